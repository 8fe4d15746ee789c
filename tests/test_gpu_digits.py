"""The FP64 scattering product in digits (rtg_scat64.cu) with its plan fixed by rtg_apply_digits, and the table that
shows which plan runs (rtg_apply_plans): so that a comparison with the FP64 pipe is one of two plans, at few angular
nodes too (one stage of 16, one row tile that is not full), where the autotuner may choose either.

Tolerance in norm as in test_gpu_scat64: 1e-14 of the terms' size."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_scat64 import CASES, _ctx

pytestmark = pytest.mark.gpu

# nodes per direction, nodes per cell, angular refinements, cells of one node more: Nth = nth 2^ang + more
SMALL = {"nth3": (3, 3, 0, 0), "nth12": (4, 3, 2, 0), "nth17": (3, 4, 2, 1), "nth40": (5, 5, 3, 0)}


def small_ctx(name, Phi=None):
    from rtg import DeviceContext, workloads as W
    from rtg.mesh import Mesh
    n, nth, ang, more = SMALL[name]
    m = Mesh([2., 2.], [False, False], [n, n, nth], True)
    for _ in range(ang):
        m.ref_mesh(kind="ang", form="h")
    for _ in range(3):
        m.ref_mesh(kind="spt", form="h")
    for ck in sorted(m.cols):
        for kk in sorted(m.cols[ck].cells)[:more]:
            m.ref_cell(ck, kk, form="p")
    spec = W.two_disc_problem()
    return DeviceContext(m, spec.kappa, spec.sigma, spec.Phi if Phi is None else Phi)


def plans(ctx, prec):
    from rtg import _lib
    table, n = np.zeros((64, 9), dtype=np.int32), C.c_int()
    _lib.check(ctx.lib.rtg_apply_plans(ctx.h, prec, _lib.ptr(table, C.c_int32), 64, C.byref(n), None))
    return table[:n.value]


def pin(ctx, digits):
    """Fixes the FP64 plan and shows that it is the one asked for."""
    from rtg import _lib
    if digits:
        _lib.check(ctx.lib.rtg_apply_digits(ctx.h, 32))
    else:
        shape = np.asarray((32, 1, 0, 0), dtype=np.int32)
        _lib.check(ctx.lib.rtg_apply_shape(ctx.h, _lib.RTG_FP64, _lib.ptr(shape, C.c_int32)))
    t = plans(ctx, _lib.RTG_FP64)
    assert [tuple(int(v) for v in r[:5]) for r in t] == [(32, 1, 0, int(digits), 1)]


def both(ctx, flags, x):
    """The product in digits (twice, equal bit by bit) and on the FP64 pipe."""
    import torch
    pin(ctx, True)
    a = ctx.apply(flags, x)
    assert torch.equal(a, ctx.apply(flags, x))
    pin(ctx, False)
    return a, ctx.apply(flags, x)


@pytest.mark.parametrize("name", sorted(CASES) + sorted(SMALL))
def test_pinned_product(name):
    import torch
    from rtg import _lib
    ctx = _ctx(name) if name in CASES else small_ctx(name)
    torch.manual_seed(0)
    x = torch.randn(ctx.N, dtype=torch.float64, device=ctx.device)
    for flags, parts in ((_lib.RTG_SYSTEM | _lib.RTG_MASK_ROWS, (_lib.RTG_MASS, _lib.RTG_SCAT)), (_lib.RTG_SCAT, (_lib.RTG_SCAT,))):
        a, r = both(ctx, flags, x)
        size = sum(float(torch.linalg.norm(ctx.apply(p, x.abs()))) for p in parts)
        assert float(torch.linalg.norm(a - r)) <= 1e-14 * size


@pytest.mark.parametrize("name", ["nth147_n6", "nth129_n7", "nth17", "nth40"])
def test_dropped_terms_are_left_out(name):
    """A beam (one angular node of x) in columns whose terms are dropped or kept by their size: where the FP64 pipe
    drops all of an output's terms, the sum is exactly zero."""
    import torch
    from rtg import DeviceContext, _lib, workloads as W
    ctx = _ctx(name) if name in CASES else small_ctx(name)
    spec = W.two_disc_problem()
    # sigma falls by 10 from strip to strip of columns, so that the drop rule cuts at every level of the kernel
    thin = DeviceContext(ctx.layout.mesh, spec.kappa, lambda x, y: 10. ** (-2. - np.floor(4. * x)) + 0. * y, spec.Phi)
    lay = thin.layout
    x = torch.zeros(thin.N, dtype=torch.float64, device=thin.device)
    rng = np.random.default_rng(0)
    for c in range(lay.ncols):
        e = int(rng.integers(lay.col_elem_start[c], lay.col_elem_start[c + 1]))
        nth = int(lay.cell_ndof[e])
        o = np.arange(int(lay.elem_off[e]) + int(rng.integers(nth)), int(lay.elem_off[e + 1]), nth)
        x[torch.as_tensor(o)] = torch.as_tensor(rng.uniform(0.5, 2., size=len(o)), device=thin.device)
    a, r = both(thin, _lib.RTG_SCAT, x)
    assert (r == 0).any() and (r != 0).any()
    assert bool((a[r == 0] == 0).all())
    assert bool((a[r != 0] != 0).all())


def _forward(th, phi):
    """A forward cone: falls by 2^57 across the circle."""
    return 3.14 * np.exp(20. * (np.cos(th - phi) - 1.))


@pytest.mark.parametrize("peaked", [False, True])
@pytest.mark.parametrize("name", ["nth256_n4", "nth147_n6", "nth160_n9", "nth17", "nth40"])
def test_every_output_against_its_own_terms(name, peaked):
    """Each output is within the rounding of an FP64 sum of its own terms, also where these are small beside the row's
    largest |W| times the node's largest |x|: a beam alone, over a floor of 1e-30, values spread over many decades.
    Both sums obey Nth 2^-53 of the sum of the terms' sizes, so twice that between them."""
    import torch
    from rtg import DeviceContext, _lib, workloads as W
    ctx = _ctx(name) if name in CASES else small_ctx(name)
    if peaked:
        spec = W.two_disc_problem()
        ctx = DeviceContext(ctx.layout.mesh, spec.kappa, spec.sigma, _forward)
    lay = ctx.layout
    nth = int(lay.cell_ndof[:lay.col_elem_start[1]].sum())
    rng = np.random.default_rng(1)
    beam = np.zeros(ctx.N)
    for c in range(lay.ncols):
        e = int(rng.integers(lay.col_elem_start[c], lay.col_elem_start[c + 1]))
        o = np.arange(int(lay.elem_off[e]) + int(rng.integers(lay.cell_ndof[e])), int(lay.elem_off[e + 1]), int(lay.cell_ndof[e]))
        beam[o] = rng.uniform(0.5, 2., size=len(o))
    noise = rng.standard_normal(ctx.N)
    xs = [torch.as_tensor(x, device=ctx.device) for x in (beam, beam + 1e-30 * noise, noise * np.exp(12. * rng.standard_normal(ctx.N)), noise)]
    pin(ctx, False)
    ref = [(ctx.apply(_lib.RTG_SCAT, x), ctx.apply(_lib.RTG_SCAT, x.abs()).abs()) for x in xs]
    pin(ctx, True)
    for x, (r, size) in zip(xs, ref):
        a = ctx.apply(_lib.RTG_SCAT, x)
        assert float(((a - r).abs() - 2. * nth * 2. ** -53 * size).max()) <= 0.


def test_tuned_table():
    """The autotuned FP64 table: one row chosen, the fastest, and the digits among the shapes of a product of 1e8."""
    from rtg import _lib
    t = plans(_ctx("nth128_n7"), _lib.RTG_FP64)
    assert int(t[:, 4].sum()) == 1 and t[t[:, 4] == 1][0][5] == t[:, 5].min()
    assert (t[:, 3] == 1).any()
    assert (t[:, 3] == 0).any()                # the FP64 pipe is timed beside them


def test_tuned_table_of_few_angles():
    """4,096 columns of 3 x 3 nodes and 12 angles: the product is large, its tiles of 128 rows are not filled."""
    from rtg import DeviceContext, _lib, workloads as W
    from rtg.mesh import Mesh
    m = Mesh([2., 2.], [False, False], [3, 3, 3], True)
    for _ in range(2):
        m.ref_mesh(kind="ang", form="h")
    for _ in range(6):
        m.ref_mesh(kind="spt", form="h")
    spec = W.two_disc_problem()
    t = plans(DeviceContext(m, spec.kappa, spec.sigma, spec.Phi), _lib.RTG_FP64)
    assert (t[:, 3] == 1).any() and (t[:, 3] == 0).any()
    assert t[t[:, 4] == 1][0][5] == t[:, 5].min()


def test_refused():
    from rtg import DeviceContext, _lib, workloads as W
    from rtg.mesh import Mesh
    m = Mesh([1., 1.], [False, False], [2, 2, 9], True)
    for _ in range(5):
        m.ref_mesh(kind="ang", form="h")       # 288 angular nodes
    spec = W.manufactured_problem()
    ctx = DeviceContext(m, spec.kappa, spec.sigma, spec.Phi)
    assert ctx.lib.rtg_apply_digits(ctx.h, 0) == _lib.RTG_ERR_ARG
    assert ctx.lib.rtg_apply_digits(ctx.h, 32) == _lib.RTG_ERR_SIZE
    assert not plans(ctx, _lib.RTG_FP64)[:, 3].any()
    assert ctx.lib.rtg_apply_digits(None, 32) == _lib.RTG_ERR_ARG

"""FP64 scattering product on the tensor cores (rtg_scat64.cu, taken for products of 1e8 multiply-adds and more)
against the FP64 pipe's (plan pinned with rtg_apply_shape), which the oracle tests hold to 1e-12.  Edges: no,
one and more rows past a 128-row tile, row counts that are no multiple of eight, 256 angular nodes (the most), node counts that fill, pad and split the 32-node
tiles, drop-rule nodes of every class, and inputs whose nodes leave the fixed-point range.

Tolerance: both sum at most 256 products of FP64 operands; the FP64 pipe's rounding is about sqrt(256) 2^-53 = 1.8e-15
of the terms' size, the digits' 2^-58 of the largest, so 1e-14 relative (the bound between plan shapes) holds."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# nodes per direction, nodes per cell, angular and spatial refinements, cells of one node more per column:
# Nth = nth 2^ang + more, 4^spt columns
CASES = {"nth256_n4": (4, 8, 5, 4, 0), "nth160_n2": (2, 5, 5, 5, 0), "nth144_n5": (5, 9, 4, 4, 0),
         "nth147_n6": (6, 9, 4, 4, 3), "nth128_n7": (7, 8, 4, 4, 0), "nth129_n7": (7, 8, 4, 4, 1),
         "nth160_n9": (9, 5, 5, 3, 0)}


def _ctx(name):
    from rtg import DeviceContext, workloads as W
    from rtg.mesh import Mesh
    n, nth, ang, spt, more = CASES[name]
    m = Mesh([2., 2.], [False, False], [n, n, nth], True)
    for _ in range(ang):
        m.ref_mesh(kind="ang", form="h")
    for _ in range(spt):
        m.ref_mesh(kind="spt", form="h")
    for ck in sorted(m.cols):
        for kk in sorted(m.cols[ck].cells)[:more]:
            m.ref_cell(ck, kk, form="p")
    # thick discs (every term kept), a thin background (terms dropped) and vacuum at x < 0.3 (no term)
    spec = W.two_disc_problem()
    sigma = lambda x, y: np.where(x < 0.3, 0., spec.sigma(x, y))   # noqa: E731
    return DeviceContext(m, spec.kappa, sigma, spec.Phi)


def _apply_both(ctx, flags, xs):
    """Results on the tensor cores (twice) and the FP64 pipe, and the size of the terms summed."""
    import torch
    from rtg import _lib
    tc = [ctx.apply(f, x) for f in flags for x in xs]
    again = [ctx.apply(f, x) for f in flags for x in xs]
    shape = np.asarray((32, 1, 0, 0), dtype=np.int32)
    _lib.check(ctx.lib.rtg_apply_shape(ctx.h, _lib.RTG_FP64, _lib.ptr(shape, C.c_int32)))
    ref = [ctx.apply(f, x) for f in flags for x in xs]
    parts = {_lib.RTG_SCAT: (_lib.RTG_SCAT,)}
    size = [sum(float(torch.linalg.norm(ctx.apply(p, x.abs()))) for p in parts.get(f, (_lib.RTG_MASS, _lib.RTG_SCAT)))
            for f in flags for x in xs]
    return tc, again, ref, size


@pytest.mark.parametrize("name", sorted(CASES))
def test_product_matches_fp64_pipe(name):
    import torch
    from rtg import _lib
    ctx = _ctx(name)
    torch.manual_seed(0)
    x = torch.randn(ctx.N, dtype=torch.float64, device=ctx.device)
    wide = x * torch.exp(6. * torch.randn(ctx.N, dtype=torch.float64, device=ctx.device))
    flags = (_lib.RTG_SYSTEM | _lib.RTG_MASK_ROWS, _lib.RTG_SCAT)
    for a, b, r, size in zip(*_apply_both(ctx, flags, (x, wide, torch.ones_like(x), torch.zeros_like(x)))):
        assert torch.equal(a, b)
        assert float(torch.linalg.norm(a - r)) <= 1e-14 * size


def test_values_outside_the_fixed_point_range():
    """Non-finite values spread as the FP64 pipe's sums spread them; nodes of 1e-300 and 1e300 keep their relative
    accuracy beside ordinary ones."""
    import torch
    from rtg import _lib
    ctx = _ctx("nth128_n7")
    torch.manual_seed(1)
    x = torch.randn(ctx.N, dtype=torch.float64, device=ctx.device)
    n = ctx.N // 4
    scaled = x.clone()
    scaled[:n] *= 1e-300
    scaled[n:2 * n] *= 1e290
    bad = x.clone()
    bad[n // 2], bad[3 * n + 5], bad[2 * n + 11] = float("nan"), float("inf"), -float("inf")
    tc, again, ref, _ = _apply_both(ctx, (_lib.RTG_SCAT,), (scaled, bad))
    for part in (slice(0, n), slice(n, 2 * n)):
        a, r = tc[0][part], ref[0][part]
        s = float(r.abs().max())
        assert s > 0. and float(torch.linalg.norm((a - r) / s)) <= 1e-14 * float(torch.linalg.norm(r / s))
    a, r = tc[1], ref[1]
    assert torch.equal(torch.isnan(a), torch.isnan(r)) and torch.equal(torch.isinf(a), torch.isinf(r))
    assert torch.isnan(r).any() or torch.isinf(r).any()
    f = torch.isfinite(r)
    assert torch.equal(a[torch.isinf(r)], r[torch.isinf(r)])
    assert float(torch.linalg.norm((a - r)[f])) <= 1e-14 * float(torch.linalg.norm(r[f]))

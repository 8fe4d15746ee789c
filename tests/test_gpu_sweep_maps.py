"""The sweep's compact upwind maps (rtg_sweep.cu) against the oracle's sweep at
the edges of their forms.  The FP32 sweep folds the angular mortars into the maps
where fewer than 128 elements share a level and forms T = Et z after the wait
otherwise; the FP64 sweep takes elements of more than two angular nodes in parts
of two.  Meshes of both kinds, of two (never in parts), three (a part of one left
over), five and eight angular nodes, with hanging faces, and with neighbouring
columns refined differently in angle (mortars that are not diagonal) or in
order (rows of several lengths on one mesh).

Tolerance: the element blocks are inverted in FP32 (about 1e-5, bound 1e-4) and
the FP32 sweep reads BF16 copies of them (about 2e-3, bound 1e-2), the bounds of
the other comparisons with the oracle's sweep."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# nodes per direction, nodes per cell, spatial and angular refinements, elements of 128 and more per level
CASES = {"dense_n2": (2, 2, 2, 6, True), "dense_n3": (4, 3, 2, 6, True), "dense_n5": (3, 5, 2, 6, True),
         "few_n3": (4, 3, 2, 2, False), "few_n5": (5, 5, 1, 3, False), "few_n8": (7, 8, 1, 3, False)}


def _mesh(name):
    from rtg.mesh import Mesh
    n, nth, spt, ang, _ = CASES[name]
    m = Mesh([2., 1.5], [False, False], [n, n, nth], True)
    for _ in range(ang):
        m.ref_mesh(kind="ang", form="h")
    for _ in range(spt):
        m.ref_mesh(kind="spt", form="h")
    cols = sorted(m.cols)
    for kk in sorted(m.cols[cols[0]].cells)[::3]:      # angularly non-conforming beside cols[1]
        m.ref_cell(cols[0], kk, form="h")
    m.ref_col(cols[1], kind="spt", form="p")           # one more node per direction than beside it
    m.ref_col(cols[-1], kind="spt", form="h")          # hanging faces
    return m


@pytest.mark.parametrize("name", sorted(CASES))
def test_maps_match_oracle_sweep(name):
    import torch
    from oracle import rt_oracle as O
    from rtg import DeviceContext, _lib, workloads as W
    mesh, spec = _mesh(name), W.smooth_variable_problem(2., 1.5)
    o = O.assemble(mesh, spec.kappa, spec.sigma, spec.Phi, spec.f, spec.bcs_dirac)
    P = O.SweepPreconditioner(o, o["layout"])
    ne, nlev = len(P.order), int(P.level.max()) + 1
    assert (ne >= 128 * nlev) == CASES[name][4], (ne, nlev)
    ctx = DeviceContext(mesh, spec.kappa, spec.sigma, spec.Phi)
    rng = np.random.default_rng(7)
    r = np.where(o["mask"], rng.standard_normal(len(o["mask"])), 0.)
    z_ref = P(r)
    for prec, tol in ((_lib.RTG_FP64, 1e-4), (_lib.RTG_FP32, 1e-2)):
        z = ctx.precondition(r, prec=prec)
        assert torch.equal(z, ctx.precondition(r, prec=prec)), (name, prec)
        err = np.linalg.norm(z.double().cpu().numpy() - z_ref) / np.linalg.norm(z_ref)
        assert err <= tol, (name, prec, err)
    ctx.close()

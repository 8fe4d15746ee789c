"""The batched solver's cycles (rtg_batch.cu) at the edges of their forms: instances
of less than one 4096-value chunk and of more than 128 (above which an instance's
sums have a launch of their own), one instance alone, restart lengths that end a
cycle before and after the instances converge, and an instance without any
right-hand side (done before the first step).

Tolerance: both solves end at a residual of 1e-11 of the right-hand side; 1e-8 is
the bound of the other comparisons of a batch with single solves."""
import pytest

pytestmark = pytest.mark.gpu


def _instances(kind):
    from rtg import workloads as W
    from rtg.mesh import Mesh
    small = [W.batch_instance(s, max_cols=8, max_cells=4, n_range=(2, 4)) for s in (3, 4, 5)]
    if kind == "small":
        return small
    m = Mesh([1., 1.], [False, False], [8, 8, 9], True)
    for _ in range(4):
        m.ref_mesh(kind="ang", form="h")
    for _ in range(3):
        m.ref_mesh(kind="spt", form="h")
    large = (m, W.gaussian_bump_problem())
    return [large] if kind == "one" else [small[0], large, small[1]]


@pytest.mark.parametrize("kind,restart", [("small", 3), ("small", 60), ("mixed", 7), ("mixed", 30), ("one", 30)])
def test_batch_matches_single_solves(kind, restart):
    import torch
    from rtg import DeviceContext
    from rtg.batch import BatchContext
    inst = _instances(kind)
    assert max(m.get_ndof() for m, _ in inst) > 128 * 4096 or kind == "small"
    bc = BatchContext(inst)
    f, g = bc.forcing(), bc.inflow()
    if len(inst) > 1:        # the last instance has nothing to solve
        f[int(bc.inst_off[-2]):] = 0.
        g[int(bc.inst_off[-2]):] = 0.
    u, infos = bc.solve(f, g, rtol=1e-11, restart=restart, max_it=6000)
    again, _ = bc.solve(f, g, rtol=1e-11, restart=restart, max_it=6000)
    assert all(i["converged"] for i in infos) and torch.equal(u, again)
    for k, (mesh, spec) in enumerate(inst):
        o0, o1 = int(bc.inst_off[k]), int(bc.inst_off[k + 1])
        if len(inst) > 1 and k == len(inst) - 1:
            assert not u[o0:o1].any()
            continue
        ctx = DeviceContext(mesh, spec.kappa, spec.sigma, spec.Phi)
        ref, info = ctx.solve(f[o0:o1].contiguous(), g[o0:o1].contiguous(), method=0, precond=1, rtol=1e-11, max_it=2000)
        assert info["converged"]
        assert float(torch.linalg.norm(u[o0:o1] - ref)) <= 1e-8 * float(torch.linalg.norm(ref)), (kind, k)
        ctx.close()

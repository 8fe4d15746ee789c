"""The FP32 apply's outputs (rtg_apply.cu) over the degrees its loops are unrolled
for (3 to 8 nodes per direction), those next to them (2, 9) and unequal degrees,
each term on its own and the masked system, with the scattering product in the
tiled kernel and on the tensor cores, against the FP64 apply.

Tolerance: FP32 rounding of sums of at most some hundred terms of mixed sign and
the TF32 hi/lo split, 2e-6 of the result, the bound between plan shapes; the
streaming terms alone cancel up to tenfold, 2e-5, the bound of the other FP32
comparisons with the operator."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nth", [(2, 2, 4), (3, 3, 3), (4, 4, 1), (5, 5, 5), (6, 6, 3), (7, 7, 2), (8, 8, 4),
                                       (9, 9, 3), (4, 6, 3), (7, 3, 2)])
def test_fp32_apply_matches_fp64(nx, ny, nth):
    import torch
    from rtg import DeviceContext, _lib, workloads as W
    from rtg.mesh import Mesh
    m = Mesh([2., 1.5], [False, False], [nx, ny, nth], True)
    for _ in range(3):
        m.ref_mesh(kind="ang", form="h")
    for _ in range(2):
        m.ref_mesh(kind="spt", form="h")
    cols = sorted(m.cols)
    for kk in sorted(m.cols[cols[0]].cells)[::3]:      # mortars in angle
        m.ref_cell(cols[0], kk, form="h")
    m.ref_col(cols[1], kind="spt", form="p")           # mortars in space
    m.ref_col(cols[-1], kind="spt", form="h")
    spec = W.smooth_variable_problem(2., 1.5)
    ctx = DeviceContext(m, spec.kappa, spec.sigma, spec.Phi)
    torch.manual_seed(0)
    x = torch.randn(ctx.N, dtype=torch.float64, device=ctx.device).float()
    for shape in ((64, 1, 0, 0), (16, 0, 0, 0), (16, 1, 0, 2), (64, 0, 0, 2)):
        arr = np.asarray(shape, dtype=np.int32)
        _lib.check(ctx.lib.rtg_apply_shape(ctx.h, _lib.RTG_FP32, _lib.ptr(arr, C.c_int32)))
        for flags, tol in ((_lib.RTG_SYSTEM | _lib.RTG_MASK_ROWS, 2e-5), (_lib.RTG_MASS, 2e-6), (_lib.RTG_SCAT, 2e-6),
                           (_lib.RTG_IC, 2e-5), (_lib.RTG_BC, 2e-5)):
            ref = ctx.apply(flags, x.double())
            y = ctx.apply(flags, x, prec=_lib.RTG_FP32).double()
            assert float(torch.linalg.norm(y - ref)) <= tol * float(torch.linalg.norm(ref)), (shape, flags)
    ctx.close()

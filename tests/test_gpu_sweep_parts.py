"""The records of the FP64 sweep's parts (two angular nodes of an element each) are made for the first FP64 sweep: a
handle that sweeps in FP32 alone does not hold them."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_parts_come_with_the_first_fp64_sweep():
    import torch
    from rtg import DeviceContext, _lib, workloads as W
    from rtg.mesh import Mesh

    def sweep(ctx, dtype):
        r = torch.ones(ctx.N, dtype=dtype, device=ctx.device)
        z = torch.empty_like(r)
        prec = _lib.RTG_FP64 if dtype == torch.float64 else _lib.RTG_FP32
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        _lib.check(ctx.lib.rtg_precondition(ctx.h, prec, C.c_void_p(r.data_ptr()), C.c_void_p(z.data_ptr()), None))
        torch.cuda.synchronize()
        return free - torch.cuda.mem_get_info()[0], z

    spec = W.two_disc_problem()

    def handle(spt):
        m = Mesh([2., 2.], [False, False], [4, 4, 5], True)
        for _ in range(5):
            m.ref_mesh(kind="ang", form="h")
        for _ in range(spt):
            m.ref_mesh(kind="spt", form="h")
        return DeviceContext(m, spec.kappa, spec.sigma, spec.Phi)

    first = handle(1)                    # loads the kernels
    sweep(first, torch.float32)
    sweep(first, torch.float64)
    ctx = handle(4)                      # 8,192 elements of 5 angular nodes: three parts each
    sweep(ctx, torch.float32)
    grew, z = sweep(ctx, torch.float64)
    assert grew >= 8192 * 3 * 64 * 4     # a record has 64 words at least
    again, z2 = sweep(ctx, torch.float64)
    assert again <= 0 and torch.equal(z, z2)

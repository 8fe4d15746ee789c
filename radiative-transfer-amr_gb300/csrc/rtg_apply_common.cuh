// Device helpers shared by the apply kernels.
#pragma once

#include "rtg_internal.h"

namespace rtg {

__device__ __forceinline__ bool bdry_node(int bm, int i, int j, int nx, int ny) {
    return ((bm & 1) && i == nx - 1) || ((bm & 2) && j == ny - 1) || ((bm & 4) && i == 0) ||
           ((bm & 8) && j == 0);
}

struct ApplyFlags {
    bool scat, mass, merged, ic, bc, mask_rows;
    float ic_sign;
};

__device__ __forceinline__ ApplyFlags decode(uint32_t flags) {
    ApplyFlags f;
    const bool sys = flags & RTG_SYSTEM;
    f.scat = sys || (flags & RTG_SCAT);
    f.mass = sys || (flags & RTG_MASS);
    f.merged = f.scat && f.mass;   // (M - S) block with the joint drop rule
    f.ic = sys || (flags & RTG_IC);
    f.ic_sign = sys ? -1.f : 1.f;
    f.bc = sys || (flags & RTG_BC);
    f.mask_rows = flags & RTG_MASK_ROWS;
    return f;
}

// bounded wait for the completion of phase `parity` of an mbarrier
__device__ __forceinline__ bool mbar_wait(uint32_t mb, uint32_t parity) {
    uint32_t done = 0;
    for (int spin = 0; spin < (1 << 22) && !done; ++spin)
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mb), "r"(parity)
            : "memory");
    return done != 0;
}

}  // namespace rtg

"""The digit tables of the FP64 scattering product (rtg_scat64.cu) when device memory runs out while they are made:
build_scat64 gives back what it has and returns null, so that the FP64 pipe's plans stand alone, as for a W that the
digits cannot hold.  Host code with the allocator replaced; no GPU."""
import os
import subprocess

import golden_io  # noqa: F401  (puts the package on the path)
from rtg import build

MAIN = r"""
#include <cstdio>
#include <cuda_runtime.h>
static int left = 0, live = 0;
template <typename T>
cudaError_t short_malloc(T** p, size_t n) {
    if (left-- <= 0) return cudaErrorMemoryAllocation;
    *p = (T*)malloc(n);
    ++live;
    return cudaSuccess;
}
static cudaError_t short_free(void* p) {
    free(p);
    --live;
    return cudaSuccess;
}
static cudaError_t no_copy() { return cudaSuccess; }
#define cudaMalloc(p, n) short_malloc(p, n)
#define cudaFree(p) short_free(p)
#define cudaMemcpy(...) no_copy()
#define cudaMemset(...) no_copy()
#include "rtg_scat64.cu"
namespace rtg {
void set_error(const std::string&) {}
void raise_smem_limit(const void*, size_t) {}
std::atomic<long long>& launch_counter() { static std::atomic<long long> n{0}; return n; }
}
int main() {
    rtg_handle h;
    rtg::ColDev c{};
    c.nx = c.ny = 2;
    c.nth_col = 4;
    h.host.cols.push_back(c);
    h.host.sig_nth.push_back(4);
    h.host.nnodes = 4;
    const uint8_t cls[4] = {1, 1, 2, 2};
    const uint64_t thr[4] = {0, 0, 1, 1};
    for (int n = 0; n < 12; ++n) {   // fewer than it makes: it never reaches its kernels
        left = n;
        try {
            if (rtg::build_scat64(&h, {1}, cls, thr, nullptr)) return 1;
        } catch (const rtg::RtgError& e) {
            printf("allocation %d: %s\n", n, e.msg.c_str());
            return 2;
        }
        if (live) return 3;
    }
    return 0;
}
"""


def test_out_of_memory_means_no_digits(tmp_path):
    main = tmp_path / "main.cu"
    main.write_text(MAIN)
    exe = str(tmp_path / "main")
    r = subprocess.run([build.nvcc()] + build.ARCH + ["-std=c++17", "--expt-relaxed-constexpr", "-I", build.INCLUDE, "-I", build.CSRC,
                                                      str(main), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, env=dict(os.environ, CUDA_VISIBLE_DEVICES=""))
    assert r.returncode == 0, (r.returncode, r.stdout)

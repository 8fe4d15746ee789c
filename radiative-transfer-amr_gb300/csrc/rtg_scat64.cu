// FP64 scattering product on the tensor cores.
//
// Y[R][ij] = sum_c W[R][c] x[c][ij] over a column's angular nodes is the dense
// contraction of the FP64 apply, and GB300 runs FP64 at 2 FMAs per SM and
// clock: on the FP64 pipe the product took 3.3 of the 4.07 ms of an apply at
// 7.95e6 DOF.  Here every operand is a sum of ten signed 8-bit digits (the
// splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012, with
// fixed-point digits): a row of W and a node's line of x are scaled by the
// power of two of their largest entry to 78-bit fixed point, whose balanced
// digits d_1 .. d_10 (|d_1| <= 64, |d_k| <= 128) are exact in FP16.  A digit
// product is an integer of at most 2^14, and D_s = sum over i + j = s of W_i x_j,
// s = 2 .. 11, accumulates in FP32 in tensor memory, without rounding for s <= 10:
// set-up checks on the digits of W that |D_s| <= 2^24 for every x (random digits
// of 270 angular nodes reach it; a column has at most 256).  The epilogue adds the
// ten integers in 80 bits and rounds once: T in units of 2^-82 to 2^-84 of
// |W|_max |x|_max.
//
// What is left out (s >= 12, and W and x below 2^-78 of their largest entry) is
// at most 578 + 128 of these units for every x that is not zero in fixed point, 64 for
// one that only fixed point makes zero, and
// D_11, if it passes 2^24, is off by at most 2 a multiply, 320.  Against the FP64 sum
// of a row that is small only where the sum is not itself small beside |W|_max
// |x|_max: so an output below 2^52 times that (kOzLost, kOzTiny, kOzRound; 2^-12 of
// the largest product at 256 nonzero x) is summed again, term by term in FP64: one in a
// few thousand outputs for random x.  The apply at 7.95e6 DOF takes 1407 us for
// random x, 1744 for a solution, 2273 for a beam in every column, 3329 for
// randn exp(12 randn); 4230 on the FP64 pipe.
// Every other output is within 2^-52 of the sum of its terms, as an FP64 sum of so
// many terms is not.  With eight digits and no second sum the apply
// at 7.95e6 DOF took 1286 us, but a beam's terms were off by 1e-13 of
// their size for the g = 0.95 kernel and 3e-7 for exp(20 (cos - 1)).
//
// Drop rule (rt/preconditioner_matrix.py:450-495): a node of class 2 keeps the
// terms with |W| >= t.  The nodes of a CTA share one threshold (a column has few:
// the four or eight nodes of a symmetric rule share theirs), and the digits of
// the dropped entries are cleared in shared memory before they are multiplied, so
// a dropped term is left out exactly.  The test |W| < t runs on FP32
// copies; the thresholds are moved at set-up to where the rounded test decides
// as the exact one.  Nodes for which none does (two W entries of one FP32 value
// on both sides of t), nodes with a non-finite x and nodes with max |x| outside
// [2^-823, 2^977] are summed term by term in the same way.
//
// One CTA takes up to 128 rows and 24 nodes of a column: 10 accumulators of 24
// columns fill half of the tensor memory, so two CTAs share an SM and one
// stages while the other multiplies.  B holds the digits of x stacked along N
// (row np (j - 1) + n, np the nodes rounded up to 8), so that one tcgen05.mma
// multiplies W_i with x_1 .. x_{11-i} into D_{i+1} .. D_11, which lie next to each
// other: 10 instructions per 16 angular nodes in place of 55.
#include <algorithm>
#include <cstring>
#include <map>
#include <vector>

#include "rtg_apply_common.cuh"
#include "rtg_scat64.h"

namespace rtg {

namespace {

constexpr int kOzThreads = 256;
constexpr int kOzM = 128;        // rows of a CTA (TMEM lanes)
constexpr int kOzN = 24;         // nodes of a CTA, at most
constexpr int kOzK = 16;         // angular nodes per stage: one tcgen05.mma step
constexpr int kOzD = 10;         // digits
// what an x, one that is zero in fixed point, and the sum may be off by (units of T)
constexpr int kOzLost = 710, kOzTiny = 64, kOzRound = 512;
constexpr int kOzMaxNth = 256;   // angular nodes a column may have (bound of the FP32 sums)
constexpr int kRowBytes = kOzD * kOzK * 2;            // digits of a row of W per stage
constexpr int kABytes = kOzM * kRowBytes;
constexpr int kBBytes = kOzD * kOzN * kOzK * 2;
constexpr int kOzSmem = 2 * (kABytes + kBBytes) + kOzMaxNth * (int)sizeof(int2);

struct OzItem {
    int32_t col, row0, rows, n0, nn;        // rows row0 .. row0 + rows - 1, nodes perm[n0] .. perm[n0 + nn - 1] of one threshold
    int64_t tile;                           // first byte of the row tile's digits of W
    int64_t wrange;                         // first of the row tile's |W| ranges (per stage, eight groups of 16 rows)
};

__device__ __forceinline__ uint64_t oz_desc(uint32_t addr) {
    const uint64_t lbo = 128, sbo = 256;   // canonical K-major, no swizzle: core matrices along K, 8-row groups
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((lbo >> 4) << 16) | ((sbo >> 4) << 32) | (1ull << 46);
}

__device__ __forceinline__ void oz_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, int acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

// The ten balanced digits of Q, v = Q 2^(E - 1100), |Q| < 2^78, for |v| < 2^(E - 1022),
// E >= 1 (bits below 2^(E - 1100) cut off), each plus 128: d_1 .. d_8 in the bytes of u,
// d_1 on top, d_9 and d_10 in the lower two of w
struct OzDigits {
    unsigned long long u;
    uint32_t w;
    __device__ bool zero() const { return u == 0x8080808080808080ull && w == 0x8080u; }
};
__device__ __forceinline__ OzDigits oz_digits(double v, int E) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    int e = (int)(b >> 52) & 0x7FF;
    unsigned long long m = b & 0xFFFFFFFFFFFFFull;
    if (e) m |= 1ull << 52;
    else e = 1;
    m <<= 9;
    const int sh = E - e;   // Q = m 2^16 >> sh, in 62 and 16 bits
    long long hi = sh < 63 ? (long long)(m >> sh) : 0ll;
    int lo = (int)(sh < 16 ? m << (16 - sh) : sh < 79 ? m >> (sh - 16) : 0ull) & 0xFFFF;
    if ((long long)b < 0) {
        hi = -hi;
        lo = -lo;
    }
    const int w = lo + 0x8080;   // the carry into d_8 above 16 bits
    OzDigits d;
    d.u = ((unsigned long long)(hi + (w >> 16)) + 0x0080808080808080ull) ^ 0x8000000000000000ull;
    d.w = (uint32_t)w & 0xFFFFu;
    return d;
}

// digits k (bytes k of u and w) as FP16, exactly: 1024 + byte - 1152
__device__ __forceinline__ uint32_t oz_pair(uint32_t u, uint32_t w, int k) {
    const uint32_t b = (__byte_perm(u, w, ((unsigned)(4 + k) << 8) | (unsigned)k) & 0x00FF00FFu) | 0x64006400u;
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(b), "r"(0x64806480u));
    return d;
}
// digit j + 1 of both
__device__ __forceinline__ uint32_t oz_pair(const OzDigits& a, const OzDigits& b, int j) {
    return j < 4   ? oz_pair((uint32_t)(a.u >> 32), (uint32_t)(b.u >> 32), 3 - j)
           : j < 8 ? oz_pair((uint32_t)a.u, (uint32_t)b.u, 7 - j)
                   : oz_pair(a.w, b.w, 9 - j);
}

// hi 2^40 + lo rounded once, for |hi| < 2^58 and 0 <= lo < 2^40, with two FP64 operations
// (the pipe takes 16 cycles for each of a warp's): its upper and lower parts
// are put into the mantissas of 3 2^99 (one unit 2^48) and of 2^52 (one unit 1)
__device__ __forceinline__ double oz_double(long long hi, long long lo) {
    const double a = __longlong_as_double(0x4638000000000000ll + (hi >> 8));
    const double b = __longlong_as_double(0x4330000000000000ll | ((hi & 0xFF) << 40) | lo);
    return (a - (0x1.8p100 + 0x1p52)) + b;
}

// v 2^e for v zero or normal, with v 2^e normal (integer work alone)
__device__ __forceinline__ double oz_times_pow2(double v, int e) {
    const int hi = __double2hiint(v);
    return (hi << 1) ? __hiloint2double(hi + (e << 20), __double2loint(v)) : v;
}

// 2^e as a double, -1022 <= e <= 1023
__host__ __device__ __forceinline__ double oz_pow2(int e) {
    const unsigned long long b = (unsigned long long)(e + 1023) << 52;
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double d;
    std::memcpy(&d, &b, 8);
    return d;
#endif
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// Warps 0-7 stage x, clear the dropped entries of W and write y; warp 8 brings
// the digits of W in, one stage ahead, and issues the multiplies.
__global__ void __launch_bounds__(kOzThreads + 32, 2)
scat64_kernel(OpView<double> v, uint32_t flags, const OzItem* __restrict__ items,
              const unsigned char* __restrict__ digits, const float4* __restrict__ w32, const int* __restrict__ frow,
              const int64_t* __restrict__ sig_row, const float2* __restrict__ wrange,
              const uint8_t* __restrict__ perm, const uint64_t* __restrict__ thr, const float* __restrict__ thr32,
              const double* __restrict__ x, double* __restrict__ y, int* __restrict__ status) {
    extern __shared__ __align__(128) unsigned char osm[];
    __shared__ __align__(8) uint64_t s_bar[6];   // W arrived 0, 1; multiplied 0, 1; x staged 0, 1
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort, s_need, s_nlist;
    __shared__ uint8_t s_any[kOzM];    // row keeps a term
    __shared__ unsigned s_max[kOzN];
    __shared__ int s_E[kOzN];          // exponent field of the node's largest |x|; 0: node not in the product
    __shared__ float2 s_wr[kOzMaxNth / kOzK][8];   // range of |W| per stage and 16 rows
    __shared__ int s_node[kOzN];       // node in the column
    __shared__ double s_g[kOzN];       // -cw 2^(E - 1064); 0: nothing to add
    __shared__ double s_cw[kOzN];      // -cw
    __shared__ int s_off[kOzN];        // units of T that the node's sums may be off by
    after_trigger();
    const OzItem it = items[blockIdx.x];
    const ColDev C = v.cols[it.col];
    const bool mask_rows = flags & RTG_MASK_ROWS;
    const int nij = C.nx * C.ny, Nth = C.nth_col, ncell = C.elem_end - C.elem_begin;
    const int np = (it.nn + 7) & ~7;
    const int tcols = np <= 8 ? 128 : 256;
    const int rows8 = (it.rows + 7) & ~7;
    const int nch = (Nth + kOzK - 1) / kOzK;
    unsigned char* As = osm;
    unsigned char* Bs = As + 2 * kABytes;
    // per angular row: DOF offset in the column; nth and, from bit 8, the inflow-boundary faces of its cell
    int2* s_row = reinterpret_cast<int2*>(Bs + 2 * kBBytes);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(s_bar);
    const unsigned char* wsrc = digits + it.tile;
    const uint32_t stage = (uint32_t)rows8 * kRowBytes;   // bytes of a stage: the digits of the rows
    const float4* w32t = w32 + it.tile / kRowBytes * (kOzK / 4);   // their FP32 copies, per stage [kOzK / 4][rows8]
    const uint32_t as_addr = (uint32_t)__cvta_generic_to_shared(As);
    // the CTA's threshold (0: nothing is dropped; NaN: term by term)
    const float thr_cta = thr32[C.node_off + perm[it.n0]];
    // node tid's constant (loaded before it is needed)
    double cw = 0.;
    float lo = INFINITY;   // smallest |W| of stage tid - 32
    if (tid < kOzN) {
        s_max[tid] = 0u;
        const int ij = perm[it.n0 + min(tid, it.nn - 1)];   // the pad nodes repeat the last (their x is zero)
        s_node[tid] = ij;
        cw = v.colc[it.col] * v.sw[C.node_off + ij];
        s_cw[tid] = -cw;
        s_off[tid] = kOzRound;
    } else if (tid >= 32 && tid - 32 < nch) {
        for (int q = 0; q < 8; ++q) {
            const float2 w = wrange[it.wrange + 8 * (tid - 32) + q];
            s_wr[tid - 32][q] = w;
            lo = fminf(lo, w.x);
        }
    }
    // the column's rows
    for (int k = warp; k < ncell; k += kOzThreads / 32 + 1) {
        const ElemDev E = v.elems[C.elem_begin + k];
        const int off = nij * E.row;
        for (int r = lane; r < E.nth; r += 32) s_row[E.row + r] = make_int2(off + r, E.nth | (E.flags >> 4) << 8);
    }
    // the tables are constant; the flags, x and y belong to the kernels ahead, whose last
    // waves these loads ran beside (with the launch, 58 -> 53 us for an apply of 218,581
    // DOF, 255 -> 249 at 1.95e6)
    after_wait();
    if ((v.stop && *v.stop) || (v.skip && v.skip[it.col])) return;
    if (tid == 0) {
        s_abort = 0;
        s_need = 0;
        s_nlist = 0;
        for (int q = 0; q < 6; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar + 8 * q), "r"(q < 4 ? 1 : kOzThreads / 32)
                         : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // the first stages' digits travel while the tables are made
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        bulk_load(as_addr, wsrc, stage, bar);
        if (nch > 1) bulk_load(as_addr + kABytes, wsrc + stage, stage, bar + 8);
    }
    if (warp == 8) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&s_tmem);
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(tcols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    // the stages in which some |W| is dropped
    if (lo < thr_cta) atomicOr(&s_need, 1 << (tid - 32));
    if (tid < kOzM) s_any[tid] = 0;
    // per node the largest |x|: a lane takes a node and, where few nodes share the
    // CTA, a warp several cells at once (apply at 7.95e6 DOF 1448 -> 1405 us)
    const double* xc = x + C.dof_off;
    const int cells = 32 / np, node = lane - lane / np * np;
    if (lane < cells * np && node < it.nn) {
        unsigned mx = 0;
        for (int k = warp * cells + lane / np; k < ncell; k += (kOzThreads / 32 + 1) * cells) {
            const ElemDev E = v.elems[C.elem_begin + k];
            const double* xk = xc + nij * E.row + s_node[node] * E.nth;
#pragma unroll 4
            for (int r = 0; r < E.nth; ++r) {
                const double xv = xk[r];
                const unsigned hi = (unsigned)__double2hiint(xv) & 0x7FFFFFFFu;
                mx = max(mx, hi ? hi : (__double2loint(xv) ? 1u : 0u));
            }
        }
        atomicMax(&s_max[node], mx);
    }
    __syncthreads();
    if (tid < kOzN) {
        int E = 0;
        double g = 0.;
        if (tid < it.nn) {
            const unsigned mx = s_max[tid];
            const int e = (int)(mx >> 20);
            if (e < 200 || e > 2000 || thr_cta != thr_cta) {
                g = mx ? -cw : 0.;          // summed term by term below, or x is zero
            } else {
                E = e;
                g = -cw * oz_pow2(e - 1064);
            }
        }
        s_E[tid] = E;
        s_g[tid] = g;
    }
    __syncthreads();
    const int needs = s_need;
    bool ok = true;
    if (warp == 8) {
        // kind::f16: D F32 (bits 4-5 = 1), A and B FP16 (bits 7-9, 10-12 = 0), K-major, N >> 3 at bit 17, M >> 4 at 24
        const uint32_t idesc0 = (1u << 4) | ((uint32_t)(kOzM >> 4) << 24);
        if (lane == 0) {
            for (int ch = 0; ch < nch && ok; ++ch) {
                const int b = ch & 1;
                const uint32_t par = (uint32_t)((ch >> 1) & 1);
                ok = mbar_wait(bar + 32 + 8 * b, par) && mbar_wait(bar + 8 * b, par);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t aa = as_addr + b * kABytes;
                const uint64_t db = oz_desc((uint32_t)__cvta_generic_to_shared(Bs + b * kBBytes));
#pragma unroll
                for (int i = 0; i < kOzD; ++i) {
                    const uint32_t n = (uint32_t)(((kOzD - i) * np + 15) & ~15);   // columns past D_11 are not read
                    oz_mma(tmem + (uint32_t)(i * np), oz_desc(aa + (uint32_t)(i * rows8 * 32)), db,
                           idesc0 | ((n >> 3) << 17), ch > 0 || i > 0);
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 bar + 16 + 8 * b)
                             : "memory");
                // stage ch - 1 multiplied: its W buffer takes stage ch + 1 (0 and 1 are on their way)
                if (ch >= 1 && ch + 1 < nch) {
                    ok = mbar_wait(bar + 16 + 8 * (b ^ 1), (uint32_t)(((ch - 1) >> 1) & 1));
                    if (ok)
                        bulk_load(as_addr + (b ^ 1) * kABytes, wsrc + (int64_t)(ch + 1) * stage, stage, bar + 8 * (b ^ 1));
                }
            }
            if (!ok) s_abort = 1;
        }
        __syncwarp();
    } else {
        // thread -> (two angular nodes, one node): ten digits of each into B
        const int kp = 8 * (warp & 1) + 2 * (lane & 3), nb = 8 * (warp >> 1) + (lane >> 2);
        const bool bact = nb < np;
        const int En = bact ? s_E[nb] : 0, ijn = s_node[min(nb, kOzN - 1)];
        auto load_x = [&](int c) -> double {
            if (!En || c >= Nth) return 0.;
            const int2 ro = s_row[c];
            return xc[ro.x + ijn * (ro.y & 0xFF)];
        };
        const uint32_t boff = (uint32_t)((nb >> 3) * 256 + (kp >> 3) * 128 + (nb & 7) * 16 + (kp & 7) * 2);
        // thread -> (row mr, eight angular nodes from 8 mh) of the entries it may clear
        const int mr = tid & (kOzM - 1), mh = tid >> 7;
        float4 wa{}, wb{};
        bool any = false;   // the row keeps one of them
        auto load_w = [&](int ch) {
            if (mr >= rows8 || ch >= nch || !(needs >> ch & 1)) return;
            const float4* p = w32t + ((int64_t)ch * (kOzK / 4) + 2 * mh) * rows8 + mr;
            wa = p[0];
            wb = p[rows8];
        };
        load_w(0);
        double x0 = load_x(kp), x1 = load_x(kp + 1);
        int off = 0;
        for (int ch = 0; ch < nch; ++ch) {
            const int b = ch & 1, c0 = ch * kOzK;
            unsigned char* Bb = Bs + b * kBBytes;
            // stage ch - 2 has been multiplied: its buffers are free
            if (ch >= 2 && !mbar_wait(bar + 16 + 8 * b, (uint32_t)(((ch >> 1) - 1) & 1))) {
                s_abort = 1;
                ok = false;
            }
            if (bact) {
                const OzDigits d0 = oz_digits(x0, max(En, 1)), d1 = oz_digits(x1, max(En, 1));   // x is zero where En is
                off += d0.zero() ? (x0 != 0. ? kOzTiny : 0) : kOzLost;
                off += d1.zero() ? (x1 != 0. ? kOzTiny : 0) : kOzLost;
#pragma unroll
                for (int j = 0; j < kOzD; ++j)
                    *reinterpret_cast<uint32_t*>(Bb + boff + j * np * 32) = oz_pair(d0, d1, j);
            }
            if (needs >> ch & 1) {
                // the digits of the dropped entries: cleared once they are there
                ok = mbar_wait(bar + 8 * b, (uint32_t)((ch >> 1) & 1)) && ok;
                if (mr < rows8 && s_wr[ch][mr >> 4].x < thr_cta) {
                    auto kept = [&](float a, float c) {
                        return (fabsf(a) >= thr_cta ? 0xFFFFu : 0u) | (fabsf(c) >= thr_cta ? 0xFFFF0000u : 0u);
                    };
                    const uint4 k4 = make_uint4(kept(wa.x, wa.y), kept(wa.z, wa.w), kept(wb.x, wb.y), kept(wb.z, wb.w));
                    any |= (k4.x | k4.y | k4.z | k4.w) != 0u;
                    unsigned char* p = As + b * kABytes + (mr >> 3) * 256 + mh * 128 + (mr & 7) * 16;
#pragma unroll
                    for (int k = 0; k < kOzD; ++k) {
                        uint4* q = reinterpret_cast<uint4*>(p + k * rows8 * 32);
                        uint4 d = *q;
                        d.x &= k4.x;
                        d.y &= k4.y;
                        d.z &= k4.z;
                        d.w &= k4.w;
                        *q = d;
                    }
                } else {
                    any = true;
                }
            } else {
                any = true;
            }
            // generic-proxy writes -> visible to the tensor cores
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar + 32 + 8 * b) : "memory");
            x0 = load_x(c0 + kOzK + kp);
            x1 = load_x(c0 + kOzK + kp + 1);
            load_w(ch + 1);
        }
        if (any) s_any[mr] = 1;
        if (off) atomicAdd(&s_off[nb], off);
        if (!ok) s_abort = 1;
    }
    // the last commit follows every multiply of the CTA
    if (ok && !mbar_wait(bar + 16 + 8 * ((nch - 1) & 1), (uint32_t)(((nch - 1) >> 1) & 1))) s_abort = 1;
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (s_abort) {
        // give the copies and multiplies in flight one more bounded wait each before the memory is let go
        for (int q = 0; q < 2; ++q) {
            mbar_wait(bar + 8 * q, 0);
            mbar_wait(bar + 16 + 8 * q, 0);
        }
        if (tid == 0 && status) atomicExch(status, RTG_ERR_TIMEOUT);
    } else {
        const int q = warp & 3, h = warp >> 2;
        const int m = 32 * q + lane, R = it.row0 + m;
        const bool valid = warp < 8 && m < it.rows;
        const int2 ro = s_row[valid ? R : it.row0];
        const int fr = valid ? frow[sig_row[C.sig] + R] : 0;
        const int nth = ro.y & 0xFF, bm = mask_rows ? ro.y >> 8 : 0;
        const float rny = __frcp_rn((float)C.ny);
        // rows of inflow-boundary nodes stay zero under RTG_MASK_ROWS
        auto masked = [&](int ij) {
            const int i = small_div(ij, rny);
            return bm && bdry_node(bm, i, ij - i * C.ny, C.nx, C.ny);
        };
        double* yc = y + C.dof_off;
        // outputs to be summed again, row + 256 node (the buffers are free)
        uint16_t* s_list = reinterpret_cast<uint16_t*>(As);
        auto again = [&](int n) { s_list[atomicAdd(&s_nlist, 1)] = (uint16_t)(m | n << 8); };
        for (int cb = 4 * h; cb < np && warp < 8; cb += 8) {
            uint32_t d[kOzD][4];
#pragma unroll
            for (int k = 0; k < kOzD; ++k)
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(d[k][0]), "=r"(d[k][1]), "=r"(d[k][2]), "=r"(d[k][3])
                             : "r"(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(k * np + cb))
                             : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (!valid) continue;
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                const int n = cb + jj;
                if (n >= it.nn || s_g[n] == 0.) continue;
                const int ij = s_node[n];
                if (masked(ij)) continue;
                if (!s_E[n]) {
                    again(n);
                    continue;
                }
                long long H = 0, L = 0;
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    H = (H << 8) + __float2int_rn(__uint_as_float(d[k][jj]));
                    L = (L << 8) + __float2int_rn(__uint_as_float(d[k + 5][jj]));
                }
                H += L >> 40;
                if (llabs(H) < (long long)s_off[n] << 12) {   // units of 2^40: |T| below 2^52 times that
                    if (s_any[m]) again(n);   // else every term is dropped
                    continue;
                }
                const double s = oz_times_pow2(oz_double(H, L & 0xFFFFFFFFFFll), fr);
                atomicAdd(yc + ro.x + ij * nth, s * s_g[n]);
            }
        }
        __syncthreads();
        // eight lanes per output: the kept terms one by one (the bits of |W| against the
        // threshold).  A warp per output spends half of its FP64 operations on the sum of the
        // lanes' parts (randn exp(12 randn) at 7.95e6 DOF: 5537 us in place of 3353)
        const int lane8 = lane & 7;
        for (int i0 = 4 * warp; i0 < s_nlist; i0 += 4 * (kOzThreads / 32 + 1)) {
            const int i = i0 + (lane >> 3);
            const int at = s_list[min(i, s_nlist - 1)], n = at >> 8, Ra = it.row0 + (at & 0xFF), ij = s_node[n];
            const double* Wr = v.W + v.W_off[C.sig] + (int64_t)Ra * Nth;
            const unsigned long long tb = thr[C.node_off + ij];
            double s = 0.;
#pragma unroll 4
            for (int c = lane8; c < Nth; c += 8) {
                const double w = Wr[c];
                const bool keep = c != Ra && ((unsigned long long)__double_as_longlong(w) & 0x7FFFFFFFFFFFFFFFull) >= tb;
                const int2 rc = s_row[c];
                s = fma(keep ? w : 0., xc[rc.x + ij * (rc.y & 0xFF)], s);
            }
            for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            const int2 ra = s_row[Ra];
            if (lane8 == 0 && i < s_nlist) atomicAdd(yc + ra.x + ij * (ra.y & 0xFF), s * s_cw[n]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 8) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tcols) : "memory");
    }
}

// One block per row of a distinct W: its digits into the row tile's image (per
// stage of kOzK columns: digit, 8-row group, 8-column group, row, column), its FP32
// copy (per stage four columns of every row together), its
// scale, and the range of the nonzero off-diagonal |W| per stage and 16 rows.  bad: an entry is not
// finite, the row's largest is outside [2^-100, 2^100], or the digits allow an x whose D_2 .. D_10 pass 2^24.
__global__ void oz_digits_kernel(const double* __restrict__ W, const float* __restrict__ W32,
                                 const int64_t* __restrict__ W_off, const int2* __restrict__ rows,
                                 const int64_t* __restrict__ sig_tile, const int64_t* __restrict__ sig_wrange,
                                 const int32_t* __restrict__ sig_n, unsigned char* __restrict__ out,
                                 float* __restrict__ out32, int* __restrict__ frow, float2* __restrict__ wrange, int* __restrict__ bad) {
    __shared__ unsigned long long s_mx[4];
    __shared__ int s_sum[kOzD];   // sum of the |d_i|
    const int sg = rows[blockIdx.x].x, R = rows[blockIdx.x].y, n = sig_n[sg];
    const double* w = W + W_off[sg] + (int64_t)R * n;
    unsigned long long mx = 0;
    for (int c = threadIdx.x; c < n; c += blockDim.x)
        if (c != R) mx = max(mx, (unsigned long long)__double_as_longlong(w[c]) & 0x7FFFFFFFFFFFFFFFull);
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) s_mx[threadIdx.x >> 5] = mx;
    if (threadIdx.x < kOzD) s_sum[threadIdx.x] = 0;
    __syncthreads();
    for (int q = 0; q < (int)blockDim.x / 32; ++q) mx = max(mx, s_mx[q]);
    const int E = (int)(mx >> 52);
    const bool ok = mx == 0 || (E >= 923 && E <= 1123);
    if (threadIdx.x == 0) {
        if (!ok) atomicExch(bad, 1);
        frow[blockIdx.x] = ok && mx ? E - 1064 : 0;
    }
    if (!ok || !mx) return;   // the digits stay zero
    const int mt = R / kOzM, rr = R % kOzM, nch = (n + kOzK - 1) / kOzK;
    const int rows8 = (min(kOzM, n - mt * kOzM) + 7) & ~7;
    const int64_t at = sig_tile[sg] + (int64_t)mt * nch * kOzM * kRowBytes;
    unsigned char* tile = out + at;
    float* tile32 = out32 + at / kRowBytes * kOzK;
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
        if (c == R) continue;
        const OzDigits u = oz_digits(w[c], E);
        unsigned char* st = tile + (int64_t)(c / kOzK) * rows8 * kRowBytes;
        unsigned char* p = st + (rr >> 3) * 256 + ((c % kOzK) >> 3) * 128 + (rr & 7) * 16 + (c & 7) * 2;
#pragma unroll
        for (int k = 0; k < kOzD; ++k) {
            *reinterpret_cast<uint16_t*>(p + k * rows8 * kOzK * 2) = (uint16_t)oz_pair(u, u, k);
            const int byte = (int)(k < 8 ? u.u >> (8 * (7 - k)) : u.w >> (8 * (9 - k))) & 0xFF;
            atomicAdd(&s_sum[k], abs(byte - 128));
        }
        const float w32 = W32[W_off[sg] + (int64_t)R * n + c];
        tile32[((int64_t)(c / 4) * rows8 + rr) * 4 + (c & 3)] = w32;
        const float a = fabsf(w32);
        if (a > 0.f) {
            float2* wr = wrange + sig_wrange[sg] + 8 * ((int64_t)mt * nch + c / kOzK) + (rr >> 4);
            atomicMin(reinterpret_cast<int*>(&wr->x), __float_as_int(a));
            atomicMax(reinterpret_cast<int*>(&wr->y), __float_as_int(a));
        }
    }
    __syncthreads();
    if (threadIdx.x >= 2 && threadIdx.x <= 10) {
        int most = 0;   // of |D_s|, s = threadIdx.x
        for (int i = 1; i < (int)threadIdx.x; ++i) most += s_sum[i - 1] * (i == (int)threadIdx.x - 1 ? 64 : 128);
        if (most > 1 << 24) atomicExch(bad, 1);
    }
}

// One block per class-2 node: the FP32 threshold that decides |W| >= t as the
// FP64 one does (rounding to FP32 is monotone, so only W that round to the
// same value as t are in doubt); NaN when W of that value lie on both sides.
__global__ void oz_threshold_kernel(const double* __restrict__ W, const int64_t* __restrict__ W_off,
                                    const int32_t* __restrict__ sig_n, const int2* __restrict__ nodes,
                                    const uint64_t* __restrict__ thr, float* __restrict__ thr32) {
    const int node = nodes[blockIdx.x].x, sg = nodes[blockIdx.x].y, n = sig_n[sg];
    const double t = __longlong_as_double((long long)thr[node]);
    const float f = (float)t;
    const double* w = W + W_off[sg];
    bool lo = false, hi = false;
    for (int64_t q = threadIdx.x; q < (int64_t)n * n; q += blockDim.x) {
        const double a = fabs(w[q]);
        if ((float)a != f || q % (n + 1) == 0) continue;   // the diagonal is not tested
        if (a < t) lo = true;
        else hi = true;
    }
    const int any_lo = __syncthreads_or(lo), any_hi = __syncthreads_or(hi);
    if (threadIdx.x == 0)
        thr32[node] = any_lo ? (any_hi ? __int_as_float(0x7FC00000) : __int_as_float(__float_as_int(f) + 1)) : f;
}

}  // namespace

struct Scat64 {
    OzItem* d_items = nullptr;
    int nitems = 0;
    unsigned char* d_digits = nullptr;
    float* d_w32 = nullptr;
    int* d_frow = nullptr;   // per row: exponent of its scale
    int64_t* d_sig_row = nullptr;
    float2* d_wrange = nullptr;
    float* d_thr32 = nullptr;
    uint8_t* d_perm = nullptr;
    const uint64_t* d_thr = nullptr;
    int* d_status = nullptr;
    std::vector<void*> allocs;
};

bool scat64_fits(const ColDev& C) { return C.nth_col <= kOzMaxNth; }

Scat64* build_scat64(const rtg_handle* h, const std::vector<char>& cols, const uint8_t* scls, const uint64_t* thr,
                     const uint64_t* d_thr) {
    const HostTables& t = h->host;
    const int nsig = (int)t.sig_nth.size();
    std::vector<char> used(nsig, 0);
    for (size_t c = 0; c < cols.size(); ++c)
        if (cols[c]) used[t.cols[c].sig] = 1;
    std::vector<int64_t> sig_tile(nsig, 0), sig_wrange(nsig, 0), sig_row(nsig, 0);
    std::vector<int2> rows;
    int64_t bytes = 0, nw = 0;
    for (int s = 0; s < nsig; ++s) {
        if (!used[s]) continue;
        const int n = t.sig_nth[s], nch = (n + kOzK - 1) / kOzK;
        sig_tile[s] = bytes;
        sig_wrange[s] = nw;
        sig_row[s] = (int64_t)rows.size();
        for (int r = 0; r < n; ++r) rows.push_back(make_int2(s, r));
        for (int r0 = 0; r0 < n; r0 += kOzM) {
            bytes += (int64_t)((std::min(kOzM, n - r0) + 7) & ~7) * nch * kRowBytes;
            nw += 8 * nch;
        }
    }
    std::vector<OzItem> items;
    std::vector<int2> nodes;
    std::vector<uint8_t> perm;
    std::vector<int64_t> cost(nsig, 0);
    for (int ci = 0; ci < (int)t.cols.size(); ++ci) {
        if (!cols[ci]) continue;
        const ColDev& C = t.cols[ci];
        const int nij = C.nx * C.ny, nch = (C.nth_col + kOzK - 1) / kOzK;
        // the nodes whose product is used, by threshold; a CTA takes nodes of one
        std::vector<uint8_t> ord;
        for (int q = 0; q < nij; ++q) {
            const uint8_t cls = scls[C.node_off + q];
            if (cls == 1 || cls == 2) ord.push_back((uint8_t)q);
            if (cls == 2) nodes.push_back(make_int2(C.node_off + q, C.sig));
        }
        std::stable_sort(ord.begin(), ord.end(),
                         [&](uint8_t a, uint8_t b) { return thr[C.node_off + a] < thr[C.node_off + b]; });
        const int na = (int)ord.size(), p0 = (int)perm.size();
        perm.insert(perm.end(), ord.begin(), ord.end());
        for (int g0 = 0, g1; g0 < na; g0 = g1) {
            for (g1 = g0; g1 < na && thr[C.node_off + ord[g1]] == thr[C.node_off + ord[g0]];) ++g1;
            const int ntl = (g1 - g0 + kOzN - 1) / kOzN, per = (g1 - g0 + ntl - 1) / ntl;
            for (int n0 = g0; n0 < g1; n0 += per)
                for (int r0 = 0; r0 < C.nth_col; r0 += kOzM) {
                    const int mt = r0 / kOzM;
                    items.push_back(OzItem{ci, r0, std::min(kOzM, C.nth_col - r0), p0 + n0, std::min(per, g1 - n0),
                                           sig_tile[C.sig] + (int64_t)mt * nch * kOzM * kRowBytes,
                                           sig_wrange[C.sig] + 8 * (int64_t)mt * nch});
                    cost[C.sig] += (int64_t)nch * kOzM;
                }
        }
    }
    // the CTAs that read one row tile run next to each other, so that its
    // digits come from L2 after the first
    std::stable_sort(items.begin(), items.end(), [&](const OzItem& a, const OzItem& b) {
        const int sa = t.cols[a.col].sig, sb = t.cols[b.col].sig;
        if (cost[sa] != cost[sb]) return cost[sa] > cost[sb];
        if (sa != sb) return sa < sb;
        return a.row0 < b.row0;
    });
    struct NoRoom {};
    Scat64* p = new Scat64();
    try {
        auto alloc = [&](size_t n) -> void* {
            void* d = nullptr;
            const cudaError_t e = cudaMalloc(&d, std::max<size_t>(n, 16));
            if (e == cudaErrorMemoryAllocation) throw NoRoom{};
            RTG_CUDA(e);
            p->allocs.push_back(d);
            return d;
        };
        auto up = [&](const void* src, size_t n) -> void* {
            void* d = alloc(n);
            if (n) RTG_CUDA(cudaMemcpy(d, src, n, cudaMemcpyHostToDevice));
            return d;
        };
        p->nitems = (int)items.size();
        p->d_items = (OzItem*)up(items.data(), sizeof(OzItem) * items.size());
        p->d_digits = (unsigned char*)alloc((size_t)bytes);
        p->d_w32 = (float*)alloc((size_t)bytes / kRowBytes * kOzK * sizeof(float));
        p->d_frow = (int*)alloc(sizeof(int) * rows.size());
        p->d_sig_row = (int64_t*)up(sig_row.data(), sizeof(int64_t) * nsig);
        p->d_wrange = (float2*)alloc(sizeof(float2) * (size_t)nw);
        p->d_thr32 = (float*)alloc(sizeof(float) * std::max<size_t>((size_t)t.nnodes, 1));
        p->d_status = (int*)alloc(sizeof(int));
        p->d_perm = (uint8_t*)up(perm.data(), perm.size());
        p->d_thr = d_thr;
        int2* d_rows = (int2*)up(rows.data(), sizeof(int2) * rows.size());
        int2* d_nodes = (int2*)up(nodes.data(), sizeof(int2) * nodes.size());
        int64_t* d_st = (int64_t*)up(sig_tile.data(), sizeof(int64_t) * nsig);
        int64_t* d_sw = (int64_t*)up(sig_wrange.data(), sizeof(int64_t) * nsig);
        int32_t* d_n = (int32_t*)up(t.sig_nth.data(), sizeof(int32_t) * nsig);
        int* d_bad = (int*)alloc(sizeof(int));
        RTG_CUDA(cudaMemset(p->d_status, 0, sizeof(int)));
        RTG_CUDA(cudaMemset(d_bad, 0, sizeof(int)));
        RTG_CUDA(cudaMemset(p->d_digits, 0, (size_t)bytes));
        RTG_CUDA(cudaMemset(p->d_w32, 0, (size_t)bytes / kRowBytes * kOzK * sizeof(float)));
        const std::vector<float2> none((size_t)nw, make_float2(3.4e38f, 0.f));
        RTG_CUDA(cudaMemcpy(p->d_wrange, none.data(), sizeof(float2) * (size_t)nw, cudaMemcpyHostToDevice));
        RTG_CUDA(cudaMemset(p->d_thr32, 0, sizeof(float) * (size_t)t.nnodes));
        if (!rows.empty()) {
            oz_digits_kernel<<<(int)rows.size(), 128>>>(h->v64.W, h->v32.W, h->v64.W_off, d_rows, d_st, d_sw, d_n,
                                                        p->d_digits, p->d_w32, p->d_frow, p->d_wrange, d_bad), count_launch();
            RTG_LAUNCHED("oz_digits_kernel");
        }
        if (!nodes.empty()) {
            oz_threshold_kernel<<<(int)nodes.size(), 256>>>(h->v64.W, h->v64.W_off, d_n, d_nodes, d_thr, p->d_thr32),
                count_launch();
            RTG_LAUNCHED("oz_threshold_kernel");
        }
        int bad = 0;
        RTG_CUDA(cudaMemcpy(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost));
        if (bad) {
            free_scat64(p);
            return nullptr;
        }
        raise_smem_limit((const void*)scat64_kernel, kOzSmem);
    } catch (const NoRoom&) {   // the FP64 pipe needs none of this
        cudaGetLastError();
        free_scat64(p);
        return nullptr;
    } catch (...) {
        free_scat64(p);
        throw;
    }
    return p;
}

void free_scat64(Scat64* p) {
    if (!p) return;
    for (void* d : p->allocs) cudaFree(d);
    delete p;
}

void launch_scat64(const Scat64* p, const OpView<double>& v, uint32_t flags, const double* x,
                   double* y, cudaStream_t s) {
    if (!p->nitems) return;
    launch_after(scat64_kernel, p->nitems, kOzThreads + 32, kOzSmem, s, v, flags, p->d_items, p->d_digits,
                 reinterpret_cast<const float4*>(p->d_w32), p->d_frow,
                 p->d_sig_row, p->d_wrange, p->d_perm, p->d_thr, p->d_thr32, x, y, p->d_status);
}

int* scat64_status(const Scat64* p) { return p->d_status; }

}  // namespace rtg

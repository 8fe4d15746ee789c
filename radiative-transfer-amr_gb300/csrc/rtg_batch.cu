// Batched solve of many independent RT instances held by one handle.
//
// The instances' meshes are concatenated into one mesh description (no
// couplings between instances), so every operator apply and every sweep
// covers all instances in one launch.  The Krylov state is per instance:
// inner products are segmented by instance, the Hessenberg matrix, Givens
// rotations and convergence flags of each instance live on the device and
// are updated by one thread per instance, and a converged instance's basis is
// frozen.  The start of a GMRES restart cycle, each Arnoldi step and the end
// (the correction and its sweep) are fixed kernel sequences, captured once in
// CUDA graphs and replayed; the host queues step j + 1, then reads whether step j
// finished the last instance, so the GPU never waits for it and a cycle runs at
// most one step (whose launches return at once) too many.  A cycle that always ran its
// m = 30 steps spent 40 % of the solve of 64 instances of 72,000 DOF on steps with
// nothing left to do.
//
// method 1 (the batched workload's method): FP64 iterative refinement around
// FP32 sweep-preconditioned GMRES; method 0: FP64 GMRES.
//
// Instances converge at different iterations; a finished instance costs
// nothing for the rest of the cycle: per-column skip flags (refreshed inside
// the captured cycle from the per-instance flags) make the operator apply and
// the sweep leave its columns out, and the vector kernels leave out its
// chunks.  Its frozen basis columns and correction are never read again.
#include <chrono>
#include <cmath>
#include <type_traits>
#include <vector>

#include "rtg_internal.h"

namespace rtg {

namespace {

constexpr int kBChunk = 4096;
constexpr int kBThreads = 256;
constexpr int kBGroup = 8;

struct BChunk {
    int64_t begin, end;
    int32_t inst, pad;
};

// partials of <v, v> per chunk (FP64), bound by reading v; the general kernel's
// reductions for eight products took 103 us at 4.65e6 values
__global__ void __launch_bounds__(kBThreads)
bnorm_kernel(const BChunk* __restrict__ ch, const double* __restrict__ v, double* __restrict__ partial) {
    __shared__ double red[kBThreads / 32];
    const BChunk c = ch[blockIdx.x];
    double s = 0.;
#pragma unroll 8
    for (int64_t i = c.begin + threadIdx.x; i < c.end; i += kBThreads) s = fma(v[i], v[i], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.;
        for (int wq = 0; wq < kBThreads / 32; ++wq) t += red[wq];
        partial[blockIdx.x] = t;
    }
}

// out[b*ldo + q] = sum of the partials of instance b
__global__ void breduce_kernel(const int32_t* __restrict__ cbeg, const double* __restrict__ partial, int k,
                               double* __restrict__ out, int ldo) {
    const int b = blockIdx.x, q = blockIdx.y;
    double s = 0.;
    for (int c = cbeg[b] + threadIdx.x; c < cbeg[b + 1]; c += blockDim.x) s += partial[(int64_t)c * k + q];
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.;
        for (int wq = 0; wq < (int)(blockDim.x + 31) / 32; ++wq) t += red[wq];
        out[b * ldo + q] = t;
    }
}

// The partials of an Arnoldi step's sums: k values each, those of instance b from
// beg[b] to beg[b + 1].  Every block that needs an instance's sums adds them itself (in one
// order, so all get the same), which saves a launch of 4.5 us between two passes of
// 10; above kOwnSums partials per instance breduce_kernel leaves one.  With instances
// of up to 92 partials the solve takes 11.62 ms with the launch and 11.31 without.
struct BSums {
    const double* partial;
    const int32_t* beg;
};
constexpr int kOwnSums = 128;

// out[q] = the sums of instance b, for the block's threads
__device__ __forceinline__ void inst_sums(BSums sums, int b, int k, double* out) {
    const int lane = threadIdx.x & 31, c0 = sums.beg[b], c1 = sums.beg[b + 1];
    for (int q = threadIdx.x >> 5; q < k; q += kBThreads / 32) {
        double s = 0.;
        for (int c = c0 + lane; c < c1; c += 32) s += sums.partial[(int64_t)c * k + q];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) out[q] = s;
    }
    __syncthreads();
}

// A chunk of a vector in the block's registers
constexpr int kBPer = kBChunk / kBThreads;
__device__ __forceinline__ void load_chunk(float (&w)[kBPer], const float* __restrict__ p, int n) {
#pragma unroll
    for (int u = 0; u < kBPer; ++u) w[u] = (int)threadIdx.x + u * kBThreads < n ? p[threadIdx.x + u * kBThreads] : 0.f;
}
__device__ __forceinline__ void store_chunk(const float (&w)[kBPer], float* __restrict__ p, int n) {
#pragma unroll
    for (int u = 0; u < kBPer; ++u)
        if ((int)threadIdx.x + u * kBThreads < n) p[threadIdx.x + u * kBThreads] = w[u];
}
// w -= sum_{q<k} h[q] V_q
__device__ __forceinline__ void axpy_chunk(float (&w)[kBPer], const float* __restrict__ V, int64_t ldv, int k,
                                           const double* h, int n) {
    for (int q = 0; q < k; ++q) {
        float v[kBPer];
        load_chunk(v, V + (int64_t)q * ldv, n);
        const float hq = (float)h[q];
#pragma unroll
        for (int u = 0; u < kBPer; ++u) w[u] = fmaf(-hq, v[u], w[u]);
    }
}
// partial of <w, w>: per element and warp in FP32, double from the warps' sums on
__device__ __forceinline__ void norm_chunk(const float (&w)[kBPer], double* partial) {
    __shared__ double red[kBThreads / 32];
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < kBPer; ++u) s = fmaf(w[u], w[u], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = (double)s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.;
        for (int wq = 0; wq < kBThreads / 32; ++wq) t += red[wq];
        *partial = t;
    }
}
// partials of <V_q, w>, q < k
__device__ __forceinline__ void dot_chunk(const float (&w)[kBPer], const float* __restrict__ V, int64_t ldv, int k,
                                          int n, double* partial) {
    __shared__ double red[kBGroup][kBThreads / 32];
    for (int g0 = 0; g0 < k; g0 += kBGroup) {
        const int gk = min(kBGroup, k - g0);
        float acc[kBGroup];
#pragma unroll
        for (int q = 0; q < kBGroup; ++q) {
            acc[q] = 0.f;
            if (q < gk) {
                float v[kBPer];
                load_chunk(v, V + (int64_t)(g0 + q) * ldv, n);
#pragma unroll
                for (int u = 0; u < kBPer; ++u) acc[q] = fmaf(v[u], w[u], acc[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < kBGroup; ++q) {
            float sw = acc[q];
            for (int o = 16; o > 0; o >>= 1) sw += __shfl_down_sync(0xffffffffu, sw, o);
            if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = (double)sw;
        }
        __syncthreads();
        if (threadIdx.x < gk) {
            double s = 0.;
            for (int wq = 0; wq < kBThreads / 32; ++wq) s += red[threadIdx.x][wq];
            partial[g0 + threadIdx.x] = s;
        }
        __syncthreads();
    }
}

// w = rhs - s and its norm's partials
__global__ void __launch_bounds__(kBThreads)
bresid_kernel(const BChunk* __restrict__ ch, const float* __restrict__ rhs, const float* __restrict__ sv,
              float* __restrict__ w, double* __restrict__ partial) {
    const BChunk c = ch[blockIdx.x];
    const int n = (int)(c.end - c.begin);
    float a[kBPer], b[kBPer];
    load_chunk(a, rhs + c.begin, n);
    load_chunk(b, sv + c.begin, n);
#pragma unroll
    for (int u = 0; u < kBPer; ++u) a[u] -= b[u];
    store_chunk(a, w + c.begin, n);
    norm_chunk(a, partial + blockIdx.x);
}

// The passes of classical Gram-Schmidt with reorthogonalisation over the k basis
// vectors of the chunk's instance, w in registers: <V, w>; then w -= V h1 and
// <V, w> again; then w -= V h2 and <w, w>.  Each is bound by reading V (twice in
// the second, the second time from L2 or L1).
__global__ void __launch_bounds__(kBThreads)
bdots_kernel(const BChunk* __restrict__ ch, const float* __restrict__ V, int64_t ldv, int k,
             const float* __restrict__ w, double* __restrict__ partial, const int32_t* __restrict__ done) {
    after_trigger();
    after_wait();
    const BChunk c = ch[blockIdx.x];
    if (done[c.inst]) return;
    const int n = (int)(c.end - c.begin);
    float wr[kBPer];
    load_chunk(wr, w + c.begin, n);
    dot_chunk(wr, V + c.begin, ldv, k, n, partial + (int64_t)blockIdx.x * k);
}

__global__ void __launch_bounds__(kBThreads)
baxpy_dots_kernel(const BChunk* __restrict__ ch, const int32_t* __restrict__ cbeg, BSums sums,
                  const float* __restrict__ V, int64_t ldv, int k, float* __restrict__ w, double* __restrict__ h1,
                  int ldh, double* __restrict__ partial, const int32_t* __restrict__ done) {
    __shared__ double h[64];
    after_trigger();
    after_wait();
    const BChunk c = ch[blockIdx.x];
    if (done[c.inst]) return;
    const int n = (int)(c.end - c.begin);
    float wr[kBPer];
    load_chunk(wr, w + c.begin, n);
    inst_sums(sums, c.inst, k, h);
    if (cbeg[c.inst] == (int)blockIdx.x && threadIdx.x < k) h1[c.inst * ldh + threadIdx.x] = h[threadIdx.x];
    axpy_chunk(wr, V + c.begin, ldv, k, h, n);
    store_chunk(wr, w + c.begin, n);
    dot_chunk(wr, V + c.begin, ldv, k, n, partial + (int64_t)blockIdx.x * k);
}

// ho = h1 + h2
__global__ void __launch_bounds__(kBThreads)
baxpy_norm_kernel(const BChunk* __restrict__ ch, const int32_t* __restrict__ cbeg, BSums sums,
                  const float* __restrict__ V, int64_t ldv, int k, float* __restrict__ w,
                  const double* __restrict__ h1, double* __restrict__ ho, int ldh, double* __restrict__ partial,
                  const int32_t* __restrict__ done) {
    __shared__ double h[64];
    after_trigger();
    after_wait();
    const BChunk c = ch[blockIdx.x];
    if (done[c.inst]) return;
    const int n = (int)(c.end - c.begin);
    float wr[kBPer];
    load_chunk(wr, w + c.begin, n);
    inst_sums(sums, c.inst, k, h);
    if (cbeg[c.inst] == (int)blockIdx.x && threadIdx.x < k)
        ho[c.inst * ldh + threadIdx.x] = h[threadIdx.x] + h1[c.inst * ldh + threadIdx.x];
    axpy_chunk(wr, V + c.begin, ldv, k, h, n);
    store_chunk(wr, w + c.begin, n);
    norm_chunk(wr, partial + blockIdx.x);
}

// out = w / ||w||, the norm into nrm[b*ldn] (first chunk of b), and the sentinel
// over z, the output of the sweep that follows (its claim counter is reset by the
// step kernels below)
__global__ void __launch_bounds__(kBThreads)
bnormalize_kernel(const BChunk* __restrict__ ch, const int32_t* __restrict__ cbeg, BSums sums,
                  const float* __restrict__ w, float* __restrict__ out, double* __restrict__ nrm, int ldn,
                  float* __restrict__ z, const int32_t* __restrict__ done) {
    __shared__ double s_sq;
    __shared__ float s_inv;
    after_trigger();
    after_wait();
    const BChunk c = ch[blockIdx.x];
    if (done && done[c.inst]) return;
    inst_sums(sums, c.inst, 1, &s_sq);
    if (threadIdx.x == 0) {
        const double nr = sqrt(s_sq);
        s_inv = (float)(nr > 0. ? 1. / nr : 0.);
        if (cbeg[c.inst] == (int)blockIdx.x) nrm[c.inst * ldn] = nr;
    }
    __syncthreads();
    const float inv = s_inv;
    Sentinel<float>::U* zq = reinterpret_cast<Sentinel<float>::U*>(z);
    for (int64_t i = c.begin + threadIdx.x; i < c.end; i += blockDim.x) {
        out[i] = w[i] * inv;
        zq[i] = Sentinel<float>::bits;
    }
}

// x = sum_{q < kb[b]} y[b][q] V_q, and the sentinel over z for the sweep of x
__global__ void __launch_bounds__(kBThreads)
bcombine_kernel(const BChunk* __restrict__ ch, float* __restrict__ x, const float* __restrict__ V, int64_t ldv,
                const int32_t* __restrict__ kb, const double* __restrict__ y, int ldy, float* __restrict__ z) {
    const BChunk c = ch[blockIdx.x];
    const int k = kb[c.inst];
    if (k == 0) return;
    Sentinel<float>::U* zq = reinterpret_cast<Sentinel<float>::U*>(z);
    for (int64_t i = c.begin + threadIdx.x; i < c.end; i += blockDim.x) {
        float sv = 0.f;
        for (int q = 0; q < k; ++q) sv = fmaf((float)y[c.inst * ldy + q], V[(int64_t)q * ldv + i], sv);
        x[i] = sv;
        zq[i] = Sentinel<float>::bits;
    }
}

// y = a[b] * x + beta * y  (a per instance; a == nullptr means ascal); a zero
// coefficient drops its term without reading it (uninitialised buffers)
template <typename TX, typename TY>
__global__ void bscale_kernel(const BChunk* __restrict__ ch, const TX* __restrict__ x, TY* __restrict__ y,
                              const double* __restrict__ a, int lda, double ascal, double beta) {
    using A = typename std::conditional<sizeof(TX) == 4 && sizeof(TY) == 4, float, double>::type;
    const BChunk c = ch[blockIdx.x];
    const double s = a ? a[c.inst * lda] : ascal;
    const A sa = (A)s, ba = (A)beta;
    for (int64_t i = c.begin + threadIdx.x; i < c.end; i += blockDim.x)
        y[i] = (TY)((s == 0. ? A(0) : sa * (A)x[i]) + (beta == 0. ? A(0) : ba * (A)y[i]));
}

// What one restart cycle knows of its instances, on the device
struct BState {
    double *H, *cs, *sn, *g, *est, *y;
    const double* tol;
    int32_t *kvalid, *done;
    int32_t* ndone;                // instances that are done, then 1 once all are (stop): [2]
    unsigned int* next;            // the sweep's claim counter
    const int32_t* col_beg;        // first column of instance b (columns of an instance are contiguous)
    int32_t* skip;                 // columns that products and sweeps leave out
    int nb, m;
};

// Columns of instance b skipped or not; the block's threads
__device__ __forceinline__ void set_skip(const BState& st, int b, int skip) {
    for (int c = st.col_beg[b] + threadIdx.x; c < st.col_beg[b + 1]; c += blockDim.x) st.skip[c] = skip;
}
__device__ __forceinline__ void count_done(const BState& st, int b) {
    st.done[b] = 1;
    if (atomicAdd(st.ndone, 1) == st.nb - 1) st.ndone[1] = 1;
}

// Start of a restart cycle, one block per instance: beta = ||r||, g = (beta, 0...).
__global__ void bstart_kernel(BState st, const double* __restrict__ nrm) {
    const int b = blockIdx.x, m = st.m;
    const double beta = nrm[b];
    const bool fin = beta <= st.tol[b];
    for (int q = threadIdx.x; q <= m; q += blockDim.x) st.g[b * (m + 1) + q] = q ? 0. : beta;
    set_skip(st, b, fin);
    if (threadIdx.x == 0) {
        if (b == 0) *st.next = 0u;
        st.kvalid[b] = 0;
        st.done[b] = 0;
        if (fin) count_done(st, b);
    }
}

// Arnoldi step j, one block per instance: store the new Hessenberg column, apply the
// previous Givens rotations, form the new one, update g and the residual estimate;
// freeze the instance and skip its columns once converged.
__global__ void barnoldi_kernel(BState st, int j, const double* __restrict__ ho, int ldh) {
    after_trigger();
    after_wait();
    const int b = blockIdx.x, m = st.m;
    if (b == 0 && threadIdx.x == 0) *st.next = 0u;
    if (st.done[b]) return;
    __shared__ int s_fin;
    if (threadIdx.x == 0) {
        double* hc = st.H + (int64_t)b * (m + 1) * m + (int64_t)j * (m + 1);
        const double* hb = ho + b * ldh;
        double* c = st.cs + b * m;
        double* s = st.sn + b * m;
        double a0 = hb[0];
        for (int q = 0; q < j; ++q) {
            const double a1 = hb[q + 1];
            hc[q] = c[q] * a0 + s[q] * a1;
            a0 = -s[q] * a0 + c[q] * a1;
        }
        const double a1 = hb[j + 1];
        const double rr = hypot(a0, a1);
        c[j] = rr > 0. ? a0 / rr : 1.;
        s[j] = rr > 0. ? a1 / rr : 0.;
        hc[j] = rr;
        hc[j + 1] = 0.;
        double* gg = st.g + b * (m + 1);
        const double gj = gg[j];
        gg[j + 1] = -s[j] * gj;
        gg[j] = c[j] * gj;
        const double e = fabs(gg[j + 1]);
        st.est[b] = e;
        st.kvalid[b] = j + 1;
        s_fin = e <= st.tol[b] || rr == 0. || !isfinite(e);
        if (s_fin) count_done(st, b);
    }
    __syncthreads();
    if (s_fin) set_skip(st, b, 1);
}

// y = H^{-1} g on the kvalid columns of each instance (back substitution), and
// the columns of instances without a correction skipped
__global__ void bsolve_kernel(BState st) {
    const int b = blockIdx.x, m = st.m;
    const int k = st.kvalid[b];
    set_skip(st, b, k == 0);
    if (threadIdx.x) return;
    if (b == 0) *st.next = 0u;
    const double* Hb = st.H + (int64_t)b * (m + 1) * m;
    double* yb = st.y + b * m;
    for (int q = k - 1; q >= 0; --q) {
        double acc = st.g[b * (m + 1) + q];
        for (int cc = q + 1; cc < k; ++cc) acc -= Hb[(int64_t)cc * (m + 1) + q] * yb[cc];
        const double d = Hb[(int64_t)q * (m + 1) + q];
        yb[q] = d != 0. ? acc / d : 0.;
    }
}

// d += z on the chunks of instances that formed a correction this cycle
__global__ void badd_kernel(const BChunk* __restrict__ ch, const float* __restrict__ z, float* __restrict__ d,
                            const int32_t* __restrict__ kvalid) {
    const BChunk c = ch[blockIdx.x];
    if (kvalid[c.inst] == 0) return;
    for (int64_t i = c.begin + threadIdx.x; i < c.end; i += blockDim.x) d[i] += z[i];
}

}  // namespace

struct BatchWs {
    int nb = 0, m = 0, nchunks = 0;
    int64_t N = 0;
    std::vector<int64_t> off;      // instance offsets
    BChunk* d_ch = nullptr;
    int32_t* d_cbeg = nullptr;
    double *b = nullptr, *r = nullptr, *x = nullptr, *t = nullptr, *gb = nullptr;
    float *V32 = nullptr, *w32 = nullptr, *z32 = nullptr, *s32 = nullptr, *d32 = nullptr, *rhs32 = nullptr;
    double *partial = nullptr, *partial2 = nullptr, *rsum = nullptr, *h1 = nullptr, *ho = nullptr, *nsq = nullptr;
    double *tin = nullptr, *scale = nullptr, *vnorm = nullptr;
    int32_t* d_one = nullptr;      // 0, 1, .., nb: one partial per instance
    bool own_sums = true;          // blocks add their instance's partials (kOwnSums)
    BState st{};
    int32_t* hstop = nullptr;      // per step, pinned: every instance is done
    cudaEvent_t ev[2] = {};
    std::vector<cudaGraphExec_t> graphs;   // start, m steps, end
    std::vector<long long> graph_kernels;  // kernels one replay runs
    std::vector<void*> allocs;
};

namespace {

template <typename T>
T* balloc(BatchWs* w, size_t n) {
    void* p = nullptr;
    RTG_CUDA(cudaMalloc(&p, sizeof(T) * std::max<size_t>(n, 1)));
    w->allocs.push_back(p);
    return (T*)p;
}

void drop_graphs(BatchWs* w) {
    for (cudaGraphExec_t g : w->graphs) cudaGraphExecDestroy(g);
    w->graphs.clear();
    w->graph_kernels.clear();
}

void free_bws(BatchWs* w) {
    if (!w) return;
    drop_graphs(w);
    for (cudaEvent_t e : w->ev)
        if (e) cudaEventDestroy(e);
    if (w->hstop) cudaFreeHost(w->hstop);
    for (void* p : w->allocs) cudaFree(p);
    delete w;
}

// per-instance squared norms into out[b*ldo]
void bnorm2(const BatchWs* w, const double* v, double* out, int ldo, cudaStream_t s) {
    bnorm_kernel<<<w->nchunks, kBThreads, 0, s>>>(w->d_ch, v, w->partial), count_launch();
    breduce_kernel<<<dim3(w->nb, 1), 128, 0, s>>>(w->d_cbeg, w->partial, 1, out, ldo), count_launch();
}

// the sums of the partials p (k per chunk), for blocks that need one instance's
BSums sums_of(const BatchWs* w, const double* p, int k, cudaStream_t s) {
    if (w->own_sums) return {p, w->d_cbeg};
    breduce_kernel<<<dim3(w->nb, k), 128, 0, s>>>(w->d_cbeg, p, k, w->rsum, k), count_launch();
    return {w->rsum, w->d_one};
}

// Part of one restart cycle of batched FP32 GMRES for A d = rhs32, sweep right
// preconditioned, d updated in place: 0 the start, 1 + j Arnoldi step j, m + 1 the
// end; each a fixed kernel sequence.
void record_part(rtg_handle* h, BatchWs* w, int part, cudaStream_t s) {
    const int m = w->m, nb = w->nb, nc = w->nchunks;
    const int64_t N = w->N;
    const int ldh = m + 2;
    const int* stop = w->st.ndone + 1;
    if (part == 0) {
        // w = rhs - A d ; V0 = w / ||w|| ; start
        launch_apply<float>(h, h->v32, RTG_SYSTEM | RTG_MASK_ROWS, w->d32, w->s32, s);
        RTG_CUDA(cudaMemsetAsync(w->st.ndone, 0, 2 * sizeof(int32_t), s));
        bresid_kernel<<<nc, kBThreads, 0, s>>>(w->d_ch, w->rhs32, w->s32, w->w32, w->partial), count_launch();
        const BSums sums = sums_of(w, w->partial, 1, s);
        bnormalize_kernel<<<nc, kBThreads, 0, s>>>(w->d_ch, w->d_cbeg, sums, w->w32, w->V32, w->nsq, 1, w->z32,
                                                   nullptr), count_launch();
        bstart_kernel<<<nb, 128, 0, s>>>(w->st, w->nsq), count_launch();
    } else if (part <= m) {
        const int j = part - 1, k = j + 1;
        float* vj = w->V32 + (int64_t)j * N;
        OpView<float> v = h->v32;       // the operator with the batch's column skip flags
        v.skip = w->st.skip;
        v.stop = stop;
        apply_sweep<float>(h, vj, w->z32, s, nullptr, w->st.skip, stop, true);
        launch_apply<float>(h, v, RTG_SYSTEM | RTG_MASK_ROWS, w->z32, w->w32, s);
        // CGS2 with per-instance coefficients; ho = h1 + h2
        if (apply_chains(h, RTG_FP32))
            launch_after(bdots_kernel, nc, kBThreads, 0, s, w->d_ch, w->V32, N, k, w->w32, w->partial, w->st.done);
        else
            bdots_kernel<<<nc, kBThreads, 0, s>>>(w->d_ch, w->V32, N, k, w->w32, w->partial, w->st.done), count_launch();
        BSums sums = sums_of(w, w->partial, k, s);
        launch_after(baxpy_dots_kernel, nc, kBThreads, 0, s, w->d_ch, w->d_cbeg, sums, w->V32, N, k, w->w32, w->h1, ldh,
                     w->partial2, w->st.done);
        sums = sums_of(w, w->partial2, k, s);
        launch_after(baxpy_norm_kernel, nc, kBThreads, 0, s, w->d_ch, w->d_cbeg, sums, w->V32, N, k, w->w32, w->h1,
                     w->ho, ldh, w->partial, w->st.done);
        sums = sums_of(w, w->partial, 1, s);
        launch_after(bnormalize_kernel, nc, kBThreads, 0, s, w->d_ch, w->d_cbeg, sums, w->w32, vj + N, w->ho + k, ldh,
                     w->z32, w->st.done);
        launch_after(barnoldi_kernel, nb, 128, 0, s, w->st, j, w->ho, ldh);
        RTG_CUDA(cudaMemcpyAsync(w->hstop + j, stop, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    } else {
        // d += P^{-1} (V y), for the instances that formed a correction
        bsolve_kernel<<<nb, 128, 0, s>>>(w->st), count_launch();
        bcombine_kernel<<<nc, kBThreads, 0, s>>>(w->d_ch, w->s32, w->V32, N, w->st.kvalid, w->st.y, m, w->z32), count_launch();
        apply_sweep<float>(h, w->s32, w->z32, s, nullptr, w->st.skip, nullptr, true);
        badd_kernel<<<nc, kBThreads, 0, s>>>(w->d_ch, w->z32, w->d32, w->st.kvalid), count_launch();
    }
}

void capture_parts(rtg_handle* h, BatchWs* w) {
    cudaStream_t cap;
    RTG_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    for (int part = 0; part <= w->m + 1; ++part) {
        cudaGraph_t graph;
        const long long n0 = launch_counter().load();
        RTG_CUDA(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
        record_part(h, w, part, cap);
        RTG_CUDA(cudaStreamEndCapture(cap, &graph));
        // recorded launches are counted when the graph runs
        w->graph_kernels.push_back(launch_counter().load() - n0);
        launch_counter().fetch_sub(w->graph_kernels.back());
        cudaGraphExec_t exec;
        RTG_CUDA(cudaGraphInstantiate(&exec, graph, 0));
        w->graphs.push_back(exec);
        RTG_CUDA(cudaGraphDestroy(graph));
    }
    RTG_CUDA(cudaStreamDestroy(cap));
}

void replay_part(BatchWs* w, int part, cudaStream_t s) {
    RTG_CUDA(cudaGraphLaunch(w->graphs[part], s));
    launch_counter().fetch_add(w->graph_kernels[part]);
}

// One restart cycle; returns the Arnoldi steps it took.
int run_cycle(BatchWs* w, cudaStream_t s) {
    replay_part(w, 0, s);
    int steps = 0;
    for (int j = 0; j < w->m; ++j) {
        replay_part(w, 1 + j, s);
        RTG_CUDA(cudaEventRecord(w->ev[j & 1], s));
        if (j > 0) {
            RTG_CUDA(cudaEventSynchronize(w->ev[(j - 1) & 1]));
            if (w->hstop[j - 1]) break;
        }
        steps = j + 1;
    }
    replay_part(w, w->m + 1, s);
    return steps;
}

}  // namespace

void free_batch(rtg_handle* h) {
    free_bws(h->bws);
    h->bws = nullptr;
}

int solve_batched(rtg_handle* h, int nb, const int64_t* inst_off, const double* f, const double* g, double* u,
                  const rtg_solve_opts* o, rtg_solve_info* infos, cudaStream_t s) {
    const auto t0 = std::chrono::steady_clock::now();
    const int64_t N = h->host.ndof;
    if (nb < 1) throw RtgError{RTG_ERR_ARG, "nbatch < 1"};
    if (inst_off[0] != 0 || inst_off[nb] != N) throw RtgError{RTG_ERR_ARG, "instance offsets must cover [0, N)"};
    for (int b = 0; b < nb; ++b)
        if (inst_off[b + 1] <= inst_off[b]) throw RtgError{RTG_ERR_ARG, "empty or unordered instance"};
    if (o->method != 1) throw RtgError{RTG_ERR_ARG, "batched solve supports method 1 (FP32 GMRES + FP64 refinement)"};
    const int m = std::max(1, std::min(o->restart, 60));
    get_sweep(h, s);
    // (re)build the workspace when the instance split or restart changes
    BatchWs* w = h->bws;
    const std::vector<int64_t> off(inst_off, inst_off + nb + 1);
    const bool same = w && w->off == off && w->m == m && w->N == N;
    std::vector<BChunk> chunks;
    std::vector<int32_t> cbeg(nb + 1, 0);
    for (int b = 0; b < nb; ++b) {
        cbeg[b] = (int32_t)chunks.size();
        for (int64_t i = inst_off[b]; i < inst_off[b + 1]; i += kBChunk)
            chunks.push_back(BChunk{i, std::min(inst_off[b + 1], i + kBChunk), b, 0});
    }
    cbeg[nb] = (int32_t)chunks.size();
    if (!same) {
        // columns of every instance (contiguous in DOF order)
        const HostTables& t = h->host;
        std::vector<int32_t> cb(nb + 1, (int32_t)t.cols.size());
        cb[0] = 0;
        int b = 0;
        for (size_t c = 0; c < t.cols.size(); ++c) {
            while (b + 1 < nb && t.cols[c].dof_off >= inst_off[b + 1]) cb[++b] = (int32_t)c;
            if (t.cols[c].dof_off < inst_off[b] || t.cols[c].dof_off + t.cols[c].ndof > inst_off[b + 1])
                throw RtgError{RTG_ERR_ARG, "an instance boundary splits a column"};
        }
        free_bws(w);
        w = new BatchWs();
        h->bws = w;
        w->nb = nb;
        w->m = m;
        w->N = N;
        w->nchunks = (int)chunks.size();
        w->d_ch = balloc<BChunk>(w, chunks.size());
        w->d_cbeg = balloc<int32_t>(w, nb + 1);
        RTG_CUDA(cudaMemcpy(w->d_ch, chunks.data(), sizeof(BChunk) * chunks.size(), cudaMemcpyHostToDevice));
        RTG_CUDA(cudaMemcpy(w->d_cbeg, cbeg.data(), sizeof(int32_t) * (nb + 1), cudaMemcpyHostToDevice));
        w->b = balloc<double>(w, N);
        w->r = balloc<double>(w, N);
        w->x = balloc<double>(w, N);
        w->t = balloc<double>(w, N);
        w->gb = balloc<double>(w, N);
        w->V32 = balloc<float>(w, (size_t)(m + 1) * N);
        w->w32 = balloc<float>(w, N);
        w->z32 = balloc<float>(w, N);
        w->s32 = balloc<float>(w, N);
        w->d32 = balloc<float>(w, N);
        w->rhs32 = balloc<float>(w, N);
        w->partial = balloc<double>(w, (size_t)chunks.size() * (m + 2));
        w->partial2 = balloc<double>(w, (size_t)chunks.size() * (m + 2));
        const int ldh = m + 2;
        w->rsum = balloc<double>(w, (size_t)nb * ldh);
        w->h1 = balloc<double>(w, (size_t)nb * ldh);
        w->ho = balloc<double>(w, (size_t)nb * ldh);
        w->nsq = balloc<double>(w, nb);
        w->tin = balloc<double>(w, nb);
        w->scale = balloc<double>(w, nb);
        w->vnorm = balloc<double>(w, nb);
        std::vector<int32_t> one(nb + 1);
        for (int b = 0; b <= nb; ++b) one[b] = b;
        for (int b = 0; b < nb; ++b) w->own_sums = w->own_sums && cbeg[b + 1] - cbeg[b] <= kOwnSums;
        w->d_one = balloc<int32_t>(w, nb + 1);
        RTG_CUDA(cudaMemcpy(w->d_one, one.data(), sizeof(int32_t) * (nb + 1), cudaMemcpyHostToDevice));
        BState& st = w->st;
        st.nb = nb;
        st.m = m;
        st.H = balloc<double>(w, (size_t)nb * (m + 1) * m);
        st.cs = balloc<double>(w, (size_t)nb * m);
        st.sn = balloc<double>(w, (size_t)nb * m);
        st.g = balloc<double>(w, (size_t)nb * (m + 1));
        st.y = balloc<double>(w, (size_t)nb * m);
        st.est = balloc<double>(w, nb);
        st.tol = w->tin;
        st.kvalid = balloc<int32_t>(w, nb);
        st.done = balloc<int32_t>(w, nb);
        st.ndone = balloc<int32_t>(w, 2);
        st.next = sweep_counter(h, s);
        RTG_CUDA(cudaMallocHost(&w->hstop, sizeof(int32_t) * m));
        for (cudaEvent_t& e : w->ev) RTG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        int32_t* d_cb = balloc<int32_t>(w, nb + 1);
        st.col_beg = d_cb;
        st.skip = balloc<int32_t>(w, t.cols.size());
        RTG_CUDA(cudaMemcpy(d_cb, cb.data(), sizeof(int32_t) * (nb + 1), cudaMemcpyHostToDevice));
        RTG_CUDA(cudaMemset(st.skip, 0, sizeof(int32_t) * t.cols.size()));
        w->off = off;   // complete from here on
    }
    const int nc = w->nchunks;
    // b = mask_I (f - A mask_B g); x = 0
    launch_mask_vector(h, 1, g, w->gb, s);
    launch_apply<double>(h, h->v64, RTG_SYSTEM | RTG_MASK_ROWS, w->gb, w->t, s);
    launch_mask_vector(h, 0, f, w->b, s);
    bscale_kernel<double, double><<<nc, kBThreads, 0, s>>>(w->d_ch, w->t, w->b, nullptr, 0, -1., 1.), count_launch();
    bscale_kernel<double, double><<<nc, kBThreads, 0, s>>>(w->d_ch, w->t, w->x, nullptr, 0, 0., 0.), count_launch();
    std::vector<double> bn(nb), rn(nb), tol(nb), tin(nb), scale(nb), inv(nb);
    bnorm2(w, w->b, w->vnorm, 1, s);
    RTG_CUDA(cudaMemcpyAsync(bn.data(), w->vnorm, sizeof(double) * nb, cudaMemcpyDeviceToHost, s));
    RTG_CUDA(cudaStreamSynchronize(s));
    for (int b = 0; b < nb; ++b) tol[b] = std::max(o->rtol * std::sqrt(bn[b]), o->atol);
    const double inner_rtol = o->inner_rtol > 0. ? o->inner_rtol : 1e-6;
    const int max_outer = o->max_outer > 0 ? o->max_outer : 20;
    const int max_cycles = std::max(1, o->max_it / m);
    std::vector<int> iters(nb, 0), outer(nb, 0), done(nb), kv(nb), conv(nb, 0);
    int fp64_applies = 1, fp32_applies = 0, sweeps = 0;
    for (int it = 0; it <= max_outer; ++it) {
        // r = b - A x (FP64), per-instance norms
        launch_apply<double>(h, h->v64, RTG_SYSTEM | RTG_MASK_ROWS, w->x, w->r, s);
        ++fp64_applies;
        bscale_kernel<double, double><<<nc, kBThreads, 0, s>>>(w->d_ch, w->b, w->r, nullptr, 0, 1., -1.), count_launch();
        bnorm2(w, w->r, w->vnorm, 1, s);
        RTG_CUDA(cudaMemcpyAsync(rn.data(), w->vnorm, sizeof(double) * nb, cudaMemcpyDeviceToHost, s));
        RTG_CUDA(cudaStreamSynchronize(s));
        bool any = false;
        for (int b = 0; b < nb; ++b) {
            rn[b] = std::sqrt(rn[b]);
            const bool act = rn[b] > tol[b] && std::isfinite(rn[b]);
            conv[b] = act ? 0 : 1;
            any = any || act;
            inv[b] = act ? 1. / rn[b] : 0.;
            scale[b] = act ? rn[b] : 0.;
            tin[b] = act ? std::max(inner_rtol, tol[b] / rn[b]) : 1e300;
            if (act) outer[b]++;
        }
        if (!any || it == max_outer) break;
        // inner FP32 solve of A d = r / ||r|| per instance
        RTG_CUDA(cudaMemcpyAsync(w->scale, inv.data(), sizeof(double) * nb, cudaMemcpyHostToDevice, s));
        RTG_CUDA(cudaMemcpyAsync(w->tin, tin.data(), sizeof(double) * nb, cudaMemcpyHostToDevice, s));
        bscale_kernel<double, float><<<nc, kBThreads, 0, s>>>(w->d_ch, w->r, w->rhs32, w->scale, 1, 0., 0.), count_launch();
        bscale_kernel<float, float><<<nc, kBThreads, 0, s>>>(w->d_ch, w->d32, w->d32, nullptr, 0, 0., 0.), count_launch();
        if ((int)w->graphs.size() != m + 2) {
            // build the FP32 apply plan and sweep launch shape before capture
            launch_apply<float>(h, h->v32, RTG_SYSTEM | RTG_MASK_ROWS, w->d32, w->s32, s);
            apply_sweep<float>(h, w->s32, w->z32, s);
            RTG_CUDA(cudaStreamSynchronize(s));
            drop_graphs(w);   // of a capture that failed half-way
            capture_parts(h, w);
        }
        for (int cyc = 0; cyc < max_cycles; ++cyc) {
            const int steps = run_cycle(w, s);
            fp32_applies += steps + 1;
            sweeps += steps + 1;
            RTG_CUDA(cudaMemcpyAsync(done.data(), w->st.done, sizeof(int32_t) * nb, cudaMemcpyDeviceToHost, s));
            RTG_CUDA(cudaMemcpyAsync(kv.data(), w->st.kvalid, sizeof(int32_t) * nb, cudaMemcpyDeviceToHost, s));
            RTG_CUDA(cudaStreamSynchronize(s));
            bool all = true;
            for (int b = 0; b < nb; ++b) {
                if (!conv[b]) iters[b] += kv[b];
                all = all && (done[b] || conv[b]);
            }
            if (all) break;
        }
        // x += ||r|| d
        RTG_CUDA(cudaMemcpyAsync(w->scale, scale.data(), sizeof(double) * nb, cudaMemcpyHostToDevice, s));
        bscale_kernel<float, double><<<nc, kBThreads, 0, s>>>(w->d_ch, w->d32, w->x, w->scale, 1, 0., 1.), count_launch();
    }
    if (sweep_status(h, s) != RTG_OK)
        throw RtgError{RTG_ERR_TIMEOUT, "a sweep wait gave up; the solution is not valid"};
    if (apply_status(h, s) != RTG_OK)
        throw RtgError{RTG_ERR_TIMEOUT, "a tensor-core wait of an apply gave up; the solution is not valid"};
    // u = x on the unknowns, g on the inflow-boundary DOFs
    bscale_kernel<double, double><<<nc, kBThreads, 0, s>>>(w->d_ch, w->x, w->gb, nullptr, 0, 1., 1.), count_launch();
    RTG_CUDA(cudaMemcpyAsync(u, w->gb, sizeof(double) * N, cudaMemcpyDeviceToDevice, s));
    RTG_CUDA(cudaStreamSynchronize(s));
    const double secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (infos)
        for (int b = 0; b < nb; ++b) {
            rtg_solve_info inf{};
            inf.converged = conv[b];
            inf.iterations = iters[b];
            inf.outer = outer[b];
            inf.fp64_applies = fp64_applies;
            inf.fp32_applies = fp32_applies;
            inf.sweeps = sweeps;
            inf.res_f = rn[b];
            inf.rhs_norm = std::sqrt(bn[b]);
            inf.seconds = secs;
            infos[b] = inf;
        }
    return RTG_OK;
}

}  // namespace rtg

// pcg.cu -- Jacobi-preconditioned CG on the device for sm_100a.
//
// Reference: conjugate_gradient::solve (src/solver/linear/linear_solver.cpp:67-109), which runs
// Eigen's ConjugateGradient<Lower|Upper> with the diagonal preconditioner, x0 = 0 and the stop
// test ||r||^2 < max(tol^2 ||b||^2, DBL_MIN), and the reference's GPU variant
// conjugate_gradient_cuda::solve (conjugate_gradient_cuda.cpp:72-192, cuSPARSE csrmv + cuBLAS
// + diagonal_matrix_vector_product.cu) which copies K to the device on every solve and reads 3
// dot products back to the host per iteration.
//
// Here K stays resident in HBM and every scalar stays on the device.  One iteration is three
// kernels:
//   k_spmv  : q = A p over the 3x3 block rows (a few lanes per block row, several rows per
//             warp in flight), fused with the p.q reduction; the last block to finish forms
//             alpha = (r.z)/(p.q);
//   k_xr    : x += alpha p, r -= alpha q, fused with r.r and r.z (z = D^-1 r); the last block
//             applies the stop test, beta and the iteration count;
//   k_p     : p = D^-1 r + beta p.
// (up to about 64^3 hex8 cells the same iteration runs in one persistent launch, cg_group.cu).
// Reductions are per-block partials summed in a fixed order by the last block (deterministic,
// no spin waits).  Kernels return at once after `done` is set, so whole blocks of iterations are
// enqueued (optionally as one CUDA graph) and the host reads the flag once per block.
// Rows of active Dirichlet DOFs are skipped (q = 0): with b = 0 there, r, z, p stay exactly 0 on
// them, so this equals neon's zeroing of those rows and columns (static_matrix.hpp:279-320).
#include <cfloat>
#include <cstdint>
#include <cmath>
#include <cstring>
#include <vector>

#include "cg_group.cuh"
#include "mf_cg.cuh"
#include "nb2_internal.cuh"
#include "reduce.cuh"

namespace nb2 {

int reduction_blocks(const nb2_ctx*) { return 148 * 4; }

template <typename T>
__device__ __forceinline__ T ld_stream(const T* p) {
    return __ldcs(p);
}

// ---------------------------------------------------------------------------------------
// matrices
// ---------------------------------------------------------------------------------------
template <typename V>
struct Bsr {
    const int* brp;
    const int* bcol;
    const V* val;
    int rows;  // block rows
};

struct Csr {
    const int* rp;
    const int* ci;
    const double* val;
    int rows;
};

// y[3a+r] for r = 0..2 of block row a, reduced across the warp (all lanes get the sums).
// A row of a hex8 mesh holds up to 27 blocks = 243 values: the first 256 values are loaded in one
// batch of 8 independent loads per lane (values, then their block columns, then the x entries),
// so a warp keeps a whole row in flight instead of one 32-value slice per round trip.
template <typename V, typename X, typename Acc>
__device__ __forceinline__ void bsr_row(const Bsr<V>& A, const X* __restrict__ x, int a, int lane,
                                        Acc& y0, Acc& y1, Acc& y2) {
    const int b0 = __ldg(A.brp + a);
    const int nval = 9 * (__ldg(A.brp + a + 1) - b0);
    const V* vals = A.val + 9ll * b0;
    const int* cols = A.bcol + b0;
    Acc a0 = 0, a1 = 0, a2 = 0;
    constexpr int U = 8;
    V v[U];
    int c[U];
#pragma unroll
    for (int t = 0; t < U; ++t) {
        const int idx = lane + 32 * t;
        const bool ok = idx < nval;
        v[t] = ok ? ld_stream(vals + idx) : (V)0;
        c[t] = ok ? __ldg(cols + idx / 9) : 0;
    }
#pragma unroll
    for (int t = 0; t < U; ++t) {
        const int idx = lane + 32 * t;
        const int e = idx % 9;
        const int r = e / 3;
        const int cc = e - 3 * r;
        const Acc prod = (Acc)v[t] * (Acc)x[3ll * c[t] + cc];
        a0 += (r == 0) ? prod : (Acc)0;
        a1 += (r == 1) ? prod : (Acc)0;
        a2 += (r == 2) ? prod : (Acc)0;
    }
    for (int idx = lane + 32 * U; idx < nval; idx += 32) {  // rows with more than 28 blocks
        const int k = idx / 9;
        const int e = idx - 9 * k;
        const int r = e / 3;
        const int cc = e - 3 * r;
        const Acc prod = (Acc)ld_stream(vals + idx) * (Acc)x[3ll * __ldg(cols + k) + cc];
        a0 += (r == 0) ? prod : (Acc)0;
        a1 += (r == 1) ? prod : (Acc)0;
        a2 += (r == 2) ? prod : (Acc)0;
    }
    y0 = warp_sum(a0);
    y1 = warp_sum(a1);
    y2 = warp_sum(a2);
}

// ---------------------------------------------------------------------------------------
// CG kernels (BSR)
// ---------------------------------------------------------------------------------------
// q = A p with LPR lanes per 3x3 block row: a warp keeps 32/LPR rows in flight; lane l of a row
// walks its blocks l, l+LPR, ... (9 values, the block column, 3 gathered p entries) and the three
// row sums are reduced over the LPR lanes with shuffles.  Plain loads with many independent rows
// per SM stream the matrix at ~80% of HBM bandwidth (hex8 rows: 27 blocks, tet4: ~15), where a
// whole warp per row or a shared-memory staging pipeline left it latency-bound.  Fused with the
// p.q reduction; the last block forms alpha = (r.z)/(p.q).
template <typename V, typename X, int LPR>
__global__ void __launch_bounds__(kRedThreads) k_spmv(Bsr<V> A, const X* __restrict__ p,
                                                      X* __restrict__ q,
                                                      const unsigned char* __restrict__ mask,
                                                      CgScalars* s, double* partials) {
    if (s->done) return;
    constexpr int RPW = 32 / LPR;
    const int lane = threadIdx.x & 31, sub = lane / LPR, sl = lane % LPR;
    const long long gw = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
    double dot[1] = {0.0};
    for (long long a0 = gw * RPW; a0 < A.rows; a0 += nw * RPW) {
        const long long a = a0 + sub;
        X y0 = 0, y1 = 0, y2 = 0;
        if (a < A.rows) {
            const int b0 = A.brp[a], b1 = A.brp[a + 1];
            for (int k = b0 + sl; k < b1; k += LPR) {
                const long long col = A.bcol[k];
                const X x0 = p[3 * col], x1 = p[3 * col + 1], x2 = p[3 * col + 2];
                const V* blk = A.val + 9ll * k;
                y0 += (X)blk[0] * x0 + (X)blk[1] * x1 + (X)blk[2] * x2;
                y1 += (X)blk[3] * x0 + (X)blk[4] * x1 + (X)blk[5] * x2;
                y2 += (X)blk[6] * x0 + (X)blk[7] * x1 + (X)blk[8] * x2;
            }
        }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) {
            y0 += __shfl_xor_sync(0xffffffffu, y0, o);
            y1 += __shfl_xor_sync(0xffffffffu, y1, o);
            y2 += __shfl_xor_sync(0xffffffffu, y2, o);
        }
        if (a < A.rows && sl < 3) {
            const long long i = 3 * a + sl;
            X y = sl == 0 ? y0 : (sl == 1 ? y1 : y2);
            if (mask && mask[i]) y = (X)0;
            q[i] = y;
            dot[0] += (double)p[i] * (double)y;
        }
    }
    if (block_partials<1>(dot, partials, &s->counter[0])) {
        double tot[1];
        final_sum<1>(partials, tot);
        if (threadIdx.x == 0) {
            s->pq = tot[0];
            s->alpha = s->abs_new / tot[0];
            // Eigen's CG carries on through p.Ap <= 0 (an indefinite tangent); only a
            // non-finite step size is a failure (neon: FE_INVALID -> computational_error)
            if (!isfinite(s->alpha)) {
                s->status = NB2_E_NAN;
                s->done = 1;
            }
            s->counter[0] = 0;
        }
    }
}

// lanes per block row of the PCG SpMV: 4 for FP64 and FP32 values (C3 on B200: FP64 0.44 ms,
// FP32 0.26 ms per iteration; 8 or 16 lanes were slower for both)
template <typename V>
constexpr int spmv_lanes() {
    return 4;
}

template <typename X>
__device__ __forceinline__ void xr_one(X& x, X& r, X p, X q, X inv, X alpha, double (&acc)[2]) {
    x += alpha * p;
    const X ri = r - alpha * q;
    r = ri;
    acc[0] += (double)ri * (double)ri;
    acc[1] += (double)ri * (double)(inv * ri);
}

// No __restrict__ on the vectors of the kernels that start early: they are resident while the kernel
// ahead still writes them, and the read-only path that __restrict__ opens is for data that nothing
// writes during a kernel's life (inv, the mask), or that the kernel itself only writes (q of the product).
template <typename X>
__global__ void __launch_bounds__(kRedThreads) k_xr(long long n, X* x, X* r, const X* p, const X* q,
                                                    const X* __restrict__ inv, CgScalars* s,
                                                    double* partials) {
    pdl_next();
    pdl_wait();
    if (s->done) return;
    using V = typename Vec16<X>::T;
    constexpr int W = Vec16<X>::W;
    const X alpha = (X)s->alpha;
    double acc[2] = {0.0, 0.0};
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long st = (long long)gridDim.x * blockDim.x;
    const long long nv = aligned16(x, r, p, q, inv) ? n / W : 0;
    for (long long j = t0; j < nv; j += st) {
        X xv[W], rv[W], pv[W], qv[W], iv[W];
        *reinterpret_cast<V*>(xv) = reinterpret_cast<const V*>(x)[j];
        *reinterpret_cast<V*>(rv) = reinterpret_cast<const V*>(r)[j];
        *reinterpret_cast<V*>(pv) = reinterpret_cast<const V*>(p)[j];
        *reinterpret_cast<V*>(qv) = reinterpret_cast<const V*>(q)[j];
        *reinterpret_cast<V*>(iv) = reinterpret_cast<const V*>(inv)[j];
#pragma unroll
        for (int w = 0; w < W; ++w) xr_one(xv[w], rv[w], pv[w], qv[w], iv[w], alpha, acc);
        reinterpret_cast<V*>(x)[j] = *reinterpret_cast<V*>(xv);
        reinterpret_cast<V*>(r)[j] = *reinterpret_cast<V*>(rv);
    }
    for (long long i = nv * W + t0; i < n; i += st) xr_one(x[i], r[i], p[i], q[i], inv[i], alpha, acc);
    if (block_partials<2>(acc, partials, &s->counter[1])) {
        double tot[2];
        final_sum<2>(partials, tot);
        if (threadIdx.x == 0) {
            s->rr = tot[0];
            if (tot[0] < s->threshold) {
                s->done = 1;
            } else if (tot[0] > s->rr_cap) {
                s->done = 1;
                s->status = NB2_E_CG_BREAKDOWN;
            } else {
                s->beta = tot[1] / s->abs_new;
                s->abs_new = tot[1];
                s->rz = tot[1];
                s->iterations += 1;
                if (s->iterations >= s->max_iterations) {
                    s->done = 1;
                    s->status = NB2_E_CG_MAXIT;
                }
            }
            if (!isfinite(tot[0])) {
                s->done = 1;
                s->status = NB2_E_NAN;
            }
            s->counter[1] = 0;
        }
    }
}

template <typename X>
__global__ void __launch_bounds__(kRedThreads) k_p(long long n, X* p, const X* r,
                                                   const X* __restrict__ inv, const CgScalars* s) {
    pdl_next();
    pdl_wait();
    if (s->done) return;
    using V = typename Vec16<X>::T;
    constexpr int W = Vec16<X>::W;
    const X beta = (X)s->beta;
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long st = (long long)gridDim.x * blockDim.x;
    const long long nv = aligned16(p, r, inv, p, r) ? n / W : 0;
    for (long long j = t0; j < nv; j += st) {
        X pv[W], rv[W], iv[W];
        *reinterpret_cast<V*>(pv) = reinterpret_cast<const V*>(p)[j];
        *reinterpret_cast<V*>(rv) = reinterpret_cast<const V*>(r)[j];
        *reinterpret_cast<V*>(iv) = reinterpret_cast<const V*>(inv)[j];
#pragma unroll
        for (int w = 0; w < W; ++w) pv[w] = iv[w] * rv[w] + beta * pv[w];
        reinterpret_cast<V*>(p)[j] = *reinterpret_cast<V*>(pv);
    }
    for (long long i = nv * W + t0; i < n; i += st) p[i] = inv[i] * r[i] + beta * p[i];
}

// x = 0, r = b (as X), p = D^-1 r; rhs_norm2, r.r, r.p; threshold and early exits.
template <typename X>
__global__ void __launch_bounds__(kRedThreads) k_init(long long n, const double* __restrict__ b,
                                                      X* __restrict__ x, X* __restrict__ r,
                                                      X* __restrict__ p,
                                                      const X* __restrict__ inv, CgScalars* s,
                                                      double* partials, double tol) {
    double acc[3] = {0, 0, 0};
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        X bi = (X)b[i];
        x[i] = (X)0;
        r[i] = bi;
        X pi = inv[i] * bi;
        p[i] = pi;
        acc[0] += b[i] * b[i];
        acc[1] += (double)bi * (double)bi;
        acc[2] += (double)bi * (double)pi;
    }
    if (block_partials<3>(acc, partials, &s->counter[2])) {
        double tot[3];
        final_sum<3>(partials, tot);
        if (threadIdx.x == 0) {
            s->rhs_norm2 = tot[0];
            s->threshold = fmax(tol * tol * tot[0], DBL_MIN);
            s->rr = tot[1];
            s->abs_new = tot[2];
            s->rz = tot[2];
            s->rr_cap = INFINITY;
            s->beta = 0.0;
            s->iterations = 0;
            s->status = 0;
            s->done = 0;
            if (tot[0] == 0.0) {
                s->done = 1;
                s->rr = 0.0;
            } else if (tot[1] < s->threshold) {
                s->done = 1;
            }
            s->counter[2] = 0;
        }
    }
}

// Jacobi inverse diagonal of a block matrix: 1/K_ii, or 1 for a zero diagonal (Eigen's
// DiagonalPreconditioner).
template <typename V, typename X>
__global__ void k_invdiag(Bsr<V> A, X* __restrict__ inv) {
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A.rows) return;
    int lo = A.brp[a], hi = A.brp[a + 1] - 1;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (A.bcol[mid] < a)
            lo = mid + 1;
        else
            hi = mid;
    }
    // a node that no element references has an empty row: its diagonal is 0 (inverse 1)
    const bool has = lo < A.brp[a + 1] && A.bcol[lo] == a;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        V d = has ? A.val[9ll * lo + 4 * r] : (V)0;
        inv[3ll * a + r] = (d != (V)0) ? (X)(1.0 / (double)d) : (X)1;
    }
}

template <typename X>
__global__ void k_copy_out(long long n, const X* __restrict__ src, double* __restrict__ dst) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        dst[i] = (double)src[i];
}

// ---------------------------------------------------------------------------------------
// generic CSR (drop-in linear_solver on a caller matrix)
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kRedThreads) k_csr_spmv(Csr A, const double* p,
                                                          double* __restrict__ q, CgScalars* s,
                                                          double* partials) {
    pdl_next();
    pdl_wait();
    if (s->done) return;
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    double dot[1] = {0.0};
    // One warp per row.  A row's first 96 entries (a hex8 row has 81) are requested at once, values and
    // columns, then the gathered p: with one entry per lane and trip the kernel waited for memory three
    // times over (per iteration, hex8 systems of 24^3 cells, 130 MB in L2: 34.5 -> 30.3 us; 30^3,
    // 255 MB from HBM: 45.3 -> 37.7).  The sums keep their order.
    constexpr int U = 3;
    int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    int b0 = 0, b1 = 0;
    if (i < A.rows) {
        b0 = A.rp[i];
        b1 = A.rp[i + 1];
    }
    for (; i < A.rows; i += warps) {
        double v[U], g[U];
        int c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = b0 + lane + 32 * u;
            const bool on = k < b1;
            v[u] = on ? A.val[k] : 0.0;
            c[u] = on ? A.ci[k] : -1;
        }
        int n0 = 0, n1 = 0;  // the next row's bounds, ahead of their use
        if (i + warps < A.rows) {
            n0 = A.rp[i + warps];
            n1 = A.rp[i + warps + 1];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) g[u] = c[u] >= 0 ? p[c[u]] : 0.0;
        const double pi = lane == 0 ? p[i] : 0.0;  // in flight with the others
        double acc = 0;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c[u] >= 0) acc += v[u] * g[u];
        for (int k = b0 + lane + 32 * U; k < b1; k += 32) acc += A.val[k] * p[A.ci[k]];
        acc = warp_sum(acc);
        if (lane == 0) {
            q[i] = acc;
            dot[0] += pi * acc;
        }
        b0 = n0;
        b1 = n1;
    }
    if (block_partials<1>(dot, partials, &s->counter[0])) {
        double tot[1];
        final_sum<1>(partials, tot);
        if (threadIdx.x == 0) {
            s->pq = tot[0];
            s->alpha = s->abs_new / tot[0];
            if (!isfinite(s->alpha)) {
                s->status = NB2_E_NAN;
                s->done = 1;
            }
            s->counter[0] = 0;
        }
    }
}

__global__ void k_csr_invdiag(Csr A, double* inv) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.rows) return;
    double v = 1.0;
    for (int k = A.rp[i]; k < A.rp[i + 1]; ++k)
        if (A.ci[k] == i) {
            if (A.val[k] != 0.0) v = 1.0 / A.val[k];
            break;
        }
    inv[i] = v;
}

// ---------------------------------------------------------------------------------------
// norms and helpers
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kRedThreads) k_norms(long long n, const double* a,
                                                       const double* b, const double* c,
                                                       const double* d, const double* e,
                                                       double* partials, unsigned int* counter,
                                                       double* out) {
    double acc[5] = {0, 0, 0, 0, 0};
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        acc[0] += a[i] * a[i];
        acc[1] += b[i] * b[i];
        acc[2] += c[i] * c[i];
        acc[3] += d[i] * d[i];
        acc[4] += e[i] * e[i];
    }
    if (block_partials<5>(acc, partials, counter)) {
        double tot[5];
        final_sum<5>(partials, tot);
        if (threadIdx.x == 0) {
            for (int j = 0; j < 5; ++j) out[j] = sqrt(tot[j]);
            *counter = 0;
        }
    }
}

template <typename V>
__global__ void __launch_bounds__(kRedThreads) k_bsr_apply(Bsr<V> A, const double* __restrict__ x,
                                                           double* __restrict__ y,
                                                           const unsigned char* __restrict__ mask) {
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int a = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); a < A.rows; a += warps) {
        double y0, y1, y2;
        bsr_row<V, double, double>(A, x, a, lane, y0, y1, y2);
        if (lane < 3) {
            long long i = 3ll * a + lane;
            double v = lane == 0 ? y0 : (lane == 1 ? y1 : y2);
            if (mask && mask[i]) v = 0.0;
            y[i] = v;
        }
    }
}

// ---------------------------------------------------------------------------------------
// host drivers
// ---------------------------------------------------------------------------------------
int wait_scalars(nb2_ctx* c) {
    NB2_CUDA(c, cudaMemcpyAsync(c->h_cgs, c->cgs, sizeof(CgScalars), cudaMemcpyDeviceToHost,
                                c->stream));
    NB2_CUDA(c, cudaStreamSynchronize(c->stream));
    return NB2_OK;
}

constexpr int kChunk = 32;

// One Jacobi-PCG on a block matrix: the captured block of kChunk iterations and the host loop
// that launches blocks until the device scalars say done.
template <typename V, typename X>
struct CgRunner {
    nb2_ctx* c;
    const V* vals;
    X *x, *r, *p, *q, *inv;
    bool use_mask, use_graphs;
    cudaGraphExec_t* cache;
    int RB = 0;
    Bsr<V> A{};

    int setup() {
        RB = reduction_blocks(c);
        A = Bsr<V>{c->brp, c->bcol, vals, c->N};
        k_invdiag<V, X><<<(c->N + 255) / 256, 256, 0, c->stream>>>(A, inv);
        c->launches++;
        return NB2_OK;
    }

    void enqueue(int count) {
        const unsigned char* mask = use_mask ? c->mask : nullptr;
        const long long n = c->n;
        for (int it = 0; it < count; ++it) {
            k_spmv<V, X, spmv_lanes<V>()><<<RB, kRedThreads, 0, c->stream>>>(A, p, q, mask, c->cgs,
                                                                            c->partials);
            k_xr<X><<<RB, kRedThreads, 0, c->stream>>>(n, x, r, p, q, inv, c->cgs, c->partials);
            k_p<X><<<RB, kRedThreads, 0, c->stream>>>(n, p, r, inv, c->cgs);
        }
    }

    // launch blocks of iterations until the scalars say done (bounded by maxit / kChunk + 4)
    int run(int maxit) {
        if (use_graphs && *cache == nullptr) {
            // capture one block of iterations; plain launches if the stream cannot be captured
            // (e.g. the legacy default stream)
            cudaGraph_t g = nullptr;
            if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) ==
                cudaSuccess) {
                enqueue(kChunk);
                if (cudaStreamEndCapture(c->stream, &g) == cudaSuccess && g) {
                    if (cudaGraphInstantiate(cache, g, 0) != cudaSuccess) *cache = nullptr;
                    cudaGraphDestroy(g);
                }
            }
            cudaGetLastError();
            if (*cache == nullptr) use_graphs = false;
        }
        int guard = 0;
        for (;;) {
            if (use_graphs)
                NB2_CUDA(c, cudaGraphLaunch(*cache, c->stream));
            else
                enqueue(kChunk);
            c->launches += 3 * kChunk;
            NB2_TRY(wait_scalars(c));
            if (c->h_cgs->done) break;
            if (++guard > (maxit / kChunk) + 4) break;  // scalars say not done: cannot happen
        }
        NB2_CUDA(c, cudaGetLastError());
        return NB2_OK;
    }
};

template <typename V, typename X>
static int run_bsr_cg(nb2_ctx* c, const V* vals, X* x, X* r, X* p, X* q, X* inv, const double* b,
                      double* xout, double tol, int maxit, bool use_mask, int* iterations,
                      double* error, bool use_graphs, cudaGraphExec_t* cache) {
    CgRunner<V, X> cg{c, vals, x, r, p, q, inv, use_mask, use_graphs, cache};
    NB2_TRY(cg.setup());
    const long long n = c->n;
    k_init<X><<<cg.RB, kRedThreads, 0, c->stream>>>(n, b, x, r, p, inv, c->cgs, c->partials, tol);
    c->launches++;
    // max_iterations is read by k_xr: set it with a tiny copy
    NB2_CUDA(c, cudaMemcpyAsync(&c->cgs->max_iterations, &maxit, sizeof(int), cudaMemcpyHostToDevice,
                                c->stream));
    // one persistent launch where its plan applies (up to about 64^3 hex8 cells, where it is as fast
    // as the kernels below: 124 against 129 us per iteration; 12 against 27 us at 37x29x32)
    SellPlan* plan = nullptr;
    NB2_TRY(sell_plan(c, {0, c->N}, sizeof(V), &plan));
    if (plan && sell_fill(c, plan, vals, use_mask ? c->mask : nullptr) == NB2_OK) {
        CgScalars* s = c->cgs;
        const GroupScalars S{&s->threshold,  &s->abs_new, &s->beta,   &s->rr,           &s->rr_cap,
                             &s->iterations, &s->done,    &s->status, &s->max_iterations};
        do {
            NB2_TRY((group_cg<V, X>(c, plan, S, {}, x, r, p, q, inv, nullptr)));
            NB2_TRY(wait_scalars(c));
            if (group_failed(c)) return NB2_E_TIMEOUT;
        } while (!c->h_cgs->done);
    } else {
        NB2_TRY(cg.run(maxit));
    }
    k_copy_out<X><<<cg.RB, kRedThreads, 0, c->stream>>>(n, x, xout);
    c->launches++;
    const CgScalars& h = *c->h_cgs;
    *iterations = h.iterations;
    *error = h.rhs_norm2 > 0 ? std::sqrt(h.rr / h.rhs_norm2) : 0.0;
    if (h.status) return h.status;
    if (!h.done) return NB2_E_TIMEOUT;
    return NB2_OK;
}

int pcg_device_fp64(nb2_ctx* c, const double* b, double* x, double tol, int maxit, bool use_mask,
                    int* iterations, double* error, bool use_graphs) {
    return run_bsr_cg<double, double>(c, c->K64, c->cg_x, c->cg_r, c->cg_p, c->cg_q, c->cg_inv, b,
                                      x, tol, maxit, use_mask, iterations, error,
                                      use_graphs && use_mask, &c->graph64[c->kbuf]);
}

int pcg_device_fp32(nb2_ctx* c, const double* b, double* x, double tol, int maxit, int* iterations,
                    double* error, bool use_graphs) {
    return run_bsr_cg<float, float>(c, c->K32, c->cg32_x, c->cg32_r, c->cg32_p, c->cg32_q,
                                    c->cg32_inv, b, x, tol, maxit, true, iterations, error,
                                    use_graphs, &c->graph32);
}

void release_graphs(nb2_ctx* c) {
    for (auto& g : c->graph64) {
        if (g) cudaGraphExecDestroy(g);
        g = nullptr;
    }
    if (c->graph32) cudaGraphExecDestroy(c->graph32);
    c->graph32 = nullptr;
    if (c->mf) {
        for (auto* g : {&c->mf->graph32[0], &c->mf->graph32[1], &c->mf->graph64}) {
            if (*g) cudaGraphExecDestroy(*g);
            *g = nullptr;
        }
    }
}

void bsr_spmv_fp64(nb2_ctx* c, const double* x, double* y, bool use_mask) {
    Bsr<double> A{c->brp, c->bcol, c->K64, c->N};
    k_bsr_apply<double><<<reduction_blocks(c), kRedThreads, 0, c->stream>>>(
        A, x, y, use_mask ? c->mask : nullptr);
    c->launches++;
}

void bsr_spmv_mixed_accum(nb2_ctx* c, const double* x, double* y) {
    Bsr<float> A{c->brp, c->bcol, c->K32, c->N};
    k_bsr_apply<float><<<reduction_blocks(c), kRedThreads, 0, c->stream>>>(A, x, y, nullptr);
    c->launches++;
}

__global__ void __launch_bounds__(kRedThreads) k_dot1(long long n, const double* a, const double* b,
                                                      double* partials, unsigned int* counter,
                                                      double* out) {
    double acc[1] = {0.0};
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        acc[0] += a[i] * b[i];
    if (block_partials<1>(acc, partials, counter)) {
        double tot[1];
        final_sum<1>(partials, tot);
        if (threadIdx.x == 0) {
            *out = tot[0];
            *counter = 0;
        }
    }
}

double device_dot_sync(nb2_ctx* c, const double* a, const double* b, int n) {
    k_dot1<<<reduction_blocks(c), kRedThreads, 0, c->stream>>>(n, a, b, c->partials,
                                                                &c->cgs->counter[3], c->norms + 5);
    c->launches++;
    cudaMemcpyAsync(c->h_norms + 5, c->norms + 5, sizeof(double), cudaMemcpyDeviceToHost, c->stream);
    cudaStreamSynchronize(c->stream);
    return c->h_norms[5];
}

int compute_norms(nb2_ctx* c) {
    k_norms<<<reduction_blocks(c), kRedThreads, 0, c->stream>>>(
        c->n, c->du, c->u, c->rhs, c->fext, c->fint, c->partials, &c->cgs->counter[3], c->norms);
    c->launches++;
    NB2_CUDA(c, cudaMemcpyAsync(c->h_norms, c->norms, 5 * sizeof(double), cudaMemcpyDeviceToHost,
                                c->stream));
    NB2_CUDA(c, cudaStreamSynchronize(c->stream));
    return NB2_OK;
}

// column indices in [0, n) over [0, rp[n]) (rp already checked); flag = 1 on any violation
__global__ void k_check_columns(int n, const int* __restrict__ rp, const int* __restrict__ ci,
                                unsigned int* flag) {
    const long long nnz = rp[n];
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
         k += (long long)gridDim.x * blockDim.x)
        if (ci[k] < 0 || ci[k] >= n) atomicOr(flag, 1u);
}

// kChunk iterations on a caller CSR.  The kernels start early (programmatic dependent launch): a small
// system is bound by the gaps between them (hex8 systems of 8^3, 16^3, 24^3 cells: 24.6 -> 15.8,
// 23.7 -> 18.2, 30.3 -> 27.6 us per iteration).
cudaError_t csr_chunk(const Csr& A, double* x, double* r, double* p, double* q, const double* inv,
                      CgScalars* s, double* partials, int RB, cudaStream_t stream) {
    const long long n = A.rows;
    cudaError_t e = cudaSuccess;
    for (int it = 0; it < kChunk && e == cudaSuccess; ++it) {
        e = launch_early(true, stream, (unsigned)RB, (unsigned)kRedThreads, 0, k_csr_spmv, A,
                         (const double*)p, q, s, partials);
        if (e == cudaSuccess)
            e = launch_early(true, stream, (unsigned)RB, (unsigned)kRedThreads, 0, k_xr<double>, n, x,
                             r, (const double*)p, (const double*)q, inv, s, partials);
        if (e == cudaSuccess)
            e = launch_early(true, stream, (unsigned)RB, (unsigned)kRedThreads, 0, k_p<double>, n, p,
                             (const double*)r, inv, (const CgScalars*)s);
    }
    return e;
}

// Standalone solve on a caller CSR (host buffers): own stream and buffers.
int pcg_csr_host(int n, const int* rowptr, const int* col, const double* val, const double* b,
                 double* x, double tol, int maxit, int* iterations, double* error,
                 std::string* err) {
    nb2_ctx tmp;
    nb2_ctx* c = &tmp;
    auto fail = [&](cudaError_t e) {
        if (err) *err = cudaGetErrorString(e);
        return NB2_E_CUDA;
    };
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)) != cudaSuccess)
        return fail(e);
    const long long nnz = rowptr[n];
    int *rp = nullptr, *ci = nullptr;
    double *v = nullptr, *bd = nullptr, *xd = nullptr, *r = nullptr, *p = nullptr, *q = nullptr,
           *inv = nullptr, *partials = nullptr;
    CgScalars* s = nullptr;
    CgScalars hs;
    const int RB = 148 * 4;
    int status = NB2_OK;
#define TRY(call)                          \
    if ((e = (call)) != cudaSuccess) {     \
        status = fail(e);                  \
        goto done;                         \
    }
    // one device block for everything: values, the vectors, partials, scalars and the indices, each
    // part rounded up to 256 bytes so that the update kernels keep their 16-byte path
    {
        auto up = [](size_t k, size_t m) { return (k + m - 1) / m * m; };
        const size_t nv = up((size_t)std::max<long long>(nnz, 1), 32), vec = up((size_t)n, 32);
        const size_t doubles = nv + 6 * vec + RB * 8 + up(sizeof(CgScalars) / 8 + 1, 32);
        const size_t ints = up((size_t)n + 1, 64) + (size_t)std::max<long long>(nnz, 1);
        TRY(cudaMalloc(&v, sizeof(double) * doubles + sizeof(int) * ints));
        bd = v + nv;
        xd = bd + vec;
        r = xd + vec;
        p = r + vec;
        q = p + vec;
        inv = q + vec;
        partials = inv + vec;
        s = reinterpret_cast<CgScalars*>(partials + RB * 8);
        rp = reinterpret_cast<int*>(v + doubles);
        ci = rp + up((size_t)n + 1, 64);
    }
    TRY(cudaMemsetAsync(s, 0, sizeof(CgScalars), c->stream));
    TRY(cudaMemcpyAsync(rp, rowptr, sizeof(int) * (n + 1), cudaMemcpyHostToDevice, c->stream));
    TRY(cudaMemcpyAsync(ci, col, sizeof(int) * nnz, cudaMemcpyHostToDevice, c->stream));
    TRY(cudaMemcpyAsync(v, val, sizeof(double) * nnz, cudaMemcpyHostToDevice, c->stream));
    TRY(cudaMemcpyAsync(bd, b, sizeof(double) * n, cudaMemcpyHostToDevice, c->stream));
    TRY(cudaMemcpyAsync(&s->max_iterations, &maxit, sizeof(int), cudaMemcpyHostToDevice, c->stream));
    // columns outside [0, n) are refused before any kernel follows one
    k_check_columns<<<RB, kRedThreads, 0, c->stream>>>(n, rp, ci, &s->counter[3]);
    TRY(cudaMemcpyAsync(&hs, s, sizeof hs, cudaMemcpyDeviceToHost, c->stream));
    TRY(cudaStreamSynchronize(c->stream));
    if (hs.counter[3] != 0) {
        status = NB2_E_INPUT;
        goto done;
    }
    {
        Csr A{rp, ci, v, n};
        k_csr_invdiag<<<(n + 255) / 256, 256, 0, c->stream>>>(A, inv);
        k_init<double><<<RB, kRedThreads, 0, c->stream>>>(n, bd, xd, r, p, inv, s, partials, tol);
        TRY(cudaMemcpyAsync(&s->max_iterations, &maxit, sizeof(int), cudaMemcpyHostToDevice,
                            c->stream));
        int guard = 0;
        for (;;) {
            if (++guard > maxit / kChunk + 4) {
                status = NB2_E_TIMEOUT;
                goto done;
            }
            TRY(csr_chunk(A, xd, r, p, q, inv, s, partials, RB, c->stream));
            TRY(cudaMemcpyAsync(&hs, s, sizeof hs, cudaMemcpyDeviceToHost, c->stream));
            TRY(cudaStreamSynchronize(c->stream));
            if (hs.done) break;
        }
        TRY(cudaGetLastError());
        TRY(cudaMemcpyAsync(x, xd, sizeof(double) * n, cudaMemcpyDeviceToHost, c->stream));
        TRY(cudaStreamSynchronize(c->stream));
        *iterations = hs.iterations;
        *error = hs.rhs_norm2 > 0 ? std::sqrt(hs.rr / hs.rhs_norm2) : 0.0;
        if (hs.status) status = hs.status;
    }
done:
#undef TRY
    cudaFree(v);
    cudaStreamDestroy(c->stream);
    c->stream = nullptr;
    return status;
}

// ---------------------------------------------------------------------------------------
// Allocation-free PCG (nb2_pcg_solve_noalloc).
//
// For callers that must not allocate device memory while they run a solve: a code that places
// every device byte itself through its own pool or arena and forbids hidden allocations, or a
// long-running service that must not trigger allocator growth in the middle of a time step.
// They pass the matrix, right-hand side and solution in device memory they own; the solver's
// own work vectors, reduction partials and scalars live in the fixed array below, which every
// GPU that loads this library holds until the process exits.  The call allocates nothing, but
// it is not asynchronous: it blocks the host on its stream after the CSR check and once every
// kChunk iterations to read the convergence flag, so it cannot run inside a stream capture.
// ---------------------------------------------------------------------------------------
constexpr int kNoAllocMaxRows = NB2_NOALLOC_MAX_ROWS;
constexpr int kNoAllocBlocks = 148 * 4;
// layout (doubles): [partials kNoAllocBlocks*8][scalars 32][r][p][q][inv] (rows each)
constexpr size_t kNoAllocPartials = (size_t)kNoAllocBlocks * 8;
constexpr size_t kNoAllocScalars = 32;  // >= sizeof(CgScalars) / 8, keeps 256-byte alignment
constexpr size_t kNoAllocDoubles = kNoAllocPartials + kNoAllocScalars + 4ull * kNoAllocMaxRows;
static_assert(sizeof(CgScalars) <= kNoAllocScalars * sizeof(double), "scalar slot too small");

static __device__ __align__(256) double g_noalloc_scratch[kNoAllocDoubles];

// row pointers monotone from 0; flag = 1 on any violation.  Run first, and its flag read back,
// so that the column check below never walks past a corrupt rp[n]
__global__ void k_check_rowptr(int n, const int* __restrict__ rp, unsigned int* flag) {
    const int nnz = rp[n];
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        if (rp[i + 1] < rp[i] || rp[i] < 0 || rp[i + 1] > nnz) atomicOr(flag, 1u);
    if (blockIdx.x == 0 && threadIdx.x == 0 && (rp[0] != 0 || nnz < 0)) atomicOr(flag, 1u);
}

}  // namespace nb2

extern "C" int nb2_pcg_solve_noalloc(int32_t n, const int32_t* rowptr, const int32_t* col,
                                     const double* values, const double* b, double* x,
                                     double tolerance, int32_t maximum_iterations, void* stream,
                                     int32_t* iterations, double* error) {
    using namespace nb2;
    if (n <= 0 || !rowptr || !col || !values || !b || !x || maximum_iterations <= 0)
        return NB2_E_INPUT;
    if (n > kNoAllocMaxRows) return NB2_E_INPUT;  // beyond the fixed workspace
    // device address of the fixed workspace, looked up on every call with the caller's device
    // current (the symbol's host-side name is not a device address).  The lookup allocates
    // nothing; doing it per call keeps no pointer that a cudaDeviceReset could leave stale.
    // The first call on a device loads the library's module there, so make it before any
    // stream capture.
    void* sym = nullptr;
    if (cudaGetSymbolAddress(&sym, g_noalloc_scratch) != cudaSuccess || !sym) return NB2_E_CUDA;
    double* base = static_cast<double*>(sym);
    double* partials = base;
    CgScalars* s = reinterpret_cast<CgScalars*>(base + kNoAllocPartials);
    double* r = base + kNoAllocPartials + kNoAllocScalars;
    double* p = r + kNoAllocMaxRows;
    double* q = p + kNoAllocMaxRows;
    double* inv = q + kNoAllocMaxRows;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int RB = kNoAllocBlocks;
    // the workspace keeps the previous call's contents: the scalars (reduction tickets, flags)
    // must start at zero
    if (cudaMemsetAsync(s, 0, sizeof(CgScalars), st) != cudaSuccess) return NB2_E_CUDA;
    unsigned int* flag = &s->counter[3];
    CgScalars hs;
    auto read_flag = [&](unsigned int* out) {
        if (cudaMemcpyAsync(&hs, s, sizeof hs, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return false;
        *out = hs.counter[3];
        return true;
    };
    unsigned int bad = 0;
    k_check_rowptr<<<RB, kRedThreads, 0, st>>>(n, rowptr, flag);
    if (!read_flag(&bad)) return NB2_E_CUDA;
    if (bad != 0) return NB2_E_INPUT;
    k_check_columns<<<RB, kRedThreads, 0, st>>>(n, rowptr, col, flag);
    if (!read_flag(&bad)) return NB2_E_CUDA;
    if (bad != 0) return NB2_E_INPUT;
    if (cudaMemsetAsync(s, 0, sizeof(CgScalars), st) != cudaSuccess) return NB2_E_CUDA;
    if (cudaMemcpyAsync(&s->max_iterations, &maximum_iterations, sizeof(int),
                        cudaMemcpyHostToDevice, st) != cudaSuccess)
        return NB2_E_CUDA;
    Csr A{rowptr, col, values, n};
    k_csr_invdiag<<<(n + 255) / 256, 256, 0, st>>>(A, inv);
    k_init<double><<<RB, kRedThreads, 0, st>>>(n, b, x, r, p, inv, s, partials, tolerance);
    int guard = 0;
    for (;;) {
        if (++guard > maximum_iterations / kChunk + 4) return NB2_E_TIMEOUT;
        if (csr_chunk(A, x, r, p, q, inv, s, partials, RB, st) != cudaSuccess) return NB2_E_CUDA;
        if (cudaMemcpyAsync(&hs, s, sizeof hs, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return NB2_E_CUDA;
        if (hs.done) break;
    }
    if (cudaGetLastError() != cudaSuccess) return NB2_E_CUDA;
    if (iterations) *iterations = hs.iterations;
    if (error) *error = hs.rhs_norm2 > 0 ? std::sqrt(hs.rr / hs.rhs_norm2) : 0.0;
    return hs.status ? hs.status : NB2_OK;
}

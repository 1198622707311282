// Dense reduced-camera-system solve S x = b_s on the device (sm_103a).
//
// Factorisation: ba_chol_fx.cu (k_chol_fx), which also inverts L's 32 x 32
// diagonal blocks (D_k = L_kk^-1).
// Triangular solves: one thread-block cluster (16 CTAs, or 8 where 16 is not
// allowed) walks the 32-row blocks with cluster barriers, each block step a
// small GEMV with D_k; the mixed form's FP64 refinement sweeps
// x += (L L^T)^-1 (b - S x) run inside the same launch and stop once the
// residual has converged.
//
// The pivot and solve tests are zeroslam's (gpdaniels/zeroslam
// source/matrix_decomposition_cholesky.hpp:40,53 and :74,80,89): a pivot must
// exceed 1e-14 * max|S_ii| and every |L_ii| must exceed 1e-7 * max|L_ii|.
#include <cooperative_groups.h>

#include <algorithm>

#include "ba_internal.h"

namespace cg = cooperative_groups;

namespace zs {

constexpr int kNB = 32;

// Loads of data that another CTA of the same launch wrote (persistent and
// cluster kernels) go through L2, never a possibly stale L1 line.
template <typename T>
__device__ __forceinline__ T ldg2(const T* p) {
    return __ldcg(p);
}
__device__ __forceinline__ int ld_ok(const LmState* st) { return __ldcg(&st->solve_ok); }

template <typename T>
__global__ void __launch_bounds__(kThreads) k_diag_max(int n, const T* __restrict__ A, LmState* st, double factor,
                                                       int which) {
    __shared__ double sh[kThreads];
    double m = 0.0;
    for (int i = threadIdx.x; i < n; i += kThreads) m = fmax(m, fabs((double)A[(int64_t)i * n + i]));
    sh[threadIdx.x] = m;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + s]);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (which == 0) st->eps_factor = sh[0] * factor;
        else st->eps_solve = sh[0] * factor;
    }
}

template <typename TS, typename TF>
__global__ void __launch_bounds__(kThreads) k_convert(int64_t N, const TS* __restrict__ src, TF* __restrict__ dst) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < N) dst[i] = (TF)src[i];
}

// Every |L_ii| must exceed 1e-7 max |L_ii|.
template <typename T>
__global__ void __launch_bounds__(kThreads) k_check_solve_eps(int n, const T* __restrict__ F, LmState* st) {
    __shared__ double sh[kThreads];
    __shared__ int bad;
    if (!st->solve_ok || st->skip_factor) return;
    double m = 0.0;
    for (int i = threadIdx.x; i < n; i += kThreads) m = fmax(m, fabs((double)F[(int64_t)i * n + i]));
    sh[threadIdx.x] = m;
    if (threadIdx.x == 0) bad = 0;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + s]);
        __syncthreads();
    }
    const double eps = sh[0] * 1e-7;
    for (int i = threadIdx.x; i < n; i += kThreads)
        if (!(fabs((double)F[(int64_t)i * n + i]) > eps)) bad = 1;
    __syncthreads();
    if (threadIdx.x == 0) {
        st->eps_solve = eps;
        if (bad) st->solve_ok = 0;
    }
}

__device__ inline double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Cluster-wide deterministic sum: each CTA publishes its partial in global
// scratch, then every CTA adds them in rank order.
__device__ inline double cluster_sum(cg::cluster_group& cl, double v, double* scratch) {
    if (threadIdx.x == 0) scratch[cl.block_rank()] = v;
    cl.sync();
    double s = 0.0;
    for (unsigned r = 0; r < cl.num_blocks(); ++r) s += ldg2(scratch + r);
    cl.sync();
    return s;
}

// Stages D_k (32 x 32, as double) and the kb entries of w_k in shared memory
// with independent loads (w_k may come from another CTA of the cluster).
template <typename T>
__device__ void stage_block(const T* Dk, const double* wk, int kb, double (*ds)[kNB + 1], double* ws) {
    T v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = Dk[threadIdx.x + q * kThreads];
    const double wv = (threadIdx.x < kb) ? ldg2(wk + threadIdx.x) : 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int e = threadIdx.x + q * kThreads;
        ds[e >> 5][e & 31] = (double)v[q];
    }
    if (threadIdx.x < kNB) ws[threadIdx.x] = wv;
    __syncthreads();
}

// x = (L L^T)^-1 rhs by blocked forward and backward substitution; w is the
// running right-hand side, y the forward result. Block b (32 rows) belongs to
// cluster CTA b % C. Ends with a cluster barrier.
template <typename T>
__device__ void cluster_trisolve(cg::cluster_group& cl, int n, const T* __restrict__ F, const T* __restrict__ D,
                                 const double* rhs, double* w, double* y, double* x, double* xs,
                                 double (*ds)[kNB + 1], double* ws) {
    const unsigned C = cl.num_blocks(), me = cl.block_rank();
    const int nblk = (n + kNB - 1) / kNB;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if ((unsigned)((i / kNB) % C) == me) w[i] = rhs[i];
    cl.sync();
    for (int k = 0; k < nblk; ++k) {
        const int k0 = k * kNB, kb = min(kNB, n - k0);
        // y_k = D_k w_k (every CTA, redundantly; w_k and D_k staged in shared memory)
        stage_block<T>(D + (int64_t)k * kNB * kNB, w + k0, kb, ds, ws);
        if (threadIdx.x < kNB) {
            const int c = threadIdx.x;
            double v = 0.0;
#pragma unroll 8
            for (int m = 0; m < kNB; ++m) v += (m <= c) ? ds[c][m] * ws[m] : 0.0;
            xs[c] = (c < kb) ? v : 0.0;
        }
        __syncthreads();
        if ((unsigned)(k % C) == me)
            for (int c = threadIdx.x; c < kb; c += blockDim.x) y[k0 + c] = xs[c];
        // w_i -= L_i,k y_k for the rows of later blocks this CTA owns, a warp per row
        for (int b = k + 1; b < nblk; ++b) {
            if ((unsigned)(b % C) != me) continue;
            const int b0 = b * kNB, bb = min(kNB, n - b0);
            for (int r = warp; r < bb; r += nw) {
                const int i = b0 + r;
                double part = (lane < kb) ? (double)F[(int64_t)i * n + k0 + lane] * xs[lane] : 0.0;
                part = warp_sum(part);
                if (lane == 0) w[i] -= part;
            }
        }
        cl.sync();
    }
    // backward: w = y, then x_k = D_k^T w_k and w_i -= sum_m L_{k0+m, i} x_m for i < k0
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if ((unsigned)((i / kNB) % C) == me) w[i] = y[i];
    cl.sync();
    for (int k = nblk - 1; k >= 0; --k) {
        const int k0 = k * kNB, kb = min(kNB, n - k0);
        stage_block<T>(D + (int64_t)k * kNB * kNB, w + k0, kb, ds, ws);
        if (threadIdx.x < kNB) {
            const int c = threadIdx.x;
            double v = 0.0;
#pragma unroll 8
            for (int m = 0; m < kNB; ++m) v += (m >= c) ? ds[m][c] * ws[m] : 0.0;
            xs[c] = (c < kb) ? v : 0.0;
        }
        __syncthreads();
        if ((unsigned)(k % C) == me)
            for (int c = threadIdx.x; c < kb; c += blockDim.x) x[k0 + c] = xs[c];
        for (int b = 0; b < k; ++b) {
            if ((unsigned)(b % C) != me) continue;
            const int b0 = b * kNB;
            for (int r = threadIdx.x; r < kNB; r += blockDim.x) {
                const int i = b0 + r;
                double acc = 0.0;
                for (int m = 0; m < kb; ++m) acc += (double)F[(int64_t)(k0 + m) * n + i] * xs[m];
                w[i] -= acc;
            }
        }
        cl.sync();
    }
}

// Solve, then (refine > 0) FP64 refinement sweeps against S until
// ||bs - S x|| <= tol ||bs||. Vectors w, y, d, r: n doubles each; scratch
// holds at least 16 doubles for the cluster sums.
template <typename TS, typename TF>
__global__ void __launch_bounds__(kThreads) k_solve_cluster(int n, const TS* __restrict__ S, const TF* __restrict__ F,
                                                            const TF* __restrict__ D, const double* __restrict__ bs,
                                                            double* x, double* w, double* y, double* d, double* r,
                                                            double* scratch, int refine, double tol, LmState* st) {
    __shared__ double xs[kNB];
    __shared__ double red[kThreads];
    __shared__ double ds[kNB][kNB + 1];
    __shared__ double ws[kNB];
    cg::cluster_group cl = cg::this_cluster();
    if (!ld_ok(st)) return;  // uniform across the cluster
    const unsigned C = cl.num_blocks(), me = cl.block_rank();
    cluster_trisolve<TF>(cl, n, F, D, bs, w, y, x, xs, ds, ws);
    if (refine <= 0) return;
    double bb = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if ((unsigned)((i / kNB) % C) == me) bb += bs[i] * bs[i];
    bb = block_sum(bb, red);
    const double bnorm2 = cluster_sum(cl, bb, scratch);
    int sweeps = 0;
    double rn2 = 0.0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int it = 0; it <= refine; ++it) {
        // r = bs - S x for this CTA's rows, a warp per row
        double part2 = 0.0;
        for (int blk = (int)me; blk * kNB < n; blk += (int)C) {
            const int b0 = blk * kNB, bnum = min(kNB, n - b0);
            for (int rr = warp; rr < bnum; rr += nw) {
                const int i = b0 + rr;
                double acc = 0.0;
                for (int c = lane; c < n; c += 32) acc += (double)S[(int64_t)i * n + c] * ldg2(x + c);
                acc = warp_sum(acc);
                const double ri = bs[i] - acc;
                if (lane == 0) {
                    r[i] = ri;
                    part2 += ri * ri;
                }
            }
        }
        part2 = block_sum(part2, red);
        rn2 = cluster_sum(cl, part2, scratch);
        if (it == refine || !(rn2 > tol * tol * bnorm2)) break;
        cluster_trisolve<TF>(cl, n, F, D, r, w, y, d, xs, ds, ws);
        for (int i = threadIdx.x; i < n; i += blockDim.x)
            if ((unsigned)((i / kNB) % C) == me) x[i] += d[i];
        cl.sync();
        ++sweeps;
    }
    if (me == 0 && threadIdx.x == 0) {
        st->resid_norm = sqrt(rn2);
        st->rhs_norm = sqrt(bnorm2);
        st->refine_sweeps = sweeps;
    }
}

template <typename TS, typename TF>
static int cluster_size() {
    static int cached = 0;
    if (cached) return cached;
    int c = 8;
    if (cudaFuncSetAttribute(k_solve_cluster<TS, TF>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
        cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(16);
        cfg.blockDim = dim3(kThreads);
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 16;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, k_solve_cluster<TS, TF>, &cfg) == cudaSuccess && clusters > 0)
            c = 16;
    }
    cudaGetLastError();
    cached = c;
    return c;
}

cudaError_t launch_factor(int n, const double* S, double* F, double* D, void* fx, LmState* st, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const cudaError_t e = launch_chol_fx(n, S, F, D, fx, st, s);
    if (e != cudaSuccess) return e;
    k_check_solve_eps<double><<<1, kThreads, 0, s>>>(n, F, st); note_launch();
    return cudaGetLastError();
}

// Preconditioner retry: armed only after a failed factorisation.
__global__ void k_retry_arm(LmState* st) {
    if (threadIdx.x == 0) {
        const int failed = !st->solve_ok;
        st->skip_factor = !failed;
        st->shifted = failed;
        if (failed) st->solve_ok = 1;
    }
}
__global__ void k_retry_disarm(LmState* st) {
    if (threadIdx.x == 0) st->skip_factor = 0;
}
// F = S + mu diag(S) (FP32) when a retry is armed.
__global__ void __launch_bounds__(kThreads) k_convert_shift(int n, const double* __restrict__ S, float* __restrict__ F,
                                                            double mu, const LmState* st) {
    if (st->skip_factor) return;
    const int64_t nn = (int64_t)n * n;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nn; i += (int64_t)gridDim.x * blockDim.x) {
        const double v = S[i];
        F[i] = (float)(i / n == i % n ? v + mu * fabs(v) : v);
    }
}

static cudaError_t launch_chol_inverse(int n, float* F, float* X, float* XT, float* scratch, TcStreams* ts,
                                       LmState* st, int* flags, int* epoch, cudaStream_t s) {
    if (scratch && ts && chol_tc_applies(n) && tc_gemm_supported(n, n, F, X))
        return launch_chol_inverse_tc(n, F, X, XT, scratch, st, flags, epoch, *ts, s);
    return launch_chol_inverse_dag(n, F, X, XT, st, flags, epoch, s);
}

cudaError_t launch_factor_dag(int n, const double* S, float* F, float* X, float* XT, float* scratch, TcStreams* ts,
                              LmState* st, int* flags, int* epoch, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int64_t nn = (int64_t)n * n;
    k_diag_max<double><<<1, kThreads, 0, s>>>(n, S, st, 1e-14, 0); note_launch();
    k_convert<double, float><<<grid_for(nn), kThreads, 0, s>>>(nn, S, F); note_launch();
    cudaError_t e = launch_chol_inverse(n, F, X, XT, scratch, ts, st, flags, epoch, s);
    if (e != cudaSuccess) return e;
    k_check_solve_eps<float><<<1, kThreads, 0, s>>>(n, F, st); note_launch();
    return cudaGetLastError();
}

cudaError_t launch_preconditioner(int n, const double* S, float* F, float* X, float* XT, float* scratch,
                                  TcStreams* ts, LmState* st, double mu, int* flags, int* epoch, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int64_t nn = (int64_t)n * n;
    cudaError_t e = launch_factor_dag(n, S, F, X, XT, scratch, ts, st, flags, epoch, s);
    if (e != cudaSuccess) return e;
    k_retry_arm<<<1, 32, 0, s>>>(st); note_launch();
    if (scratch && ts && chol_tc_applies(n)) {
        // The blocked form's retry would be some 200 launches that return at
        // once; the host reads the arm flag instead (one synchronisation,
        // against milliseconds of factorisation) and launches the retry only
        // when it is armed.
        int32_t armed = 0;
        if ((e = cudaMemcpyAsync(&armed, &st->shifted, sizeof(armed), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
            (e = cudaStreamSynchronize(s)) != cudaSuccess)
            return e;
        if (!armed) {
            k_retry_disarm<<<1, 32, 0, s>>>(st); note_launch();
            return cudaGetLastError();
        }
    }
    k_convert_shift<<<std::min<int64_t>(grid_for(nn), 4096), kThreads, 0, s>>>(n, S, F, mu, st); note_launch();
    e = launch_chol_inverse(n, F, X, XT, scratch, ts, st, flags, epoch, s);
    if (e != cudaSuccess) return e;
    k_check_solve_eps<float><<<1, kThreads, 0, s>>>(n, F, st); note_launch();
    k_retry_disarm<<<1, 32, 0, s>>>(st); note_launch();
    return cudaGetLastError();
}

template <typename TS, typename TF>
cudaError_t launch_solve_refine(int n, const TS* S, const TF* F, const TF* D, const double* bs, double* x,
                                double* work, LmState* st, int refine_iters, double tol, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int C = cluster_size<TS, TF>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = C;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    double* w = work;
    double* y = work + n;
    double* d = work + 2 * (int64_t)n;
    double* r = work + 3 * (int64_t)n;
    double* scratch = work + 4 * (int64_t)n;
    cudaError_t e =
        cudaLaunchKernelEx(&cfg, k_solve_cluster<TS, TF>, n, S, F, D, bs, x, w, y, d, r, scratch, refine_iters, tol, st);
    if (e != cudaSuccess) return e;
    note_launch();
    return cudaSuccess;
}

cudaError_t launch_reduced_solve(int n, const double* S, double* F, double* D, void* fx, const double* bs, double* x,
                                 double* work, LmState* st, cudaStream_t s) {
    const cudaError_t e = launch_factor(n, S, F, D, fx, st, s);
    if (e != cudaSuccess) return e;
    return launch_solve_refine<double, double>(n, S, F, D, bs, x, work, st, 0, 0.0, s);
}

template cudaError_t launch_solve_refine<double, double>(int, const double*, const double*, const double*,
                                                         const double*, double*, double*, LmState*, int, double,
                                                         cudaStream_t);

}  // namespace zs

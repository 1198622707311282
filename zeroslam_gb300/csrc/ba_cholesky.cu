// The dense reduced camera system's solves: in FP64 the factor (ba_chol_fx.cu)
// and the triangular solves (ba_trisolve.cu); the mixed form's FP32
// preconditioner around ba_chol_dag.cu and ba_chol_tc.cu.
//
// The pivot and solve tests are zeroslam's (gpdaniels/zeroslam
// source/matrix_decomposition_cholesky.hpp:40,53 and :74,80,89): a pivot must
// exceed 1e-14 * max|S_ii| and every |L_ii| must exceed 1e-7 * max|L_ii|.
#include <algorithm>

#include "ba_internal.h"

namespace zs {

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

cudaError_t launch_reduced_solve(int n, const double* S, double* F, void* fx, const double* bs, double* x, double* work,
                                 LmState* st, cudaStream_t s) {
    const cudaError_t e = launch_chol_fx(n, S, F, fx, st, s);
    if (e != cudaSuccess) return e;
    return launch_trisolve(n, F, bs, x, work, st, s);
}

}  // namespace zs

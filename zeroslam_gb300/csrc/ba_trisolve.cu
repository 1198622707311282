// x = (L L^T)^-1 b for the FP64 factor, by blocks of 32 rows in one launch
// (matrix::solve_cholesky, source/matrix_decomposition_cholesky.hpp:63-95,
// with its test |L_ii| > 1e-7 max |L_ii|).
//
// Block row i has one owner CTA. Forward, it adds L_ik y_k for k < i as each
// y_k appears, then y_i = D_i (b_i - sum), D_i = L_ii^-1 formed before the
// chain reaches it; backward the same with L^T from the last block. A step
// of the chain is then the last product, two sums over eight lanes and the
// product with D_i, each a few FP64 instructions of 64 cycles, and one
// transfer through L2.
//
// The values carry their own flags: y and x are filled with all-ones words
// (a NaN no arithmetic here yields) before the launch and a reader polls the
// words that it needs, so a transfer costs one round trip and no fence. A
// poll gives up after a bounded number of tries: the launch is then marked
// aborted (every other poll returns), st->timeout set and st->solve_ok
// cleared. Every sum has one owner and a fixed order.
#include <cooperative_groups.h>

#include <cstdlib>

#include "ba_internal.h"

namespace zs {

namespace {

constexpr int kB = 32;
constexpr int kBL = kB + 1;
constexpr int kTriThreads = 256;
constexpr long long kPollLimit = 1ll << 20;  // about a second
constexpr unsigned long long kUnset = ~0ull;

struct Tri {
    int n, nblk;
    const double* F;
    const double* b;
    double* x;     // the solution
    double* y;     // [n] forward values, [n] solution, both unset; then the abort word
    int* abort;
    LmState* st;
    int stall;     // a block that is never published (failure-path tests), else -1
};

__device__ __forceinline__ double load_relaxed(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

// p[0 .. count) (count <= 4, zeros beyond) once they are set, all loads in
// flight together; ok = false when the launch was aborted or the polls ran out.
__device__ __forceinline__ void poll4(const Tri& d, const double* p, int count, double (&v)[4], bool& ok) {
    for (long long it = 1;; ++it) {
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = u < count ? load_relaxed(p + u) : 0.0;
        bool set = true;
#pragma unroll
        for (int u = 0; u < 4; ++u) set = set && (unsigned long long)__double_as_longlong(v[u]) != kUnset;
        if (set) return;
        if ((it & 255) == 0) {
            int a;
            asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(a) : "l"(d.abort) : "memory");
            if (a) ok = false;
            if (it > kPollLimit) {
                d.st->timeout = 1;
                d.st->solve_ok = 0;
                asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(d.abort), "r"(1) : "memory");
                ok = false;
            }
        }
        if (!ok) return;
    }
}

__device__ __forceinline__ void put(double* p, double v) {
    // a NaN of all ones would read as unset
    if ((unsigned long long)__double_as_longlong(v) == kUnset) v = __longlong_as_double(0x7ff8000000000000ll);
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

__device__ __forceinline__ double sum8(double v) {
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// D = L_kk^-1 (identity beyond n) into D (row stride kBL): X = I, then per
// column k row k is divided by L_kk and taken off the rows below.
__device__ void invert_block(const Tri& d, int k0, double* D, double (*l)[kBL], double* inv) {
    const int t = threadIdx.x, r = t >> 3, q = t & 7;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int row = k0 + r, c = 8 * m + q, col = k0 + c;
        l[r][c] = row < d.n && col < d.n && c <= r ? __ldg(d.F + (int64_t)row * d.n + col) : (r == c ? 1.0 : 0.0);
    }
    __syncthreads();
    if (t < kB) inv[t] = 1.0 / l[t][t];
    double w[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) w[m] = 8 * m + q == r ? 1.0 : 0.0;
    __syncthreads();
    const int mtop = (r | 3) >> 3;  // the warp's last column group
    for (int k = 0; k < kB; ++k) {
        if (r == k) {
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (m <= mtop) {
                    w[m] *= inv[k];
                    D[k * kBL + 8 * m + q] = w[m];
                }
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (m > mtop) D[k * kBL + 8 * m + q] = 0.0;
        }
        __syncthreads();
        if (r > k) {
            const double a = l[r][k];
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (m <= (k >> 3)) w[m] = fma(-a, D[k * kBL + 8 * m + q], w[m]);
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kTriThreads, 1) k_trisolve(Tri d) {
    extern __shared__ double D[];  // the owned blocks' inverses
    __shared__ double l[kB][kBL];
    __shared__ double w[kB];
    __shared__ double red[kTriThreads / 32][kBL];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, r = t >> 3, q = t & 7;
    const int n = d.n, G = gridDim.x;
    if (!__ldcg(&d.st->solve_ok)) return;
    // the solve test, in every CTA alike
    {
        double m = 0.0;
        for (int i = t; i < n; i += kTriThreads) m = fmax(m, fabs(__ldg(d.F + (int64_t)i * n + i)));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
        if (lane == 0) w[warp] = m;
        __syncthreads();
        m = w[lane & 7];
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
        const double eps = m * 1e-7;
        int bad = 0;
        for (int i = t; i < n; i += kTriThreads)
            if (!(fabs(__ldg(d.F + (int64_t)i * n + i)) > eps)) bad = 1;
        bad = __syncthreads_or(bad);
        if (blockIdx.x == 0 && t == 0) {
            d.st->eps_solve = eps;
            if (bad) d.st->solve_ok = 0;
        }
        if (bad) return;
    }
    int owned = 0;
    for (int i = blockIdx.x; i < d.nblk; i += G) invert_block(d, kB * i, D + (owned++) * kB * kBL, l, &red[0][0]);
    bool ok = true;
    double* xs = d.y + n;
    // forward: thread (r, q) takes columns 4 q .. 4 q + 3 of row r
    int o = 0;
    for (int i = blockIdx.x; i < d.nblk; i += G, ++o) {
        const int row = kB * i + r;
        const double* Lr = d.F + (int64_t)min(row, n - 1) * n + 4 * q;
        double acc = 0.0;
        double a[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u] = i > 0 ? __ldg(Lr + u) : 0.0;
        for (int k = 0; k < i; ++k) {
            double c[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                c[u] = a[u];
                if (k + 1 < i) a[u] = __ldg(Lr + kB * (k + 1) + u);
            }
            double yk[4];
            poll4(d, d.y + kB * k + 4 * q, 4, yk, ok);
#pragma unroll
            for (int u = 0; u < 4; ++u) acc = fma(c[u], yk[u], acc);
        }
        acc = sum8(acc);
        if (q == 0) w[r] = row < n ? __ldg(d.b + row) - acc : 0.0;
        if (__syncthreads_or(!ok)) return;
        const double* Di = D + o * kB * kBL + r * kBL + 4 * q;
        double v = 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u) v = fma(Di[u], w[4 * q + u], v);
        v = sum8(v);
        if (q == 0 && row < n && i != d.stall) put(d.y + row, v);
        __syncthreads();
    }
    // backward: lane c takes column c, warp g rows 4 g .. 4 g + 3 of a tile
    for (int i = (d.nblk - 1 - (int)blockIdx.x) / G * G + blockIdx.x; i >= 0; i -= G) {
        --o;
        const int col = min(kB * i + lane, n - 1);
        const double* Lc = d.F + col;
        double acc = 0.0;
        double a[4];
        auto load = [&](int k, double (&v)[4]) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int rr = kB * k + 4 * warp + u;
                v[u] = rr < n ? __ldg(Lc + (int64_t)rr * n) : 0.0;
            }
        };
        if (i + 1 < d.nblk) load(d.nblk - 1, a);
        for (int k = d.nblk - 1; k > i; --k) {
            double c[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) c[u] = a[u];
            if (k - 1 > i) load(k - 1, a);
            const int r0 = kB * k + 4 * warp;
            double xk[4];
            poll4(d, xs + r0, min(4, n - r0), xk, ok);  // (c is 0 beyond n)
#pragma unroll
            for (int u = 0; u < 4; ++u) acc = fma(c[u], xk[u], acc);
        }
        red[warp][lane] = acc;
        if (__syncthreads_or(!ok)) return;
        const int row = kB * i + r;  // thread (r, q) adds warp q's part of column r
        const double s = sum8(red[q][r]);
        // (y of an owned block was written by this CTA)
        if (q == 0) w[r] = row < n ? load_relaxed(d.y + row) - s : 0.0;
        __syncthreads();
        const double* Di = D + o * kB * kBL + r;
        double v = 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u) v = fma(Di[(4 * q + u) * kBL], w[4 * q + u], v);
        v = sum8(v);
        if (q == 0 && row < n) {
            put(xs + row, v);
            d.x[row] = v;
        }
        __syncthreads();
    }
}

int stall_block_from_env() {
    const char* v = std::getenv("ZS_TEST_STALL_TRISOLVE");
    return v && *v ? std::atoi(v) : -1;
}

}  // namespace

cudaError_t launch_trisolve(int n, const double* F, const double* b, double* x, double* work, LmState* st,
                            cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    static const int stall = stall_block_from_env();
    static std::atomic<int> sm_count[kMaxDevices];
    const int sms = per_device(sm_count, [&] {
        int dev = 0, v = 0, most = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (cudaFuncSetAttribute(k_trisolve, cudaFuncAttributeMaxDynamicSharedMemorySize, most - 16384) != cudaSuccess)
            return 0;
        return v;
    });
    if (sms < 1) {
        const cudaError_t e = cudaGetLastError();
        return e != cudaSuccess ? e : cudaErrorInvalidConfiguration;
    }
    Tri d;
    d.n = n;
    d.nblk = (n + kB - 1) / kB;
    d.F = F;
    d.b = b;
    d.x = x;
    d.y = work;
    d.abort = reinterpret_cast<int*>(work + 2 * (int64_t)n);
    d.st = st;
    d.stall = stall;
    cudaError_t e = cudaMemsetAsync(work, 0xff, 2 * sizeof(double) * (size_t)n, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(d.abort, 0, sizeof(double), s);
    if (e != cudaSuccess) return e;
    const int G = d.nblk < sms ? d.nblk : sms;
    const size_t smem = sizeof(double) * kB * kBL * (size_t)((d.nblk + G - 1) / G);
    void* args[] = {(void*)&d};
    e = cudaLaunchCooperativeKernel((const void*)k_trisolve, dim3(G), dim3(kTriThreads), args, smem, s);
    if (e == cudaSuccess) note_launch();
    return e;
}

}  // namespace zs

// The FP64 Cholesky factor S = L L^T of the reduced camera system
// (source/matrix_decomposition_cholesky.hpp:26-59, with its pivot test) in
// one launch, its products on the integer pipe.
//
// A GB300 SM quarter takes one FP64 multiply-add per two cycles, a warp's
// instruction 64 cycles (measured, whether its lanes are in use or not), and
// a 32 x 32 -> 64-bit integer multiply-add per 2.2. So the factor's products,
// nearly all of its work, run in fixed point, and FP64 is kept for what is
// sequential: the 32 x 32 diagonal blocks.
//
// Fixed point. Row r is scaled by 2^-e_r, 2^e_r >= sqrt(S_rr): for a positive
// definite S every |L_rc| 2^-e_r <= 1, every Schur complement's entry
// |C_rc| 2^-(e_r + e_c) <= 1, and every sum of products of scaled rows is at
// most 1 in magnitude (Cauchy-Schwarz), partial sums of absolute values
// included. A scaled value is q 2^-60, q = a1 2^30 + a0 with a0 in [-2^29,
// 2^29): a product is four integer multiply-adds (a1 b1; a1 b0 + a0 b1; the
// upper half of a0 b0), sums are exact. An entry is rounded at 2^-61 of its
// row's scale, where FP64's own sums round at 2^-53 of it. (It takes those
// bits: unlike FP64's, the rounding of a small entry is no smaller, and over
// the rows of a large matrix it adds up. With 2^-56 and a0 b0 dropped, the
// step of the 6,000-row loop was 4.6 times further from 64 bits than FP64's,
// with 2^-58 twice.)
// The diagonal entries' differences S_rr - sum and the diagonal blocks'
// elimination, with its pivot test, are FP64.
//
// Where a bound above does not hold, S is not positive definite and the
// factor fails, as the pivot test of the FP64 factor would: a scaled entry
// of C above 1.5 (or not finite), a tile row of L whose squares sum to more
// than 1.25, or a diagonal sum above 1.25. These are tested before a value is
// used, so that no sum can wrap unnoticed: a wrapped sum needs a row whose
// squares exceed its S_rr, and that row's diagonal task sees it.
//
// Tiles are T x T (32 or 64); every tile has one owner CTA that computes it
// completely, in a fixed order, and publishes it with a flag (cleared by
// k_fx_prepare): tile (i, j), i > j, is C_ij = S_ij - sum_{k<j} L_ik L_jk^T
// times L_jj^-T, by products with the inverses of L_jj's 32 x 32 diagonal
// blocks; such a product's error grows with the block's condition number, so
// each is corrected once with its residual, L += (C - L L_kk^T) L_kk^-T. Tasks are numbered column block by column block, CTA
// t mod G takes its tasks in increasing order, every dependency has a
// smaller number and all CTAs are co-resident (cooperative launch), so the
// lowest unfinished task can always proceed. With T = 32 the task of tile
// (c + 1, c) also factors diagonal tile c + 1. A wait gives up after a bounded number of polls: the
// launch is then marked aborted (every other wait returns), st->timeout set
// and st->solve_ok cleared.
#include <cooperative_groups.h>

#include <cstdlib>

#include "ba_fixed.cuh"
#include "ba_internal.h"

namespace zs {

namespace {

using namespace fixed;

constexpr int kFxThreads = 256;
constexpr int kFrac = 60;                       // q = scaled value x 2^kFrac
constexpr int kAccFrac = 2 * (kFrac - kLow);    // the sum of a1 b1 is in units of 2^-kAccFrac
constexpr ll kMaxQ = 3ll << (kFrac - 1);        // 1.5
constexpr ll kMaxDiag = 5ll << (kAccFrac - 2);  // 1.25
constexpr float kMaxRow = 1.25f;
constexpr long long kSpinLimit = 1ll << 20;  // polls of one flag before a wait gives up (about a second)

struct Fx {
    int n, N;
    const double* S;
    double* F;
    int2* Q;      // tiles (i, j), i >= j, at (i (i + 1) / 2 + j) T^2: (a0, a1) of L's entries in panels of 32
                  // columns (diagonal tiles unused)
    int2* G;      // per diagonal tile kBlocks<T> 32 x 32 blocks: scaled inverse, L (T = 64: X_11, L_21, L_11, L_22, X_22)
    const int* e; // [N T] row scales
    int* f;       // [N T] shifts of the products with the inverses' rows
    LmState* st;
    int* flag;    // tiles as Q: 1 once final
    int* abort;   // 1 once the launch has given up
    int stall;    // a task whose flags are never published (failure-path tests), else -1
};

__device__ __forceinline__ int64_t tri(int i, int j) { return (int64_t)i * (i + 1) / 2 + j; }

__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// As fixed::quantize, at most kMaxQ.
__device__ __forceinline__ ll quantize(double v, int sh, int& bad) { return fixed::quantize(v, sh, kMaxQ, bad); }

template <int RA, int RB>
struct Acc {
    ll hi[RA][RB], mid[RA][RB];  // sums of a1 b1 and a1 b0 + a0 b1
    int lo[RA][RB];              // sums of a0 b0 >> 32
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < RA; ++i)
#pragma unroll
            for (int j = 0; j < RB; ++j) {
                hi[i][j] = mid[i][j] = 0;
                lo[i][j] = 0;
            }
    }
    __device__ __forceinline__ void add(int i, int j, int a0, int a1, int b0, int b1) {
        hi[i][j] += (ll)a1 * b1;
        mid[i][j] += (ll)a1 * b0;
        mid[i][j] += (ll)a0 * b1;
        lo[i][j] += __mulhi(a0, b0);
    }
    // the carries: out of lo, of at most 16 products; out of mid, of 32 products
    // of scaled rows (at most 2^62.7, Cauchy-Schwarz) or of 8 others
    __device__ __forceinline__ void carry_lo() {
#pragma unroll
        for (int i = 0; i < RA; ++i)
#pragma unroll
            for (int j = 0; j < RB; ++j) {
                mid[i][j] += (ll)lo[i][j] << (32 - kLow);
                lo[i][j] = 0;
            }
    }
    __device__ __forceinline__ void carry() {
#pragma unroll
        for (int i = 0; i < RA; ++i)
#pragma unroll
            for (int j = 0; j < RB; ++j) {
                const ll c = mid[i][j] >> kLow;
                hi[i][j] += c;
                mid[i][j] -= c << kLow;
            }
    }
    // the sum in units of 2^-kAccFrac, to nearest
    __device__ __forceinline__ ll value(int i, int j) const { return hi[i][j] + ((mid[i][j] + (1ll << (kLow - 1))) >> kLow); }
    // the same in units of 2^-kFrac
    __device__ __forceinline__ ll value_q(int i, int j) const { return shift(value(i, j), kFrac - kAccFrac); }
};

constexpr int kE = 32;       // the diagonal blocks, and the columns of a panel
constexpr int kEL = kE + 1;
constexpr int kPL = kE + 2;  // pairs from row to row of a panel in shared memory: 16-byte aligned, an odd number of
                             // 16-byte words (16 consecutive rows fall in distinct banks)
constexpr int kBlk = kE * kPL;
template <int T>
constexpr int kBlocks = T == 64 ? 5 : 2;

// acc(i, j) += sum_{m < 32} A[ty + 16 i][m] B[tx + 16 j][m], thread (ty, tx) =
// (tid / 16, tid % 16); kLower: j <= i only; kRows: A and B are scaled rows.
template <bool kLower, bool kRows, int RA, int RB>
__device__ __forceinline__ void mac(const int2* A, const int2* B, Acc<RA, RB>& acc) {
    constexpr int kStep = kRows ? 16 : 8;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 1
    for (int m0 = 0; m0 < kE; m0 += kStep) {
#pragma unroll 2
        for (int m = m0; m < m0 + kStep; m += 2) {
            int4 a[RA], b[RB];
#pragma unroll
            for (int i = 0; i < RA; ++i) a[i] = *reinterpret_cast<const int4*>(A + (ty + 16 * i) * kPL + m);
#pragma unroll
            for (int j = 0; j < RB; ++j) b[j] = *reinterpret_cast<const int4*>(B + (tx + 16 * j) * kPL + m);
#pragma unroll
            for (int i = 0; i < RA; ++i)
#pragma unroll
                for (int j = 0; j < RB; ++j) {
                    if (kLower && j > i) continue;
                    acc.add(i, j, a[i].x, a[i].y, b[j].x, b[j].y);
                    acc.add(i, j, a[i].z, a[i].w, b[j].z, b[j].w);
                }
        }
        acc.carry_lo();
        if (!kRows) acc.carry();
    }
    if (kRows) acc.carry();
}

// Two CTAs fit an SM: while one waits for a tile or runs a diagonal block, the
// other's products fill the integer pipe.
template <int T>
struct Smem {
    // the sums' operand panels; then buf[0], buf[1]: C and L of a panel, or the
    // FP64 diagonal tile; from buf[2] on: the diagonal tile's blocks
    __align__(16) int2 buf[4][T * kPL];
    __align__(16) int2 extra[T == 64 ? 2 : 1][T == 64 ? kBlk : 2];
    double lraw[kE * kEL];  // the elimination's columns a_rc
    double x[kE * kEL];     // L^-1 of the diagonal block
    double row[2][kE];      // the published row
    double pinv[2];
    double piv[kE], rs[kE];  // d_c, d_c^-1/2
    int shift[T];
    __device__ __forceinline__ int2* blk(int i) { return i < 4 ? buf[2] + i * kBlk : extra[0]; }
    __device__ __forceinline__ double* c() { return reinterpret_cast<double*>(buf[0]); }
};
static_assert(sizeof(double) * 64 * 65 <= sizeof(int2) * 2 * 64 * kPL, "the diagonal tile fits two panels");

// 1 / d: the hardware's approximation and one step of Halley's iteration
// y (1 + e + e^2), e = 1 - d y, which cubes its error.
__device__ __forceinline__ double reciprocal(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// Factors the 32 x 32 block C (row stride cl, lower triangle read, kb valid
// rows) by elimination on [C | I] in place: at step c column c, with its
// pivot's reciprocal, is published, every row r > c takes a_rc / d_c times
// row c (by symmetry column c) away from its part left of the diagonal, and
// column c, done, becomes column c of the right half. It ends with E = L'^-1,
// C = L' D L'^T, so L^-1 = D^-1/2 E (to x) and L_rc = a_rc d_c^-1/2 (a_rc in
// lraw, d_c^-1/2 in rs). Row c is taken from column c, not from a copy above
// the diagonal: two copies drift apart by rounding, which a small pivot would
// magnify. Thread t owns row t / 8 and columns 8 m + t % 8 <= row. A step is
// one barrier and six FP64 instructions deep, and those hold the FP64 pipe
// (each 64 cycles a warp). Returns 0 when a pivot fails its test (uniform).
template <int T>
__device__ __noinline__ int eliminate(Smem<T>& sm, const double* C, int cl, int kb, double eps) {
    const int t = threadIdx.x, r = t >> 3, q = t & 7, grp = t & 31 & ~7;
    const int mtop = (r | 3) >> 3;  // the warp's last column group
    double w[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int j = 8 * m + q;
        w[m] = j <= r ? C[r * cl + j] : 0.0;
    }
    int fail = 0;
#pragma unroll
    for (int c = 0; c < kE; ++c) {
        const int mc = c >> 3, qc = c & 7;
        double* row = sm.row[c & 1];
        const double arc = __shfl_sync(0xffffffffu, w[mc], grp | qc);
        if (r == c) {
            if (q == qc) {
                const double d = w[mc];
                if (c < kb && !(d > eps)) fail = 1;
                sm.piv[c] = d;
                sm.pinv[c & 1] = reciprocal(d);
            }
#pragma unroll
            for (int m = 0; m <= mc; ++m)
                if (8 * m + q < c) row[8 * m + q] = w[m];
        } else if (r > c && q == qc) {
            row[r] = arc;
            sm.lraw[r * kEL + c] = arc;
        }
        __syncthreads();
        if (r > c) {
            const double coef = arc * sm.pinv[c & 1];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int m = (k + ((c + 1) >> 3)) & 3;  // the next pivot's column first
                if (m > mtop) continue;
                if (m == mc && q == qc) w[m] = -coef;
                else w[m] = fma(-coef, row[8 * m + q], w[m]);
            }
        }
    }
    if (__syncthreads_or(fail)) return 0;
    if (t < kE) sm.rs[t] = rsqrt(sm.piv[t]);
    __syncthreads();
    const double rr = sm.rs[r];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int j = 8 * m + q;
        sm.x[r * kEL + j] = j < r ? w[m] * rr : (j == r ? rr : 0.0);
    }
    __syncthreads();
    return 1;
}

// The diagonal block's L (zeros above the diagonal) into F. k0: its first row.
template <int T>
__device__ void store_block(const Fx& d, const Smem<T>& sm, int k0) {
    const int kb = min(kE, d.n - k0);
#pragma unroll
    for (int m = 0; m < kE * kE / kFxThreads; ++m) {
        const int el = threadIdx.x + m * kFxThreads, r = el >> 5, c = el & 31;
        if (r < kb && c < kb)
            d.F[(int64_t)(k0 + r) * d.n + k0 + c] =
                c < r ? sm.lraw[r * kEL + c] * sm.rs[c] : (c == r ? sm.piv[r] * sm.rs[r] : 0.0);
    }
}

// Scales the inverse's rows: row c of X 2^{e_m} (column m) is below 2^F, kept
// as X 2^{e_m - F - 3}, so that a product of 32 entries of C with it cannot
// overflow; the product times 2^{F + 3} is the scaled L, shift_out[c] takes
// its value() to kFrac. Lb: the block's L, scaled.
template <int T>
__device__ void scale_blocks(const Fx& d, Smem<T>& sm, int k0, int2* X, int2* Lb, int* shift_out, int& bad) {
    const int t = threadIdx.x, r = t >> 3, q = t & 7;
    const int er = d.e[k0 + r];
    double v[4];
    int em[4], top = -8192;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int j = 8 * m + q;
        v[m] = sm.x[r * kEL + j];
        em[m] = d.e[k0 + j];
        top = max(top, exponent(v[m]) + em[m]);
    }
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, off));
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int j = 8 * m + q;
        X[r * kPL + j] = split(quantize(v[m], kFrac - 3 + em[m] - top, bad));
        const double l = j < r ? sm.lraw[r * kEL + j] * sm.rs[j] : (j == r ? sm.piv[r] * sm.rs[r] : 0.0);
        Lb[r * kPL + j] = split(quantize(l, kFrac - er, bad));
    }
    if (q == 0) shift_out[r] = top + 3 + kFrac - kAccFrac;
}

// The rows ty + 16 a, columns tx + 16 b (b < 2) of L = C L_kk^-T from the
// scaled C in c: the product with the inverse X, then its correction with the
// residual against Lb = L_kk. bufC, bufL: panels of 16 RA rows; L stays in
// bufL (visible after the caller's barrier), bad is set where a row of L
// leaves its bound.
template <int RA>
__device__ __forceinline__ void solve_panel(const ll (&c)[RA][2], ll (&l)[RA][2], const int2* X, const int2* Lb,
                                            const int (&sh)[2], int2* bufC, int2* bufL, int& bad) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    Acc<RA, 2> u;
    auto at = [&](int a, int b) { return (ty + 16 * a) * kPL + tx + 16 * b; };
#pragma unroll
    for (int a = 0; a < RA; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            if (llabs(c[a][b]) > kMaxQ) bad = 1;
            bufC[at(a, b)] = split(c[a][b]);
        }
    __syncthreads();
    u.zero();
    mac<false, false>(bufC, X, u);
#pragma unroll
    for (int a = 0; a < RA; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const ll v = u.value(a, b);
            if (llabs(v) > (sh[b] > 0 ? kMaxQ >> min(sh[b], 63) : (1ll << 62))) bad = 1;
            l[a][b] = shift(v, sh[b]);
            bufL[at(a, b)] = split(l[a][b]);
        }
    __syncthreads();
    u.zero();
    mac<false, true>(bufL, Lb, u);
#pragma unroll
    for (int a = 0; a < RA; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) bufC[at(a, b)] = split(c[a][b] - u.value_q(a, b));
    __syncthreads();
    u.zero();
    mac<false, false>(bufC, X, u);
#pragma unroll
    for (int a = 0; a < RA; ++a) {
        float sq = 0.f;
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            l[a][b] += shift(u.value(a, b), sh[b]);
            bufL[at(a, b)] = split(l[a][b]);
            const float f = (float)(int)(l[a][b] >> 32) * (1.f / (1 << (kFrac - 32)));
            sq = fmaf(f, f, sq);
        }
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
        if (!(sq <= kMaxRow)) bad = 1;
    }
}

__device__ __forceinline__ void give_up(const Fx& d) {
    if (threadIdx.x == 0) {
        d.st->solve_ok = 0;
        __threadfence();
        st_release(d.abort, 1);
    }
}

// Threads 0 and 32 wait for the two flags; false (uniform) when the launch
// was aborted or a wait ran out.
__device__ bool wait_flags(const Fx& d, const int* fa, const int* fb) {
    int ok = 1;
    if (threadIdx.x == 0 || threadIdx.x == 32) {
        const int* p = threadIdx.x == 0 ? fa : fb;
        long long it = 0;
        unsigned ns = 32;
        while (ld_acquire(p) == 0) {
            if (ld_acquire(d.abort) != 0) {
                ok = 0;
                break;
            }
            if (++it > kSpinLimit) {
                d.st->timeout = 1;
                d.st->solve_ok = 0;
                __threadfence();
                st_release(d.abort, 1);
                ok = 0;
                break;
            }
            __nanosleep(ns);
            if (ns < 256) ns *= 2;
        }
    }
    return __syncthreads_and(ok) != 0;
}

__device__ bool flags_ready(const int* fa, const int* fb) {
    int ok = 1;
    if (threadIdx.x == 0) ok = ld_acquire(fa) != 0;
    if (threadIdx.x == 32) ok = ld_acquire(fb) != 0;
    return __syncthreads_and(ok) != 0;
}

__device__ void publish(const Fx& d, int* f, int task) {
    __syncthreads();
    if (threadIdx.x == 0 && task != d.stall) {
        __threadfence();
        st_release(f, 1);
    }
}

// kRows x 32 contiguous pairs into a panel in shared memory, asynchronously.
template <int kRows>
__device__ __forceinline__ void load_panel(const int2* src, int2* dst) {
#pragma unroll
    for (int k = 0; k < kRows * kE / 2 / kFxThreads; ++k) {
        const int el = threadIdx.x + k * kFxThreads, r = el >> 4, c = 2 * (el & 15);
        cp_async16(dst + r * kPL + c, src + r * kE + c);
    }
}

// accL += sum_{k<j} L_ik L_jk^T (kL) and accD += sum_{k<j} L_ik L_ik^T (kD,
// lower triangle), a panel of 32 columns at a time; the next panels are
// copied while the current ones are multiplied when their flags are already
// set. bad: a diagonal sum left its bound.
template <int T, bool kL, bool kD>
__device__ bool accumulate(const Fx& d, int i, int j, Smem<T>& sm, Acc<T / 16, T / 16>& accL, Acc<T / 16, T / 16>& accD,
                           int& bad) {
    constexpr int H = T / kE;
    if (j <= 0) return true;
    const int64_t ri = tri(i, 0), rj = kL ? tri(j, 0) : ri;
    auto issue = [&](int p, int buf) {
        load_panel<T>(d.Q + ri * T * T + (int64_t)p * T * kE, sm.buf[buf]);
        if (kL) load_panel<T>(d.Q + rj * T * T + (int64_t)p * T * kE, sm.buf[2 + buf]);
        cp_async_commit();
    };
    if (!wait_flags(d, d.flag + ri, d.flag + rj)) return false;
    issue(0, 0);
    for (int p = 0; p < j * H; ++p) {
        const int buf = p & 1, k1 = (p + 1) / H;
        const bool more = p + 1 < j * H;
        bool pre = false;
        if (more && ((p + 1) % H != 0 || flags_ready(d.flag + ri + k1, d.flag + rj + k1))) {
            issue(p + 1, buf ^ 1);
            pre = true;
        }
        if (pre) cp_async_wait<1>();
        else cp_async_wait<0>();
        __syncthreads();
        if (kL) {
            mac<false, true>(sm.buf[buf], sm.buf[2 + buf], accL);
        }
        if (kD) {
            mac<true, true>(sm.buf[buf], sm.buf[buf], accD);
            if ((threadIdx.x & 15) == threadIdx.x >> 4) {
#pragma unroll
                for (int a = 0; a < T / 16; ++a)
                    if (accD.hi[a][a] > kMaxDiag) bad = 1;
            }
        }
        __syncthreads();
        if (more && !pre) {
            if (!wait_flags(d, d.flag + ri + k1, d.flag + rj + k1)) return false;
            issue(p + 1, buf ^ 1);
        }
    }
    return true;
}

// The diagonal tile jb from its FP64 lower triangle in sm.c(): factor, scaled
// blocks and L.
template <int T>
__device__ bool finish_diag(const Fx& d, int jb, int task, Smem<T>& sm, int bad) {
    constexpr int CL = T + 1;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int k0 = T * jb;
    const double eps = __ldcg(&d.st->eps_factor);
    double* c = sm.c();
    int ok = eliminate<T>(sm, c, CL, min(kE, d.n - k0), eps);
    if (!ok) bad = 1;
    ll l21[2][2];
    if constexpr (T == 32) {
        if (ok) scale_blocks<T>(d, sm, k0, sm.blk(0), sm.blk(1), sm.shift, bad);
    } else if (ok) {
        scale_blocks<T>(d, sm, k0, sm.blk(0), sm.blk(2), sm.shift, bad);
        // L_21 = C_21 L_11^-T, then C_22 -= L_21 L_21^T
        ll q[2][2];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int r = kE + ty + 16 * a, cc = tx + 16 * b;
                q[a][b] = quantize(c[r * CL + cc], kFrac - d.e[k0 + r] - d.e[k0 + cc], bad);
            }
        __syncthreads();
        const int sh[2] = {sm.shift[tx], sm.shift[tx + 16]};
        solve_panel<2>(q, l21, sm.blk(0), sm.blk(2), sh, sm.extra[1], sm.blk(1), bad);
        store_block<T>(d, sm, k0);
        __syncthreads();
        Acc<2, 2> u;
        u.zero();
        mac<false, true>(sm.blk(1), sm.blk(1), u);
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const int r = kE + ty + 16 * a;
            const double sr = pow2(d.e[k0 + r] - kAccFrac);
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int cc = kE + tx + 16 * b;
                if (cc <= r)
                    c[r * CL + cc] = fma(-(double)u.value(a, b) * sr, pow2(d.e[k0 + cc]), c[r * CL + cc]);
            }
        }
        __syncthreads();
        ok = eliminate<T>(sm, c + kE * CL + kE, CL, min(kE, d.n - k0 - kE), eps);
        if (!ok) bad = 1;
        if (ok) scale_blocks<T>(d, sm, k0 + kE, sm.blk(4), sm.blk(3), sm.shift + kE, bad);
    }
    if (__syncthreads_or(bad)) {
        give_up(d);
        return false;
    }
    int2* out = d.G + (int64_t)jb * kBlocks<T> * kE * kE;
#pragma unroll
    for (int k = 0; k < kBlocks<T> * kE * kE / kFxThreads; ++k) {
        const int el = threadIdx.x + k * kFxThreads, bl = el >> 10, r = (el >> 5) & 31;
        out[el] = sm.blk(bl)[r * kPL + (el & 31)];
    }
    if (threadIdx.x < T) d.f[k0 + threadIdx.x] = sm.shift[threadIdx.x];
    publish(d, d.flag + tri(jb, jb), task);
    if (k0 + T - kE < d.n) store_block<T>(d, sm, k0 + T - kE);
    if constexpr (T == 64) {
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const int row = k0 + kE + ty + 16 * a;
            const double sr = pow2(d.e[row] - kFrac);
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int col = k0 + tx + 16 * b;
                if (row < d.n && col < d.n) d.F[(int64_t)row * d.n + col] = (double)l21[a][b] * sr;
            }
        }
    }
    __syncthreads();
    return true;
}

__device__ __forceinline__ double load_s(const Fx& d, int row, int col) {
    return row < d.n && col < d.n ? __ldg(d.S + (int64_t)row * d.n + col) : (row == col ? 1.0 : 0.0);
}

// sm.c() = S_ii - accD in FP64 (lower triangle; s: the thread's entries of S_ii).
template <int T>
__device__ void diag_difference(const Fx& d, int i, Smem<T>& sm, const Acc<T / 16, T / 16>& accD,
                                const double (&s)[T / 16][T / 16]) {
    constexpr int R = T / 16;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double* out = sm.c();
#pragma unroll
    for (int a = 0; a < R; ++a) {
        const double sr = pow2(d.e[T * i + ty + 16 * a] - kAccFrac);
#pragma unroll
        for (int b = 0; b <= a; ++b) {
            const int r = ty + 16 * a, c = tx + 16 * b;
            out[r * (T + 1) + c] = fma(-(double)accD.value(a, b) * sr, pow2(d.e[T * i + c]), s[a][b]);
        }
    }
}

template <int T>
__device__ __forceinline__ void load_diag_s(const Fx& d, int i, double (&s)[T / 16][T / 16]) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int a = 0; a < T / 16; ++a)
#pragma unroll
        for (int b = 0; b <= a; ++b) s[a][b] = load_s(d, T * i + ty + 16 * a, T * i + tx + 16 * b);
}

// Tile (i, j), i > j; with kD (T = 32) also the diagonal tile i = j + 1, whose
// sums share the tiles L_ik: the chain of diagonal tiles then passes one flag
// a column.
template <int T, bool kD>
__device__ bool task_tile(const Fx& d, int i, int j, int task, Smem<T>& sm) {
    constexpr int R = T / 16, H = T / kE;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    int bad = 0;
    ll cq[H][R][2];  // the tile's entries of S, scaled; then of C; then of L
    auto load = [&] {
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int row = T * i + ty + 16 * a, col = T * j + kE * h + tx + 16 * b;
                    cq[h][a][b] = quantize(load_s(d, row, col), kFrac - d.e[row] - d.e[col], bad);
                }
    };
    if constexpr (T == 32) load();  // before anything is waited for (T = 64: after the sums, for their registers)
    {
        Acc<R, R> accL, accD;
        accL.zero();
        if (kD) accD.zero();
        if (!accumulate<T, true, kD>(d, i, j, sm, accL, accD, bad)) return false;
        if constexpr (T == 64) load();
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b) cq[h][a][b] -= accL.value_q(a, 2 * h + b);
        if (!wait_flags(d, d.flag + tri(j, j), d.flag + tri(j, j))) return false;
#pragma unroll
        for (int bl = 0; bl < kBlocks<T>; ++bl)
            load_panel<kE>(d.G + ((int64_t)j * kBlocks<T> + bl) * kE * kE, sm.blk(bl));
        cp_async_commit();
        int sh[H][2];
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
            for (int b = 0; b < 2; ++b) sh[h][b] = __ldcg(d.f + T * j + kE * h + tx + 16 * b);
        double s[R][R];
        if (kD) load_diag_s<T>(d, i, s);
        cp_async_wait<0>();
        // (the barrier in solve_panel makes the copies visible)
#pragma unroll
        for (int h = 0; h < H; ++h) {
            if (h > 0) {  // C_2 -= L_1 L_21^T
                Acc<R, 2> u;
                u.zero();
                mac<false, true>(sm.buf[1], sm.blk(1), u);
#pragma unroll
                for (int a = 0; a < R; ++a)
#pragma unroll
                    for (int b = 0; b < 2; ++b) cq[h][a][b] -= u.value_q(a, b);
                __syncthreads();
            }
            ll l[R][2];
            solve_panel<R>(cq[h], l, sm.blk(h == 0 ? 0 : 4), sm.blk(T == 32 ? 1 : 2 + h), sh[h], sm.buf[0], sm.buf[1], bad);
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    cq[h][a][b] = l[a][b];
                    d.Q[tri(i, j) * T * T + (h * T + ty + 16 * a) * kE + tx + 16 * b] = split(l[a][b]);
                }
            if (h + 1 < H) __syncthreads();
        }
        if (__syncthreads_or(bad)) {
            give_up(d);
            return false;
        }
        publish(d, d.flag + tri(i, j), task);
        if constexpr (kD) {
            mac<true, true>(sm.buf[1], sm.buf[1], accD);
            if (tx == ty) {
#pragma unroll
                for (int a = 0; a < R; ++a)
                    if (accD.hi[a][a] > kMaxDiag) bad = 1;
            }
            diag_difference<T>(d, i, sm, accD, s);
            __syncthreads();
        }
    }
    if constexpr (kD) {
        if (!finish_diag<T>(d, i, task, sm, bad)) return false;
    }
#pragma unroll
    for (int h = 0; h < H; ++h)
#pragma unroll
        for (int a = 0; a < R; ++a) {
            const int row = T * i + ty + 16 * a;
            const double sr = pow2(d.e[row] - kFrac);
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int col = T * j + kE * h + tx + 16 * b;
                if (row < d.n && col < d.n) d.F[(int64_t)row * d.n + col] = (double)cq[h][a][b] * sr;
            }
        }
    __syncthreads();
    return true;
}

// The diagonal tile j on its own.
template <int T>
__device__ bool task_diag(const Fx& d, int j, int task, Smem<T>& sm) {
    int bad = 0;
    {
        Acc<T / 16, T / 16> none, accD;
        accD.zero();
        if (!accumulate<T, false, true>(d, j, j, sm, none, accD, bad)) return false;
        double s[T / 16][T / 16];
        load_diag_s<T>(d, j, s);
        diag_difference<T>(d, j, sm, accD, s);
    }
    __syncthreads();
    return finish_diag<T>(d, j, task, sm, bad);
}

template <int T>
__global__ void __launch_bounds__(kFxThreads, 2) k_chol_fx(Fx d) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem<T>& sm = *reinterpret_cast<Smem<T>*>(smem_raw);
    if (!__ldcg(&d.st->solve_ok)) return;  // written by earlier launches: uniform
    const int tasks = (int)tri(d.N, 0);
    int c = 0, first = 0;  // column c's tasks are [first, first + N - c)
    for (int t = blockIdx.x; t < tasks; t += gridDim.x) {
        while (t >= first + d.N - c) {
            first += d.N - c;
            ++c;
        }
        const int r = t - first;
        bool ok = true;
        if (r == 0) {
            if (T == 64 || c == 0) ok = task_diag<T>(d, c, t, sm);
            // (T = 32, c > 0: the diagonal tile came with tile (c, c - 1))
        } else if (T == 32 && r == 1) {
            ok = task_tile<T, T == 32>(d, c + 1, c, t, sm);
        } else {
            ok = task_tile<T, false>(d, c + r, c, t, sm);
        }
        if (!ok) return;
    }
}

// eps_factor = 1e-14 max |S_ii|, the rows' scales, cleared flags. A diagonal
// entry at most eps fails at once: its pivot cannot exceed it.
__global__ void __launch_bounds__(1024) k_fx_prepare(int n, int rows, const double* __restrict__ S, int* e, int* flags,
                                                     int nflags, LmState* st) {
    __shared__ double sh[32];
    double m = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmax(m, fabs(S[(int64_t)i * n + i]));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    m = sh[threadIdx.x & 31];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
    const double eps = 1e-14 * m;
    int bad = 0;
    for (int i = threadIdx.x; i < rows; i += blockDim.x) {
        int p = 0;
        if (i < n) {
            const double v = S[(int64_t)i * n + i];
            if (!(v > eps) || !isfinite(v)) bad = 1;
            // 2^(p - 1) <= S_ii < 2^p (a subnormal's p is larger)
            p = (int)((__double_as_longlong(v) >> 52) & 0x7ff) - 1022;
        }
        e[i] = (p + 1) >> 1;
    }
    for (int i = threadIdx.x; i < nflags; i += blockDim.x) flags[i] = 0;
    if (__syncthreads_or(bad)) bad = 1;
    if (threadIdx.x == 0) {
        st->eps_factor = eps;
        if (bad) st->solve_ok = 0;
    }
}

int stall_task_from_env() {
    const char* v = std::getenv("ZS_TEST_STALL_FX_TASK");
    return v && *v ? std::atoi(v) : -1;
}

template <int T>
cudaError_t launch_fx(Fx& d, int tasks, cudaStream_t s) {
    static std::atomic<int> resident[kMaxDevices];
    const size_t smem = sizeof(Smem<T>);
    const int co = per_device(resident, [&] {
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaFuncSetAttribute(k_chol_fx<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_chol_fx<T>, kFxThreads, smem) != cudaSuccess)
            return 0;
        return sms * per_sm;
    });
    if (co < 1) {
        const cudaError_t e = cudaGetLastError();
        return e != cudaSuccess ? e : cudaErrorInvalidConfiguration;
    }
    void* args[] = {(void*)&d};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_chol_fx<T>, dim3(tasks < co ? tasks : co),
                                                      dim3(kFxThreads), args, smem, s);
    if (e == cudaSuccess) note_launch();
    return e;
}

}  // namespace

cudaError_t launch_chol_fx(int n, const double* S, double* F, void* work, LmState* st, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    static const int stall = stall_task_from_env();
    const FxLayout l = fx_layout(n);
    unsigned char* w = static_cast<unsigned char*>(work);
    Fx d;
    d.n = n;
    d.N = l.N;
    d.S = S;
    d.F = F;
    d.Q = reinterpret_cast<int2*>(w);
    d.G = reinterpret_cast<int2*>(w + l.g);
    int* e = reinterpret_cast<int*>(w + l.e);
    d.e = e;
    d.f = reinterpret_cast<int*>(w + l.f);
    d.flag = reinterpret_cast<int*>(w + l.flag);
    d.abort = d.flag + l.tiles;
    d.st = st;
    d.stall = stall;
    k_fx_prepare<<<1, 1024, 0, s>>>(n, l.N * l.T, S, e, d.flag, l.tiles + 1, st); note_launch();
    return l.T == 32 ? launch_fx<32>(d, l.tiles, s) : launch_fx<64>(d, l.tiles, s);
}

}  // namespace zs

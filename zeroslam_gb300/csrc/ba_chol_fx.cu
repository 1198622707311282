// The FP64 Cholesky factor S = L L^T of the reduced camera system
// (source/matrix_decomposition_cholesky.hpp:26-59, with its pivot test) in
// one launch, its products on the integer pipe.
//
// A GB300 SM quarter takes one FP64 multiply-add per two cycles, a warp's
// instruction 64 cycles (measured, whether its lanes are in use or not), and
// a 32 x 32 -> 64-bit integer multiply-add per about three. So the factor
// runs in fixed point: its products, nearly all of its work, and the chain of
// pivots, whose every step would otherwise wait on several FP64
// instructions.
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
// with 2^-58 twice. With 2^-60 the solutions of the reduced systems of arcs, walks
// and loops are 1.6 to 60 times nearer to extended precision than with FP64 sums.
// What is below 2^-60 of its row's scale is lost, where FP64 would hold it: parts
// of a solution that many orders below the rest.) A pivot is compared with 1e-14 max |S_ii| in its row's scale.
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
// times L_jj^-T by substitution; the diagonal tile j is factored in blocks of
// 32 columns. Tasks are numbered column block by column block, CTA
// t mod G takes its tasks in increasing order, every dependency has a
// smaller number and all CTAs are co-resident (cooperative launch), so the
// lowest unfinished task can always proceed. With T = 32 the task of tile
// (c + 1, c) also factors diagonal tile c + 1. A wait gives up after a
// bounded number of polls: the launch is then marked aborted (every other
// wait returns), st->timeout set and st->solve_ok cleared.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>

#include "ba_fixed.cuh"
#include "ba_internal.h"

namespace zs {

namespace {

using namespace fixed;

constexpr int kFxThreads = 256;
constexpr int kFrac = 60;                       // q = scaled value x 2^kFrac
static_assert(2 * (kFrac - kLow) == kFrac, "sums of a1 b1 are in units of 2^-kFrac");
constexpr ll kMaxQ = 3ll << (kFrac - 1);        // 1.5
constexpr ll kMaxDiag = 5ll << (kFrac - 2);  // 1.25
constexpr float kMaxRow = 1.25f;
constexpr long long kSpinLimit = 1ll << 20;  // polls of one flag before a wait gives up (about a second)

struct Fx {
    int n, N;
    const double* S;
    double* F;
    int2* Q;      // tiles (i, j), i >= j, at (i (i + 1) / 2 + j) T^2: (a0, a1) of L's entries in panels of 32
                  // columns (diagonal tiles unused)
    int2* G;      // per diagonal tile kBlocks<T> 32 x 32 blocks of its L (T = 64: L_11, L_21, L_22)
    const int* e; // [N T] row scales
    int4* f;      // [N T] columns' pivots: Pivot
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
    // the sum in units of 2^-kFrac, to nearest
    __device__ __forceinline__ ll value(int i, int j) const {
        return hi[i][j] + ((mid[i][j] + ((ll)lo[i][j] << (32 - kLow)) + (1ll << (kLow - 1))) >> kLow);
    }
};

constexpr int kE = 32;       // the diagonal blocks, and the columns of a panel
constexpr int kEL = kE + 1;
constexpr int kPL = kE + 2;  // pairs from row to row of a panel in shared memory: 16-byte aligned, an odd number of
                             // 16-byte words (16 consecutive rows fall in distinct banks)
constexpr int kBlk = kE * kPL;
template <int T>
constexpr int kBlocks = T == 64 ? 3 : 1;

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
// other's products fill the integer multiply pipe (n = 4700: 69% busy; at 1200, where
// the diagonal tiles' chain is all, 16%).
template <int T>
struct Smem {
    // the sums' operand panels; then buf[0]: C of a panel, buf[1]: L of a panel,
    // from buf[2] on: the diagonal tile's blocks
    __align__(16) int2 buf[4][T * kPL];
    __align__(16) int4 piv[T];
    float part[kFxThreads];
    // (row-major blocks, stride kPL: L_21; by columns, stride kE: L_11, L_22)
    __device__ __forceinline__ int2* blk(int i) { return buf[2] + i * kBlk; }
    // the columns of the L that substitute() works on
    __align__(16) int2 cols[T * kE];
    __device__ __forceinline__ ll* c() { return reinterpret_cast<ll*>(buf[0]); }
};
static_assert(sizeof(ll) * 64 * kEL <= sizeof(int2) * 64 * kPL, "C of a panel fits");

// Reciprocal square root of a pivot: y 2^-61 2^((s - 3) / 2) for some s, y < 2^62; as
// int4 (y low, y high, the shift of a product with it, -).
struct Pivot {
    ll y;
    int sh;
};
__device__ __forceinline__ int4 pack(const Pivot& p) { return make_int4((int)p.y, (int)(p.y >> 32), p.sh, 0); }
__device__ __forceinline__ Pivot unpack(const int4& v) { return {(ll)(unsigned)v.x | (ll)v.y << 32, v.z}; }

// 1 / sqrt(d 2^-kFrac), d > 0: v = d 2^s 2^-63 in [1/4, 1), the hardware's
// approximation y0 of v^-1/2 and one step of the third-order iteration
// y0 (1 + h / 2 + 3 h^2 / 8), h = 1 - v y0^2 (the series of (1 - h)^-1/2; h is
// about 2^-21, so its error is below 2^-62).
__device__ __forceinline__ Pivot rsqrt_pivot(ll d) {
    int s = __clzll(d) - 1;
    s -= (s & 1) ^ 1;  // odd: d 2^-60 = v 2^(3 - s) is then v times a power of four
    const unsigned long long m = (unsigned long long)d << s;
    const float v = (float)(unsigned)(m >> 32) * 0x1p-31f;
    float yf;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(v));
    const unsigned y0 = (unsigned)(yf * 0x1p30f);
    const ll h = (1ll << 59) - (ll)__umul64hi(m, (unsigned long long)y0 * y0);  // 2^-59 steps
    const int hh = (int)(h >> 10);
    const ll e = (h >> 1) + ((3 * ((ll)hh * hh)) >> 42);
    const ll y1 = (ll)y0 << 31;
    // (v = 1/4 ends at 2^62, which the upper of scale_by's limbs does not hold)
    return {min(y1 + (__mul64hi(y1, e << 24) >> 19), (1ll << 62) - 1), 61 - ((s - 3) >> 1)};
}

// a times the pivot's reciprocal square root, to nearest, from limbs of 31
// bits; bad: far above 1 (the row's squares are checked too).
__device__ __forceinline__ ll scale_by(ll a, const Pivot& p, bool mine, int& bad) {
    constexpr int kMask = 0x7fffffff;
    const int a1 = (int)(a >> 31), a0 = (int)(a & kMask), y1 = (int)(p.y >> 31), y0 = (int)(p.y & kMask);
    const ll top = (ll)a1 * y1;
    const ll t = (ll)a1 * y0 + (ll)a0 * y1 + ((ll)a0 * y0 >> 31);
    if (mine && (llabs(top) >> (p.sh - 1)) != 0) bad = 1;
    return (top << (62 - p.sh)) + (t >> (p.sh - 31)) + ((t >> (p.sh - 32)) & 1);
}

// sq + (l 2^-kFrac)^2.
__device__ __forceinline__ float add_square(float sq, ll l) {
    const float f = (float)(int)(l >> 32) * (1.f / (1 << (kFrac - 32)));
    return fmaf(f, f, sq);
}

// The sequential parts, a column at a time. Lane = row, and the columns of a
// block are dealt to the NW warps of its rows: the warp that owns column c
// finishes it (a reciprocal square root, a 64-bit product: some 60 integer
// instructions, run by that warp alone), one barrier, and every warp takes it
// off its own later columns. Sums are kept whole until their column is due.
// (The inner loop stays a loop: a step's code runs once a block, and unrolled
// 32 times it does not fit the instruction cache. Threads of one row sharing
// its columns, with shuffles, took twice the time: every lane then runs the
// owner's instructions.)
//
// Lt: the diagonal block's L by columns (row j of column c at c kE + j); part:
// a float per thread.

// Every row's squares, summed over the NW warps of its group, are within
// their bound (uniform over the row's lanes of each group's first warp).
template <int NW>
__device__ __forceinline__ void check_rows(float sq, float* part, int& bad) {
    part[threadIdx.x] = sq;
    __syncthreads();
    if ((threadIdx.x >> 5) % NW == 0) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) v += part[threadIdx.x + 32 * w];
        if (!(v <= kMaxRow)) bad = 1;
    }
}

// Factors the 32 x 32 block C = L L^T (64-bit, row stride kEL, lower triangle
// read): Lt (zeros above the diagonal) and piv; a pivot of the block's kb rows
// must exceed eps in its row's scale. Returns 0 when one fails (uniform).
__device__ __noinline__ int factor_block(const ll* C, int2* Lt, int4* piv, float* part, int kb, const Fx& d, int k0,
                                         double eps) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ll a[4];
    Acc<1, 4> acc;
    acc.zero();
#pragma unroll
    for (int m = 0; m < 4; ++m) a[m] = 8 * m + warp <= lane ? C[lane * kEL + 8 * m + warp] : 0;
    int bad = 0;
    float sq = 0.f;
    ll limit = 0;  // of row lane's pivot
    if (lane < kb) {
        int none = 0;
        limit = max(quantize(eps, kFrac - 2 * d.e[k0 + lane], none), 0ll);
    }
    auto take = [&](int m, int c) {
        const int2 l = Lt[c * kE + lane], u = Lt[c * kE + 8 * m + warp];
        acc.add(0, m, l.x, l.y, u.x, u.y);
    };
#pragma unroll
    for (int mc = 0; mc < 4; ++mc) {
#pragma unroll 1
        for (int qc = 0; qc < 8; ++qc) {
            const int c = 8 * mc + qc;
            if (warp == qc) {
                if (c > 0) take(mc, c - 1);  // the column before, to this one alone
                const ll v = a[mc] - acc.value(0, mc);
                if (lane == c && !(v > limit)) bad = 1;
                const Pivot p = rsqrt_pivot(max(__shfl_sync(0xffffffffu, v, c), 1ll));
                ll l = scale_by(v, p, lane >= c, bad);
                if (lane < c) l = 0;
                Lt[c * kE + lane] = split(l);
                if (lane == 0) piv[c] = pack(p);
                sq = add_square(sq, l);
            }
            if (c > 0) {  // while the owner works, and to its other columns when it is done
#pragma unroll
                for (int m = mc; m < 4; ++m)
                    if (m > mc || warp > qc) take(m, c - 1);
            }
            __syncthreads();
        }
        if (mc == 1) acc.carry_lo();
    }
    check_rows<8>(sq, part, bad);
    return __syncthreads_or(bad) == 0;
}

// L = C L_b^-T for 8 / NW groups of 32 rows: the warp's rows are lane of its
// group, its columns NW m + its number in the group. C: row stride kEL; Lt,
// piv: the diagonal block; out: L's rows (stride kPL), colbuf: its columns (32
// pairs a group and column); l: the thread's entries. bad: an entry or a row's
// squares leave their bound.
template <int NW>
__device__ __forceinline__ void substitute(const ll* C, const int2* Lt, const int4* piv, int2* out, int2* colbuf,
                                           float* part, ll (&l)[kE / NW], int& bad) {
    constexpr int CN = kE / NW;
    const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % NW, group = (threadIdx.x >> 5) / NW;
    const int r = 32 * group + lane;
    int2* mine = colbuf + group * kE * kE + lane;
    ll a[CN];
    Acc<1, CN> acc;
    acc.zero();
#pragma unroll
    for (int m = 0; m < CN; ++m) a[m] = C[r * kEL + NW * m + warp];
    float sq = 0.f;
    auto take = [&](int m, int c) {
        const int2 p = mine[c * kE], u = Lt[c * kE + NW * m + warp];
        acc.add(0, m, p.x, p.y, u.x, u.y);
    };
#pragma unroll
    for (int mc = 0; mc < CN; ++mc) {
#pragma unroll 1
        for (int qc = 0; qc < NW; ++qc) {
            const int c = NW * mc + qc;
            if (warp == qc) {
                if (c > 0) take(mc, c - 1);
                const ll v = scale_by(a[mc] - acc.value(0, mc), unpack(piv[c]), true, bad);
                const int2 p = split(v);
                mine[c * kE] = p;
                out[r * kPL + c] = p;
                l[mc] = v;
                sq = add_square(sq, v);
            }
            if (c > 0) {
#pragma unroll
                for (int m = mc; m < CN; ++m)
                    if (m > mc || warp > qc) take(m, c - 1);
            }
            __syncthreads();
        }
        if (mc == CN / 2 - 1) acc.carry_lo();
    }
    check_rows<NW>(sq, part, bad);
}

__device__ __forceinline__ double to_double(const int2& p, int e) {
    return (double)(((ll)p.y << kLow) + p.x) * pow2(e - kFrac);
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
__device__ __forceinline__ void load_panel(const int2* src, int2* dst, int stride = kPL) {
#pragma unroll
    for (int k = 0; k < kRows * kE / 2 / kFxThreads; ++k) {
        const int el = threadIdx.x + k * kFxThreads, r = el >> 4, c = 2 * (el & 15);
        cp_async16(dst + r * stride + c, src + r * kE + c);
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

__device__ __forceinline__ ll load_scaled(const Fx& d, int row, int col, int& bad) {
    // (not by the read-only path: the windows' factors are written over S in the same launch)
    const double v = row < d.n && col < d.n ? d.S[(int64_t)row * d.n + col] : (row == col ? 1.0 : 0.0);
    return quantize(v, kFrac - d.e[row] - d.e[col], bad);
}

// The diagonal tile jb from its scaled lower triangle: thread (ty, tx) holds
// c[a][b] at (ty + 16 a, tx + 16 b), b <= a.
template <int T>
__device__ bool finish_diag(const Fx& d, int jb, int task, Smem<T>& sm, ll (&c)[T / 16][T / 16], int bad) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int k0 = T * jb;
    const double eps = __ldcg(&d.st->eps_factor);
    ll* C = sm.c();
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b <= a; ++b) C[(ty + 16 * a) * kEL + tx + 16 * b] = c[a][b];
    __syncthreads();
    if (!factor_block(C, sm.blk(0), sm.piv, sm.part, min(kE, d.n - k0), d, k0, eps)) bad = 1;
    if constexpr (T == 64) {
        // L_21 = C_21 L_11^-T, C_22 -= L_21 L_21^T
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) C[(ty + 16 * a) * kEL + tx + 16 * b] = c[2 + a][b];
        __syncthreads();
        ll l[4];
        substitute<8>(C, sm.blk(0), sm.piv, sm.blk(1), sm.cols, sm.part, l, bad);
        __syncthreads();
        Acc<2, 2> u;
        u.zero();
        mac<true, true>(sm.blk(1), sm.blk(1), u);
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b <= a; ++b) C[(ty + 16 * a) * kEL + tx + 16 * b] = c[2 + a][2 + b] - u.value(a, b);
        __syncthreads();
        if (!factor_block(C, sm.blk(2), sm.piv + kE, sm.part, min(kE, d.n - k0 - kE), d, k0 + kE, eps)) bad = 1;
    }
    if (__syncthreads_or(bad)) {
        give_up(d);
        return false;
    }
    int2* out = d.G + (int64_t)jb * kBlocks<T> * kE * kE;
#pragma unroll
    for (int k = 0; k < kBlocks<T> * kE * kE / kFxThreads; ++k) {
        const int el = threadIdx.x + k * kFxThreads, bl = el >> 10, r = (el >> 5) & 31;
        out[el] = sm.blk(bl)[r * (bl == 1 ? kPL : kE) + (el & 31)];
    }
    if (threadIdx.x < T) d.f[k0 + threadIdx.x] = sm.piv[threadIdx.x];
    publish(d, d.flag + tri(jb, jb), task);
    // L into F, zeros above the diagonal
#pragma unroll
    for (int k = 0; k < kBlocks<T> * kE * kE / kFxThreads; ++k) {
        const int el = threadIdx.x + k * kFxThreads, bl = el >> 10;
        const int r = (el >> 5) & 31, cc = el & 31, at = bl == 1 ? r * kPL + cc : cc * kE + r;
        const int row = k0 + r + (bl > 0 ? kE : 0), col = k0 + cc + (bl > 1 ? kE : 0);
        if (row < d.n && col < d.n) d.F[(int64_t)row * d.n + col] = to_double(sm.blk(bl)[at], d.e[row]);
    }
    __syncthreads();
    return true;
}

// c = S_ii - accD, scaled (lower triangle).
template <int T>
__device__ __forceinline__ void diag_difference(const Fx& d, int i, const Acc<T / 16, T / 16>& accD,
                                                ll (&c)[T / 16][T / 16], int& bad) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int a = 0; a < T / 16; ++a)
#pragma unroll
        for (int b = 0; b <= a; ++b)
            c[a][b] = load_scaled(d, T * i + ty + 16 * a, T * i + tx + 16 * b, bad) - accD.value(a, b);
}

// Tile (i, j), i > j; with kD (T = 32) also the diagonal tile i = j + 1, whose
// sums share the tiles L_ik: the chain of diagonal tiles then passes one flag
// a column.
template <int T, bool kD>
__device__ bool task_tile(const Fx& d, int i, int j, int task, Smem<T>& sm) {
    constexpr int R = T / 16, H = T / kE, NW = kFxThreads / T, CN = kE / NW;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int r = (threadIdx.x >> 5) / NW * 32 + (threadIdx.x & 31), q = (threadIdx.x >> 5) % NW;  // as substitute()
    int bad = 0;
    ll cq[R][R];  // the tile's entries of S, scaled; then of C
    auto load = [&] {
#pragma unroll
        for (int a = 0; a < R; ++a)
#pragma unroll
            for (int b = 0; b < R; ++b) cq[a][b] = load_scaled(d, T * i + ty + 16 * a, T * j + tx + 16 * b, bad);
    };
    if constexpr (T == 32) load();  // before anything is waited for (T = 64: after the sums, for their registers)
    Acc<R, R> accD;
    if (kD) accD.zero();
    {
        Acc<R, R> accL;
        accL.zero();
        if (!accumulate<T, true, kD>(d, i, j, sm, accL, accD, bad)) return false;
        if constexpr (T == 64) load();
#pragma unroll
        for (int a = 0; a < R; ++a)
#pragma unroll
            for (int b = 0; b < R; ++b) cq[a][b] -= accL.value(a, b);
    }
    if (!wait_flags(d, d.flag + tri(j, j), d.flag + tri(j, j))) return false;
#pragma unroll
    for (int bl = 0; bl < kBlocks<T>; ++bl)
        load_panel<kE>(d.G + ((int64_t)j * kBlocks<T> + bl) * kE * kE, sm.blk(bl), bl == 1 ? kPL : kE);
    if (threadIdx.x < T) cp_async16(sm.piv + threadIdx.x, d.f + T * j + threadIdx.x);
    cp_async_commit();
    ll* C = sm.c();
    ll l[H][CN];
#pragma unroll
    for (int h = 0; h < H; ++h) {
        if (h > 0) {  // C_2 -= L_1 L_21^T
            Acc<R, 2> u;
            u.zero();
            mac<false, true>(sm.buf[1], sm.blk(1), u);
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b) cq[a][2 * h + b] -= u.value(a, b);
            // (C's and L's buffers are free: the barrier before h = 1, and the one below)
        }
#pragma unroll
        for (int a = 0; a < R; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) C[(ty + 16 * a) * kEL + tx + 16 * b] = cq[a][2 * h + b];
        if (h == 0) cp_async_wait<0>();
        __syncthreads();
        substitute<NW>(C, sm.blk(2 * h), sm.piv + kE * h, sm.buf[1], sm.cols, sm.part, l[h], bad);
        __syncthreads();
        int2* Qh = d.Q + tri(i, j) * T * T + h * T * kE;
#pragma unroll
        for (int k = 0; k < T * kE / kFxThreads; ++k) {
            const int el = threadIdx.x + k * kFxThreads;
            Qh[el] = sm.buf[1][(el >> 5) * kPL + (el & 31)];
        }
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
        ll c[R][R];
        diag_difference<T>(d, i, accD, c, bad);
        __syncthreads();
        if (!finish_diag<T>(d, i, task, sm, c, bad)) return false;
    }
    const int row = T * i + r;
    if (row < d.n) {
        const double sr = pow2(d.e[row] - kFrac);
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
            for (int m = 0; m < CN; ++m) {
                const int col = T * j + kE * h + NW * m + q;
                if (col < d.n) d.F[(int64_t)row * d.n + col] = (double)l[h][m] * sr;
            }
    }
    __syncthreads();
    return true;
}

// The diagonal tile j on its own.
template <int T>
__device__ bool task_diag(const Fx& d, int j, int task, Smem<T>& sm) {
    int bad = 0;
    ll c[T / 16][T / 16];
    {
        Acc<T / 16, T / 16> none, accD;
        accD.zero();
        if (!accumulate<T, false, true>(d, j, j, sm, none, accD, bad)) return false;
        diag_difference<T>(d, j, accD, c, bad);
    }
    return finish_diag<T>(d, j, task, sm, c, bad);
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

// A batch of windows: the same tiles, tasks (window, i, j) column by column
// over all windows, largest window first, taken from a queue. Whoever took a
// task's dependencies runs or has finished, so the lowest unfinished task can
// proceed whatever the grid. A window that fails or is not active is passed
// over by its abort flag.
__global__ void __launch_bounds__(kFxThreads, 2) k_chol_fx_windows(const FxWindow* __restrict__ win,
                                                                   const uint32_t* __restrict__ tasks, int ntasks,
                                                                   int* next, char* work, double* S, LmState* st,
                                                                   int stall) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem<32>& sm = *reinterpret_cast<Smem<32>*>(smem_raw);
    __shared__ int s_task;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_task = atomicAdd(next, 1);
        __syncthreads();
        const int t = s_task;
        if (t >= ntasks) return;
        const uint32_t task = tasks[t];
        const int w = (int)(task >> 8), i = (int)(task >> 4 & 15), j = (int)(task & 15);
        const FxWindow v = win[w];
        const FxLayout l = fx_layout(v.n);
        char* base = work + v.work;
        Fx d;
        d.n = v.n;
        d.N = l.N;
        d.S = S + v.s;
        d.F = S + v.s;  // (an entry is read by the one CTA that writes it, before it does)
        d.Q = reinterpret_cast<int2*>(base);
        d.G = reinterpret_cast<int2*>(base + l.g);
        d.e = reinterpret_cast<const int*>(base + l.e);
        d.f = reinterpret_cast<int4*>(base + l.f);
        d.flag = reinterpret_cast<int*>(base + l.flag);
        d.abort = d.flag + l.tiles;
        d.st = st + w;
        d.stall = stall;
        if (__syncthreads_or(threadIdx.x == 0 && ld_acquire(d.abort) != 0)) continue;
        if (i == j) task_diag<32>(d, j, t, sm);
        else if (i == j + 1) task_tile<32, true>(d, i, j, t, sm);
        else task_tile<32, false>(d, i, j, t, sm);
    }
}

// eps_factor = 1e-14 max |S_ii|, the rows' scales, cleared flags (the last one
// is the abort flag). A diagonal entry at most eps fails at once: its pivot
// cannot exceed it. Returns whether one did (in thread 0).
__device__ int fx_prepare(int n, int rows, const double* S, int* e, int* flags, int nflags, LmState* st) {
    __shared__ double sh[32];
    if (threadIdx.x < 32) sh[threadIdx.x] = 0.0;
    __syncthreads();
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
    if (threadIdx.x == 0) st->eps_factor = eps;
    return bad;
}

__global__ void __launch_bounds__(1024) k_fx_prepare(int n, int rows, const double* __restrict__ S, int* e, int* flags,
                                                     int nflags, LmState* st) {
    if (fx_prepare(n, rows, S, e, flags, nflags, st) && threadIdx.x == 0) st->solve_ok = 0;
}

// A CTA per window; st->solve_ok of active windows is set here.
__global__ void __launch_bounds__(128) k_fx_prepare_windows(const FxWindow* __restrict__ win, int* next, char* work,
                                                            const double* __restrict__ S, LmState* st,
                                                            const WinCtl* __restrict__ ctl) {
    const int w = blockIdx.x;
    if (w == 0 && threadIdx.x == 0) *next = 0;
    const FxWindow v = win[w];
    const FxLayout l = fx_layout(v.n);
    char* base = work + v.work;
    int* flag = reinterpret_cast<int*>(base + l.flag);
    int skip = 1;
    if (ctl[w].active) {
        skip = fx_prepare(v.n, l.N * l.T, S + v.s, reinterpret_cast<int*>(base + l.e), flag, l.tiles + 1, st + w);
        if (threadIdx.x == 0) st[w].solve_ok = !skip;
    }
    __syncthreads();
    if (threadIdx.x == 0) flag[l.tiles] = skip;
}

int stall_task_from_env() {
    const char* v = std::getenv("ZS_TEST_STALL_FX_TASK");
    return v && *v ? std::atoi(v) : -1;
}

// CTAs of the kernel that are resident together (0: an error is pending).
int resident_ctas(const void* kernel, size_t smem) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kFxThreads, smem) != cudaSuccess)
        return 0;
    return sms * per_sm;
}

template <int T>
cudaError_t launch_fx(Fx& d, int tasks, cudaStream_t s) {
    static std::atomic<int> resident[kMaxDevices];
    const size_t smem = sizeof(Smem<T>);
    const int co = per_device(resident, [&] { return resident_ctas((const void*)k_chol_fx<T>, smem); });
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
    d.f = reinterpret_cast<int4*>(w + l.f);
    d.flag = reinterpret_cast<int*>(w + l.flag);
    d.abort = d.flag + l.tiles;
    d.st = st;
    d.stall = stall;
    k_fx_prepare<<<1, 1024, 0, s>>>(n, l.N * l.T, S, e, d.flag, l.tiles + 1, st); note_launch();
    return l.T == 32 ? launch_fx<32>(d, l.tiles, s) : launch_fx<64>(d, l.tiles, s);
}

size_t fx_batch_plan(const std::vector<int>& n, const std::vector<int64_t>& s, std::vector<FxWindow>& win,
                     std::vector<uint32_t>& tasks) {
    win.assign(n.size(), FxWindow{});
    tasks.clear();
    size_t bytes = 0;
    std::vector<int> order(n.size());
    for (size_t w = 0; w < n.size(); ++w) {
        win[w] = {n[w], s[w], (int64_t)bytes};
        bytes += (chol_fx_bytes(n[w]) + 255) / 256 * 256;
        order[w] = (int)w;
    }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return n[a] > n[b]; });
    const int most = order.empty() ? 0 : fx_layout(n[order[0]]).N;
    for (int j = 0; j < most; ++j)
        for (int d = 0; j + d < most; ++d)  // (every window's diagonal tile, then the tiles below it)
            for (int w : order) {
                const int i = j + d;
                if (i >= fx_layout(n[w]).N) break;
                if (d == 0 && j > 0) break;  // with tile (j, j - 1)
                tasks.push_back((uint32_t)w << 8 | (uint32_t)i << 4 | (uint32_t)j);
            }
    return bytes;
}

cudaError_t launch_chol_fx_windows(const FxBatch& b, int nwin, double* S, LmState* st, const WinCtl* ctl,
                                   cudaStream_t s) {
    if (nwin < 1) return cudaSuccess;
    static const int stall = stall_task_from_env();
    static std::atomic<int> resident[kMaxDevices];
    const size_t smem = sizeof(Smem<32>);
    const int co = per_device(resident, [&] { return resident_ctas((const void*)k_chol_fx_windows, smem); });
    if (co < 1) {
        const cudaError_t e = cudaGetLastError();
        return e != cudaSuccess ? e : cudaErrorInvalidConfiguration;
    }
    k_fx_prepare_windows<<<nwin, 128, 0, s>>>(b.win, b.next, b.work, S, st, ctl);
    note_launch();
    if (b.ntasks > 0) {
        k_chol_fx_windows<<<std::min(b.ntasks, co), kFxThreads, smem, s>>>(b.win, b.tasks, b.ntasks, b.next, b.work, S,
                                                                          st, stall);
        note_launch();
    }
    return cudaGetLastError();
}

}  // namespace zs

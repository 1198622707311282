// Pose-only problems (every landmark fixed: zeroslam's tracking mode,
// map optimise(1, true, 50), source/slam.hpp:316,387,469) solved in one
// cooperative launch that runs the whole Levenberg-Marquardt loop of
// factor_graph::solve (source/factor_graph.hpp:489-615) on the device, with no
// host round trip per attempt.
//
// With every landmark fixed the landmark blocks vanish: no H_ll, no H_pl, and
// the reduced system is H_pp + lambda I, block diagonal with one 6 x 6 block
// per pose. Every CTA holds all poses, current and trial, and takes every
// decision itself from the same values by the same arithmetic; one grid
// barrier an attempt, around the observations' sums, is all they exchange:
//   * a warp factors a pose's damped block, a lane per entry of the lower
//     triangle with the right-hand side as its last row, with the reference's
//     pivot test (d > 1e-14 max |S_ii|,
//     source/matrix_decomposition_cholesky.hpp:41-57) and solve test
//     (|L_ii| > 1e-7 max |L_ii|, :74-89), and solves for the step;
//   * the trial poses (pose_plus in three parts, a warp each) and the model's
//     gain;
//   * one pass at the trial state gives its cost and, for the next iteration
//     if it is accepted, its system, on different SMs: a CTA takes a chunk of
//     256 observations' cost, or four warps' sums of a free pose's 27 terms
//     (J_p^T W J_p upper triangle and -J_p^T g, each observation's with the
//     rounding of the plain form's k_linearize); after the barrier every CTA
//     adds the warps' and chunks' sums in the same order;
//   * the reference's accept / reject decision (source/factor_graph.hpp:542-606):
//     a rejected step's poses and system are simply not taken.
//
// Bound by FP64 issue: any FP64 instruction of a warp holds its SM quarter's
// pipe for 64 cycles, so the time is the longest chain of one warp. Hence a
// warp per quarter (CTAs of four), one observation a lane (some 150 FP64
// instructions), sums by recursive halving (31 additions for 27 values where
// butterflies take 135), and no chain of one thread where lanes can share it.
// 6,802 observations, one free pose of five, three attempts: 375 us with a
// barrier and a pass for each of cost, system and sums and a thread a pose in
// the solve, 102 us now, the results bit for bit the same. The outer loop,
// its stopping rules and the attempt history follow the host loop of the
// general path (solve_impl). Both precisions take this path in FP64: there is
// no Schur complement or dense factor to make cheaper. Every sum has a fixed
// order for a given number of observations: results repeat bit for bit.
//
// Batches of such windows (many tracking problems at once) run the same loop
// with one CTA per window (k_pose_only_windows): the window's sums stay in
// its CTA, and the loop is shared with the single-problem kernel through a
// team type (GridTeam / WindowTeam: who sums, who synchronises).
#include <cooperative_groups.h>

#include <algorithm>

#include "../../include/zeroslam_ba.h"
#include "ba_internal.h"

namespace cg = cooperative_groups;

namespace zs {

namespace {

constexpr int kPoThreads = 128;     // a CTA of the grid: a warp per SM quarter
constexpr int kPoWinThreads = 256;  // a window's CTA
// Sums are formed as if by CTAs of 256 threads, ~64 observations of the
// problem a CTA: chunk c holds places 256 c .. 256 c + 255 of a range, and
// those a multiple of 256 pose_only_chunks(M) further on.
constexpr int kChunk = 256;
constexpr int kSys = 27;  // a pose's sums: J^T W J's upper triangle, row by row, then b
constexpr int kRec = 28;  // doubles from one warp's sums to the next's

// Places of a pose's sums: entry (i, j), i >= j, of the lower triangle; row 6 is b.
__device__ __forceinline__ constexpr int place(int i, int j) {
    return i == 6 ? 21 + j : 6 * j - j * (j - 1) / 2 + (i - j);
}

struct Observed {
    double X[3], Xc[3], r[2];
    const double* om;
    int front;
};
__device__ __forceinline__ Observed see(const DevProblem& P, const double p[7], int64_t o) {
    Observed v;
    const double* xp = P.lm + (int64_t)P.obs_lm[o] * kLmStride;
    const double2 uv = P.obs_uv[o];
    v.om = P.obs_info ? P.obs_info + 4 * o : nullptr;
#pragma unroll
    for (int i = 0; i < 3; ++i) v.X[i] = __ldg(xp + i);
    v.front = residual(p, v.X, uv.x, uv.y, P.intr, v.Xc, v.r);
    return v;
}

// Observation o's cost term at pose p (k_cost_partial's).
__device__ __forceinline__ double obs_cost(const DevProblem& P, const double p[7], int64_t o) {
    const Observed v = see(P, p, o);
    const double e2 = chi2_of(v.r, v.om);
    if (P.loss.kind) {
        double rho[3];
        loss_rho(P.loss, e2, rho);
        return rho[0];
    }
    return e2;
}

// Observation o's 27 pose terms added to acc: J_p^T W J_p (upper triangle) and
// -J_p^T g, formed as the plain form's k_linearize forms them, without the
// products with the zeros of the projection's Jacobian (c0, 0, c2; 0, c4, c5).
__device__ __forceinline__ void add_terms(const DevProblem& P, const double p[7], int64_t o, double acc[32]) {
    const Observed v = see(P, p, o);
    const double* r = v.r;
    const double* om = v.om;
    double c0 = 0.0, c2 = kBehindPenalty, c4 = 0.0, c5 = kBehindPenalty;
    if (v.front) {
        const double iz = 1.0 / v.Xc[2], iz2 = iz * iz;
        c0 = P.intr.fx * iz;
        c2 = -P.intr.fx * v.Xc[0] * iz2;
        c4 = P.intr.fy * iz;
        c5 = -P.intr.fy * v.Xc[1] * iz2;
    }
    double W[4] = {1.0, 0.0, 0.0, 1.0};
    double orr0 = r[0], orr1 = r[1], drho = 1.0;
    if (om) {
#pragma unroll
        for (int i = 0; i < 4; ++i) W[i] = om[i];
        orr0 = dot2_first(om[0], r[0], om[1], r[1]);
        orr1 = dot2_first(om[2], r[0], om[3], r[1]);
    }
    if (P.loss.kind) {
        const double e2 = chi2_of(r, om);
        double rho[3];
        loss_rho(P.loss, e2, rho);
        drho = rho[1];
#pragma unroll
        for (int i = 0; i < 4; ++i) W[i] *= rho[1];
        // rho' + 2 rho'' e2 as separately rounded multiply and add (no FMA),
        // as the reference evaluates it (its sign decides the rank-one term)
        if (rho[2] != 0.0 && __dadd_rn(rho[1], __dmul_rn(2.0 * rho[2], e2)) > 0.0) {
            const double k2 = 2.0 * rho[2];
            W[0] += k2 * orr0 * orr0;
            W[1] += k2 * orr0 * orr1;
            W[2] += k2 * orr1 * orr0;
            W[3] += k2 * orr1 * orr1;
        }
    }
    const double x = v.Xc[0], y = v.Xc[1], z = v.Xc[2];
    // rows 0 and 1 of J_p; row 0 has no entry 4, row 1 no entry 3
    const double j0[6] = {-(c2 * y), -(c0 * z - c2 * x), c0 * y, -c0, 0.0, -c2};
    const double j1[6] = {-(c5 * y - c4 * z), c5 * x, -(c4 * x), 0.0, -c4, -c5};
    const double g0 = drho * orr0, g1 = drho * orr1;
#pragma unroll
    for (int a = 0; a < 6; ++a) {
        double A0, A1;
        if (a == 3) {
            A0 = j0[a] * W[0];
            A1 = j0[a] * W[1];
        } else if (a == 4) {
            A0 = j1[a] * W[2];
            A1 = j1[a] * W[3];
        } else {
            A0 = dot2_second(j0[a], W[0], j1[a], W[2]);
            A1 = dot2_second(j0[a], W[1], j1[a], W[3]);
        }
#pragma unroll
        for (int c = a; c < 6; ++c) {
            double& t = acc[place(c, a)];
            if (c == 3) t += __dmul_rn(A0, j0[c]);
            else if (c == 4) t += __dmul_rn(A1, j1[c]);
            else t += dot2_first(A0, j0[c], A1, j1[c]);
        }
        double& t = acc[21 + a];
        if (a == 3) t -= __dmul_rn(j0[a], g0);
        else if (a == 4) t -= __dmul_rn(j1[a], g1);
        else t -= dot2_second(j0[a], g0, j1[a], g1);
    }
}

// Largest |v| as fmax forms it (a NaN counts as nothing), on the integer pipe.
__device__ __forceinline__ unsigned long long abs_bits(double v) {
    return isnan(v) ? 0ull : (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ double warp_max_bits(unsigned long long v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, off));
    return __longlong_as_double((long long)v);
}
template <int Lanes = 32>
__device__ __forceinline__ double lanes_add(double v) {
#pragma unroll
    for (int off = Lanes / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// The warp's sums of 32 values a lane, value l in lane l: lanes_add's tree by
// recursive halving (half of the values that are left go to the other half of
// the lanes each time: 31 additions where butterflies take 5 a value).
__device__ __forceinline__ double warp_sums(double (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < off; ++i) {
            const double give = up ? v[i] : v[i + off], keep = up ? v[i + off] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
    }
    return v[0];
}

// MK, MF: the most poses, and free ones among them; NT threads. Two states:
// the current one and the trial one. Free poses go by their number f, pose
// order[f].
template <int MK, int MF, int NT>
struct Shared {
    double pose[2][MK][kPoseStride];
    double sys[2][MF][kSys];
    double delta[MF][6];
    double lo[MF], hi[MF];  // of a pose's L_ii; lo = 0 where a pivot failed
    double plus[MF][kPlusParts];  // a trial pose's parts (pose_plus_part)
    double gain[64];        // the poses' shares of the model's gain
    double red[NT];
    double wpart[NT / 32][kRec];
    double lambda, nu, chi2, rho, scale;
    int order[MK];  // the free poses, in order
    int nfree;
    int good;
};

// The damped blocks' factors and the step delta of state b. A warp takes
// free poses warp, warp + NT / 32, ... (a fixed pose's block is lambda I and
// its step zero); uniform result over the CTA.
template <int MK, int MF, int NT>
__device__ bool solve_step(int K, int b, Shared<MK, MF, NT>& sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nf = sh.nfree;
    const double lam = sh.lambda;
    unsigned long long m = K > nf ? abs_bits(lam) : 0;
    for (int i = lane; i < 6 * nf; i += 32) m = max(m, abs_bits(sh.sys[b][i / 6][place(i % 6, i % 6)] + lam));
    const double eps_f = warp_max_bits(m) * 1e-14;
    // lane e < 27 holds entry (row, col) of [L; (L^-1 b)^T]
    int row = lane < kSys ? 6 : -1, col = lane - 21;
    if (lane < 21) {
        col = 0;
        while (lane > place(5, col)) ++col;
        row = col + lane - place(col, col);
    }
    for (int f = warp; f < nf; f += NT / 32) {
        double v = lane < kSys ? sh.sys[b][f][lane] : 0.0;
        if (row == col) v += lam;
        bool ok = true;
        double inv[6], x[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            const double d = __shfl_sync(0xffffffffu, v, place(c, c));
            ok = ok && d > eps_f;
            const double piv = sqrt(d);
            inv[c] = 1.0 / piv;
            if (col == c) v = row == c ? piv : v * inv[c];
            const bool due = lane < kSys && col > c;
            const double lr = __shfl_sync(0xffffffffu, v, due ? place(row, c) : lane);
            const double lc = __shfl_sync(0xffffffffu, v, due ? place(col, c) : lane);
            if (due) v = fma(-lr, lc, v);
        }
        const double hi = warp_max_bits(row == col ? abs_bits(v) : 0ull);
        unsigned long long lo = row == col ? abs_bits(v) : ~0ull;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, off));
#pragma unroll
        for (int i = 5; i >= 0; --i) {
            double t = __shfl_sync(0xffffffffu, v, 21 + i);
#pragma unroll
            for (int n = i + 1; n < 6; ++n) t = fma(-__shfl_sync(0xffffffffu, v, place(n, i)), x[n], t);
            x[i] = t * inv[i];
            if (lane == i) sh.delta[f][i] = x[i];
        }
        if (lane == 0) {
            sh.lo[f] = ok ? __longlong_as_double((long long)lo) : 0.0;
            sh.hi[f] = hi;
        }
    }
    __syncthreads();
    const double lfix = K > nf ? sqrt(lam) : 0.0;  // of the fixed poses' blocks
    unsigned long long h = abs_bits(lfix);
    for (int f = lane; f < nf; f += 32) h = max(h, abs_bits(sh.hi[f]));
    const double eps_s = warp_max_bits(h) * 1e-7;
    int good = K <= nf || (lam > eps_f && lfix > eps_s);
    for (int f = lane; f < nf; f += 32)
        if (!(sh.lo[f] > eps_s)) good = 0;
    return __all_sync(0xffffffffu, good) != 0;
}

// State b ^ 1: the free poses of state b moved by delta, and the model's gain
// delta^T (lambda delta + b) + 1e-3 into sh.scale. pose_plus
// (source/factor_graph.hpp:947-960) in three parts that do not wait on one
// another, a warp each; the gain is the fourth's.
template <int MK, int MF, int NT>
__device__ void trial_state(int b, Shared<MK, MF, NT>& sh) {
    static_assert(NT >= 128 && MF <= 32 && MK <= 64, "a warp per part, a lane per free pose");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nf = sh.nfree;
    if (warp < 3 && lane < nf) pose_plus_part(warp, sh.pose[b][sh.order[lane]], sh.delta[lane], sh.plus[lane]);
    if (warp == 3) {
        if (lane < nf) {
            double sc = 0.0;
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const double d = sh.delta[lane][i];
                sc += d * (sh.lambda * d + sh.sys[b][lane][21 + i]);
            }
            sh.gain[sh.order[lane]] = sc;
        }
        __syncwarp();
        const double v = lanes_add(sh.gain[lane] + sh.gain[lane + 32]);
        if (lane == 0) sh.scale = v + 1e-3;
    }
    __syncthreads();
    if (threadIdx.x < nf) {
        pose_plus_join(sh.plus[threadIdx.x], sh.delta[threadIdx.x], sh.pose[b ^ 1][sh.order[threadIdx.x]]);
    }
    __syncthreads();
}

// Who works on one problem: the whole cooperative grid (a single problem,
// poses 0 .. P.K) or one CTA (a window of a batch, poses k0 .. k0 + K).
// cost: of state b, the same in every thread. system: the free poses' sums at
// b (sh.sys[b]); the grid forms them with the cost, on SMs that would idle.
struct GridTeam {
    static constexpr int kThreadsOf = kPoThreads;
    using Sh = Shared<kPoseOnlyMaxK, kPoseOnlyMaxFree, kPoThreads>;
    cg::grid_group grid;
    double* scratch;  // of two passes by turns: chunks' costs [chunks], warps' sums [free poses][8 chunks][kRec]
    int chunks, turn;
    __device__ bool lead() const { return blockIdx.x == 0; }
    // 32 observations a lane apart from a free pose's, and the 8 warps of a chunk
    __device__ int warps_of(const DevProblem& P, int k) const {
        return min(8 * chunks, (P.pose_ptr[k + 1] - P.pose_ptr[k] + 31) / 32);
    }
    // the chunks' sums of free pose f, from their warps' in order, and the sum
    // over the chunks: lane l those of chunks l, l + Lanes, ..., then a butterfly
    template <int Lanes>
    __device__ void add_chunks(const double* wsum, int warps, double* sys) const {
        constexpr int kGroups = kPoThreads / Lanes;
        const int l = threadIdx.x % Lanes, g = threadIdx.x / Lanes;
        for (int e0 = 0; e0 < kSys; e0 += kGroups) {  // (uniform: every lane takes part in the butterfly)
            const int e = e0 + g;
            double v = 0.0;
            if (e < kSys) {
                for (int c = l; 8 * c < warps; c += Lanes) {
                    double t = 0.0, x[8];
#pragma unroll
                    for (int w = 0; w < 8; ++w) x[w] = 8 * c + w < warps ? __ldcg(wsum + (8 * c + w) * kRec + e) : 0.0;
#pragma unroll
                    for (int w = 0; w < 8; ++w) t += x[w];
                    v += t;
                }
            }
            v = lanes_add<Lanes>(v);
            if (l == 0 && e < kSys) sys[e] = v;
        }
    }
    __device__ void system(const DevProblem&, int, Sh&) {}
    __device__ double cost(const DevProblem& P, int b, Sh& sh) {
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nf = sh.nfree;
        const int64_t stride = (int64_t)kChunk * chunks;
        double* cpart = scratch + (int64_t)turn * (chunks + (int64_t)kPoseOnlyMaxFree * 8 * chunks * kRec);
        double* wsums = cpart + chunks;
        turn ^= 1;
        // tasks of a CTA: a chunk's cost, or four warps' sums of a free pose
        const int nc = (int)min((int64_t)chunks, (P.M + kChunk - 1) / kChunk);
        int t0 = nc;
        for (int t = blockIdx.x; t < nc; t += gridDim.x) {
            double h[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                h[i] = 0.0;
                for (int64_t o = (int64_t)t * kChunk + tid + i * kPoThreads; o < P.M; o += stride) {
                    const double* pp = sh.pose[b][P.obs_pose[o]];
                    double p[7];
#pragma unroll
                    for (int j = 0; j < 7; ++j) p[j] = pp[j];
                    h[i] += obs_cost(P, p, o);
                }
            }
            __syncthreads();
            sh.red[tid] = h[0] + h[1];
            __syncthreads();
            if (warp == 0) {
                const double v = lanes_add((sh.red[lane] + sh.red[lane + 64]) + (sh.red[lane + 32] + sh.red[lane + 96]));
                if (lane == 0) __stcg(cpart + t, v);
            }
        }
        for (int f = 0; f < nf; ++f) {
            const int k = sh.order[f], warps = warps_of(P, k), nt = (warps + 3) / 4;
            // the first task of this pose that is this CTA's
            const int skip = (int)((blockIdx.x + gridDim.x - t0 % gridDim.x) % gridDim.x);
            for (int t = skip; t < nt; t += gridDim.x) {
                const int w = 4 * t + warp;
                if (w >= warps) break;  // (of this warp; no barrier in this loop)
                double v[32], p[7];
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = 0.0;
#pragma unroll
                for (int i = 0; i < 7; ++i) p[i] = sh.pose[b][k][i];
                const int q1 = P.pose_ptr[k + 1];
                for (int64_t q = P.pose_ptr[k] + 32 * w + lane; q < q1; q += stride) add_terms(P, p, P.pose_obs[q], v);
                const double s = warp_sums(v);
                if (lane < kSys) __stcg(wsums + ((int64_t)f * 8 * chunks + w) * kRec + lane, s);
            }
            t0 += nt;
        }
        // (a CTA writes this pass's scratch again two passes on, when every
        // other one has come to the next pass's barrier)
        grid.sync();
        for (int f = 0; f < nf; ++f) {
            const int warps = warps_of(P, sh.order[f]);
            const double* w = wsums + (int64_t)f * 8 * chunks * kRec;
            if (warps <= 64) add_chunks<8>(w, warps, sh.sys[b][f]);
            else if (warps <= 128) add_chunks<16>(w, warps, sh.sys[b][f]);
            else add_chunks<32>(w, warps, sh.sys[b][f]);
        }
        // every warp adds the chunks' costs the same way
        double c = 0.0;
        for (int i = lane; i < nc; i += 32) c += __ldcg(cpart + i);
        c = lanes_add(c);
        __syncthreads();
        return c;
    }
};
struct WindowTeam {
    static constexpr int kThreadsOf = kPoWinThreads;
    using Sh = Shared<kBatchMaxK, kBatchMaxK, kPoWinThreads>;
    int k0, k1;
    __device__ bool lead() const { return true; }
    __device__ void system(const DevProblem& P, int b, Sh& sh) {
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        for (int f = 0; f < sh.nfree; ++f) {
            const int k = sh.order[f];
            const int q0 = P.pose_ptr[k0 + k], q1 = P.pose_ptr[k0 + k + 1];
            double t = 0.0;
            if (32 * warp < q1 - q0) {  // (else the warp has no observation: zeros)
                double v[32], p[7];
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = 0.0;
#pragma unroll
                for (int i = 0; i < 7; ++i) p[i] = sh.pose[b][k][i];
                for (int q = q0 + tid; q < q1; q += kPoWinThreads) add_terms(P, p, P.pose_obs[q], v);
                t = warp_sums(v);
            }
            if (lane < kSys) sh.wpart[warp][lane] = t;
            __syncthreads();
            if (tid < kSys) {
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < kPoWinThreads / 32; ++w) s += sh.wpart[w][tid];
                sh.sys[b][f][tid] = s;
            }
            __syncthreads();
        }
    }
    __device__ double cost(const DevProblem& P, int b, Sh& sh) {
        const int tid = threadIdx.x, lane = tid & 31;
        double v = 0.0;
        for (int q = P.pose_ptr[k0] + tid; q < P.pose_ptr[k1]; q += kPoWinThreads) {
            const int64_t o = P.pose_obs[q];
            const double* pp = sh.pose[b][P.obs_pose[o] - k0];
            double p[7];
#pragma unroll
            for (int j = 0; j < 7; ++j) p[j] = pp[j];
            v += obs_cost(P, p, o);
        }
        __syncthreads();
        sh.red[tid] = v;
        __syncthreads();
        // every warp the same tree: threads 128 apart, 64, 32, then the lanes
        double h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = sh.red[lane + 32 * i] + sh.red[lane + 32 * i + 128];
        return lanes_add((h[0] + h[2]) + (h[1] + h[3]));
    }
};

// The Levenberg-Marquardt loop of factor_graph::solve
// (source/factor_graph.hpp:506-615) over poses k0 .. k0 + K (every landmark
// fixed). active = false skips the loop (the window reports no iteration).
// hist (may be null): the attempts, up to ctl.hist_cap. Every CTA takes the
// same decisions; the lead CTA writes the poses at the end.
template <typename Team>
__device__ PoseOnlyOut lm_loop(const DevProblem& P, int k0, int K, const PoseOnlyCtl& ctl, bool active, Team& team,
                               typename Team::Sh& sh, zs_ba_attempt* hist) {
    constexpr int NT = Team::kThreadsOf;
    const int t = threadIdx.x, lane = t & 31;
    const bool lead = team.lead();
    for (int i = t; i < K * kPoseStride; i += NT) {
        const double v = P.pose[(int64_t)k0 * kPoseStride + i];
        sh.pose[0][i / kPoseStride][i % kPoseStride] = v;
        sh.pose[1][i / kPoseStride][i % kPoseStride] = v;
    }
    if (t == 0) {
        int n = 0;
        for (int k = 0; k < K; ++k)
            if (!P.pose_fixed[k0 + k]) sh.order[n++] = k;
        sh.nfree = n;
    }
    if (t < 64) sh.gain[t] = 0.0;
    __syncthreads();
    int cur = 0;
    // the initial system, cost and damping (tau min(clamp, max diag H))
    team.system(P, 0, sh);
    const double c0 = team.cost(P, 0, sh);
    unsigned long long m = 0;
    for (int i = lane; i < 6 * sh.nfree; i += 32) m = max(m, abs_bits(sh.sys[0][i / 6][place(i % 6, i % 6)]));
    const double mdiag = warp_max_bits(m);
    if (t == 0) {
        sh.chi2 = c0;
        sh.lambda = ctl.tau * fmin(ctl.clamp, mdiag);
        sh.nu = 2.0;
    }
    __syncthreads();
    int iterations = 0, attempts = 0, accepted = 0, chol_fail = 0, nhist = 0;
    const double legacy = ctl.legacy_stop * c0;
    for (int it = 0; active && it < ctl.iterations; ++it) {
        iterations = it + 1;
        const double last = sh.chi2;
        int failures = 0;
        while (failures < ctl.max_failures) {
            const bool ok = solve_step(K, cur, sh);
            double chi2_new = sh.chi2;
            if (ok) {
                trial_state(cur, sh);
                chi2_new = team.cost(P, cur ^ 1, sh);
            }
            __syncthreads();
            // source/factor_graph.hpp:542-591 (k_decide), in every CTA
            if (t == 0) {
                if (!ok) {
                    sh.lambda *= sh.nu;
                    sh.nu *= 2.0;
                    sh.good = 0;
                } else {
                    const double rho = (sh.chi2 - chi2_new) / sh.scale;
                    sh.rho = rho;
                    if (rho > 0 && isfinite(chi2_new)) {
                        double alpha = 1.0 - pow(2.0 * rho - 1.0, 3.0);
                        alpha = fmin(alpha, 2.0 / 3.0);
                        sh.lambda *= fmax(1.0 / 3.0, alpha);
                        sh.nu = 2.0;
                        sh.chi2 = chi2_new;
                        sh.good = 1;
                    } else {
                        sh.lambda *= sh.nu;
                        sh.nu *= 2.0;
                        sh.good = 0;
                    }
                }
            }
            __syncthreads();
            const bool good = sh.good != 0;
            const double lam = sh.lambda;
            ++attempts;
            if (hist && lead && t == 0 && nhist < ctl.hist_cap) {
                zs_ba_attempt a{};
                a.iteration = it;
                a.attempt = failures;
                a.solved = ok ? 1 : 0;
                a.accepted = ok && good ? 1 : 0;
                a.chi2 = ok ? chi2_new : sh.chi2;
                a.rho = ok ? sh.rho : 0.0;
                a.lambda = lam;
                hist[nhist] = a;
            }
            ++nhist;
            if (!ok) {
                ++chol_fail;
                ++failures;
                if (!isfinite(lam)) break;
                continue;
            }
            // (a rejected step is rolled back while lambda stays finite)
            if (good || !isfinite(lam)) cur ^= 1;
            if (good) {
                ++accepted;
                if (isfinite(lam)) team.system(P, cur, sh);  // the next iteration's, where it did not come with the cost
                break;
            }
            if (!isfinite(lam)) break;
            ++failures;
        }
        const double thr = ctl.use_relative ? ctl.rel_tol * fmax(last, ctl.floor) : legacy;
        if (failures >= ctl.max_failures || (last - sh.chi2) < thr || !isfinite(sh.lambda)) break;
    }
    if (lead)
        for (int i = t; i < K * kPoseStride; i += NT)
            if (!P.pose_fixed[k0 + i / kPoseStride])
                P.pose[(int64_t)k0 * kPoseStride + i] = sh.pose[cur][i / kPoseStride][i % kPoseStride];
    PoseOnlyOut o;
    o.iterations = iterations;
    o.attempts = attempts;
    o.accepted = accepted;
    o.cholesky_failures = chol_fail;
    o.history = nhist;
    o.chi2_initial = c0;
    o.chi2_final = sh.chi2;
    o.lambda_final = sh.lambda;
    return o;
}

__global__ void __launch_bounds__(kPoThreads) k_pose_only_lm(DevProblem P, PoseOnlyCtl ctl, PoseOnlyOut* out,
                                                             zs_ba_attempt* hist, double* scratch, int chunks) {
    __shared__ GridTeam::Sh sh;
    GridTeam team{cg::this_grid(), scratch, chunks, 0};
    const PoseOnlyOut o = lm_loop(P, 0, P.K, ctl, true, team, sh, hist);
    if (blockIdx.x == 0 && threadIdx.x == 0) *out = o;
}

// A batch of windows whose landmarks are all fixed (tracking problems solved
// together): one CTA per window runs the loop above on the window's poses,
// each window with its own damping, decisions and stops, as the general
// batched path (ba_batch.cu) runs them, and reports into the batch's
// per-window control and state. A window without observations, or with
// neither poses nor landmarks, runs no iteration (k_binit's rule).
__global__ void __launch_bounds__(kPoWinThreads) k_pose_only_windows(DevProblem P, PoseOnlyCtl ctl, WinCtl* wctl,
                                                                  LmState* wst) {
    __shared__ WindowTeam::Sh sh;
    const int w = blockIdx.x;
    const int k0 = P.win_pose0[w], k1 = P.win_pose0[w + 1];
    WindowTeam team{k0, k1};
    const bool has_obs = P.pose_ptr[k1] > P.pose_ptr[k0];
    const bool active = ctl.iterations > 0 && ctl.max_failures > 0 && has_obs &&
                        (k1 > k0 || P.win_lm0[w + 1] > P.win_lm0[w]);
    const PoseOnlyOut o = lm_loop(P, k0, k1 - k0, ctl, active, team, sh, nullptr);
    if (threadIdx.x == 0) {
        WinCtl c{};
        c.iterations = o.iterations;
        c.it = o.iterations;
        c.accepted = o.accepted;
        c.attempts = o.attempts;
        c.chol_failures = o.cholesky_failures;
        c.last = o.chi2_final;
        c.legacy = ctl.legacy_stop * o.chi2_initial;
        c.chi2_initial = o.chi2_initial;
        wctl[w] = c;
        LmState st{};
        st.chi2 = o.chi2_final;
        st.chi2_new = o.chi2_final;
        st.lambda = o.lambda_final;
        st.solve_ok = 1;
        wst[w] = st;
    }
}

}  // namespace

// CTAs that are surely resident together: at most one per SM.
static int pose_only_resident() {
    static std::atomic<int> cache[kMaxDevices];
    return per_device(cache, [] {
        int dev = 0, sms = 0, per = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pose_only_lm, kPoThreads, 0);
        cudaGetLastError();
        return std::max(1, std::min(sms, sms * per));
    });
}

// About 64 observations a chunk, at most a chunk per SM.
static int pose_only_chunks(int64_t M) {
    return (int)std::max<int64_t>(1, std::min<int64_t>(pose_only_resident(), (M + 63) / 64));
}

size_t pose_only_scratch(int64_t M) {
    return 2 * (size_t)pose_only_chunks(M) * (1 + (size_t)kPoseOnlyMaxFree * 8 * kRec);
}

cudaError_t launch_pose_only_windows(const DevProblem& P, const PoseOnlyCtl& ctl, WinCtl* wctl, LmState* wst,
                                    cudaStream_t s) {
    if (P.nwin < 1) return cudaSuccess;
    k_pose_only_windows<<<P.nwin, kPoWinThreads, 0, s>>>(P, ctl, wctl, wst);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_pose_only_lm(const DevProblem& P, const PoseOnlyCtl& ctl, PoseOnlyOut* out, zs_ba_attempt* hist,
                                double* scratch, cudaStream_t s) {
    if (P.K > kPoseOnlyMaxK) return cudaErrorInvalidValue;
    int chunks = pose_only_chunks(P.M);
    // a CTA per task of a pass (chunks' costs, four warps' sums), at most one per SM
    const int64_t tasks = (P.M + kChunk - 1) / kChunk + P.M / kPoThreads + kPoseOnlyMaxFree;
    const int grid = (int)std::min<int64_t>(pose_only_resident(), tasks);
    DevProblem Pv = P;
    PoseOnlyCtl c = ctl;
    void* args[] = {(void*)&Pv, (void*)&c, (void*)&out, (void*)&hist, (void*)&scratch, (void*)&chunks};
    cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_pose_only_lm, dim3(grid), dim3(kPoThreads), args, 0, s);
    if (e == cudaSuccess) note_launch();
    return e;
}

}  // namespace zs

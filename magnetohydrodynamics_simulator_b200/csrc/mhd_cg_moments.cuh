// The implicit solve with a fixed number of passes over the data: conjugate gradients whose scalars
// come from moments (reference: solvers.hpp:404-489 with Eigen's ConjugateGradient defaults, the
// same iterates and the same stopping rule as k_cg_sweep).
//
// With t = 2 (cx + cy) the matrix is A = I + t D, where D = I - (weighted mean of the four
// neighbours) is positive semidefinite with spectrum in [0, 2]. CG started at x0 = 0 with a constant
// Jacobi diagonal only ever builds polynomials of D applied to the right-hand side b, and all of its
// scalars are functions of the moments mu_l = b . D^l b: the residual of iterate k is
// pi_k(D) b / pi_k(-1/t), pi_k being the monic orthogonal polynomials of those moments. So
//   pass 1  forms w_l = D^l b, l <= M, in registers while the rows stream by, and sums
//           w_l . w_{l-1} and w_l . w_l: mu_0 .. mu_2M with full relative accuracy (every sum has
//           terms of one sign up to rounding; smooth right-hand sides need that);
//   plan    one warp runs the Chebyshev algorithm (moments -> recurrence coefficients and norms of
//           pi_k): |r_k|^2 = norm_k / pi_k(-1/t)^2 for k <= M, the first k below the threshold, and
//           the coefficients of x_k = q_{k-1}(D) b, (1 + t z) q_{k-1}(z) = 1 - pi_k(z) / pi_k(-1/t);
//   pass 2  evaluates x_k = q_{k-1}(D) b as it streams the rows once more.
// Each pass reads the two face planes (16 bytes a zone) and pass 2 writes x (8 bytes): 40 bytes a
// solve, whatever k is, where one CG iteration moves 32-48.
//
// The Chebyshev algorithm loses about a factor 30 of accuracy per step, so every norm carries a
// running error bound (the sums' relative error is far below kCmNoise), and only norms well above
// it are used. If the residual has not passed the threshold at the last usable k, the ordinary
// iterations go on from there: r, p and x of an earlier iterate are evaluated from their polynomials
// (three more passes) and the sweeps of mhd_cg_sweep.cuh go on, in k_solve or in the k_cg_sweep launched
// behind it. With no usable norm, beyond kCmMaxT, or in front of a k_cg_band, which takes up no iterate (it
// gains nothing by the passes then: beyond kCmSureT), they start from the right-hand side.
//
// Bound by instruction issue at two warps a scheduler (FP64 pipe 40%, DRAM 30%), not by DRAM. Measured on
// B200, one solve: 4096^2, eta 1e-4 (6 products) 792 -> 308 us; 2048^2, eta 1e-3 (9 products) 360 -> 172 us;
// 512^2 (7 products) 64 -> 60 us. Tried: levels skewed by a row, so that a row's levels do not wait for one
// another (three rows of each level kept): 96 us instead of 109 for five levels, but seven spill.
#pragma once

#include "mhd_cg_sweep.cuh"

namespace mhd {

constexpr int CM_NT = 256;  // threads per block: 8 warps of up to 255 registers, one block a SM
constexpr int CM_NW = CM_NT / 32;
constexpr int CM_RING = 8;  // prefetched rows per warp (power of two)
constexpr int CM_MAXM = 9;  // levels of the longest pass 1
constexpr int CM_NMU = 2 * CM_MAXM + 1;
// A pass works on C adjacent columns per lane: 3 (odd: conflict-free shared-memory reads), or 1 where the grid
// has too few rows to keep the warps busy -- a row then takes a third of the instructions, which is what a
// lone warp waits for, for twice the halo. Halo lanes on each side of a pass of M levels (M columns, whole
// lanes) and output columns per warp. Measured at 4096^2, M = 7, C = 3: 137 us; two columns on 12 warps of
// 168 registers 156 us, on 16 warps of 128 registers the levels spill.
constexpr int CM_C = 3;
__host__ __device__ constexpr int cm_halo_lanes(int M, int C) { return (M + C - 1) / C; }
__host__ __device__ constexpr int cm_out(int M, int C) { return (32 - 2 * cm_halo_lanes(M, C)) * C; }
// Doubles of a ring slot (bx row, by row, by left of the first column) and of a warp's shared memory: ring,
// then the staging of an output row.
__host__ __device__ constexpr int cm_slot(int C) { return 2 * 32 * C + 2; }
constexpr int CM_WARP = CM_RING * cm_slot(CM_C) + 32 * CM_C;
constexpr size_t kCmSmemBytes = (size_t)CM_NW * CM_WARP * sizeof(double);
static_assert(CG_RING * CG_SLOT <= CM_WARP, "the sweeps' rings fit the passes' shared memory");
constexpr double kCmNoise = 5.7e-14;  // relative error allowed to the moment sums (256 eps)
constexpr double kCmTrust = 8.0;      // a norm counts when it exceeds its error bound this many times
constexpr double kCmMaxT = 0.06;      // largest t = 2 (cx + cy) of the moment form
constexpr double kCmSureT = 0.033;    // beyond it CM_MAXM levels may not suffice (cm_levels)

// Levels of pass 1. The a-priori CG bound, 2 sqrt(kappa) zeta^k with zeta = (sqrt(kappa) - 1) / (sqrt(kappa)
// + 1) and kappa = 1 + 2 t, reaches machine precision by k = 5 up to t = 1.2e-3, by k = 7 up to t = 0.0105 and by
// k = 9 up to 0.034; flows need one product less (7 at t = 0.0155, 9 at 0.053), noise does not. Where the levels do
// not suffice the ordinary iterations finish. (9 levels from 0.0105 on: a CFL step of a flow at 512^2 takes 159 us for
// 144, one of a noisy field 168 for 246.)
__host__ __device__ inline int cm_levels(double t) { return t < 1.2e-3 ? 5 : (t < 0.0155 ? 7 : CM_MAXM); }
// Whether they suffice for any right-hand side.
__host__ __device__ inline bool cm_sure(double t) { return t < 0.0105 || (t >= 0.0155 && t <= kCmSureT); }

struct CmSpan {
    int strips, seg_h, n;  // column strips, rows per segment, segments in all
};
// Split of the grid over `warps` warps: strips of `out` columns, row segments of equal height (at least 4
// rows: a segment repeats 2 M halo rows).
__device__ __forceinline__ CmSpan cm_span(int nx, int ny, int out, int warps) {
    CmSpan s;
    s.strips = (nx + out - 1) / out;
    const int segs = max(1, warps / s.strips);
    s.seg_h = max(4, (ny + segs - 1) / segs);
    s.n = s.strips * ((ny + s.seg_h - 1) / s.seg_h);
    return s;
}
// Whether a pass of M levels is shorter with one column a lane: the rows of a warp's segment, weighed by what
// a row takes a warp that has its scheduler nearly to itself (1700 cycles with three columns, 600 with one).
__device__ __forceinline__ bool cm_narrow(int nx, int ny, int M, int warps) {
    const CmSpan w = cm_span(nx, ny, cm_out(M, CM_C), warps), n = cm_span(nx, ny, cm_out(M, 1), warps);
    const int rounds = (n.n + warps - 1) / warps;  // (a strip for every warp and more: very wide grids)
    return rounds * (n.seg_h + 2 * M) * 6 < (w.seg_h + 2 * M) * 17;
}

struct CmGeom {
    int nx, ny;
    double ratio;          // dx / dy: the passes work on b / scale = (by - by_left) - ratio (bx - bx_below),
                           // with scale = eta / dx
    double ax, ay;         // weights of D: D w = w - ax (left + right) - ay (below + above)
    const double* bxf;
    const double* byf;
};

// This warp's shared memory. The functions that are not inlined ask for it themselves: a pointer argument
// would be a generic address, and every access through it one of the slower generic loads and stores.
__device__ __forceinline__ double* cm_warp_smem() {
#if defined(__CUDA_ARCH__)
    extern __shared__ __align__(16) double cm_mem[];
#else
    static double cm_mem[kCmSmemBytes / sizeof(double)];
#endif
    return cm_mem + (size_t)(threadIdx.x >> 5) * CM_WARP;
}

// A warp's stream of right-hand-side rows: cp.async into the ring, coalesced; each lane then reads
// its C adjacent columns. Sweep row k holds grid row j0 + k (k = -1: only bx, the row below the
// first). The caller runs next() once per row, in order.
template <int C>
struct CmRows {
    const CmGeom& g;
    double* ring;
    int lane, j0, last;  // grid row of sweep row 0, last sweep row
    int col[C], coll;    // wrapped columns this lane copies; the one left of the strip

    __device__ __forceinline__ CmRows(const CmGeom& g_, double* ring_, int c0, int j0_, int rows)
        : g(g_), ring(ring_), lane(threadIdx.x & 31), j0(j0_), last(rows - 1) {
#pragma unroll
        for (int q = 0; q < C; ++q) col[q] = wrap(c0 + lane + 32 * q, g.nx);
        coll = wrap(c0 - 1, g.nx);
#pragma unroll
        for (int k = -1; k < CM_RING - 2; ++k) issue(k);
    }
    __device__ __forceinline__ double* slot(int k) const { return ring + ((k + 1) & (CM_RING - 1)) * cm_slot(C); }
    __device__ __forceinline__ void issue(int k) const {
        if (k <= last) {
            const size_t rp = (size_t)wrap(j0 + k, g.ny) * g.nx;
            double* s = slot(k);
            const double* px = g.bxf + rp;
            const double* py = g.byf + rp;
#pragma unroll
            for (int q = 0; q < C; ++q) {
                cp_async8(&s[lane + 32 * q], &px[col[q]]);
                cp_async8(&s[(32 * C) + lane + 32 * q], &py[col[q]]);
            }
            if (lane == 0) cp_async8(&s[2 * (32 * C)], &py[coll]);
        }
        cp_async_commit();
    }
    // b / scale of sweep row k at the lane's columns
    __device__ __forceinline__ void next(int k, double (&b)[C]) {
        cp_async_wait<CM_RING - 3>();  // row k has landed (row k + 1 may be in flight)
        __syncwarp();                  // ... for every lane, and every lane is done with row k - 1's slot
        const double* s = slot(k) + lane * C;
        const double* sb = slot(k - 1) + lane * C;  // the row below, still in its slot
        double by[C];
#pragma unroll
        for (int c = 0; c < C; ++c) by[c] = s[(32 * C) + c];
        double byl = __shfl_up_sync(0xffffffffu, by[C - 1], 1);
        if (lane == 0) byl = s[2 * (32 * C)];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            b[c] = fma(g.ratio, sb[c] - s[c], by[c] - (c ? by[c - 1] : byl));
        }
        issue(k + CM_RING - 2);  // into row k - 2's slot
    }
};

// D at one row: out = ctr - ax (left + right) - ay (below + above).
template <int C>
__device__ __forceinline__ void cm_apply(const CmGeom& g, const double (&below)[C], const double (&ctr)[C],
                                         const double (&above)[C], double (&out)[C]) {
    const double l = __shfl_up_sync(0xffffffffu, ctr[C - 1], 1);
    const double r = __shfl_down_sync(0xffffffffu, ctr[0], 1);
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const double lr = (c ? ctr[c - 1] : l) + (c < C - 1 ? ctr[c + 1] : r);
        out[c] = fma(-g.ay, below[c] + above[c], fma(-g.ax, lr, ctr[c]));
    }
}

// A double with its high word cleared where the mask is 0: below 2e-314, nothing in any sum. One
// integer instruction where a select takes two.
__device__ __forceinline__ double cm_mask(double v, int m) {
#if defined(__CUDA_ARCH__)
    return __hiloint2double(__double2hiint(v) & m, __double2loint(v));
#else
    return m ? v : 0.0;
#endif
}

template <bool V>
struct CmTag {
    static constexpr bool value = V;
};

// Pass 1 over rows [r0, r1) of strip sx: acc[2l] += w_l . w_l, acc[2l - 1] += w_l . w_{l-1}. FULL: every
// column of the strip's output lanes counts (halo lanes' sums are dropped by the caller); else columns are
// masked one by one.
template <int M, int C, bool FULL>
__device__ __forceinline__ void cm_moments_segment(const CmGeom& g, int sx, int r0, int r1, double* smem,
                                                   double (&acc)[2 * M + 1]) {
    constexpr int LH = cm_halo_lanes(M, C);
    const int lane = threadIdx.x & 31;
    const int c0 = sx * cm_out(M, C) - LH * C;
    const int h = r1 - r0;
    int own[C];  // all ones where the lane's column counts
#pragma unroll
    for (int c = 0; c < C; ++c)
        own[c] = FULL || (lane >= LH && lane < 32 - LH && c0 + lane * C + c < g.nx) ? -1 : 0;
    const int rows = h + 2 * M;
    CmRows<C> in(g, smem, c0, r0 - M, rows);
    // the two latest rows of w_0 .. w_{M-1}: S[k & 1] holds row k's, written over row k - 2's
    double S[2][M][C];
#pragma unroll
    for (int l = 0; l < M; ++l)
#pragma unroll
        for (int c = 0; c < C; ++c) S[0][l][c] = S[1][l][c] = 0.0;
    // A: row k - 2 of each level (overwritten with the new one), B: row k - 1. Level l of sweep row k is
    // row k - l - M of the segment; EDGE: some of them may lie outside it. Masks instead of branches keep
    // a row one basic block, in which the levels' instructions interleave.
    auto row = [&](int k, double (&A)[M][C], const double (&B)[M][C], auto edge) {
        constexpr bool kEdge = decltype(edge)::value;
        auto counted = [&](double v, int l, int c) {
            int m = own[c];
            if constexpr (kEdge) m = (unsigned)(k - l - M) < (unsigned)h ? m : 0;
            return kEdge || !FULL ? cm_mask(v, m) : v;
        };
        double cur[C];
        in.next(k, cur);
#pragma unroll
        for (int c = 0; c < C; ++c) acc[0] = fma(counted(cur[c], 0, c), cur[c], acc[0]);
#pragma unroll
        for (int l = 0; l < M; ++l) {
            double nw[C];
            cm_apply<C>(g, A[l], B[l], cur, nw);  // w_{l+1} of sweep row k - l - 1
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const double v = counted(nw[c], l + 1, c);
                acc[2 * l + 1] = fma(v, B[l][c], acc[2 * l + 1]);
                acc[2 * l + 2] = fma(v, nw[c], acc[2 * l + 2]);
                A[l][c] = cur[c];
                cur[c] = nw[c];
            }
        }
    };
    int k = 0;
    for (; k < 2 * M; k += 2) {
        row(k, S[0], S[1], CmTag<true>{});
        row(k + 1, S[1], S[0], CmTag<true>{});
    }
    for (; k + 1 < h + M; k += 2) {
        row(k, S[0], S[1], CmTag<false>{});
        row(k + 1, S[1], S[0], CmTag<false>{});
    }
    for (; k < rows; k += 2) {  // (the last row may lie one past the sweep: nothing of it counts)
        row(k, S[0], S[1], CmTag<true>{});
        row(k + 1, S[1], S[0], CmTag<true>{});
    }
    cp_async_wait<0>();
    __syncwarp();
}

// out = q(D) b over rows [r0, r1) of strip sx, q of degree DEG with coefficients q[0 .. DEG] (shared
// memory): a row's partial sum goes down the levels with it.
template <int DEG, int C>
__device__ __forceinline__ void cm_poly_segment(const CmGeom& g, int sx, int r0, int r1, double* smem,
                                                const double* q, double* __restrict__ out) {
    constexpr int LH = cm_halo_lanes(DEG, C);
    const int lane = threadIdx.x & 31;
    const int c0 = sx * cm_out(DEG, C) - LH * C;
    const int h = r1 - r0;
    const int rows = h + 2 * DEG;
    double* const stage = smem + CM_RING * cm_slot(C);
    CmRows<C> in(g, smem, c0, r0 - DEG, rows);
    double S[2][DEG][C], X[DEG][C];  // X[l]: the sum up to level l of sweep row k - 1 - l
#pragma unroll
    for (int l = 0; l < DEG; ++l)
#pragma unroll
        for (int c = 0; c < C; ++c) S[0][l][c] = S[1][l][c] = X[l][c] = 0.0;
    auto row = [&](int k, double (&A)[DEG][C], const double (&B)[DEG][C]) {
        double cur[C], sum[C];
        in.next(k, cur);
#pragma unroll
        for (int c = 0; c < C; ++c) sum[c] = q[0] * cur[c];
#pragma unroll
        for (int l = 0; l < DEG; ++l) {
            double nw[C];
            cm_apply<C>(g, A[l], B[l], cur, nw);
            const double ql = q[l + 1];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const double x = X[l][c];
                X[l][c] = sum[c];
                sum[c] = fma(ql, nw[c], x);
                A[l][c] = cur[c];
                cur[c] = nw[c];
            }
        }
        const int ro = k - 2 * DEG;  // the finished row, r0 + ro
        if ((unsigned)ro < (unsigned)h) {
            double* const po = out + (size_t)(r0 + ro) * g.nx;
            // through shared memory, so that the row is written in full sectors
#pragma unroll
            for (int c = 0; c < C; ++c) stage[lane * C + c] = sum[c];
            __syncwarp();
#pragma unroll
            for (int e = 0; e < C; ++e) {
                const int m = lane + 32 * e, i = c0 + m;
                if (m >= LH * C && m < 32 * C - LH * C && i < g.nx) po[i] = stage[m];
            }
        }
    };
    for (int k = 0; k < rows; k += 2) {
        row(k, S[0], S[1]);
        row(k + 1, S[1], S[0]);  // (may lie one past the sweep: nothing of it is written)
    }
    cp_async_wait<0>();
    __syncwarp();
}

// What the moments say about the solve; identical in every block.
enum CmMode : int { kCmZero = 0, kCmBreakdown, kCmDone, kCmCapped, kCmContinue, kCmScratch };
struct CmPlan {
    int mode;
    int k;             // kCmDone / kCmCapped: products; kCmContinue: the iteration to go on with (odd)
    double bb, rr;     // |b|^2; |r_k|^2
    double q[CM_MAXM + 2];  // polynomial of x
    double qr[CM_MAXM + 2], qp[CM_MAXM + 2];  // kCmContinue: polynomials of r_k and p_{k-1}
    double alpha, alpha_prev, beta, absNew, pAp, threshold;
};

// The plan, by one warp: lane l holds mu_l (l <= 2 M; 0 in the other lanes). Two runs of the Chebyshev
// algorithm over the same numbers: the first finds the residuals and the polynomial of x; the second,
// only when the residual has not passed the threshold, follows CG's own polynomials to the last odd
// iteration that the norms resolve.
// The polynomials come out times `scale`: the passes evaluate them on b / scale (mu is b's own).
__device__ __forceinline__ void cm_plan(double mu, int M, double t, double diag, double scale, double tol,
                                        long long max_iters, CmPlan* P) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const double bb = __shfl_sync(kAll, mu, 0);
    const double threshold = smax(tol * tol * bb, 2.2250738585072014e-308);
    if (lane == 0) {
        P->bb = bb;
        P->threshold = threshold;
        P->rr = 0.0;
        P->k = 0;
    }
    int mode = kCmScratch;
    if (!isfinite(bb)) mode = kCmBreakdown;
    else if (bb == 0.0 || bb < threshold) mode = kCmZero;
    if (mode != kCmScratch) {
        if (lane == 0) P->mode = mode;
        return;
    }
    const double zs = -1.0 / t;  // the matrix's zero in D
    const double a0 = __shfl_sync(kAll, mu, 1) / bb;
    // One step of the algorithm, from pi_{k-1} (recurrence coefficients a, b) to pi_k.
    struct State {
        double sp, sc, ep, ec;  // <pi_{k-2}, z^l>, <pi_{k-1}, z^l> and their error bounds, l = lane
        double vp, vc;          // pi_{k-2}(zs), pi_{k-1}(zs)
        double cp, cc;          // coefficients of pi_{k-2}, pi_{k-1}
        double a, b;
        double norm, inorm;     // <pi_{k-1}, pi_{k-1}> and its reciprocal
        double ratio;           // <pi_{k-1}, z^k> / norm
        double vn, cn, err, nn; // pi_k(zs), pi_k's coefficients, error bound and value of its norm
        double sn, en;
    };
    auto begin = [&]() {
        State S{};
        S.sc = mu;
        S.ec = fabs(mu) * kCmNoise;
        S.vc = 1.0;
        S.cc = lane == 0 ? 1.0 : 0.0;
        S.a = a0;
        S.norm = bb;
        S.inorm = 1.0 / bb;
        S.ratio = a0;
        return S;
    };
    auto form = [&](State& S, int k) {  // pi_k and its norm; false when the norm is not resolved
        const double s1 = __shfl_down_sync(kAll, S.sc, 1), e1 = __shfl_down_sync(kAll, S.ec, 1);
        const double up = __shfl_up_sync(kAll, S.cc, 1);
        S.sn = s1 - S.a * S.sc - S.b * S.sp;
        S.en = e1 + fabs(S.a) * S.ec + fabs(S.b) * S.ep;
        S.nn = __shfl_sync(kAll, S.sn, k);
        S.err = __shfl_sync(kAll, S.en, k);
        S.vn = (zs - S.a) * S.vc - S.b * S.vp;
        S.cn = (lane ? up : 0.0) - S.a * S.cc - S.b * S.cp;
        return S.nn > kCmTrust * S.err && S.nn > 0.0 && isfinite(S.nn) && isfinite(S.vn * S.vn);
    };
    auto advance = [&](State& S, int k) {
        const double in = 1.0 / S.nn;
        const double ratio = __shfl_sync(kAll, S.sn, (k + 1) & 31) * in;
        S.a = ratio - S.ratio;
        S.b = S.nn * S.inorm;
        S.ratio = ratio;
        S.norm = S.nn;
        S.inorm = in;
        S.sp = S.sc;
        S.sc = S.sn;
        S.ep = S.ec;
        S.ec = S.en;
        S.vp = S.vc;
        S.vc = S.vn;
        S.cp = S.cc;
        S.cc = S.cn;
    };
    State S = begin();
    int usable = 0;  // norms of pi_1 .. pi_usable are resolved
    for (int k = 1; k <= M; ++k) {
        if (!form(S, k)) break;
        usable = k;
        const double v2 = S.vn * S.vn;
        const bool passed = S.nn < threshold * v2;  // |r_k|^2 = nn / v2
        if (passed || k == max_iters) {
            // x_k: (1 + t z) q(z) = 1 - pi_k(z) / pi_k(zs)
            const double e = (lane == 0 ? 1.0 : 0.0) - S.cn / S.vn;
            double ql = 0.0, prev = 0.0;
            for (int l = 0; l < k; ++l) {
                prev = __shfl_sync(kAll, e, l) - t * prev;
                if (lane == l) ql = prev;
            }
            if (lane < CM_MAXM + 2) P->q[lane] = scale * ql;
            if (lane == 0) {
                P->mode = passed ? kCmDone : kCmCapped;
                P->k = k;
                P->rr = S.nn / v2;
            }
            return;
        }
        advance(S, k);
    }
    // iteration kc (odd) is the last whose alpha the norms give: that takes pi_{kc+1}
    const int kc = usable >= 2 ? ((usable - 1) & 1 ? usable - 1 : usable - 2) : 0;
    if (kc == 0) {
        if (lane == 0) P->mode = kCmScratch;
        return;
    }
    S = begin();
    double rr = bb, alpha_p = 0.0, beta = 0.0;
    double pk = S.cc / diag, pk_p = 0.0;  // p_{k-1}, p_{k-2}: p_0 = r_0 / d
    double x = 0.0, x_p = 0.0;            // x_{k-1}, x_{k-2}
    for (int k = 1; k <= kc + 1; ++k) {
        form(S, k);
        const double alpha = -diag * S.vc / (t * S.vn);  // alpha_{k-1}, from the leading coefficients
        if (k == kc + 1) {
            if (lane < CM_MAXM + 2) {
                P->q[lane] = scale * x_p;               // x_{kc-1}
                P->qr[lane] = scale * (S.cc / S.vc);    // r_kc
                P->qp[lane] = scale * pk_p;             // p_{kc-1}
            }
            if (lane == 0) {
                P->mode = kCmContinue;
                P->k = kc;
                P->alpha = alpha;
                P->alpha_prev = alpha_p;
                P->beta = beta;
                P->absNew = rr / diag;
                P->pAp = (rr / diag) / alpha;
            }
            return;
        }
        const double rr_k = S.nn / (S.vn * S.vn);
        beta = rr_k / rr;
        rr = rr_k;
        x_p = x;
        x = fma(alpha, pk, x);
        pk_p = pk;
        pk = S.cn / (S.vn * diag) + beta * pk;
        alpha_p = alpha;
        advance(S, k);
    }
}

// Publish the block's sums of NV moments as partials[v * gridDim + block].
template <int NV>
__device__ __forceinline__ void cm_publish(double (&acc)[NV], double* partials, double (*red)[CM_NMU]) {
#pragma unroll
    for (int v = 0; v < NV; ++v)
        for (int o = 16; o > 0; o >>= 1) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], o);
    const int wi = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) red[wi][v] = acc[v];
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double s = 0.0;
        for (int w = 0; w < CM_NW; ++w) s += red[w][threadIdx.x];
        partials[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = s;
    }
}

// The passes and sweeps are functions of their own, not inlined: each gets its registers without the
// others' values alive around it.
template <int M, int C>
static __device__ __noinline__ void cm_pass1(CmGeom g, int wfirst, int warps, double* partials,
                                             double (*red)[CM_NMU]) {
    constexpr int LH = cm_halo_lanes(M, C), OUT = cm_out(M, C);
    double* const smem = cm_warp_smem();
    const CmSpan sp = cm_span(g.nx, g.ny, OUT, warps);
    double acc[2 * M + 1];
#pragma unroll
    for (int v = 0; v < 2 * M + 1; ++v) acc[v] = 0.0;
    for (int w = wfirst; w < sp.n; w += warps) {
        const int sx = w % sp.strips, r0 = (w / sp.strips) * sp.seg_h, r1 = min(r0 + sp.seg_h, g.ny);
        if ((sx + 1) * OUT <= g.nx) cm_moments_segment<M, C, true>(g, sx, r0, r1, smem, acc);
        else cm_moments_segment<M, C, false>(g, sx, r0, r1, smem, acc);
    }
    const int lane = threadIdx.x & 31;
    if (lane < LH || lane >= 32 - LH) {
#pragma unroll
        for (int v = 0; v < 2 * M + 1; ++v) acc[v] = 0.0;
    }
    cm_publish<2 * M + 1>(acc, partials, red);
}
template <int M>
__device__ __forceinline__ void cm_pass1_any(const CmGeom& g, int wfirst, int warps, double* partials,
                                             double (*red)[CM_NMU]) {
    if (cm_narrow(g.nx, g.ny, M, warps)) cm_pass1<M, 1>(g, wfirst, warps, partials, red);
    else cm_pass1<M, CM_C>(g, wfirst, warps, partials, red);
}

template <int DEG, int C>
static __device__ __noinline__ void cm_pass2(CmGeom g, int wfirst, int warps, const double* q,
                                             double* out) {
    double* const smem = cm_warp_smem();
    const CmSpan sp = cm_span(g.nx, g.ny, cm_out(DEG, C), warps);
    for (int w = wfirst; w < sp.n; w += warps) {
        const int r0 = (w / sp.strips) * sp.seg_h;
        cm_poly_segment<DEG, C>(g, w % sp.strips, r0, min(r0 + sp.seg_h, g.ny), smem, q, out);
    }
}

// out = q(D) b over the whole grid, for a polynomial of degree deg <= CM_MAXM - 1.
__device__ __forceinline__ void cm_pass2_any(const CmGeom& g, int deg, int wfirst, int warps,
                                             const double* q, double* out) {
    if (cm_narrow(g.nx, g.ny, deg, warps)) {
        if (deg <= 4) cm_pass2<4, 1>(g, wfirst, warps, q, out);
        else if (deg <= 6) cm_pass2<6, 1>(g, wfirst, warps, q, out);
        else cm_pass2<CM_MAXM - 1, 1>(g, wfirst, warps, q, out);
    } else if (deg <= 3) cm_pass2<3, CM_C>(g, wfirst, warps, q, out);
    else if (deg <= 4) cm_pass2<4, CM_C>(g, wfirst, warps, q, out);
    else if (deg <= 5) cm_pass2<5, CM_C>(g, wfirst, warps, q, out);
    else if (deg <= 6) cm_pass2<6, CM_C>(g, wfirst, warps, q, out);
    else if (deg <= 7) cm_pass2<7, CM_C>(g, wfirst, warps, q, out);
    else cm_pass2<CM_MAXM - 1, CM_C>(g, wfirst, warps, q, out);
}

}  // namespace mhd

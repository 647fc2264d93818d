// The batch's implicit solves in the single context's forms (mhd_cg_moments.cuh, mhd_cg_cluster.cuh):
//   k_cluster_batch  one cluster per instance that fits one: every instance converges on its own;
//   k_solve_batch    the moment form for all other instances of a chunk in one persistent kernel: pass 1 over
//                    tiles of every instance, one plan per instance, pass 2 over tiles. What it cannot settle
//                    (t beyond kCmMaxT, more products than the moments resolve) it leaves to k_cg_batch by
//                    setting the instance's todo flag.
// k_cg_batch's phases run in lockstep, one per product, each with a grid barrier and 32-48 bytes a zone; here
// there are two passes and two barriers whatever the products.
#pragma once

#include "mhd_batch.cuh"
#include "mhd_cg_cluster.cuh"
#include "mhd_cg_moments.cuh"

namespace mhd {

// A solve's outcome in its instance's status and record (one thread).
__device__ __forceinline__ void batch_report(const BatchInst& I, int inst, int solve, int rec_stride, long long* prods_rec,
                                             const CgResult& r) {
    I.st->cg_products[solve] = r.products;
    I.st->cg_products_sum[solve] += r.products;
    I.st->cg_last_rr[solve] = (r.bb > 0.0) ? r.rr / r.bb : 0.0;
    if (prods_rec) prods_rec[((size_t)inst * rec_stride + I.C->cur) * 2 + solve] = r.products;
    if (r.breakdown) atomicOr(&I.st->flags, (unsigned)(kStatusCgBreakdown | kStatusNonFinite));
    else if (!r.converged) atomicOr(&I.st->flags, (unsigned)kStatusCgNotConverged);
}

// Cluster c solves instance list[c]. Dynamic shared memory: that of the largest.
static __global__ void __launch_bounds__(CC_NT, 1)
k_cluster_batch(const BatchInst* __restrict__ insts, const int* __restrict__ list, int cluster_blocks, int solve,
                int rec_stride, long long* prods_rec, double timeout_s) {
    __shared__ CcTable tab;
#if defined(__CUDA_ARCH__)
    extern __shared__ __align__(16) double cc_mem[];
#else
    static double cc_mem[CC_SMEM_DOUBLES];
#endif
    const int inst = list[blockIdx.x / cluster_blocks];
    const BatchInst& I = insts[inst];
    const unsigned long long deadline = global_timer_ns() + (unsigned long long)(timeout_s * 1e9);
    CgResult res{};
    const bool ok = cc_solve_any(I.D, cluster_blocks, I.C->alpha, solve == 0 ? I.T[4] : I.A[4], solve == 0 ? I.T[5] : I.A[5],
                                 I.x, I.tol, I.max_iters, deadline, cc_mem, &tab, res);
    if (blockIdx.x % cluster_blocks == 0 && threadIdx.x == 0) {
        if (ok) batch_report(I, inst, solve, rec_stride, prods_rec, res);
        else atomicOr(&I.st->flags, (unsigned)kStatusTimeout);
    }
    cooperative_groups::this_cluster().sync();  // no block leaves while another may write into its shared memory
}

// ------------------------------------------------------------------------------------------

struct BatchPlan {
    int mode, k;
    double q[CM_MAXM];  // the solution's polynomial, degree k - 1
};

struct SolveBatchArgs {
    const BatchInst* insts;  // descriptors of this step's parity
    const int* list;         // instances of this launch
    int n;                   // <= CGB_MAX_INST
    int solve;
    double* partials;        // [tiles][CM_NMU], at least kCmTileMinRows rows a tile
    BatchPlan* plans;        // [CGB_MAX_INST]
    int* todo;               // [count]: set for the instances left to k_cg_batch
    CgSync* sync;
    int rec_stride;
    long long* prods_rec;
    double timeout_s;
};

constexpr int kCmTileMinRows = 8;
constexpr int kCmNHeights = 16;
__device__ __constant__ const int kCmHeights[kCmNHeights] = {8, 10, 12, 16, 20, 24, 32, 40, 48, 64, 80, 96, 128, 160, 192, 256};

struct CmBInst {
    int nx, ny, M;    // M: levels of pass 1; 0: not in the moment form
    int strips;       // of the current pass
    double t, diag, scale;
};

__device__ __forceinline__ CmGeom batch_geom(const BatchInst& I, int solve, double t) {
    CmGeom g;
    const double alpha = I.C->alpha;
    g.nx = I.D.nx;
    g.ny = I.D.ny;
    g.ratio = I.D.dx / I.D.dy;
    g.ax = alpha / (I.D.dx * I.D.dx) / t;
    g.ay = alpha / (I.D.dy * I.D.dy) / t;
    g.bxf = solve == 0 ? I.T[4] : I.A[4];
    g.byf = solve == 0 ? I.T[5] : I.A[5];
    return g;
}

// The pass's tile height -- the one that gives the busiest warp the fewest rows, `halo` rows repeated per
// tile -- and the prefix sums of the instances' tiles, by the first warp; then a block barrier. Every block
// computes the same from the same sizes.
// Instances are taken in the order of `key`, largest first (ord): a variant of a pass is 10-20 KB of straight-
// line code, and warps of an SM that run different ones at a time wait for instructions (pass 1 of the mixed
// batch: 970 us in instance order).
__device__ __forceinline__ int cm_tiles(const CmBInst* sh, const int* key, int n, int halo, int* ord, int* pref, int* h_out) {
    static_assert(CGB_MAX_INST <= 64, "two instances per lane");
    if (threadIdx.x < n) {
        const int me = key[threadIdx.x];
        int rank = 0;
        for (int j = 0; j < n; ++j) rank += key[j] > me || (key[j] == me && j < (int)threadIdx.x);
        ord[rank] = threadIdx.x;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int l = threadIdx.x;
        const long long W = (long long)gridDim.x * CM_NW;
        int h = kCmHeights[l % kCmNHeights];
        long long tiles = 0;
        for (int li = 0; li < n; ++li) tiles += (long long)sh[li].strips * ((sh[li].ny + h - 1) / h);
        long long cost = ((tiles + W - 1) / W) * (h + halo);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {  // lowest cost, then the taller tile
            const long long oc = __shfl_xor_sync(0xffffffffu, cost, o);
            const int oh = __shfl_xor_sync(0xffffffffu, h, o);
            if (oc < cost || (oc == cost && oh > h)) {
                cost = oc;
                h = oh;
            }
        }
        auto count = [&](int pos) { return pos < n ? sh[ord[pos]].strips * ((sh[ord[pos]].ny + h - 1) / h) : 0; };
        const int u0 = count(l), u1 = count(l + 32);
        int s0 = u0, s1 = u1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y0 = __shfl_up_sync(0xffffffffu, s0, o), y1 = __shfl_up_sync(0xffffffffu, s1, o);
            if (l >= o) {
                s0 += y0;
                s1 += y1;
            }
        }
        const int first = __shfl_sync(0xffffffffu, s0, 31);
        if (l < n) pref[l] = s0 - u0;
        if (l + 32 < n) pref[l + 32] = first + s1 - u1;
        if (l == 31) pref[n] = first + s1;
        if (l == 0) *h_out = h;
    }
    __syncthreads();
    return *h_out;
}

// A tile of pass 1: its sums go to part[0 .. 2 M].
template <int M>
static __device__ __noinline__ void cm_tile_moments(CmGeom g, int sx, int r0, int r1, double* part) {
    constexpr int LH = cm_halo_lanes(M, CM_C), NV = 2 * M + 1;
    double* const smem = cm_warp_smem();
    const int lane = threadIdx.x & 31;
    double acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
    cm_moments_segment<M, CM_C, false>(g, sx, r0, r1, smem, acc);  // (one variant: see k_solve_batch on code size)
    const bool halo = lane < LH || lane >= 32 - LH;
    double mine = 0.0;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        double a = halo ? 0.0 : acc[v];
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == v) mine = a;
    }
    if (lane < NV) part[lane] = mine;
}

// A tile of pass 2.
template <int DEG>
static __device__ __noinline__ void cm_tile_poly(CmGeom g, int sx, int r0, int r1, const double* q, double* x) {
    cm_poly_segment<DEG, CM_C>(g, sx, r0, r1, cm_warp_smem(), q, x);
}
__device__ __forceinline__ int cm_batch_degree(int k) { return k <= 5 ? 4 : (k <= 7 ? 6 : CM_MAXM - 1); }

static __global__ void __launch_bounds__(CM_NT, 1)
k_solve_batch(const __grid_constant__ SolveBatchArgs a) {
    __shared__ CmBInst sh[CGB_MAX_INST];
    __shared__ BatchPlan plans[CGB_MAX_INST];
    __shared__ int pref[CGB_MAX_INST + 1], ord[CGB_MAX_INST], key[CGB_MAX_INST];
    __shared__ double mu[32];
    __shared__ CmPlan plan;
    __shared__ int tile_h, sflag;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int W = gridDim.x * CM_NW;
    const int wfirst = wid * gridDim.x + blockIdx.x;
    unsigned long long target = barrier_base(a.sync);
    const unsigned long long deadline = global_timer_ns() + (unsigned long long)(a.timeout_s * 1e9);
    auto barrier = [&]() {
        if (grid_barrier(a.sync, target, deadline, &sflag)) return true;
        if (tid == 0)
            for (int li = 0; li < a.n; ++li) {
                atomicOr(&a.insts[a.list[li]].st->flags, (unsigned)kStatusTimeout);
                a.todo[a.list[li]] = 0;
            }
        return false;
    };
    for (int li = tid; li < a.n; li += CM_NT) {
        const BatchInst& I = a.insts[a.list[li]];
        const double alpha = I.C->alpha;
        CmBInst& S = sh[li];
        const double cx = alpha / (I.D.dx * I.D.dx), cy = alpha / (I.D.dy * I.D.dy);
        S.t = 2 * (cx + cy);
        S.diag = 1 + S.t;
        S.scale = I.D.eta / I.D.dx;
        S.nx = I.D.nx;
        S.ny = I.D.ny;
        S.M = S.t >= 1e-30 && S.t <= kCmMaxT ? cm_levels(S.t) : 0;
        const int out = S.M == 5 ? cm_out(5, CM_C) : (S.M == 7 ? cm_out(7, CM_C) : cm_out(CM_MAXM, CM_C));
        S.strips = S.M ? (S.nx + out - 1) / out : 0;
        key[li] = S.M;
    }
    __syncthreads();
    // ---- pass 1
    int h = cm_tiles(sh, key, a.n, 2 * 7, ord, pref, &tile_h);
    auto tiles = [&](auto&& f) {
        int pos = 0;
        for (int j = wfirst; j < pref[a.n]; j += W) {
            while (pref[pos + 1] <= j) ++pos;
            const int li = ord[pos], w = j - pref[pos];
            const int sx = w % sh[li].strips, r0 = (w / sh[li].strips) * h;
            f(j, li, sx, r0, min(r0 + h, sh[li].ny));
        }
    };
    tiles([&](int j, int li, int sx, int r0, int r1) {
        const CmGeom g = batch_geom(a.insts[a.list[li]], a.solve, sh[li].t);
        double* const part = a.partials + (size_t)j * CM_NMU;
        if (sh[li].M == 5) cm_tile_moments<5>(g, sx, r0, r1, part);
        else if (sh[li].M == 7) cm_tile_moments<7>(g, sx, r0, r1, part);
        else cm_tile_moments<CM_MAXM>(g, sx, r0, r1, part);
    });
    if (!barrier()) return;
    // ---- plans: block b does instances b, b + G, ...; the tiles' sums in a fixed order
    for (int pos = blockIdx.x; pos < a.n; pos += gridDim.x) {
        const int li = ord[pos], M = sh[li].M, inst = a.list[li];
        const BatchInst& I = a.insts[inst];
        int mode = kCmScratch;
        if (M) {
            if (tid < 32) mu[tid] = 0.0;
            __syncthreads();
            const double s2 = sh[li].scale * sh[li].scale;
            for (int v = wid; v <= 2 * M; v += CM_NW) {
                double x = 0.0;
#pragma unroll 4
                for (int j = pref[pos] + lane; j < pref[pos + 1]; j += 32) x += __ldcg(&a.partials[(size_t)j * CM_NMU + v]);
                for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                if (lane == 0) mu[v] = x * s2;
            }
            __syncthreads();
            if (wid == 0) cm_plan(mu[lane], M, sh[li].t, sh[li].diag, sh[li].scale, I.tol, I.max_iters, &plan);
            __syncthreads();
            mode = plan.mode == kCmContinue ? kCmScratch : plan.mode;
        }
        BatchPlan& P = a.plans[li];
        if (tid < CM_MAXM) P.q[tid] = (mode == kCmDone || mode == kCmCapped) ? plan.q[tid] : 0.0;
        if (tid == 0) {
            P.mode = mode;
            P.k = M ? plan.k : 0;
            a.todo[inst] = mode == kCmScratch;
            if (mode != kCmScratch) {
                CgResult res{};
                res.products = (mode == kCmDone || mode == kCmCapped) ? plan.k : 0;
                res.bb = plan.bb;
                res.rr = plan.rr;
                res.breakdown = mode == kCmBreakdown;
                res.converged = mode == kCmDone || mode == kCmZero;
                batch_report(I, inst, a.solve, a.rec_stride, a.prods_rec, res);
            }
        }
        __syncthreads();
    }
    if (!barrier()) return;
    // ---- pass 2
    for (int li = tid; li < a.n; li += CM_NT) {
        BatchPlan P;
        P.mode = __ldcg(&a.plans[li].mode);
        P.k = __ldcg(&a.plans[li].k);
#pragma unroll
        for (int v = 0; v < CM_MAXM; ++v) P.q[v] = __ldcg(&a.plans[li].q[v]);
        plans[li] = P;
        const int deg = cm_batch_degree(P.k);
        const int out = deg == 4 ? cm_out(4, CM_C) : (deg == 6 ? cm_out(6, CM_C) : cm_out(CM_MAXM - 1, CM_C));
        sh[li].strips = P.mode == kCmScratch ? 0 : (sh[li].nx + out - 1) / out;
        key[li] = deg;
    }
    __syncthreads();
    h = cm_tiles(sh, key, a.n, 2 * 5, ord, pref, &tile_h);
    tiles([&](int, int li, int sx, int r0, int r1) {
        const BatchInst& I = a.insts[a.list[li]];
        const int mode = plans[li].mode, deg = cm_batch_degree(plans[li].k);
        if (mode == kCmZero || mode == kCmBreakdown) {
            const int out = cm_out(4, CM_C), i1 = min((sx + 1) * out, sh[li].nx);
            for (int j = r0; j < r1; ++j)
                for (int i = sx * out + lane; i < i1; i += 32) I.x[(size_t)j * sh[li].nx + i] = 0.0;
            return;
        }
        const CmGeom g = batch_geom(I, a.solve, sh[li].t);
        if (deg == 4) cm_tile_poly<4>(g, sx, r0, r1, plans[li].q, I.x);
        else if (deg == 6) cm_tile_poly<6>(g, sx, r0, r1, plans[li].q, I.x);
        else cm_tile_poly<CM_MAXM - 1>(g, sx, r0, r1, plans[li].q, I.x);
    });
}

}  // namespace mhd

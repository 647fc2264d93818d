// The implicit solve of a context, an adjoint and the allocation-free call: its kernels (one copy in the library: the
// other translation units see the functions of mhd_solve.h only) and the choice between them.
#include "mhd_solve.h"

#include "mhd_cg_band.cuh"
#include "mhd_cg_cluster.cuh"

namespace mhd {

// START: behind k_solve, which says in a.start what is left to do.
template <bool START>
static __global__ void __launch_bounds__(CGS_NT, MHD_CG_MIN_BLOCKS)
k_cg_sweep(const __grid_constant__ CgSweepArgs a) {
    __shared__ double red[CGS_NT / 32 * 4];
    __shared__ double scal[8];
    __shared__ int sflag;
#if defined(__CUDA_ARCH__)
    extern __shared__ __align__(16) double cg_ring_mem[];
#else
    // host compilation of the kernel sources (single-block logic tests): one shared copy
    static double cg_ring_mem[(CGS_NT / 32) * CG_RING * CG_SLOT];
#endif
    CgStart start{};
    if constexpr (START) {
        start = *a.start;
        if (start.k < 0) return;
    }
    double* const ring = cg_ring_mem + (size_t)(threadIdx.x >> 5) * CG_RING * CG_SLOT;
    const int tid = threadIdx.x;
    CgScal s = cg_scalars(a);
    unsigned long long target = barrier_base(a.sync);
    const unsigned long long deadline =
        global_timer_ns() + (unsigned long long)(a.timeout_s * 1e9);
    auto barrier = [&]() -> bool {
        if (grid_barrier(a.sync, target, deadline, &sflag)) return true;
        // (any block: one that gives up leaves its part undone)
        if (tid == 0) atomicOr(&a.st->flags, (unsigned)kStatusTimeout);
        return false;
    };
    CgResult res{};
    if (cg_iterate<CGS_NT, true, START>(a, a.strips_x, a.seg_h, a.nwarps, s, ring, a.partials, red, scal, barrier, start, res) && blockIdx.x == 0 && tid == 0)
        cg_report(a, res);
}

static __global__ void __launch_bounds__(CC_NT, 1)
k_cg_cluster(const __grid_constant__ CgSweepArgs a) {
    __shared__ CcTable tab;
#if defined(__CUDA_ARCH__)
    extern __shared__ __align__(16) double cc_mem[];
#else
    static double cc_mem[CC_SMEM_DOUBLES];
#endif
    const unsigned long long deadline = global_timer_ns() + (unsigned long long)(a.timeout_s * 1e9);
    CgResult res{};
    const bool ok = cc_solve_any(a.D, gridDim.x, a.C->alpha, a.bxf, a.byf, a.x, a.tol, a.max_iters, deadline, cc_mem, &tab, res);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (ok) cg_report(a, res);
        else atomicOr(&a.st->flags, (unsigned)kStatusTimeout);
    }
    cooperative_groups::this_cluster().sync();  // no block leaves while another may write into its shared memory
}

static __global__ void __launch_bounds__(CM_NT, 1)
k_solve(const __grid_constant__ CgSweepArgs a) {
    __shared__ double red[CM_NW][CM_NMU];
    __shared__ double mu[32];
    __shared__ double scal[8];
    __shared__ CmPlan plan;
    __shared__ int sflag;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    CgScal s = cg_scalars(a);
    const double t = 2 * (s.cx + s.cy);
    const bool in_range = t >= 1e-30 && t <= (a.from_rhs ? kCmSureT : kCmMaxT);
    if (a.start && !in_range) {  // the CG kernel launched next does all of it
        if (blockIdx.x == 0 && tid == 0) a.start->k = 0;
        return;
    }
    const int G = gridDim.x, warps = G * CM_NW;
    // consecutive segments go to different SMs, so that few of them spread out
    const int wfirst = wid * G + blockIdx.x;
    unsigned long long target = barrier_base(a.sync);
    const unsigned long long deadline = global_timer_ns() + (unsigned long long)(a.timeout_s * 1e9);
    CmGeom g;
    g.nx = a.D.nx;
    g.ny = a.D.ny;
    g.ratio = a.D.dx / a.D.dy;
    g.ax = s.cx / t;
    g.ay = s.cy / t;
    g.bxf = a.bxf;
    g.byf = a.byf;
    const double scale = a.D.eta / a.D.dx;
    bool alive = true;
    auto barrier = [&]() {
        if (alive && !grid_barrier(a.sync, target, deadline, &sflag)) {
            alive = false;
            // (any block: one that gives up leaves its part of x unwritten)
            if (tid == 0) atomicOr(&a.st->flags, (unsigned)kStatusTimeout);
        }
        return alive;
    };
    int mode = kCmScratch;
    if (in_range) {
        const int M = cm_levels(t);
        if (M == 5) cm_pass1_any<5>(g, wfirst, warps, a.partials, red);
        else if (M == 7) cm_pass1_any<7>(g, wfirst, warps, a.partials, red);
        else cm_pass1_any<CM_MAXM>(g, wfirst, warps, a.partials, red);
        if (barrier()) {
            // every block adds the blocks' partials in the same order
            if (tid < 32) mu[tid] = 0.0;
            __syncthreads();
            for (int v = wid; v <= 2 * M; v += CM_NW) {
                double x = 0.0;
#pragma unroll 5
                for (int b = lane; b < G; b += 32) x += __ldcg(&a.partials[(size_t)v * G + b]);
                for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                if (lane == 0) mu[v] = x * (scale * scale);
            }
            __syncthreads();
            if (wid == 0) cm_plan(mu[lane], M, t, s.diag, scale, a.tol, a.max_iters, &plan);
            __syncthreads();
            mode = plan.mode;
            if (mode == kCmContinue && a.from_rhs) mode = kCmScratch;
            if (mode == kCmDone || mode == kCmCapped || mode == kCmContinue)
                cm_pass2_any(g, plan.k - 1, wfirst, warps, plan.q, a.x);
        }
    }
    CgResult res{};
    bool report = alive;
    if (alive && (mode == kCmScratch || mode == kCmContinue)) {
        CgStart start{};
        if (mode == kCmContinue) {
            // r_k into the buffer iteration k reads, p_{k-1} likewise (k is odd)
            cm_pass2_any(g, plan.k, wfirst, warps, plan.qr, a.r[1]);
            cm_pass2_any(g, plan.k - 1, wfirst, warps, plan.qp, a.p[0]);
            start.k = plan.k;
            start.alpha = plan.alpha;
            start.alpha_prev = plan.alpha_prev;
            start.beta = plan.beta;
            start.absNew = plan.absNew;
            start.pAp = plan.pAp;
            start.bb = plan.bb;
            start.threshold = plan.threshold;
        }
        if (a.start) {  // the CG kernel launched next takes over
            report = false;
            if (blockIdx.x == 0 && tid == 0) *a.start = start;
        } else {
            __syncthreads();  // the rings change their layout
            if (mode == kCmScratch || barrier()) {
                const int strips = (g.nx + CG_W - 1) / CG_W;
                const int segs = max(1, warps / strips);
                const int seg_h = max(4, (g.ny + segs - 1) / segs);
                // (partials of its own: other blocks may still read the moments')
                cg_iterate<CM_NT, false, true>(a, strips, seg_h, strips * ((g.ny + seg_h - 1) / seg_h), s,
                                  cm_warp_smem(), a.partials + (size_t)CM_NMU * G, &red[0][0],
                                  scal, barrier, start, res);
            }
            report = alive;
        }
    } else if (alive) {
        res.products = (mode == kCmDone || mode == kCmCapped) ? plan.k : 0;
        res.bb = plan.bb;
        res.rr = plan.rr;
        res.breakdown = mode == kCmBreakdown;
        res.converged = mode == kCmDone || mode == kCmZero;
        if (mode == kCmZero || mode == kCmBreakdown) {
            const size_t n = (size_t)g.nx * g.ny;
            for (size_t e = (size_t)blockIdx.x * CM_NT + tid; e < n; e += (size_t)G * CM_NT) a.x[e] = 0.0;
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        if (report) cg_report(a, res);
        // solved, or given up: nothing is left for the CG kernel
        if (a.start && (report || !alive)) a.start->k = -1;
    }
}

// a.start: behind k_solve, which says there whether anything is left to do.
static __global__ void __launch_bounds__(CB_NT, 1)
k_cg_band(const __grid_constant__ CgSweepArgs a) {
    __shared__ CbShared sh;
#if defined(__CUDA_ARCH__)
    extern __shared__ __align__(16) double cb_mem[];
#else
    static double cb_mem[CB_SMEM_DOUBLES];
#endif
    if (a.start && a.start->k < 0) return;
    unsigned long long target = barrier_base(a.sync);
    const unsigned long long deadline = global_timer_ns() + (unsigned long long)(a.timeout_s * 1e9);
    auto barrier = [&]() -> bool {
        if (grid_barrier(a.sync, target, deadline, &sh.flag)) return true;
        if (threadIdx.x == 0) atomicOr(&a.st->flags, (unsigned)kStatusTimeout);
        return false;
    };
    const int Rmax = (a.D.ny + (int)gridDim.x - 1) / (int)gridDim.x;
    const long long runs = (long long)a.D.nx * ((Rmax + CB_V - 1) / CB_V);
    CgResult res{};
    const bool ok = runs <= CB_NT ? cb_solve<1>(a, cb_mem, &sh, barrier, res)
                    : runs <= 2 * CB_NT ? cb_solve<2>(a, cb_mem, &sh, barrier, res)
                                        : cb_solve<CB_ITEMS>(a, cb_mem, &sh, barrier, res);
    if (ok && blockIdx.x == 0 && threadIdx.x == 0) cg_report(a, res);
}

}  // namespace mhd

namespace mhd_host {

mhd_status solve_setup(const SolveGeom* g) {
    const bool cluster = !g || g->cluster, others = !g || !g->cluster;
    int occ = 0;
    if (cluster)
        MHD_TRY(cudaFuncSetAttribute(mhd::k_cg_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(mhd::CC_SMEM_DOUBLES * sizeof(double))));
    if (others) {
        MHD_TRY(cudaFuncSetAttribute(mhd::k_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mhd::kCmSmemBytes));
        MHD_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, mhd::k_solve, mhd::CM_NT, mhd::kCmSmemBytes));
        if (occ < 1) return MHD_ERR_CUDA;
    }
    if (others && (!g || g->band))
        MHD_TRY(cudaFuncSetAttribute(mhd::k_cg_band, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(mhd::CB_SMEM_DOUBLES * sizeof(double))));
    if (others && (!g || !g->band)) {
        for (auto k : {mhd::k_cg_sweep<false>, mhd::k_cg_sweep<true>}) {
            MHD_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mhd::kCgRingBytes));
            MHD_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, mhd::CGS_NT, mhd::kCgRingBytes));
            if (occ < 1) return MHD_ERR_CUDA;
        }
    }
    return MHD_OK;
}

// One wave of co-resident blocks, no more than there are rows of work for their warps.
SolveGeom solve_geometry(int nx, int ny, int num_sms) {
    SolveGeom g;
    constexpr int NW = mhd::CGS_NT / 32;
    g.strips_x = (nx + mhd::CG_W - 1) / mhd::CG_W;
    const long long rows = (long long)g.strips_x * ny;
    g.grid = (int)std::max(1LL, std::min((long long)num_sms, (rows + NW * 4 - 1) / (NW * 4)));
    const int segs = std::max(1, g.grid * NW / g.strips_x);
    g.seg_h = std::max(4, (ny + segs - 1) / segs);
    g.nwarps = g.strips_x * ((ny + g.seg_h - 1) / g.seg_h);
    // k_solve: narrow segments of 12 rows, one a warp, until every SM has a block. Spread thinner (4 rows, half
    // the warps of a block) a solve is 2-6% shorter on a grid of some 60 000 cells, but takes every SM for it: three
    // contexts stepping 444 x 209, 73 x 914 and 51 x 747 grids on streams of their own then took 250, 562 and 695 us
    // for 168, 342 and 405 (two, five and seven steps each).
    const int out = mhd::cm_out(mhd::CM_MAXM, 1);
    const long long nseg = (long long)((nx + out - 1) / out) * ((ny + 11) / 12);
    g.mgrid = (int)std::max(1LL, std::min((long long)num_sms, (nseg + mhd::CM_NW - 1) / mhd::CM_NW));
    // the largest cluster whose bands have at least one row
    int cs = mhd::CC_MAX;
    while (cs > 1 && ny < cs) cs /= 2;
    g.cluster = mhd::cc_fits(nx, ny, cs) ? cs : 0;
    g.band = mhd::cb_bands(nx, ny, num_sms);
    return g;
}

// Cells from which on a caller's field takes the two passes. Their length does not depend on the field; smooth fields of
// few modes take two products up to t = 8e-3 or so and three or four beyond, and the sweeps are then shorter up to the
// grids below (k_cg_sweep against k_solve, us a call):
//   t = 1e-3, 2 products   1800^2 130, 141   2048^2 155, 166   2200^2 176, 172   2700^2 239, 215
//   t = 2e-3, 2 products   2048^2 156, 177   2400^2 205, 217   2700^2 252, 256
//   t = 1e-2, 3 products   1500^2 141, 131   2048^2 219, 179
//   t = 0.03, 3 products   1500^2 142, 154   1600^2 156, 160   1800^2 188, 178   2048^2 226, 203
//   t = 0.05, 4 products   1600^2 157, 158   1800^2 185, 181   2048^2 224, 206
// (noise, 4 to 9 products, gains from the two passes on any of these: 1.2 to 2 times.)
static long long field_line(double t) {
    if (t < 1.2e-3) return 4800000;
    if (t < 8e-3) return 7000000;
    return t < 0.0155 ? 1 << 21 : 2900000;
}

mhd_status launch_solve(mhd::CgSweepArgs a, const SolveGeom& g, double t, bool field, SolveSync* dev,
                        cudaStream_t stream) {
    cudaLaunchConfig_t cfg{};
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    if (g.cluster) {
        cfg.gridDim = dim3(g.cluster);
        cfg.blockDim = dim3(mhd::CC_NT);
        cfg.dynamicSmemBytes =
            (size_t)mhd::cc_smem_doubles(a.D.nx, (a.D.ny + g.cluster - 1) / g.cluster) * sizeof(double);
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = g.cluster;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        MHD_TRY(cudaLaunchKernelEx(&cfg, mhd::k_cg_cluster, a));
        return MHD_OK;
    }
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    a.strips_x = g.strips_x;
    a.seg_h = g.seg_h;
    a.nwarps = g.nwarps;
    const bool moments = t <= (g.band ? mhd::kCmSureT : mhd::kCmMaxT) &&
                         !(field && (long long)a.D.nx * a.D.ny < field_line(t));
    const bool sweep = t < 0.0 || !moments || !mhd::cm_sure(t);
    a.start = moments && sweep ? &dev->start : nullptr;
    a.from_rhs = a.start && g.band;
    if (moments) {
        a.sync = &dev->sync[0];
        cfg.gridDim = dim3(g.mgrid);
        cfg.blockDim = dim3(mhd::CM_NT);
        cfg.dynamicSmemBytes = mhd::kCmSmemBytes;
        MHD_TRY(cudaLaunchKernelEx(&cfg, mhd::k_solve, a));
    }
    if (sweep && g.band) {
        a.sync = &dev->sync[1];
        cfg.gridDim = dim3(g.band);
        cfg.blockDim = dim3(mhd::CB_NT);
        cfg.dynamicSmemBytes =
            (size_t)mhd::cb_smem_doubles(a.D.nx, (a.D.ny + g.band - 1) / g.band) * sizeof(double);
        MHD_TRY(cudaLaunchKernelEx(&cfg, mhd::k_cg_band, a));
    } else if (sweep) {
        a.sync = &dev->sync[1];
        cfg.gridDim = dim3(g.grid);
        cfg.blockDim = dim3(mhd::CGS_NT);
        cfg.dynamicSmemBytes = mhd::kCgRingBytes;
        MHD_TRY(cudaLaunchKernelEx(&cfg, a.start ? mhd::k_cg_sweep<true> : mhd::k_cg_sweep<false>, a));
    }
    return MHD_OK;
}

}  // namespace mhd_host

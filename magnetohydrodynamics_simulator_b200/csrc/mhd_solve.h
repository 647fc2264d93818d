// Host side of one implicit solve: launch geometry and the choice between its two kernels.
#pragma once

#include <algorithm>

#include "mhd_cg_band.cuh"
#include "mhd_cg_moments.cuh"
#include "mhd_host_util.h"

namespace mhd_host {

struct SolveGeom {
    int strips_x = 0, seg_h = 0, nwarps = 0;  // k_cg_sweep: column strips, rows per warp, warps
    int grid = 0;                             // k_cg_sweep's blocks
    int mgrid = 0;                            // k_solve's blocks
    int cluster = 0;                          // k_cg_cluster's blocks; 0: the grid does not fit a cluster
    int band = 0;                             // k_cg_band's blocks; 0: the grid does not fit the chip's shared memory
    // doubles of the partial sums of either kernel
    size_t partials() const {
        return std::max((size_t)2 * std::max(grid, band) * 4, (size_t)mgrid * (mhd::CM_NMU + 8));
    }
};

// Device memory of the solves of one object besides its planes: two barriers (zeroed when created and
// after a solve that ran out of time) and the hand-over from k_solve to k_cg_sweep.
struct SolveSync {
    mhd::CgSync sync[2];
    mhd::CgStart start;
};

// Once per device: the kernels' shared-memory limits. (static, as the kernels: every translation unit has its own.)
static inline mhd_status solve_setup() {
    int occ = 0;
    for (auto k : {mhd::k_cg_sweep<false>, mhd::k_cg_sweep<true>}) {
        MHD_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mhd::kCgRingBytes));
        MHD_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, mhd::CGS_NT, mhd::kCgRingBytes));
        if (occ < 1) return MHD_ERR_CUDA;
    }
    MHD_TRY(cudaFuncSetAttribute(mhd::k_cg_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(mhd::CC_SMEM_DOUBLES * sizeof(double))));
    MHD_TRY(cudaFuncSetAttribute(mhd::k_cg_band, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(mhd::CB_SMEM_DOUBLES * sizeof(double))));
    MHD_TRY(cudaFuncSetAttribute(mhd::k_solve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)mhd::kCmSmemBytes));
    MHD_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, mhd::k_solve, mhd::CM_NT, mhd::kCmSmemBytes));
    return occ < 1 ? MHD_ERR_CUDA : MHD_OK;
}

// Both kernels: one wave of co-resident blocks, no more than there are rows of work for their warps.
static inline SolveGeom solve_geometry(int nx, int ny, int num_sms) {
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

// t = 2 alpha (1/dx^2 + 1/dy^2) of a solve, which decides its form (mhd_cg_moments.cuh).
inline double solve_t(double alpha, double dx, double dy) {
    return 2.0 * alpha * (1.0 / (dx * dx) + 1.0 / (dy * dy));
}

// Launch the solve of `a` (its geometry, sync and start are set here). t: solve_t where the host knows
// alpha, else negative (the step's dt is chosen on the device). Up to kCmMaxT k_solve alone (two passes
// over the face planes), beyond it CG alone: k_cg_band where the chip's shared memory holds the grid, else
// k_cg_sweep (one sweep per product). Where the host does not know, k_solve comes first and CG behind it
// finds the solve done, or does it: an idle kernel costs 1 us. (k_cg_band starts from the right-hand side;
// k_cg_sweep also takes up an iteration that k_solve left.)
// Grids that fit one cluster take k_cg_cluster, whatever the matrix.
// field: the right-hand side is a caller's field, not an evolved one. Smooth fields take two to four products,
// and below 1448^2 as many are shorter than the two passes, whose length does not depend on them
// (1024^2 with k_cg_sweep: 3 products 66 against 76 us; 2048^2: 198 against 154); in a step there are five or more.
static inline mhd_status launch_solve(mhd::CgSweepArgs a, const SolveGeom& g, double t, bool field, SolveSync* dev,
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
    const bool moments = t <= mhd::kCmMaxT && !(field && (long long)a.D.nx * a.D.ny < (1 << 21));
    const bool sweep = t < 0.0 || !moments;
    a.start = (t < 0.0 && sweep) ? &dev->start : nullptr;
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

// Host side of one implicit solve: launch geometry and the choice between its two kernels.
#pragma once

#include <algorithm>

#include "mhd_cg_moments.cuh"
#include "mhd_host_util.h"

namespace mhd_host {

struct SolveGeom {
    int strips_x = 0, seg_h = 0, nwarps = 0;  // k_cg_sweep: column strips, rows per warp, warps
    int grid = 0;                             // k_cg_sweep's blocks
    int mgrid = 0;                            // k_solve's blocks
    bool small = false;                       // k_solve alone, whatever the matrix
    // doubles of the partial sums of either kernel
    size_t partials() const {
        return std::max((size_t)2 * grid * 4, (size_t)mgrid * (mhd::CM_NMU + 8));
    }
};

// Device memory of the solves of one object besides its planes: two barriers (zeroed when created and
// after a solve that ran out of time) and the hand-over from k_solve to k_cg_sweep.
struct SolveSync {
    mhd::CgSync sync[2];
    mhd::CgStart start;
};

// Once per device: the kernels' shared-memory limits.
inline mhd_status solve_setup() {
    int occ = 0;
    for (auto k : {mhd::k_cg_sweep<false>, mhd::k_cg_sweep<true>}) {
        MHD_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mhd::kCgRingBytes));
        MHD_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, mhd::CGS_NT, mhd::kCgRingBytes));
        if (occ < 1) return MHD_ERR_CUDA;
    }
    MHD_TRY(cudaFuncSetAttribute(mhd::k_solve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)mhd::kCmSmemBytes));
    MHD_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, mhd::k_solve, mhd::CM_NT, mhd::kCmSmemBytes));
    return occ < 1 ? MHD_ERR_CUDA : MHD_OK;
}

// Both kernels: one wave of co-resident blocks, no more than there are rows of work for their warps.
inline SolveGeom solve_geometry(int nx, int ny, int num_sms) {
    SolveGeom g;
    constexpr int NW = mhd::CGS_NT / 32;
    g.strips_x = (nx + mhd::CG_W - 1) / mhd::CG_W;
    const long long rows = (long long)g.strips_x * ny;
    g.grid = (int)std::max(1LL, std::min((long long)num_sms, (rows + NW * 4 - 1) / (NW * 4)));
    const int segs = std::max(1, g.grid * NW / g.strips_x);
    g.seg_h = std::max(4, (ny + segs - 1) / segs);
    g.nwarps = g.strips_x * ((ny + g.seg_h - 1) / g.seg_h);
    // k_solve: segments of 4 rows or more, two per block until every SM has a block
    const int out = mhd::cm_out(mhd::CM_MAXM);
    const long long nseg = (long long)((nx + out - 1) / out) * ((ny + 3) / 4);
    g.mgrid = (int)std::max(1LL, std::min((long long)num_sms, (nseg + 1) / 2));
    g.small = (long long)nx * ny <= 256 * 256;
    return g;
}

// t = 2 alpha (1/dx^2 + 1/dy^2) of a solve, which decides its form (mhd_cg_moments.cuh).
inline double solve_t(double alpha, double dx, double dy) {
    return 2.0 * alpha * (1.0 / (dx * dx) + 1.0 / (dy * dy));
}

// Launch the solve of `a` (its geometry, sync and start are set here). t: solve_t where the host knows
// alpha, else negative (the step's dt is chosen on the device). Up to kCmMaxT k_solve alone (two passes
// over the face planes), beyond it k_cg_sweep alone (one sweep per product). Where the host does not
// know, k_solve comes first and k_cg_sweep behind it finds the solve done, or does it: an idle kernel
// costs 1 us, the sweeps on k_solve's half as many warps a quarter more time (1024^2: 188 against 150 us).
// Small grids, whose t is small (it grows with eta / dx under the CFL rule), take k_solve alone.
inline mhd_status launch_solve(mhd::CgSweepArgs a, const SolveGeom& g, double t, SolveSync* dev, cudaStream_t stream) {
    cudaLaunchConfig_t cfg{};
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    a.strips_x = g.strips_x;
    a.seg_h = g.seg_h;
    a.nwarps = g.nwarps;
    const bool sweep = t > mhd::kCmMaxT || (t < 0.0 && !g.small);
    a.start = (t < 0.0 && sweep) ? &dev->start : nullptr;
    if (t <= mhd::kCmMaxT) {
        a.sync = &dev->sync[0];
        cfg.gridDim = dim3(g.mgrid);
        cfg.blockDim = dim3(mhd::CM_NT);
        cfg.dynamicSmemBytes = mhd::kCmSmemBytes;
        MHD_TRY(cudaLaunchKernelEx(&cfg, mhd::k_solve, a));
    }
    if (sweep) {
        a.sync = &dev->sync[1];
        cfg.gridDim = dim3(g.grid);
        cfg.blockDim = dim3(mhd::CGS_NT);
        cfg.dynamicSmemBytes = mhd::kCgRingBytes;
        MHD_TRY(cudaLaunchKernelEx(&cfg, a.start ? mhd::k_cg_sweep<true> : mhd::k_cg_sweep<false>, a));
    }
    return MHD_OK;
}

}  // namespace mhd_host

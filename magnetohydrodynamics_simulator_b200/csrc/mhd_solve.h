// One implicit solve: its launch geometry, and the choice between its kernels (mhd_solve.cu).
#pragma once

#include <algorithm>

#include "mhd_cg_moments.cuh"
#include "mhd_host_util.h"

namespace mhd_host {

struct SolveGeom {
    int strips_x = 0, seg_h = 0, nwarps = 0;  // k_cg_sweep: column strips, rows per warp, warps
    int grid = 0;                             // k_cg_sweep's blocks
    int mgrid = 0;                            // k_solve's blocks
    int cluster = 0;                          // k_cg_cluster's blocks; 0: the grid does not fit a cluster
    int band = 0;                             // k_cg_band's blocks; 0: the grid does not fit the chip's shared memory
    // doubles of the partial sums of any of them
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

// The shared-memory limits of the kernels that a grid's solves may take (null: of all of them), on the current device.
mhd_status solve_setup(const SolveGeom* g);

SolveGeom solve_geometry(int nx, int ny, int num_sms);

// t = 2 alpha (1/dx^2 + 1/dy^2) of a solve, which decides its form (mhd_cg_moments.cuh).
inline double solve_t(double alpha, double dx, double dy) {
    return 2.0 * alpha * (1.0 / (dx * dx) + 1.0 / (dy * dy));
}

// Launch the solve of `a` (its geometry, sync and start are set here). t: solve_t where the host knows
// alpha, else negative (the step's dt is chosen on the device).
// Up to kCmSureT k_solve (two passes over the face planes). Beyond it the levels may not suffice, and the passes are then
// lost: grids that the chip's shared memory holds take k_cg_band (steps of fixed dt at t = 0.06, 10 products a solve, with
// the two passes first and with k_cg_band alone: 300^2 249 and 156 us, 512^2 307 and 197, 1000^2 619 and 363; with 9
// products, which the passes settle, 177 and 143, 168 and 179, 343 and 330), larger ones k_solve up to kCmMaxT and
// k_cg_sweep (one sweep per product) after that.
// A CG kernel behind k_solve finds the solve done, or does it: where the host does not know t, and where the levels are
// not sure to suffice. An idle kernel costs 4 us; without it k_solve goes on with sweeps of its own, which are slower
// (t = 0.06, 10 products: a step at 1448^2 900 us, 780 with k_cg_sweep behind).
// Grids that fit one cluster take k_cg_cluster, whatever the matrix.
// field: the right-hand side is a caller's field, not an evolved one, which in a step takes five products or more: below
// field_line(t) cells it takes CG alone.
mhd_status launch_solve(mhd::CgSweepArgs a, const SolveGeom& g, double t, bool field, SolveSync* dev,
                        cudaStream_t stream);

}  // namespace mhd_host

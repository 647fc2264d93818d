// The implicit solve of a small grid: conjugate gradients by one cluster of thread blocks, with every
// vector in its shared memory and registers (reference: solvers.hpp:404-489 with Eigen's
// ConjugateGradient defaults, as in mhd_cg_sweep.cuh).
//
// Small grids are bound by latency: a product of k_cg_sweep costs a grid-wide barrier through L2 and a
// pass over memory, 4-6 us whatever the size. Here block `rank` of the cluster owns a band of rows; r
// (with a halo row on each side), p and s = A p live in its shared memory, x in registers. A block writes
// its edge rows into its neighbours' halos and its sums into every block's table (distributed shared
// memory), and the hardware's cluster barrier is the only wait. A product is (Chronopoulos and Gear 1989,
// one reduction instead of two):
//   A r and the sums r.r, r.Ar;  barrier;
//   beta = g / g_old, alpha = g / (d - beta g / alpha_old) with g = r.z, d = z.Az, z = r / diag;
//   p = z + beta p, s = A z + beta s, x += alpha p, r -= alpha s, edges;  barrier.
// In exact arithmetic these are CG's iterates. The blocks' sums are added in rank order by every block, so
// all take the same decisions and the result is deterministic.
//
// Measured on B200, one solve against k_cg_sweep: 64^2 (5 products) 40 -> 21 us, 128^2 (6) 45 -> 27 us.
//
// A thread owns runs of V rows of a column (V = 4: the rows above and below are its own registers but
// two; V = 1 while the band has few cells).
#pragma once

#include <cooperative_groups.h>

#include "mhd_cg_sweep.cuh"

namespace mhd {

constexpr int CC_NT = 512;    // threads per block
constexpr int CC_MAX = 8;     // blocks per cluster (the portable limit)
constexpr int CC_ITEMS = 2;   // most runs per thread
constexpr int CC_SMEM_DOUBLES = 14336;  // 112 KB
// Doubles of dynamic shared memory of a block whose band has at most R rows: r with halos, p, s.
__host__ __device__ constexpr long long cc_smem_doubles(long long nx, long long R) { return nx * (3 * R + 2); }

// Whether a grid's solve fits a cluster of `blocks` blocks: at most 4096 cells a block (32768 for eight, 181^2).
// Larger bands would fit the shared memory, but its bandwidth then costs more than the grid's barriers: 6.2 us
// a product at 256^2 against 2.0 at 128^2 and 1.8 at 64^2.
__host__ __device__ inline bool cc_fits(int nx, int ny, int blocks) {
    const long long R = ((long long)ny + blocks - 1) / blocks;
    return ny >= blocks && cc_smem_doubles(nx, R) <= CC_SMEM_DOUBLES &&
           (long long)nx * ((R + 3) / 4) <= (long long)CC_ITEMS * CC_NT;
}

struct CcTable {
    double sums[CC_MAX][3];  // r.r, r.Ar, time ran out -- of every rank
    double red[CC_NT / 32][2];
};

// One solve by this cluster. `deadline`: the wall-clock limit, checked once a product by rank 0.
// Returns false when it ran out (res is not set).
template <int V, int ITEMS>
__device__ __forceinline__ bool cc_solve(const Domain& D, double alpha_m, const double* __restrict__ bxf,
                                         const double* __restrict__ byf, double* __restrict__ x_out, double tol,
                                         long long max_iters, unsigned long long deadline, double* smem, CcTable* tab,
                                         CgResult& res) {
    namespace cgr = cooperative_groups;
    auto cluster = cgr::this_cluster();
    const int CS = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int nx = D.nx, ny = D.ny, tid = threadIdx.x;
    auto first_row = [&](int k) { return (int)((long long)ny * k / CS); };
    const int j0 = first_row(rank), R = first_row(rank + 1) - j0, Rmax = (ny + CS - 1) / CS;
    const int below = (rank + CS - 1) % CS, above = (rank + 1) % CS;
    const int R_below = first_row(below + 1) - first_row(below);
    double* const r = smem;                         // row 0 and row R + 1: halos
    double* const p = smem + (size_t)(Rmax + 2) * nx;
    double* const s = p + (size_t)Rmax * nx;
    double* const r_below = cluster.map_shared_rank(r, below) + (size_t)(R_below + 1) * nx;  // its upper halo
    double* const r_above = cluster.map_shared_rank(r, above);                               // its lower halo
    const double cx = alpha_m / (D.dx * D.dx), cy = alpha_m / (D.dy * D.dy);
    const double diag = 1 + 2 * (cx + cy);
    const double invdiag = (diag == 0.0) ? 1.0 : 1.0 / diag;

    // this thread's runs: column, its neighbours, first row and length
    int col[ITEMS], cl[ITEMS], cr[ITEMS], row0[ITEMS], len[ITEMS];
    const int runs = (R + V - 1) / V;
#pragma unroll
    for (int m = 0; m < ITEMS; ++m) {
        const int it = tid + CC_NT * m;
        const int q = it / nx;
        col[m] = it - q * nx;
        cl[m] = col[m] == 0 ? nx - 1 : col[m] - 1;
        cr[m] = col[m] == nx - 1 ? 0 : col[m] + 1;
        row0[m] = q * V;
        len[m] = q < runs ? min(V, R - q * V) : 0;
    }
    auto put_r = [&](int m, int row, double v) {
        r[(size_t)(row + 1) * nx + col[m]] = v;
        if (row == 0) r_below[col[m]] = v;
        if (row == R - 1) r_above[col[m]] = v;
    };

    cluster.sync();  // the neighbours' shared memory exists, and an earlier solve is done with it
    const double idx = 1.0 / D.dx, idy = 1.0 / D.dy;
    double x[ITEMS * V], ar[ITEMS * V];
#pragma unroll
    for (int m = 0; m < ITEMS; ++m)
#pragma unroll
        for (int v = 0; v < V; ++v) {
            x[m * V + v] = 0.0;
            if (v < len[m]) {
                const int row = row0[m] + v, j = j0 + row, jb = j == 0 ? ny - 1 : j - 1;
                const size_t g = (size_t)j * nx;
                put_r(m, row, corner_rhs(D, idx, idy, byf[g + col[m]], byf[g + cl[m]], bxf[g + col[m]],
                                         bxf[(size_t)jb * nx + col[m]]));
                p[(size_t)row * nx + col[m]] = 0.0;
                s[(size_t)row * nx + col[m]] = 0.0;
            }
        }

    double bb = 0.0, threshold = 0.0, rr = 0.0, g_old = 0.0, alpha = 0.0;
    bool breakdown = false, converged = false, zero = false;
    long long k = 0;
    for (;; ++k) {
        cluster.sync();  // r and its halos
        double acc[2] = {0.0, 0.0};
#pragma unroll
        for (int m = 0; m < ITEMS; ++m) {
            if (len[m] == 0) continue;
            const double* rc = r + (size_t)(row0[m] + 1) * nx;
            double lo = rc[col[m] - nx], ce = rc[col[m]];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                if (v < len[m]) {
                    const double hi = rc[(size_t)(v + 1) * nx + col[m]];
                    const double lr = rc[(size_t)v * nx + cl[m]] + rc[(size_t)v * nx + cr[m]];
                    const double a = fma(-cy, lo + hi, fma(-cx, lr, diag * ce));
                    ar[m * V + v] = a;
                    acc[0] = fma(ce, ce, acc[0]);
                    acc[1] = fma(ce, a, acc[1]);
                    lo = ce;
                    ce = hi;
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
            for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
        if ((tid & 31) == 0) {
            tab->red[tid >> 5][0] = acc[0];
            tab->red[tid >> 5][1] = acc[1];
        }
        __syncthreads();
        if (tid < CS) {  // thread q writes this block's sums to rank q
            double a0 = 0.0, a1 = 0.0;
#pragma unroll
            for (int w = 0; w < CC_NT / 32; ++w) {
                a0 += tab->red[w][0];
                a1 += tab->red[w][1];
            }
            CcTable* t = cluster.map_shared_rank(tab, tid);
            t->sums[rank][0] = a0;
            t->sums[rank][1] = a1;
            t->sums[rank][2] = (rank == 0 && global_timer_ns() > deadline) ? 1.0 : 0.0;
        }
        cluster.sync();
        double rar = 0.0;
        rr = 0.0;
        for (int q = 0; q < CS; ++q) {
            rr += tab->sums[q][0];
            rar += tab->sums[q][1];
        }
        if (k == 0) {
            bb = rr;
            threshold = smax(tol * tol * bb, 2.2250738585072014e-308);
            zero = bb == 0.0 || bb < threshold;
            breakdown = !isfinite(bb);
            converged = zero;
            if (zero || breakdown) break;
        } else {
            if (!isfinite(rr) || !isfinite(alpha)) { breakdown = true; break; }
            if (rr < threshold) { converged = true; break; }
        }
        if (tab->sums[0][2] != 0.0) return false;
        if (k >= max_iters) break;
        const double g = rr * invdiag, d = rar * (invdiag * invdiag);
        const double beta = k == 0 ? 0.0 : g / g_old;
        const double pAp = k == 0 ? d : d - beta * (g / alpha);
        if (!(pAp > 0.0)) { breakdown = true; break; }
        alpha = g / pAp;
        g_old = g;
#pragma unroll
        for (int m = 0; m < ITEMS; ++m)
#pragma unroll
            for (int v = 0; v < V; ++v)
                if (v < len[m]) {
                    const int row = row0[m] + v;
                    const size_t e = (size_t)row * nx + col[m];
                    const double rv = r[e + nx];
                    const double pv = fma(beta, p[e], invdiag * rv);
                    const double sv = fma(beta, s[e], invdiag * ar[m * V + v]);
                    p[e] = pv;
                    s[e] = sv;
                    x[m * V + v] = fma(alpha, pv, x[m * V + v]);
                    put_r(m, row, fma(-alpha, sv, rv));
                }
    }
#pragma unroll
    for (int m = 0; m < ITEMS; ++m)
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (v < len[m])
                x_out[(size_t)(j0 + row0[m] + v) * nx + col[m]] = (zero || breakdown) ? 0.0 : x[m * V + v];
    res.products = k;
    res.bb = bb;
    res.rr = k == 0 ? 0.0 : rr;
    res.breakdown = breakdown;
    res.converged = converged;
    return true;
}

// The variant for a band of R rows: one cell a thread at a time while that keeps most threads busy once or
// twice, else runs of four rows.
__device__ __forceinline__ bool cc_solve_any(const Domain& D, int blocks, double alpha_m, const double* bxf, const double* byf,
                                             double* x, double tol, long long max_iters, unsigned long long deadline,
                                             double* smem, CcTable* tab, CgResult& res) {
    const int R = (D.ny + blocks - 1) / blocks;
    if ((long long)D.nx * R <= 2 * CC_NT)
        return cc_solve<1, 2>(D, alpha_m, bxf, byf, x, tol, max_iters, deadline, smem, tab, res);
    if ((long long)D.nx * ((R + 3) / 4) <= CC_NT)
        return cc_solve<4, 1>(D, alpha_m, bxf, byf, x, tol, max_iters, deadline, smem, tab, res);
    return cc_solve<4, CC_ITEMS>(D, alpha_m, bxf, byf, x, tol, max_iters, deadline, smem, tab, res);
}

}  // namespace mhd

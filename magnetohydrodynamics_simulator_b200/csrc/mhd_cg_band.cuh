// The implicit solve of a mid-size grid where the two-pass form does not apply (large t, callers' smooth fields):
// conjugate gradients over the whole chip with every vector on it (reference: solvers.hpp:404-489 with Eigen's
// ConjugateGradient defaults, as in mhd_cg_sweep.cuh).
//
// Block b owns a band of rows; r and s = A p (with a halo row on each side) and p live in its shared memory, x in
// registers. A product is Chronopoulos and Gear's (1989) one-reduction form, as in mhd_cg_cluster.cuh, with one
// grid-wide barrier: a block publishes its sums r.r, r.Ar and the first and last row of A r, and after the barrier
// brings its own halo rows of s and r forward with the neighbours' A r -- the operations, and the bits, of the
// rows' owners. (Exchanging r would take a second barrier.) The blocks' sums are added in the same order by every
// block, so all take the same decisions and the result is deterministic.
//
// Bound by the barrier and two trips to L2, then by shared memory (nine accesses a cell). Against k_cg_sweep, which
// streams p, r and x through L2 in every product: 512^2 at eta 10 (125 products a solve) 10.6 -> 6.7 us a product
// on 128 SMs; 1000 x 700 (13 products) 146 -> 128 us a solve; 1024^2 with 11 and 35 products 284 -> 212 and
// 647 -> 455 us a call.
#pragma once

#include "mhd_cg_cluster.cuh"

namespace mhd {

constexpr int CB_NT = 512;
constexpr int CB_V = 4;                  // rows of a run (a thread's consecutive cells of one column)
constexpr int CB_ITEMS = 4;              // most runs per thread
constexpr int CB_SMEM_DOUBLES = 28672;   // 224 KB
// Cells of a band at least: below it the barrier sets the time of a product, and more SMs only keep other streams
// off the chip (200 x 200, three fixed steps, three contexts on three streams: 499 us with two-row bands, 219 with
// 1600 cells, 251 with 3200; one alone 649, 627 and 737).
constexpr int CB_MIN_CELLS = 1600;
// Doubles of dynamic shared memory of a block whose band has at most R rows.
__host__ __device__ constexpr long long cb_smem_doubles(long long nx, long long R) { return nx * (3 * R + 4); }

// Bands of an nx x ny grid on num_sms SMs; 0: does not fit. Every band has two rows or more (their edge rows share
// the planes a.r with room for two a band).
// Half of the SMs where their shared memory holds the grid (up to some 680^2): a solve is then up to 15% longer, but two
// run side by side. A step of fixed dt at eta 10 (257 to 423 products), one context alone, and each of three on streams
// of their own, in us, with bands for all SMs and for half of them:
//            400^2       450^2       512^2       520^2       560^2       600^2       640^2       660^2
//   alone  1320 1407   1590 1573   1729 1887   2037 2262   2265 2423   2695 2820   2794 2937   3107 3149
//   three  1256  687   1565  769   1684  964   2002 1112   2232 1193   2649 1384   2746 1471   3058 1625
//          682x888     1000x592    1024x592    1024x444    512x888     400x1100    300x1400
//   alone  3998 3973   3660 4179   3725 4274   3454 3840   3036 3277   3717 3896   4262 4690
//   three  4015 2041   3669 2130   3738 2172   3459 1963   3055 1663   3697 1969   4270 2368
// (up to 350^2 CB_MIN_CELLS makes the bands, the same for both.)
inline int cb_bands(int nx, int ny, int num_sms) {
    if (ny < 2 || nx < 2) return 0;
    auto fit = [&](int sms) {
        const int R = std::max({2, (ny + sms - 1) / sms, (CB_MIN_CELLS + nx - 1) / nx});
        const int bands = std::max(1, std::min(ny / R, num_sms));
        const long long Rmax = (ny + bands - 1) / bands;
        return cb_smem_doubles(nx, Rmax) <= CB_SMEM_DOUBLES &&
                       (long long)nx * ((Rmax + CB_V - 1) / CB_V) <= (long long)CB_ITEMS * CB_NT
                   ? bands : 0;
    };
    const int half = fit(std::max(1, num_sms / 2));
    return half ? half : fit(num_sms);
}

struct CbShared {
    double red[CB_NT / 32][2];
    double sum[2];
    int flag;
};

template <bool FULL>
struct CbTag {
    static constexpr bool value = FULL;
};

// The solve; false when time ran out (res is not set).
template <int ITEMS, class Barrier>
__device__ __forceinline__ bool cb_solve(const CgSweepArgs& a, double* smem, CbShared* sh, Barrier& barrier,
                                         CgResult& res) {
    constexpr int V = CB_V, HALO = 2 * ITEMS;
    const int G = (int)gridDim.x, b = (int)blockIdx.x, tid = threadIdx.x;
    const int nx = a.D.nx, ny = a.D.ny;
    auto first_row = [&](int k) { return (int)((long long)ny * k / G); };
    const int j0 = first_row(b), R = first_row(b + 1) - j0, Rmax = (ny + G - 1) / G;
    double* const r = smem;                              // rows 0 and R + 1: halos
    double* const s = r + (size_t)(Rmax + 2) * nx;       // likewise
    double* const p = s + (size_t)(Rmax + 2) * nx;
    const CgScal sc = cg_scalars(a);
    const double cx = sc.cx, cy = sc.cy, diag = sc.diag, invdiag = sc.invdiag;

    // this thread's runs: column, steps to its neighbours in the row, first cell (row * nx + column), length
    int col[ITEMS], dl[ITEMS], dr[ITEMS], row0[ITEMS], at0[ITEMS], len[ITEMS];
    const int runs = (R + V - 1) / V;
#pragma unroll
    for (int m = 0; m < ITEMS; ++m) {
        const int it = tid + CB_NT * m;
        const int q = it / nx;
        col[m] = it - q * nx;
        dl[m] = col[m] == 0 ? nx - 1 : -1;
        dr[m] = col[m] == nx - 1 ? 1 - nx : 1;
        row0[m] = q * V;
        at0[m] = row0[m] * nx + col[m];
        len[m] = q < runs ? min(V, R - q * V) : 0;
    }
    const double idx = 1.0 / a.D.dx, idy = 1.0 / a.D.dy;
#pragma unroll 2
    for (int row = -1; row <= R; ++row) {
        const int j = wrap(j0 + row, ny), jb = j == 0 ? ny - 1 : j - 1;
        const size_t g = (size_t)j * nx;
        for (int i = tid; i < nx; i += CB_NT) {
            r[(row + 1) * nx + i] = corner_rhs(a.D, idx, idy, a.byf[g + i], a.byf[g + (i == 0 ? nx - 1 : i - 1)],
                                                       a.bxf[g + i], a.bxf[(size_t)jb * nx + i]);
            s[(row + 1) * nx + i] = 0.0;
            if (row >= 0 && row < R) p[row * nx + i] = 0.0;
        }
    }
    double x[ITEMS * V], ar[ITEMS * V];
#pragma unroll
    for (int e = 0; e < ITEMS * V; ++e) x[e] = 0.0;
    __syncthreads();

    // where this block's neighbours publish the rows next to its band
    const size_t edge_below = (size_t)(2 * ((b + G - 1) % G) + 1) * nx, edge_above = (size_t)(2 * ((b + 1) % G)) * nx;
    double bb = 0.0, threshold = 0.0, rr = 0.0, g_old = 0.0, alpha = 0.0;
    bool breakdown = false, converged = false, zero = false;
    long long k = 0;
    for (;; ++k) {
        double* const edges = a.r[k & 1];
        double* const part = a.partials + (size_t)(k & 1) * 2 * G;
        double acc[2] = {0.0, 0.0};
        auto product = [&](int m, auto full) {
            constexpr bool kFull = decltype(full)::value;
            const double* rc = r + nx + at0[m];
            double lo = rc[-nx], ce = rc[0];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                if (kFull || v < len[m]) {
                    const double hi = rc[nx];
                    const double lr = rc[dl[m]] + rc[dr[m]];
                    const double w = fma(-cy, lo + hi, fma(-cx, lr, diag * ce));
                    ar[m * V + v] = w;
                    acc[0] = fma(ce, ce, acc[0]);
                    acc[1] = fma(ce, w, acc[1]);
                    lo = ce;
                    ce = hi;
                    rc += nx;
                }
            }
            if (row0[m] == 0) __stcg(&edges[(size_t)(2 * b) * nx + col[m]], ar[m * V]);
            if (row0[m] + len[m] == R) {
                double w = ar[m * V];
#pragma unroll
                for (int v = 1; v < V; ++v)
                    if (kFull || v < len[m]) w = ar[m * V + v];
                __stcg(&edges[(size_t)(2 * b + 1) * nx + col[m]], w);
            }
        };
#pragma unroll
        for (int m = 0; m < ITEMS; ++m) {
            if (len[m] == V) product(m, CbTag<true>{});
            else if (len[m] > 0) product(m, CbTag<false>{});
        }
#pragma unroll
        for (int c = 0; c < 2; ++c)
            for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
        if ((tid & 31) == 0) {
            sh->red[tid >> 5][0] = acc[0];
            sh->red[tid >> 5][1] = acc[1];
        }
        __syncthreads();
        if (tid < 2) {
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < CB_NT / 32; ++w) t += sh->red[w][tid];
            __stcg(&part[(size_t)tid * G + b], t);
        }
        if (!barrier()) return false;
        if (tid < 64) {  // one warp a sum, in block order
            const int c = tid >> 5, l = tid & 31;
            double t = 0.0;
#pragma unroll 5
            for (int q = l; q < G; q += 32) t += __ldcg(&part[(size_t)c * G + q]);
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (l == 0) sh->sum[c] = t;
        }
        double halo[HALO];
#pragma unroll
        for (int h = 0; h < HALO; ++h) {
            const int e = tid + CB_NT * h;
            halo[h] = e < 2 * nx ? __ldcg(&edges[e < nx ? edge_below + e : edge_above + (e - nx)]) : 0.0;
        }
        __syncthreads();
        rr = sh->sum[0];
        const double rar = sh->sum[1];
        if (k == 0) {
            bb = rr;
            threshold = smax(a.tol * a.tol * bb, 2.2250738585072014e-308);
            zero = bb == 0.0 || bb < threshold;
            breakdown = !isfinite(bb);
            converged = zero;
            if (zero || breakdown) break;
        } else {
            if (!isfinite(rr) || !isfinite(alpha)) { breakdown = true; break; }
            if (rr < threshold) { converged = true; break; }
        }
        if (k >= a.max_iters) break;
        const double g = rr * invdiag, d = rar * (invdiag * invdiag);
        const double beta = k == 0 ? 0.0 : g / g_old;
        const double pAp = k == 0 ? d : d - beta * (g / alpha);
        if (!(pAp > 0.0)) { breakdown = true; break; }
        alpha = g / pAp;
        g_old = g;
#pragma unroll
        for (int h = 0; h < HALO; ++h) {
            const int e = tid + CB_NT * h;
            if (e < 2 * nx) {
                const int at = e < nx ? e : (R + 1) * nx + (e - nx);
                const double sv = fma(beta, s[at], invdiag * halo[h]);
                s[at] = sv;
                r[at] = fma(-alpha, sv, r[at]);
            }
        }
        auto update = [&](int m, auto full) {
            constexpr bool kFull = decltype(full)::value;
            int e = at0[m];
#pragma unroll
            for (int v = 0; v < V; ++v)
                if (kFull || v < len[m]) {
                    const double rv = r[e + nx];
                    const double pv = fma(beta, p[e], invdiag * rv);
                    const double sv = fma(beta, s[e + nx], invdiag * ar[m * V + v]);
                    p[e] = pv;
                    s[e + nx] = sv;
                    x[m * V + v] = fma(alpha, pv, x[m * V + v]);
                    r[e + nx] = fma(-alpha, sv, rv);
                    e += nx;
                }
        };
#pragma unroll
        for (int m = 0; m < ITEMS; ++m) {
            if (len[m] == V) update(m, CbTag<true>{});
            else if (len[m] > 0) update(m, CbTag<false>{});
        }
        __syncthreads();  // r and its halos
    }
#pragma unroll
    for (int m = 0; m < ITEMS; ++m)
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (v < len[m])
                a.x[(size_t)(j0 + row0[m] + v) * nx + col[m]] = (zero || breakdown) ? 0.0 : x[m * V + v];
    res.products = k;
    res.bb = bb;
    res.rr = k == 0 ? 0.0 : rr;
    res.breakdown = breakdown;
    res.converged = converged;
    return true;
}

}  // namespace mhd

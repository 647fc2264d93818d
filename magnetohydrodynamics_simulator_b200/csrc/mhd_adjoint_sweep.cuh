// F'(U)^T w of the explicit rate as one warp column sweep: out = base + scale * F'(U)^T w.
//
// A warp owns a strip of AS_OUT = 25 output columns [c0, c0+25) and sweeps its rows upwards; lane l holds column
// i = c0 - 4 + l. A cell's adjoint needs the limited slopes of its neighbours, their faces' adjoints and, for the
// face field, the cell and the face on its left: four columns on the left, three on the right. At sweep row c:
//   PRIM    row c+2
//   CORNER  adjoint of the corner field at (i, c+1) from w, weighted by the branch of its upwind test
//   YFACE   top face of row c: HLL VJP -> adjoint of row c's upper and row c+1's lower extrapolation; row c's
//           slope adjoint is then complete and goes to rows c-1, c and c+1
//   XFACE   right face of column i in row c, and the same along the row by shuffles
//   OUT     row c-1: primitive -> conserved VJP, face fields from the cell-centred adjoints and the normal fields
// U and w come through a per-warp ring of AS_ROWS rows in shared memory, filled by cp.async three rows ahead; a
// lane reads back only what it copied itself, so there is no block-level barrier. What passes from row to row
// (the adjoints of a row that its upper neighbours still add to) stays with the lane.
//
// Lane validity: PRIM 0-31, CORNER 1-31, XFACE 1-29, cells 3-28, outputs 4-28.
//
// Why one kernel: as passes over whole planes (primitives, x faces, y faces, gather, face fields) the 24 planes
// between them were written once and read back up to three times, 305 us at 1024^2 for 150 MB of arguments and
// results (23 us of copy). The sweep takes 113 us there, 20 us at 256^2 (28 with the flux differentiated component
// by component): it is bound by issue and FP64, with 32 lanes at work for 25 columns and two warps a sub-partition.
#pragma once

#include "mhd_adjoint.cuh"

namespace mhd {

constexpr int AS_OUT = 25;
constexpr int AS_ROWS = 8;            // ring rows: c-1 .. c+6
constexpr int AS_SLOT = 12 * 32 + 2;  // U (6 planes), w (6 planes), lane 31's right-hand neighbour of bxf
constexpr int AS_CARRY = 10 * 32;     // row adjoints carried in shared memory
constexpr size_t kAdjSweepSmemBytes = (size_t)(AS_ROWS * AS_SLOT + AS_CARRY) * sizeof(double);
constexpr int AS_PRE_FACE = 3;        // y faces start this many rows before the first output row
constexpr int AS_PRE = 6;             // ... and the primitives this many
// Rows of a segment at least: 3 and 6 take the same time on a 256^2 grid (20 us), 9 take 7% more of a whole
// gradient; 6 sweeps half the extra rows of 3.
constexpr int AS_MIN_ROWS = 6;

// The sweep of output rows [r0, r1) of strip sx. Returns r1 + 1, or the sweep row c at which a cell was not of ordinary
// size: output rows below c - 1 are then written, and nothing of the others. ANY: every cell is.
template <bool ANY>
__device__ __forceinline__ int adj_rate_rows(const Domain& D, const CPlanes& U, const CPlanes& w, const CPlanes& base,
                                             double scale, const Planes& out, int sx, int r0, int r1, double* ring) {
    double* const carry = ring + AS_ROWS * AS_SLOT + (threadIdx.x & 31);
    const int lane = threadIdx.x & 31;
    const int nx = D.nx;
    const int i = sx * AS_OUT - 4 + lane;
    const int iw = wrap(i, nx), iw_r = wrap(i + 1, nx);
    const bool out_lane = lane >= 4 && lane < 4 + AS_OUT && i < nx;
    const double idx = 1.0 / D.dx, idy = 1.0 / D.dy;

    double Prho[4], Pvx[4], Pvy[4], Pp[4], Pbx[4], Pby[4];  // rows c-1 .. c+2
#pragma unroll
    for (int k = 0; k < 4; ++k) { Prho[k] = 1.0; Pvx[k] = 0.0; Pvy[k] = 0.0; Pp[k] = 1.0; Pbx[k] = 0.0; Pby[k] = 0.0; }
    // adjoints of row c's primitives: of its lower y extrapolation (Lo), that plus the slope of row c-1 (Half)
    auto Lo = [&](int k) -> double& { return carry[k * 32]; };
    auto Half = [&](int k) -> double& { return carry[(5 + k) * 32]; };
    double Acc[6];  // of row c-1, but for the slope of row c
#pragma unroll
    for (int k = 0; k < 5; ++k) { Lo(k) = 0.0; Half(k) = 0.0; }
#pragma unroll
    for (int k = 0; k < 6; ++k) Acc[k] = 0.0;
    double p0_prev = 0.0;                     // corner (i, c): weighted for the x face
    double abyc_prev = 0.0;                   // cell-centred by adjoint of row c-2
    double ybn1 = 0.0, ybn2 = 0.0, xbn1 = 0.0;  // normal-field adjoints: y faces c-1, c-2; x face of row c-1

    const int cstart = r0 - AS_PRE;
    auto slot = [&](int r) -> double* { return ring + ((r - cstart) & (AS_ROWS - 1)) * AS_SLOT; };
    auto issue_row = [&](int r) {
        if (r <= r1 + 3) {
            const size_t rp = (size_t)wrap(r, D.ny) * nx;
            double* s = slot(r);
#pragma unroll
            for (int q = 0; q < 6; ++q) cp_async8(&s[q * 32 + lane], &U.f[q][rp + iw]);
            if (lane == 31) cp_async8(&s[12 * 32], &U.f[4][rp + iw_r]);
            if (r >= r0 - AS_PRE_FACE && r <= r1 + 1) {
#pragma unroll
                for (int q = 0; q < 6; ++q) cp_async8(&s[(6 + q) * 32 + lane], &w.f[q][rp + iw]);
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int r = 2; r < AS_ROWS - 1; ++r) issue_row(cstart + r);

    bool wild = false;  // this lane met a cell for the sweep of any cell
    int c = cstart;
    for (; c <= r1; ++c) {
        cp_async_wait<3>();  // rows up to c+3 have landed
        double ob[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const bool out_row = out_lane && c - 1 >= r0;
        const size_t g = (size_t)(c - 1) * nx + i;
        if (out_row) {
            if (base.f[0]) {
#pragma unroll
                for (int q = 0; q < 4; ++q) ob[q] = base.f[q][g];
            }
            if (base.f[4]) {
                ob[4] = base.f[4][g];
                ob[5] = base.f[5][g];
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            Prho[k] = Prho[k + 1]; Pvx[k] = Pvx[k + 1]; Pvy[k] = Pvy[k + 1];
            Pp[k] = Pp[k + 1]; Pbx[k] = Pbx[k + 1]; Pby[k] = Pby[k + 1];
        }
        {
            const double* s2 = slot(c + 2) + lane;
            const double bxf2 = s2[4 * 32];
            double bxr2 = __shfl_down_sync(0xffffffffu, bxf2, 1);
            if (lane == 31) bxr2 = slot(c + 2)[12 * 32];
            Pbx[3] = (bxf2 + bxr2) / 2.0;
            Pby[3] = (s2[5 * 32] + slot(c + 3)[5 * 32 + lane]) / 2.0;
            double rho = s2[0];
            Pp[3] = primitives_of<ANY>(rho, s2[32], s2[64], s2[96], Pbx[3], Pby[3], Pvx[3], Pvy[3]);
            Prho[3] = rho;
            if constexpr (!ANY) {
                const unsigned face = max((unsigned)high_word(bxf2) & 0x7fffffffu, (unsigned)high_word(s2[5 * 32]) & 0x7fffffffu);
                wild |= !ordinary(rho, Pvx[3], Pvy[3], Pp[3], Pbx[3], Pby[3]) || face >= kOrdinaryHigh;
            }
        }
        if (c < r0 - AS_PRE_FACE) {
            issue_row(c + AS_ROWS - 1);
            continue;
        }
        const double* w0 = slot(c) + 6 * 32 + lane;
        const double* w1 = slot(c + 1) + 6 * 32 + lane;
        auto up = [](double v) { return __shfl_up_sync(0xffffffffu, v, 1); };
        auto dn = [](double v) { return __shfl_down_sync(0xffffffffu, v, 1); };
        // ---- CORNER (i, c+1): Fx.bt is -eN of corner (i+1, c) and -eS of (i+1, c+1), Fy.bt is eE of (i, c+1) and
        //      eW of (i+1, c+1)
        double xbt, ybt;
        {
            const double wby = w1[5 * 32];
            const double cfa = (w1[4 * 32] - w0[4 * 32]) * idy + (up(wby) - wby) * idx;
            const double vxc = 0.25 * (Pvx[2] + up(Pvx[2]) + Pvx[1] + up(Pvx[1]));
            const double vyc = 0.25 * (Pvy[2] + up(Pvy[2]) + Pvy[1] + up(Pvy[1]));
            xbt = -dn(p0_prev + cfa * ct_weight(vyc, D.ct_mode, 1));
            p0_prev = cfa * ct_weight(vyc, D.ct_mode, 0);
            ybt = cfa * ct_weight(vxc, D.ct_mode, 0) + dn(cfa * ct_weight(vxc, D.ct_mode, 1));
        }
        // ---- XFACE: right face of (i, c), then row c's adjoints along x
        double ax[5] = {0.0, 0.0, 0.0, 0.0, 0.0}, xbn = 0.0;
        if (c >= r0 - 1 && c < r1) {
            FaceState L, R;
            int br = 0;
            auto recon = [&](double q, int k, double& hi, double& lo_right) {
                const double dl = q - up(q);
                const double dr = dn(dl);
                const double s = minmod<ANY>(dl, dr);
                hi = q + 0.5 * s;
                lo_right = dn(q - 0.5 * s);
                br |= minmod_branch(dl, dr) << (2 * k);
            };
            recon(Prho[1], 0, L.rho, R.rho);
            recon(Pvx[1], 1, L.vn, R.vn);
            recon(Pvy[1], 2, L.vt, R.vt);
            recon(Pp[1], 3, L.p, R.p);
            recon(Pby[1], 4, L.bt, R.bt);
            L.bn = R.bn = dn(slot(c)[4 * 32 + lane]);
            const FluxAdj f = {(dn(w0[0]) - w0[0]) * idx, (dn(w0[32]) - w0[32]) * idx, (dn(w0[64]) - w0[64]) * idx,
                               (dn(w0[96]) - w0[96]) * idx, xbt};
            FaceState aL, aR;
            hll_vjp<ANY>(L, R, f, aL, aR);
            xbn = aL.bn + aR.bn;
            auto gather = [&](int k, double hi, double lo_right) {
                const double lo = up(lo_right);
                const double as = 0.5 * (hi - lo);  // adjoint of the limited slope
                const int b = (br >> (2 * k)) & 3;
                const double m = b == 1 ? as : 0.0, n = b == 2 ? as : 0.0;
                ax[k] = (hi + lo) + (m - n) + (up(n) - dn(m));
            };
            gather(0, aL.rho, aR.rho);
            gather(1, aL.vn, aR.vn);
            gather(2, aL.vt, aR.vt);
            gather(3, aL.p, aR.p);
            gather(4, aL.bt, aR.bt);
        }
        // ---- YFACE: top face of (i, c), then the adjoints of rows c-1 .. c+1 along y
        double ybn;
        double a[6];  // row c-1, complete
        {
            FaceState Dn, Up;
            auto recon = [](const double (&q)[4], double& hi, double& lo_up) {
                hi = recon_hi<ANY>(q[0], q[1], q[2]);
                lo_up = recon_lo<ANY>(q[1], q[2], q[3]);
            };
            recon(Prho, Dn.rho, Up.rho);
            recon(Pvx, Dn.vt, Up.vt);
            recon(Pvy, Dn.vn, Up.vn);
            recon(Pp, Dn.p, Up.p);
            recon(Pbx, Dn.bt, Up.bt);
            Dn.bn = Up.bn = slot(c + 1)[5 * 32 + lane];
            const FluxAdj f = {(w1[0] - w0[0]) * idy, (w1[64] - w0[64]) * idy, (w1[32] - w0[32]) * idy,
                               (w1[96] - w0[96]) * idy, ybt};
            FaceState aD, aU;
            hll_vjp<ANY>(Dn, Up, f, aD, aU);
            ybn = aD.bn + aU.bn;
            auto gather = [&](int k, const double (&q)[4], double hi, double lo_up) {
                const double as = 0.5 * (hi - Lo(k));
                const int b = minmod_branch(q[1] - q[0], q[2] - q[1]);
                const double m = b == 1 ? as : 0.0, n = b == 2 ? as : 0.0;
                a[k] = Acc[k] - m;
                Acc[k] = hi + Half(k) + (m - n);
                Lo(k) = lo_up;
                Half(k) = lo_up + n;
            };
            gather(0, Prho, aD.rho, aU.rho);
            gather(1, Pvx, aD.vt, aU.vt);
            gather(2, Pvy, aD.vn, aU.vn);
            gather(3, Pp, aD.p, aU.p);
            gather(4, Pbx, aD.bt, aU.bt);
            a[5] = Acc[5];
#pragma unroll
            for (int k = 0; k < 4; ++k) Acc[k] += ax[k];
            Acc[5] = ax[4];
        }
        const bool stop = !ANY && __any_sync(0xffffffffu, wild);
        // ---- OUT row c-1: primitive -> conserved (Grid.hpp:100-136): vx = mx/rho, vy = my/rho (density as stored),
        //      rho_f = max(rho, floor), p = max((gamma-1)(E - rho_f v^2/2 - |Bc|^2/2), floor)
        {
            const double* s = slot(c - 1) + lane;
            const double rho = s[0], E = s[96];
            const double vx = Pvx[0], vy = Pvy[0], rho_f = Prho[0], bxc = Pbx[0], byc = Pby[0];
            const double eint = E - 0.5 * rho_f * (vx * vx + vy * vy) - (bxc * bxc + byc * byc) / 2;
            const double gm1ap = (kGammaGas - 1) * eint < kPFloor ? 0.0 : (kGammaGas - 1) * a[3];
            const double arho_f = a[0] - gm1ap * 0.5 * (vx * vx + vy * vy);
            const double avx = a[1] - gm1ap * rho_f * vx;
            const double avy = a[2] - gm1ap * rho_f * vy;
            const double abxc = a[4] - gm1ap * bxc;
            const double abyc = a[5] - gm1ap * byc;
            const double ir = ANY ? 1.0 / rho : rcp_nr(rho);
            double arho = -(avx * vx + avy * vy) * ir;
            if (!(rho < kRhoFloor)) arho += arho_f;
            // bxc(i) = (bxf(i) + bxf(i+1))/2, and bxf(i) is the normal field of x face i-1
            const double abx = 0.5 * (abxc + up(abxc)) + up(xbn1);
            const double aby = 0.5 * (abyc + abyc_prev) + ybn2;
            if (out_row && !stop) {
                out.f[0][g] = ob[0] + scale * arho;
                out.f[1][g] = ob[1] + scale * (avx * ir);
                out.f[2][g] = ob[2] + scale * (avy * ir);
                out.f[3][g] = ob[3] + scale * gm1ap;
                out.f[4][g] = ob[4] + scale * abx;
                out.f[5][g] = ob[5] + scale * aby;
            }
            abyc_prev = abyc;
        }
        ybn2 = ybn1;
        ybn1 = ybn;
        xbn1 = xbn;
        issue_row(c + AS_ROWS - 1);  // into the slot of row c-1, no longer read
        if (stop) break;
    }
    cp_async_wait<0>();  // leave no copy in flight into the ring
    return c;
}

static __global__ void __launch_bounds__(32, 8)
k_adj_rate_sweep(Domain D, CPlanes U, CPlanes w, CPlanes base, double scale, Planes out, SweepGeom G) {
#if defined(__CUDA_ARCH__)
    extern __shared__ __align__(16) double as_ring_mem[];
#else
    static double as_ring_mem[AS_ROWS * AS_SLOT + AS_CARRY];
#endif
    const int sx = blockIdx.x % G.strips_x, sy = blockIdx.x / G.strips_x;
    const int r0 = sy * G.seg_h, r1 = min(r0 + G.seg_h, D.ny);
    if (r0 >= r1) return;
    const int c = adj_rate_rows<false>(D, U, w, base, scale, out, sx, r0, r1, as_ring_mem);
    if (c > r1) return;
    __syncwarp();
    adj_rate_rows<true>(D, U, w, base, scale, out, sx, max(c - 1, r0), r1, as_ring_mem);  // (inlined: no stack frame)
}

}  // namespace mhd

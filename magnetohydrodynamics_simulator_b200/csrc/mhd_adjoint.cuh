// Discrete adjoint of the ARS(2,2,2) IMEX step (FP64): hand-written vector-Jacobian products of
// the explicit rate (MUSCL-minmod reconstruction, HLL flux, upwind CT, flux divergence) and the
// linear stencils of the resistive term.
//
// Notation. F(U) is the explicit rate of solvers.hpp:393-402 (six planes). For a given adjoint
// w of the rate, F'(U)^T w is one sweep without atomics (mhd_adjoint_sweep.cuh): per face the flux
// adjoint from w (divergence and CT transposed) and the HLL VJP below, per cell the gather of the
// reconstruction adjoints (minmod branches recomputed) and the primitive -> conserved VJP.
// The branches of minmod, of the HLL wave-speed min/max and of the CT corner test are those of
// the forward evaluation (the derivative of a selection is that of the selected operand); floors
// contribute zero derivative where they are active.
//
// The resistive operators are symmetric: with Jz the corner current of face B
// (solvers.hpp:450-461 without eta) and C the face rate of a corner field (solvers.hpp:478-486),
// Jz^T = -C and C^T = -Jz, so the explicit rate eta*C*Jz and the implicit rate
// eta*C*(I - alpha L)^-1*Jz are both self-adjoint (Jz*C = L, the corner Laplacian of the matrix).
#pragma once

#include "mhd_kernels.cuh"

namespace mhd {

// ------------------------------------------------------------------------------------------
// Per-face vector-Jacobian product of the HLL flux (HLL.hpp:31-218).
//
// In components normal (n) and tangential (t) to the face both directions read the same. With the clamped wave
// speeds sL <= 0 <= sR of the forward (hll), i = 1/(sR - sL), a = sR i, b = sL i and for a flux adjoint f
//   F = a F_L - b F_R + a sL (U_R - U_L)
//   J_L^T f = a (F'_L - sL U'_L)^T f,   J_R^T f = -b (F'_R - sR U'_R)^T f   at fixed speeds,
//   dF.f / dsR = i b (X - sL Y),        dF.f / dsL = -i a (X - sR Y),      X = f.(F_R - F_L), Y = f.(U_R - U_L),
// so neither F nor any scaled copy of f is formed. A clamped speed has no derivative; straight-line code, as a
// branch to the supersonic cases costs a warp all of them. (Flux, average and their derivatives component by
// component, with those branches: 169 us a launch of the sweep at 1024^2 for 113.)

struct FaceState {  // primitives, or their adjoints, in face components
    double rho, vn, vt, p, bn, bt;
};
struct FluxAdj {
    double rho, mn, mt, E, bt;
};

// fast_speed with the two reciprocals its derivative needs.
struct FastSpeed {
    double c;   // sqrt(X / rho), X = S + sqrt(D)
    double iz;  // 1 / sqrt(X rho)
    double id;  // 1 / sqrt(D), 0 where D counts as 0
    double S;
};
__device__ __forceinline__ FastSpeed fast_speed_parts(const FaceState& w) {
    const double b2 = w.bn * w.bn + w.bt * w.bt;
    const double gp = kGammaGas * w.p;
    FastSpeed f;
    f.S = 0.5 * (gp + b2);
    const double D = fma(f.S, f.S, -(gp * (w.bn * w.bn)));
    const bool pos = high_word(D) > 0x03f00000;
    const double root = sqrt_nr(D), inv = rsqrt_nr(D);
    const double X = f.S + (pos ? root : 0.0);
    f.id = pos ? inv : 0.0;
    f.iz = rsqrt_nr(X * w.rho);
    f.c = X * f.iz;
    return f;
}
// Adjoint ac of the speed: into a.
__device__ __forceinline__ void fast_speed_vjp(const FaceState& w, const FastSpeed& f, double ac, FaceState& a) {
    const double h = 0.5 * ac * f.iz;  // adjoint of X
    const double k = h * f.id;
    const double aS = fma(k, f.S, h);
    a.rho -= h * (f.c * f.c);
    a.p += (0.5 * kGammaGas) * fma(-k, w.bn * w.bn, aS);
    a.bn += w.bn * fma(-k, kGammaGas * w.p, aS);
    a.bt += w.bt * aS;
}

// The speed and its VJP with the quotients first, as the reference forms them: for cells of any size.
__device__ __forceinline__ double fast_speed_any(const FaceState& w) {
    const double ir = 1.0 / w.rho;
    const double a2 = kGammaGas * w.p * ir;
    const double sum = (w.bn * w.bn + w.bt * w.bt) * ir + a2;
    const double term = sum * sum - 4.0 * a2 * (w.bn * w.bn * ir);
    return sqrt(0.5 * (sum + sqrt(term > 0.0 ? term : 0.0)));
}
__device__ __forceinline__ void fast_speed_any_vjp(const FaceState& w, double ac, FaceState& a) {
    const double b2 = w.bn * w.bn + w.bt * w.bt;
    const double ir = 1.0 / w.rho;
    const double a2 = kGammaGas * w.p * ir, n2 = w.bn * w.bn * ir;
    const double sum = b2 * ir + a2;
    const double term = sum * sum - 4.0 * a2 * n2;
    const double sq = term > 0.0 ? sqrt(term) : 0.0;
    const double c = sqrt(0.5 * (sum + sq));
    const double h = c > 0.0 ? 0.25 * ac / c : 0.0;           // adjoint of sum + sq
    const double t = sq > 0.0 ? 0.5 * h / sq : 0.0;           // of term
    const double asum = h + 2.0 * t * sum, aa2 = asum - 4.0 * n2 * t, an2 = -4.0 * a2 * t;
    a.rho -= (aa2 * kGammaGas * w.p + asum * b2 + an2 * (w.bn * w.bn)) * ir * ir;
    a.p += aa2 * kGammaGas * ir;
    a.bn += 2.0 * w.bn * (asum + an2) * ir;
    a.bt += 2.0 * w.bt * asum * ir;
}

// One side's f.F and f.U (less the terms in bn alone, which cancel between the sides), and what the VJP shares.
struct FaceSide {
    double K, Mn, Mt, G, hp, phi, ups;
};
__device__ __forceinline__ FaceSide face_side(const FaceState& w, const FluxAdj& f) {
    FaceSide s;
    const double v2 = fma(w.vn, w.vn, w.vt * w.vt), hbt2 = 0.5 * (w.bt * w.bt);
    s.K = fma(0.5 * f.E, v2, fma(f.mt, w.vt, fma(f.mn, w.vn, f.rho)));
    s.Mn = fma(f.E, w.vn, f.mn);
    s.Mt = fma(f.E, w.vt, f.mt);
    s.G = fma(f.E, w.bt, f.bt);
    s.hp = (kGammaGas * kInvGm1) * w.p * f.E;
    const double rK = w.rho * s.K;
    const double eb = fma(w.vn, w.bt, -(w.vt * w.bn));
    s.phi = fma(w.vn, rK + s.hp, fma(eb, s.G, fma(f.mn, w.p + hbt2, -(f.mt * (w.bn * w.bt)))));
    s.ups = fma(f.E, fma(w.p, kInvGm1, hbt2), fma(f.bt, w.bt, rK));
    return s;
}
// wt (F' - sp U')^T f
__device__ __forceinline__ FaceState face_side_vjp(const FaceState& w, const FluxAdj& f, const FaceSide& s, double sp,
                                                   double wt) {
    const double q = w.vn - sp;
    FaceState a;
    a.rho = wt * (q * s.K);
    a.vn = wt * fma(w.rho, fma(q, s.Mn, s.K), fma(w.bt, s.G, s.hp));
    a.vt = wt * fma(q * w.rho, s.Mt, -(w.bn * s.G));
    a.p = wt * fma(q * kInvGm1, f.E, s.Mn);
    a.bn = wt * fma(w.bn, fma(q, f.E, -s.Mn), -fma(w.bt, s.Mt, f.bt * w.vt));
    a.bt = wt * fma(q, s.G, fma(w.bt, s.Mn, -(w.bn * s.Mt)));
    return a;
}

// L, R: lower and upper state; f: the flux adjoint. The normal field enters both states: its adjoint is the sum of
// both sides' bn. Selections (HLL.hpp:139-141: std::min, std::max) as in the forward. ANY: for cells of any size, with
// the one-sided cases as the forward has them there.
template <bool ANY>
__device__ __forceinline__ void hll_vjp(const FaceState& L, const FaceState& R, const FluxAdj& f, FaceState& aL,
                                        FaceState& aR) {
    FastSpeed cL, cR;
    if constexpr (ANY) {
        cL.c = fast_speed_any(L);
        cR.c = fast_speed_any(R);
    } else {
        cL = fast_speed_parts(L);
        cR = fast_speed_parts(R);
    }
    const FaceSide l = face_side(L, f), r = face_side(R, f);
    const double mnL = L.vn - cL.c, mnR = R.vn - cR.c, mxL = L.vn + cL.c, mxR = R.vn + cR.c;
    const bool lowR = mnR < mnL, highR = mxL < mxR;
    const double mn = lowR ? mnR : mnL, mx = highR ? mxR : mxL;
    if constexpr (ANY) {
        if (mn >= 0.0) {
            aL = face_side_vjp(L, f, l, 0.0, 1.0);
            aR = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            return;
        }
        if (mx <= 0.0) {
            aL = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            aR = face_side_vjp(R, f, r, 0.0, 1.0);
            return;
        }
    }
    const double sL = mn < 0.0 ? mn : 0.0, sR = mx > 0.0 ? mx : 0.0;
    const double inv = ANY ? 1.0 / (sR - sL) : rcp_nr(sR - sL);
    const double a = sR * inv, b = sL * inv;
    const double X = r.phi - l.phi, Y = r.ups - l.ups;
    const double asR = mx > 0.0 ? (inv * b) * fma(-sL, Y, X) : 0.0;
    const double asL = mn < 0.0 ? -(inv * a) * fma(-sR, Y, X) : 0.0;
    aL = face_side_vjp(L, f, l, sL, a);
    aR = face_side_vjp(R, f, r, sR, -b);
    const double lL = lowR ? 0.0 : asL, lR = lowR ? asL : 0.0, hL = highR ? 0.0 : asR, hR = highR ? asR : 0.0;
    aL.vn += lL + hL;
    aR.vn += lR + hR;
    if constexpr (ANY) {
        fast_speed_any_vjp(L, hL - lL, aL);
        fast_speed_any_vjp(R, hR - lR, aR);
    } else {
        fast_speed_vjp(L, cL, hL - lL, aL);
        fast_speed_vjp(R, cR, hR - lR, aR);
    }
}

// Which operand minmod(a, b) returned (MUSCL.hpp:11-17): 1 = a, 2 = b, 0 = none.
__device__ __forceinline__ int minmod_branch(double a, double b) {
    if (a * b > 0.0) return (fabs(a) < fabs(b)) ? 1 : 2;
    return 0;
}

// Weight of the north (sel = 0) or south (sel = 1) face value in the corner field for a corner
// velocity v (solvers.hpp:314-340): the corner field is (ezx + ezy) / 2.
__device__ __forceinline__ double ct_weight(double v, int mode, int second) {
    if (ct_average(v, mode)) return 0.25;
    // upwind: v > 0 takes the second operand (eS for ezy, eW for ezx)
    return ((v > 0.0) == (second != 0)) ? 0.5 : 0.0;
}

// ------------------------------------------------------------------------------------------
// Linear stencils of the resistive term and plane algebra.

// Each kernel below is one pass that also forms one term of dL/deta: a thread's cells in row order, a block's
// sum in partial[block] (launch shape adj_grid). They take the place of a corner current, a curl, a dot product
// and a plane combination at a time: at 1024^2 those were 9-11 us each, most of it launch and tail.

struct Planes6C {
    const double* f[6];
};

// Jz(bx, by) at corner (i, j); im, jm: the wrapped column to the left, the row below (offsets).
__device__ __forceinline__ double adj_jz(const double* __restrict__ bx, const double* __restrict__ by, size_t row, size_t rowm,
                                         int i, int im, double idx, double idy) {
    return (by[row + i] - by[row + im]) * idx - (bx[row + i] - bx[rowm + i]) * idy;
}

// Where a resistive term with field B2 = B + t C(x) (x: the solution of the term's solve) meets the adjoint
// lam: c2 = Jz(B) + t L x = Jz(B2); fb = s C(Jz(lam)); partial sums of Jz(lam) . c2. FIELD: also B2 itself.
template <bool FIELD>
static __global__ void __launch_bounds__(256)
k_adj_resistive(Domain D, const double* __restrict__ lbx, const double* __restrict__ lby, const double* __restrict__ bx,
                const double* __restrict__ by, const double* __restrict__ x, double t, double s, double* __restrict__ c2,
                double* __restrict__ fbx, double* __restrict__ fby, double* __restrict__ b2x, double* __restrict__ b2y,
                double* __restrict__ partial) {
    __shared__ double red[64];
    const int nx = D.nx, ny = D.ny;
    const double idx = 1.0 / D.dx, idy = 1.0 / D.dy;
    double acc[1] = {0.0};
    for (int j = blockIdx.y; j < ny; j += gridDim.y)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nx; i += gridDim.x * blockDim.x) {
        const int im = wrap(i - 1, nx), ip = wrap(i + 1, nx);
        const size_t row = (size_t)j * nx, rowm = (size_t)wrap(j - 1, ny) * nx, rowp = (size_t)wrap(j + 1, ny) * nx;
        const size_t g = row + i;
        const double e = adj_jz(lbx, lby, row, rowm, i, im, idx, idy);
        const double er = adj_jz(lbx, lby, row, rowm, ip, i, idx, idy);
        const double eu = adj_jz(lbx, lby, rowp, row, i, im, idx, idy);
        const double xc = x[g], xr = x[row + ip], xu = x[rowp + i];
        double v = adj_jz(bx, by, row, rowm, i, im, idx, idy);
        const double lap = (xr + x[row + im] - 2.0 * xc) * (idx * idx) + (xu + x[rowm + i] - 2.0 * xc) * (idy * idy);
        v += t * lap;
        c2[g] = v;
        fbx[g] = s * (-(eu - e) * idy);
        fby[g] = s * ((er - e) * idx);
        if (FIELD) {
            b2x[g] = t * (-(xu - xc) * idy) + bx[g];
            b2y[g] = t * ((xr - xc) * idx) + by[g];
        }
        acc[0] += e * v;
    }
    block_sum<256, 1>(acc, red);
    if (threadIdx.x == 0) partial[blockIdx.y * gridDim.x + blockIdx.x] = acc[0];
}

// lam_B += fb + eta C(y), and the partial sums of y . c2.
static __global__ void __launch_bounds__(256)
k_adj_implicit(Domain D, double eta, const double* __restrict__ y, const double* __restrict__ c2,
               const double* __restrict__ fbx, const double* __restrict__ fby, double* __restrict__ lbx,
               double* __restrict__ lby, double* __restrict__ partial) {
    __shared__ double red[64];
    const int nx = D.nx, ny = D.ny;
    const double idx = 1.0 / D.dx, idy = 1.0 / D.dy;
    double acc[1] = {0.0};
    for (int j = blockIdx.y; j < ny; j += gridDim.y)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nx; i += gridDim.x * blockDim.x) {
        const size_t row = (size_t)j * nx, g = row + i;
        const double yc = y[g], yr = y[row + wrap(i + 1, nx)], yu = y[(size_t)wrap(j + 1, ny) * nx + i];
        lbx[g] = eta * (-(yu - yc) * idy) + lbx[g] + fbx[g];
        lby[g] = eta * ((yr - yc) * idx) + lby[g] + fby[g];
        acc[0] += yc * c2[g];
    }
    block_sum<256, 1>(acc, red);
    if (threadIdx.x == 0) partial[blockIdx.y * gridDim.x + blockIdx.x] = acc[0];
}

// The end of the adjoint step: lamT_B += eta C(y), the explicit-rate adjoint of stage 1 w = cd lam + cg lamT,
// lam += lamT, and the partial sums of y . c2.
static __global__ void __launch_bounds__(256)
k_adj_close(Domain D, double eta, const double* __restrict__ y, const double* __restrict__ c2, double cd, double cg,
            Planes lam, Planes6C lamT, Planes w, double* __restrict__ partial) {
    __shared__ double red[64];
    const int nx = D.nx, ny = D.ny;
    const double idx = 1.0 / D.dx, idy = 1.0 / D.dy;
    double acc[1] = {0.0};
    for (int j = blockIdx.y; j < ny; j += gridDim.y)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nx; i += gridDim.x * blockDim.x) {
        const size_t row = (size_t)j * nx, g = row + i;
        const double yc = y[g], yr = y[row + wrap(i + 1, nx)], yu = y[(size_t)wrap(j + 1, ny) * nx + i];
        double t[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) t[k] = lamT.f[k][g];
        t[4] = eta * (-(yu - yc) * idy) + t[4];
        t[5] = eta * ((yr - yc) * idx) + t[5];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const double a = lam.f[k][g];
            w.f[k][g] = cd * a + cg * t[k];
            lam.f[k][g] = a + t[k];
        }
        acc[0] += yc * c2[g];
    }
    block_sum<256, 1>(acc, red);
    if (threadIdx.x == 0) partial[blockIdx.y * gridDim.x + blockIdx.x] = acc[0];
}

// *acc += sum_k scale[k] * (sum of the kth nblocks partials), one warp a term, in a fixed order.
struct DotScales {
    double s[4];
};
static __global__ void __launch_bounds__(128)
k_adj_dot_final(const double* __restrict__ partial, int nblocks, DotScales scale, double* acc) {
    __shared__ double term[4];
    const int k = threadIdx.x >> 5, l = threadIdx.x & 31;
    double v = 0.0;
#pragma unroll 8
    for (int b = l; b < nblocks; b += 32) v += partial[(size_t)k * nblocks + b];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (l == 0) term[k] = scale.s[k] * v;
    __syncthreads();
    if (threadIdx.x == 0) *acc += term[0] + term[1] + term[2] + term[3];
}

}  // namespace mhd

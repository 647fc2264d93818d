// Per-cell and per-face FP64 physics of the reference solver, as device functions.
//
// The same expressions as the reference's, to rounding: quotients and roots by the approximations below, the fast
// speed with one quotient under the root, the HLL cases through clamped wave speeds, and FMA contraction. Cells beyond
// ordinary size keep the reference's own forms (ANY). References are to RikibabManos/Magnetohydrodynamics_Simulator.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

namespace mhd {

constexpr double kGammaGas = 5.0 / 3.0;  // Grid.hpp:104, HLL.hpp:31,62,85,108, diagnostics.hpp:48
// p / (gamma - 1) of the ideal-gas energy (HLL.hpp:43, 69, 92) as a product with the folded
// reciprocal: what the reference's -ffast-math build computes (CMakeLists.txt:21), within 1 ulp of
// the quotient, and one FP64 multiply instead of a division sequence.
constexpr double kInvGm1 = 1.0 / (kGammaGas - 1.0);
constexpr double kRhoFloor = 1e-8;       // Grid.hpp:115, diagnostics.hpp:64
constexpr double kPFloor = 1e-8;         // Grid.hpp:124, diagnostics.hpp:65

struct Prim {
    double rho, vx, vy, p, bx, by;
};

struct Flux {
    double rho, mx, my, E, bt;  // bt: the tangential induction flux (F^By in x, F^Bx in y)
};

// Reciprocal and square root as straight-line code: the hardware's approximation (relative error below
// 2^-19; PTX rcp/rsqrt.approx.ftz.f64) and one third-order step (Householder 1970) for 1/a and 1/sqrt(a), one
// Goldschmidt step and one residual correction (Markstein 1990) for sqrt(a). Largest error found over 2^24 arguments of
// 2^-300 .. 2^300 (a GPU test asserts these): 0.507 ulp for 1/a, 0.509 for sqrt(a), 1.00 for 1/sqrt(a), 1.94 for sqrt(X/r). Their
// arguments are normal numbers, positive for the root (0, infinities and subnormals give NaN). The library's
// division and root branch to a slow path, and each such branch ends a basic block: with the eight roots and
// seven reciprocals of a cell's two faces inline, both faces' arithmetic interleaves.
__device__ __forceinline__ double rcp_nr(double a) {
#if defined(__CUDA_ARCH__)
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-a, y, 1.0);
    return fma(y, fma(e, e, e), y);
#else
    return 1.0 / a;
#endif
}
__device__ __forceinline__ double sqrt_nr(double a) {
#if defined(__CUDA_ARCH__)
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double g = a * y, h = 0.5 * y;
    const double g1 = fma(g, fma(-g, h, 0.5), g);
    return fma(fma(-g1, g1, a), h, g1);
#else
    return sqrt(a);
#endif
}

// 1 / sqrt(z), z > 0: one third-order step.
__device__ __forceinline__ double rsqrt_nr(double z) {
#if defined(__CUDA_ARCH__)
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(z));
    const double e = fma(-(z * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
#else
    return 1.0 / sqrt(z);
#endif
}

// X * rsqrt(X * r) = sqrt(X / r) for X, r > 0: one reciprocal root instead of a reciprocal and a root.
__device__ __forceinline__ double sqrt_quotient(double X, double r) {
#if defined(__CUDA_ARCH__)
    return X * rsqrt_nr(X * r);
#else
    return sqrt(X / r);
#endif
}

// High word of a double, for tests of sign and magnitude by integer instructions.
__device__ __forceinline__ int high_word(double v) {
#if defined(__CUDA_ARCH__)
    return __double2hiint(v);
#else
    long long b;
    memcpy(&b, &v, sizeof(b));
    return (int)(b >> 32);
#endif
}

// std::min / std::max semantics (b < a ? b : a), not fmin/fmax.
__device__ __forceinline__ double smin(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double smax(double a, double b) { return (a < b) ? b : a; }

// MUSCL.hpp:11-17. The test a * b > 0 by the sign bits: an integer instruction for a product and a
// comparison of the FP64 pipe. (Where it differs -- a zero, a product that underflows -- the smaller operand
// is below 1e-154.) ANY: the product, for which a NaN makes the slope 0.
template <bool ANY = false>
__device__ __forceinline__ double minmod(double a, double b) {
#if defined(__CUDA_ARCH__)
    if constexpr (!ANY) {
        const double s = (fabs(a) < fabs(b)) ? a : b;
        // (the high word decides: cleared, what is left of s is below 1e-313)
        return __hiloint2double((__double2hiint(a) ^ __double2hiint(b)) >= 0 ? __double2hiint(s) : 0, __double2loint(s));
    }
#endif
    if (a * b > 0.0) return (fabs(a) < fabs(b)) ? a : b;
    return 0.0;
}

// MUSCL.hpp:26-47, lower (c - s/2) face value of a cell from (left, centre, right)
template <bool ANY = false>
__device__ __forceinline__ double recon_lo(double fm, double f0, double fp) {
    return f0 - 0.5 * minmod<ANY>(f0 - fm, fp - f0);
}
// upper (c + s/2) face value
template <bool ANY = false>
__device__ __forceinline__ double recon_hi(double fm, double f0, double fp) {
    return f0 + 0.5 * minmod<ANY>(f0 - fm, fp - f0);
}

// The straight-line forms (rcp_nr, sqrt_nr and what is built on them) are for values of ordinary size: no products
// that overflow, no arguments outside the approximations' range. A cell within these limits cannot take them out of
// it; zero densities, infinities, NaN and values beyond 2^100 (velocity, field) or 2^200 (density, pressure) take the
// operators' division and root and the reference's own selections instead (ANY).
constexpr unsigned kOrdinaryHigh = (1023u + 200u) << 20;  // high word of 2^200

__device__ __forceinline__ bool ordinary(double rho, double vx, double vy, double p, double bx, double by) {
    // none of the four is negative, except a NaN, whose high word is above every number's either way
    const unsigned a = max((unsigned)high_word(rho), (unsigned)high_word(p));
    const unsigned b = max((unsigned)high_word(vx * vx + vy * vy), (unsigned)high_word(bx * bx + by * by));
    return max(a, b) < kOrdinaryHigh;
}

// Grid.hpp:100-136 computePrimitives for one cell. `rho` is replaced by the floored density;
// velocities divide by the density as stored (before the floor), as the reference does.
// Returns the (floored) pressure.
template <bool ANY>
__device__ __forceinline__ double primitives_of(double& rho, double mx, double my, double E,
                                                double bxc, double byc, double& vx, double& vy) {
    // one reciprocal instead of two divisions (<= 1 ulp from m/rho; the reference's fast-math
    // build is free to do the same)
    const double ir = ANY ? 1.0 / rho : rcp_nr(rho);
    vx = mx * ir;
    vy = my * ir;
    if (rho < kRhoFloor) rho = kRhoFloor;
    const double kin = 0.5 * rho * (vx * vx + vy * vy);
    const double mag = (bxc * bxc + byc * byc) / 2;
    const double eint = E - kin - mag;
    double p = (kGammaGas - 1) * eint;
    if (p < kPFloor) p = kPFloor;
    return p;
}
// ... of any cell
__device__ __forceinline__ double primitives(double& rho, double mx, double my, double E,
                                             double bxc, double byc, double& vx, double& vy) {
    const double stored = rho;
    double p = primitives_of<false>(rho, mx, my, E, bxc, byc, vx, vy);
    if (!ordinary(rho, vx, vy, p, bxc, byc)) {
        rho = stored;
        p = primitives_of<true>(rho, mx, my, E, bxc, byc, vx, vy);
    }
    return p;
}

// HLL.hpp:107-122 fast magnetosonic speed, c^2 = (s + sqrt(s^2 - 4 a^2 n^2)) / 2 with s = (gamma p + B^2) / rho,
// a^2 = gamma p / rho, n^2 = Bn^2 / rho. All terms share 1 / rho, so it is taken once, under the root:
// c = sqrt(X / rho), X = S + sqrt(S^2 - gamma p Bn^2), S = (gamma p + B^2) / 2.
// ANY: the quotients first, as the reference forms them (p and B^2 may then be beyond 1e154).
template <bool ANY = false>
__device__ __forceinline__ double fast_speed(const Prim& w, double bn) {
    const double b2 = w.bx * w.bx + w.by * w.by;
    if constexpr (ANY) {
        const double ir = 1.0 / w.rho;
        const double a2 = kGammaGas * w.p * ir;
        const double sum = b2 * ir + a2;
        const double term = sum * sum - 4.0 * a2 * (bn * bn * ir);
        return sqrt(0.5 * (sum + sqrt(term > 0.0 ? term : 0.0)));
    }
    const double gp = kGammaGas * w.p;
    const double S = 0.5 * (gp + b2);
    const double D = fma(S, S, -(gp * (bn * bn)));
    const double root = sqrt_nr(D);
    // D <= 0 up to rounding, or below 2^-960, counts as 0 (S > 0: the pressure is floored)
    return sqrt_quotient(S + (high_word(D) > 0x03f00000 ? root : 0.0), w.rho);
}

// HLL.hpp:61-104 physical flux normal to direction DIR (0 = x, 1 = y), together with the
// conserved energy of HLL.hpp:31-47 (needed by the HLL average).
template <int DIR>
__device__ __forceinline__ Flux phys_flux(const Prim& w) {
    const double v2 = w.vx * w.vx + w.vy * w.vy;
    const double b2 = w.bx * w.bx + w.by * w.by;
    const double pt = w.p + 0.5 * b2;
    const double vb = w.vx * w.bx + w.vy * w.by;
    const double E = w.p * kInvGm1 + 0.5 * (w.rho * v2 + b2);
    Flux F;
    if (DIR == 0) {
        F.rho = w.rho * w.vx;
        F.mx = w.rho * w.vx * w.vx + pt - w.bx * w.bx;
        F.my = w.rho * w.vx * w.vy - w.bx * w.by;
        F.E = (E + pt) * w.vx - w.bx * vb;
        F.bt = w.vx * w.by - w.vy * w.bx;
    } else {
        F.rho = w.rho * w.vy;
        F.my = w.rho * w.vy * w.vy + pt - w.by * w.by;
        F.mx = w.rho * w.vx * w.vy - w.bx * w.by;
        F.E = (E + pt) * w.vy - w.by * vb;
        F.bt = w.vy * w.bx - w.vx * w.by;
    }
    return F;
}

// HLL.hpp:31-47 ConservedState::fromPrimitive (the components the HLL average uses).
template <int DIR>
__device__ __forceinline__ Flux conserved(const Prim& w) {
    Flux U;
    U.rho = w.rho;
    U.mx = w.rho * w.vx;
    U.my = w.rho * w.vy;
    const double v2 = w.vx * w.vx + w.vy * w.vy;
    const double b2 = w.bx * w.bx + w.by * w.by;
    U.E = w.p * kInvGm1 + 0.5 * (w.rho * v2 + b2);  // as phys_flux forms it: one value for both
    U.bt = (DIR == 0) ? w.by : w.bx;
    return U;
}

// HLL.hpp:126-172 (DIR = 0) and :177-218 (DIR = 1). L is the lower/left state. The reference takes F_L where
// sL >= 0, F_R where sR <= 0 and the average between; with sL and sR clamped to the two sides of 0 the
// average's own weights give those cases, to rounding: straight-line code without selects per component.
// ANY: the cases themselves (the side that does not count may be infinite or NaN).
template <int DIR, bool ANY = false>
__device__ __forceinline__ Flux hll(const Prim& L, const Prim& R) {
    const Flux FL = phys_flux<DIR>(L);
    const Flux FR = phys_flux<DIR>(R);
    const double cL = fast_speed<ANY>(L, DIR == 0 ? L.bx : L.by);
    const double cR = fast_speed<ANY>(R, DIR == 0 ? R.bx : R.by);
    const double vL = DIR == 0 ? L.vx : L.vy;
    const double vR = DIR == 0 ? R.vx : R.vy;
    const double mn = smin(vL - cL, vR - cR), mx = smax(vL + cL, vR + cR);
    if constexpr (ANY) {
        if (mn >= 0) return FL;
        if (mx <= 0) return FR;
        const Flux UL = conserved<DIR>(L);
        const Flux UR = conserved<DIR>(R);
        const double inv = 1.0 / (mx - mn), sLR = mn * mx;
        auto avg = [&](double fl, double fr, double ul, double ur) { return (mx * fl - mn * fr + sLR * (ur - ul)) * inv; };
        return {avg(FL.rho, FR.rho, UL.rho, UR.rho), avg(FL.mx, FR.mx, UL.mx, UR.mx), avg(FL.my, FR.my, UL.my, UR.my),
                avg(FL.E, FR.E, UL.E, UR.E), avg(FL.bt, FR.bt, UL.bt, UR.bt)};
    }
    const double sL = high_word(mn) < 0 ? mn : 0.0, sR = high_word(mx) < 0 ? 0.0 : mx;
    const Flux UL = conserved<DIR>(L);
    const Flux UR = conserved<DIR>(R);
    const double inv = rcp_nr(sR - sL);
    const double a = sR * inv, b = sL * inv, c = sR * b;
    auto avg = [&](double fl, double fr, double ul, double ur) { return fma(c, ur - ul, fma(a, fl, -(b * fr))); };
    Flux F;
    F.rho = avg(FL.rho, FR.rho, UL.rho, UR.rho);
    F.mx = avg(FL.mx, FR.mx, UL.mx, UR.mx);
    F.my = avg(FL.my, FR.my, UL.my, UR.my);
    F.E = avg(FL.E, FR.E, UL.E, UR.E);
    F.bt = avg(FL.bt, FR.bt, UL.bt, UR.bt);
    return F;
}

// solvers.hpp:326,333 corner-velocity test. GCC resolves the unqualified abs(double) there to
// int abs(int), so the reference averages whenever (int)v == 0, i.e. |v| < 1 (and, as x86
// converts NaN / out-of-range values to INT_MIN, also for those). mode 1 is the literal
// |v| < 1e-12 test, for physics studies.
__device__ __forceinline__ bool ct_average(double v, int mode) {
    if (mode == 1) return fabs(v) < 1e-12;
    const unsigned a = (unsigned)high_word(v) & 0x7fffffffu;  // |v| >= 1 and |v| < 2^31 by the exponent
    return !(a >= 0x3ff00000u && a < 0x41e00000u);
}

// solvers.hpp:314-340 corner electric field from the four face fluxes and the corner velocity.
template <bool ANY = false>
__device__ __forceinline__ double corner_ez(double eN, double eS, double eE, double eW, double vxc,
                                            double vyc, int mode) {
    double ezy, ezx;
    if (ct_average(vyc, mode)) ezy = 0.5 * (eS + eN);
    else ezy = (ANY ? vyc > 0.0 : high_word(vyc) > 0) ? eS : eN;
    if (ct_average(vxc, mode)) ezx = 0.5 * (eE + eW);
    else ezx = (ANY ? vxc > 0.0 : high_word(vxc) > 0) ? eW : eE;
    return 0.5 * (ezx + ezy);
}

// diagnostics.hpp:60-77 fastest signal speed of one cell from its stored primitives.
template <bool ANY>
__device__ __forceinline__ double cfl_speed_of(double rho_f, double vx, double vy, double p,
                                               double bxc, double byc) {
    const double r = smax(rho_f, 1e-8);
    const double pr = smax(p, 1e-8);
    const double ir = ANY ? 1.0 / r : rcp_nr(r);
    const double a2 = kGammaGas * pr * ir;
    const double b2 = (bxc * bxc + byc * byc) * ir;
    const double v2 = vx * vx + vy * vy;
    if constexpr (ANY) return sqrt(a2 + b2) + sqrt(v2);
    const double v = sqrt_nr(v2);
    return sqrt_nr(a2 + b2) + (v2 > 1e-290 ? v : 0.0);
}
// Both, of any cell, from its conserved values (`rho` is replaced by the floored density); the speed is infinite where
// it overflows or the density is zero.
__device__ __forceinline__ double cell_cfl_speed(double& rho, double mx, double my, double E, double bxc, double byc) {
    const double stored = rho;
    double vx, vy;
    double p = primitives_of<false>(rho, mx, my, E, bxc, byc, vx, vy);
    double speed = cfl_speed_of<false>(rho, vx, vy, p, bxc, byc);
    if (!ordinary(rho, vx, vy, p, bxc, byc)) {
        rho = stored;
        p = primitives_of<true>(rho, mx, my, E, bxc, byc, vx, vy);
        speed = cfl_speed_of<true>(rho, vx, vy, p, bxc, byc);
    }
    return speed;
}

}  // namespace mhd

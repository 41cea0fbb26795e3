// fvm2d_math.cuh -- per-cell and per-interface arithmetic of the split step.
//
// One sweep treats its direction as "normal" (n) and the other as
// "tangential" (t): a cell is (rho, p, un, ut).  In an x-sweep un = u; in a
// y-sweep un = v, exactly as the reference's anti-transposed copy swaps the
// u and v slots (src/basicFuns.cuh:249-262).
//
// The functions below keep the reference's operation order: with FMA
// contraction off (-fmad=false) an FP64 build rounds every operation in the
// same order as the reference built the same way, so the two agree bit for
// bit.  The product build contracts (the nvcc default, as the reference's own
// build does) and is checked against the reference within a relative L1
// tolerance.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <string.h>
#include <type_traits>

#ifndef FVM2D_VARIANT
#error "define FVM2D_VARIANT (the namespace of this build of the kernels) first"
#endif

namespace fvm2d {
namespace FVM2D_VARIANT {

template <typename Real>
struct Cell {
    Real rho, p, un, ut;
};

template <typename Real>
__device__ __forceinline__ Real rmin(Real a, Real b) { return (b < a) ? b : a; }
template <typename Real>
__device__ __forceinline__ Real rmax(Real a, Real b) { return (a < b) ? b : a; }
// single precision: the min/max instructions (equal to the selects unless an
// argument is NaN)
__device__ __forceinline__ float rmin(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ float rmax(float a, float b) { return fmaxf(a, b); }
// 1/x and 1/sqrt(x).
//
// Builds that define FVM2D_FAST_RCP (the FP64 product build, and the FP64
// wave speed of the FP32 build) take the hardware's approximate seeds --
// PTX rcp.approx.ftz.f64 and rsqrt.approx.ftz.f64, about 20 correct bits --
// and refine each by one third-order step (Householder's method of order 3),
// written from the series
//   1/x       = r / (1 - e)       = r (1 + e + e^2 + ...),         e = 1 - x r
//   1/sqrt(x) = y / sqrt(1 - e)   = y (1 + e/2 + 3 e^2/8 + ...),   e = 1 - x y^2
// truncated after the quadratic term: the relative error falls from about
// 2^-20 to about 2^-58, below the rounding of the result, so the results are
// within a couple of ulp of correctly rounded ones (not bit-identical: that
// build is held to the reference within a relative L1 tolerance; a further
// Newton step towards correct rounding was measured to leave its distance
// from the oracle no smaller, 5% slower).  Each costs the seed and three to
// five FP64 operations instead of a full IEEE division or square-root
// sequence.  The
// seeds flush subnormal arguments to zero, so the arguments must be normal
// numbers: the solver's reciprocals take densities, pressures, sound speeds
// and their products, which are, in any state that is not degenerate
// (vacuum) or corrupt; the wave speed, whose velocity part can be
// arbitrarily small, clamps its arguments (wave_speed).  Other builds use
// IEEE division and CUDA's rsqrt (1 ulp); rsqrtf is within 2 ulp; the
// dual-number overloads live with the dual type, and other number types
// divide.
#if defined(FVM2D_FAST_RCP)
__device__ __forceinline__ double rcp_seed(double x)
{
#if defined(__CUDA_ARCH__)
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
#else
    return (1.0 / x) * (1.0 + 0x1p-21);  // host builds of this file (tests): a seed 2^-21 off
#endif
}
__device__ __forceinline__ double rsqrt_seed(double x)
{
#if defined(__CUDA_ARCH__)
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
#else
    return (1.0 / sqrt(x)) * (1.0 - 0x1p-21);
#endif
}
__device__ __forceinline__ double rrcp(double x)
{
    const double r = rcp_seed(x);
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double rrsqrt(double x)
{
    const double y = rsqrt_seed(x);
    const double e = fma(-(x * y), y, 1.0);
    return fma(y, e * fma(e, 0.375, 0.5), y);
}
#else
__device__ __forceinline__ double rrcp(double x) { return 1.0 / x; }
__device__ __forceinline__ double rrsqrt(double x) { return ::rsqrt(x); }
#endif
__device__ __forceinline__ float rrcp(float x) { return 1.0f / x; }
__device__ __forceinline__ float rrsqrt(float x) { return ::rsqrtf(x); }
template <typename Real>
__device__ __forceinline__ Real rrcp(Real x) { return Real(1) / x; }

// Generalized-minmod slope of one component from its left (m), centre (c)
// and right (p) values.  src/basicFuns.cuh:49-68.
template <typename Real>
__device__ __forceinline__ Real limited_slope(Real m, Real c, Real p, Real rh, Real alpha)
{
    Real central = (p - m) * Real(0.5) * rh;
    Real back = (c - m) * rh * alpha;
    Real fwd = (p - c) * rh * alpha;
    Real p13 = central * fwd, p23 = back * fwd;
    if (p13 > Real(0) && p23 > Real(0)) {
        Real sign = (central <= Real(0)) ? Real(-1) : Real(1);
        return sign * rmin(fabs(central), rmin(fabs(back), fabs(fwd)));
    }
    return Real(0);
}

// Interface state W = (rho, p, un, ut, e) and its time derivative Wt.
template <typename Real>
struct Interface {
    Real rho, p, un, ut, e;
    Real rho_t, p_t, un_t, ut_t, e_t;
};

// Relaxation GRP at one interface from the left/right face states (L, R)
// and the slopes of the two cells (sL, sR).  src/basicFuns.cuh:86-189.
// The star-region coefficients k_l, k_r, d_l, d_r read the velocity before
// it receives the star value (basicFuns.cuh:151-155 see the initial 0.0 of
// basicFuns.cuh:110); the literal `u0` keeps that.
template <typename Real>
__device__ __forceinline__ Interface<Real> relaxation_grp(const Cell<Real> &L, const Cell<Real> &R,
                                                          const Cell<Real> &sL, const Cell<Real> &sR,
                                                          Real g)
{
    const Real rho_l = L.rho, pi_l = L.p, u_l = L.un, v_l = L.ut;
    const Real rho_r = R.rho, pi_r = R.p, u_r = R.un, v_r = R.ut;
    const Real rho_lx = sL.rho, pi_lx = sL.p, u_lx = sL.un, v_lx = sL.ut;
    const Real rho_rx = sR.rho, pi_rx = sR.p, u_rx = sR.un, v_rx = sR.ut;
    const Real one = Real(1), two = Real(2), half = Real(0.5), zero = Real(0);

    Real e_l = pi_l / rho_l / (g - one);
    Real e_r = pi_r / rho_r / (g - one);
    Real e_lx = pi_lx / rho_l / (g - one) - pi_l * rho_lx / rho_l / rho_l / (g - one);
    Real e_rx = pi_rx / rho_r / (g - one) - pi_r * rho_rx / rho_r / rho_r / (g - one);
    Real c_lx = half * sqrt(g / pi_l / rho_l) * (pi_l * rho_lx + rho_l * pi_lx);
    Real c_rx = half * sqrt(g / pi_r / rho_r) * (pi_r * rho_rx + rho_r * pi_rx);

    Interface<Real> o;
    Real c_l, c_r;
    Real a_l = sqrt(g * pi_l / rho_l), a_r = sqrt(g * pi_r / rho_r);
    Real kappa = (g + one) / two;
    if (pi_r >= pi_l) {
        c_l = rho_l * (a_l + kappa * rmax(zero, (pi_r - pi_l) / rho_r / a_r + u_l - u_r));
        c_r = rho_r * (a_r + kappa * rmax(zero, (pi_l - pi_r) / c_l + u_l - u_r));
    } else {
        c_r = rho_r * (a_r + kappa * rmax(zero, (pi_l - pi_r) / rho_l / a_l + u_l - u_r));
        c_l = rho_l * (a_l + kappa * rmax(zero, (pi_r - pi_l) / c_r + u_l - u_r));
    }

    if (u_l - c_l / rho_l >= zero) {
        // the whole wave fan moves right: left state (basicFuns.cuh:129-137)
        Real rho = rho_l, pi = pi_l, u = u_l;
        o.rho = rho_l; o.p = pi_l; o.un = u_l; o.ut = v_l; o.e = e_l;
        o.rho_t = -rho * u_lx - u * rho_lx;
        o.un_t = -u * u_lx - pi_lx / rho;
        o.e_t = -u * e_lx - pi / rho * u_lx;
        o.ut_t = -u * v_lx;
        o.p_t = -u * pi_lx - c_l * c_l / rho_l * u_lx;
    } else if (u_r + c_r / rho_r <= zero) {
        // the whole wave fan moves left: right state (basicFuns.cuh:138-146)
        Real rho = rho_r, pi = pi_r, u = u_r;
        o.rho = rho_r; o.p = pi_r; o.un = u_r; o.ut = v_r; o.e = e_r;
        o.rho_t = -rho * u_rx - u * rho_rx;
        o.un_t = -u * u_rx - pi_rx / rho;
        o.e_t = -u * e_rx - pi / rho * u_rx;
        o.ut_t = -u * v_rx;
        o.p_t = -u * pi_rx - c_r * c_r / rho * u_rx;
    } else {
        // star region (basicFuns.cuh:147-186)
        const Real u0 = zero;
        Real u_m = (u_l * c_l + u_r * c_r + pi_l - pi_r) / (c_l + c_r);
        Real pi_m = ((u_l - u_r) * c_l * c_r + c_l * pi_r + c_r * pi_l) / (c_l + c_r);
        Real k_l = -pi_lx - c_l * u_lx + half * (u0 - u_l) * c_lx;
        Real k_r = -pi_rx + c_r * u_rx - half * (u0 - u_r) * c_rx;
        Real d_l = Real(-2.0) * c_l * c_l / rho_l * u_lx - two * c_l / rho_l * pi_lx + c_l / rho_l * (u0 - u_l) * c_lx;
        Real d_r = two * c_r * c_r / rho_r * u_rx - two * c_r / rho_r * pi_rx + c_r / rho_r * (u_r - u0) * c_rx;
        Real Dpi_Dt = (c_r * d_l - c_l * d_r) / two / (c_l + c_r);
        Real pi = pi_m, u = u_m, rho, e;
        o.p = pi_m;
        o.un = u_m;
        if (u <= zero) {
            Real rho_mr = c_r / (u_r - u_m + c_r / rho_r);
            Real e_mr = e_r + (pi_m - pi_r) * (pi_m + pi_r) / two / c_r / c_r;
            rho = rho_mr;
            e = e_mr;
            o.ut = v_r;
            o.rho_t = -u * rho * rho * rho / (rho_r * c_r * c_r) * (c_r * c_r / rho_r / rho_r * rho_rx - c_r * u_rx + Real(1.5) * (u - u_r) * c_rx) + rho * rho * rho / (c_r * c_r * c_r) * (u + c_r / rho) * Dpi_Dt;
            o.p_t = one / (c_l + c_r) * (c_l * c_r / rho_l * (one + u * rho / c_r) * k_l - c_l * c_r / rho_r * (one - u * rho / c_l) * k_r);
            o.un_t = one / (c_l + c_r) * (c_l / rho_l * (one + u * rho / c_r) * k_l + c_r / rho_r * (one - u * rho * c_l / c_r / c_r) * k_r);
            o.e_t = -u * rho / rho_r / c_r / c_r / c_r * (-pi_r * c_r * pi_rx + c_r * c_r * c_r * e_rx + two * (e_r - e) * c_r * c_r * c_rx) + pi / c_r / c_r * o.p_t;
            Real v_x = rho / rho_r * v_rx;
            o.ut_t = -u * v_x;
        } else {
            Real rho_ml = c_l / (u_m - u_l + c_l / rho_l);
            Real e_ml = e_l + (pi_m - pi_l) * (pi_m + pi_l) / two / c_l / c_l;
            rho = rho_ml;
            e = e_ml;
            o.ut = v_l;
            o.rho_t = -u * rho * rho * rho / (rho_l * c_l * c_l) * (c_l * c_l / rho_l / rho_l * rho_lx + c_l * u_lx + Real(1.5) * (u - u_l) * c_lx) - rho * rho * rho / (c_l * c_l * c_l) * (u - c_l / rho) * Dpi_Dt;
            o.p_t = one / (c_l + c_r) * (c_l * c_r / rho_l * (one + u * rho / c_r) * k_l - c_l * c_r / rho_r * (one - u * rho / c_l) * k_r);
            o.un_t = one / (c_l + c_r) * (c_l / rho_l * (one + u * rho * c_r / c_l / c_l) * k_l + c_r / rho_r * (one - u * rho / c_l) * k_r);
            o.e_t = -u * rho / rho_l / c_l / c_l / c_l * (-pi_l * c_l * pi_lx + c_l * c_l * c_l * e_lx + two * (e_l - e) * c_l * c_l * c_lx) + pi / c_l / c_l * o.p_t;
            Real v_x = rho / rho_l * v_lx;
            o.ut_t = -u * v_x;
        }
        o.rho = rho;
        o.e = e;
    }
    return o;
}

// Midpoint flux F(W) + k/2 dF/dt in the sweep's conserved ordering
// (mass, normal momentum, energy, tangential momentum).
// src/basicFuns.cuh:14-34.
template <typename Real>
__device__ __forceinline__ Cell<Real> midpoint_flux(const Interface<Real> &w, Real k)
{
    const Real rho = w.rho, pi = w.p, u = w.un, v = w.ut, e = w.e;
    const Real rho_t = w.rho_t, pi_t = w.p_t, u_t = w.un_t, v_t = w.ut_t, e_t = w.e_t;
    const Real two = Real(2);
    Cell<Real> F;
    F.rho = rho * u + k / two * (rho * u_t + u * rho_t);
    F.p = rho * u * u + pi + k / two * (rho_t * u * u + two * rho * u * u_t + pi_t);
    F.un = rho * u * (e + u * u / two + v * v / two) + pi * u + k / two * (rho_t * u * e + rho * u_t * e + rho * u * e_t + rho_t * u * u * u / two + Real(1.5) * rho * u * u * u_t + rho_t * u * v * v / two + rho * u * v * v_t + rho * u_t * v * v / two + pi_t * u + pi * u_t);
    F.ut = rho * u * v + k / two * (rho * u_t * v + u * rho_t * v + u * rho * v_t);
    return F;
}

// Conservative update of one cell, primitive in and out:
// W = cons(U); W -= (F_R - F_L) * lambda; U = prim(W).
// src/basicFuns.cuh:195-212, 240-244.  Field slots of the flux Cell are
// (mass, normal momentum, energy, tangential momentum).
template <typename Real>
__device__ __forceinline__ Cell<Real> conservative_update(const Cell<Real> &U, const Cell<Real> &FL,
                                                          const Cell<Real> &FR, Real lambda, Real g)
{
    const Real one = Real(1), two = Real(2);
    Real m0 = U.rho;
    Real m1 = U.rho * U.un;
    Real m2 = U.p / (g - one) + U.rho * (U.un * U.un + U.ut * U.ut) / two;
    Real m3 = U.rho * U.ut;
    m0 = m0 - (FR.rho - FL.rho) * lambda;
    m1 = m1 - (FR.p - FL.p) * lambda;
    m2 = m2 - (FR.un - FL.un) * lambda;
    m3 = m3 - (FR.ut - FL.ut) * lambda;
    Cell<Real> o;
    o.rho = m0;
    o.p = (g - one) * (m2 - m1 * m1 / m0 / two - m3 * m3 / m0 / two);
    o.un = m1 / m0;
    o.ut = m3 / m0;
    return o;
}

// ---------------------------------------------------------------------------
// Arithmetic policies.  A sweep kernel calls Phys::interface_flux once per
// interface and Phys::update once per cell.
//
// RefOrder: the reference's expressions in the reference's order (above).
// Hoisted:  the same mathematics with the reciprocals hoisted and shared
//           (1/rho of the contact's side only; 1/(rho a) per side as
//           1/sqrt(g p rho), with a = g p/(rho a); the second side's 1/c and
//           1/(c_l + c_r) from one division; 1/c of the first side and
//           1/rho_star: 4 divisions and 2 reciprocal square roots per
//           interface in the star region, 3 and 2 when the wave fan is
//           one-sided, where the reference's expressions divide by a
//           variable 61 times (27-28) and take 4 square roots),
//           sqrt(g/(p rho)) rewritten as g/(rho a), and the midpoint flux
//           written through the mass flux
//           m = rho u and its time derivative; the limiter tests signs on
//           the raw differences and scales its minimum once, and h/2 is
//           folded into the face states.  Rounding differs from the
//           reference at the ulp level; results are checked against the
//           reference within a relative L1 tolerance.
// ---------------------------------------------------------------------------
template <typename Real>
struct SweepConsts {
    Real h, rh, alpha, g;  // spacing, 1/h, limiter parameter, gamma
    Real k, lambda;        // dt and dt/h
    Real igm1, kappa;      // 1/(gamma-1), (gamma+1)/2   (Hoisted only)
    // 1/(gamma-1) and gamma-1 as hi + lo pairs of the arithmetic type (lo = 0
    // unless Real is float), for the compensated FP32 update: it converts p
    // to E and back once per sweep, and with the rounded constants alone
    // (2.5f and 1.4f - 1 for gamma 1.4) every round trip scales the internal
    // energy by 1 - 6e-8, a bias that grows with the number of sweeps
    Real igm1_lo, gm1, gm1_lo;
    Real lambda_lo;  // dt/h - lambda (0 unless Real is float): the FP64 update of residual builds
};

// The part of x that Real does not hold: 0 unless Real is float.
template <typename Real>
__host__ __device__ inline double lo_part(double x)
{
    if constexpr (std::is_same<Real, float>::value)
        return x - double(float(x));
    else
        return 0.0;
}

// The constants of gamma in SweepConsts.
template <typename Real>
__host__ __device__ inline void set_gamma_consts(SweepConsts<Real> &K, double gamma)
{
    const double gm1 = gamma - 1.0, igm1 = 1.0 / gm1;
    K.g = Real(gamma);
    K.igm1 = Real(igm1);
    K.igm1_lo = Real(lo_part<Real>(igm1));
    K.gm1 = Real(gm1);
    K.gm1_lo = Real(lo_part<Real>(gm1));
    K.kappa = Real((gamma + 1.0) / 2.0);
}

template <typename Real>
__device__ __forceinline__ Cell<Real> cell_slope(const Cell<Real> &m, const Cell<Real> &c, const Cell<Real> &p,
                                                 const SweepConsts<Real> &K)
{
    Cell<Real> s;
    s.rho = limited_slope(m.rho, c.rho, p.rho, K.rh, K.alpha);
    s.p = limited_slope(m.p, c.p, p.p, K.rh, K.alpha);
    s.un = limited_slope(m.un, c.un, p.un, K.rh, K.alpha);
    s.ut = limited_slope(m.ut, c.ut, p.ut, K.rh, K.alpha);
    return s;
}

// Face states of the interface between cells L and R: U_L + s_L h/2 and
// U_R - s_R h/2 (src/basicFuns.cuh:69-70).
template <typename Real>
__device__ __forceinline__ void face_states(const Cell<Real> &UL, const Cell<Real> &UR, const Cell<Real> &sL,
                                            const Cell<Real> &sR, Real h, Cell<Real> &fL, Cell<Real> &fR)
{
    fL.rho = UL.rho + sL.rho * h * Real(0.5);
    fL.p = UL.p + sL.p * h * Real(0.5);
    fL.un = UL.un + sL.un * h * Real(0.5);
    fL.ut = UL.ut + sL.ut * h * Real(0.5);
    fR.rho = UR.rho - sR.rho * h * Real(0.5);
    fR.p = UR.p - sR.p * h * Real(0.5);
    fR.un = UR.un - sR.un * h * Real(0.5);
    fR.ut = UR.ut - sR.ut * h * Real(0.5);
}

struct RefOrder {
    template <typename Real>
    __device__ static __forceinline__ Cell<Real> slope(const Cell<Real> &m, const Cell<Real> &c, const Cell<Real> &p,
                                                       const SweepConsts<Real> &K)
    {
        return cell_slope(m, c, p, K);
    }
    template <typename Real>
    __device__ static __forceinline__ Cell<Real> interface_flux(const Cell<Real> &UL, const Cell<Real> &UR,
                                                                const Cell<Real> &sL, const Cell<Real> &sR,
                                                                const SweepConsts<Real> &K)
    {
        Cell<Real> fL, fR;
        face_states(UL, UR, sL, sR, K.h, fL, fR);
        return midpoint_flux(relaxation_grp(fL, fR, sL, sR, K.g), K.k);
    }
    template <typename Real>
    __device__ static __forceinline__ Cell<Real> update(const Cell<Real> &U, const Cell<Real> &FL,
                                                        const Cell<Real> &FR, const SweepConsts<Real> &K)
    {
        return conservative_update(U, FL, FR, K.lambda, K.g);
    }
};

// Generalized minmod on raw differences: the reference's sign tests on the
// scaled differences are sign tests on the differences themselves (rh and
// alpha are positive), and the minimum is scaled once.
template <typename Real>
__device__ __forceinline__ Real limited_slope_hoisted(Real m, Real c, Real p, Real hrh, Real rha)
{
    const Real d1 = c - m, d2 = p - c, dc = p - m;
    if (dc * d2 > Real(0) && d1 * d2 > Real(0)) {
        const Real a = rmin(fabs(dc) * hrh, rha * rmin(fabs(d1), fabs(d2)));
        return dc <= Real(0) ? -a : a;
    }
    return Real(0);
}

// Double precision: the same result with one product and one test.  d1 d2 > 0
// implies dc d2 > 0: d1, d2 nonzero of one sign puts m, c, p in strict order,
// so dc = fl(p - m) has that sign and |dc| >= |d1| (rounding is monotonic),
// hence |dc d2| >= |d1 d2| > 0; then dc != 0 and the result takes its sign.
// The minima are formed for every cell and selected: four fields without a
// branch between them overlap their chains (4096^2 step of a varied flow in
// tiles: 1627 -> 1587 us).
__device__ __forceinline__ double limited_slope_hoisted(double m, double c, double p, double hrh, double rha)
{
    const double d1 = c - m, d2 = p - c, dc = p - m;
    const double a = rmin(fabs(dc) * hrh, rha * rmin(fabs(d1), fabs(d2)));
    return d1 * d2 > 0.0 ? copysign(a, dc) : 0.0;
}

// Single precision: the same choices with the min/max and sign instructions
// (they differ from the selects above only when an argument is NaN); the
// sign test is d1 d2 > 0 alone, for the reason given above.
__device__ __forceinline__ float limited_slope_hoisted(float m, float c, float p, float hrh, float rha)
{
    const float d1 = c - m, d2 = p - c, dc = p - m;
    const float a = fminf(fabsf(dc) * hrh, rha * fminf(fabsf(d1), fabsf(d2)));
    return d1 * d2 > 0.f ? copysignf(a, dc) : 0.f;
}

// The limiter as a kernel with constants of type Consts takes it.  The sweep
// kernels, which wait more for memory, gain nothing by the select (4096^2 slab
// step of a varied flow 1816 us with a branch around the minima, 1808 with the
// select) and lose where the flow is constant (plain quadrants: 1591, 1722): the
// branch, with the same result.
template <typename Real, class Consts>
__device__ __forceinline__ Real limiter(Real m, Real c, Real p, Real hrh, Real rha, const Consts &)
{
    return limited_slope_hoisted(m, c, p, hrh, rha);
}
__device__ __forceinline__ double limiter(double m, double c, double p, double hrh, double rha,
                                          const SweepConsts<double> &)
{
    const double d1 = c - m, d2 = p - c, dc = p - m;
    if (d1 * d2 > 0.0) return copysign(rmin(fabs(dc) * hrh, rha * rmin(fabs(d1), fabs(d2))), dc);
    return 0.0;
}

// Products of the constants of a sweep, formed where they are used; a kernel
// that keeps its constants in memory keeps the products there (TileConsts in
// fvm2d_tile.cuh) and overloads these.
template <typename Real>
__device__ __forceinline__ Real half_h(const SweepConsts<Real> &K) { return K.h * Real(0.5); }
template <typename Real>
__device__ __forceinline__ Real half_rh(const SweepConsts<Real> &K) { return K.rh * Real(0.5); }
template <typename Real>
__device__ __forceinline__ Real alpha_rh(const SweepConsts<Real> &K) { return K.rh * K.alpha; }
template <typename Real>
__device__ __forceinline__ Real half_k(const SweepConsts<Real> &K) { return K.k * Real(0.5); }
// and the constants kept as hi + lo pairs, joined
template <typename Real>
__device__ __forceinline__ double joined_lambda(const SweepConsts<Real> &K) { return double(K.lambda) + double(K.lambda_lo); }
template <typename Real>
__device__ __forceinline__ double joined_igm1(const SweepConsts<Real> &K) { return double(K.igm1) + double(K.igm1_lo); }
template <typename Real>
__device__ __forceinline__ double joined_gm1(const SweepConsts<Real> &K) { return double(K.gm1) + double(K.gm1_lo); }

// Every sum of a product below is written as an fma or as two roundings, and
// the FP64 build is compiled without contraction, so each copy of this
// arithmetic (walkers, tiles, batches, taped steps) rounds alike.
struct Hoisted {
    template <typename Real, class Consts>
    __device__ static __forceinline__ Cell<Real> slope(const Cell<Real> &m, const Cell<Real> &c, const Cell<Real> &p,
                                                       const Consts &K)
    {
        Cell<Real> s;
        const Real hrh = half_rh(K), rha = alpha_rh(K);
        s.rho = limiter(m.rho, c.rho, p.rho, hrh, rha, K);
        s.p = limiter(m.p, c.p, p.p, hrh, rha, K);
        s.un = limiter(m.un, c.un, p.un, hrh, rha, K);
        s.ut = limiter(m.ut, c.ut, p.ut, hrh, rha, K);
        return s;
    }
    // The reference's formulas (src/basicFuns.cuh:86-189) with common parts
    // taken out.  With k_l, k_r as there and s = c / rho, its d_l = 2 s_l k_l
    // and d_r = 2 s_r k_r, so Dpi_Dt = (c_r s_l k_l - c_l s_r k_r) / (c_l + c_r).
    // On the side of the contact (c, the face's rho, u, ...; sg = 1 on the
    // right, -1 on the left) z = 1 / (sg (u_s - u) + c / rho_s) is the star
    // density over c; with w = u z and h = 1 + sg w
    //   rho_t = z (z h Dpi_Dt - w (rho / rho_s) S),
    //   S     = s^2 rho_x - sg c u_x + 3/2 (u - u_s) c_x,
    // and u rho / c = w in the factors of p_t and u_t: about 125 operations from
    // the face states to the star region's derivatives, where the formulas term
    // by term take about 165.
    template <typename Real, class Consts>
    __device__ static __forceinline__ Interface<Real> grp(const Cell<Real> &L, const Cell<Real> &R,
                                                          const Cell<Real> &sL, const Cell<Real> &sR,
                                                          const Consts &K)
    {
        const Real one = Real(1), half = Real(0.5), zero = Real(0);
        const Real g = K.g, igm1 = K.igm1, kappa = K.kappa;
        const Real rho_l = L.rho, pi_l = L.p, u_l = L.un, v_l = L.ut;
        const Real rho_r = R.rho, pi_r = R.p, u_r = R.un, v_r = R.ut;
        const Real rho_lx = sL.rho, pi_lx = sL.p, u_lx = sL.un, v_lx = sL.ut;
        const Real rho_rx = sR.rho, pi_rx = sR.p, u_rx = sR.un, v_rx = sR.ut;

        // 1/(rho a) = 1/sqrt(g p rho) and a = sqrt(g p / rho) = g p / sqrt(g p rho):
        // one reciprocal square root per side
        const Real gpl = g * pi_l, gpr = g * pi_r;
        const Real il = rrsqrt(gpl * rho_l), ir = rrsqrt(gpr * rho_r);
        const Real a_l = gpl * il, a_r = gpr * ir;
        const Real hg = half * g;
        const Real c_lx = fma(pi_l, rho_lx, rho_l * pi_lx) * (hg * il);
        const Real c_rx = fma(pi_r, rho_rx, rho_r * pi_rx) * (hg * ir);
        const Real du = u_l - u_r, dp = pi_r - pi_l;
        // the side computed second gets its reciprocal and 1/(c_l + c_r)
        // from one division
        Real c_l, c_r, icl, icr, isum, sl, sr;  // s = c/rho: the fan's edge speeds relative to u
        if (pi_r >= pi_l) {
            sl = fma(kappa, rmax(zero, fma(dp, ir, du)), a_l);
            c_l = rho_l * sl;
            icl = rrcp(c_l);
            sr = fma(kappa, rmax(zero, fma(-dp, icl, du)), a_r);
            c_r = rho_r * sr;
            const Real sc = c_l + c_r, q = rrcp(c_r * sc);
            icr = sc * q;
            isum = c_r * q;
        } else {
            sr = fma(kappa, rmax(zero, fma(-dp, il, du)), a_r);
            c_r = rho_r * sr;
            icr = rrcp(c_r);
            sl = fma(kappa, rmax(zero, fma(dp, icr, du)), a_l);
            c_l = rho_l * sl;
            const Real sc = c_l + c_r, q = rrcp(c_l * sc);
            icl = sc * q;
            isum = c_l * q;
        }
        Interface<Real> o;
        if (u_l - sl >= zero) {
            const Real irl = rrcp(rho_l), iri = irl * igm1, tp = pi_l * irl;
            o.rho = rho_l; o.p = pi_l; o.un = u_l; o.ut = v_l; o.e = pi_l * iri;
            o.rho_t = -fma(rho_l, u_lx, u_l * rho_lx);
            o.un_t = -fma(u_l, u_lx, pi_lx * irl);
            o.e_t = -fma(u_l, fma(-tp, rho_lx, pi_lx) * iri, tp * u_lx);
            o.ut_t = -(u_l * v_lx);
            o.p_t = -fma(u_l, pi_lx, (c_l * sl) * u_lx);
        } else if (u_r + sr <= zero) {
            const Real irr = rrcp(rho_r), iri = irr * igm1, tp = pi_r * irr;
            o.rho = rho_r; o.p = pi_r; o.un = u_r; o.ut = v_r; o.e = pi_r * iri;
            o.rho_t = -fma(rho_r, u_rx, u_r * rho_rx);
            o.un_t = -fma(u_r, u_rx, pi_rx * irr);
            o.e_t = -fma(u_r, fma(-tp, rho_rx, pi_rx) * iri, tp * u_rx);
            o.ut_t = -(u_r * v_rx);
            o.p_t = -fma(u_r, pi_rx, (c_r * sr) * u_rx);
        } else {
            const Real u = (fma(u_l, c_l, u_r * c_r) - dp) * isum;
            const Real pm = fma(du * c_l, c_r, fma(c_l, pi_r, c_r * pi_l)) * isum;
            // b_l = -s_l k_l, b_r = s_r k_r, nDp = -Dpi_Dt
            const Real b_l = sl * fma(half * u_l, c_lx, fma(c_l, u_lx, pi_lx));
            const Real b_r = sr * fma(half * u_r, c_rx, fma(c_r, u_rx, -pi_rx));
            const Real nDp = fma(c_r, b_l, c_l * b_r) * isum;
            o.p = pm;
            o.un = u;
            if (u <= zero) {
                const Real irr = rrcp(rho_r), z = rrcp((u_r - u) + sr);
                const Real rho = c_r * z, w = u * z, h = one + w, q = rho * irr;
                const Real S = fma(sr * sr, rho_rx, fma(-c_r, u_rx, (Real(1.5) * (u - u_r)) * c_rx));
                const Real P = b_l * h;
                const Real icr2 = icr * icr, E2 = (pm - pi_r) * (pm + pi_r) * icr2;
                const Real iri = irr * igm1, tp = pi_r * irr;
                const Real G = fma(-icr, fma(E2, c_rx, (icr * pi_r) * pi_rx), fma(-tp, rho_rx, pi_rx) * iri);
                const Real uq = u * q;
                o.rho = rho;
                o.e = fma(half, E2, pi_r * iri);
                o.ut = v_r;
                o.rho_t = -(z * fma(z * h, nDp, (w * q) * S));
                o.p_t = -(isum * fma(c_r, P, b_r * fma(-u, rho, c_l)));
                o.un_t = isum * fma(b_r, fma(-(w * c_l), icr, one), -P);
                o.e_t = fma(pm * icr2, o.p_t, -(uq * G));
                o.ut_t = -(uq * v_rx);
            } else {
                const Real irl = rrcp(rho_l), z = rrcp((u - u_l) + sl);
                const Real rho = c_l * z, w = u * z, h = one - w, q = rho * irl;
                const Real S = fma(sl * sl, rho_lx, fma(c_l, u_lx, (Real(1.5) * (u - u_l)) * c_lx));
                const Real P = b_r * h;
                const Real icl2 = icl * icl, E2 = (pm - pi_l) * (pm + pi_l) * icl2;
                const Real iri = irl * igm1, tp = pi_l * irl;
                const Real G = fma(-icl, fma(E2, c_lx, (icl * pi_l) * pi_lx), fma(-tp, rho_lx, pi_lx) * iri);
                const Real uq = u * q;
                o.rho = rho;
                o.e = fma(half, E2, pi_l * iri);
                o.ut = v_l;
                o.rho_t = -(z * fma(z * h, nDp, (w * q) * S));
                o.p_t = -(isum * fma(b_l, fma(u, rho, c_r), c_l * P));
                o.un_t = isum * fma(-b_l, fma(w * c_r, icl, one), P);
                o.e_t = fma(pm * icl2, o.p_t, -(uq * G));
                o.ut_t = -(uq * v_lx);
            }
        }
        return o;
    }

    // Single precision keeps the formulas term by term, and each rounding where
    // it was: the midpoint flux jumps where the contact speed u (or a fan edge's
    // speed) crosses zero, the star density and tangential velocity changing
    // sides and k/2 rho u_t with them.  Where such a speed is within FP32
    // rounding of zero the order of the operations decides, and cells there
    // change by 1e-5 to 1e-4, so the order is part of what these builds return.
    // Every fma is written (cfma) and they are compiled without contraction: left
    // to the compiler, tiles and sweeps chose differently (17% of the velocities
    // of one step apart in the last bit).  Two roundings belong to some sweeps,
    // whose results keep them: `sound`, the sound speed's product rounded by
    // itself in the impedances (PackedResidual); `once`, c_r u_rx - p_rx rounded
    // once (PackedBatch).
    // (host builds, for tests, round the product and the sum as the formulas read)
    __device__ static __forceinline__ float cfma(float a, float b, float c)
    {
#if defined(__CUDA_ARCH__)
        return fmaf(a, b, c);
#else
        return a * b + c;
#endif
    }
    struct Fan {  // the two fans' speeds, as forward and adjoint take them
        float irl, irr, il, ir, c_lx, c_rx, zl, zr, c_l, c_r, icl, icr, isum, sl, sr;
    };
    template <class Consts>
    __device__ static __forceinline__ Fan fan(const Cell<float> &L, const Cell<float> &R, const Cell<float> &sL,
                                              const Cell<float> &sR, const Consts &K, bool sound = false)
    {
        const float zero = 0.f, kappa = K.kappa, hg = 0.5f * K.g;
        Fan w;
        // 1/rho_l and 1/rho_r from one division
        const float irlr = rrcp(L.rho * R.rho);
        w.irl = R.rho * irlr;
        w.irr = L.rho * irlr;
        // 1/(rho a) = 1/sqrt(g p rho) and a = sqrt(g p / rho) = g p / sqrt(g p rho):
        // one reciprocal square root per side
        const float gpl = K.g * L.p, gpr = K.g * R.p;
        w.il = rrsqrt(gpl * L.rho);
        w.ir = rrsqrt(gpr * R.rho);
        w.c_lx = hg * cfma(L.p, sL.rho, L.rho * sL.p) * w.il;
        w.c_rx = hg * cfma(R.p, sR.rho, R.rho * sR.p) * w.ir;
        const float du = L.un - R.un, dp = R.p - L.p;
        auto speed = [&](float gp, float i, float z) {  // a + kappa max(0, z)
            return sound ? cfma(kappa, rmax(zero, z), gp * i) : cfma(gp, i, kappa * rmax(zero, z));
        };
        // the side computed second gets its reciprocal and 1/(c_l + c_r)
        // from one division
        if (R.p >= L.p) {
            w.zl = cfma(dp, w.ir, du);
            w.c_l = L.rho * speed(gpl, w.il, w.zl);
            w.icl = rrcp(w.c_l);
            w.zr = cfma(-dp, w.icl, du);
            w.c_r = R.rho * speed(gpr, w.ir, w.zr);
            const float sc = w.c_l + w.c_r, q = rrcp(w.c_r * sc);
            w.icr = sc * q;
            w.isum = w.c_r * q;
        } else {
            w.zr = cfma(-dp, w.il, du);
            w.c_r = R.rho * speed(gpr, w.ir, w.zr);
            w.icr = rrcp(w.c_r);
            w.zl = cfma(dp, w.icr, du);
            w.c_l = L.rho * speed(gpl, w.il, w.zl);
            const float sc = w.c_l + w.c_r, q = rrcp(w.c_l * sc);
            w.icl = sc * q;
            w.isum = w.c_l * q;
        }
        w.sl = w.c_l * w.irl;  // c/rho: the fan's edge speeds relative to u
        w.sr = w.c_r * w.irr;
        return w;
    }
    __device__ static __forceinline__ float contact_speed(float u_l, float c_l, float p_l, float u_r, float c_r, float p_r,
                                                          float isum)
    {
        return (cfma(u_l, c_l, u_r * c_r) + p_l - p_r) * isum;
    }
    __device__ static __forceinline__ float contact_pressure(float du, float c_l, float p_l, float c_r, float p_r,
                                                             float isum)
    {
        return cfma(c_r, p_l, cfma(c_l, p_r, du * c_l * c_r)) * isum;
    }
    template <class Consts>
    __device__ static __forceinline__ Interface<float> grp(const Cell<float> &L, const Cell<float> &R,
                                                           const Cell<float> &sL, const Cell<float> &sR,
                                                           const Consts &K, bool sound = false, bool once = false)
    {
        const float one = 1.f, half = 0.5f, zero = 0.f, igm1 = K.igm1;
        const float rho_l = L.rho, pi_l = L.p, u_l = L.un, v_l = L.ut;
        const float rho_r = R.rho, pi_r = R.p, u_r = R.un, v_r = R.ut;
        const float rho_lx = sL.rho, pi_lx = sL.p, u_lx = sL.un, v_lx = sL.ut;
        const float rho_rx = sR.rho, pi_rx = sR.p, u_rx = sR.un, v_rx = sR.ut;
        const Fan w = fan(L, R, sL, sR, K, sound);
        const float irl = w.irl, irr = w.irr, c_lx = w.c_lx, c_rx = w.c_rx, c_l = w.c_l, c_r = w.c_r;
        const float icl = w.icl, icr = w.icr, isum = w.isum, sl = w.sl, sr = w.sr;
        // a side's e and (gamma - 1) e_x, wanted on one side only
        auto energy = [&](float p, float ir) { return p * ir * igm1; };
        auto energy_x = [&](float p, float rho_x, float p_x, float ir) { return cfma(-(p * rho_x), ir, p_x) * ir; };
        Interface<float> o;
        if (u_l - sl >= zero) {
            o.rho = rho_l; o.p = pi_l; o.un = u_l; o.ut = v_l; o.e = energy(pi_l, irl);
            o.rho_t = cfma(-rho_l, u_lx, -(u_l * rho_lx));
            o.un_t = cfma(-u_l, u_lx, -(pi_lx * irl));
            o.e_t = cfma(-u_l, energy_x(pi_l, rho_lx, pi_lx, irl) * igm1, -(pi_l * irl * u_lx));
            o.ut_t = -u_l * v_lx;
            o.p_t = cfma(-u_l, pi_lx, -(c_l * sl * u_lx));
        } else if (u_r + sr <= zero) {
            o.rho = rho_r; o.p = pi_r; o.un = u_r; o.ut = v_r; o.e = energy(pi_r, irr);
            o.rho_t = cfma(-rho_r, u_rx, -(u_r * rho_rx));
            o.un_t = cfma(-u_r, u_rx, -(pi_rx * irr));
            o.e_t = cfma(-u_r, energy_x(pi_r, rho_rx, pi_rx, irr) * igm1, -(pi_r * irr * u_rx));
            o.ut_t = -u_r * v_rx;
            o.p_t = cfma(-u_r, pi_rx, -(c_r * sr * u_rx));
        } else {
            const float u = contact_speed(u_l, c_l, pi_l, u_r, c_r, pi_r, isum);
            const float pm = contact_pressure(u_l - u_r, c_l, pi_l, c_r, pi_r, isum);
            const float cu_l = c_l * u_lx, cu_r = c_r * u_rx;
            const float f_r = once ? cfma(c_r, u_rx, -pi_rx) : cu_r - pi_rx;
            const float k_l = cfma(-(half * u_l), c_lx, -pi_lx - cu_l);
            const float k_r = cfma(half * u_r, c_rx, f_r);
            const float d_l = sl * cfma(-2.f, cu_l + pi_lx, -(u_l * c_lx));
            const float d_r = sr * cfma(u_r, c_rx, 2.f * f_r);
            const float Dp = cfma(c_r, d_l, -(c_l * d_r)) * half * isum;
            o.p = pm;
            o.un = u;
            if (u <= zero) {
                const float irho = (u_r - u + sr) * icr;
                const float rho = rrcp(irho), icr2 = icr * icr;
                const float e_r = energy(pi_r, irr), e = cfma((pm - pi_r) * (pm + pi_r) * half, icr2, e_r);
                const float rho3 = rho * rho * rho, urho = u * rho;
                const float h_l = cfma(urho, icr, one), h_r = cfma(-urho, icl, one);
                const float S = cfma(1.5f * (u - u_r), c_rx, cfma(sr * sr, rho_rx, -cu_r));
                const float G = cfma(2.f * (e_r - e) * c_rx, icr, cfma(energy_x(pi_r, rho_rx, pi_rx, irr), igm1, -(pi_r * pi_rx * icr2)));
                o.rho = rho; o.e = e; o.ut = v_r;
                o.rho_t = cfma(rho3 * icr2 * icr * cfma(c_r, irho, u), Dp, -u * rho3 * irr * icr2 * S);
                o.p_t = isum * cfma(c_r * sl * h_l, k_l, -(c_l * sr * h_r * k_r));
                o.un_t = isum * cfma(sl * h_l, k_l, sr * cfma(-(urho * c_l), icr2, one) * k_r);
                o.e_t = cfma(-urho * irr, G, pm * icr2 * o.p_t);
                o.ut_t = -urho * irr * v_rx;
            } else {
                const float irho = (u - u_l + sl) * icl;
                const float rho = rrcp(irho), icl2 = icl * icl;
                const float e_l = energy(pi_l, irl), e = cfma((pm - pi_l) * (pm + pi_l) * half, icl2, e_l);
                const float rho3 = rho * rho * rho, urho = u * rho;
                const float h_l = cfma(urho, icr, one), h_r = cfma(-urho, icl, one);
                const float S = cfma(1.5f * (u - u_l), c_lx, cfma(sl * sl, rho_lx, cu_l));
                const float G = cfma(2.f * (e_l - e) * c_lx, icl, cfma(energy_x(pi_l, rho_lx, pi_lx, irl), igm1, -(pi_l * pi_lx * icl2)));
                o.rho = rho; o.e = e; o.ut = v_l;
                o.rho_t = cfma(-u * rho3 * irl * icl2, S, -(rho3 * icl2 * icl * cfma(-c_l, irho, u) * Dp));
                o.p_t = isum * cfma(c_r * sl * h_l, k_l, -(c_l * sr * h_r * k_r));
                o.un_t = isum * cfma(sr * h_r, k_r, sl * cfma(urho * c_r, icl2, one) * k_l);
                o.e_t = cfma(-urho * irl, G, pm * icl2 * o.p_t);
                o.ut_t = -urho * irl * v_lx;
            }
        }
        return o;
    }

    // F + k/2 dF/dt through m = rho u and m_t = d(rho u)/dt (the product rule
    // applied to src/basicFuns.cuh:28-33), gathered around the midpoint mass
    // flux M = m + k/2 m_t and pressure Q = p + k/2 p_t.
    template <typename Real, class Consts>
    __device__ static __forceinline__ Cell<Real> flux_of(const Interface<Real> &w, const Consts &K)
    {
        const Real hk = half_k(K), half = Real(0.5);
        const Real m = w.rho * w.un, m_t = fma(w.rho, w.un_t, w.un * w.rho_t);
        const Real M = fma(hk, m_t, m), hm = hk * m;
        const Real es = fma(half, fma(w.un, w.un, w.ut * w.ut), w.e);
        const Real et = fma(w.un, w.un_t, fma(w.ut, w.ut_t, w.e_t));
        Cell<Real> F;
        F.rho = M;
        const Real Q = fma(hk, w.p_t, w.p);
        F.p = fma(M, w.un, fma(hm, w.un_t, Q));
        F.un = fma(es, M, fma(hm, et, fma(w.un, Q, (hk * w.p) * w.un_t)));
        F.ut = fma(M, w.ut, hm * w.ut_t);
        return F;
    }
    // and term by term in single precision (grp)
    template <class Consts>
    __device__ static __forceinline__ Cell<float> flux_of(const Interface<float> &w, const Consts &K)
    {
        const float hk = half_k(K);
        const float m = w.rho * w.un, m_t = cfma(w.un, w.rho_t, w.rho * w.un_t);
        const float es = cfma(0.5f, cfma(w.un, w.un, w.ut * w.ut), w.e);
        const float et = cfma(w.ut, w.ut_t, cfma(w.un, w.un_t, w.e_t));
        Cell<float> F;
        F.rho = cfma(hk, m_t, m);
        F.p = cfma(hk, cfma(m, w.un_t, m_t * w.un) + w.p_t, cfma(m, w.un, w.p));
        F.un = cfma(hk, cfma(w.p, w.un_t, cfma(w.p_t, w.un, cfma(m_t, es, m * et))), cfma(w.p, w.un, m * es));
        F.ut = cfma(m, w.ut, hk * cfma(m, w.ut_t, m_t * w.ut));
        return F;
    }

    template <typename Real, class Consts>
    __device__ static __forceinline__ Cell<Real> interface_flux(const Cell<Real> &UL, const Cell<Real> &UR,
                                                                const Cell<Real> &sL, const Cell<Real> &sR,
                                                                const Consts &K)
    {
        const Real hh = half_h(K);
        Cell<Real> fL, fR;  // U_L + s_L h/2, U_R - s_R h/2 with h/2 folded in
        fL.rho = fma(sL.rho, hh, UL.rho);
        fL.p = fma(sL.p, hh, UL.p);
        fL.un = fma(sL.un, hh, UL.un);
        fL.ut = fma(sL.ut, hh, UL.ut);
        fR.rho = fma(-sR.rho, hh, UR.rho);
        fR.p = fma(-sR.p, hh, UR.p);
        fR.un = fma(-sR.un, hh, UR.un);
        fR.ut = fma(-sR.ut, hh, UR.ut);
        return flux_of(grp(fL, fR, sL, sR, K), K);
    }

    template <typename Real, class Consts>
    __device__ static __forceinline__ Cell<Real> update(const Cell<Real> &U, const Cell<Real> &FL,
                                                        const Cell<Real> &FR, const Consts &K)
    {
        const Real half = Real(0.5);
        // W + lambda (F_L - F_R): momenta with the change rounded before the
        // product it joins, one rounding each; the energy with the pressure's
        // part rounded by itself, as the reference does (with the change rounded
        // first, pressures ended 1.5 to 2.4 times as far from the formulas in
        // the reference's order, over 40 steps of four flows)
        const Real m0 = fma(FL.rho - FR.rho, K.lambda, U.rho);
        const Real m1 = fma(U.rho, U.un, (FL.p - FR.p) * K.lambda);
        const Real m2 = fma(FL.un - FR.un, K.lambda, fma(half * U.rho, fma(U.un, U.un, U.ut * U.ut), U.p * K.igm1));
        const Real m3 = fma(U.rho, U.ut, (FL.ut - FR.ut) * K.lambda);
        const Real ir = rrcp(m0);
        Cell<Real> o;
        o.rho = m0;
        o.un = m1 * ir;
        o.ut = m3 * ir;
        o.p = K.gm1 * fma(-(half * fma(m3, m3, m1 * m1)), ir, m2);
        return o;
    }
};

// ---------------------------------------------------------------------------
// Compensated conservative update for FP32 storage.  The cell's conserved
// vector and its update are carried as unevaluated sums hi + lo built from
// error-free transformations (TwoSum, and TwoProd through fma), so the sum
// W - lambda (F_R - F_L) loses nothing to rounding before the primitive
// variables are recovered; the recovery divides and subtracts with the same
// residual terms.  The only roundings left are the flux difference itself and
// the final rounding of each primitive to its FP32 plane.
// ---------------------------------------------------------------------------
template <typename Real>
__device__ __forceinline__ void two_sum(Real a, Real b, Real &s, Real &e)
{
    s = a + b;
    const Real bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

template <typename Real>
__device__ __forceinline__ void two_prod(Real a, Real b, Real &p, Real &e)
{
    p = a * b;
    e = fma(a, b, -p);
}

struct HoistedCompensated : Hoisted {
    template <typename Real, class Consts>
    __device__ static __forceinline__ Cell<Real> update(const Cell<Real> &U, const Cell<Real> &FL,
                                                        const Cell<Real> &FR, const Consts &K)
    {
        const Real half = Real(0.5);
        // conserved vector of the cell: (rho, rho un, E, rho ut) as hi + lo
        Real m1, m1e, m3, m3e;
        two_prod(U.rho, U.un, m1, m1e);
        two_prod(U.rho, U.ut, m3, m3e);
        Real ka, kae, kb, kbe, kin, kine;
        two_prod(m1, U.un, ka, kae);
        two_prod(m3, U.ut, kb, kbe);
        two_sum(ka, kb, kin, kine);
        kine += kae + kbe + m1e * U.un + m3e * U.ut;  // rho (un^2 + ut^2) = kin + kine
        Real pe, pee, E, Ee;
        two_prod(U.p, K.igm1, pe, pee);
        pee = fma(U.p, K.igm1_lo, pee);  // p / (gamma - 1) = pe + pee
        two_sum(pe, half * kin, E, Ee);
        Ee += pee + half * kine;
        // W - lambda (F_R - F_L), compensated
        Real s0, e0, s1, e1, s2, e2, s3, e3;
        two_sum(U.rho, -(FR.rho - FL.rho) * K.lambda, s0, e0);
        two_sum(m1, -(FR.p - FL.p) * K.lambda, s1, e1);
        two_sum(E, -(FR.un - FL.un) * K.lambda, s2, e2);
        two_sum(m3, -(FR.ut - FL.ut) * K.lambda, s3, e3);
        e1 += m1e;
        e2 += Ee;
        e3 += m3e;
        // primitives from (s + e)
        Cell<Real> o;
        o.rho = s0 + e0;
        const Real ir = Real(1) / o.rho;
        const Real qu = s1 * ir, qv = s3 * ir;
        o.un = fma(fma(-qu, o.rho, s1) + e1, ir, qu);
        o.ut = fma(fma(-qv, o.rho, s3) + e3, ir, qv);
        Real ku, kue, kv, kve, k2, k2e;
        two_prod(s1, o.un, ku, kue);
        two_prod(s3, o.ut, kv, kve);
        two_sum(ku, kv, k2, k2e);
        k2e += kue + kve + e1 * o.un + e3 * o.ut;  // m . u = k2 + k2e
        Real d, de;
        two_sum(s2, -half * k2, d, de);
        const Real ei = d + (de + e2 - half * k2e);  // internal energy
        o.p = fma(K.gm1, ei, K.gm1_lo * ei);        // (gamma - 1) ei with the constant's low part
        return o;
    }
};

// |(u, v)| + sqrt(gamma p / rho) in the array's own (u, v) order.
// src/basicFuns.cuh:223-224.
template <typename Real>
__device__ __forceinline__ double wave_speed(Real rho, Real p, Real u, Real v, double g)
{
    double du = double(u), dv = double(v);
#if defined(FVM2D_FAST_RCP)
    // sqrt(q) = q / sqrt(q) and sqrt(g p / rho) = |g p| / sqrt(g p rho):
    // two reciprocal square roots, no division.  The reciprocal square root
    // wants a normal argument: q below 2^-998 (zero and the subnormal squares
    // of vanishing velocities ahead of a wave included) takes that bound, so
    // the speed stays below 2^-499 (0 for q = 0), which adds nothing to the
    // maximum; g p rho is clamped to [2^-998, 2^998], which changes nothing
    // but degenerate states (vacuum, or pressure and density both below
    // 1e-150), and where it is negative or NaN the sound speed is NaN, as the
    // reference's square root makes it (a NaN never wins the maximum)
    // (every product and sum is rounded on its own -- no contraction choice
    // left to the compiler -- so the init, final-sweep and ghost kernels give
    // the same bits for the same cell, and a resumed run the same dt)
    const double q = fma(du, du, __dmul_rn(dv, dv));
    const double velo = __dmul_rn(q, rrsqrt(fmax(q, 0x1p-998)));
    const double gp = __dmul_rn(g, double(p)), gpr = __dmul_rn(gp, double(rho));
    const double c = __dmul_rn(fabs(gp), rrsqrt(fmin(fmax(gpr, 0x1p-998), 0x1p998)));
    return __dadd_rn(velo, gpr >= 0.0 ? c : nan(""));
#else
    double velo = sqrt(du * du + dv * dv);
    double c = sqrt(g * double(p) / double(rho));
    return fabs(velo) + c;
#endif
}

} // namespace FVM2D_VARIANT
} // namespace fvm2d

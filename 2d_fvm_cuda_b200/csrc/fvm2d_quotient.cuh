// fvm2d_quotient.cuh -- the reference's operation order with its quotients
// from shared reciprocals, each correctly rounded: the same bits as division.
//
// The reference's interface divides by a variable up to 61 times, 44 of them
// by one of six values (both densities, both wave impedances, their sum,
// gamma - 1).  An IEEE division is 20 instructions and a branch to its slow
// path, so the contraction-free step issued 1990 instructions for 32
// interfaces where the product build issues 480.  Here a divisor b is inverted
// once, y = RN(1/b) and the rest yl of 1/b - y, and a quotient takes
//   q0 = RN(a y + a yl)     within (1/2 + 2^-50) units in the last place of a/b
//   r  = a - b q0           exact, q0 being faithful
//   q  = RN(q0 + r y)       = RN(a/b)
// which is Markstein's theorem (IBM J. Res. Dev. 34, 1990; Muller et al.,
// Handbook of Floating-Point Arithmetic, on division with an FMA): with y the
// correctly rounded reciprocal and q0 a faithful quotient, q is the correctly
// rounded one, as long as nothing over- or underflows.  So b must lie in
// [2^-60, 2^60] and a be zero or in [2^-900, 2^900] in magnitude; the sign of
// a zero is a's, b being positive.  Where an interface or an update meets
// anything else (NaN, vacuum, velocities that vanish ahead of a wave) it is
// computed once more with division.
#pragma once

#include "fvm2d_math.cuh"

namespace fvm2d {
namespace FVM2D_VARIANT {

__device__ __forceinline__ unsigned int high_word(double x)
{
#if defined(__CUDA_ARCH__)
    return (unsigned int)__double2hiint(x);
#else
    unsigned long long b;
    memcpy(&b, &x, 8);
    return (unsigned int)(b >> 32);
#endif
}
__device__ __forceinline__ unsigned int low_word(double x)
{
#if defined(__CUDA_ARCH__)
    return (unsigned int)__double2loint(x);
#else
    unsigned long long b;
    memcpy(&b, &x, 8);
    return (unsigned int)b;
#endif
}

// A divisor and its reciprocal y + yl; ok: false once anything was out of range.
struct Divisor {
    double b, y, yl;
    __device__ __forceinline__ Divisor(double x, double rx, bool &ok) : b(x), y(rx)
    {
        yl = fma(-b, y, 1.0) * y;
        ok = ok & (high_word(b) - 0x3c300000u <= 0x07800000u);
    }
#if defined(__CUDA_ARCH__)
    __device__ __forceinline__ Divisor(double x, bool &ok) : Divisor(x, __drcp_rn(x), ok) {}
#else
    __device__ __forceinline__ Divisor(double x, bool &ok) : Divisor(x, 1.0 / x, ok) {}
#endif
};

__device__ __forceinline__ double quotient(double a, const Divisor &d, bool &ok)
{
    const double q0 = fma(a, d.y, a * d.yl);
    const double q = fma(fma(-d.b, q0, a), d.y, q0);
    const unsigned int h = high_word(a) & 0x7fffffffu;
    ok = ok & ((h - 0x07b00000u <= 0x70800000u) | ((h | low_word(a)) == 0u));
    return copysign(q, a);
}

// relaxation_grp, expression by expression.
__device__ __forceinline__ Interface<double> relaxation_grp_shared(const Cell<double> &L, const Cell<double> &R,
                                                                   const Cell<double> &sL, const Cell<double> &sR,
                                                                   double g, double gm1, double igm1, bool &ok)
{
    const double rho_l = L.rho, pi_l = L.p, u_l = L.un, v_l = L.ut;
    const double rho_r = R.rho, pi_r = R.p, u_r = R.un, v_r = R.ut;
    const double rho_lx = sL.rho, pi_lx = sL.p, u_lx = sL.un, v_lx = sL.ut;
    const double rho_rx = sR.rho, pi_rx = sR.p, u_rx = sR.un, v_rx = sR.ut;
    const Divisor G(gm1, igm1, ok), Dl(rho_l, ok), Dr(rho_r, ok);
    auto by = [&](double a, const Divisor &d) { return quotient(a, d, ok); };

    // the internal energy and its slope, wanted on the contact's side only
    auto energy = [&](double pi, const Divisor &d) { return by(by(pi, d), G); };
    auto energy_x = [&](double pi_x, double pi, double rho_x, const Divisor &d) {
        return by(by(pi_x, d), G) - by(by(by(pi * rho_x, d), d), G);
    };
    const double c_lx = 0.5 * sqrt(by(g / pi_l, Dl)) * (pi_l * rho_lx + rho_l * pi_lx);
    const double c_rx = 0.5 * sqrt(by(g / pi_r, Dr)) * (pi_r * rho_rx + rho_r * pi_rx);

    Interface<double> o;
    double c_l, c_r;
    const double a_l = sqrt(by(g * pi_l, Dl)), a_r = sqrt(by(g * pi_r, Dr));
    const double kappa = (g + 1.0) / 2.0;
    // the side of the larger pressure's neighbour comes first (relaxation_grp);
    // its impedance divides again in the star region
    const bool left_first = pi_r >= pi_l;
    const double dp = left_first ? pi_r - pi_l : pi_l - pi_r;
    const double rise = by(dp, left_first ? Dr : Dl) / (left_first ? a_r : a_l);
    const double c1 = (left_first ? rho_l : rho_r) *
                      ((left_first ? a_l : a_r) + kappa * rmax(0.0, rise + u_l - u_r));
    const Divisor D1(c1, ok);
    const double c2 = (left_first ? rho_r : rho_l) *
                      ((left_first ? a_r : a_l) +
                       kappa * rmax(0.0, by(left_first ? pi_l - pi_r : pi_r - pi_l, D1) + u_l - u_r));
    c_l = left_first ? c1 : c2;
    c_r = left_first ? c2 : c1;
    const double s_l = by(c_l, Dl), s_r = by(c_r, Dr);

    if (u_l - s_l >= 0.0) {
        o.rho = rho_l; o.p = pi_l; o.un = u_l; o.ut = v_l; o.e = energy(pi_l, Dl);
        o.rho_t = -rho_l * u_lx - u_l * rho_lx;
        o.un_t = -u_l * u_lx - by(pi_lx, Dl);
        o.e_t = -u_l * energy_x(pi_lx, pi_l, rho_lx, Dl) - by(pi_l, Dl) * u_lx;
        o.ut_t = -u_l * v_lx;
        o.p_t = -u_l * pi_lx - by(c_l * c_l, Dl) * u_lx;
    } else if (u_r + s_r <= 0.0) {
        o.rho = rho_r; o.p = pi_r; o.un = u_r; o.ut = v_r; o.e = energy(pi_r, Dr);
        o.rho_t = -rho_r * u_rx - u_r * rho_rx;
        o.un_t = -u_r * u_rx - by(pi_rx, Dr);
        o.e_t = -u_r * energy_x(pi_rx, pi_r, rho_rx, Dr) - by(pi_r, Dr) * u_rx;
        o.ut_t = -u_r * v_rx;
        o.p_t = -u_r * pi_rx - by(c_r * c_r, Dr) * u_rx;
    } else {
        const double u0 = 0.0;
        const Divisor S(c_l + c_r, ok), D2(c2, ok);
        const Divisor Cl = left_first ? D1 : D2, Cr = left_first ? D2 : D1;
        const double u = by(u_l * c_l + u_r * c_r + pi_l - pi_r, S);
        const double pi = by((u_l - u_r) * c_l * c_r + c_l * pi_r + c_r * pi_l, S);
        const double k_l = -pi_lx - c_l * u_lx + 0.5 * (u0 - u_l) * c_lx;
        const double k_r = -pi_rx + c_r * u_rx - 0.5 * (u0 - u_r) * c_rx;
        // (factors of two pass through a quotient exactly)
        const double cc_l = by(c_l * c_l, Dl), cc_r = by(c_r * c_r, Dr);
        const double d_l = -2.0 * cc_l * u_lx - 2.0 * s_l * pi_lx + s_l * (u0 - u_l) * c_lx;
        const double d_r = 2.0 * cc_r * u_rx - 2.0 * s_r * pi_rx + s_r * (u_r - u0) * c_rx;
        const double Dpi_Dt = by((c_r * d_l - c_l * d_r) * 0.5, S);
        o.p = pi;
        o.un = u;
        double rho, e;
        const double cl_cr = c_l * c_r;
        if (u <= 0.0) {
            rho = c_r / (u_r - u + s_r);
            const double e_r = energy(pi_r, Dr);
            e = e_r + by(by((pi - pi_r) * (pi + pi_r) * 0.5, Cr), Cr);
            o.ut = v_r;
            const double ur = u * rho, m_l = 1.0 + by(ur, Cr);
            o.rho_t = -u * rho * rho * rho / (rho_r * c_r * c_r) *
                          (by(cc_r, Dr) * rho_rx - c_r * u_rx + 1.5 * (u - u_r) * c_rx) +
                      rho * rho * rho / (c_r * c_r * c_r) * (u + c_r / rho) * Dpi_Dt;
            o.p_t = S.y * (by(cl_cr, Dl) * m_l * k_l - by(cl_cr, Dr) * (1.0 - by(ur, Cl)) * k_r);
            o.un_t = S.y * (s_l * m_l * k_l + s_r * (1.0 - by(by(ur * c_l, Cr), Cr)) * k_r);
            o.e_t = by(by(by(by(-u * rho, Dr), Cr), Cr), Cr) *
                        (-pi_r * c_r * pi_rx + c_r * c_r * c_r * energy_x(pi_rx, pi_r, rho_rx, Dr) +
                         2.0 * (e_r - e) * c_r * c_r * c_rx) +
                    by(by(pi, Cr), Cr) * o.p_t;
            o.ut_t = -u * (by(rho, Dr) * v_rx);
        } else {
            rho = c_l / (u - u_l + s_l);
            const double e_l = energy(pi_l, Dl);
            e = e_l + by(by((pi - pi_l) * (pi + pi_l) * 0.5, Cl), Cl);
            o.ut = v_l;
            const double ur = u * rho, m_r = 1.0 - by(ur, Cl);
            o.rho_t = -u * rho * rho * rho / (rho_l * c_l * c_l) *
                          (by(cc_l, Dl) * rho_lx + c_l * u_lx + 1.5 * (u - u_l) * c_lx) -
                      rho * rho * rho / (c_l * c_l * c_l) * (u - c_l / rho) * Dpi_Dt;
            o.p_t = S.y * (by(cl_cr, Dl) * (1.0 + by(ur, Cr)) * k_l - by(cl_cr, Dr) * m_r * k_r);
            o.un_t = S.y * (s_l * (1.0 + by(by(ur * c_r, Cl), Cl)) * k_l + s_r * m_r * k_r);
            o.e_t = by(by(by(by(-u * rho, Dl), Cl), Cl), Cl) *
                        (-pi_l * c_l * pi_lx + c_l * c_l * c_l * energy_x(pi_lx, pi_l, rho_lx, Dl) +
                         2.0 * (e_l - e) * c_l * c_l * c_lx) +
                    by(by(pi, Cl), Cl) * o.p_t;
            o.ut_t = -u * (by(rho, Dl) * v_lx);
        }
        o.rho = rho;
        o.e = e;
    }
    return o;
}

#if defined(__CUDACC__)
#define FVM2D_OUT_OF_LINE __noinline__
#else
#define FVM2D_OUT_OF_LINE
#endif
__device__ FVM2D_OUT_OF_LINE static Interface<double> relaxation_grp_divided(Cell<double> L, Cell<double> R,
                                                                             Cell<double> sL, Cell<double> sR, double g)
{
    return relaxation_grp(L, R, sL, sR, g);
}
__device__ FVM2D_OUT_OF_LINE static Cell<double> update_divided(Cell<double> U, Cell<double> FL, Cell<double> FR,
                                                                double lambda, double g)
{
    return conservative_update(U, FL, FR, lambda, g);
}

// RefOrder's bits, without most of its divisions.
struct RefOrderShared : RefOrder {
    template <class Consts>
    __device__ static __forceinline__ Cell<double> interface_flux(const Cell<double> &UL, const Cell<double> &UR,
                                                                  const Cell<double> &sL, const Cell<double> &sR,
                                                                  const Consts &K)
    {
        Cell<double> fL, fR;
        face_states(UL, UR, sL, sR, K.h, fL, fR);
        bool ok = true;
        Interface<double> w = relaxation_grp_shared(fL, fR, sL, sR, K.g, K.gm1, K.igm1, ok);
        if (!ok) w = relaxation_grp_divided(fL, fR, sL, sR, K.g);
        return midpoint_flux(w, K.k);
    }
    template <class Consts>
    __device__ static __forceinline__ Cell<double> update(const Cell<double> &U, const Cell<double> &FL,
                                                          const Cell<double> &FR, const Consts &K)
    {
        double m1 = U.rho * U.un, m3 = U.rho * U.ut;
        bool ok = true;
        double m2 = quotient(U.p, Divisor(K.gm1, K.igm1, ok), ok) + U.rho * (U.un * U.un + U.ut * U.ut) * 0.5;
        const double m0 = U.rho - (FR.rho - FL.rho) * K.lambda;
        m1 = m1 - (FR.p - FL.p) * K.lambda;
        m2 = m2 - (FR.un - FL.un) * K.lambda;
        m3 = m3 - (FR.ut - FL.ut) * K.lambda;
        const Divisor D(m0, ok);
        Cell<double> o;
        o.rho = m0;
        o.p = K.gm1 * (m2 - quotient(m1 * m1, D, ok) * 0.5 - quotient(m3 * m3, D, ok) * 0.5);
        o.un = quotient(m1, D, ok);
        o.ut = quotient(m3, D, ok);
        return ok ? o : update_divided(U, FL, FR, K.lambda, K.g);
    }
};

} // namespace FVM2D_VARIANT
} // namespace fvm2d

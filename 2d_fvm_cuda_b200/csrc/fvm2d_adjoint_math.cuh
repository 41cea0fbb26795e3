// fvm2d_adjoint_math.cuh -- reverse-mode (adjoint) versions of the per-cell
// and per-interface arithmetic of one sweep, for the builds with shared
// reciprocals (Hoisted in fvm2d_math.cuh), in the arithmetic type FVM2D_REAL.  Each function recomputes the
// forward values it needs and then applies the transposed Jacobian of the
// forward statements in reverse order.  Branches (limiter selection, wave
// cases, max(0, .)) follow the forward values, so the derivative is the one
// of the branch taken (almost everywhere).  dt is an input, not a variable:
// the time step is fixed while differentiating.
#pragma once

#include "fvm2d_math.cuh"

namespace fvm2d {
namespace FVM2D_VARIANT {

using A = FVM2D_REAL;

struct Cell5 {
    A rho, p, un, ut, e;
};

// ---- limiter -------------------------------------------------------------
// The slope itself (Hoisted's limiter) with its choice: which difference was
// selected (0 none, 1 central, 2 backward, 3 forward), for the adjoint.
__device__ __forceinline__ A slope_with_choice(A m, A c, A p, A hrh, A rha, int &choice)
{
    const A d1 = c - m, d2 = p - c, dc = p - m;
    const A a1 = fabs(d1), a2 = fabs(d2);
    const bool forward = a2 < a1;
    const A inner = rha * (forward ? a2 : a1), outer = fabs(dc) * hrh;
    const bool one_sided = inner < outer, sloped = d1 * d2 > A(0);
    choice = !sloped ? 0 : !one_sided ? 1 : forward ? 3 : 2;
    return sloped ? copysign(one_sided ? inner : outer, dc) : A(0);
}

// The adjoints a slope component passes to its right cell (the return value)
// and left cell (mbar); its own cell gets minus their sum.
__device__ __forceinline__ A slope_parts(int choice, A sbar, A hrh, A rha, A &mbar)
{
    const A x = (choice == 1 ? hrh : rha) * sbar;
    mbar = choice == 1 || choice == 2 ? -x : A(0);
    return choice & 1 ? x : A(0);
}

#if !defined(__CUDACC__)  // host builds: the limiter's choice and adjoint each by itself, for tests
// s = Hoisted::slope's limiter (limited_slope_hoisted) on (m, c, p): which
// difference was selected (0 none, 1 central, 2 backward, 3 forward), for the
// adjoint.  Same tests and tie order (d1 d2 > 0 alone: it implies dc d2 > 0).
__device__ __forceinline__ int slope_choice(A m, A c, A p, A rh, A alpha)
{
    const A d1 = c - m, d2 = p - c, dc = p - m;
    if (!(d1 * d2 > A(0))) return 0;
    const A a1 = fabs(d1), a2 = fabs(d2);
    const A inner = (rh * alpha) * ((a2 < a1) ? a2 : a1);
    if (!(inner < fabs(dc) * (rh * A(0.5)))) return 1;
    return (a2 < a1) ? 3 : 2;
}

// Adds the adjoint of one slope component (sbar) to its three cells.
__device__ __forceinline__ void slope_adjoint(int choice, A sbar, A rh, A alpha, A &mbar, A &cbar, A &pbar)
{
    if (choice == 1) {
        pbar += A(0.5) * rh * sbar;
        mbar -= A(0.5) * rh * sbar;
    } else if (choice == 2) {
        cbar += rh * alpha * sbar;
        mbar -= rh * alpha * sbar;
    } else if (choice == 3) {
        pbar += rh * alpha * sbar;
        cbar -= rh * alpha * sbar;
    }
}
#endif

// ---- conservative update ---------------------------------------------------
// Adjoint of Hoisted::update.  Given the output adjoint Ub (rho, p, un, ut),
// adds the adjoint of the input cell to Uin_b and returns the adjoint of the
// post-update conserved vector m' (slots mass, normal momentum, energy,
// tangential momentum); the flux adjoints are then +lambda mb' for F_L and
// -lambda mb' for F_R.
__device__ __forceinline__ Cell<A> update_adjoint(const Cell<A> &U, const Cell<A> &FL, const Cell<A> &FR,
                                                  const SweepConsts<A> &K, const Cell<A> &Ub, Cell<A> &Uin_b)
{
    const A half = A(0.5), gm1 = K.g - A(1);
    // forward
    const A m1 = U.rho * U.un, m3 = U.rho * U.ut;
    const A n0 = U.rho - (FR.rho - FL.rho) * K.lambda;
    const A n1 = m1 - (FR.p - FL.p) * K.lambda;
    const A n3 = m3 - (FR.ut - FL.ut) * K.lambda;
    const A ir = rrcp(n0);
    // reverse of the primitive recovery
    A n0b = Ub.rho, n1b = ir * Ub.un, n3b = ir * Ub.ut, n2b = gm1 * Ub.p;
    A irb = n1 * Ub.un + n3 * Ub.ut;
    n1b += -gm1 * n1 * ir * Ub.p;
    n3b += -gm1 * n3 * ir * Ub.p;
    irb += -gm1 * half * (n1 * n1 + n3 * n3) * Ub.p;
    n0b += -ir * ir * irb;
    // m' = m - lambda (F_R - F_L): dm = dm'
    // conserved from primitive
    Uin_b.rho += n0b + U.un * n1b + U.ut * n3b + half * (U.un * U.un + U.ut * U.ut) * n2b;
    Uin_b.un += U.rho * n1b + U.rho * U.un * n2b;
    Uin_b.ut += U.rho * n3b + U.rho * U.ut * n2b;
    Uin_b.p += K.igm1 * n2b;
    Cell<A> mb;
    mb.rho = n0b;
    mb.p = n1b;
    mb.un = n2b;
    mb.ut = n3b;
    return mb;
}

// ---- interface: face states, relaxation GRP, midpoint flux -------------------
// One side of an interface in Hoisted::grp's terms: the face state and its
// slopes, i = 1/(rho a), the relaxation speed c with ic = 1/c and s = c/rho,
// the sound-speed slope cx = (gamma/2) Y i with Y = p rho_x + rho p_x.
struct Side {
    A r, p, u, v, rx, px, ux, vx;
    A gp, i, Y, cx, c, ic, s;
};
// The adjoints of a side's quantities.
struct SideAdjoint {
    A r = 0, p = 0, u = 0, v = 0, rx = 0, px = 0, ux = 0, vx = 0, i = 0, cx = 0, c = 0, ic = 0, s = 0;
};

// Adjoint of Hoisted::flux_of at the interface state W and its derivative Wt.
__device__ __forceinline__ void flux_adjoint(const Cell5 &W, const Cell5 &Wt, A hk, const Cell<A> &Fb, Cell5 &Wb,
                                             Cell5 &Wtb)
{
    const A half = A(0.5);
    const A m = W.rho * W.un, M = fma(hk, fma(W.rho, Wt.un, W.un * Wt.rho), m), Q = fma(hk, Wt.p, W.p), hm = hk * m;
    const A es = fma(half, fma(W.un, W.un, W.ut * W.ut), W.e), et = fma(W.un, Wt.un, fma(W.ut, Wt.ut, Wt.e));
    // F = (M, M un + hm un_t + Q, es M + hm et + un Q + hk p un_t, M ut + hm ut_t)
    const A Mb = fma(W.un, Fb.p, fma(es, Fb.un, fma(W.ut, Fb.ut, Fb.rho))), Qb = fma(W.un, Fb.un, Fb.p);
    const A hmb = fma(Wt.un, Fb.p, fma(et, Fb.un, Wt.ut * Fb.ut));
    const A esb = M * Fb.un, etb = hm * Fb.un, he = hk * Fb.un;
    const A mb = fma(hk, hmb, Mb), mtb = hk * Mb;
    Wb.rho = fma(Wt.un, mtb, W.un * mb);
    Wb.p = fma(he, Wt.un, Qb);
    Wb.un = fma(M, Fb.p, fma(Q, Fb.un, fma(Wt.un, etb, fma(W.un, esb, fma(Wt.rho, mtb, W.rho * mb)))));
    Wb.ut = fma(M, Fb.ut, fma(Wt.ut, etb, W.ut * esb));
    Wb.e = esb;
    Wtb.rho = W.un * mtb;
    Wtb.p = hk * Qb;
    Wtb.un = fma(hm, Fb.p, fma(W.p, he, fma(W.un, etb, W.rho * mtb)));
    Wtb.ut = fma(hm, Fb.ut, W.ut * etb);
    Wtb.e = etb;
}

// Reverse of a fan that lies on one side: the interface state is the face
// state of side S.
__device__ __forceinline__ void one_sided_adjoint(const Side &S, SideAdjoint &b, A igm1, A hk, const Cell<A> &Fb)
{
    const A ir = rrcp(S.r), iri = ir * igm1, tp = S.p * ir, X = fma(-tp, S.rx, S.px), ex = X * iri, cs = S.c * S.s;
    const Cell5 W = {S.r, S.p, S.u, S.v, S.p * iri};
    const Cell5 Wt = {-fma(S.r, S.ux, S.u * S.rx), -fma(S.u, S.px, cs * S.ux), -fma(S.u, S.ux, S.px * ir),
                      -(S.u * S.vx), -fma(S.u, ex, tp * S.ux)};
    Cell5 Wb, Wtb;
    flux_adjoint(W, Wt, hk, Fb, Wb, Wtb);
    const A tr = -Wtb.rho, tn = -Wtb.un, te = -Wtb.e, tv = -Wtb.ut, tq = -Wtb.p;
    const A exb = S.u * te, Xb = iri * exb, tpb = fma(S.ux, te, -(S.rx * Xb)), irib = fma(S.p, Wb.e, X * exb);
    const A irb = fma(S.px, tn, fma(S.p, tpb, igm1 * irib));
    b.r = fma(S.ux, tr, Wb.rho) - ir * ir * irb;
    b.p = fma(iri, Wb.e, fma(ir, tpb, Wb.p));
    b.u = fma(S.rx, tr, fma(S.ux, tn, fma(ex, te, fma(S.vx, tv, fma(S.px, tq, Wb.un)))));
    b.v = Wb.ut;
    b.rx = fma(S.u, tr, -(tp * Xb));
    b.px = fma(ir, tn, fma(S.u, tq, Xb));
    b.ux = fma(S.r, tr, fma(S.u, tn, fma(tp, te, cs * tq)));
    b.vx = S.u * tv;
    const A uq = S.ux * tq;
    b.c = S.s * uq;
    b.s = S.c * uq;
}

// Reverse of the star region, on the contact's side S (SG = 1: right, -1:
// left; O the other side).  Forward, as Hoisted::grp has it:
//   z = 1 / (SG (u_s - u) + s_s), rho = c_s z, w = u z, h = 1 + SG w, q = rho / rho_s,
//   Sx = s_s^2 rho_sx - SG c_s u_sx + 3/2 (u - u_s) c_sx, rho_t = -z (z h nD + w q Sx),
//   P = b_o h, N = c_o - SG u rho, p_t = -isum (c_s P + b_s N),
//   H = 1 - SG w c_o ic_s, un_t = SG isum (b_s H - P),
//   E2 = (pm^2 - p_s^2) ic_s^2, e = p_s iri + E2 / 2, iri = igm1 / rho_s,
//   G = (p_sx - p_s rho_sx / rho_s) iri - ic_s (E2 c_sx + ic_s p_s p_sx),
//   e_t = pm ic_s^2 p_t - u q G, ut_t = -u q v_sx.
// Adds the adjoints of the sides' quantities; ub, pmb, nDb, bsb and bob
// receive those of u, pm, nD, b_s and b_o, and xb un_t un_tb + p_t p_tb,
// their part of isum's.
template <int SG>
__device__ __forceinline__ void star_adjoint(const Side &S, const Side &O, SideAdjoint &Sb, SideAdjoint &Ob, A u, A pm,
                                             A nD, A b_s, A b_o, A isum, A igm1, A hk, const Cell<A> &Fb, A &ub,
                                             A &pmb, A &nDb, A &bsb, A &bob, A &xb)
{
    const A one = A(1), half = A(0.5), sg = A(SG);
    const A z = rrcp(SG > 0 ? (S.u - u) + S.s : (u - S.u) + S.s);
    const A rho = S.c * z, w = u * z, h = fma(sg, w, one), irs = rrcp(S.r), q = rho * irs;
    const A du15 = A(1.5) * (u - S.u), ss = S.s * S.s;
    const A Sx = fma(ss, S.rx, fma(-sg * S.c, S.ux, du15 * S.cx));
    const A zh = z * h, wq = w * q, Kz = fma(zh, nD, wq * Sx);
    const A P = b_o * h, N = fma(-sg * u, rho, O.c), wc = w * O.c, H = fma(-sg * wc, S.ic, one);
    const A ic2 = S.ic * S.ic, dE = (pm - S.p) * (pm + S.p), E2 = dE * ic2;
    const A iri = irs * igm1, tp = S.p * irs, X = fma(-tp, S.rx, S.px), ppx = S.p * S.px;
    const A Y = fma(E2, S.cx, S.ic * ppx), G = fma(-S.ic, Y, X * iri), uq = u * q, pmi = pm * ic2;
    Cell5 W = {rho, pm, u, S.v, fma(half, E2, S.p * iri)}, Wt;
    Wt.rho = -(z * Kz);
    Wt.p = -(isum * fma(S.c, P, b_s * N));
    Wt.un = sg * isum * fma(b_s, H, -P);
    Wt.e = fma(pmi, Wt.p, -(uq * G));
    Wt.ut = -(uq * S.vx);
    Cell5 Wb, Wtb;
    flux_adjoint(W, Wt, hk, Fb, Wb, Wtb);
    // ut_t, e_t, e
    Sb.v = Wb.ut;
    Sb.vx = -(uq * Wtb.ut);
    const A uqb = -fma(S.vx, Wtb.ut, G * Wtb.e), Gb = -(uq * Wtb.e), pe = Wt.p * Wtb.e;
    pmb = fma(ic2, pe, Wb.p);
    const A ptb = fma(pmi, Wtb.e, Wtb.p);
    // G: X, Y
    const A Xb = iri * Gb, Yb = -(S.ic * Gb), m = S.ic * Yb, tpb = -(S.rx * Xb);
    const A E2b = fma(S.cx, Yb, half * Wb.e), f = (ic2 + ic2) * E2b;
    pmb = fma(pm, f, pmb);
    Sb.p = fma(iri, Wb.e, fma(S.px, m, fma(irs, tpb, -(S.p * f))));
    Sb.px = fma(S.p, m, Xb);
    Sb.cx = E2 * Yb;
    A icb = fma(ppx, Yb, -(Y * Gb));
    icb = fma(S.ic + S.ic, fma(dE, E2b, pm * pe), icb);  // ic2 = ic^2
    A irb = fma(S.p, tpb, igm1 * fma(S.p, Wb.e, X * Gb));
    // un_t
    const A j1 = sg * isum * Wtb.un, t1 = -(sg * b_s) * j1;
    A wb = O.c * S.ic * t1;
    icb = fma(wc, t1, icb);
    // p_t
    const A j2 = -(isum * ptb), Nb = b_s * j2, Pb = fma(S.c, j2, -j1);
    bsb = fma(H, j1, N * j2);
    Ob.c = fma(w * S.ic, t1, Nb);
    xb = fma(Wt.un, Wtb.un, Wt.p * ptb);
    bob = h * Pb;
    A rhob = fma(-sg * u, Nb, Wb.rho);
    // rho_t
    const A j3 = -(z * Wtb.rho), zhb = nD * j3, wqb = Sx * j3, Sxb = wq * j3;
    nDb = zh * j3;
    const A hb = fma(z, zhb, b_o * Pb), qb = fma(w, wqb, u * uqb);
    wb = fma(q, wqb, fma(sg, hb, wb));
    Sb.rx = fma(ss, Sxb, -(tp * Xb));
    Sb.ux = -(sg * S.c) * Sxb;
    Sb.cx = fma(du15, Sxb, Sb.cx);
    const A m5 = A(1.5) * S.cx * Sxb;
    rhob = fma(irs, qb, rhob);
    irb = fma(rho, qb, irb);
    // z, and through it rho, w, h
    const A zb = fma(h, zhb, fma(u, wb, fma(S.c, rhob, -(Kz * Wtb.rho)))), d = -(z * z) * zb;
    ub = fma(-sg * rho, Nb, fma(q, uqb, fma(z, wb, fma(-sg, d, Wb.un + m5))));
    Sb.u = fma(sg, d, -m5);
    Sb.s = fma(A(2) * S.s * S.rx, Sxb, d);
    Sb.c = fma(P, j2, fma(-sg * S.ux, Sxb, z * rhob));
    Sb.r = -(irs * irs) * irb;
    Sb.ic = icb;
}

// Reverse of the relaxation speeds: of the two sides the one computed first
// (from the other's i) and second (from the first's 1/c), e = the pressure
// rise from first to second.  zf, zs: the arguments of max(0, .).
__device__ __forceinline__ void speeds_adjoint(const Side &f, const Side &s, SideAdjoint &fb, SideAdjoint &sb, A e,
                                               A kappa, A zf, A zs, A &eb, A &dub)
{
    sb.c = fma(-(s.ic * s.ic), sb.ic, sb.c);
    sb.r = fma(s.s, sb.c, sb.r);
    sb.s = fma(s.r, sb.c, sb.s);
    const A ts = zs > A(0) ? kappa * sb.s : A(0);
    fb.ic = fma(-e, ts, fb.ic);
    fb.c = fma(-(f.ic * f.ic), fb.ic, fb.c);
    fb.r = fma(f.s, fb.c, fb.r);
    fb.s = fma(f.r, fb.c, fb.s);
    const A tf = zf > A(0) ? kappa * fb.s : A(0);
    sb.i = e * tf;
    fb.i = A(0);
    eb = fma(s.i, tf, -(f.ic * ts));
    dub += ts + tf;
}

// Reverse of a side's sound speed a = gp i (adjoint s), of cx and of
// i = 1/sqrt(gp rho), gp = gamma p.
__device__ __forceinline__ void sound_adjoint(const Side &S, SideAdjoint &b, A g)
{
    const A hg = A(0.5) * g, t = hg * S.i * b.cx;
    const A ib = fma(hg * S.Y, b.cx, fma(S.gp, b.s, b.i));
    const A yb = A(-0.5) * (S.i * S.i) * (S.i * ib);
    b.p = fma(S.rx, t, fma(g, fma(S.i, b.s, S.r * yb), b.p));
    b.r = fma(S.px, t, fma(S.gp, yb, b.r));
    b.rx = fma(S.p, t, b.rx);
    b.px = fma(S.r, t, b.px);
}

// The sides' i, cx, c, ic and s, the arguments of max(0, .) and 1/(c_l + c_r),
// each with the forward's own roundings, so that the reverse takes its
// branches: Hoisted::grp's grouping, in single precision Hoisted::fan.
template <typename Real>
__device__ __forceinline__ void side_speeds(Side &l, Side &r, const Cell<Real> &sL, const Cell<Real> &sR,
                                            const SweepConsts<Real> &K, Real du, Real dp, Real &zl, Real &zr, Real &isum)
{
    if constexpr (std::is_same<Real, float>::value) {
        const auto w = Hoisted::fan(Cell<Real>{l.r, l.p, l.u, l.v}, Cell<Real>{r.r, r.p, r.u, r.v}, sL, sR, K);
        l.i = w.il, l.cx = w.c_lx, l.c = w.c_l, l.ic = w.icl, l.s = w.sl;
        r.i = w.ir, r.cx = w.c_rx, r.c = w.c_r, r.ic = w.icr, r.s = w.sr;
        zl = w.zl, zr = w.zr, isum = w.isum;
    } else {
        const Real zero = Real(0), kappa = K.kappa, hg = Real(0.5) * K.g;
        l.i = rrsqrt(l.gp * l.r), r.i = rrsqrt(r.gp * r.r);
        l.cx = l.Y * (hg * l.i), r.cx = r.Y * (hg * r.i);
        if (r.p >= l.p) {
            zl = fma(dp, r.i, du);
            l.s = fma(kappa, rmax(zero, zl), l.gp * l.i);
            l.c = l.r * l.s;
            l.ic = rrcp(l.c);
            zr = fma(-dp, l.ic, du);
            r.s = fma(kappa, rmax(zero, zr), r.gp * r.i);
            r.c = r.r * r.s;
            const Real sc = l.c + r.c, q = rrcp(r.c * sc);
            r.ic = sc * q;
            isum = r.c * q;
        } else {
            zr = fma(-dp, l.i, du);
            r.s = fma(kappa, rmax(zero, zr), r.gp * r.i);
            r.c = r.r * r.s;
            r.ic = rrcp(r.c);
            zl = fma(dp, r.ic, du);
            l.s = fma(kappa, rmax(zero, zl), l.gp * l.i);
            l.c = l.r * l.s;
            const Real sc = l.c + r.c, q = rrcp(l.c * sc);
            l.ic = sc * q;
            isum = l.c * q;
        }
    }
}
template <typename Real>
__device__ __forceinline__ Real contact_speed(const Side &l, const Side &r, Real dp, Real isum)
{
    if constexpr (std::is_same<Real, float>::value)
        return Hoisted::contact_speed(l.u, l.c, l.p, r.u, r.c, r.p, isum);
    else
        return (fma(l.u, l.c, r.u * r.c) - dp) * isum;
}
template <typename Real>
__device__ __forceinline__ Real contact_pressure(const Side &l, const Side &r, Real du, Real isum)
{
    if constexpr (std::is_same<Real, float>::value)
        return Hoisted::contact_pressure(du, l.c, l.p, r.c, r.p, isum);
    else
        return fma(du * l.c, r.c, fma(l.c, r.p, r.c * l.p)) * isum;
}

// Adjoint of Hoisted::interface_flux(UL, UR, sL, sR): given the flux adjoint
// Fb (slots mass, normal momentum, energy, tangential momentum), adds the
// adjoints of the two cells and the two slopes.  The forward is recomputed
// as Hoisted::grp has it, so the reverse takes the forward's branches.
__device__ __forceinline__ void interface_flux_adjoint(const Cell<A> &UL, const Cell<A> &UR, const Cell<A> &sL,
                                                       const Cell<A> &sR, const SweepConsts<A> &K, const Cell<A> &Fb,
                                                       Cell<A> &ULb, Cell<A> &URb, Cell<A> &sLb, Cell<A> &sRb)
{
    const A half = A(0.5), zero = A(0);
    const A g = K.g, igm1 = K.igm1, kappa = K.kappa, hk = K.k * half, hh = K.h * half;
    Side l, r;
    l.r = fma(sL.rho, hh, UL.rho), l.p = fma(sL.p, hh, UL.p), l.u = fma(sL.un, hh, UL.un), l.v = fma(sL.ut, hh, UL.ut);
    r.r = fma(-sR.rho, hh, UR.rho), r.p = fma(-sR.p, hh, UR.p), r.u = fma(-sR.un, hh, UR.un);
    r.v = fma(-sR.ut, hh, UR.ut);
    l.rx = sL.rho, l.px = sL.p, l.ux = sL.un, l.vx = sL.ut;
    r.rx = sR.rho, r.px = sR.p, r.ux = sR.un, r.vx = sR.ut;
    l.gp = g * l.p, r.gp = g * r.p;
    l.Y = fma(l.p, l.rx, l.r * l.px), r.Y = fma(r.p, r.rx, r.r * r.px);
    const A du = l.u - r.u, dp = r.p - l.p;
    const bool left_first = r.p >= l.p;
    A zl, zr, isum;
    side_speeds(l, r, sL, sR, K, du, dp, zl, zr, isum);
    SideAdjoint lb, rb;
    A dub = zero, dpb = zero;
    if (l.u - l.s >= zero) {
        one_sided_adjoint(l, lb, igm1, hk, Fb);
    } else if (r.u + r.s <= zero) {
        one_sided_adjoint(r, rb, igm1, hk, Fb);
    } else {
        const A u = contact_speed(l, r, dp, isum);
        const A pm = contact_pressure(l, r, du, isum);
        const A Bl = fma(half * l.u, l.cx, fma(l.c, l.ux, l.px)), Br = fma(half * r.u, r.cx, fma(r.c, r.ux, -r.px));
        const A b_l = l.s * Bl, b_r = r.s * Br, nD = fma(r.c, b_l, l.c * b_r) * isum;
        A ub, pmb, nDb, blb, brb, xb;
        if (u <= zero)
            star_adjoint<1>(r, l, rb, lb, u, pm, nD, b_r, b_l, isum, igm1, hk, Fb, ub, pmb, nDb, brb, blb, xb);
        else
            star_adjoint<-1>(l, r, lb, rb, u, pm, nD, b_l, b_r, isum, igm1, hk, Fb, ub, pmb, nDb, blb, brb, xb);
        // nD, u and pm are brackets times isum = 1/(c_l + c_r), whose adjoint
        // reaches c_l and c_r as -isum sum(X Xb)
        const A jD = isum * nDb, ju = isum * ub, jp = isum * pmb;
        const A jc = -(isum * fma(u, ub, fma(pm, pmb, fma(nD, nDb, xb))));
        blb = fma(r.c, jD, blb);
        brb = fma(l.c, jD, brb);
        const A tl = l.s * blb, tr = r.s * brb;
        lb.c += fma(b_r, jD, fma(l.u, ju, fma(fma(du, r.c, r.p), jp, fma(l.ux, tl, jc))));
        rb.c += fma(b_l, jD, fma(r.u, ju, fma(fma(du, l.c, l.p), jp, fma(r.ux, tr, jc))));
        lb.p += r.c * jp;
        rb.p += l.c * jp;
        dub = l.c * r.c * jp;
        dpb = -ju;
        // b = s B
        lb.s = fma(Bl, blb, lb.s);
        rb.s = fma(Br, brb, rb.s);
        lb.u += fma(l.c, ju, half * l.cx * tl);
        rb.u += fma(r.c, ju, half * r.cx * tr);
        lb.cx = fma(half * l.u, tl, lb.cx);
        rb.cx = fma(half * r.u, tr, rb.cx);
        lb.ux = fma(l.c, tl, lb.ux);
        rb.ux = fma(r.c, tr, rb.ux);
        lb.px += tl;
        rb.px -= tr;
    }
    A eb;
    if (left_first) {
        speeds_adjoint(l, r, lb, rb, dp, kappa, zl, zr, eb, dub);
        dpb += eb;
    } else {
        speeds_adjoint(r, l, rb, lb, -dp, kappa, zr, zl, eb, dub);
        dpb -= eb;
    }
    sound_adjoint(l, lb, g);
    sound_adjoint(r, rb, g);
    lb.u += dub;
    rb.u -= dub;
    lb.p -= dpb;
    rb.p += dpb;
    // face states
    ULb.rho += lb.r;
    ULb.p += lb.p;
    ULb.un += lb.u;
    ULb.ut += lb.v;
    URb.rho += rb.r;
    URb.p += rb.p;
    URb.un += rb.u;
    URb.ut += rb.v;
    sLb.rho += fma(hh, lb.r, lb.rx);
    sLb.p += fma(hh, lb.p, lb.px);
    sLb.un += fma(hh, lb.u, lb.ux);
    sLb.ut += fma(hh, lb.v, lb.vx);
    sRb.rho += fma(-hh, rb.r, rb.rx);
    sRb.p += fma(-hh, rb.p, rb.px);
    sRb.un += fma(-hh, rb.u, rb.ux);
    sRb.ut += fma(-hh, rb.v, rb.vx);
}

} // namespace FVM2D_VARIANT
} // namespace fvm2d

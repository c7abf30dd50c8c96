// fast64.cuh -- the plain path's physics with fewer FP64 operations.
//
// The plain path must round as the reference's CPU build does, and it is
// bound by the FP64 pipe, on which one operation costs as much as 64 others
// (0.5 lanes per clock and scheduler, measured; 128 lanes per clock and SM
// elsewhere).  The functions here return the bits of their counterparts in
// physics_fp64.cuh (which name the reference's routines) from a third of the
// FP64 operations:
//  * divisions and square roots in integers (ieee64.cuh), those by one divisor
//    sharing its reciprocal;
//  * each zone's slopes once, for the faces on both of its sides;
//  * multiplications by powers of two on the exponent, comparisons on the bit
//    patterns;
//  * the face normal at compile time: a product with one of its zeros is a
//    zero, of which only the sign can matter, and that is kept (add_zero).
//    The y normal keeps its x component cos(pi/2) = 6.1e-17;
//  * eigenvalues only where they can be the largest or the smallest: rounding
//    is monotone, so e.g. max(vn - c, vn, vn + c) is RN(vn + c).
// They hold for ordinary operands: zero or of magnitude 2^-300 to 2^200
// (ordinary()), positive densities and pressures, no division by zero.
// Anything else clears `ok`, and the caller repeats the face or zone with the
// general functions, so NaNs, infinities and error codes stay theirs.
#pragma once

#include "ieee64.cuh"
#include "physics_fp64.cuh"

#define F64_FN __device__ __forceinline__

namespace mara {
namespace fast64 {

using ieee64::Divisor;
using ieee64::bits;
using ieee64::from_bits;
typedef ieee64::u32 u32;
typedef ieee64::u64 u64;

constexpr u64 SIGN = 0x8000000000000000ull;

F64_FN u64 mag(double x) { return bits(x) & ~SIGN; }
F64_FN bool is_zero(double x) { return (bits(x) << 1) == 0; }
F64_FN bool sign_bit(double x) { return (bits(x) >> 63) != 0; }
F64_FN u32 expo(double x) { return (u32) (bits(x) >> 52) & 0x7ffu; }

// zero, or of magnitude 2^-300 .. 2^201: products and quotients of a few of
// these stay far inside the normal range, and so do their non-zero differences
F64_FN bool ordinary(double x) { return expo(x) - 723u <= 500u || is_zero(x); }

// x 2^k for ordinary x (and what ordinary values were combined to)
F64_FN double scale(double x, int k)
{
    return is_zero(x) ? x : from_bits(bits(x) + ((u64) (ieee64::i64) k << 52));
}
F64_FN double half(double x) { return scale(x, -1); }

// x + z for a zero z of the given sign: x, or the zero the addition gives
F64_FN double add_zero(double x, bool z_negative)
{
    return is_zero(x) ? from_bits(z_negative ? bits(x) : 0ull) : x;
}

// the larger of two non-negative finite values, the smaller of two
// non-positive ones (a zero counts as +0)
F64_FN double max_pos(double a, double b) { return bits(a) > bits(b) ? a : b; }
F64_FN double min_neg(double a, double b) { return bits(a) > bits(b) ? a : b; }
// max(x, +0) and min(x, +0) for x without -0
F64_FN double clamp_pos(double x) { return sign_bit(x) ? 0.0 : x; }
F64_FN double clamp_neg(double x) { return sign_bit(x) ? x : 0.0; }

// The constants of a run that the functions use (one copy per kernel launch).
struct Consts {
    double gamma, gm1, theta, ny0;   // ny0: x component of the y normal
    double shenzha_A;
    int weno_is;
    Divisor gm1_div;
    bool ok;                         // the constants themselves are ordinary
};

// ---------------------------------------------------------------------------
// The generalised minmod's half slope, 0.5 minmod(theta, l, c, r), from its
// one-sided differences a = theta (c - l), d = theta (r - c) and r - l.  The
// reference's factor 0.25 |sgn a + sgn b| (sgn a + sgn d) is 0 or +-1 unless
// one of the three vanishes, and then their minimum is 0; a zero result has
// the sign of the factor.
F64_FN double half_slope(double a, double rl, double d)
{
    const u64 xa = mag(a), xd = mag(d);
    const u64 xb = mag(half(rl));
    u64 m = xa < xd ? xa : xd;
    m = m < xb ? m : xb;
    const bool same = ((bits(a) ^ bits(d)) >> 63) == 0 && ((bits(a) ^ bits(rl)) >> 63) == 0;
    const int sa = xa == 0 ? 0 : sign_bit(a) ? -1 : 1, sd = xd == 0 ? 0 : sign_bit(d) ? -1 : 1;
    const u64 neg = sa + sd < 0 ? SIGN : 0ull;
    return from_bits((same && m != 0 ? m - (1ull << 52) : 0ull) | neg);
}

// weno5 at both edges of a zone, from v[-2 .. 2] of magnitude below 2^61: the
// smoothness indicators and the products that both edges use once
F64_FN bool weno_ordinary(double x) { return expo(x) - 723u <= 360u || is_zero(x); }

F64_FN double sq(double x) { return x * x; }

F64_FN void weno5_edges(const Consts& c, const double* v, double& left, double& right, bool& ok)
{
    const double q = 1. / 4., t = 13. / 12.;
    double B0 = t * sq(v[0] - scale(v[1], 1) + v[2]) + q * sq(3 * v[0] - scale(v[1], 2) + v[2]);
    double B1 = t * sq(v[-1] - scale(v[0], 1) + v[1]) + q * sq(v[-1] - v[1]);
    double B2 = t * sq(v[-2] - scale(v[-1], 1) + v[0]) + q * sq(v[-2] - scale(v[-1], 2) + 3 * v[0]);
    // w = d / e for the three stencils
    double wl[3], wr[3];
    if (c.weno_is == WENO_BORGES08) {
        const double eps = 1e-14;
        const double tau5 = fabs(B0 - B2);
        const double r0 = 1.0 + ieee64::div(tau5, B0 + eps, ok);
        const double r1 = 1.0 + ieee64::div(tau5, B1 + eps, ok);
        const double r2 = 1.0 + ieee64::div(tau5, B2 + eps, ok);
        wr[0] = 0.3 * r0; wr[1] = 0.6 * r1; wr[2] = 0.1 * r2;
        wl[0] = 0.1 * r0; wl[1] = wr[1]; wl[2] = 0.3 * r2;
    } else {
        double ep = 1e-6;
        if (c.weno_is == WENO_SHENZHA10) {
            ep = 1e-10;
            const double lo = bits(B0) < bits(B1) ? (bits(B0) < bits(B2) ? B0 : B2) : (bits(B1) < bits(B2) ? B1 : B2);
            const double hi = max_pos(max_pos(B0, B1), B2);
            const double add = ieee64::div(lo, hi + ep, ok) * c.shenzha_A * lo;
            B0 = add + B0;
            B1 = add + B1;
            B2 = add + B2;
        }
        const Divisor e0 = ieee64::divisor(sq(ep + B0), ok);
        const Divisor e1 = ieee64::divisor(sq(ep + B1), ok);
        const Divisor e2 = ieee64::divisor(sq(ep + B2), ok);
        wr[0] = ieee64::div(0.3, e0, ok); wr[1] = ieee64::div(0.6, e1, ok); wr[2] = ieee64::div(0.1, e2, ok);
        wl[0] = ieee64::div(0.1, e0, ok); wl[1] = wr[1]; wl[2] = ieee64::div(0.3, e2, ok);
    }
    const double third = 1. / 3., sixth = 1. / 6., a56 = 5. / 6., a76 = 7. / 6., a116 = 11. / 6.;
    const double r0 = third * v[0] + a56 * v[1] - sixth * v[2];
    const double r1 = -sixth * v[-1] + a56 * v[0] + third * v[1];
    const double r2 = third * v[-2] - a76 * v[-1] + a116 * v[0];
    const double l0 = a116 * v[0] - a76 * v[1] + third * v[2];
    const double l1 = third * v[-1] + a56 * v[0] - sixth * v[1];
    const double l2 = -sixth * v[-2] + a56 * v[-1] + third * v[0];
    right = ieee64::div(wr[0] * r0 + wr[1] * r1 + wr[2] * r2, wr[0] + wr[1] + wr[2], ok);
    left = ieee64::div(wl[0] * l0 + wl[1] * l1 + wl[2] * l2, wl[0] + wl[1] + wl[2], ok);
}

// ---------------------------------------------------------------------------
// vector component along the normal of AXIS: x n0 + y n1 + z n2
template <int AXIS>
F64_FN double along(const Consts& c, double x, double y, double z)
{
    if constexpr (AXIS == 1) return add_zero(x * c.ny0 + y, sign_bit(z));
    const double v = AXIS == 0 ? x : z;
    return is_zero(v) ? from_bits(bits(x) & bits(y) & bits(z) & SIGN) : v;
}

// x + p n_d for the component d of the normal
template <int AXIS>
F64_FN double add_normal(const Consts& c, int d, double x, double p)
{
    if (d == AXIS) return x + p;
    if (AXIS == 1 && d == 0) return x + p * c.ny0;
    return add_zero(x, sign_bit(p));
}

// a product v_n x with v_n = along(v): P0 v_axis is already there for a flux
// along a coordinate axis (y's normal has two components)
template <int AXIS>
F64_FN double times_along(double vn, double x, double x_times_axis)
{
    if constexpr (AXIS == 1) return vn * x;
    return is_zero(vn) ? from_bits((bits(vn) ^ bits(x)) & SIGN) : x_times_axis;
}

// One side of a face: primitives, conserved densities, fluxes and the clamped
// extreme wave speeds (slot_max, slot_min of physics_fp64.cuh).
template <int NQ> struct Side {
    double U[NQ], F[NQ];
    double vn, ap, am;
};

// hydro_prim
template <int AXIS>
F64_FN void hydro_side(const Consts& c, const double* P, Side<5>& S, bool& ok)
{
    const double cs = ieee64::sqrt_rn(ieee64::div(c.gamma * P[4], P[0], ok), ok);
    const double vv = P[1] * P[1] + P[2] * P[2] + P[3] * P[3];
    const double vn = along<AXIS>(c, P[1], P[2], P[3]);
    S.vn = vn;
    S.U[0] = P[0];
    S.U[1] = P[0] * P[1];
    S.U[2] = P[0] * P[2];
    S.U[3] = P[0] * P[3];
    S.U[4] = half(P[0] * vv) + ieee64::div(P[4], c.gm1_div, ok);
    S.F[0] = times_along<AXIS>(vn, S.U[0], S.U[1 + AXIS]);
    S.F[1] = add_normal<AXIS>(c, 0, vn * S.U[1], P[4]);
    S.F[2] = add_normal<AXIS>(c, 1, vn * S.U[2], P[4]);
    S.F[3] = add_normal<AXIS>(c, 2, vn * S.U[3], P[4]);
    S.F[4] = vn * S.U[4] + P[4] * vn;
    S.ap = clamp_pos(vn + cs);
    S.am = clamp_neg(vn - cs);
    ok = ok && !is_zero(cs);
}

// mhd_prim; an auxiliary field (index 8) is carried without a flux
template <int AXIS, int NQ>
F64_FN void mhd_side(const Consts& c, const double* P, Side<NQ>& S, bool& ok)
{
    const Divisor rho = ieee64::divisor(P[0], ok);
    const double cs2 = ieee64::div(c.gamma * P[4], rho, ok);
    const double vv = P[1] * P[1] + P[2] * P[2] + P[3] * P[3];
    const double BB = P[5] * P[5] + P[6] * P[6] + P[7] * P[7];
    const double Bv = P[5] * P[1] + P[6] * P[2] + P[7] * P[3];
    const double vn = along<AXIS>(c, P[1], P[2], P[3]);
    const double Bn = along<AXIS>(c, P[5], P[6], P[7]);
    const double ps = P[4] + half(BB);
    S.vn = vn;
    S.U[0] = P[0];
#pragma unroll
    for (int d = 1; d < 4; ++d) S.U[d] = P[0] * P[d];
    S.U[4] = half(P[0] * vv) + half(BB) + ieee64::div(P[4], c.gm1_div, ok);
#pragma unroll
    for (int d = 5; d < NQ; ++d) S.U[d] = P[d];
    S.F[0] = times_along<AXIS>(vn, S.U[0], S.U[1 + AXIS]);
#pragma unroll
    for (int d = 0; d < 3; ++d) S.F[1 + d] = add_normal<AXIS>(c, d, vn * S.U[1 + d] - Bn * P[5 + d], ps);
    S.F[4] = vn * S.U[4] - Bn * Bv + ps * vn;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (AXIS != 1 && d == AXIS) {
            // v_n B_n - B_n v_n: +0, or the difference of two zeros
            const bool zero = is_zero(vn) || is_zero(Bn);
            const bool p = sign_bit(vn) != sign_bit(P[5 + d]), q = sign_bit(Bn) != sign_bit(P[1 + d]);
            S.F[5 + d] = from_bits(zero && p && !q ? SIGN : 0ull);
        } else {
            S.F[5 + d] = vn * S.U[5 + d] - Bn * P[1 + d];
        }
    }
    if constexpr (NQ > 8) S.F[8] = 0.0;
    // the fast speed; an Alfven speed that rounding puts above it wins
    const double ca2 = ieee64::div(BB, rho, ok);
    const double cn2 = ieee64::div(Bn * Bn, rho, ok);
    const double s = cs2 + ca2;
    const double cF2 = half(s + ieee64::sqrt_rn(s * s - scale(cs2 * cn2, 2), ok));
    const double cf = ieee64::sqrt_rn(max_pos(cF2, cn2), ok);
    S.ap = clamp_pos(vn + cf);
    S.am = clamp_neg(vn - cf);
    ok = ok && !is_zero(cf) && !sign_bit(P[4]);
}

template <int LAW, int AXIS>
F64_FN void side(const Consts& c, const double* P, Side<LawInfo<LAW>::NQ>& S, bool& ok)
{
    if constexpr (LAW == LAW_HYDRO) hydro_side<AXIS>(c, P, S, ok);
    else mhd_side<AXIS, LawInfo<LAW>::NQ>(c, P, S, ok);
}

// ---------------------------------------------------------------------------
template <int NQ>
F64_FN void hlle(const Side<NQ>& L, const Side<NQ>& R, double* F, bool& ok)
{
    const double ap = max_pos(L.ap, R.ap), am = min_neg(L.am, R.am);
    const Divisor den = ieee64::divisor(ap - am, ok);
    const double apam = ap * am;
#pragma unroll
    for (int q = 0; q < NQ; ++q)
        F[q] = ieee64::div(ap * L.F[q] - am * R.F[q] + apam * (R.U[q] - L.U[q]), den, ok);
}

// the star state of the side the contact moves away from, chosen first
template <int AXIS>
F64_FN void hllc(const Consts& c, const double* Pl, const double* Pr, const Side<5>& L, const Side<5>& R, double* F,
                 bool& ok)
{
    const double ap = max_pos(L.ap, R.ap), am = min_neg(L.am, R.am);
    const double sl = am - L.vn, sr = ap - R.vn;
    const double ml = Pl[0] * sl, mr = Pr[0] * sr;
    const double lc = ieee64::div((Pr[4] - R.F[0] * sr) - (Pl[4] - L.F[0] * sl), ml - mr, ok);
    const bool left = !sign_bit(lc) || is_zero(lc);
    const double s = left ? am : ap, m = left ? ml : mr, vn = left ? L.vn : R.vn;
    double P[5], U[5], G[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        P[q] = left ? Pl[q] : Pr[q];
        U[q] = left ? L.U[q] : R.U[q];
        G[q] = left ? L.F[q] : R.F[q];
    }
    const double f = ieee64::div(m, s - lc, ok);
    const double w = lc - vn;
    double Us[5];
    Us[0] = f;
    Us[4] = f * (ieee64::div(U[4], P[0], ok) + w * (lc + ieee64::div(P[4], m, ok)));
#pragma unroll
    for (int d = 0; d < 3; ++d) Us[1 + d] = f * add_normal<AXIS>(c, d, P[1 + d], w);
    const bool supersonic = is_zero(am);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        const double star = G[q] + s * (Us[q] - U[q]);
        F[q] = supersonic ? L.F[q] : star;
    }
}

// ---------------------------------------------------------------------------
// hydro_cons; mhd_cons where it accepts the state as it is
template <int LAW>
F64_FN void cons(const Consts& c, const double* U, double* P, bool& ok)
{
    constexpr int NQ = LawInfo<LAW>::NQ;
    const Divisor rho = ieee64::divisor(U[0], ok);
    const double p2 = U[1] * U[1] + U[2] * U[2] + U[3] * U[3];
    double e = U[4] - ieee64::div(half(p2), rho, ok);
    if constexpr (LAW != LAW_HYDRO) {
        e = e - half(U[5] * U[5] + U[6] * U[6] + U[7] * U[7]);
#pragma unroll
        for (int q = 5; q < NQ; ++q) P[q] = U[q];
        ok = ok && !sign_bit(e) && !sign_bit(U[0]) && !sign_bit(U[4]);
    }
    P[0] = U[0];
    P[4] = e * c.gm1;
#pragma unroll
    for (int q = 1; q < 4; ++q) P[q] = ieee64::div(U[q], rho, ok);
}

// hydro_p2u, mhd_p2u
template <int LAW>
F64_FN void p2u(const Consts& c, const double* P, double* U, bool& ok)
{
    constexpr int NQ = LawInfo<LAW>::NQ;
    const double vv = P[1] * P[1] + P[2] * P[2] + P[3] * P[3];
    U[0] = P[0];
#pragma unroll
    for (int d = 1; d < 4; ++d) U[d] = P[0] * P[d];
    double e = half(P[0] * vv);
    if constexpr (LAW != LAW_HYDRO) {
        e = e + half(P[5] * P[5] + P[6] * P[6] + P[7] * P[7]);
#pragma unroll
        for (int q = 5; q < NQ; ++q) U[q] = P[q];
    }
    U[4] = e + ieee64::div(P[4], c.gm1_div, ok);
}

// The largest max_eigen_magnitude over the three face normals: on each,
// RN(|vn| + c) with the fast speed c.
template <int LAW>
F64_FN double fastest(const Consts& c, const double* P, bool& ok)
{
    const double v[3] = {P[1], P[1] * c.ny0 + P[2], P[3]};
    const Divisor rho = ieee64::divisor(P[0], ok);
    const double cs2 = ieee64::div(c.gamma * P[4], rho, ok);
    if constexpr (LAW == LAW_HYDRO) {
        u64 vmax = mag(v[0]) > mag(v[1]) ? mag(v[0]) : mag(v[1]);
        vmax = vmax > mag(v[2]) ? vmax : mag(v[2]);
        return from_bits(vmax) + ieee64::sqrt_rn(cs2, ok);
    } else {
        const double BB = P[5] * P[5] + P[6] * P[6] + P[7] * P[7];
        const double B[3] = {P[5], P[5] * c.ny0 + P[6], P[7]};
        const double s = cs2 + ieee64::div(BB, rho, ok);
        const double s2 = s * s;
        double m = 0.0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double cn2 = ieee64::div(B[a] * B[a], rho, ok);
            const double cF2 = half(s + ieee64::sqrt_rn(s2 - scale(cs2 * cn2, 2), ok));
            m = max_pos(m, from_bits(mag(v[a])) + ieee64::sqrt_rn(max_pos(cF2, cn2), ok));
        }
        return m;
    }
}

} // namespace fast64
} // namespace mara

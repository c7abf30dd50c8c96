// fast64_rmhd.cuh -- relativistic MHD of the plain path with fewer FP64
// operations (see fast64.cuh): rmhd_prim, rmhd_cons and their eigenvalue
// checks, bit for bit the functions of physics_fp64.cuh where `ok` stays set.
//
// The quartic's pow(x, 1/3), acos, cos and sin take their first phase
// (ziv64.cuh) and only where that cannot round the hundreds of FP64
// operations of crmath.cuh.
#pragma once

#include "fast64.cuh"
#include "ziv64.cuh"

#if defined(__CUDACC__)
#define F64_COLD static __device__ __noinline__
#else
#define F64_COLD static
#endif

namespace mara {
namespace fast64 {

F64_COLD double acos_slow(double z) { return crm::acos_cr(z); }
F64_COLD double cos_slow(double t) { return crm::cos_cr(t); }
F64_COLD double sin_slow(double t) { return crm::sin_cr(t); }
F64_COLD double pow_third_slow(double x) { return crm::pow_third(x); }

// (s >= 0) ? pow(s, 1/3) : -pow(-s, 1/3)
F64_FN double signed_third(double s)
{
    bool ok = true;
    const double w = from_bits(mag(s));
    double r = ziv64::pow_third(w, ok);
    if (!ok) r = pow_third_slow(w);
    return sign_bit(s) && !is_zero(s) ? -r : r;
}

// The real root u1 of the resolvent cubic u^3 + a2 u^2 + a1 u + a0 that
// quartic_roots takes (solve_cubic with c3 = 1).
F64_FN double resolvent_root(const Consts& c, double a2, double a1, double a0, bool& ok)
{
    const double t = div(a2, c.d3, ok);   // a2 / 3
    const double q = div(a1, c.d3, ok) - div(a2 * a2, c.d9, ok);
    const double r = div(a1 * a2 - 3.0 * a0, c.d6, ok) - div(a2 * a2 * a2, c.d27, ok);
    const double delta = q * q * q + r * r;
    if (is_zero(delta)) {
        const double s = signed_third(r);
        const double x1 = 2.0 * s - t, x3 = -s - t;
        return x1 > x3 ? x1 : x3;
    }
    if (!sign_bit(delta)) {
        const double sd = sqrt_rn(delta, ok);
        return (signed_third(r + sd) + signed_third(r - sd)) - t;
    }
    const double z = div(r, sqrt_rn(-q * q * q, ok), ok);
    bool fine = true;
    double th = ziv64::arccos(z, fine);
    if (!fine) th = acos_slow(z);
    th = div(th, c.d3, ok);
    double cs, sn;
    fine = true;
    ziv64::sincos_third(th, cs, sn, fine);
    if (!fine) {
        cs = cos_slow(th);
        sn = sin_slow(th);
    }
    const double sq = sqrt_rn(-q, ok);
    const double x1 = 2.0 * sq * cs - t;
    const double x3 = -sq * cs - t + 1.7320508075688772 * sq * sn;
    return less(x3, x1) ? x1 : x3;
}

// The smallest and the largest real root of d4 x^4 + ... + d0 (quartic_roots);
// ok cleared where there is none.
F64_FN void quartic_range(const Consts& c, double d4, double d3, double d2, double d1, double d0, double& lo,
                          double& hi, bool& ok)
{
    const Divisor v = ieee64::divisor(d4, ok);
    const double a3 = div(d3, v, ok), a2 = div(d2, v, ok), a1 = div(d1, v, ok), a0 = div(d0, v, ok);
    const double u1 = resolvent_root(c, -a2, a1 * a3 - 4 * a0, 4.0 * a0 * a2 - a1 * a1 - a0 * a3 * a3, ok);
    const double R2 = 0.25 * a3 * a3 + u1 - a2;
    double R = 0.0, f1, f2;
    if (!sign_bit(R2) && !is_zero(R2)) {
        R = sqrt_rn(R2, ok);
        f1 = 0.75 * a3 * a3 - R2 - 2.0 * a2;
        f2 = div(0.25 * (4.0 * a3 * a2 - 8.0 * a1 - a3 * a3 * a3), R, ok);
    } else {
        f1 = 0.75 * a3 * a3 - 2.0 * a2;
        f2 = 2.00 * sqrt_rn(u1 * u1 - 4.0 * a0, ok);
    }
    const double D2 = f1 + f2, E2 = f1 - f2;
    const double b = -0.25 * a3, h = 0.5 * R;
    bool any = false;
    if (!sign_bit(D2) || is_zero(D2)) {
        const double D = sqrt_rn(D2, ok);
        lo = b + h - 0.5 * D;
        hi = b + h + 0.5 * D;
        any = true;
    }
    if (!sign_bit(E2) || is_zero(E2)) {
        const double E = sqrt_rn(E2, ok);
        const double l = b - h - 0.5 * E, m = b - h + 0.5 * E;
        lo = any && less(lo, l) ? lo : l;
        hi = any && less(m, hi) ? hi : m;
        any = true;
    }
    ok = ok && any;
}

// What rmhd_prim forms of a state before its fluxes.
struct RmhdState {
    double vv, BB, vn, Bn, W2, W0, b0, bb, b[3], bn, ps, h0, hs;
};

template <int AXIS>
F64_FN void rmhd_state(const Consts& c, const double* P, RmhdState& s, bool& ok)
{
    s.vv = P[1] * P[1] + P[2] * P[2] + P[3] * P[3];
    s.BB = P[5] * P[5] + P[6] * P[6] + P[7] * P[7];
    const double Bv = P[5] * P[1] + P[6] * P[2] + P[7] * P[3];
    s.vn = along<AXIS>(c, P[1], P[2], P[3]);
    s.Bn = along<AXIS>(c, P[5], P[6], P[7]);
    ok = ok && less(s.vv, 1.0) && edge_pos(P[0]) && edge_pos(P[4]);
    s.W2 = div(1.0, 1.0 - s.vv, ok);
    s.W0 = sqrt_rn(s.W2, ok);
    s.b0 = s.W0 * Bv;
    s.bb = div(s.BB + s.b0 * s.b0, s.W2, ok);
    const Divisor W = ieee64::divisor(s.W0, ok);
    const double k = s.b0 * s.W0;
#pragma unroll
    for (int d = 0; d < 3; ++d) s.b[d] = div(P[5 + d] + k * P[1 + d], W, ok);
    ok = ok && steep(s.b[0]) && (is_zero(s.bb) || expo(s.bb) > 1);   // for along() and half()
    s.bn = along<AXIS>(c, s.b[0], s.b[1], s.b[2]);
    const Divisor rho = ieee64::divisor(P[0], ok);
    const double pr = div(P[4], rho, ok);
    const double e0 = div(pr, c.gm1_div, ok);
    const double es = e0 + div(half(s.bb), rho, ok);
    s.ps = P[4] + half(s.bb);
    s.h0 = 1.0 + e0 + pr;
    s.hs = 1.0 + es + div(s.ps, rho, ok);
}

// the clamped extreme wave speeds (slot_max and slot_min of the eigenvalues)
F64_FN void rmhd_speeds(const Consts& c, const double* P, const RmhdState& s, double& ap, double& am, bool& ok)
{
    const double rh = P[0] * s.h0;
    const double cs2 = div(c.gamma * P[4], rh, ok);
    const double v2 = s.vn * s.vn;
    double hi = s.vn, lo = s.vn;
    if (is_zero(s.BB)) {
        const double K = sqrt_rn(cs2 * (1 - s.vv) * (1 - s.vv * cs2 - v2 * (1 - cs2)), ok);
        const Divisor den = ieee64::divisor(1 - s.vv * cs2, ok);
        const double l = div(s.vn * (1 - cs2) - K, den, ok), h = div(s.vn * (1 - cs2) + K, den, ok);
        lo = less(l, lo) ? l : lo;
        hi = less(hi, h) ? h : hi;
    } else {
        const double W4 = s.W2 * s.W2;
        const double v3 = s.vn * v2, v4 = s.vn * v3;
        const Divisor c2 = ieee64::divisor(cs2, ok);
        const double K = W4 * (rh * (div(1.0, c2, ok) - 1.));
        const double L = -s.W2 * (rh + div(s.bb, c2, ok));
        const double b00 = s.b0 * s.b0, bnn = s.bn * s.bn, b0n = 2 * s.b0 * s.bn, Lv = L * s.vn * 2, K4 = -4 * K;
        double l, h;
        quartic_range(c, K - L - b00, K4 * s.vn + Lv + b0n, 6 * K * v2 + L * (1. - v2) + b00 - bnn,
                      K4 * v3 - Lv - b0n, K * v4 + L * v2 + bnn, l, h, ok);
        const double C = sqrt_rn(s.h0 + s.bb, ok);
        const double x = C * s.vn * s.W0, y = C * s.W0;
        const double a1 = div(s.bn - x, s.b0 - y, ok), a6 = div(s.bn + x, s.b0 + y, ok);
        lo = less(l, lo) ? l : lo;
        hi = less(hi, h) ? h : hi;
        lo = less(a1, lo) ? a1 : lo;
        hi = less(hi, a1) ? a1 : hi;
        lo = less(a6, lo) ? a6 : lo;
        hi = less(hi, a6) ? a6 : hi;
    }
    ok = ok && !is_zero(hi) && !is_zero(lo);   // the general form keeps the sign of a zero
    ap = clamp_pos(hi);
    am = clamp_neg(lo);
}

// rmhd_prim
template <int AXIS>
F64_FN void rmhd_side(const Consts& c, const double* P, Side<8>& S, bool& ok)
{
    RmhdState s;
    rmhd_state<AXIS>(c, P, s, ok);
    const double x = P[0] * s.hs * s.W2;
    const double vn = s.vn, Bn = s.Bn;
    S.vn = vn;
    S.U[0] = P[0] * s.W0;
    S.U[4] = x - s.ps - s.b0 * s.b0 - S.U[0];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        S.U[1 + d] = x * P[1 + d] - s.b0 * s.b[d];
        S.U[5 + d] = P[5 + d];
    }
    const Divisor W = ieee64::divisor(s.W0, ok);
    S.F[0] = vn * S.U[0];
#pragma unroll
    for (int d = 0; d < 3; ++d)
        S.F[1 + d] = add_normal<AXIS>(c, d, vn * S.U[1 + d] - div(Bn * s.b[d], W, ok), s.ps);
    S.F[4] = vn * S.U[4] - div(Bn * s.b0, W, ok) + s.ps * vn;
#pragma unroll
    for (int d = 0; d < 3; ++d) S.F[5 + d] = vn * S.U[5 + d] - Bn * P[1 + d];
    rmhd_speeds(c, P, s, S.ap, S.am, ok);
}

// Whether rmhd_prim's eigenvalues along x surely exist (quartic_roots finds
// two or four), from FP32: the fast speeds' quartic is
//   K (x - v)^4 + (1 - x^2) (L (x - v)^2 + (b0 x - bn)^2),  K > 0 > L,
// positive at x = +-1, so a point inside where it lies below zero by a
// thousandth of its terms brackets two real roots on each side.  The points:
// the minimum of the first two terms, and of all of them for a fluid at rest
// (a field along x there, as in an unshocked medium, leaves the first point
// above zero), at least 0.02 from v, so that the roots are far enough apart
// not to drown in FP64's rounding of the quartic.  With the first point alone
// nearly every zone of such a medium needed its roots (mixed 512^2 blast,
// 16 steps 4.19 -> 4.09 ms; plain 160x131, 2 steps 1.64 -> 1.44).
// The thousandth covers the rounding of value and terms (1.2e-4 of the terms at
// most in 32 M random states); of 96 M states with v^2 up to 0.999, p / rho of
// 1e-6 to 1e4 and gamma of 1.0001 to 5/3, the general functions refused none
// of the 70 % certified here.
F64_FN bool rmhd_roots_certain(const Consts& c, const double* P)
{
    float p[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) p[q] = (float) P[q];
    const float g = (float) c.gamma, vv = p[1] * p[1] + p[2] * p[2] + p[3] * p[3];
    const float BB = p[5] * p[5] + p[6] * p[6] + p[7] * p[7], Bv = p[5] * p[1] + p[6] * p[2] + p[7] * p[3];
    if (!(vv < 0.999f)) return false;
    const float W2 = 1.0f / (1.0f - vv), W = sqrtf(W2), b0 = W * Bv, bb = BB / W2 + Bv * Bv, bn = p[5] / W + b0 * p[1];
    const float rh = p[0] + p[4] / (float) c.gamf, cs2 = g * p[4] / rh, v = p[1];
    if (BB == 0.0f) return P[5] == 0.0 && P[6] == 0.0 && P[7] == 0.0;   // no quartic then
    const float K = W2 * W2 * rh * (1.0f / cs2 - 1.0f), L = -W2 * (rh + bb / cs2);
    const float y0 = b0 * v - bn, d1 = sqrtf(-L * (1.0f - v * v) / (2.0f * K));
    const float d2 = sqrtf((y0 * y0 - L * (1.0f - v * v)) / (2.0f * (K - L)));
    bool certain = false;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const float d = m & 2 ? d2 : d1;
        const float x = m & 1 ? v + d : v - d, y = b0 * x - bn, k4 = K * d * d * d * d, w = 1.0f - x * x;
        const float value = k4 + w * (L * d * d + y * y), terms = k4 + w * (-L * d * d + y * y);
        certain = certain || (d > 0.02f && w > 1e-3f && terms < 1e30f && value < -1e-3f * terms);
    }
    return certain;
}

// the same from the eigenvalues themselves
F64_COLD bool rmhd_roots_exist(const Consts& c, double rho, double v1, double v2, double v3, double p, double B1,
                               double B2, double B3)
{
    const double P[8] = {rho, v1, v2, v3, p, B1, B2, B3};
    RmhdState s;
    double ap, am;
    bool ok = true;
    rmhd_state<0>(c, P, s, ok);
    rmhd_speeds(c, P, s, ap, am, ok);
    return ok;
}
F64_FN bool rmhd_roots(const Consts& c, const double* P)
{
    return rmhd_roots_certain(c, P) || rmhd_roots_exist(c, P[0], P[1], P[2], P[3], P[4], P[5], P[6], P[7]);
}

// conserved densities of rmhd_prim, with its eigenvalue check along x
F64_FN void rmhd_p2u(const Consts& c, const double* P, double* U, bool& ok)
{
    RmhdState s;
    rmhd_state<0>(c, P, s, ok);
    const double x = P[0] * s.hs * s.W2;
    U[0] = P[0] * s.W0;
    U[4] = x - s.ps - s.b0 * s.b0 - U[0];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        U[1 + d] = x * P[1 + d] - s.b0 * s.b[d];
        U[5 + d] = P[5 + d];
    }
    ok = ok && rmhd_roots(c, P);
}

// max_eigen_magnitude along the normal of axis a: the extremes clamped at
// zero hold the largest magnitude
F64_FN double rmhd_fastest(const Consts& c, const double* P, int a, bool& ok)
{
    RmhdState s;
    rmhd_state<0>(c, P, s, ok);
    s.vn = a == 0 ? s.vn : a == 1 ? along<1>(c, P[1], P[2], P[3]) : along<2>(c, P[1], P[2], P[3]);
    s.bn = a == 0 ? s.bn : a == 1 ? along<1>(c, s.b[0], s.b[1], s.b[2]) : along<2>(c, s.b[0], s.b[1], s.b[2]);
    double ap, am;
    rmhd_speeds(c, P, s, ap, am, ok);
    return max_pos(ap, from_bits(mag(am)));
}

// rm_anton2dzw with its reconstruction and checks, from rmhd_cons's start or
// the given one (Z0 > 0); ok cleared where it does not succeed
F64_FN void rmhd_newton(const Consts& c, const double* U, double* P, bool& ok, double Z0 = 0.0, double W0 = 0.0)
{
    const double D = U[0], Tau = U[4];
    const double S2 = U[1] * U[1] + U[2] * U[2] + U[3] * U[3];
    const double B2 = U[5] * U[5] + U[6] * U[6] + U[7] * U[7];
    const double BS = U[5] * U[1] + U[6] * U[2] + U[7] * U[3];
    const double BS2 = BS * BS;
    const double g = c.gamf;
    double Z = Z0, W = W0;
    if (Z0 == 0.0) {
        Z = sqrt_rn(S2 + D * D, ok);
        W = div(Z, D, ok);
    }
    double error = 1.0;
    int it = 0;
    while (ok && less(1e-12, error)) {
        const double Z2 = Z * Z, Z3 = Z * Z2, W2 = W * W, W3 = W * W2;
        const Divisor vW2 = ieee64::divisor(W2, ok), vW3 = ieee64::divisor(W3, ok);
        const Divisor vZ2 = ieee64::divisor(Z2, ok), vZ3 = ieee64::divisor(Z3, ok);
        const double BZ = B2 + Z, w1 = W2 - 1, DW = D * W;
        const double Pre = div(D, W, ok) * (div(Z, DW, ok) - 1.0) * g;
        const double j00 = div(2 * BZ * (BS2 * W2 + w1 * Z3), W2 * Z3, ok);
        const double j01 = div(2 * BZ * BZ, vW3, ok);
        const double j10 = 1.0 + div(BS2, vZ3, ok) - div(g, vW2, ok);
        const double j11 = div(B2, vW3, ok) + div(2 * Z - DW, vW3, ok) * g;
        const double f0 = -S2 + div(BZ * BZ * w1, vW2, ok) - div((2 * Z + B2) * BS2, vZ2, ok);
        const double f1 = -Tau + Z + B2 - Pre - div(0.5 * B2, vW2, ok) - div(0.5 * BS2, vZ2, ok) - D;
        const Divisor det = ieee64::divisor(j00 * j11 - j01 * j10, ok);
        const double G0 = div(j11, det, ok), G1 = div(-j01, det, ok), G2 = div(-j10, det, ok), G3 = div(j00, det, ok);
        const double dZ = -(G0 * f0 + G1 * f1);
        const double dW = -(G2 * f0 + G3 * f1);
        double Zn = Z + dZ, Wn = W + dW;
        Zn = from_bits(mag(Zn));
        Zn = less(Zn, 1e20) ? Zn : Z;
        Wn = less(1.0, Wn) ? Wn : 1.0;
        Wn = less(Wn, 1e12) ? Wn : 1e12;
        Z = Zn;
        W = Wn;
        error = fabs(div(dZ, Z, ok)) + fabs(div(dW, W, ok));
        if (++it == 250) ok = false;
    }
    const Divisor vW = ieee64::divisor(W, ok);
    const double b0 = div(BS * W, Z, ok);
    const double dw = div(D, vW, ok);
    P[0] = dw;
    P[4] = dw * (div(Z, D * W, ok) - 1.0) * g;
    const Divisor ZB = ieee64::divisor(Z + B2, ok);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        P[1 + d] = div(U[1 + d] + div(b0 * U[5 + d], vW, ok), ZB, ok);
        P[5 + d] = U[5 + d];
    }
    const double v2 = P[1] * P[1] + P[2] * P[2] + P[3] * P[3];
    ok = ok && less(v2, 1.0) && less(0.0, P[4]) && less(0.0, P[0]);
}

// rmhd_cons (U ordinary), with its closing eigenvalue check along x
F64_FN void rmhd_cons(const Consts& c, const double* U, double* P, bool& ok)
{
    rmhd_newton(c, U, P, ok);
    bool fine = true;
#pragma unroll
    for (int q = 0; q < 8; ++q) fine = fine && ordinary_field<LAW_RMHD>(q, P[q]);
    ok = ok && fine && rmhd_roots(c, P);
}

} // namespace fast64
} // namespace mara

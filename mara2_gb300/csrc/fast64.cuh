// fast64.cuh -- the plain path's physics with fewer FP64 operations.
//
// The plain path must round as the reference's CPU build does, and it is
// bound by the FP64 pipe, on which one operation costs as much as 64 others
// (0.5 lanes per clock and scheduler, measured; 128 lanes per clock and SM
// elsewhere).  The functions here return the bits of their counterparts in
// physics_fp64.cuh (which name the reference's routines) from a third of the
// FP64 operations:
//  * divisions, square roots and most products in integers (ieee64.cuh), the
//    divisions by one divisor sharing its reciprocal: written mul(a, b) and
//    div(a, b).  a * b stays on the FP64 pipe: the split between the two is
//    flat (all products in integers against two thirds: within 1 % on KH
//    1024^2 and MHD 64x56x48, 4 % for the latter on a 1024-zone tube);
//  * each zone's slopes once, for the faces on both of its sides;
//  * multiplications by powers of two on the exponent, comparisons on the bit
//    patterns;
//  * the face normal at compile time: a product with one of its zeros is a
//    zero, of which only the sign can matter, and that is kept (add_zero).
//    The y normal keeps its x component cos(pi/2) = 6.1e-17;
//  * eigenvalues only where they can be the largest or the smallest: rounding
//    is monotone, so e.g. max(vn - c, vn, vn + c) is RN(vn + c).
// They hold for ordinary operands (ordinary(), ordinary_pos()) and where no
// divisor vanishes.  Anything else clears `ok`, and the caller repeats the face or zone with the
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

// Ordinary operands: a density or pressure of 2^-100 to 2^101, another field
// zero or of magnitude 2^-330 to 2^101.  An edge value then is at least
// 2^-154 (edge_pos) and 2^-383 (or zero), and the products that the functions
// below form without a check stay normal: the smallest is rho v v above 2^-974,
// its v_n along y a difference of two such values.  PLM gives no smaller
// edges (the last place of 2^-331); WENO's weighted sum cancels a second time,
// down to 2^-436 found, so weno5_edges checks (EDGE).
F64_FN bool ordinary_pos(double x) { return (u32) (bits(x) >> 32) - (923u << 20) <= (200u << 20); }
F64_FN bool ordinary(double x) { return ((u32) (bits(x) >> 32) & 0x7fffffffu) - (693u << 20) <= (430u << 20) || is_zero(x); }
// field q of a primitive (or conserved: density and energy) state
F64_FN bool ordinary_field(int q, double x) { return q == 0 || q == 4 ? ordinary_pos(x) : ordinary(x); }
// Ahead of a wave into a medium at rest, transverse fields fall by orders of
// magnitude from zone to zone and stay behind for good, at 1e-99 to 1e-270
// (magnetic laws, field along x or y: the transverse field in 49 % of the zones
// of 256^2 after 40 steps with WENO5 and 39 % with PLM, a velocity in 37 % of
// 64^3 after 20; in a third of a relativistic blast 512^2 after 43; never in
// hydro).  The magnetic laws take fields down to 2^-900 for it.  Relativistic
// forms multiply with FP64 instructions, which underflow as the general forms
// do; mhd_side does so where an operand is below 2^-330 (SMALL), p2u, cons and
// fastest use mul_any and times_pow2.  Products without a check remain with y's
// normal, whose factors are steep() or zero, and with pressures.  Against the
// general functions for these zones: relativistic blast, 45 steps, 631 -> 321 ms
// (with rmhd_roots_certain's second point); hot region in MHD at rest, 64^3 PLM,
// 6 steps, 16.7 -> 7.0 ms, 256^2 WENO5, 20 steps, 43.8 -> 17.1.
constexpr int STEEP = 68;   // exponent field of 2^-955
F64_FN bool steep(double x) { return ((u32) (bits(x) >> 32) & 0x7fffffffu) >= (u32) STEEP << 20 || is_zero(x); }
template <int LAW>
F64_FN bool ordinary_field(int q, double x)
{
    if (LAW == LAW_HYDRO || q == 0 || q == 4) return ordinary_field(q, x);
    return ((u32) (bits(x) >> 32) & 0x7fffffffu) - (123u << 20) <= (1000u << 20) || is_zero(x);
}
constexpr int EDGE = 640;   // exponent field of 2^-383
// a reconstructed density or pressure
F64_FN bool edge_pos(double x) { return (u32) (bits(x) >> 32) - (869u << 20) <= (256u << 20); }

using ieee64::mul;
using ieee64::div;
using ieee64::sqrt_rn;

// x 2^k for x zero or well inside the normal range
F64_FN double scale(double x, int k)
{
    return is_zero(x) ? x : from_bits(bits(x) + ((u64) (ieee64::i64) k << 52));
}
F64_FN double half(double x) { return scale(x, -1); }

// a b on the FP64 pipe, as a call: predicated in line it would take its slot
// of the pipe also where no thread needs it
#if defined(__CUDACC__)
static __device__ __noinline__ double mul_seldom(double a, double b) { return __dmul_rn(a, b); }
#else
static inline double mul_seldom(double a, double b) { return a * b; }
#endif

// a b for any operands: on the FP64 pipe only where the integer product does
// not hold
F64_FN double mul_any(double a, double b)
{
    bool ok = true;
    double r = mul(a, b, ok);
    if (!ok) r = mul_seldom(a, b);
    return r;
}

// x 2^k, -3 <= k <= 1: on the exponent where x and the result are normal
F64_FN double times_pow2(double x, int k)
{
    const u32 e = expo(x);
    if (e - 1u < 2046u && e + (u32) k - 1u < 2046u) return from_bits(bits(x) + ((u64) (ieee64::i64) k << 52));
    if (is_zero(x)) return x;
    return mul_seldom(x, k == 1 ? 2.0 : k == -1 ? 0.5 : k == -2 ? 0.25 : 0.125);
}

// x + z for a zero z of the given sign: x, or the zero the addition gives
F64_FN double add_zero(double x, bool z_negative)
{
    return is_zero(x) ? from_bits(z_negative ? bits(x) : 0ull) : x;
}

// the larger of two non-negative finite values, the smaller of two
// non-positive ones (a zero counts as +0)
F64_FN double max_pos(double a, double b) { return bits(a) > bits(b) ? a : b; }
F64_FN double min_neg(double a, double b) { return bits(a) > bits(b) ? a : b; }
// a < b for numbers, -0 below +0
F64_FN bool less(double a, double b)
{
    const ieee64::i64 x = (ieee64::i64) bits(a), y = (ieee64::i64) bits(b), m = 0x7fffffffffffffffll;
    return (x ^ ((x >> 63) & m)) < (y ^ ((y >> 63) & m));
}
// max(x, +0) and min(x, +0) for x without -0
F64_FN double clamp_pos(double x) { return sign_bit(x) ? 0.0 : x; }
F64_FN double clamp_neg(double x) { return sign_bit(x) ? x : 0.0; }

// The constants of a run that the functions use (one copy per kernel launch).
struct Consts {
    double gamma, gm1, theta, ny0;   // ny0: x component of the y normal
    double shenzha_A;
    int weno_is;
    double gamf;                     // (gamma - 1) / gamma
    Divisor gm1_div, d3, d6, d9, d27;
    bool ok;                         // the constants themselves are ordinary
};

// The constants of a configuration, with the normals CartesianMeshGeometry
// gives (ny0: its yhat's x component).
static inline Consts make_consts(double gamma, double theta, double shenzha_A, int weno_is, double ny0)
{
    Consts c;
    c.ok = true;
    c.gamma = gamma;
    c.gm1 = gamma - 1.0;
    c.gamf = (gamma - 1.0) / gamma;
    c.theta = theta;
    c.shenzha_A = shenzha_A;
    c.weno_is = weno_is;
    c.ny0 = ny0;
    c.gm1_div = ieee64::divisor(c.gm1, c.ok);
    c.d3 = ieee64::divisor(3.0, c.ok);
    c.d6 = ieee64::divisor(6.0, c.ok);
    c.d9 = ieee64::divisor(9.0, c.ok);
    c.d27 = ieee64::divisor(27.0, c.ok);
    // gamma - 1 only divides, or multiplies with a check: nearly isothermal
    // gases (1.001) would otherwise pay the lean forms and then the general
    // ones (MHD 192^2, 6 steps, 2.18 ms against 1.75 by the general ones alone)
    const double small = 1e-3, large = 1e3;
    c.ok = c.ok && gamma < large && c.gm1 > 1e-8 && (theta == 0.0 || theta > small) && theta < large &&
           shenzha_A >= 0.0 && shenzha_A < 1e9 && ny0 > 1e-20 && ny0 < small;
    return c;
}

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

// weno5 at both edges of a zone, from ordinary v[-2 .. 2]: the smoothness
// indicators and the products that both edges use once.  SMALL: from values
// whose squares may underflow.

F64_FN double sq(double x) { return mul(x, x); }
template <bool SMALL> F64_FN double indicator(double t, double a, double b)
{
    return SMALL ? t * (a * a) + 0.25 * (b * b) : t * sq(a) + scale(sq(b), -2);
}
template <bool SMALL> F64_FN double quotient(double x, double d, bool& ok) { return SMALL ? x / d : div(x, d, ok); }

template <bool SMALL = false>
F64_FN void weno5_edges(const Consts& c, const double* v, double& left, double& right, bool& ok)
{
    const double t = 13. / 12.;
    const double v3 = 3 * v[0];
    double B0 = indicator<SMALL>(t, v[0] - scale(v[1], 1) + v[2], v3 - scale(v[1], 2) + v[2]);
    double B1 = indicator<SMALL>(t, v[-1] - scale(v[0], 1) + v[1], v[-1] - v[1]);
    double B2 = indicator<SMALL>(t, v[-2] - scale(v[-1], 1) + v[0], v[-2] - scale(v[-1], 2) + v3);
    // w = d / e for the three stencils
    double wl[3], wr[3];
    if (c.weno_is == WENO_BORGES08) {
        const double eps = 1e-14;
        const double tau5 = fabs(B0 - B2);
        const double r0 = 1.0 + quotient<SMALL>(tau5, B0 + eps, ok);
        const double r1 = 1.0 + quotient<SMALL>(tau5, B1 + eps, ok);
        const double r2 = 1.0 + quotient<SMALL>(tau5, B2 + eps, ok);
        wr[0] = 0.3 * r0; wr[1] = 0.6 * r1; wr[2] = 0.1 * r2;
        wl[0] = 0.1 * r0; wl[1] = wr[1]; wl[2] = 0.3 * r2;
    } else {
        double ep = 1e-6;
        if (c.weno_is == WENO_SHENZHA10) {
            ep = 1e-10;
            const double lo = bits(B0) < bits(B1) ? (bits(B0) < bits(B2) ? B0 : B2) : (bits(B1) < bits(B2) ? B1 : B2);
            const double hi = max_pos(max_pos(B0, B1), B2);
            const double add = quotient<SMALL>(lo, hi + ep, ok) * c.shenzha_A * lo;
            B0 = add + B0;
            B1 = add + B1;
            B2 = add + B2;
        }
        const Divisor e0 = ieee64::divisor(sq(ep + B0), ok);
        const Divisor e1 = ieee64::divisor(sq(ep + B1), ok);
        const Divisor e2 = ieee64::divisor(sq(ep + B2), ok);
        wr[0] = div(0.3, e0, ok); wr[1] = div(0.6, e1, ok); wr[2] = div(0.1, e2, ok);
        wl[0] = div(0.1, e0, ok); wl[1] = wr[1]; wl[2] = div(0.3, e2, ok);
    }
    const double third = 1. / 3., sixth = 1. / 6., a56 = 5. / 6., a76 = 7. / 6., a116 = 11. / 6.;
    const double c0 = mul(a56, v[0]), t0 = mul(third, v[0]), e0 = mul(a116, v[0]);
    const double tp = mul(third, v[1]), tm = mul(third, v[-1]), sp = mul(sixth, v[1]), sm = mul(sixth, v[-1]);
    const double tp2 = mul(third, v[2]), tm2 = mul(third, v[-2]), sp2 = mul(sixth, v[2]), sm2 = mul(sixth, v[-2]);
    const double cp = mul(a56, v[1]), cm = mul(a56, v[-1]), gp = mul(a76, v[1]), gm = mul(a76, v[-1]);
    const double r0 = t0 + cp - sp2, r1 = -sm + c0 + tp, r2 = tm2 - gm + e0;
    const double l0 = e0 - gp + tp2, l1 = tm + c0 - sp, l2 = -sm2 + cm + t0;
    // (the quotient's own range check, raised: no edge between zero and what
    // the functions below assume)
    constexpr int LOW = SMALL ? STEEP : EDGE;
    right = div<LOW>(mul(wr[0], r0) + mul(wr[1], r1) + mul(wr[2], r2), wr[0] + wr[1] + wr[2], ok);
    left = div<LOW>(mul(wl[0], l0) + mul(wl[1], l1) + mul(wl[2], l2), wl[0] + wl[1] + wl[2], ok);
}

// ---------------------------------------------------------------------------
// vector component along the normal of AXIS: x n0 + y n1 + z n2
template <int AXIS>
F64_FN double along(const Consts& c, double x, double y, double z)
{
    if constexpr (AXIS == 1) return add_zero(mul(x, c.ny0) + y, sign_bit(z));
    const double v = AXIS == 0 ? x : z;
    return is_zero(v) ? from_bits(bits(x) & bits(y) & bits(z) & SIGN) : v;
}

// x + p n_d for the component d of the normal
template <int AXIS>
F64_FN double add_normal(const Consts& c, int d, double x, double p)
{
    if (d == AXIS) return x + p;
    if (AXIS == 1 && d == 0) return x + mul(p, c.ny0);
    return add_zero(x, sign_bit(p));
}

// a product v_n x with v_n = along(v): P0 v_axis is already there for a flux
// along a coordinate axis (y's normal has two components)
template <int AXIS>
F64_FN double times_along(double vn, double x, double x_times_axis)
{
    if constexpr (AXIS == 1) return mul(vn, x);
    return is_zero(vn) ? from_bits((bits(vn) ^ bits(x)) & SIGN) : x_times_axis;
}

// One side of a face: primitives, conserved densities, fluxes and the clamped
// extreme wave speeds (slot_max, slot_min of physics_fp64.cuh).
template <int NQ> struct Side {
    double U[NQ], F[NQ];
    double vn, ap, am;
};

F64_FN double dot(double a, double b, double c, double x, double y, double z)
{
    return a * x + b * y + c * z;
}

// hydro_prim
template <int AXIS>
F64_FN void hydro_side(const Consts& c, const double* P, Side<5>& S, bool& ok)
{
    ok = ok && edge_pos(P[0]) && edge_pos(P[4]);
    const double cs = sqrt_rn(div(mul(c.gamma, P[4]), P[0], ok), ok);
    const double vv = dot(P[1], P[2], P[3], P[1], P[2], P[3]);
    const double vn = along<AXIS>(c, P[1], P[2], P[3]);
    S.vn = vn;
    S.U[0] = P[0];
    S.U[1] = mul(P[0], P[1]);
    S.U[2] = mul(P[0], P[2]);
    S.U[3] = mul(P[0], P[3]);
    S.U[4] = half(mul(P[0], vv)) + div(P[4], c.gm1_div, ok);
    S.F[0] = times_along<AXIS>(vn, S.U[0], S.U[1 + AXIS]);
    S.F[1] = add_normal<AXIS>(c, 0, mul(vn, S.U[1]), P[4]);
    S.F[2] = add_normal<AXIS>(c, 1, mul(vn, S.U[2]), P[4]);
    S.F[3] = add_normal<AXIS>(c, 2, mul(vn, S.U[3]), P[4]);
    S.F[4] = mul(vn, S.U[4]) + mul(P[4], vn);
    S.ap = clamp_pos(vn + cs);
    S.am = clamp_neg(vn - cs);
}

// mhd_prim; an auxiliary field (index 8) is carried without a flux.  SMALL:
// from fields whose products may underflow.
template <bool SMALL> F64_FN double prod(double a, double b) { return SMALL ? a * b : mul(a, b); }
template <bool SMALL> F64_FN double halved(double x) { return SMALL ? 0.5 * x : half(x); }

template <int AXIS, bool SMALL, int NQ>
F64_FN void mhd_side(const Consts& c, const double* P, Side<NQ>& S, bool& ok)
{
    ok = ok && edge_pos(P[0]) && edge_pos(P[4]);
    const Divisor rho = ieee64::divisor(P[0], ok);
    const double cs2 = div(mul(c.gamma, P[4]), rho, ok);
    const double vv = dot(P[1], P[2], P[3], P[1], P[2], P[3]);
    const double BB = dot(P[5], P[6], P[7], P[5], P[6], P[7]);
    const double Bv = dot(P[5], P[6], P[7], P[1], P[2], P[3]);
    const double vn = along<AXIS>(c, P[1], P[2], P[3]);
    const double Bn = along<AXIS>(c, P[5], P[6], P[7]);
    const double ps = P[4] + halved<SMALL>(BB);
    S.vn = vn;
    S.U[0] = P[0];
#pragma unroll
    for (int d = 1; d < 4; ++d) S.U[d] = prod<SMALL>(P[0], P[d]);
    S.U[4] = halved<SMALL>(prod<SMALL>(P[0], vv)) + halved<SMALL>(BB) + div(P[4], c.gm1_div, ok);
#pragma unroll
    for (int d = 5; d < NQ; ++d) S.U[d] = P[d];
    S.F[0] = SMALL ? vn * S.U[0] : times_along<AXIS>(vn, S.U[0], S.U[1 + AXIS]);
#pragma unroll
    for (int d = 0; d < 3; ++d)
        S.F[1 + d] = add_normal<AXIS>(c, d, prod<SMALL>(vn, S.U[1 + d]) - prod<SMALL>(Bn, P[5 + d]), ps);
    S.F[4] = prod<SMALL>(vn, S.U[4]) - Bn * Bv + prod<SMALL>(ps, vn);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (!SMALL && AXIS != 1 && d == AXIS) {
            // v_n B_n - B_n v_n: +0, or the difference of two zeros
            const bool zero = is_zero(vn) || is_zero(Bn);
            const bool p = sign_bit(vn) != sign_bit(P[5 + d]), q = sign_bit(Bn) != sign_bit(P[1 + d]);
            S.F[5 + d] = from_bits(zero && p && !q ? SIGN : 0ull);
        } else {
            S.F[5 + d] = prod<SMALL>(vn, S.U[5 + d]) - prod<SMALL>(Bn, P[1 + d]);
        }
    }
    if constexpr (NQ > 8) S.F[8] = 0.0;
    // the fast speed; an Alfven speed that rounding puts above it wins
    const double ca2 = div(BB, rho, ok);
    const double cn2 = div(prod<SMALL>(Bn, Bn), rho, ok);
    const double s = cs2 + ca2;
    const double cF2 = half(s + sqrt_rn(mul(s, s) - scale(cs2, 2) * cn2, ok));
    const double cf = sqrt_rn(max_pos(cF2, cn2), ok);
    S.ap = clamp_pos(vn + cf);
    S.am = clamp_neg(vn - cf);
}

template <int LAW, int AXIS, bool SMALL = false>
F64_FN void side(const Consts& c, const double* P, Side<LawInfo<LAW>::NQ>& S, bool& ok)
{
    if constexpr (LAW == LAW_HYDRO) hydro_side<AXIS>(c, P, S, ok);
    else mhd_side<AXIS, SMALL>(c, P, S, ok);
}

// ---------------------------------------------------------------------------
// hlle of one field, from the sides' clamped wave speeds
F64_FN double hlle(double apl, double apr, double aml, double amr, double fl, double fr, double ul, double ur, bool& ok)
{
    const double ap = max_pos(apl, apr), am = min_neg(aml, amr);
    return div(mul(ap, fl, ok) - mul(am, fr, ok) + ap * am * (ur - ul), ap - am, ok);
}

// the star state of the side the contact moves away from, chosen first
template <int AXIS>
F64_FN void hllc(const Consts& c, const double* Pl, const double* Pr, const Side<5>& L, const Side<5>& R, double* F,
                 bool& ok)
{
    const double ap = max_pos(L.ap, R.ap), am = min_neg(L.am, R.am);
    const double sl = am - L.vn, sr = ap - R.vn;
    const double ml = mul(Pl[0], sl, ok), mr = mul(Pr[0], sr, ok);
    const double lc = div((Pr[4] - mul(R.F[0], sr, ok)) - (Pl[4] - mul(L.F[0], sl, ok)), ml - mr, ok);
    const bool left = !sign_bit(lc) || is_zero(lc);
    const double s = left ? am : ap, m = left ? ml : mr, vn = left ? L.vn : R.vn;
    double P[5], U[5], G[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        P[q] = left ? Pl[q] : Pr[q];
        U[q] = left ? L.U[q] : R.U[q];
        G[q] = left ? L.F[q] : R.F[q];
    }
    const double f = div(m, s - lc, ok);
    const double w = lc - vn;
    double Us[5];
    Us[0] = f;
    Us[4] = mul(f, div(U[4], P[0], ok) + mul(w, lc + div(P[4], m, ok), ok), ok);
#pragma unroll
    for (int d = 0; d < 3; ++d) Us[1 + d] = mul(f, add_normal<AXIS>(c, d, P[1 + d], w), ok);
    const bool supersonic = is_zero(am);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        const double star = G[q] + mul(s, Us[q] - U[q], ok);
        F[q] = supersonic ? L.F[q] : star;
    }
}

// ---------------------------------------------------------------------------
// hydro_cons; mhd_cons where it accepts the state as it is (U ordinary)
template <int LAW>
F64_FN void cons(const Consts& c, const double* U, double* P, bool& ok)
{
    constexpr int NQ = LawInfo<LAW>::NQ;
    const Divisor rho = ieee64::divisor(U[0], ok);
    const double pp = dot(U[1], U[2], U[3], U[1], U[2], U[3]);
    double e = U[4] - div(LAW == LAW_HYDRO ? half(pp) : times_pow2(pp, -1), rho, ok);
    if constexpr (LAW != LAW_HYDRO) {
        e = e - times_pow2(dot(U[5], U[6], U[7], U[5], U[6], U[7]), -1);
#pragma unroll
        for (int q = 5; q < NQ; ++q) P[q] = U[q];
        ok = ok && !sign_bit(e);
    }
    P[0] = U[0];
    P[4] = mul(e, c.gm1, ok);
#pragma unroll
    for (int q = 1; q < 4; ++q) P[q] = div(U[q], rho, ok);
}

// hydro_p2u, mhd_p2u
template <int LAW>
F64_FN void p2u(const Consts& c, const double* P, double* U, bool& ok)
{
    constexpr int NQ = LawInfo<LAW>::NQ;
    const double vv = dot(P[1], P[2], P[3], P[1], P[2], P[3]);
    double e;
    U[0] = P[0];
    if constexpr (LAW == LAW_HYDRO) {
#pragma unroll
        for (int d = 1; d < 4; ++d) U[d] = mul(P[0], P[d]);
        e = half(mul(P[0], vv));
    } else {
#pragma unroll
        for (int d = 1; d < 4; ++d) U[d] = mul_any(P[0], P[d]);
        e = times_pow2(mul_any(P[0], vv), -1) + times_pow2(dot(P[5], P[6], P[7], P[5], P[6], P[7]), -1);
#pragma unroll
        for (int q = 5; q < NQ; ++q) U[q] = P[q];
    }
    U[4] = e + div(P[4], c.gm1_div, ok);
}

// The largest max_eigen_magnitude over the three face normals: on each,
// RN(|vn| + c) with the fast speed c.
template <int LAW>
F64_FN double fastest(const Consts& c, const double* P, bool& ok)
{
    const double v[3] = {P[1], mul(P[1], c.ny0) + P[2], P[3]};
    const Divisor rho = ieee64::divisor(P[0], ok);
    const double cs2 = div(mul(c.gamma, P[4]), rho, ok);
    if constexpr (LAW == LAW_HYDRO) {
        u64 vmax = mag(v[0]) > mag(v[1]) ? mag(v[0]) : mag(v[1]);
        vmax = vmax > mag(v[2]) ? vmax : mag(v[2]);
        return from_bits(vmax) + sqrt_rn(cs2, ok);
    } else {
        const double BB = dot(P[5], P[6], P[7], P[5], P[6], P[7]);
        const double B[3] = {P[5], mul(P[5], c.ny0) + P[6], P[7]};
        const double s = cs2 + div(BB, rho, ok);
        const double s2 = mul(s, s);
        double m = 0.0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double cn2 = div(mul_any(B[a], B[a]), rho, ok);
            const double cF2 = half(s + sqrt_rn(s2 - scale(cs2, 2) * cn2, ok));
            m = max_pos(m, from_bits(mag(v[a])) + sqrt_rn(max_pos(cF2, cn2), ok));
        }
        return m;
    }
}

} // namespace fast64
} // namespace mara

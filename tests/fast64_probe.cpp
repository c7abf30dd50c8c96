// Host build of the plain path's device functions: the forms with fewer FP64
// operations (fast64.cuh, ieee64.cuh) against the general ones
// (physics_fp64.cuh) and the host's own division and square root, on seeded
// operands of many kinds.  Every function returns the number of results whose
// bits differ; *accepted counts the operands the fast form took.
#include <math.h>
#include <string.h>

#include <cuda_runtime.h>

static inline long long __double_as_longlong(double x) { long long b; memcpy(&b, &x, 8); return b; }
static inline double __longlong_as_double(long long b) { double x; memcpy(&x, &b, 8); return x; }

#ifdef PROBE_IEEE_ONLY
#include "../mara2_gb300/csrc/ieee64.cuh"
#else
#include "../mara2_gb300/csrc/fast64_rmhd.cuh"
#endif

#ifndef PROBE_IEEE_ONLY
using namespace mara;
#endif
typedef unsigned long long u64;

static u64 state;
static u64 rnd()
{
    state += 0x9E3779B97F4A7C15ull;
    u64 z = state;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
static double uni() { return (double) (rnd() >> 11) * 0x1p-53; }
static bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b); }

// a significand near the edges of rounding as often as a random one
static u64 significand()
{
    const u64 m = rnd() >> 12, all = 0xfffffffffffffull;
    switch (rnd() % 10) {
        case 0: return 0;
        case 1: return all;
        case 2: return m & 0xff;
        case 3: return (m | ~0xffull) & all;
        case 4: return 1ull << (rnd() % 52);
        case 5: return (all << (rnd() % 52)) & all;
        case 6: return all - (rnd() & 7);
        default: return m;
    }
}
static double wide(int spread)
{
    const u64 e = 1023 + rnd() % (2 * spread + 1) - spread;
    return __longlong_as_double((long long) ((rnd() & 1) << 63 | e << 52 | significand()));
}
static double any()
{
    switch (rnd() % 6) {
        case 0: return (rnd() & 1) ? 0.0 : -0.0;
        case 1: return __longlong_as_double((long long) rnd());
        case 2: return (rnd() & 1) ? INFINITY : NAN;
        default: return wide(1000);
    }
}

#ifndef PROBE_IEEE_ONLY
// A zone's primitives.  kind 0: smooth, 1: zeros and equal values, 2: strong
// jumps, 3: wide magnitudes, 4: anything, 5: small fields and zeros, 6: small
// magnetic fields and zeros; hydro
// pressure and density positive for all but kind 4
static void zone(int law, int kind, int nq, const double* base, double* P)
{
    for (int q = 0; q < nq; ++q) {
        const bool pos = q == 0 || q == 4;
        double v;
        if (kind == 0) v = base[q] * (1 + 0.1 * (uni() - 0.5));
        else if (kind == 1) v = pos ? (rnd() & 1 ? 1.0 : base[q]) : rnd() % 4 == 0 ? base[q] : rnd() % 3 == 0 ? -0.0 : 0.0;
        else if (kind == 2) v = pos ? exp(8 * (uni() - 0.5)) : 6 * (uni() - 0.5);
        else if (kind == 5 || kind == 6) v = pos || rnd() % 8 ? base[q] * (1 + 0.1 * (uni() - 0.5)) : 0.0;
        else if (kind == 3) v = pos ? fabs(wide(30)) : wide(rnd() % 8 ? 20 : 320);
        else v = any();
        if (law == LAW_RMHD && kind < 4 && !pos && q < 4) v *= kind == 2 ? 0.16 : 0.5;   // mostly below light speed
        P[q] = v;
    }
}

// some fields (kind 6: from the magnetic ones on) down to 2^-930
static void shrink(int nq, double* base, int kind)
{
    for (int q = kind == 6 ? 5 : 0; q < nq; ++q)
        if (q != 0 && q != 4 && rnd() % 2) base[q] *= pow(2.0, -930 * uni());
}

template <int LAW, int RECON, int RIEMANN, int AXIS>
static long faces(long n, const PhysParams& pp, const fast64::Consts& C, const double (*nrm)[3], int kind, long* accepted)
{
    constexpr int NQ = LawInfo<LAW>::NQ, S = RECON == RECON_PCM ? 1 : RECON == RECON_PLM ? 2 : 3;
    long bad = 0;
    for (long m = 0; m < n; ++m) {
        double Z[2 * S][NQ], base[NQ];
        for (int q = 0; q < NQ; ++q) base[q] = q == 0 || q == 4 ? exp(2 * (uni() - 0.5)) : 2 * (uni() - 0.5);
        if (kind >= 5) shrink(NQ, base, kind);
        for (int s = 0; s < 2 * S; ++s) zone(LAW, kind, NQ, base, Z[s]);
        if (kind == 1 && rnd() % 3 == 0) for (int s = 1; s < 2 * S; ++s) memcpy(Z[s], Z[0], sizeof(Z[0]));
        double PL[NQ], PR[NQ], QL[NQ], QR[NQ];
        bool ok = C.ok, all = true;   // all: every field of every zone is large
        for (int q = 0; q < NQ; ++q) {
            double v[2 * S];
            bool strict = true;
            for (int s = 0; s < 2 * S; ++s) {
                v[s] = Z[s][q];
                ok = ok && fast64::ordinary_field<LAW>(q, v[s]);
                strict = strict && fast64::ordinary_field(q, v[s]);
            }
            all = all && strict;
            if constexpr (RECON == RECON_PCM) { PL[q] = QL[q] = v[0]; PR[q] = QR[q] = v[1]; }
            else if constexpr (RECON == RECON_PLM) {
                QL[q] = v[1] + +1.0 * 0.5 * minmod(pp.plm_theta, v[0], v[1], v[2]);
                QR[q] = v[2] + -1.0 * 0.5 * minmod(pp.plm_theta, v[1], v[2], v[3]);
                const double a = C.theta * (v[1] - v[0]), b = C.theta * (v[2] - v[1]), c = C.theta * (v[3] - v[2]);
                PL[q] = v[1] + fast64::half_slope(a, v[2] - v[0], b);
                PR[q] = v[2] - fast64::half_slope(b, v[3] - v[1], c);
            } else {
                QL[q] = weno5<true>(&v[2], pp.weno_is, pp.shenzha_A);
                QR[q] = weno5<false>(&v[3], pp.weno_is, pp.shenzha_A);
                double x;
                if (strict) {
                    fast64::weno5_edges(C, &v[2], x, PL[q], ok);
                    fast64::weno5_edges(C, &v[3], PR[q], x, ok);
                } else {
                    fast64::weno5_edges<true>(C, &v[2], x, PL[q], ok);
                    fast64::weno5_edges<true>(C, &v[3], PR[q], x, ok);
                }
            }
        }
        double F[NQ], H[NQ];
        StateD<NQ> L, R;
        const int e = law_prim<LAW>(pp, QL, nrm[AXIS], L) | law_prim<LAW>(pp, QR, nrm[AXIS], R);
        fast64::Side<NQ> l, r;
        if constexpr (LAW == LAW_RMHD) {
            fast64::rmhd_side<AXIS>(C, PL, l, ok);
            fast64::rmhd_side<AXIS>(C, PR, r, ok);
        } else if (all) {
            fast64::side<LAW, AXIS>(C, PL, l, ok);
            fast64::side<LAW, AXIS>(C, PR, r, ok);
        } else {
            fast64::side<LAW, AXIS, true>(C, PL, l, ok);
            fast64::side<LAW, AXIS, true>(C, PR, r, ok);
        }
        if constexpr (RIEMANN == RIEMANN_HLLC) {
            hllc<NQ>(L, R, nrm[AXIS], H);
            fast64::hllc<AXIS>(C, PL, PR, l, r, F, ok);
        } else {
            hlle<NQ>(L, R, H);
            for (int q = 0; q < NQ; ++q)
                F[q] = fast64::hlle(l.ap, r.ap, l.am, r.am, l.F[q], r.F[q], l.U[q], r.U[q], ok);
        }
        if (!ok) continue;
        ++*accepted;
        bool wrong = e != ST_OK;
        for (int q = 0; q < NQ; ++q) wrong = wrong || !same(F[q], H[q]);
        bad += wrong;
    }
    return bad;
}

static void constants(PhysParams& pp, fast64::Consts& C, double (*nrm)[3], int weno, double gamma, double theta)
{
    memset(&pp, 0, sizeof(pp));
    pp.gamma = gamma;
    pp.plm_theta = theta;
    pp.shenzha_A = 50.0;
    pp.pressure_floor = -1.0;
    pp.weno_is = weno;
    const double n[3][3] = {{1, 0, 0}, {cos(M_PI / 2), 1, 0}, {0, 0, 1}};
    memcpy(nrm, n, sizeof(n));
    C = fast64::make_consts(gamma, theta, 50.0, weno, n[1][0]);
}

extern "C" long probe_faces(long n, u64 seed, int law, int recon, int riemann, int axis, int weno, double gamma,
                            double theta, int kind, long* accepted)
{
    state = seed;
    *accepted = 0;
    PhysParams pp;
    fast64::Consts C;
    double nrm[3][3];
    constants(pp, C, nrm, weno, gamma, theta);
#define AXES(LAW, RECON, RIEMANN)                                                                                  \
    return axis == 0 ? faces<LAW, RECON, RIEMANN, 0>(n, pp, C, nrm, kind, accepted)                                 \
         : axis == 1 ? faces<LAW, RECON, RIEMANN, 1>(n, pp, C, nrm, kind, accepted)                                 \
                     : faces<LAW, RECON, RIEMANN, 2>(n, pp, C, nrm, kind, accepted)
#define RECONS(LAW, RIEMANN)                                                                                       \
    if (recon == RECON_PCM) { AXES(LAW, RECON_PCM, RIEMANN); }                                                      \
    if (recon == RECON_PLM) { AXES(LAW, RECON_PLM, RIEMANN); }                                                      \
    AXES(LAW, RECON_WENO5, RIEMANN)
    if (law == LAW_HYDRO && riemann == RIEMANN_HLLC) { RECONS(LAW_HYDRO, RIEMANN_HLLC); }
    if (law == LAW_HYDRO) { RECONS(LAW_HYDRO, RIEMANN_HLLE); }
    if (law == LAW_MHD) { RECONS(LAW_MHD, RIEMANN_HLLE); }
    if (law == LAW_RMHD) { RECONS(LAW_RMHD, RIEMANN_HLLE); }
    RECONS(LAW_MHD_COOL, RIEMANN_HLLE);
}

// The hydro WENO5 HLLE flux along x of the face between zones 2 and 3 of
// Z[6][5]: 1 where the lean form took it with other bits, 0 where it took it
// with the same, -1 where it refused.
extern "C" int probe_hydro_weno_face(const double* Z, int weno)
{
    PhysParams pp;
    fast64::Consts C;
    double nrm[3][3];
    constants(pp, C, nrm, weno, 5.0 / 3, 1.5);
    double PL[5], PR[5], QL[5], QR[5], x;
    bool ok = C.ok;
    for (int q = 0; q < 5; ++q) {
        double v[6];
        for (int s = 0; s < 6; ++s) {
            v[s] = Z[s * 5 + q];
            ok = ok && fast64::ordinary_field(q, v[s]);
        }
        QL[q] = weno5<true>(&v[2], pp.weno_is, pp.shenzha_A);
        QR[q] = weno5<false>(&v[3], pp.weno_is, pp.shenzha_A);
        fast64::weno5_edges(C, &v[2], x, PL[q], ok);
        fast64::weno5_edges(C, &v[3], PR[q], x, ok);
    }
    StateD<5> L, R;
    law_prim<LAW_HYDRO>(pp, QL, nrm[0], L);
    law_prim<LAW_HYDRO>(pp, QR, nrm[0], R);
    double H[5];
    hlle<5>(L, R, H);
    fast64::Side<5> l, r;
    fast64::side<LAW_HYDRO, 0>(C, PL, l, ok);
    fast64::side<LAW_HYDRO, 0>(C, PR, r, ok);
    bool wrong = false;
    for (int q = 0; q < 5; ++q)
        wrong = wrong || !same(H[q], fast64::hlle(l.ap, r.ap, l.am, r.am, l.F[q], r.F[q], l.U[q], r.U[q], ok));
    return !ok ? -1 : wrong;
}

template <int LAW>
static long zones(long n, const PhysParams& pp, const fast64::Consts& C, const double (*nrm)[3], int kind, long* accepted)
{
    constexpr int NQ = LawInfo<LAW>::NQ;
    long bad = 0;
    for (long m = 0; m < n; ++m) {
        double base[NQ], P[NQ];
        for (int q = 0; q < NQ; ++q) base[q] = q == 0 || q == 4 ? exp(2 * (uni() - 0.5)) : 2 * (uni() - 0.5);
        if (kind >= 5) shrink(NQ, base, kind);
        zone(LAW, kind, NQ, base, P);
        bool ord = C.ok;
        for (int q = 0; q < NQ; ++q) ord = ord && fast64::ordinary_field<LAW>(q, P[q]);
        double U[NQ], W[NQ];
        bool ok = ord;
        bool wrong = false;
        const int ep = law_p2u<LAW>(pp, P, U);
        if constexpr (LAW == LAW_RMHD) {
            fast64::rmhd_p2u(C, P, W, ok);
            wrong = ok && ep != ST_OK;
        } else {
            fast64::p2u<LAW>(C, P, W, ok);
        }
        if (ok) for (int q = 0; q < NQ; ++q) wrong = wrong || !same(U[q], W[q]);
        *accepted += ok;
        // the same numbers as conserved densities, and the zone's own
        for (int t = 0; t < 2; ++t) {
            double D[NQ], A[NQ], B[NQ];
            bool o2 = C.ok;
            for (int q = 0; q < NQ; ++q) { D[q] = t ? U[q] : P[q]; o2 = o2 && fast64::ordinary_field<LAW>(q, D[q]); A[q] = 0; }
            int code = 0;
            const int e = law_cons<LAW>(pp, D, A, &code);
            if constexpr (LAW == LAW_RMHD) fast64::rmhd_cons(C, D, B, o2);
            else fast64::cons<LAW>(C, D, B, o2);
            if (o2) { wrong = wrong || e != ST_OK; for (int q = 0; q < NQ; ++q) wrong = wrong || !same(A[q], B[q]); }
        }
        double lmax = 0;
        for (int a = 0; a < 3; ++a) {
            StateD<NQ> S;
            law_prim<LAW>(pp, P, nrm[a], S);
            double x = 0;
            for (int q = 0; q < NQ; ++q) if (x < fabs(S.A[q])) x = fabs(S.A[q]);
            if (a == 0 || lmax < x) lmax = x;
        }
        ok = ord;
        double f;
        if constexpr (LAW == LAW_RMHD) {
            f = 0;
            for (int a = 0; a < 3; ++a) { const double x = fast64::rmhd_fastest(C, P, a, ok); if (f < x) f = x; }
        }
        else f = fast64::fastest<LAW>(C, P, ok);
        if (ok) wrong = wrong || !same(f, lmax);
        bad += wrong;
    }
    return bad;
}

extern "C" long probe_zones(long n, u64 seed, int law, double gamma, int kind, long* accepted)
{
    state = seed;
    *accepted = 0;
    PhysParams pp;
    fast64::Consts C;
    double nrm[3][3];
    constants(pp, C, nrm, WENO_SHENZHA10, gamma, 1.5);
    if (law == LAW_HYDRO) return zones<LAW_HYDRO>(n, pp, C, nrm, kind, accepted);
    if (law == LAW_RMHD) return zones<LAW_RMHD>(n, pp, C, nrm, kind, accepted);
    if (law == LAW_MHD) return zones<LAW_MHD>(n, pp, C, nrm, kind, accepted);
    return zones<LAW_MHD_COOL>(n, pp, C, nrm, kind, accepted);
}

#endif  // PROBE_IEEE_ONLY

extern "C" long probe_ieee(long n, u64 seed, long* accepted)
{
    state = seed;
    *accepted = 0;
    long bad = 0;
    for (long m = 0; m < n; ++m) {
        double x = m % 16 == 0 ? any() : wide(m % 16 == 1 ? 1022 : 100), d = m % 16 == 0 ? any() : wide(100);
        if (m % 8 == 2) d = __longlong_as_double(__double_as_longlong(x) + (long long) (rnd() % 5) - 2);
        if (m % 8 == 3) x = (double) ((long double) d * (1.0L + (long double) (rnd() >> 11) * 0x1p-53L));  // near a midpoint
        bool ok = true;
        const double q = ieee64::div(x, d, ok);
        if (ok) { ++*accepted; bad += !same(q, x / d); }
        double a = fabs(x);
        if (m % 8 == 4) { a = d * d; a = rnd() & 1 ? nextafter(a, 2 * a) : rnd() & 1 ? nextafter(a, 0) : a; }
        ok = true;
        const double p = ieee64::mul(x, d, ok);
        if (ok) { ++*accepted; bad += !same(p, x * d); }
        ok = true;
        const double r = ieee64::sqrt_rn(a, ok);
        if (ok) { ++*accepted; bad += !same(r, sqrt(a)); }
    }
    return bad;
}

#ifndef PROBE_IEEE_ONLY
// ziv64.cuh against crmath.cuh: arc cosines, sines and cosines of their
// thirds, cube roots
extern "C" long probe_ziv(long n, u64 seed, long* accepted)
{
    state = seed;
    *accepted = 0;
    long bad = 0;
    for (long m = 0; m < n; ++m) {
        const double u = uni();
        const double z = m % 4 == 0 ? 2 * u - 1 : m % 4 == 1 ? -1 + exp(-36 * u) : m % 4 == 2 ? 1 - exp(-10 * u)
                                                             : (m % 8 == 3 ? -1.0 : (2 * u - 1) * exp(-20 * uni()));
        bool ok = true;
        const double a = ziv64::arccos(z, ok);
        if (ok) { ++*accepted; bad += !same(a, crm::acos_cr(z)); }
        const double t = m & 1 ? crm::acos_cr(z) / 3.0 : uni() * 1.05;
        double c, s;
        ok = true;
        ziv64::sincos_third(t, c, s, ok);
        if (ok) { ++*accepted; bad += !same(c, crm::cos_cr(t)) || !same(s, crm::sin_cr(t)); }
        const double x = exp((uni() - 0.5) * (m & 1 ? 10 : 400));
        ok = true;
        const double y = ziv64::pow_third(x, ok);
        if (ok) { ++*accepted; bad += !same(y, crm::pow_third(x)); }
    }
    return bad;
}
#endif

// plain_kernels.cuh -- the kernels of the plain FP64 path: one launch of face
// fluxes over all fleshed axes (runs of faces: one per axis), then one fused
// update kernel per RK stage, plus the Courant reduction.  Compiled with
// --fmad=false (see mara2_gb300/build.py) so that the arithmetic rounds as
// the reference's CPU build does.
//
// Per stage (MethodOfLinesTVD::advance, SolutionSchemes.cpp:191-274):
//   flux kernels        MeshOperator::godunov (MeshOperator.cpp:443-525): the
//                       2s-cell stencil along the axis, intercell flux
//                       (reconstruction + fromPrimitive x2 + Riemann), raw
//                       flux stored per face.  Faces are those the interior
//                       update reads: along the axis the interior faces,
//                       across it the interior rows plus one guard row on
//                       each side when flux CT needs transverse neighbours.
//                       flux_tile_kernel: a block per 32 faces; flux_run_kernel:
//                       a thread per run of faces (large hydro grids, PLM,
//                       HLLC); flux_general_kernel: a thread per face (magnetic
//                       laws with HLLC).  Zones whose values the lean forms of
//                       fast64.cuh do not cover go to face_general.
//   update_kernel       per interior zone: CellCenteredFieldCT's flux CT on
//                       the magnetic fluxes of the zone's six faces
//                       (CellCenteredFieldCT.cpp:14-134), the divergence
//                       (MeshOperator.cpp:323-381), the RK combine
//                       (SolutionSchemes.cpp:232-235), fromConserved
//                       (FieldOperator::recoverPrimitive, FieldOperator.cpp:
//                       41-82) and the guard fill: boundary conditions are
//                       copies (periodic, outflow) or mirrored copies
//                       (reflecting) of interior zones applied axis by axis,
//                       so every guard zone equals one interior zone (velocity
//                       components negated on reflecting axes) and the zone
//                       that owns a value writes all of its guard images.
#pragma once

#include "../../include/mara_gpu.h"
#include "internal.h"
#include "fast64.cuh"
#include "fast64_rmhd.cuh"
#include "physics_fp64.cuh"

namespace mara {

using fast64::times_pow2;

template <int RECON> struct ReconInfo;
template <> struct ReconInfo<RECON_PCM> { static constexpr int S = 1; };
template <> struct ReconInfo<RECON_PLM> { static constexpr int S = 2; };
template <> struct ReconInfo<RECON_WENO5> { static constexpr int S = 3; };

__device__ __forceinline__ void record_status(DevStatus* st, int code)
{
    atomicCAS(&st->code, 0, code);
}

// ---------------------------------------------------------------------------
// The Godunov flux of one face with the general functions, written to F; the
// cell on its right is P[base].  Returns the status of the face's states.
template <int LAW, int RECON, int RIEMANN>
__device__ __noinline__ int face_general(const double* P, long long sP, long long stride, double n0, double n1,
                                         double n2, const PhysParams* __restrict__ ppp, double* F, long long sF)
{
    constexpr int NQ = LawInfo<LAW>::NQ;
    constexpr int S = ReconInfo<RECON>::S;
    const PhysParams& pp = *ppp;
    const double n[3] = {n0, n1, n2};
    double PL[NQ], PR[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        double v[2 * S];
#pragma unroll
        for (int c = 0; c < 2 * S; ++c) v[c] = P[q * sP + (c - S) * stride];
        if constexpr (RECON == RECON_PCM) {
            PL[q] = v[0];
            PR[q] = v[1];
        } else if constexpr (RECON == RECON_PLM) {
            PL[q] = v[1] + +1.0 * 0.5 * minmod(pp.plm_theta, v[0], v[1], v[2]);
            PR[q] = v[2] + -1.0 * 0.5 * minmod(pp.plm_theta, v[1], v[2], v[3]);
        } else {
            PL[q] = weno5<true>(&v[2], pp.weno_is, pp.shenzha_A);
            PR[q] = weno5<false>(&v[3], pp.weno_is, pp.shenzha_A);
        }
    }
    StateD<NQ> L, R;
    int e = law_prim<LAW>(pp, PL, n, L);
    if (e == ST_OK) e = law_prim<LAW>(pp, PR, n, R);
    if (e != ST_OK) return e;
    double Fh[NQ];
    if constexpr (RIEMANN == RIEMANN_HLLC) hllc<NQ>(L, R, n, Fh);
    else hlle<NQ>(L, R, Fh);
#pragma unroll
    for (int q = 0; q < NQ; ++q) F[q * sF] = Fh[q];
    return ST_OK;
}

// The faces of one axis with the general functions: HLLC with a magnetic law,
// which the solver is not meant for (it leaves the magnetic fluxes zero).
struct FaceSpace {
    int lo[3];   // first face (right cell) and row of each axis
    int nb[3];   // faces and rows per axis
    int axis;
};

template <int LAW, int RECON, int RIEMANN>
__global__ void __launch_bounds__(128) flux_general_kernel(const double* P, double* __restrict__ F,
                                                           const __grid_constant__ GridDesc G,
                                                           const __grid_constant__ PhysParams pp,
                                                           const __grid_constant__ FaceSpace X,
                                                           DevStatus* __restrict__ st)
{
    pdl_wait();
    if (st->code != 0 || st->done) return;
    if (st->failures != 0) { st->halt = 1; return; }  // failures are final once the stage ended
    const unsigned lin = blockIdx.x * blockDim.x + threadIdx.x;
    if (lin >= (unsigned) X.nb[0] * (unsigned) X.nb[1]) return;
    const int i = X.lo[0] + (int) (lin % (unsigned) X.nb[0]), j = X.lo[1] + (int) (lin / (unsigned) X.nb[0]);
    const int k = X.lo[2] + (int) blockIdx.y;
    const long long stride = X.axis == 0 ? 1 : X.axis == 1 ? (long long) G.N[0] : (long long) G.N[0] * G.N[1];
    const double* n = G.nrm[X.axis];
    const int e = face_general<LAW, RECON, RIEMANN>(P + ((long long) k * G.N[1] + j) * G.N[0] + i, G.sP, stride, n[0],
                                                    n[1], n[2], &pp,
                                                    F + ((long long) k * (G.N[1] + 1) + j) * (G.N[0] + 1) + i, G.sF);
    if (e != ST_OK) record_status(st, e);
}

// ---------------------------------------------------------------------------
// The faces of one axis, a block's threads sharing a tile of them in three
// phases through shared memory: the edge values of every (zone, field), the
// state of every (face, side), the HLLE flux of every (face, field) or the
// HLLC flux of every face.  A face whose operands are not ordinary
// (fast64.cuh) goes through face_general.  Each phase is a short loop over independent items, so its code stays in the
// instruction cache and small grids still fill the schedulers.  Bound by the
// FP64 pipe (66 to 72 % busy).  Against a thread per run of faces: MHD
// 64x56x48 115 to 138 -> 91 to 102 us an axis, a 1024-zone tube's run 2.95 ->
// 2.77 ms.  Blocks of 32, 64, 128 and 256 threads: 3.26, 3.27, 3.32, 3.43 ms
// (MHD 64x56x48, two steps and their transfers).
struct TileSpace {
    int lo[3];      // first face (right cell) and rows of each axis
    int nf;         // faces along the axis
    int ncol;       // rows of the axis that runs across the tile
    int len;        // faces along a tile
    int na, nc;     // tiles along and across
};

constexpr int TILE_THREADS = 64, TILE_FACES = TILE_THREADS / 2, TILE_ZONES = TILE_FACES + 4;

static __device__ __noinline__ void weno5_edges_small(const fast64::Consts& C, const double* p, long long s, double& left,
                                                      double& right, bool* ok)
{
    const double w[5] = {p[-2 * s], p[-s], p[0], p[s], p[2 * s]};
    fast64::weno5_edges<true>(C, &w[2], left, right, *ok);
}

template <int LAW> constexpr bool NEWTONIAN_MHD = LAW == LAW_MHD || LAW == LAW_MHD_COOL;

// whether zone_edges takes a field: for Newtonian MHD only large ones, small
// ones are left to odd_sides
template <int LAW> __device__ __forceinline__ bool lean_field(int q, double x)
{
    if constexpr (LAW == LAW_RMHD) return fast64::ordinary_field<LAW>(q, x);
    else return fast64::ordinary_field(q, x);
}

template <int LAW, int RECON>
__device__ __forceinline__ void zone_edges(const fast64::Consts& C, const double* p, long long s, int q, double& left,
                                           double& right, bool& ok)
{
    if constexpr (RECON == RECON_PCM) {
        left = right = p[0];
        ok = ok && lean_field<LAW>(q, p[0]);
    } else if constexpr (RECON == RECON_PLM) {
        const double l = p[-s], c = p[0], r = p[s];
        const double h = fast64::half_slope(fast64::mul(C.theta, c - l), r - l, fast64::mul(C.theta, r - c));
        left = c - h;
        right = c + h;
        ok = ok && lean_field<LAW>(q, l) && lean_field<LAW>(q, c) && lean_field<LAW>(q, r);
    } else {
        const double w[5] = {p[-2 * s], p[-s], p[0], p[s], p[2 * s]};
#pragma unroll
        for (int m = 0; m < 5; ++m) ok = ok && fast64::ordinary_field(q, w[m]);
        if constexpr (LAW == LAW_RMHD) {
            if (!ok) {
                ok = true;
                for (int m = 0; m < 5; ++m) ok = ok && fast64::ordinary_field<LAW>(q, w[m]);
                if (ok) weno5_edges_small(C, p, s, left, right, &ok);
                return;
            }
        }
        fast64::weno5_edges(C, &w[2], left, right, ok);
    }
}

// a block's shared memory
template <int NQ> struct TileShared {
    double edge[2][NQ][TILE_ZONES];           // left and right edge of each zone
    double U[2][NQ][TILE_FACES], F[2][NQ][TILE_FACES], A[2][2][TILE_FACES];   // states by side; ap, am
    unsigned char odd_zone[TILE_ZONES], odd_face[TILE_FACES];                 // operands out of the ordinary
    alignas(4) unsigned char odd_field[NQ][TILE_ZONES];                       // Newtonian MHD: the zone's fields not taken by zone_edges
};

// the state on side s of face f, from zone z's edge
template <int LAW, int AXIS, bool SMALL>
__device__ __forceinline__ void face_side(const fast64::Consts& C, TileShared<LawInfo<LAW>::NQ>& sm, int s, int f, int z)
{
    constexpr int NQ = LawInfo<LAW>::NQ;
    double P[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) P[q] = sm.edge[1 - s][q][z];
    fast64::Side<NQ> S;
    bool ok = C.ok && !sm.odd_zone[z];
    if constexpr (LAW == LAW_RMHD) fast64::rmhd_side<AXIS>(C, P, S, ok);
    else fast64::side<LAW, AXIS, SMALL>(C, P, S, ok);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        sm.U[s][q][f] = S.U[q];
        sm.F[s][q][f] = S.F[q];
    }
    sm.A[s][0][f] = S.ap;
    sm.A[s][1][f] = S.am;
    if (!ok) sm.odd_face[f] = 1;
}
// The states of a tile of Newtonian MHD with fields that zone_edges did not
// take: their edges first, then the states, all by the SMALL form (of two forms
// a warp would run both).
// As a call for the whole block, so that other tiles do not pay for it: with a
// call and a branch per item they took 1 to 2 % longer, with the flags as bits
// set by atomics 1 %.
template <int LAW, int RECON, int AXIS>
__device__ __noinline__ void odd_sides(const fast64::Consts& C, TileShared<LawInfo<LAW>::NQ>& sm, const double* p,
                                       long long sP, long long stride, long long cstride, int faces, int width)
{
    constexpr int NQ = LawInfo<LAW>::NQ, WIDTH = AXIS == 0 ? 1 : 4;
    constexpr int S = ReconInfo<RECON>::S - 1;   // zones on either side
    const int zones = faces + WIDTH;
    for (int it = threadIdx.x; it < NQ * zones; it += TILE_THREADS) {
        const int q = it / zones, z = it - q * zones;
        if (!sm.odd_field[q][z]) continue;
        const double* v = p + q * sP + (z / WIDTH - 1) * stride + z % WIDTH * cstride;
        bool ok = true;
        for (int m = -S; m <= S; ++m) ok = ok && fast64::ordinary_field<LAW>(q, v[m * stride]);
        double left = v[0], right = v[0];
        if constexpr (RECON == RECON_PLM) {
            const double l = v[-stride], r = v[stride];
            const double h = fast64::half_slope(fast64::mul(C.theta, left - l), r - l, fast64::mul(C.theta, r - left));
            left -= h;
            right += h;
        } else if constexpr (RECON == RECON_WENO5) {
            if (ok) weno5_edges_small(C, v, stride, left, right, &ok);
        }
        sm.edge[0][q][z] = left;
        sm.edge[1][q][z] = right;
        if (!ok) sm.odd_zone[z] = 1;
    }
    __syncthreads();
    const int tid = threadIdx.x;
    if (tid < 2 * faces && tid % WIDTH < width) {
        const int s = tid >= faces ? 1 : 0, f = tid - s * faces, z = f + s * WIDTH;
        face_side<LAW, AXIS, true>(C, sm, s, f, z);
    }
}

// tile b of the faces along AXIS
template <int LAW, int RECON, int RIEMANN, int AXIS>
__device__ __forceinline__ void flux_tile(TileShared<LawInfo<LAW>::NQ>& sm, const double* P,
                                          double* __restrict__ F, const GridDesc& G, const PhysParams& pp,
                                          const fast64::Consts& C, const TileSpace& X, int b, DevStatus* st)
{
    constexpr int NQ = LawInfo<LAW>::NQ;
    const int tid = threadIdx.x;
    // across the tile: one row for faces along x, else four zones of x (a
    // 32-byte sector; at the grid's edge fewer, their items skipped)
    constexpr int WIDTH = AXIS == 0 ? 1 : 4;
    const int a0 = (b % X.na) * X.len, c0 = (b / X.na) % X.nc * WIDTH, o = b / X.na / X.nc;
    const int len = min(X.len, X.nf - a0), width = min(WIDTH, X.ncol - c0);
    const int faces = len * WIDTH, zones = faces + WIDTH;
    const int i = X.lo[0] + (AXIS == 0 ? a0 : c0);
    const int j = X.lo[1] + (AXIS == 1 ? a0 : AXIS == 0 ? c0 : o);
    const int k = X.lo[2] + (AXIS == 2 ? a0 : o);
    const long long s0 = 1, s1 = G.N[0], s2 = (long long) G.N[0] * G.N[1];
    const long long stride = AXIS == 0 ? s0 : AXIS == 1 ? s1 : s2, cstride = AXIS == 0 ? s1 : s0;
    const double* p = P + ((long long) k * G.N[1] + j) * G.N[0] + i;   // cell on the right of the tile's first face
    bool odd = false;
    for (int q = 0, z = tid; q < NQ; z += TILE_THREADS) {
        for (; z >= zones && q < NQ; z -= zones) ++q;
        const int s = z / WIDTH, w = z % WIDTH;
        if (q >= NQ) break;
        if (w >= width) continue;
        bool ok = true;
        double l, r;
        zone_edges<LAW, RECON>(C, p + q * G.sP + (s - 1) * stride + w * cstride, stride, q, l, r, ok);
        sm.edge[0][q][z] = l;
        sm.edge[1][q][z] = r;
        if (!ok) {
            if constexpr (NEWTONIAN_MHD<LAW>) sm.odd_field[q][z] = 1;
            else sm.odd_zone[z] = 1;
            odd = true;
        }
    }
    if (__syncthreads_or(odd) && NEWTONIAN_MHD<LAW>) {
        odd_sides<LAW, RECON, AXIS>(C, sm, p, G.sP, stride, cstride, faces, width);
    } else if (tid < 2 * faces && tid % WIDTH < width) {
        const int s = tid >= faces ? 1 : 0, f = tid - s * faces;
        face_side<LAW, AXIS, false>(C, sm, s, f, f + s * WIDTH);
    }
    __syncthreads();
    const long long f0 = 1, f1 = G.N[0] + 1, f2 = (long long) (G.N[0] + 1) * (G.N[1] + 1);
    const long long fstride = AXIS == 0 ? f0 : AXIS == 1 ? f1 : f2, fcstride = AXIS == 0 ? f1 : f0;
    double* out = F + ((long long) k * (G.N[1] + 1) + j) * (G.N[0] + 1) + i;
    if constexpr (RIEMANN == RIEMANN_HLLE) {
        for (int q = 0, f = tid; q < NQ; f += TILE_THREADS) {
            for (; f >= faces && q < NQ; f -= faces) ++q;
            const int s = f / WIDTH, w = f % WIDTH;
            if (q >= NQ) break;
            if (w >= width) continue;
            bool ok = !sm.odd_face[f];
            const double h = fast64::hlle(sm.A[0][0][f], sm.A[1][0][f], sm.A[0][1][f], sm.A[1][1][f], sm.F[0][q][f],
                                          sm.F[1][q][f], sm.U[0][q][f], sm.U[1][q][f], ok);
            double* to = out + s * fstride + w * fcstride;
            if (ok) to[q * G.sF] = h;
            else sm.odd_face[f] = 1;   // every field of the face by the general functions, below
        }
    } else if (tid < faces && tid % WIDTH < width) {
        // HLLC's star state couples the fields: a thread per face
        const int f = tid, s = f / WIDTH, w = f % WIDTH;
        double Pl[NQ], Pr[NQ], h[NQ];
        fast64::Side<NQ> L, R;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            Pl[q] = sm.edge[1][q][f];
            Pr[q] = sm.edge[0][q][f + WIDTH];
            L.U[q] = sm.U[0][q][f];
            R.U[q] = sm.U[1][q][f];
            L.F[q] = sm.F[0][q][f];
            R.F[q] = sm.F[1][q][f];
        }
        L.ap = sm.A[0][0][f];
        L.am = sm.A[0][1][f];
        R.ap = sm.A[1][0][f];
        R.am = sm.A[1][1][f];
        L.vn = fast64::along<AXIS>(C, Pl[1], Pl[2], Pl[3]);
        R.vn = fast64::along<AXIS>(C, Pr[1], Pr[2], Pr[3]);
        bool ok = !sm.odd_face[f];
        fast64::hllc<AXIS>(C, Pl, Pr, L, R, h, ok);
        double* to = out + s * fstride + w * fcstride;
        if (ok) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) to[q * G.sF] = h[q];
        } else {
            sm.odd_face[f] = 1;
        }
    }
    __syncthreads();
    if (tid < faces && sm.odd_face[tid]) {
        const int s = tid / WIDTH, w = tid % WIDTH;
        const int e = face_general<LAW, RECON, RIEMANN>(p + s * stride + w * cstride, G.sP, stride,
                                                             G.nrm[AXIS][0], G.nrm[AXIS][1], G.nrm[AXIS][2], &pp,
                                                             out + s * fstride + w * fcstride, G.sF);
        if (e != ST_OK) record_status(st, e);
    }
}

// All axes in one launch: the tiles of axis a are blocks first[a] to
// first[a + 1] - 1, so that small grids run their axes side by side.
struct TileSpaces {
    TileSpace axis[3];
    int first[4];
    double* F[3];
};

template <int LAW, int RECON, int RIEMANN>
__global__ void __launch_bounds__(TILE_THREADS, 512 / TILE_THREADS)
    flux_tile_kernel(const double* P, const __grid_constant__ TileSpaces X,
                     const __grid_constant__ GridDesc G, const __grid_constant__ PhysParams pp,
                     const __grid_constant__ fast64::Consts C, DevStatus* __restrict__ st)
{
    pdl_wait();
    __shared__ TileShared<LawInfo<LAW>::NQ> sm;
    const int tid = threadIdx.x;
    for (int z = tid; z < TILE_ZONES; z += TILE_THREADS) sm.odd_zone[z] = 0;
    if constexpr (NEWTONIAN_MHD<LAW>)
        for (int w = tid; w < (int) sizeof(sm.odd_field) / 4; w += TILE_THREADS) ((unsigned*) sm.odd_field)[w] = 0;
    if (tid < TILE_FACES) sm.odd_face[tid] = 0;
    const int code = st->code, failures = st->failures;
    if (__syncthreads_or(code != 0 || st->done || failures != 0)) {
        if (code == 0 && failures != 0) st->halt = 1;    // failures are final once the stage ended
        return;
    }
    const int b = blockIdx.x;
    if (b < X.first[1]) flux_tile<LAW, RECON, RIEMANN, 0>(sm, P, X.F[0], G, pp, C, X.axis[0], b, st);
    else if (b < X.first[2]) flux_tile<LAW, RECON, RIEMANN, 1>(sm, P, X.F[1], G, pp, C, X.axis[1], b - X.first[1], st);
    else flux_tile<LAW, RECON, RIEMANN, 2>(sm, P, X.F[2], G, pp, C, X.axis[2], b - X.first[2], st);
}

// ---------------------------------------------------------------------------
// The PLM HLLC faces of one axis of a large hydro grid, each thread a run of
// consecutive faces along it: a zone's slopes serve the faces on both of its
// sides without a trip through shared memory.  Bound by the FP64 pipe (KH
// 1024^2 658 to 714 -> about 185 us an axis, of which the additions alone
// take 170).
struct RunSpace {
    int lo[3];   // first face (right cell) and row of each axis
    int nb[3];   // threads per axis: runs along the faces' axis, rows across it
    int nf, run; // faces along the axis, faces per run
};

// Three blocks per SM (168 registers): 4, 5 and 6 lose 1, 6 and 11 % to spills.
template <int AXIS>
__global__ void __launch_bounds__(128, 3) flux_run_kernel(const double* P, double* __restrict__ F,
                                                          const __grid_constant__ GridDesc G,
                                                          const __grid_constant__ PhysParams pp,
                                                          const __grid_constant__ fast64::Consts C,
                                                          const __grid_constant__ RunSpace X,
                                                          DevStatus* __restrict__ st)
{
    constexpr int NQ = LawInfo<LAW_HYDRO>::NQ;
    pdl_wait();
    if (st->code != 0 || st->done) return;
    if (st->failures != 0) { st->halt = 1; return; }  // failures are final once the stage ended
    const unsigned lin = blockIdx.x * blockDim.x + threadIdx.x;
    if (lin >= (unsigned) X.nb[0] * (unsigned) X.nb[1]) return;
    int x[3] = {(int) (lin % (unsigned) X.nb[0]), (int) (lin / (unsigned) X.nb[0]), (int) blockIdx.y};
    const int first = (AXIS == 0 ? x[0] : AXIS == 1 ? x[1] : x[2]) * X.run;
    const int count = min(X.run, X.nf - first);
    if (AXIS == 0) x[0] = first;
    else if (AXIS == 1) x[1] = first;
    else x[2] = first;
    const int i = X.lo[0] + x[0], j = X.lo[1] + x[1], k = X.lo[2] + x[2];
    const long long stride = AXIS == 0 ? 1 : AXIS == 1 ? (long long) G.N[0] : (long long) G.N[0] * G.N[1];
    const long long fstride = AXIS == 0   ? 1
                              : AXIS == 1 ? (long long) (G.N[0] + 1)
                                          : (long long) (G.N[0] + 1) * (G.N[1] + 1);
    const double* p = P + ((long long) k * G.N[1] + j) * G.N[0] + i;  // cell on the right of the face
    double* f = F + ((long long) k * (G.N[1] + 1) + j) * (G.N[0] + 1) + i;

    // PL: the right edge of the zone on the face's left; d: the scaled
    // difference across the face; fine: one bit per zone of the stencil, set
    // where its values are ordinary
    double PL[NQ], d[NQ];
    unsigned fine = 0;
#pragma unroll
    for (int z = -2; z < 1; ++z) {
        bool o = true;
#pragma unroll
        for (int q = 0; q < NQ; ++q) o = o && fast64::ordinary_field(q, p[q * G.sP + z * stride]);
        fine = 2 * fine + o;
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const double* v = p + q * G.sP;
        const double a = C.theta * (v[-stride] - v[-2 * stride]);
        d[q] = C.theta * (v[0] - v[-stride]);
        PL[q] = v[-stride] + fast64::half_slope(a, v[0] - v[-2 * stride], d[q]);
    }
    for (int m = 0; m < count; ++m, p += stride, f += fstride) {
        double PR[NQ], next[NQ];
        bool o = true;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const double* v = p + q * G.sP;
            const double c = v[0], r = v[stride];
            const double b = C.theta * (r - c);
            const double h = fast64::half_slope(d[q], r - v[-stride], b);
            d[q] = b;
            PR[q] = c - h;
            next[q] = c + h;
            o = o && fast64::ordinary_field(q, r);
        }
        fine = 2 * fine + o;
        bool ok = C.ok && (fine & 15u) == 15u;
        // the two sides in a loop: its code once (the kernel runs out of the
        // instruction cache; KH 1024^2, four steps, 5.42 -> 5.27 ms)
        fast64::Side<NQ> L, R;
        double Ps[NQ], h[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) Ps[q] = PL[q];
#pragma unroll 1
        for (int s = 0; s < 2; ++s) {
            fast64::hydro_side<AXIS>(C, Ps, R, ok);
            if (s == 0) {
                L = R;
#pragma unroll
                for (int q = 0; q < NQ; ++q) Ps[q] = PR[q];
            }
        }
        fast64::hllc<AXIS>(C, PL, PR, L, R, h, ok);
        if (ok) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) f[q * G.sF] = h[q];
        } else {
            const int e = face_general<LAW_HYDRO, RECON_PLM, RIEMANN_HLLC>(p, G.sP, stride, G.nrm[AXIS][0],
                                                                           G.nrm[AXIS][1], G.nrm[AXIS][2], &pp, f, G.sF);
            if (e != ST_OK) { record_status(st, e); return; }
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) PL[q] = next[q];
    }
}

// ---------------------------------------------------------------------------
struct FluxView {
    const double* F[3];
    long long sF;
    int M0, M1; // (N0+1), (N1+1)
    __device__ __forceinline__ double at(int a, int q, int i, int j, int k) const
    {
        return F[a][q * sF + ((long long) k * M1 + j) * M0 + i];
    }
};

// Flux of field q through the face of axis a at flux index (i, j, k), after
// CellCenteredFieldCT::correctGodunovFluxes when ct is on (magnetic index 5):
// 1/8 of (2 F + ...), its powers of two on the exponents.
template <int NQ>
__device__ __forceinline__ double face_flux(const FluxView& V, const GridDesc& G, int a, int q, int i, int j, int k)
{
    if ((NQ == 8 || NQ == 9) && G.ct && q >= 5 && q <= 7) {
        const int B0 = 5, B1 = 6, B2 = 7;
        const bool fx = G.n[0] > 1, fy = G.n[1] > 1, fz = G.n[2] > 1;
        if (a == 0) {
            if (q == B0) return 0.0;
            if (q == B1 && fy)
                return times_pow2(times_pow2(V.at(0, B1, i, j, k), 1) + V.at(0, B1, i, j + 1, k) + V.at(0, B1, i, j - 1, k)
                                - V.at(1, B0, i, j + 1, k) - V.at(1, B0, i - 1, j + 1, k)
                                - V.at(1, B0, i, j, k) - V.at(1, B0, i - 1, j, k), -3);
            if (q == B2 && fz)
                return times_pow2(times_pow2(V.at(0, B2, i, j, k), 1) + V.at(0, B2, i, j, k + 1) + V.at(0, B2, i, j, k - 1)
                                - V.at(2, B0, i, j, k + 1) - V.at(2, B0, i - 1, j, k + 1)
                                - V.at(2, B0, i, j, k) - V.at(2, B0, i - 1, j, k), -3);
        } else if (a == 1) {
            if (q == B1) return 0.0;
            if (q == B2 && fz)
                return times_pow2(times_pow2(V.at(1, B2, i, j, k), 1) + V.at(1, B2, i, j, k + 1) + V.at(1, B2, i, j, k - 1)
                                - V.at(2, B1, i, j, k + 1) - V.at(2, B1, i, j - 1, k + 1)
                                - V.at(2, B1, i, j, k) - V.at(2, B1, i, j - 1, k), -3);
            if (q == B0 && fx)
                return times_pow2(times_pow2(V.at(1, B0, i, j, k), 1) + V.at(1, B0, i + 1, j, k) + V.at(1, B0, i - 1, j, k)
                                - V.at(0, B1, i + 1, j, k) - V.at(0, B1, i + 1, j - 1, k)
                                - V.at(0, B1, i, j, k) - V.at(0, B1, i, j - 1, k), -3);
        } else {
            if (q == B2) return 0.0;
            if (q == B0 && fx)
                return times_pow2(times_pow2(V.at(2, B0, i, j, k), 1) + V.at(2, B0, i + 1, j, k) + V.at(2, B0, i - 1, j, k)
                                - V.at(0, B2, i + 1, j, k) - V.at(0, B2, i + 1, j, k - 1)
                                - V.at(0, B2, i, j, k) - V.at(0, B2, i, j, k - 1), -3);
            if (q == B1 && fy)
                return times_pow2(times_pow2(V.at(2, B1, i, j, k), 1) + V.at(2, B1, i, j + 1, k) + V.at(2, B1, i, j - 1, k)
                                - V.at(1, B2, i, j + 1, k) - V.at(1, B2, i, j + 1, k - 1)
                                - V.at(1, B2, i, j, k) - V.at(1, B2, i, j, k - 1), -3);
        }
    }
    return V.at(a, q, i, j, k);
}

// The weight b of an RK stage (SolutionSchemes.cpp:135-138) and 1 - b.
struct RkWeight {
    int kind;        // 0: b = 1, 1: 1/2, 2: 1/4, 3: any
    double b, rest;
};
__host__ __device__ inline RkWeight rk_weight(int order, int stage)
{
    const double b = order == 1 || stage == 0 ? 1.0 : order == 2 ? 0.5 : stage == 1 ? 1. / 4 : 2. / 3;
    return {b == 1.0 ? 0 : b == 0.5 ? 1 : b == 0.25 ? 2 : 3, b, 1 - b};
}

// U0 (1 - b) + (U + dt L) b
__device__ __forceinline__ double rk_combine_plain(double Uo, double Up, double L, double dt, const RkWeight& w)
{
    const double X = Up + fast64::mul_any(dt, L);
    if (w.kind == 0)   // U0 0 + X: a zero plus X (NaN for an infinite U0)
        return fast64::expo(Uo) == 0x7ffu ? Uo * w.rest + X : fast64::add_zero(X, fast64::sign_bit(Uo));
    if (w.kind == 1) return times_pow2(Uo, -1) + times_pow2(X, -1);
    if (w.kind == 2) return fast64::mul_any(Uo, w.rest) + times_pow2(X, -2);
    return fast64::mul_any(Uo, w.rest) + fast64::mul_any(X, w.b);
}

// One RK stage's update of a zone (see the file's comment).  Bound by the
// FP64 pipe, so the face area products of flat axes (zeros) are left out, and
// the RK weights 1, 1/2 and 1/4 act on exponents.
// Resident blocks: hydro 1 to 5 a SM 5.60 ms, 8 5.39 (KH 1024^2, four steps);
// MHD 1 3.94, 4 3.66, 5 3.57, 8 3.67 (64x56x48).
template <int LAW>
__global__ void __launch_bounds__(128, LAW == LAW_HYDRO ? 8 : LAW == LAW_RMHD ? 1 : 5) update_kernel(const double* Pin, double* __restrict__ Pout,
                                                     double* __restrict__ U0, double* __restrict__ U,
                                                     const __grid_constant__ FluxView V,
                                                     const __grid_constant__ GridDesc G,
                                                     const __grid_constant__ PhysParams pp,
                                                     const __grid_constant__ fast64::Consts C, double fv,
                                                     const __grid_constant__ RkWeight w, int stage, const double* dtp,
                                                     DevStatus* __restrict__ st, const double* S)
{
    constexpr int NQ = LawInfo<LAW>::NQ;
    pdl_wait();
    if (st->code != 0 || st->halt || st->done) return;
    const unsigned lin = blockIdx.x * blockDim.x + threadIdx.x;
    if (lin >= (unsigned) G.n[0] * (unsigned) G.n[1]) return;
    const int ii = (int) (lin % (unsigned) G.n[0]), jj = (int) (lin / (unsigned) G.n[0]), kk = blockIdx.y;
    const int i = ii + G.g[0], j = jj + G.g[1], k = kk + G.g[2];
    const long long pc = ((long long) k * G.N[1] + j) * G.N[0] + i;
    const long long uc = ((long long) kk * G.n[1] + jj) * G.n[0] + ii;
    const double dt = *dtp;
    const bool fx = G.n[0] > 1, fy = G.n[1] > 1, fz = G.n[2] > 1;

    double Pc[NQ], Uo[NQ], Up[NQ], Un[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) Pc[q] = Pin[q * G.sP + pc];

    if (stage == 0) {
        bool ok = C.ok;
#pragma unroll
        for (int q = 0; q < NQ; ++q) ok = ok && fast64::ordinary_field<LAW>(q, Pc[q]);
        if constexpr (LAW == LAW_RMHD) fast64::rmhd_p2u(C, Pc, Uo, ok);
        else fast64::p2u<LAW>(C, Pc, Uo, ok);
        if (!ok) {
            const int e = law_p2u<LAW>(pp, Pc, Uo);
            if (e != ST_OK) { record_status(st, e); return; }
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) { U0[q * G.sU + uc] = Uo[q]; Up[q] = Uo[q]; }
    } else {
#pragma unroll
        for (int q = 0; q < NQ; ++q) { Uo[q] = U0[q * G.sU + uc]; Up[q] = U[q * G.sU + uc]; }
    }

    bool fine = C.ok;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        // the sum over the faces in the reference's order; a flat axis adds
        // and subtracts a zero, which only makes a -0 a +0.  (These products
        // in integers too: the two pipes out of balance, KH 1024^2, four
        // steps, 4.84 -> 5.09 ms.)
        double sum = 0.0;
        if (fx) sum = face_flux<NQ>(V, G, 0, q, i + 1, j, k) * G.dA[0] - face_flux<NQ>(V, G, 0, q, i, j, k) * G.dA[0];
        if (fy) sum = sum + face_flux<NQ>(V, G, 1, q, i, j + 1, k) * G.dA[1] - face_flux<NQ>(V, G, 1, q, i, j, k) * G.dA[1];
        else sum = fast64::add_zero(sum, false);
        if (fz) sum = sum + face_flux<NQ>(V, G, 2, q, i, j, k + 1) * G.dA[2] - face_flux<NQ>(V, G, 2, q, i, j, k) * G.dA[2];
        else sum = fast64::add_zero(sum, false);
        double L = fast64::mul_any(fv, sum);
        if constexpr (LAW == LAW_MHD_COOL) {
            // NewtonianMHD::addSourceTerms (ConservationLaws.cpp:489-501)
            if (q == 4) L -= Pc[4] / (pp.gamma - 1.0) * pp.cooling_rate;
            if (q == 8) L += Pc[4] / (pp.gamma - 1.0) * pp.cooling_rate;
        }
        if (S) L += S[q * G.sP + pc];  // the source terms function's array (SolutionSchemes.cpp:219-228)
        Un[q] = rk_combine_plain(Uo[q], Up[q], L, dt, w);
        U[q * G.sU + uc] = Un[q];
        fine = fine && fast64::ordinary_field<LAW>(q, Un[q]);
    }

    double Pn[NQ];
    if constexpr (LAW == LAW_RMHD) fast64::rmhd_cons(C, Un, Pn, fine);
    else fast64::cons<LAW>(C, Un, Pn, fine);
    if (!fine) {
        int code = ST_OK;
        const int e = law_cons<LAW>(pp, Un, Pn, &code);
        if (e == ST_INVERSION_FAILURE) {
            atomicAdd(&st->failures, 1);
            const unsigned long long z = (unsigned long long) uc;
            const unsigned long long prev = atomicMin(&st->first_zone, z);
            if (z < prev) atomicExch(&st->first_code, code);
#pragma unroll
            for (int q = 0; q < NQ; ++q) Pn[q] = Pc[q]; // a failed zone keeps its value
        } else if (e != ST_OK) {
            record_status(st, e);
            return;
        }
    }

    // the zone's cell, then (zones within a guard width of an edge) its guard
    // images on every combination of axes
    for (int c = 0; c <= G.g[2]; ++c) {
        int oz, sz;
        if (!guard_image(c, kk, G.n[2], G.g[2], G.bc, oz, sz)) continue;
        for (int bb = 0; bb <= G.g[1]; ++bb) {
            int oy, sy;
            if (!guard_image(bb, jj, G.n[1], G.g[1], G.bc, oy, sy)) continue;
            for (int a = 0; a <= G.g[0]; ++a) {
                int ox, sx;
                if (!guard_image(a, ii, G.n[0], G.g[0], G.bc, ox, sx)) continue;
                const long long o = ((long long) oz * G.N[1] + oy) * G.N[0] + ox;
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    double v = Pn[q];
                    if ((q == 1 && sx) || (q == 2 && sy) || (q == 3 && sz)) v *= -1;
                    Pout[q * G.sP + o] = v;
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// FieldOperator::getCourantTimestep: min over interior zones of
// lmin / max_direction(maxEigenvalueMagnitude).  Positive doubles order like
// their bit patterns, so the minimum is an atomicMin on the bits; NaN and
// +inf (bit patterns above DBL_MAX) never win, as in the reference's
// "if (dt < courantTimestep)" starting from DBL_MAX.
// lmin / lambda falls with lambda, also after rounding, so a block divides
// once, by its largest eigenvalue.
template <int LAW>
__global__ void __launch_bounds__(128) courant_kernel(const double* P,
                                                      const __grid_constant__ GridDesc G,
                                                      const __grid_constant__ PhysParams pp,
                                                      const __grid_constant__ fast64::Consts C,
                                                      DevStatus* __restrict__ st)
{
    constexpr int NQ = LawInfo<LAW>::NQ;
    pdl_wait();
    // the relativistic law's three normals cost a quartic each: a thread each
    constexpr int AXES = LAW == LAW_RMHD ? 3 : 1;
    const unsigned slice = (unsigned) G.n[0] * (unsigned) G.n[1];
    const unsigned item = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long mine = 0;
    if (item < AXES * slice && st->code == 0) {
        const int axis = (int) (item / slice);
        const unsigned lin = item - axis * slice;
        const int ii = (int) (lin % (unsigned) G.n[0]), jj = (int) (lin / (unsigned) G.n[0]), kk = blockIdx.y;
        const long long pc = ((long long) (kk + G.g[2]) * G.N[1] + (jj + G.g[1])) * G.N[0] + (ii + G.g[0]);
        double Pc[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) Pc[q] = P[q * G.sP + pc];
        double lmax = 0.0;
        bool ok = C.ok;
#pragma unroll
        for (int q = 0; q < NQ; ++q) ok = ok && fast64::ordinary_field<LAW>(q, Pc[q]);
        if constexpr (LAW == LAW_RMHD) lmax = fast64::rmhd_fastest(C, Pc, axis, ok);
        else lmax = fast64::fastest<LAW>(C, Pc, ok);
        if (!ok) {
            int e = ST_OK;
            lmax = 0.0;
            for (int a = AXES == 3 ? axis : 0; a <= (AXES == 3 ? axis : 2) && e == ST_OK; ++a) {
                StateD<NQ> S;
                e = law_prim<LAW>(pp, Pc, G.nrm[a], S);
                const double lam = max_eigen_magnitude<NQ>(S.A);
                if (e == ST_OK && lmax < lam) lmax = lam;
            }
            if (e != ST_OK) {
                record_status(st, e);
                lmax = 0.0;
            }
        }
        mine = (unsigned long long) __double_as_longlong(lmax);
    }
    // warp then block maximum
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_down_sync(0xffffffffu, mine, off);
        mine = o > mine ? o : mine;
    }
    __shared__ unsigned long long red[4];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) red[w] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int m = 1; m < (int) (blockDim.x >> 5); ++m) mine = red[m] > mine ? red[m] : mine;
        const double dt = G.lmin / __longlong_as_double((long long) mine);
        if (dt < 1.7976931348623157e308) atomicMin(&st->dt_bits, (unsigned long long) __double_as_longlong(dt));
    }
}

// ---------------------------------------------------------------------------
static PhysParams to_dev(const PhysParamsH& h)
{
    PhysParams p;
    p.gamma = h.gamma;
    p.plm_theta = h.plm_theta;
    p.shenzha_A = h.shenzha_A;
    p.pressure_floor = h.pressure_floor;
    p.weno_is = h.weno_is;
    p.cooling_rate = h.cooling_rate;
    return p;
}

static fast64::Consts to_fast(const PhysParamsH& h, const GridDesc& G)
{
    fast64::Consts c = fast64::make_consts(h.gamma, h.plm_theta, h.shenzha_A, h.weno_is, G.nrm[1][0]);
    for (int a = 0; a < 3; ++a)
        for (int d = 0; d < 3; ++d)
            if (!(a == 1 && d == 0)) c.ok = c.ok && G.nrm[a][d] == (a == d ? 1.0 : 0.0);
    return c;
}

// Threads per block: few warps are spread over the SMs' schedulers, each of
// which has its own half lane of FP64 per clock.
static int block_size(long long threads) { return threads <= 152ll * 4 * 32 ? 32 : 128; }

// faces along the axis: the interior faces; across: interior rows, plus one
// guard row per side on fleshed axes when flux CT is on
static void face_rows(const GridDesc& G, int axis, int* lo, int* nb)
{
    for (int a = 0; a < 3; ++a) {
        const int e = G.n[a] > 1 && a != axis && G.ct ? 1 : 0;
        lo[a] = G.g[a] - e;
        nb[a] = G.n[a] + 2 * e + (a == axis ? 1 : 0);
    }
}

// From this size on a thread per run of faces (KH with PLM, tiles against
// runs: 128^2, 16 steps 1.09 and 1.25 ms; 256^2, 16 steps 2.21 and 2.25;
// 400^2, 8 steps 2.28 and 2.15; 1024^2, 4 steps 6.63 and 5.23; with WENO5 the
// tiles win at all of them, 640^2 by 7.3 to 11.9)
constexpr long long HLLC_RUN_ZONES = 1ll << 17;
inline bool in_face_runs(int law, int recon, int riemann, const GridDesc& G)
{
    return law == LAW_HYDRO && recon == RECON_PLM && riemann == RIEMANN_HLLC &&
           (long long) G.n[0] * G.n[1] * G.n[2] >= HLLC_RUN_ZONES;
}

template <int LAW>
static void flux_runs(int launch, const GridDesc& G, const PhysParams& pp, const fast64::Consts& C, const double* P,
                      double* const* F, DevStatus* st, cudaStream_t s)
{
    for (int axis = 0; axis < 3; ++axis) {
        if (G.n[axis] <= 1 || launch-- != 0) continue;
        RunSpace X;
        face_rows(G, axis, X.lo, X.nb);
        // a run of one forms every zone's slopes twice, one of eight 1/8 too
        // many: runs as long as four waves of resident threads remain (KH
        // 1024^2, four steps: 5.42 ms at 4 faces a run, 5.61 at 8 and 2, 6.28 at 1)
        const long long faces = (long long) X.nb[0] * X.nb[1] * X.nb[2], want = 152ll * 1536;
        X.nf = X.nb[axis];
        X.run = (int) (faces < 2 * want ? 1 : faces > 8 * want ? 8 : faces / want);
        X.nb[axis] = (X.nf + X.run - 1) / X.run;
        const long long slice = (long long) X.nb[0] * X.nb[1];
        const dim3 grid((unsigned) ((slice + 127) / 128), X.nb[2]);
        switch (axis) {
            case 0: chain_launch(flux_run_kernel<0>, grid, dim3(128), s, P, F[0], G, pp, C, X, st); break;
            case 1: chain_launch(flux_run_kernel<1>, grid, dim3(128), s, P, F[1], G, pp, C, X, st); break;
            default: chain_launch(flux_run_kernel<2>, grid, dim3(128), s, P, F[2], G, pp, C, X, st); break;
        }
    }
}

template <int LAW, int RECON, int RIEMANN>
static void flux_launch(int launch, const GridDesc& G, const PhysParams& pp, const fast64::Consts& C, const double* P,
                        double* const* F, DevStatus* st, cudaStream_t s)
{
    if constexpr (RIEMANN == RIEMANN_HLLC && LAW != LAW_HYDRO) {
        for (int axis = 0; axis < 3; ++axis) {
            if (G.n[axis] <= 1 || launch-- != 0) continue;
            FaceSpace X;
            face_rows(G, axis, X.lo, X.nb);
            X.axis = axis;
            const long long slice = (long long) X.nb[0] * X.nb[1];
            const int block = block_size(slice * X.nb[2]);
            const dim3 grid((unsigned) ((slice + block - 1) / block), X.nb[2]);
            chain_launch(flux_general_kernel<LAW, RECON, RIEMANN>, grid, dim3(block), s, P, F[axis], G, pp, X, st);
        }
    } else {
        if constexpr (LAW == LAW_HYDRO && RIEMANN == RIEMANN_HLLC && RECON == RECON_PLM) {
            if (in_face_runs(LAW, RECON, RIEMANN, G)) {
                flux_runs<LAW>(launch, G, pp, C, P, F, st, s);
                return;
            }
        }
        TileSpaces X;
        X.first[0] = 0;
        for (int axis = 0; axis < 3; ++axis) {
            X.first[axis + 1] = X.first[axis];
            X.F[axis] = F[axis];
            if (G.n[axis] <= 1) continue;
            TileSpace& T = X.axis[axis];
            int nb[3];
            face_rows(G, axis, T.lo, nb);
            const int width = axis == 0 ? 1 : 4;
            const int cross = axis == 0 ? 1 : 0, outer = axis == 2 ? 1 : 2;
            const int most = TILE_FACES / width;
            T.nf = nb[axis];
            T.ncol = nb[cross];
            T.na = (T.nf + most - 1) / most;
            T.len = (T.nf + T.na - 1) / T.na;   // tiles of equal length
            T.nc = (T.ncol + width - 1) / width;
            X.first[axis + 1] += T.na * T.nc * nb[outer];
        }
        chain_launch(flux_tile_kernel<LAW, RECON, RIEMANN>, dim3(X.first[3]), dim3(TILE_THREADS), s, P, X, G, pp, C, st);
    }
}

template <int LAW, int RECON>
static void flux_dispatch_r(int launch, int riemann, const GridDesc& G, const PhysParams& pp, const fast64::Consts& C,
                            const double* P, double* const* F, DevStatus* st, cudaStream_t s)
{
    if (riemann == RIEMANN_HLLC) flux_launch<LAW, RECON, RIEMANN_HLLC>(launch, G, pp, C, P, F, st, s);
    else flux_launch<LAW, RECON, RIEMANN_HLLE>(launch, G, pp, C, P, F, st, s);
}

template <int LAW>
void plain_flux_law(int launch, int recon, int riemann, const GridDesc& G, const PhysParamsH& ph, const double* P,
                    double* const* F, DevStatus* st, cudaStream_t s)
{
    const PhysParams pp = to_dev(ph);
    const fast64::Consts C = to_fast(ph, G);
    switch (recon) {
        case RECON_PCM: flux_dispatch_r<LAW, RECON_PCM>(launch, riemann, G, pp, C, P, F, st, s); break;
        case RECON_PLM: flux_dispatch_r<LAW, RECON_PLM>(launch, riemann, G, pp, C, P, F, st, s); break;
        default: flux_dispatch_r<LAW, RECON_WENO5>(launch, riemann, G, pp, C, P, F, st, s); break;
    }
}

template <int LAW>
void plain_update_law(const GridDesc& G, const PhysParamsH& ph, const double* Pin, double* Pout, double* U0, double* U,
                      const double* Fx, const double* Fy, const double* Fz, int order, int stage, const double* dt,
                      DevStatus* st, cudaStream_t s, const double* S)
{
    const RkWeight w = rk_weight(order, stage);
    FluxView V;
    V.F[0] = Fx; V.F[1] = Fy; V.F[2] = Fz;
    V.sF = G.sF;
    V.M0 = G.N[0] + 1;
    V.M1 = G.N[1] + 1;
    const double factor = -1.0;
    const long long slice = (long long) G.n[0] * G.n[1];
    const int block = block_size(slice * G.n[2]);
    const dim3 grid((unsigned) ((slice + block - 1) / block), G.n[2]);
    chain_launch(update_kernel<LAW>, grid, dim3(block), s, Pin, Pout, U0, U, V, G, to_dev(ph), to_fast(ph, G),
                 factor / G.dV, w, stage, dt, st, S);
}

template <int LAW>
void plain_courant_law(const GridDesc& G, const PhysParamsH& ph, const double* P, DevStatus* st, cudaStream_t s)
{
    const long long slice = (long long) G.n[0] * G.n[1] * (LAW == LAW_RMHD ? 3 : 1);
    const int block = block_size(slice * G.n[2]);
    const dim3 grid((unsigned) ((slice + block - 1) / block), G.n[2]);
    chain_launch(courant_kernel<LAW>, grid, dim3(block), s, P, G, to_dev(ph), to_fast(ph, G), st);
}

// one translation unit per law instantiates the kernels (plain_*.cu)
#define MARA_PLAIN_LAW(EXTERN, LAW)                                                                                  \
    EXTERN template void plain_flux_law<LAW>(int, int, int, const GridDesc&, const PhysParamsH&, const double*,      \
                                             double* const*, DevStatus*, cudaStream_t);                              \
    EXTERN template void plain_update_law<LAW>(const GridDesc&, const PhysParamsH&, const double*, double*, double*, \
                                               double*, const double*, const double*, const double*, int, int,      \
                                               const double*, DevStatus*, cudaStream_t, const double*);             \
    EXTERN template void plain_courant_law<LAW>(const GridDesc&, const PhysParamsH&, const double*, DevStatus*,      \
                                                cudaStream_t)

} // namespace mara

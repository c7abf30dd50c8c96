// plain_cluster.cuh -- many driver-loop steps of a small 1-D hydro grid of
// the plain FP64 path in one launch, on one thread-block cluster.
//
// A step of a small 1-D grid is a chain of dependent latencies: eight
// launches, each with a warp or less per scheduler (1024 zones, PLM, HLLE,
// RK2: 43 us a step, 17 us here).  Here the grid stays in the shared memory of a cluster
// of up to 16 CTAs, each holding m zones.  Per RK stage the cluster
// synchronises once, each CTA reads its halo from its neighbours' shared
// memory (distributed shared memory) or from the boundary images, and its
// threads share the edge values by (zone, field), the states by (face, side),
// the fluxes by (face, field), the RK combine by (zone, field) and the
// recovery by zone, so that every scheduler's half lane of FP64 has work.
// The Courant step is reduced across the cluster between a step's first states
// and its first update, so dt never leaves it.  Arithmetic, dt sequence, clock and buffers are those of the step
// kernels (plain_kernels.cuh), bit for bit; hydro has no error codes.
#pragma once

#include <cooperative_groups.h>

#include <cfloat>

#include "plain_kernels.cuh"

namespace mara {

// doubles of a CTA's shared memory for m zones with a halo of S: two buffers
// of primitives with halo, U0 and U, edges of m + 2 zones, states of m + 1
// faces' sides and their wave speeds, fluxes, two Courant slots
__host__ __device__ constexpr size_t plain_cluster_doubles(int m, int S)
{
    return 2 * 5 * (size_t) (m + 2 * S) + 10 * (size_t) m + 10 * (size_t) (m + 2) + 24 * (size_t) (m + 1) +
           5 * (size_t) (m + 1) + 2;
}

template <int RECON, int RIEMANN>
__global__ void __launch_bounds__(512) plain_cluster_kernel(double* __restrict__ Pa, double* __restrict__ Pb,
                                                            const __grid_constant__ GridDesc G,
                                                            const __grid_constant__ PhysParams pp,
                                                            const __grid_constant__ fast64::Consts C, double fv,
                                                            double cfl, double t_final, int order, int nsteps,
                                                            DevStatus* st)
{
    namespace cg = cooperative_groups;
    using fast64::u64;
    constexpr int NQ = 5, S = ReconInfo<RECON>::S;
    cg::cluster_group cluster = cg::this_cluster();
    const int nc = (int) cluster.num_blocks(), r = (int) cluster.block_rank();
    // the same words for every CTA: nothing writes them before the last barrier
    if (st->code != 0 || st->done || st->failures != 0 || st->halt) return;
    const int n = G.n[0], m = (n + nc - 1) / nc, z0 = r * m;
    const int mine = max(0, min(m, n - z0));
    const int tid = threadIdx.x, nt = blockDim.x, W = m + 2 * S;

    extern __shared__ double smem[];
    double* Pbuf = smem;                       // 2 x [5][W], zone z at z + S
    double* U0 = Pbuf + 2 * NQ * W;            // [5][m]
    double* U = U0 + NQ * m;                   // [5][m]
    double* E = U + NQ * m;                    // left, right edges: 2 x [5][m + 2], zone z at z + 1
    double* sU = E + 2 * NQ * (m + 2);         // [2][5][m + 1], side (left, right) of face f (left of zone f)
    double* sF = sU + 2 * NQ * (m + 1);
    double* sA = sF + 2 * NQ * (m + 1);        // [2][ap, am][m + 1]
    double* Fx = sA + 4 * (m + 1);             // [5][m + 1]
    u64* red = (u64*) (Fx + NQ * (m + 1));     // largest eigenvalue of this CTA's zones, by step parity
    __shared__ u64 wmax[16];
    __shared__ unsigned char odd_zone[4096 + 2], odd_face[4096 + 1];

    auto fastest = [&](const double* P) {      // P: the zone's five fields
        bool ok = C.ok;
#pragma unroll
        for (int q = 0; q < NQ; ++q) ok = ok && fast64::ordinary_field(q, P[q]);
        double lmax = fast64::fastest<LAW_HYDRO>(C, P, ok);
        if (!ok) {
            lmax = 0.0;
            for (int a = 0; a < 3; ++a) {
                StateD<NQ> T;
                law_prim<LAW_HYDRO>(pp, P, G.nrm[a], T);
                const double lam = max_eigen_magnitude<NQ>(T.A);
                if (lmax < lam) lmax = lam;
            }
        }
        return (u64) __double_as_longlong(lmax);
    };
    auto reduce = [&](u64 v, int slot) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const u64 o = __shfl_down_sync(0xffffffffu, v, off);
            v = o > v ? o : v;
        }
        if ((tid & 31) == 0) wmax[tid >> 5] = v;
        __syncthreads();
        if (tid == 0) {
            for (int k = 1; k < nt / 32; ++k) v = wmax[k] > v ? wmax[k] : v;
            red[slot] = v;
        }
    };

    // the state, and (first stage) the guards as they were uploaded
    for (int it = tid; it < NQ * (mine + 2 * S); it += nt) {
        const int q = it / (mine + 2 * S), z = it - q * (mine + 2 * S) - S;
        Pbuf[q * W + S + z] = Pa[q * G.sP + G.g[0] + z0 + z];
    }
    double t = st->t, dt = st->dt;
    u64 bits = 0;
    bool done = false, fresh = true;
    int par = 0, step = 0;
    for (; step < nsteps; ++step) {
        for (int rk = 0; rk < order; ++rk, par ^= 1, fresh = false) {
            const RkWeight w = rk_weight(order, rk);
            double* Ps = Pbuf + par * NQ * W;
            double* Pn = Pbuf + (par ^ 1) * NQ * W;
            cluster.sync();
            if (!fresh && tid < 2 * S) {
                const int local = tid < S ? tid - S : mine + (tid - S);
                int flip = 0;
                int z = z0 + local;
                if (z < 0 || z >= n) {
                    if (G.bc == BC_PERIODIC) z += z < 0 ? n : -n;
                    else if (G.bc == BC_OUTFLOW) z = z < 0 ? 0 : n - 1;
                    else { flip = 1; z = z < 0 ? -1 - z : 2 * n - 1 - z; }
                }
                const int owner = z / m;
                const double* src = cluster.map_shared_rank(Ps, owner);
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    double v = src[q * W + S + (z - owner * m)];
                    if (flip && q == 1) v *= -1;
                    Ps[q * W + S + local] = v;
                }
            }
            for (int z = tid; z < mine + 2; z += nt) odd_zone[z] = 0;
            for (int f = tid; f < mine + 1; f += nt) odd_face[f] = 0;
            __syncthreads();
            // edges of zones -1 .. mine
            for (int it = tid; it < NQ * (mine + 2); it += nt) {
                const int q = it / (mine + 2), z = it - q * (mine + 2);
                bool ok = true;
                double l, h;
                zone_edges<LAW_HYDRO, RECON>(C, Ps + q * W + S + z - 1, 1, q, l, h, ok);
                E[q * (m + 2) + z] = l;
                E[(NQ + q) * (m + 2) + z] = h;
                if (!ok) odd_zone[z] = 1;
            }
            __syncthreads();
            // the states of both sides of every face; at a step's start, on
            // warps of their own, the zones' conserved densities and largest
            // eigenvalues
            const int sides = 2 * (mine + 1), warped = (sides + 31) / 32 * 32, zoned = (mine + 31) / 32 * 32;
            u64 v = 0;
            for (int it = tid; it < warped + (rk == 0 ? 2 * zoned : 0); it += nt) {
                if (it < sides) {
                    const int s = it > mine ? 1 : 0, f = it - s * (mine + 1);
                    double P[NQ];
#pragma unroll
                    for (int q = 0; q < NQ; ++q) P[q] = E[((1 - s) * NQ + q) * (m + 2) + f + s];
                    fast64::Side<NQ> T;
                    bool ok = C.ok && !odd_zone[f + s];
                    fast64::hydro_side<0>(C, P, T, ok);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        sU[(s * NQ + q) * (m + 1) + f] = T.U[q];
                        sF[(s * NQ + q) * (m + 1) + f] = T.F[q];
                    }
                    sA[(2 * s) * (m + 1) + f] = T.ap;
                    sA[(2 * s + 1) * (m + 1) + f] = T.am;
                    if (!ok) odd_face[f] = 1;
                } else if (it >= warped) {
                    const bool speeds = it >= warped + zoned;
                    const int z = it - warped - (speeds ? zoned : 0);
                    if (z >= mine) continue;
                    double P[NQ];
                    bool ok = C.ok;
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        P[q] = Ps[q * W + S + z];
                        ok = ok && fast64::ordinary_field(q, P[q]);
                    }
                    if (speeds) {
                        const u64 l = fastest(P);
                        v = l > v ? l : v;
                    } else {
                        double D[NQ];
                        fast64::p2u<LAW_HYDRO>(C, P, D, ok);
                        if (!ok) law_p2u<LAW_HYDRO>(pp, P, D);
#pragma unroll
                        for (int q = 0; q < NQ; ++q) U0[q * m + z] = U[q * m + z] = D[q];
                    }
                }
            }
            if (rk == 0) {
                reduce(v, step & 1);
                cluster.barrier_arrive();   // its wait: where dt is needed
            }
            __syncthreads();
            if constexpr (RIEMANN == RIEMANN_HLLE) {
                for (int it = tid; it < NQ * (mine + 1); it += nt) {
                    const int q = it / (mine + 1), f = it - q * (mine + 1);
                    bool ok = true;
                    const double* a = sA + f;
                    const double h = fast64::hlle(a[0], a[2 * (m + 1)], a[m + 1], a[3 * (m + 1)],
                                                  sF[q * (m + 1) + f], sF[(NQ + q) * (m + 1) + f],
                                                  sU[q * (m + 1) + f], sU[(NQ + q) * (m + 1) + f], ok);
                    Fx[q * (m + 1) + f] = h;
                    if (!ok) odd_face[f] = 1;
                }
                __syncthreads();
            }
            for (int f = tid; f < mine + 1; f += nt) {
                bool ok = !odd_face[f];
                if constexpr (RIEMANN == RIEMANN_HLLC) {
                    double Pl[NQ], Pr[NQ], h[NQ];
                    fast64::Side<NQ> L, R;
#pragma unroll
                    for (int q = 0; q < NQ; ++q) {
                        Pl[q] = E[(NQ + q) * (m + 2) + f];
                        Pr[q] = E[q * (m + 2) + f + 1];
                        L.U[q] = sU[q * (m + 1) + f];
                        R.U[q] = sU[(NQ + q) * (m + 1) + f];
                        L.F[q] = sF[q * (m + 1) + f];
                        R.F[q] = sF[(NQ + q) * (m + 1) + f];
                    }
                    L.ap = sA[f];
                    L.am = sA[(m + 1) + f];
                    R.ap = sA[2 * (m + 1) + f];
                    R.am = sA[3 * (m + 1) + f];
                    L.vn = fast64::along<0>(C, Pl[1], Pl[2], Pl[3]);
                    R.vn = fast64::along<0>(C, Pr[1], Pr[2], Pr[3]);
                    fast64::hllc<0>(C, Pl, Pr, L, R, h, ok);
#pragma unroll
                    for (int q = 0; q < NQ; ++q) Fx[q * (m + 1) + f] = h[q];
                }
                if (!ok)
                    face_general<LAW_HYDRO, RECON, RIEMANN>(Ps + S + f, W, 1, G.nrm[0][0], G.nrm[0][1], G.nrm[0][2], &pp,
                                                            Fx + f, m + 1);
            }
            if (rk == 0) {
                cluster.barrier_wait();
                u64 l = 0;
                for (int k = 0; k < nc; ++k) {
                    const u64 o = cluster.map_shared_rank(red, k)[step & 1];
                    l = o > l ? o : l;
                }
                const double courant = G.lmin / __longlong_as_double((long long) l);
                bits = (u64) __double_as_longlong(courant < DBL_MAX ? courant : DBL_MAX);
                const double c = cfl * __longlong_as_double((long long) bits);
                if (t_final >= 0.0) {
                    if (!(t < t_final)) { done = true; break; }
                    const double rest = t_final - t;
                    dt = c < rest ? c : rest;
                } else {
                    dt = c;
                }
            }
            __syncthreads();
            for (int it = tid; it < NQ * mine; it += nt) {
                const int q = it / mine, z = it - q * mine;
                const double sum = fast64::add_zero(fast64::mul_any(Fx[q * (m + 1) + z + 1], G.dA[0]) -
                                                    fast64::mul_any(Fx[q * (m + 1) + z], G.dA[0]), false);
                U[q * m + z] = rk_combine_plain(U0[q * m + z], U[q * m + z], fast64::mul_any(fv, sum), dt, w);
            }
            __syncthreads();
            for (int z = tid; z < mine; z += nt) {
                double D[NQ], P[NQ];
                bool ok = C.ok;
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    D[q] = U[q * m + z];
                    ok = ok && fast64::ordinary_field(q, D[q]);
                }
                fast64::cons<LAW_HYDRO>(C, D, P, ok);
                if (!ok) {
                    int code = 0;
                    law_cons<LAW_HYDRO>(pp, D, P, &code);
                }
#pragma unroll
                for (int q = 0; q < NQ; ++q) Pn[q * W + S + z] = P[q];
            }
        }
        if (done) break;
        t += dt;
    }
    cluster.sync();   // no CTA leaves while another reads its halo or slot
    if (step > 0) {
        const double* Ps = Pbuf + par * NQ * W;
        double* out = (step * order) & 1 ? Pb : Pa;
        for (int it = tid; it < NQ * mine; it += nt) {
            const int q = it / mine, z = it - q * mine;
            const double v = Ps[q * W + S + z];
            for (int a = 0; a <= G.g[0]; ++a) {
                int ox, sx;
                if (!guard_image(a, z0 + z, n, G.g[0], G.bc, ox, sx)) continue;
                out[q * G.sP + ox] = q == 1 && sx ? v * -1 : v;
            }
        }
    }
    if (r == 0 && tid == 0) {
        st->t = t;
        st->dt = dt;
        st->dt_bits = bits;
        st->steps += step;
        st->taken += step;
        if (done) st->done = 1;
    }
}

// Zones.  A chosen limit, not the shared memory's (16 CTAs hold about 7500) nor
// where the step kernels catch up: a step on the cluster at 4096 zones and by
// step kernels at 4097 takes 35.6 and 37.4 us (PLM, HLLE, RK2), 36.1 and 39.4
// (PLM, HLLC, RK2), but 115 and 83 (WENO5, HLLC, RK3).
constexpr int PLAIN_CLUSTER_MAX = 4096;

template <int RECON, int RIEMANN>
static cudaError_t plain_cluster_config(int n, int ctas, cudaStream_t s, cudaLaunchAttribute* at, cudaLaunchConfig_t& lc)
{
    const int m = (n + ctas - 1) / ctas;
    const size_t smem = sizeof(double) * plain_cluster_doubles(m, ReconInfo<RECON>::S);
    auto k = plain_cluster_kernel<RECON, RIEMANN>;
    const cudaError_t e = allow_cluster(k, smem, ctas > 8);
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned) ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc = {};
    lc.gridDim = dim3((unsigned) ctas);
    const int want = (5 * (m + 2) + 31) / 32 * 32;
    lc.blockDim = dim3((unsigned) (want < 128 ? 128 : want > 512 ? 512 : want));
    lc.dynamicSmemBytes = smem;
    lc.stream = s;
    lc.attrs = at;
    lc.numAttrs = 1;
    return e;
}

// CTAs of the cluster that holds a grid of n zones (0: it does not fit here):
// at least 32 zones a CTA, and 16 CTAs where the GPU can place them
template <int RECON, int RIEMANN>
static int plain_cluster_ctas_r(int n)
{
    for (int cap = 16; cap >= 8; cap /= 2) {
        const int c = n / 32 < 1 ? 1 : n / 32 > cap ? cap : n / 32;
        cudaLaunchAttribute at[1];
        cudaLaunchConfig_t lc;
        int count = 0;
        if (plain_cluster_config<RECON, RIEMANN>(n, c, nullptr, at, lc) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&count, plain_cluster_kernel<RECON, RIEMANN>, &lc) == cudaSuccess && count > 0)
            return c;
        cudaGetLastError();
    }
    return 0;
}

template <int RECON, int RIEMANN>
static int plain_cluster_steps_r(int ctas, const GridDesc& G, const PhysParamsH& ph, double* Pcur, double* Pother,
                                 double cfl, double t_final, int order, int nsteps, DevStatus* st, cudaStream_t s)
{
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t lc;
    if (plain_cluster_config<RECON, RIEMANN>(G.n[0], ctas, s, at, lc) != cudaSuccess) return MARA_ERR_CUDA;
    const double factor = -1.0;
    const cudaError_t e = cudaLaunchKernelEx(&lc, plain_cluster_kernel<RECON, RIEMANN>, Pcur, Pother, G, to_dev(ph),
                                             to_fast(ph, G), factor / G.dV, cfl, t_final, order, nsteps, st);
    return e == cudaSuccess ? MARA_OK : MARA_ERR_CUDA;
}

} // namespace mara

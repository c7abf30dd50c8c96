// plain_fp64.cu -- the plain FP64 path's entry points by law (the kernels:
// plain_kernels.cuh) and the uniform-gravity source terms.
#include "plain_kernels.cuh"

namespace mara {

MARA_PLAIN_LAW(extern, LAW_HYDRO);
MARA_PLAIN_LAW(extern, LAW_MHD);
MARA_PLAIN_LAW(extern, LAW_MHD_COOL);
MARA_PLAIN_LAW(extern, LAW_RMHD);

int plain_flux_launches(int law, int recon, int riemann, const GridDesc& G)
{
    int axes = 0;
    for (int a = 0; a < 3; ++a) axes += G.n[a] > 1;
    return in_face_runs(law, recon, riemann, G) || (riemann == RIEMANN_HLLC && law != LAW_HYDRO) ? axes : 1;
}

void plain_flux(int launch, int law, int recon, int riemann, const GridDesc& G, const PhysParamsH& ph,
                const double* P, double* const* F, DevStatus* st, cudaStream_t s)
{
    switch (law) {
        case LAW_HYDRO: plain_flux_law<LAW_HYDRO>(launch, recon, riemann, G, ph, P, F, st, s); break;
        case LAW_MHD: plain_flux_law<LAW_MHD>(launch, recon, riemann, G, ph, P, F, st, s); break;
        case LAW_MHD_COOL: plain_flux_law<LAW_MHD_COOL>(launch, recon, riemann, G, ph, P, F, st, s); break;
        default: plain_flux_law<LAW_RMHD>(launch, recon, riemann, G, ph, P, F, st, s); break;
    }
}

void plain_update(int law, const GridDesc& G, const PhysParamsH& ph, const double* Pin, double* Pout,
                  double* U0, double* U, const double* Fx, const double* Fy, const double* Fz,
                  int order, int stage, const double* dt, DevStatus* st, cudaStream_t s, const double* S)
{
    switch (law) {
        case LAW_HYDRO: plain_update_law<LAW_HYDRO>(G, ph, Pin, Pout, U0, U, Fx, Fy, Fz, order, stage, dt, st, s, S); break;
        case LAW_MHD: plain_update_law<LAW_MHD>(G, ph, Pin, Pout, U0, U, Fx, Fy, Fz, order, stage, dt, st, s, S); break;
        case LAW_MHD_COOL: plain_update_law<LAW_MHD_COOL>(G, ph, Pin, Pout, U0, U, Fx, Fy, Fz, order, stage, dt, st, s, S); break;
        default: plain_update_law<LAW_RMHD>(G, ph, Pin, Pout, U0, U, Fx, Fy, Fz, order, stage, dt, st, s, S); break;
    }
}

void plain_courant(int law, const GridDesc& G, const PhysParamsH& ph, const double* P, DevStatus* st, cudaStream_t s)
{
    switch (law) {
        case LAW_HYDRO: plain_courant_law<LAW_HYDRO>(G, ph, P, st, s); break;
        case LAW_MHD: plain_courant_law<LAW_MHD>(G, ph, P, st, s); break;
        case LAW_MHD_COOL: plain_courant_law<LAW_MHD_COOL>(G, ph, P, st, s); break;
        default: plain_courant_law<LAW_RMHD>(G, ph, P, st, s); break;
    }
}

} // namespace mara

// ---------------------------------------------------------------------------
// The ready-made uniform-gravity source terms function (include/mara_gpu.h).
__global__ void k_uniform_gravity(const double* __restrict__ P, double* __restrict__ S, long long sP, long long cells,
                                  int nq, double g1, double g2, double g3)
{
    const long long c = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    if (c >= cells) return;
    const double rho = P[c], v1 = P[sP + c], v2 = P[2 * sP + c], v3 = P[3 * sP + c];
    S[c] = 0.0;
    S[sP + c] = rho * g1;
    S[2 * sP + c] = rho * g2;
    S[3 * sP + c] = rho * g3;
    S[4 * sP + c] = rho * (v1 * g1 + v2 * g2 + v3 * g3);
    for (int q = 5; q < nq; ++q) S[q * sP + c] = 0.0;
}

extern "C" int mara_source_uniform_gravity(void* user, const MaraSourceTermsArgs* a)
{
    if (!user || !a) return MARA_ERR_ARGUMENT;
    const double* g = (const double*) user;
    const long long cells = (long long) a->N[0] * a->N[1] * a->N[2];
    k_uniform_gravity<<<(unsigned) ((cells + 255) / 256), 256, 0, (cudaStream_t) a->stream>>>(
        a->P, a->S, a->sP, cells, a->nq, g[0], g[1], g[2]);
    return cudaGetLastError() == cudaSuccess ? MARA_OK : MARA_ERR_CUDA;
}

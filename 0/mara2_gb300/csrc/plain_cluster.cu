// plain_cluster.cu -- the cluster form of the plain path's 1-D hydro loop.
#include "plain_cluster.cuh"

namespace mara {

#define MARA_PLAIN_CLUSTER(CALL)                                                                                    \
    if (riemann == RIEMANN_HLLC) {                                                                                   \
        switch (recon) {                                                                                             \
            case RECON_PCM: return CALL<RECON_PCM, RIEMANN_HLLC> ARGS;                                                \
            case RECON_PLM: return CALL<RECON_PLM, RIEMANN_HLLC> ARGS;                                                \
            default: return CALL<RECON_WENO5, RIEMANN_HLLC> ARGS;                                                     \
        }                                                                                                            \
    }                                                                                                                \
    switch (recon) {                                                                                                 \
        case RECON_PCM: return CALL<RECON_PCM, RIEMANN_HLLE> ARGS;                                                    \
        case RECON_PLM: return CALL<RECON_PLM, RIEMANN_HLLE> ARGS;                                                    \
        default: return CALL<RECON_WENO5, RIEMANN_HLLE> ARGS;                                                         \
    }

int plain_cluster_ctas(int law, int recon, int riemann, const GridDesc& G)
{
    if (law != LAW_HYDRO || G.n[0] < 2 || G.n[1] > 1 || G.n[2] > 1 || G.n[0] > PLAIN_CLUSTER_MAX) return 0;
#define ARGS (G.n[0])
    MARA_PLAIN_CLUSTER(plain_cluster_ctas_r)
#undef ARGS
}

int plain_cluster_steps(int ctas, int recon, int riemann, const GridDesc& G, const PhysParamsH& ph, double* Pcur,
                        double* Pother, double cfl, double t_final, int order, int nsteps, DevStatus* st, cudaStream_t s)
{
#define ARGS (ctas, G, ph, Pcur, Pother, cfl, t_final, order, nsteps, st, s)
    MARA_PLAIN_CLUSTER(plain_cluster_steps_r)
#undef ARGS
}

} // namespace mara

// Fehlberg 7(8) FP64 team sweeps of the one-thread models (va_team64.cuh).
// Built with -fmad=false, like va_inst_small_fp64.cu.
#include "va_models.cuh"
#include "va_registry.h"
#include "va_team64.cuh"

namespace va {

template <class M, int G>
static TeamKernels team()
{
    return {G, (const void *)forward_team_kernel<M, TabRKF78, G>, (const void *)backward_team_kernel<M, TabRKF78, G>,
            (const void *)backward_team_kernel_2level<M, TabRKF78, G>};
}

template <class M>
static void fill(Fp64Kernels &k)
{
    k.team[2][0] = team<M, 32>();
    k.team[2][1] = team<M, 16>();
    k.team[2][2] = team<M, 8>();
}

void fill_team_rkf78_vdp(Fp64Kernels &k) { fill<ModelVdP>(k); }
void fill_team_rkf78_vdp_petsc(Fp64Kernels &k) { fill<ModelVdPPetsc>(k); }
void fill_team_rkf78_dho(Fp64Kernels &k) { fill<ModelDHO>(k); }
void fill_team_rkf78_decay(Fp64Kernels &k) { fill<ModelDecay>(k); }

} // namespace va

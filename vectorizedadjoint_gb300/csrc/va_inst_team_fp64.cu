// FP64 team sweeps of the one-thread models (small batches, va_team64.cuh).
// Built with -fmad=false, like va_inst_small_fp64.cu, so they reproduce the
// oracle bit for bit.
#include "va_models.cuh"
#include "va_registry.h"
#include "va_team64.cuh"

namespace va {

template <class M, class Tab, int G>
static TeamKernels team()
{
    return {G, (const void *)forward_team_kernel<M, Tab, G>, (const void *)backward_team_kernel<M, Tab, G>,
            (const void *)backward_team_kernel_2level<M, Tab, G>};
}

template <class M>
static void fill(Fp64Kernels &k)
{
    k.team[0][0] = team<M, TabDopri5, 16>();
    k.team[0][1] = team<M, TabDopri5, 8>();
    k.team[0][2] = team<M, TabDopri5, 4>();
    k.team[0][3] = team<M, TabDopri5, 2>();
    k.team[1][0] = team<M, TabCK54, 16>();
    k.team[1][1] = team<M, TabCK54, 8>();
    k.team[1][2] = team<M, TabCK54, 4>();
    k.team[1][3] = team<M, TabCK54, 2>();
}

void fill_team_vdp(Fp64Kernels &k) { fill<ModelVdP>(k); }
void fill_team_vdp_petsc(Fp64Kernels &k) { fill<ModelVdPPetsc>(k); }
void fill_team_dho(Fp64Kernels &k) { fill<ModelDHO>(k); }
void fill_team_decay(Fp64Kernels &k) { fill<ModelDecay>(k); }

} // namespace va

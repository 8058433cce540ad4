// FP64 sweeps of the one-thread models with their products on the integer
// pipe (va_step64.cuh).  Built with -fmad=false, like va_inst_small_fp64.cu,
// so they reproduce the oracle bit for bit.
#include "../../include/va.h"
#include "va_kernels.cuh"
#include "va_models.cuh"
#include "va_registry.h"

namespace va {

template <class M>
static Fp64Kernels make(void (*team)(Fp64Kernels &), void (*rkf78)(Fp64Kernels &))
{
    Fp64Kernels k{};
    k.int_fwd[0] = (const void *)forward_kernel<M, TabDopri5, double, true>;
    k.int_fwd[1] = (const void *)forward_kernel<M, TabCK54, double, true>;
    k.int_bwd[0] = (const void *)backward_kernel<M, TabDopri5, double, true>;
    k.int_bwd[1] = (const void *)backward_kernel<M, TabCK54, double, true>;
    team(k);
    rkf78(k);
    return k;
}

const Fp64Kernels *fp64_kernels(int model, int n)
{
    static const Fp64Kernels vdp = make<ModelVdP>(fill_team_vdp, fill_team_rkf78_vdp),
                             petsc = make<ModelVdPPetsc>(fill_team_vdp_petsc, fill_team_rkf78_vdp_petsc),
                             dho = make<ModelDHO>(fill_team_dho, fill_team_rkf78_dho),
                             decay = make<ModelDecay>(fill_team_decay, fill_team_rkf78_decay);
    return model == VA_MODEL_VDP ? &vdp
         : model == VA_MODEL_VDP_PETSC ? &petsc
         : model == VA_MODEL_DHO ? &dho
         : model == VA_MODEL_DECAY ? &decay
         : model == VA_MODEL_GLV ? fp64_kernels_glv(n) : nullptr;
}

} // namespace va

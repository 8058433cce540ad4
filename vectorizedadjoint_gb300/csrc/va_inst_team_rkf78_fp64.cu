// Fehlberg 7(8) FP64 team sweeps of the one-thread models (va_team64.cuh).
// Built with -fmad=false, like va_inst_small_fp64.cu.
#include "va_models.cuh"
#include "va_registry.h"
#include "va_team64.cuh"

namespace va {

// Limits as in va_inst_team_fp64.cu.  Van der Pol, tol 1e-9, T = 10 (load =
// 0.6 B), 32 / 16 / 8 lanes, one lane with FP64 products; forward, then backward:
//     B = 600    1.18 / 1.51 / 1.79   3.52    0.70 / 1.01 / 1.48   5.86
//     B = 2,400  2.97 / 2.27 / 1.78   3.66    1.50 / 1.58 / 1.48   6.00
//     B = 5,003  4.61 / 3.77 / 2.73   3.72    1.98 / 1.76 / 2.51   6.10
//     B = 9,600  6.84 / 4.39 / 3.54   3.70    3.78 / 3.29 / 3.03   6.10
//     B = 19,000 13.3 / 8.27 / 5.44   3.72    7.36 / 6.68 / 6.23   6.13
// Two-level backward, stride 16 (32 / 16 lanes, one lane): 200: 1.1 / 1.4, 17.4;
// 5,000: 5.4 / 4.3, 16.6; 20,000: 20.7 / 18.8, 27.2; 60,000: 62 / 57, 36.
template <class M>
static void fill(Fp64Kernels &k)
{
    auto &t = k.team[2];
    t[FP64_FORWARD][0] = {(const void *)forward_team_kernel<M, TabRKF78, 32>, 32, 2, 0.7f};
    t[FP64_FORWARD][1] = {(const void *)forward_team_kernel<M, TabRKF78, 16>, 16, 2, 1.4f};
    t[FP64_FORWARD][2] = {(const void *)forward_team_kernel<M, TabRKF78, 8>, 8, 2, 9.5f};
    t[FP64_BACKWARD][0] = {(const void *)backward_team_kernel<M, TabRKF78, 32>, 32, 2, 1.2f};
    t[FP64_BACKWARD][1] = {(const void *)backward_team_kernel<M, TabRKF78, 16>, 16, 2, 7.0f};
    t[FP64_BACKWARD][2] = {(const void *)backward_team_kernel<M, TabRKF78, 8>, 8, 2, 18.0f};
    t[FP64_TWO_LEVEL][0] = {(const void *)backward_team_kernel_2level<M, TabRKF78, 32>, 32, 0, 0.5f};
    t[FP64_TWO_LEVEL][1] = {(const void *)backward_team_kernel_2level<M, TabRKF78, 16>, 16, 0, 35.0f};
}

void fill_team_rkf78_vdp(Fp64Kernels &k) { fill<ModelVdP>(k); }
void fill_team_rkf78_vdp_petsc(Fp64Kernels &k) { fill<ModelVdPPetsc>(k); }
void fill_team_rkf78_dho(Fp64Kernels &k) { fill<ModelDHO>(k); }
void fill_team_rkf78_decay(Fp64Kernels &k) { fill<ModelDecay>(k); }

} // namespace va

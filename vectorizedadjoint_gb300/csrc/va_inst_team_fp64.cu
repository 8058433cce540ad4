// FP64 team sweeps of the one-thread models (small batches, va_team64.cuh).
// Built with -fmad=false, like va_inst_small_fp64.cu, so they reproduce the
// oracle bit for bit.
#include "va_models.cuh"
#include "va_registry.h"
#include "va_team64.cuh"

namespace va {

// Limits: where the next narrower team, or one lane with integer products, is
// measured faster (forward + backward, ms; load = 0.55 B for Van der Pol T = 20,
// 0.11 B for the oscillators with horizons to 50).
//     Van der Pol, 16 / 8 / 4 / 2 lanes, one lane:
//     B = 1,216   1.96 / 2.72 / 3.51 / 4.67   4.60
//     B = 2,400   2.79 / 2.72 / 3.50 / 4.68   4.83
//     B = 4,800   5.25 / 3.95 / 3.51 / 4.69   4.85
//     B = 9,600   7.44 / 7.67 / 5.47 / 4.66   5.18
//     B = 19,000  13.3 / 10.8 / 10.2 / 7.70   5.20
//     oscillators (teams of 16 in two blocks per SM, the others in one):
//     B = 5,000   10.5 / 12.1 / 15.0 / 19.5   25.0
//     B = 19,000  12.8 / 13.7 / 15.7 / 21.0   25.6
// The oscillators gain from wide teams at loads where Van der Pol no longer
// does (their steps are cheaper beside the fixed part of an attempt); the
// limits lie between the two.
// Two seed rows in the halves of a warp, backward alone (two seeds; 32 lanes for
// both, then the teams above one seed after the other), by load per quadrant:
//     Van der Pol  0.54: 0.55, 1.27; 2.2: 0.97, 1.92; 5.4: 2.16, 3.68; 8.2: 3.34, 4.99; 12.7: 4.8, 4.7; 18: 7.2, 5.0
//     oscillators  0.02: 2.20, 4.98; 0.8: 3.16, 7.15; 3.9: 8.4, 10.8
// With one seed row the second half repeats it, and the recompute of 32 steps
// instead of 16 still pays while the warps have the quadrants to themselves:
// Van der Pol 0.54: 0.55, 0.63; 1.08: 0.77, 0.64; oscillators 0.02: 2.20, 2.49.
// Two-level backward alone, Van der Pol, stride 16 (32 / 16 / 8 lanes, one
// lane): 200: 0.73 / 1.11, 11.2; 1,200: 1.16 / 1.21, 11.3; 9,001: 5.97 / 4.69 /
// 5.34, 11.0; 30,000: 16.2 (16 lanes), 22.3; 100,000: 63.6 / 54.9, 37.4.  Longer
// segments are fewer to share out, and launch_teams lowers the limits for them
// (stride 50, ~250 steps: 9,001 instances 7.7 with 16 lanes, 7.3 with one).
template <class M, class Tab>
static void fill(TeamKernel (&t)[kFp64Sweeps][kTeams], float &seeds_per_quad)
{
    t[FP64_FORWARD][0] = {(const void *)forward_team_kernel<M, Tab, 16>, 16, 2, 4.0f};
    t[FP64_FORWARD][1] = {(const void *)forward_team_kernel<M, Tab, 4>, 4, 1, 6.6f};
    t[FP64_FORWARD][2] = {(const void *)forward_team_kernel<M, Tab, 2>, 2, 1, 13.0f};
    t[FP64_BACKWARD][0] = {(const void *)backward_team_kernel<M, Tab, 32, 2>, 32, 2, 0.8f};
    t[FP64_BACKWARD][1] = {(const void *)backward_team_kernel<M, Tab, 16>, 16, 2, 4.0f};
    t[FP64_BACKWARD][2] = {(const void *)backward_team_kernel<M, Tab, 4>, 4, 1, 6.6f};
    t[FP64_BACKWARD][3] = {(const void *)backward_team_kernel<M, Tab, 2>, 2, 1, 13.0f};
    seeds_per_quad = 13.0f;
    t[FP64_TWO_LEVEL][0] = {(const void *)backward_team_kernel_2level<M, Tab, 32>, 32, 0, 0.75f};
    t[FP64_TWO_LEVEL][1] = {(const void *)backward_team_kernel_2level<M, Tab, 16>, 16, 0, 50.0f};
}
template <class M>
static void fill_model(Fp64Kernels &k)
{
    fill<M, TabDopri5>(k.team[0], k.seeds_per_quad[0]);
    fill<M, TabCK54>(k.team[1], k.seeds_per_quad[1]);
}

void fill_team_vdp(Fp64Kernels &k) { fill_model<ModelVdP>(k); }
void fill_team_vdp_petsc(Fp64Kernels &k) { fill_model<ModelVdPPetsc>(k); }
void fill_team_dho(Fp64Kernels &k) { fill_model<ModelDHO>(k); }
void fill_team_decay(Fp64Kernels &k) { fill_model<ModelDecay>(k); }

} // namespace va

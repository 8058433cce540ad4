// FP64 sweeps of the per-instance GLV model, built with -fmad=false so that
// they reproduce the CPU oracle bit for bit (see va_inst_small_fp64.cu).
#include "va_group.cuh"
#include "va_registry.h"
#include "va_team_glv64.cuh"

namespace va {

template <int NN>
static void fill(KernelSet &k)
{
    using M = ModelGLVLane<NN>;
    k.fwd[0][0] = (const void *)forward_group_kernel<M, TabDopri5, double>;
    k.fwd[1][0] = (const void *)forward_group_kernel<M, TabCK54, double>;
    k.bwd[0][0] = (const void *)backward_group_kernel<M, TabDopri5, double>;
    k.bwd[1][0] = (const void *)backward_group_kernel<M, TabCK54, double>;
}

// With the products on the integer pipe (va_step64.cuh).  Forward, 16,384
// instances: N = 10 3.96 -> 2.85 ms, N = 5 1.70 -> 1.21; 777 instances: N = 10
// 0.88 -> 0.71, N = 5 the same.  Backward, 16,384 instances: N = 5 3.16 -> 2.52;
// N = 10 needs more registers than there are (9.1 -> 9.3), and with few warps
// the longer code loses for both (777 instances, N = 5: 1.04 -> 1.41).
// (one instance, N = 10: 0.48 -> 0.51 forward.)
constexpr float kTwoWarps5 = 2 * 6; // groups of 5 that fill two warps
template <int NN>
static Fp64Kernels make_int()
{
    using M = ModelGLVLane<NN>;
    Fp64Kernels k{};
    k.int_fwd[0] = (const void *)forward_group_kernel<M, TabDopri5, double, true>;
    k.int_fwd[1] = (const void *)forward_group_kernel<M, TabCK54, double, true>;
    if constexpr (NN == 5) {
        k.int_bwd[0] = (const void *)backward_group_kernel<M, TabDopri5, double, true>;
        k.int_bwd[1] = (const void *)backward_group_kernel<M, TabCK54, double, true>;
    }
    k.int_fwd_min = NN == 5 ? kTwoWarps5 : 0.05f;
    k.int_bwd_min = kTwoWarps5;
    // A warp per instance (va_team_glv64.cuh); limits where the lane groups are
    // faster, ms (load ~0.8 B):
    //     N = 5    forward: 100: 0.32, groups 0.61; 777: 0.48, 0.59; 3,000: 1.15, 0.62
    //              backward: 0.25, 0.89; 0.38, 0.86; 0.97, 0.91
    //     N = 10   forward: 0.51, 0.72; 0.79, 0.71; 2.08, 0.79
    //              backward: 0.54, 1.53; 0.85, 1.51; 2.36, 1.88
    const float fq = NN == 5 ? 1.5f : 0.95f, bq = NN == 5 ? 3.8f : 2.8f;
    k.team[0][FP64_FORWARD][0] = {(const void *)forward_glv_warp_kernel<NN, TabDopri5>, 32, 2, fq};
    k.team[1][FP64_FORWARD][0] = {(const void *)forward_glv_warp_kernel<NN, TabCK54>, 32, 2, fq};
    k.team[0][FP64_BACKWARD][0] = {(const void *)backward_glv_warp_kernel<NN, TabDopri5>, 32, 2, bq};
    k.team[1][FP64_BACKWARD][0] = {(const void *)backward_glv_warp_kernel<NN, TabCK54>, 32, 2, bq};
    return k;
}
const Fp64Kernels *fp64_kernels_glv(int n)
{
    static const Fp64Kernels k5 = make_int<5>(), k10 = make_int<10>();
    return n == 5 ? &k5 : n == 10 ? &k10 : nullptr;
}

void fill_fp64_glv5(KernelSet &k) { fill<5>(k); }
void fill_fp64_glv10(KernelSet &k) { fill<10>(k); }

} // namespace va

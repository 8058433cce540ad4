// Longest-first work order for the persistent sweeps (va_order.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace va {

// Batches up to this size are sorted in one block, without a split.
constexpr int kSmallBatch = 4096;

struct OrderArgs {
    int B;
    const int *steps;  // backward: accepted steps per instance (or null)
    const double *t0;  // forward: horizons t1 - t0 (used when steps is null and
    const double *t1;  //   no previous sweep's counts are valid)
    int *prev_work;        // forward: attempts per instance of the previous forward sweep,
                           //   taken from here (0 afterwards)
    const int *prev_valid; //   and its flag (device int, 1 once written); may be null
    int *work;         // order_work_ints(B) ints, kept between calls
    int *order;        // [B] output permutation, longest first
    const int *reuse;  // backward: the forward's order, copied instead of sorting when
                       //   that order came from counts (flag in work) and they were
                       //   this batch's; may be null
    const int *now;    // with reuse: attempts per instance of that forward sweep
    float keep_from;   //   and the load above which its order stays in any case
    // When the batch may be split (order_split): above this load and up to
    // that one (0: never), and the most load that goes into the longest part
    float split_from, split_to, split_load;
};

#ifdef __CUDACC__
// Whether an instance did not have the length that the order took it for.
__device__ __forceinline__ bool length_moved(int before, int now)
{
    return (now < before ? before - now : now - before) > before / 8 + 2;
}
#endif

size_t order_work_ints(int B);
// In `work`, on the device: the batch's load, the sum of its instances'
// lengths in units of the longest, set with the order (see va_order.cu).
const float *order_load(const int *work);
// The number of longest instances that a sweep of their own should take.
const int *order_split(const int *work);
cudaError_t enqueue_order(const OrderArgs &a, cudaStream_t s);

} // namespace va

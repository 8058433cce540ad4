// Longest-first work order for the persistent sweeps.  A lane that takes a
// long instance late holds the whole kernel open (the tail); handing out the
// longest instances first removes most of it.  The backward sweep orders by
// the accepted-step count the forward produced.  The forward sweep orders by
// the attempt count of the handle's previous forward sweep when there is one
// (repeated solves of a batch -- optimisation loops, sensitivity sweeps --
// change step counts little between calls), else by the horizon t1 - t0.
// Only the order comes from the previous sweep: every step is computed
// again, and each instance's result does not depend on the order.  On a
// batch with one horizon (every instance to the same T) the horizon order
// is the index order, and lanes whose last instances run long idle the rest
// of their warp.  A counting sort over 4096
// buckets (descending) builds the permutation on the device, so it can sit
// inside the captured graph.  The atomics here only decide the order; each
// instance's result does not depend on it.  The backward can take the
// forward's order when that one came from step counts (the previous sweep's
// attempts, nearly the same ranking as this sweep's accepted steps): no
// second sort, and the backward then visits the checkpoint chunks in the
// order the forward allocated them (the caller decides; one-thread models).
// Not when the inputs are others than the call's before: when the lengths of
// more than 1 in 32 instances moved by more than an eighth, or the longest did,
// the backward sorts by its own step counts, and its load and its longest part
// are this batch's too.  Where the load fills four warps per quadrant a lane
// carries several instances, the order matters less than the chunks' locality, and
// the forward's order stays (262,144 double-word Van der Pol instances on new
// inputs: backward 3.52 ms with it, 3.64 sorted; 65,536: 1.12 with it, 0.72 sorted).
//
// The sort also leaves the batch's load, sum(length) / max(length), by which
// the one-thread sweeps choose on the device how many warps they keep busy
// (resting) and how many lanes carry an instance (gated_off): with uneven
// lengths the longest instance sets the pace, and whatever shares its SM
// quadrant only delays it.  More warps per quadrant raise the throughput
// (1.9x with four, double-word Van der Pol) but slow each of them by more.
// One warp per quadrant finishes a batch in max(1, load / lanes) times its
// longest instance; the sweeps keep ceil(load / (1.25 lanes)) warps per
// quadrant.  Measured, forward + backward: 65,536 double-word oscillators
// (lengths to 1,737, mean ~190: load 0.4 lanes) 5.15 ms with one warp, 6.44
// with four; FP64 27.0 against 32.1 with two; Van der Pol (mean 0.55 of the
// longest) 20,000 instances (0.6) 1.06 with one, 1.23 with four; 65,536 (1.9)
// 2.31 with one, 1.57 with two, 1.90 with four; 262,144 (7.4) 8.25 with one,
// 5.11 with four.
#include <cuda_runtime.h>

#include <cstdint>

#include "va_order.h"

namespace va {

namespace {

constexpr int kBuckets = 4096;

__device__ __forceinline__ int horizon_bucket(double h)
{
    // 64 buckets per octave of t1 - t0, from 2^-32 to 2^32
    if (!(h > 0.0))
        return 0;
    const double l = log2(h);
    const int k = (int)((l + 32.0) * 64.0);
    return k < 0 ? 0 : k >= kBuckets ? kBuckets - 1 : k;
}

__device__ __forceinline__ int count_bucket(int n) { return n < kBuckets ? (n < 0 ? 0 : n) : kBuckets - 1; }

// work[0 ..): the buckets' counts, then, zeroed with them, how many instances
// moved and the longest of now (order_hist)
constexpr int kMovedSlot = kBuckets, kLongestSlot = kBuckets + 1, kZeroed = kBuckets + 2;
// work[kOffsets ..): the buckets' offsets
constexpr int kOffsets = kZeroed;

// 1 when the last forward order came from step counts
constexpr int kCountedFlag = kOffsets + kBuckets;

// the load (a float)
constexpr int kLoadSlot = kCountedFlag + 1;

// the size of the longest part
constexpr int kSplitSlot = kLoadSlot + 1;

// the longest length by which the last forward order went, and all of them
// (B ints), when it came from step counts
constexpr int kTopSlot = kSplitSlot + 1, kTaken = kTopSlot + 1;

// the backward reuses the forward's order when that one was count-based and the
// counts were this batch's, all but a few
__device__ __forceinline__ bool reusing(const OrderArgs &a, int moved, int longest)
{
    return a.reuse && a.work[kCountedFlag] == 1 && moved <= a.B / 32 &&
           !length_moved(a.work[kTopSlot], count_bucket(longest));
}
__device__ __forceinline__ bool reusing(const OrderArgs &a)
{
    return reusing(a, a.work[kMovedSlot], a.work[kLongestSlot]);
}
// For the order of a forward sweep: what it takes instance b's length to be, out
// of the place where the sweep puts it when it is known.  After the last key_of.
__device__ __forceinline__ void keep_length(const OrderArgs &a, int b)
{
    if (!a.steps && a.prev_work) {
        a.work[kTaken + b] = a.prev_work[b];
        a.prev_work[b] = 0;
    }
}

__device__ __forceinline__ int key_of(const OrderArgs &a, int b)
{
    if (a.steps)
        return count_bucket(a.steps[b]);
    if (a.prev_work && *a.prev_valid)
        return count_bucket(a.prev_work[b]);
    return horizon_bucket(a.t1[b] - a.t0[b]);
}

// the length a bucket stands for (any unit)
__device__ __forceinline__ float bucket_length(bool counted, int k)
{
    return counted ? (float)k : exp2f((float)k * (1.0f / 64.0f) - 32.0f);
}

// The buckets' counts and, where the forward's order may be reused, how many
// instances moved and the longest of now: two loads an instance more, and one
// atomic a block (one a warp, 8,192 on one address for 262,144 instances, took
// 20 us; a launch of its own 4 us).
__global__ void __launch_bounds__(1024) order_hist(OrderArgs a)
{
    __shared__ int h[kBuckets], block_moved, block_top;
    const bool compare = a.reuse && a.work[kCountedFlag] == 1;
    for (int i = threadIdx.x; i < kBuckets; i += blockDim.x)
        h[i] = 0;
    if (threadIdx.x == 0)
        block_moved = block_top = 0;
    __syncthreads();
    int moved = 0, top = 0;
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < a.B; b += gridDim.x * blockDim.x) {
        atomicAdd(&h[key_of(a, b)], 1);
        if (compare) {
            const int n = a.now[b];
            moved += length_moved(a.work[kTaken + b], n) ? 1 : 0;
            top = n > top ? n : top;
        }
    }
    moved = __reduce_add_sync(0xffffffffu, moved);
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&block_moved, moved);
        atomicMax(&block_top, top);
    }
    __syncthreads();
    if (compare && threadIdx.x == 0) {
        atomicAdd(&a.work[kMovedSlot], block_moved);
        atomicMax(&a.work[kLongestSlot], block_top);
    }
    for (int i = threadIdx.x; i < kBuckets; i += blockDim.x)
        if (h[i])
            atomicAdd(&a.work[i], h[i]);
}

// Over one block of 1024 threads, thread t holding the counts v[j] of buckets
// kBuckets - 1 - (4 t + j): the number of instances in the buckets above its
// first (the exclusive scan from the top bucket down); and what the sort
// leaves for the sweeps, the load and where a forward order came from.
// Shuffles within the warps and two barriers; with a barrier for each of the
// ten scan steps and the load summed by one thread the scan took ~2 us more.
__device__ __forceinline__ int scan_from_top(const OrderArgs &a, const int (&v)[4])
{
    __shared__ int part[32];
    __shared__ float sum[32], top[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const bool prev = a.prev_work && a.prev_valid && *a.prev_valid;
    const bool counted = a.steps || prev;
    const int s = v[0] + v[1] + v[2] + v[3];
    int run = s;
    float s1 = 0.0f, m1 = 0.0f;
    if (s) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float l = v[j] ? bucket_length(counted, kBuckets - 1 - (t * 4 + j)) : 0.0f;
            s1 += l * (float)v[j];
            m1 = fmaxf(m1, l);
        }
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, run, o);
        run += lane >= o ? x : 0;
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    }
    if (lane == 31) {
        part[warp] = run;
        sum[warp] = s1;
        top[warp] = m1;
    }
    __syncthreads();
    if (warp == 0) {
        const int own = part[lane];
        int x = own;
        s1 = sum[lane];
        m1 = top[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            x += lane >= o ? y : 0;
            s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
        }
        part[lane] = x - own;
        if (t == 0) {
            // at most one per instance, at least one instance's (a batch of length 0 too)
            const float load = m1 > 0.0f ? s1 / m1 : 1.0f;
            a.work[kLoadSlot] = __float_as_int(fminf(fmaxf(load, 1.0f), (float)a.B));
            if (!a.steps) { // a forward order: say whether it came from counts
                a.work[kCountedFlag] = prev ? 1 : 0;
                a.work[kTopSlot] = prev ? (int)m1 : 0;
            }
        }
    }
    __syncthreads();
    return part[warp] + run - s;
}

// The longest part: the instances above a share of the longest's length, the
// smallest share whose part is no more than split_load.  0.4 is where a lane
// and a team of 16 take the same time: an attempt and its back step are 2.4
// times faster by the team (25.0 against 10.5 ms for 1,900 of them).
constexpr int kNShares = 4;
__device__ __forceinline__ float share(int i) { return i == 0 ? 0.4f : i == 1 ? 0.5f : i == 2 ? 0.6f : 0.75f; }
__device__ void find_split(const OrderArgs &a, const int (&v)[4], int above)
{
    if (!(a.split_to > 0.0f))
        return;
    __shared__ int top, count[kNShares];
    __shared__ float part[kNShares];
    const int t = threadIdx.x;
    const bool counted = a.steps || (a.prev_work && a.prev_valid && *a.prev_valid);
    const float load = __int_as_float(a.work[kLoadSlot]); // scan_from_top ends with a barrier
    if (t < kNShares) {
        count[t] = 0;
        part[t] = 0.0f;
    }
    __syncthreads();
    int run = above;
#pragma unroll
    for (int j = 0; j < 4; j++)
        if (v[j]) {
            if (run == 0)
                top = kBuckets - 1 - (t * 4 + j);
            run += v[j];
        }
    __syncthreads();
    const float most = bucket_length(counted, top);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int k = kBuckets - 1 - (t * 4 + j);
        const float l = v[j] ? bucket_length(counted, k) : 0.0f;
        for (int i = 0; i < kNShares; i++)
            if (l > share(i) * most) {
                atomicAdd(&count[i], v[j]);
                atomicAdd(&part[i], l / most * (float)v[j]);
            }
    }
    __syncthreads();
    if (t == 0) {
        int n = 0;
        if (load > a.split_from && load <= a.split_to)
            for (int i = kNShares - 1; i >= 0; i--)
                n = part[i] <= a.split_load ? count[i] : n;
        a.work[kSplitSlot] = n;
    }
}

__global__ void __launch_bounds__(1024) order_scan(OrderArgs a)
{
    if (reusing(a))
        return;
    const int t = threadIdx.x;
    int v[4];
#pragma unroll
    for (int j = 0; j < 4; j++)
        v[j] = a.work[kBuckets - 1 - (t * 4 + j)];
    const int above = scan_from_top(a, v);
    int run = above;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        a.work[kOffsets + (kBuckets - 1 - (t * 4 + j))] = run;
        run += v[j];
    }
    find_split(a, v, above);
}

// The whole sort of a small batch in one block, the buckets in shared memory
// and four keys a thread in registers: one launch where the large batch's
// memset and three kernels are four, ~2 us each.
static_assert(kSmallBatch == 4 * 1024, "four keys a thread");
__global__ void __launch_bounds__(1024) order_small(OrderArgs a)
{
    __shared__ int cnt[kBuckets], top;
    const int t = threadIdx.x;
    if (a.reuse && a.work[kCountedFlag] == 1) { // the same for every thread
        if (t == 0)
            top = 0;
        __syncthreads();
        int moved = 0;
        for (int i = 0; i < 4; i++) {
            const int b = t + 1024 * i, n = b < a.B ? a.now[b] : 0;
            moved += __syncthreads_count(b < a.B && length_moved(a.work[kTaken + b], n));
            atomicMax(&top, n);
        }
        __syncthreads();
        if (reusing(a, moved, top)) {
            for (int b = t; b < a.B; b += 1024)
                a.order[b] = a.reuse[b];
            return;
        }
    }
    int key[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        cnt[t + 1024 * i] = 0;
        key[i] = t + 1024 * i < a.B ? key_of(a, t + 1024 * i) : -1;
        if (key[i] >= 0)
            keep_length(a, t + 1024 * i);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (key[i] >= 0)
            atomicAdd(&cnt[key[i]], 1);
    __syncthreads();
    int v[4];
#pragma unroll
    for (int j = 0; j < 4; j++)
        v[j] = cnt[kBuckets - 1 - (t * 4 + j)];
    int run = scan_from_top(a, v);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        cnt[kBuckets - 1 - (t * 4 + j)] = run;
        run += v[j];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (key[i] >= 0)
            a.order[atomicAdd(&cnt[key[i]], 1)] = t + 1024 * i;
}

// Each block takes a contiguous range of instances: it counts its range per
// bucket in shared memory, reserves one slice of every bucket it touches
// with a single global atomic, then writes its instances into the slices
// (ranks from the shared-memory atomics).  One global atomic per instance
// on the few hundred buckets a batch's step counts fall into serialised on
// those counters.
__global__ void __launch_bounds__(1024) order_scatter(OrderArgs a)
{
    __shared__ int cnt[kBuckets];
    const int per = (a.B + gridDim.x - 1) / gridDim.x;
    const int lo = blockIdx.x * per, hi = min(a.B, lo + per);
    if (reusing(a) ||
        (a.reuse && a.work[kCountedFlag] == 1 && __int_as_float(a.work[kLoadSlot]) > a.keep_from)) {
        for (int b = lo + threadIdx.x; b < hi; b += blockDim.x)
            a.order[b] = a.reuse[b];
        return;
    }
    for (int i = threadIdx.x; i < kBuckets; i += blockDim.x)
        cnt[i] = 0;
    __syncthreads();
    for (int b = lo + threadIdx.x; b < hi; b += blockDim.x)
        atomicAdd(&cnt[key_of(a, b)], 1);
    __syncthreads();
    for (int i = threadIdx.x; i < kBuckets; i += blockDim.x)
        if (cnt[i])
            cnt[i] = atomicAdd(&a.work[kOffsets + i], cnt[i]); // this block's slice of bucket i
    __syncthreads();
    for (int b = lo + threadIdx.x; b < hi; b += blockDim.x) {
        a.order[atomicAdd(&cnt[key_of(a, b)], 1)] = b;
        keep_length(a, b);
    }
}

} // namespace

size_t order_work_ints(int B) { return kTaken + (size_t)B; }
const float *order_load(const int *work) { return reinterpret_cast<const float *>(work + kLoadSlot); }

const int *order_split(const int *work) { return work + kSplitSlot; }

cudaError_t enqueue_order(const OrderArgs &a, cudaStream_t s)
{
    if (a.B <= kSmallBatch) {
        order_small<<<1, 1024, 0, s>>>(a);
        return cudaGetLastError();
    }
    cudaError_t e = cudaMemsetAsync(a.work, 0, sizeof(int) * kZeroed, s);
    if (e != cudaSuccess)
        return e;
    const int grid = (a.B + 1023) / 1024 < 256 ? (a.B + 1023) / 1024 : 256;
    order_hist<<<grid, 1024, 0, s>>>(a);
    order_scan<<<1, 1024, 0, s>>>(a);
    order_scatter<<<grid, 1024, 0, s>>>(a);
    return cudaGetLastError();
}

} // namespace va

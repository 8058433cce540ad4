// Kernels of the tensor-core dA contraction (va_contract.cuh): the factor-row
// offsets of each instance, the contraction on tcgen05 with tensor-memory
// accumulators, and the fixed-order sum of the CTA partials.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/va.h"
#include "../../include/va_probe.h"
#include "va_contract.cuh"
#include "va_tcgen05.cuh"
#include "va_kernels.cuh"

namespace va {

// ------------------------------------------------------------ row offsets

// k_base[b] = nsv * sum_{b' < b, OK} T_b' (the first factor row of instance
// b), k_base[B] = K.  One block; each thread a contiguous range of instances.
__global__ void __launch_bounds__(1024) factor_offsets_kernel(const int *inst_T, const int *inst_status, int B,
                                                              int nsv, int *k_base)
{
    __shared__ long long part[1024];
    const int t = threadIdx.x, per = (B + 1023) / 1024;
    const int lo = min(B, t * per), hi = min(B, lo + per);
    long long s = 0;
    for (int b = lo; b < hi; b++)
        s += inst_status[b] == ST_OK ? (long long)inst_T[b] * nsv : 0;
    part[t] = s;
    __syncthreads();
    // inclusive scan of the 1024 partial sums (Hillis-Steele)
    for (int o = 1; o < 1024; o <<= 1) {
        const long long v = t >= o ? part[t - o] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    long long run = t > 0 ? part[t - 1] : 0;
    for (int b = lo; b < hi; b++) {
        k_base[b] = (int)run;
        run += inst_status[b] == ST_OK ? (long long)inst_T[b] * nsv : 0;
    }
    if (t == 1023)
        k_base[B] = (int)part[1023];
}

// ------------------------------------------------------------ contraction

// |hi| of a packed double-word (for the exponent bound)
__device__ __forceinline__ float dw_abs_hi(double packed) { return fabsf(dw_unpack(packed).hi); }

// exponent e with |x| < 2^e for every entry whose leading word is at most m
__device__ __forceinline__ int bound_exponent(float m) { return m > 0.0f ? ilogbf(m) + 1 : -120; }

// two digits as a bf16 pair: a digit has at most 8 significant bits, so its
// bf16 is the upper half of its float
__device__ __forceinline__ uint32_t pack_digits(float a, float b)
{
    return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}

// One column's 8 consecutive rows (a core-matrix row of 16 bytes) as Q digit
// planes: vals are packed double-words, sc the column's scale.
__device__ __forceinline__ void slice_row8(const double *vals, DigitScale sc, uint8_t *plane0, size_t plane_stride)
{
    uint32_t q[kContractQ][4];
#pragma unroll
    for (int r = 0; r < 8; r += 2) {
        const dword w0 = dw_unpack(vals[r]), w1 = dw_unpack(vals[r + 1]);
        float d0[kContractQ], d1[kContractQ];
        split_digits_in_place(w0.hi, w0.lo, sc, d0);
        split_digits_in_place(w1.hi, w1.lo, sc, d1);
#pragma unroll
        for (int s = 0; s < kContractQ; s++)
            q[s][r / 2] = pack_digits(d0[s], d1[s]);
    }
#pragma unroll
    for (int s = 0; s < kContractQ; s++)
        *reinterpret_cast<uint4 *>(plane0 + s * plane_stride) = make_uint4(q[s][0], q[s][1], q[s][2], q[s][3]);
}

// A chunk's column exponents and scales 2^(e - 8) (0 outside the fold's fast
// range; the column then takes its exponent).
struct ContractScales {
    int ev[kContractTileM], ex[kContractTileN];
    alignas(16) float pv[kContractTileM], px[kContractTileN];
};
__device__ __forceinline__ float fold_scale(int e) { return e >= -100 && e <= 100 ? pow2f(e - 8) : 0.0f; }

// Slices chunk c of the CTA's tile into one shared-memory stage and stores
// the column exponents.  A warp holds all 64 rows of its columns (8 of v, 4
// of x), so each factor is read once and a column's maximum is a few
// shuffles: no barrier between the maximum and the digits.
__device__ __forceinline__ void slice_chunk(const ContractParams &p, int c, int K, int ti, int tj, uint8_t *stage,
                                            ContractScales &sc, const double *const *xrow)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k0 = c * kContractKC;
    const bool whole = k0 + kContractKC <= K;
    // v: column i, rows 16 h .. 16 h + 15; x: column j, rows 8 q .. 8 q + 7
    const int i = warp * 8 + (lane & 7), h = lane >> 3;
    const int j = warp * 4 + (lane & 3), q = lane >> 2;
    double v[16], x[8];
    const double *col = p.v + (size_t)(k0 + 16 * h) * kContractN + ti * kContractTileM + i;
    const int xc = tj * kContractTileN + j;
    if (whole) {
#pragma unroll
        for (int r = 0; r < 16; r++)
            v[r] = __ldg(col + (size_t)r * kContractN);
#pragma unroll
        for (int r = 0; r < 8; r++)
            x[r] = __ldg(xrow[8 * q + r] + xc);
    } else {
#pragma unroll
        for (int r = 0; r < 16; r++)
            v[r] = k0 + 16 * h + r < K ? __ldg(col + (size_t)r * kContractN) : 0.0;
#pragma unroll
        for (int r = 0; r < 8; r++)
            x[r] = k0 + 8 * q + r < K ? __ldg(xrow[8 * q + r] + xc) : 0.0;
    }
    // v planes [slice][kgroup 8][row 128][8]
    {
        float m = 0.0f;
#pragma unroll
        for (int r = 0; r < 16; r++)
            m = fmaxf(m, dw_abs_hi(v[r]));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
        const int e = bound_exponent(m);
        if (h == 0) {
            sc.ev[i] = e;
            sc.pv[i] = fold_scale(e);
        }
        const DigitScale ds = digit_scale(e);
#pragma unroll
        for (int g = 0; g < 2; g++)
            slice_row8(v + 8 * g, ds, stage + (size_t)(2 * h + g) * kVGroupBytes + i * 16, 8 * kVGroupBytes);
    }
    // x planes [slice][kgroup 8][row 64][8]
    {
        float m = 0.0f;
#pragma unroll
        for (int r = 0; r < 8; r++)
            m = fmaxf(m, dw_abs_hi(x[r]));
#pragma unroll
        for (int o = 4; o < 32; o *= 2)
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const int e = bound_exponent(m);
        if (q == 0) {
            sc.ex[j] = e;
            sc.px[j] = fold_scale(e);
        }
        slice_row8(x, digit_scale(e), stage + kTileVBytes + (size_t)q * kXGroupBytes + j * 16, 8 * kXGroupBytes);
    }
}

// The x-row pointer that this thread stages of chunk c (threads 0 .. 255:
// row t & 63; null past K, never dereferenced)
__device__ __forceinline__ const double *chunk_row(const ContractParams &p, int c, int K)
{
    const int kx = c * kContractKC + (threadIdx.x & 63);
    return threadIdx.x < 256 && kx < K ? p.xp[kx] : nullptr;
}

// The x-row pointers of chunk c into xrow[64], and a prefetch of the chunk's
// rows of the CTA's tile into L2 (the factor rows are read once from DRAM;
// the slicing loads then wait on L2 instead)
__device__ __forceinline__ void prefetch_chunk(const ContractParams &p, int c, int K, int ti, int tj,
                                               const double *base, const double **xrow)
{
    const int t = threadIdx.x;
    // v: 64 rows of 128 doubles, 8 threads a row; x: 64 rows of 64, 4 threads a row
    const int kv = c * kContractKC + (t >> 3);
    if (kv < K)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p.v + (size_t)kv * kContractN + ti * kContractTileM +
                                                      (t & 7) * 16));
    if (t < 64)
        xrow[t] = base;
    if (base)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(base + tj * kContractTileN + (t >> 6) * 16));
}

// The 40 MMAs of one chunk: for every group g = s + t the digit pairs
// (s, t), each over the chunk's four K steps of 16, into accumulator g.
__device__ __forceinline__ void issue_chunk(uint32_t tmem_acc, const uint8_t *stage)
{
    constexpr uint32_t idesc = umma_idesc_bf16(kContractTileM, kContractTileN);
    const uint32_t vbase = smem_u32(stage), xbase = smem_u32(stage + kTileVBytes);
    constexpr uint32_t vplane = 8 * kVGroupBytes, xplane = 8 * kXGroupBytes;
#pragma unroll
    for (int g = 0; g < kContractQ; g++) {
        bool first = true;
#pragma unroll
        for (int s = 0; s <= g; s++) {
            const int tq = g - s;
#pragma unroll
            for (int kk = 0; kk < kContractKC / 16; kk++) {
                // K step kk covers kgroups 2kk and 2kk + 1
                const uint64_t ad = umma_desc(vbase + s * vplane + kk * 2 * kVGroupBytes, kVGroupBytes, 128);
                const uint64_t bd = umma_desc(xbase + tq * xplane + kk * 2 * kXGroupBytes, kXGroupBytes, 128);
                umma_bf16(tmem_acc + g * kContractTileN, ad, bd, idesc, first ? 0u : 1u);
                first = false;
            }
        }
    }
}

// (ah, al) += v + lo
__device__ __forceinline__ void fold_add(float &ah, float &al, float v, float lo)
{
    const float s = ah + v;
    const float bb = s - ah;
    const float e = (ah - (s - bb)) + (v - bb);
    const float l = lo + e;
    ah = s + l;
    al = l - (ah - s);
}

// Folds one chunk's group sums into the double-word accumulators of this
// thread's row and 16 columns.  The digits carry their weights, so group g
// holds S_g = R_g 2^(-8g), a multiple of 2^(-8g) below 2^(24 - 8g): S_0 + S_1,
// S_2 + S_3 and the sum of both lose nothing in fast two-sums, and one
// double-word addition of 2^(e_v + e_x - 16) times the result replaces one
// per group.
__device__ __forceinline__ void fold_chunk(uint32_t tmem_row, const ContractScales &sc, int row, int col0,
                                           float (&ah)[kContractFoldCols], float (&al)[kContractFoldCols])
{
    constexpr int C = 8;
    const float pv = sc.pv[row];
#pragma unroll
    for (int c0 = 0; c0 < kContractFoldCols; c0 += C) {
        float S[kContractQ][C], p2[C];
        tmem_ld8_groups<kContractQ>(tmem_row + c0, 0, S);
        float lo = pv, hi = pv;
#pragma unroll
        for (int c = 0; c < C; c += 4) {
            const float4 w = *reinterpret_cast<const float4 *>(&sc.px[col0 + c0 + c]);
            p2[c] = pv * w.x;
            p2[c + 1] = pv * w.y;
            p2[c + 2] = pv * w.z;
            p2[c + 3] = pv * w.w;
        }
#pragma unroll
        for (int c = 0; c < C; c++) {
            lo = fminf(lo, p2[c]);
            hi = fmaxf(hi, p2[c]);
        }
        // every product below is then a normal float
        if (lo >= 0x1p-70f && hi <= 0x1p100f) {
#pragma unroll
            for (int c = 0; c < C; c++) {
                float s, e, u, f, w, g;
                fast_two_sum(S[0][c], S[1][c], s, e);
                fast_two_sum(S[2][c], S[3][c], u, f);
                fast_two_sum(s, u, w, g);
                fold_add(ah[c0 + c], al[c0 + c], w * p2[c], al[c0 + c] + (e + f + g) * p2[c]);
            }
        } else {
#pragma unroll
            for (int c = 0; c < C; c++) {
                const int esum = sc.ev[row] + sc.ex[col0 + c0 + c] - 16;
#pragma unroll
                for (int g = 0; g < kContractQ; g++)
                    fold_add(ah[c0 + c], al[c0 + c], ldexpf(S[g][c], esum), al[c0 + c]);
            }
        }
    }
}

// grid = tiles x splits, kContractThreads threads, kContractSmem dynamic shared memory
__global__ void __launch_bounds__(kContractThreads, 1) contract_kernel(ContractParams p)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t *done = reinterpret_cast<uint64_t *>(smem + 2 * kStageBytes); // [2]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 2);
    __shared__ ContractScales scales[3];             // of chunk idx in idx % 3: see the loop
    __shared__ const double *xrow_s[2][kContractKC]; // x-row pointers of the chunk in each stage

    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int tile = blockIdx.x % kContractTiles, split = blockIdx.x / kContractTiles;
    const int ti = tile / (kContractN / kContractTileN), tj = tile % (kContractN / kContractTileN);
    const int K = *p.k_total;
    const int nc = (K + kContractKC - 1) / kContractKC;
    const int c0 = (int)((long long)split * nc / p.splits), c1 = (int)((long long)(split + 1) * nc / p.splits);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (t == 0) {
        mbar_init(&done[0], 1);
        mbar_init(&done[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // this thread's accumulator row and columns: warp w reads tensor-memory
    // lanes 32 (w % 4) .. +31, columns 16 (w / 4) .. +15 of each group
    const int row = 32 * (warp & 3) + lane, col0 = kContractFoldCols * (warp >> 2);
    const uint32_t lane_addr = (uint32_t)(32 * (warp & 3)) << 16;
    float ah[kContractFoldCols], al[kContractFoldCols];
#pragma unroll
    for (int c = 0; c < kContractFoldCols; c++)
        ah[c] = al[c] = 0.0f;

    // One barrier a chunk: a thread slices chunk idx, meets the others, and
    // folds chunk idx - 1 while the MMAs of idx run.  What the next chunk
    // overwrites is free by then:
    // - stage and accumulators of idx - 2: every thread has waited for its
    //   MMAs and folded it before the barrier of idx;
    // - the scales of idx - 1 are read after that barrier, while a thread that
    //   is ahead already writes those of idx + 1: three sets;
    // - the row pointers of idx are read before it: two sets.
    // ok is uniform in a warp, and in the block from barrier to barrier (a
    // bounded wait that gave up stops the work of all).
    bool ok = true;
    int issued = 0, waited = 0; // chunks committed / chunks whose commit was awaited
    const int n = c1 - c0;
    const double *base = nullptr;
    if (n > 0) {
        prefetch_chunk(p, c0, K, ti, tj, chunk_row(p, c0, K), xrow_s[0]);
        if (n > 1)
            base = chunk_row(p, c0 + 1, K);
    }
    __syncthreads();
    int cur = 0, last = 2; // idx % 3, (idx - 1) % 3
    for (int idx = 0; idx < n; idx++) {
        const int st = idx & 1;
        if (ok) {
            slice_chunk(p, c0 + idx, K, ti, tj, smem + st * kStageBytes, scales[cur], xrow_s[st]);
            if (idx + 1 < n)
                prefetch_chunk(p, c0 + idx + 1, K, ti, tj, base, xrow_s[st ^ 1]);
            if (idx + 2 < n)
                base = chunk_row(p, c0 + idx + 2, K);
        }
        // the digit planes, written by this CTA's threads, feed the tensor core
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        ok = __syncthreads_and(ok) != 0;
        if (ok) {
            if (t == kContractThreads - 32) {
                tc_fence_after();
                issue_chunk(tmem + st * kContractQ * kContractTileN, smem + st * kStageBytes);
                umma_commit(&done[st]);
            }
            __syncwarp();
            issued = idx + 1;
            if (idx > 0) {
                // the previous chunk's group sums
                const int pst = st ^ 1;
                ok = __all_sync(0xffffffffu, mbar_wait_bounded(&done[pst], ((idx - 1) >> 1) & 1, p.error)) != 0;
                if (ok) {
                    waited = idx;
                    tc_fence_after();
                    fold_chunk(tmem + lane_addr + pst * kContractQ * kContractTileN + col0, scales[last], row, col0,
                               ah, al);
                }
            }
        }
        last = cur;
        cur = cur == 2 ? 0 : cur + 1;
    }
    if (ok && issued == n && n > 0) {
        const int idx = n - 1, st = idx & 1;
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(&done[st], (idx >> 1) & 1, p.error)) != 0;
        if (ok) {
            waited = n;
            tc_fence_after();
            fold_chunk(tmem + lane_addr + st * kContractQ * kContractTileN + col0, scales[last], row, col0, ah, al);
        }
    }
    // after an error: wait (bounded) for the MMAs still in flight before the
    // tensor memory is released
    for (int c = waited; c < issued; c++)
        (void)mbar_wait_bounded(&done[c & 1], (c >> 1) & 1, p.error);
    // partial[split][j][i] (transposed, as the fixed-order reduction reads it)
    const int i = ti * kContractTileM + row;
#pragma unroll
    for (int c = 0; c < kContractFoldCols; c++) {
        const int j = tj * kContractTileN + col0 + c;
        p.partials[((size_t)split * kContractN + j) * kContractN + i] = (double)ah[c] + (double)al[c];
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// x_k pointers of a dense [K][256] factor matrix (the diagnostic entry point)
__global__ void dense_rows_kernel(const double *x, int K, const double **xp)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < K)
        xp[k] = x + (size_t)k * kContractN;
}

// dA[i][j] = sum over splits, in split order, of partial[split][j][i]; NaN
// everywhere when a wait of the contraction gave up
__global__ void reduce_partials_kernel(const double *part, int nparts, const unsigned *error, double *dA)
{
    constexpr int NT = kContractN;
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; // k = j * NT + i
    if (k >= (size_t)NT * NT)
        return;
    double s = 0.0;
    for (int c = 0; c < nparts; c++)
        s += part[(size_t)c * NT * NT + k];
    if (*error)
        s = __longlong_as_double(0x7ff8000000000000ll);
    const size_t j = k / NT, i = k % NT;
    dA[i * NT + j] = s;
}

int contract_splits(int sm_count) { return std::max(1, sm_count / kContractTiles); }

cudaError_t enqueue_factor_offsets(const int *inst_T, const int *inst_status, int B, int nsv, int *k_base,
                                   cudaStream_t s)
{
    factor_offsets_kernel<<<1, 1024, 0, s>>>(inst_T, inst_status, B, nsv, k_base);
    return cudaGetLastError();
}

cudaError_t contract_prepare()
{
    return cudaFuncSetAttribute(contract_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kContractSmem);
}

cudaError_t enqueue_contract(const ContractParams &p, double *dA, cudaStream_t s)
{
    contract_kernel<<<kContractTiles * p.splits, kContractThreads, kContractSmem, s>>>(p);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    constexpr int NN = kContractN * kContractN;
    reduce_partials_kernel<<<(NN + 255) / 256, 256, 0, s>>>(p.partials, p.splits, p.error, dA);
    return cudaGetLastError();
}

} // namespace va

extern "C" VA_API int32_t va_contract_dA(int32_t K, const double *v, const double *x, double *dA, void *stream)
{
    if (K < 0 || !v || !x || !dA)
        return VA_BAD_ARGS;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return VA_CUDA_ERROR;
    cudaStream_t s = (cudaStream_t)stream;
    const int splits = va::contract_splits(sms);
    const double **xp = nullptr;
    int *k_total = nullptr;
    unsigned *err = nullptr;
    double *part = nullptr;
    const size_t nn = (size_t)va::kContractN * va::kContractN;
    int32_t st = VA_OK;
    if (cudaMalloc(&xp, sizeof(double *) * (size_t)std::max(K, 1)) != cudaSuccess ||
        cudaMalloc(&k_total, sizeof(int)) != cudaSuccess || cudaMalloc(&err, sizeof(unsigned)) != cudaSuccess ||
        cudaMalloc(&part, sizeof(double) * nn * splits) != cudaSuccess)
        st = VA_CUDA_ERROR;
    if (st == VA_OK) {
        va::dense_rows_kernel<<<(K + 255) / 256 + 1, 256, 0, s>>>(x, K, xp);
        cudaMemcpyAsync(k_total, &K, sizeof(int), cudaMemcpyHostToDevice, s);
        cudaMemsetAsync(err, 0, sizeof(unsigned), s);
        va::ContractParams p{};
        p.v = v;
        p.xp = xp;
        p.k_total = k_total;
        p.partials = part;
        p.splits = splits;
        p.error = err;
        if (va::contract_prepare() != cudaSuccess || va::enqueue_contract(p, dA, s) != cudaSuccess)
            st = VA_CUDA_ERROR;
        unsigned e = 0;
        if (cudaMemcpyAsync(&e, err, sizeof(unsigned), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            st = VA_CUDA_ERROR;
        else if (e)
            st = VA_CUDA_ERROR;
    }
    cudaFree(xp);
    cudaFree(k_total);
    cudaFree(err);
    cudaFree(part);
    return st;
}

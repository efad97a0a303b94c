// Deterministic reductions and the exclusive scan used by the CIC bucketing.
//
// Every FP64 sum in the step (MG residual norms, kinetic energy) is reduced in a
// fixed order: a fixed shuffle tree inside each warp, a fixed order across the
// warps of a block, one partial per block, then one block that walks the
// partials in index order.  The result is bit-identical run to run for a given
// grid size, unlike the reference's OpenMP REDUCTION whose order follows the
// thread count (scripts/compare_residuals.py checks exactly that drift).
#include "mgg_internal.cuh"
#include "reduce.cuh"

namespace mgg {

namespace {

// The scan of the CIC row counts (up to 2^20 + 1 of them) is a latency chain, not a
// bandwidth problem: 8192 counts per block (eight in a row per thread, then warp
// shuffles), one launch up to 8192 counts and a second one that adds the totals of
// the blocks before each block otherwise.
constexpr int kScanThreads = 1024, kScanPer = 8, kScanItems = kScanThreads * kScanPer;

// exclusive sum of v over the block's threads; total: the block's sum (every thread)
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t& total) {
    __shared__ uint32_t wsum[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    uint32_t t = wsum[lane];   // 32 warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += y;
    }
    total = __shfl_sync(0xffffffffu, t, 31);
    const uint32_t before = __shfl_sync(0xffffffffu, t, w == 0 ? 0 : w - 1);
    return x - v + (w == 0 ? 0u : before);
}

__global__ void __launch_bounds__(kScanThreads) k_scan_block(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                             uint32_t* __restrict__ block_sums, int64_t n) {
    const int64_t g = (int64_t)blockIdx.x * kScanItems + kScanPer * threadIdx.x;
    uint32_t v[kScanPer];
    if (g + kScanPer <= n) {   // in and out are 16-byte aligned
        const uint4 a = *reinterpret_cast<const uint4*>(in + g), b = *reinterpret_cast<const uint4*>(in + g + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < kScanPer; ++i) v[i] = g + i < n ? in[g + i] : 0u;
    }
    uint32_t sum = 0;
#pragma unroll
    for (int i = 0; i < kScanPer; ++i) {
        const uint32_t t = v[i];
        v[i] = sum;
        sum += t;
    }
    uint32_t total;
    const uint32_t base = block_scan(sum, total);
    if (g + kScanPer <= n) {
        *reinterpret_cast<uint4*>(out + g) = make_uint4(base + v[0], base + v[1], base + v[2], base + v[3]);
        *reinterpret_cast<uint4*>(out + g + 4) = make_uint4(base + v[4], base + v[5], base + v[6], base + v[7]);
    } else {
#pragma unroll
        for (int i = 0; i < kScanPer; ++i)
            if (g + i < n) out[g + i] = base + v[i];
    }
    if (threadIdx.x == 0 && block_sums) block_sums[blockIdx.x] = total;
}

// adds the totals of blocks 0 .. blockIdx.x (of at most 1024) to block blockIdx.x + 1
__global__ void __launch_bounds__(kScanThreads) k_scan_add(uint32_t* __restrict__ out,
                                                           const uint32_t* __restrict__ block_sums, int64_t n) {
    uint32_t add;
    block_scan(threadIdx.x <= blockIdx.x ? block_sums[threadIdx.x] : 0u, add);
    const int64_t g = (int64_t)(blockIdx.x + 1) * kScanItems + kScanPer * threadIdx.x;
    if (g + kScanPer <= n) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint4 a = *reinterpret_cast<uint4*>(out + g + 4 * h);
            a.x += add; a.y += add; a.z += add; a.w += add;
            *reinterpret_cast<uint4*>(out + g + 4 * h) = a;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kScanPer; ++i)
            if (g + i < n) out[g + i] += add;
    }
}

__global__ void k_sum_partials(const double* __restrict__ part, int n, double* __restrict__ out) {
    double v = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) v += part[i];
    v = block_sum_fixed(v);
    if (threadIdx.x == 0) out[0] = v;
}

}  // namespace

void scan_exclusive(const uint32_t* in, uint32_t* out, uint32_t* sums, int64_t n, cudaStream_t s) {
    const int nb = div_up(n, kScanItems);
    if (nb > kScanThreads) throw Error{MGG_ERR_ARG, "scan: too many elements"};
    k_scan_block<<<nb, kScanThreads, 0, s>>>(in, out, sums, n);
    MGG_CHECK_LAUNCH();
    if (nb == 1) return;
    k_scan_add<<<nb - 1, kScanThreads, 0, s>>>(out, sums, n);
    MGG_CHECK_LAUNCH();
}

void ensure_partials(Ctx& c, int n) {
    if (n <= c.red_capacity) return;
    if (c.red_partial) MGG_CUDA(cudaFree(c.red_partial));
    c.red_partial = nullptr;
    int cap = n < 4096 ? 4096 : n;
    MGG_CUDA(cudaMalloc(&c.red_partial, sizeof(double) * cap));
    c.red_capacity = cap;
}

void reduce_sum_blocks_async(Ctx& c, int nblocks, double* out) {
    ProfScope ps(c, K_MG_REDUCE, 8.0 * nblocks);
    k_sum_partials<<<1, 1024, 0, c.stream>>>(c.red_partial, nblocks, out);
    MGG_CHECK_LAUNCH();
}

double reduce_sum_blocks(Ctx& c, int nblocks) {
    reduce_sum_blocks_async(c, nblocks, c.red_out);
    MGG_CUDA(cudaMemcpyAsync(c.h_red, c.red_out, sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    MGG_CUDA(cudaStreamSynchronize(c.stream));
    return c.h_red[0];
}

}  // namespace mgg

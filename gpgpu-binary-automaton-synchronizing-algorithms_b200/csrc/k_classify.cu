// k_classify.cu -- bucket a mixed-size batch by size class on the device.
//
// The reference bakes one n into the kernel at JIT time (GlobalVariableSymbol,
// GPGPU/GPU/SlimGPUQueue.cs:21,78,216) and therefore cannot run mixed sizes in
// one batch (AlgorithmCorrectnessTestProject/IntegrityTest.cs:68-70).  Here a
// batch with per-automaton n is split into size classes by one small kernel
// whose output -- an order array and a (offset, count) pair per class -- feeds
// each class's persistent kernel without a round trip to the host, so the whole
// chain can be captured in a CUDA graph.
#include "classes.cuh"
#include "common.cuh"

namespace sbfs {
namespace {

constexpr int kBucketThreads = 256;

// Class c's members go to order[c * count ..], counted in ranges[2 * c + 1]: with
// a part of its own per class there are no offsets to wait for, and one launch
// buckets the batch.  A block takes places for its 256 automata with one global
// atomic per class (per warp: 20 us per 200K automata, the five counters being
// the bottleneck; histogram, offsets and scatter together 28 us).
__global__ void __launch_bounds__(kBucketThreads) k_bucket(const uint8_t *ns, int64_t count,
                                                           unsigned long long *ranges, int32_t *order)
{
    __shared__ unsigned int warp_count[kBucketThreads / 32][kNumClasses];
    __shared__ unsigned long long block_base[kNumClasses];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x == 0 && threadIdx.x < kNumClasses) ranges[2 * threadIdx.x] = threadIdx.x * (unsigned long long)count;
    for (int64_t base = blockIdx.x * (int64_t)kBucketThreads; base < count; base += (int64_t)gridDim.x * kBucketThreads) {
        const int64_t i = base + threadIdx.x;
        const int c = i < count ? class_of_n(ns[i]) : -1;
        unsigned rank = 0;
#pragma unroll
        for (int k = 0; k < kNumClasses; ++k) {
            const unsigned m = __ballot_sync(kFull, c == k);
            if (c == k) rank = __popc(m & ((1u << lane) - 1u));
            if (lane == 0) warp_count[warp][k] = __popc(m);
        }
        __syncthreads();
        if (threadIdx.x < kNumClasses) {
            unsigned sum = 0;
            for (int w = 0; w < kBucketThreads / 32; ++w) {
                const unsigned x = warp_count[w][threadIdx.x];
                warp_count[w][threadIdx.x] = sum;
                sum += x;
            }
            block_base[threadIdx.x] = sum ? atomicAdd(&ranges[2 * threadIdx.x + 1], (unsigned long long)sum) : 0ull;
        }
        __syncthreads();
        if (c >= 0) order[c * count + (int64_t)(block_base[c] + warp_count[warp][c] + rank)] = (int32_t)i;
        __syncthreads();
    }
}

}  // namespace

cudaError_t launch_classify(const uint8_t *d_ns, int64_t count, unsigned long long *ranges, int32_t *order,
                            int sm_count, cudaStream_t st)
{
    const int64_t want = (count + kBucketThreads - 1) / kBucketThreads;
    const int blocks = (int)(want < 1 ? 1 : (want > 4 * sm_count ? 4 * sm_count : want));
    k_bucket<<<blocks, kBucketThreads, 0, st>>>(d_ns, count, ranges, order);
    return cudaGetLastError();
}

}  // namespace sbfs

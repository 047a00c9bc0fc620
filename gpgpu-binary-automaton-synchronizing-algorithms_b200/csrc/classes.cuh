// classes.cuh -- size classes: which kernel and which visited-store placement
// serve an automaton with n states.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace sbfs {

// class 0: n <= 8   one automaton per lane, 32-byte bitmap in shared memory
// class 1: n <= 12  one automaton per lane, 192-byte bitmap over the letters' images
//                   (larger ones from a pool of the warp's, or an idle lane's column)
// class 2: n <= 16  one automaton per warp, 4 KiB bitmap over the letters' images or hash
//                   set; what outgrows it: one per CTA, 16 KiB.  A uniform batch of n = 13
//                   or 14: one per lane
// class 3: n <= 20  one automaton per warp (8 KiB), then per CTA: 16 KiB over the images,
//                   or a bit per subset (<= 128 KiB)
// class 4: n <= 28  one automaton per warp, then per CTA, with a hash set in shared
//                   memory; what outgrows both: level-synchronous, bitmap (<= 32 MiB)
//                   and frontier in HBM
// (Classes 0 to 2 also have a warp-pooled kernel, which a handle can ask for and the
// autotuner can choose.)
constexpr int kNumClasses = 5;
constexpr int kClassMaxN[kNumClasses] = {8, 12, 16, 20, 28};
// Out-of-range n (0 or > 28) is routed to class 0, whose kernel rejects it
// as a malformed record.

__host__ __device__ __forceinline__ int class_of_n(int n)
{
    return (n >= 1 && n <= 8) ? 0 : n <= 12 ? 1 : n <= 16 ? 2 : n <= 20 ? 3 : n <= 28 ? 4 : 0;
}

// Buckets d_ns[0..count): ranges[2 * c], ranges[2 * c + 1] = class c's offset into
// order (kNumClasses * count entries) and its members.  The counts start at 0.
cudaError_t launch_classify(const uint8_t *d_ns, int64_t count, unsigned long long *ranges, int32_t *order,
                            int sm_count, cudaStream_t st);

}  // namespace sbfs

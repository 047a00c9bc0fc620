// buffers.hpp -- grow-only device and pinned host allocations of the engine.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <initializer_list>

#include <cuda_runtime_api.h>

namespace sbfs {

struct Buf {
    void *ptr = nullptr;
    size_t bytes = 0;
    uint64_t generation = 0;   // allocations made so far
    template <class T> T *as() const { return static_cast<T *>(ptr); }
};

// What a captured launch sequence depends on: the buffers' addresses and which
// allocation each one is.  An address alone does not tell: a buffer that grew can
// come back at the place of the one it replaced, and the graph's copies still
// refer to the allocation that is gone (cudaGraphLaunch then crashed).
inline uint64_t buffers_signature(std::initializer_list<const Buf *> buffers, uint64_t x = 1469598103934665603ull)
{
    for (const Buf *b : buffers)
        for (const uint64_t v : {(uint64_t) reinterpret_cast<uintptr_t>(b->ptr), b->generation})
            x = (x ^ v) * 1099511628211ull;
    return x;
}

// Device allocation.
struct DevBuf : Buf {
    cudaError_t reserve(size_t want)
    {
        if (want <= bytes && ptr) return cudaSuccess;
        release();
        const size_t sz = std::max<size_t>(want, 256);
        const cudaError_t e = cudaMalloc(&ptr, sz);
        if (e != cudaSuccess) {
            ptr = nullptr;
            cudaGetLastError();
            return e;
        }
        bytes = sz;
        ++generation;
        return cudaSuccess;
    }

    void release()
    {
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
    }
};

// Pinned host allocation, mapped, so kernels may store into it (the streamed host
// path's chunk flags).
struct HostBuf : Buf {
    cudaError_t reserve(size_t want)
    {
        if (want <= bytes && ptr) return cudaSuccess;
        release();
        const size_t sz = std::max<size_t>(want, 256);
        const cudaError_t e = cudaHostAlloc(&ptr, sz, cudaHostAllocMapped);
        if (e != cudaSuccess) {
            ptr = nullptr;
            cudaGetLastError();
            return e;
        }
        bytes = sz;
        ++generation;
        return cudaSuccess;
    }

    void release()
    {
        if (ptr) cudaFreeHost(ptr);
        ptr = nullptr;
        bytes = 0;
    }
};

}  // namespace sbfs

// k_wide.cu -- power-set BFS of automata with up to 28 states, one automaton
// per CTA, with the visited set, the queue and the parents in shared memory.
//
// It takes the automata of 21..28 states whose search outgrows a warp's hash
// set (k_hash.cu: 3072 subsets; 5 % of random automata at n = 24, 12 % at
// n = 28) and is not settled backwards either.  The CTA holds 24,576 subsets:
// all but about 0.2 % of random n = 28.  What is wider still goes on to the
// level slots in HBM (k_level.cu), whose levels each cost a launch.
//   * set: 32,768 slots of a 32-bit subset (0 = free), linear probing, filled
//     with atomicCAS and cleared for every automaton;
//   * queue: 16-bit entries, set slot | letter-is-b << 15, in level order, with
//     a 16-bit parent index each, retained for the word
//     (GPGPU/CPU/CPU.cs:203-205,262-269);
//   * nibble tables of 64-bit entries, a-image << 32 | b-image.
// 225 KB in all: one CTA per SM.  Level-synchronous like
// GPGPU/CPU/SlimCPUUntweaked.cs:119-184, one barrier per level (see k_cta.cu
// for the rotation of the counters).  Bound by the barrier and the dependent
// shared-memory accesses of a level; a level is a microsecond or two.
// n = 24, 26, 28 x (64 random + C_n + permutation-plus-merge), one Verify call:
// 18.0 ms with every automaton on the level slots, 0.73 ms with k_hash and this
// kernel before them.
#include <atomic>

#include "common.cuh"

namespace sbfs {
namespace {

constexpr int kWideThreads = 1024;
constexpr int kWideCapBits = 15;
constexpr int kWideCap = 1 << kWideCapBits;
constexpr uint32_t kWideLimit = 3u * kWideCap / 4u;
constexpr int kWideChunks = 7;

struct WideSmem {
    uint64_t table[16 * kWideChunks];
    uint32_t set[kWideCap];
    uint16_t queue[kWideLimit];
    uint16_t parent[kWideLimit];
};

struct WideCtl {
    int64_t k;
    int n;
    uint32_t found[2];    // min over (queue index << 1 | letter) of a level's singleton hits
    uint32_t cnt[3];
    uint32_t over[2];     // the level found more subsets than the queue holds
    uint32_t single_a[32], single_b[32];
};

// Slot of x when it was not in the set yet, -1 otherwise.  Warps stop at the
// first push past kWideLimit, so at most 64 inserts per warp come after it and
// the set never fills up.
__device__ __forceinline__ int wide_insert(uint32_t *set, uint32_t x)
{
    uint32_t p = (x * 0x9E3779B1u) >> (32 - kWideCapBits);
    for (int probe = 0; probe < kWideCap; ++probe) {
        uint32_t v = set[p];
        if (v == 0u) {
            v = atomicCAS(&set[p], 0u, x);
            if (v == 0u) return (int)p;
        }
        if (v == x) return -1;
        p = (p + 1) & (kWideCap - 1);
    }
    return -1;
}

__global__ void __launch_bounds__(kWideThreads, 1)
    k_wide(const __grid_constant__ Batch b, int32_t *left_list, unsigned long long *left_count,
           unsigned long long *ticket)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WideSmem &S = *reinterpret_cast<WideSmem *>(smem_raw);
    __shared__ WideCtl ctl;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    int64_t count;
    const int32_t *order;
    resolve_work(b, count, order);
    unsigned long long expanded = 0;

    while (true) {
        if (tid == 0) {
            const unsigned long long pos = atomicAdd(ticket, 1ull);
            ctl.k = pos < (unsigned long long)count ? automaton_at(order, (int64_t)pos) : -1;
            if (ctl.k >= 0) ctl.n = automaton_n(b, ctl.k);
        }
        __syncthreads();
        const int64_t k = ctl.k;
        if (k < 0) break;
        const int n = ctl.n;
        // the records were checked by the kernel that handed the automaton on
        if (tid < n) {
            const uint8_t *rec = b.maps + (size_t)k * 2u * (size_t)b.lstride;
            ctl.single_a[tid] = 1u << (rec[tid] & 31);
            ctl.single_b[tid] = 1u << (rec[b.lstride + tid] & 31);
        }
        uint4 *set4 = reinterpret_cast<uint4 *>(S.set);
        for (int i = tid; i < kWideCap / 4; i += kWideThreads) set4[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        if (tid < 16 * kWideChunks) {
            const int c = tid >> 4, v = tid & 15;
            uint32_t ta = 0, tb = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (((v >> j) & 1) && 4 * c + j < n) {
                    ta |= ctl.single_a[4 * c + j];
                    tb |= ctl.single_b[4 * c + j];
                }
            S.table[tid] = ((uint64_t)ta << 32) | tb;
        }
        if (tid == 0) {
            S.queue[0] = (uint16_t)wide_insert(S.set, (1u << n) - 1u);
            ctl.found[0] = ctl.found[1] = ~0u;
            ctl.cnt[0] = ctl.cnt[1] = ctl.cnt[2] = 0u;
            ctl.over[0] = ctl.over[1] = 0u;
        }
        __syncthreads();

        uint32_t ls = 0, le = n > 1 ? 1u : 0u, level = 0;
        while (true) {
            uint32_t *cnt = &ctl.cnt[level % 3];
            uint32_t *found = &ctl.found[level & 1];
            volatile uint32_t *over = &ctl.over[level & 1];
            if (tid == 0) ctl.cnt[(level + 1) % 3] = 0u;
            for (uint32_t base = ls + (tid & ~31); base < le; base += kWideThreads) {
                if (__any_sync(kFull, *over)) break;
                const uint32_t i = base + lane;
                uint32_t ya = 0, yb = 0;
                int sa = -1, sb = -1;
                if (i < le) {
                    const uint32_t x = S.set[S.queue[i] & 0x7FFFu];
                    uint64_t t = S.table[x & 15u];
#pragma unroll
                    for (int c = 1; c < kWideChunks; ++c) t |= S.table[16 * c + ((x >> (4 * c)) & 15u)];
                    ya = (uint32_t)(t >> 32);
                    yb = (uint32_t)t;
                    ++expanded;
                    // no singleton is visited before the first one is generated
                    if (is_singleton(ya))
                        atomicMin(found, i << 1);
                    else
                        sa = wide_insert(S.set, ya);
                    if (is_singleton(yb))
                        atomicMin(found, (i << 1) | 1u);
                    else
                        sb = wide_insert(S.set, yb);
                }
                const unsigned ma = __ballot_sync(kFull, sa >= 0), mb = __ballot_sync(kFull, sb >= 0);
                const uint32_t c = (uint32_t)(__popc(ma) + __popc(mb));
                if (!c) continue;
                uint32_t pos = 0;
                if (lane == 0) {
                    pos = le + atomicAdd(cnt, c);
                    if (pos + c > kWideLimit) *over = 1u;
                }
                pos = __shfl_sync(kFull, pos, 0);
                if (pos + c > kWideLimit) break;
                const unsigned lt = (1u << lane) - 1u;
                pos += __popc(ma & lt) + __popc(mb & lt);
                if (!SBFS_CHECK(pos + (sa >= 0 ? 1u : 0u) + (sb >= 0 ? 1u : 0u) <= kWideLimit, b.error)) sa = sb = -1;
                if (sa >= 0) {
                    S.queue[pos] = (uint16_t)sa;
                    S.parent[pos++] = (uint16_t)i;
                }
                if (sb >= 0) {
                    S.queue[pos] = (uint16_t)(sb | 0x8000);
                    S.parent[pos] = (uint16_t)i;
                }
            }
            __syncthreads();
            const uint32_t f = *found, added = *cnt;
            const bool outgrown = *over != 0u;
            if (f != ~0u) {
                if (tid == 0) {
                    record_result(b, k, n, (int32_t)level + 1);
                    if (b.out_words) {
                        uint64_t *w = b.out_words + (size_t)k * (size_t)b.word_stride;
                        for (int c = 0; c < b.word_stride; ++c) w[c] = 0ull;
                        if (level < 64u * (uint32_t)b.word_stride) {
                            w[level >> 6] |= (uint64_t)(f & 1u) << (level & 63u);
                            uint32_t i = f >> 1;
                            for (int d = (int)level - 1; d >= 0; --d) {
                                w[d >> 6] |= (uint64_t)(S.queue[i] >> 15) << (d & 63);
                                i = S.parent[i];
                            }
                        }
                    }
                    publish_result(b, k);
                }
                break;
            }
            if (outgrown) {
                if (tid == 0) left_list[atomicAdd(left_count, 1ull)] = (int32_t)k;
                break;
            }
            if (added == 0) {
                if (tid == 0) {
                    record_result(b, k, n, kLenNonSync);
                    if (b.out_words)
                        for (int c = 0; c < b.word_stride; ++c) b.out_words[(size_t)k * b.word_stride + c] = 0ull;
                    publish_result(b, k);
                }
                break;
            }
            ls = le;
            le += added;
            ++level;
        }
        __syncthreads();
    }
    for (int o = 16; o; o >>= 1) expanded += __shfl_down_sync(kFull, expanded, o);
    if (lane == 0 && b.expanded && expanded) atomicAdd(b.expanded, expanded);
}

}  // namespace

// Solves the automata of b (n <= 28, one CTA per SM); those that need more
// than kWideLimit subsets are appended to left_list.
cudaError_t launch_wide(int sm_count, const Batch &b, int32_t *left_list, unsigned long long *left_count,
                        unsigned long long *ticket, cudaStream_t st)
{
    if (sm_count < 1 || !left_list || !left_count) return cudaErrorInvalidValue;
    // set once per device: the enqueue paths ask on every launch
    constexpr int kMaxDevices = 16;
    static std::atomic<int> done[kMaxDevices];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool cached = dev >= 0 && dev < kMaxDevices;
    if (!cached || !done[dev].load(std::memory_order_acquire)) {
        e = cudaFuncSetAttribute(k_wide, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WideSmem));
        if (e != cudaSuccess) return e;
        if (cached) done[dev].store(1, std::memory_order_release);
    }
    k_wide<<<sm_count, kWideThreads, sizeof(WideSmem), st>>>(b, left_list, left_count, ticket);
    return cudaGetLastError();
}

}  // namespace sbfs

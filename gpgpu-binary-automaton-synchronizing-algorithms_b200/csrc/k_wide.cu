// k_wide.cu -- power-set BFS of automata with up to 28 states, one automaton
// per CTA, with the visited set, the queue and the parents in shared memory.
//
// It takes the automata of 21..28 states whose search outgrows what a warp
// keeps (k_hash.cu: 1024 subsets; 25 % of random automata at n = 24 pass 1536,
// 5 % pass 3072) and is not settled backwards either.  The CTA holds 24,576 subsets:
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
// 18.0 ms with every automaton on the level slots, 0.42 ms with k_hash and this
// kernel before them.
#include <algorithm>
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
                if (tid == 0) hand_off(b, left_list, left_count, k);
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

// ---- n <= 20 -----------------------------------------------------------------
// The automata of 13..20 states that outgrow a warp (k_hash.cu: 1536 subsets;
// 0.4 % of random automata at n = 16, 4 % at n = 20).  Same search with the
// bitmap of k_hash.cu as its visited store -- states relabelled by image,
// 2^rank(a) + 2^rank(b) bits, 2^17 at most -- and a queue whose first 8192
// subsets stay on chip: 65 KB, so three CTAs per SM instead of the one that
// k_cta.cu's 2^20-bit bitmap allows, and no trips to global memory but for the
// widest searches.  Those continue in a spill of 2^17 entries per CTA, those on
// chip included (2^16 for n <= 16), which no search can outgrow: its subsets have
// different bits.  k_hash sends ranks that need more bits (n > 17 only) to k_cta,
// which runs beside this kernel: after it 600 n = 18 of two rank 17 letters took
// 736 us, so 546 (k_cta alone for all of them: 587), 30K random n = 20 322 and 295.
// The widest search of a batch bounds the launch, hence 512 threads: 30K random
// n = 20 took 0.330 ms with k_cta alone, 0.334 with 256 threads here, 0.315 with
// 512, 0.326 with 1024 (two CTAs per SM); 200K mixed n = 6..20 0.611, 0.599, 0.591
// and 0.611 ms (all with k_cta after it).
constexpr int kMidThreads = 512;
constexpr uint32_t kMidLimit = 8192;
constexpr int kMidWords = kMidBits / 32;
constexpr int kMidChunks = 5;

struct MidSmem {
    uint32_t store[kMidWords];
    uint64_t table[16 * kMidChunks];
    uint32_t queue[kMidLimit];      // subset | letter-is-b << 31
    uint16_t parent[kMidLimit];
};

struct MidCtl {
    int64_t k;
    int n;
    uint32_t low_end, index0, shift, bits;
    uint32_t found[2], cnt[3];            // as in WideCtl
    uint64_t single[32];                  // a's << 32 | b's image of the state with that label
};

__global__ void __launch_bounds__(kMidThreads, 3)
    k_mid(const __grid_constant__ Batch b, uint2 *spill_base, uint32_t spill_entries, unsigned long long *ticket)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MidSmem &S = *reinterpret_cast<MidSmem *>(smem_raw);
    __shared__ MidCtl ctl;
    // {subset | letter-is-b << 31, parent} of the queue entries from kMidLimit on
    uint2 *const spill = spill_base + (size_t)blockIdx.x * spill_entries;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const unsigned lt = (1u << lane) - 1u;
    int64_t count;
    const int32_t *order;
    resolve_work(b, count, order);
    unsigned long long expanded = 0;

    while (true) {
        if (tid < 32) {
            unsigned long long pos = 0;
            if (lane == 0) pos = atomicAdd(ticket, 1ull);
            pos = __shfl_sync(kFull, pos, 0);
            const int64_t k = pos < (unsigned long long)count ? automaton_at(order, (int64_t)pos) : -1;
            int n = 0;
            uint32_t av = 0, bv = 0;
            if (k >= 0) {
                // the record was checked by the kernel that handed the automaton on
                n = automaton_n(b, k);
                const uint8_t *rec = b.maps + (size_t)k * 2u * (size_t)b.lstride;
                if (lane < n) {
                    av = rec[lane] & 31u;
                    bv = rec[b.lstride + lane] & 31u;
                }
            }
            const uint32_t A = __reduce_or_sync(kFull, lane < n ? 1u << av : 0u);
            const uint32_t B = __reduce_or_sync(kFull, lane < n ? 1u << bv : 0u);
            const int ra = __popc(A), rb = __popc(B);
            const bool in_a = (A >> lane) & 1u, in_b = (B >> lane) & 1u;
            int label = in_a ? (in_b ? __popc(A & ~B) + __popc(A & B & lt) : __popc(A & ~B & lt))
                             : (in_b ? ra + __popc(B & ~A & lt) : __popc(A | B) + __popc(~(A | B) & lt));
            if (lane >= n) label = lane;
            const int la = __shfl_sync(kFull, label, (int)av), lb = __shfl_sync(kFull, label, (int)bv);
            ctl.single[label] = lane < n ? ((uint64_t)(1u << la) << 32) | (1u << lb) : 0ull;
            if (lane == 0) {
                ctl.k = k;
                ctl.n = n;
                uint32_t bits = (1u << ra) + ((B & ~A) ? 1u << rb : 0u);
                ctl.low_end = ctl.index0 = 1u << ra;
                ctl.shift = (uint32_t)__popc(A & ~B);
                if (bits > 1u << n) {
                    bits = 1u << n;
                    ctl.index0 = ctl.shift = 0u;
                }
                ctl.bits = SBFS_CHECK(bits <= kMidBits, b.error) ? bits : kMidBits;
                ctl.found[0] = ctl.found[1] = ~0u;
                ctl.cnt[0] = ctl.cnt[1] = ctl.cnt[2] = 0u;
            }
        }
        __syncthreads();
        const int64_t k = ctl.k;
        if (k < 0) break;
        const int n = ctl.n;
        const uint32_t low_end = ctl.low_end, index0 = ctl.index0, shift = ctl.shift, bits = ctl.bits;
        if (tid < 16 * kMidChunks) {
            const int c = tid >> 4, v = tid & 15;
            uint64_t acc = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if ((v >> j) & 1) acc |= ctl.single[4 * c + j];
            S.table[tid] = acc;
        }
        uint4 *store4 = reinterpret_cast<uint4 *>(S.store);
        for (uint32_t i = tid; i < (bits + 127u) / 128u; i += kMidThreads) store4[i] = make_uint4(0u, 0u, 0u, 0u);
        const uint32_t full = (1u << n) - 1u;
        if (tid == 0) S.queue[0] = full;
        __syncthreads();
        // the root comes back only through a permutation, and then the index is plain:
        // the first level sets its bit before any other thread reads the store
        uint32_t ls = 0, le = n > 1 ? 1u : 0u, level = 0;
        if (tid == 0 && (index0 == 0u || low_end > full) && SBFS_CHECK((full >> 5) < (uint32_t)kMidWords, b.error))
            S.store[full >> 5] |= 1u << (full & 31u);
        while (true) {
            uint32_t *cnt = &ctl.cnt[level % 3];
            uint32_t *found = &ctl.found[level & 1];
            if (tid == 0) ctl.cnt[(level + 1) % 3] = 0u;
            for (uint32_t base = ls + (tid & ~31); base < le; base += kMidThreads) {
                const uint32_t i = base + lane;
                uint32_t ya = 0, yb = 0;
                bool fa = false, fb = false;
                if (i < le) {
                    const uint32_t x = (i < kMidLimit ? S.queue[i] : spill[i - kMidLimit].x) & 0x7FFFFFFFu;
                    uint64_t t = S.table[x & 15u];
#pragma unroll
                    for (int c = 1; c < kMidChunks; ++c) t |= S.table[16 * c + ((x >> (4 * c)) & 15u)];
                    ya = (uint32_t)(t >> 32);
                    yb = (uint32_t)t;
                    ++expanded;
                    // no singleton is visited before the first one is generated
                    const bool sa = is_singleton(ya), sb = is_singleton(yb);
                    if (sa || sb) atomicMin(found, (i << 1) | (sa ? 0u : 1u));
                    const uint32_t ib = yb < low_end ? yb : index0 + (yb >> shift);
                    if (SBFS_CHECK(ya < 32u * kMidWords && ib < 32u * kMidWords, b.error)) {
                        const uint32_t ma = 1u << (ya & 31u), mb = 1u << (ib & 31u);
                        const uint32_t oa = atomicOr(&S.store[ya >> 5], ma);
                        const uint32_t ob = atomicOr(&S.store[ib >> 5], mb);
                        fa = !(oa & ma);
                        fb = !(ob & mb);
                    }
                }
                const unsigned ma = __ballot_sync(kFull, fa), mb = __ballot_sync(kFull, fb);
                const uint32_t c = (uint32_t)(__popc(ma) + __popc(mb));
                if (!c) continue;
                uint32_t pos = 0;
                if (lane == 0) pos = le + atomicAdd(cnt, c);
                pos = __shfl_sync(kFull, pos, 0) + __popc(ma & lt) + __popc(mb & lt);
                // (a parent below kMidLimit fits 16 bits; one past it pushes past it)
                auto push = [&](uint32_t p, uint32_t e) {
                    if (p < kMidLimit) {
                        S.queue[p] = e;
                        S.parent[p] = (uint16_t)i;
                    } else if (SBFS_CHECK(p - kMidLimit < spill_entries, b.error)) {
                        spill[p - kMidLimit] = make_uint2(e, i);
                    }
                };
                if (fa) push(pos++, ya);
                if (fb) push(pos, yb | 0x80000000u);
            }
            __syncthreads();
            const uint32_t f = *found, added = *cnt;
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
                                const uint2 e = i < kMidLimit ? make_uint2(S.queue[i], S.parent[i])
                                                              : spill[i - kMidLimit];
                                w[d >> 6] |= (uint64_t)(e.x >> 31) << (d & 63);
                                i = e.y;
                            }
                        }
                    }
                    publish_result(b, k);
                }
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

// Dynamic shared memory of a kernel, set once per device: the enqueue paths ask
// on every launch.
template <class F>
cudaError_t allow_smem(F *kernel, size_t bytes, std::atomic<int> (&done)[16])
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool cached = dev >= 0 && dev < 16;
    if (cached && done[dev].load(std::memory_order_acquire)) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess && cached) done[dev].store(1, std::memory_order_release);
    return e;
}

}  // namespace

// CTAs that `count` hand-offs at most can keep busy
int mid_ctas(int sm_count, int64_t count)
{
    return (int)std::max<int64_t>(1, std::min<int64_t>(3 * (int64_t)sm_count, count));
}

// uint64 entries per CTA of the spill that launch_mid takes, for automata of
// up to max_n states
size_t mid_spill_entries(int max_n)
{
    const size_t most = max_n < 17 ? (size_t)1 << max_n : kMidBits;   // by its bitmap
    return most > kMidLimit ? most - kMidLimit : 0;
}

// Solves the automata of b (at most max_n <= 20 states, images of at most
// kMidBits bits).
cudaError_t launch_mid(int ctas, int max_n, const Batch &b, uint64_t *spill, unsigned long long *ticket,
                       cudaStream_t st)
{
    if (ctas < 1) return cudaErrorInvalidValue;
    static std::atomic<int> done[16];
    const cudaError_t e = allow_smem(k_mid, sizeof(MidSmem), done);
    if (e != cudaSuccess) return e;
    k_mid<<<ctas, kMidThreads, sizeof(MidSmem), st>>>(b, reinterpret_cast<uint2 *>(spill),
                                                      (uint32_t)mid_spill_entries(max_n), ticket);
    return cudaGetLastError();
}

// Solves the automata of b (n <= 28, one CTA per SM); those that need more
// than kWideLimit subsets are appended to left_list.
cudaError_t launch_wide(int sm_count, const Batch &b, int32_t *left_list, unsigned long long *left_count,
                        unsigned long long *ticket, cudaStream_t st)
{
    if (sm_count < 1 || !left_list || !left_count) return cudaErrorInvalidValue;
    static std::atomic<int> done[16];
    const cudaError_t e = allow_smem(k_wide, sizeof(WideSmem), done);
    if (e != cudaSuccess) return e;
    k_wide<<<sm_count, kWideThreads, sizeof(WideSmem), st>>>(b, left_list, left_count, ticket);
    return cudaGetLastError();
}

}  // namespace sbfs

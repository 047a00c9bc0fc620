// k_hash.cu -- power-set BFS of automata with 13..28 states (size classes 2,
// 3 and 4) with one warp per automaton and an open-addressed hash set as the
// visited store.
//
// A random automaton of 13..20 states is settled after a few hundred subsets
// over ~11 levels (its shortest word is at most ~36 letters), so neither a
// 2^n-bit bitmap (128 KiB at n = 20) nor a 1024-thread CTA (k_cta.cu) pays for
// itself: the CTA's per-level barriers and round trips dominate.  Here each
// warp keeps in shared memory
//   * nibble tables: table[c][v] = (a-image << 32) | b-image of the states
//     4c..4c+3 selected by v, so both images of a subset are 4, 5 or 7 loads
//     (instances for n <= 16, 20 and 28: four instead of five at n = 16 is
//     1.124 -> 1.120 ms per 200K automata);
//   * a hash set of 2^CAP_BITS slots, each holding subset | generation << MAXN;
//     the generation changes with every search, so a slot from an earlier one
//     reads as empty and the set is cleared when the generations (2^(32 - MAXN))
//     wrap;
//   * a level-ordered queue of 16-bit entries, set slot | letter-is-b << 15
//     (a slot keeps its subset for the whole search), with a 16-bit parent
//     index per entry, retained for the word (GPGPU/CPU/CPU.cs:203-205).
// 15 KB per warp at 2048 slots: five warps per CTA, three CTAs per SM.  Sizes
// above 20 take 4096 slots (29 KB, seven warps per SM): at n = 24 5 % of random
// automata pass 3072 subsets, 25 % would pass 1536.
// The warp expands 32 subsets of the current level per step (level-
// synchronous, as GPGPU/CPU/SlimCPUUntweaked.cs:119-184), tests the images
// against the set (atomicCAS insert), and appends the new ones compacted by
// ballots in queue order.  An automaton that needs more than 3/4 of the set's
// slots or kHashLevelCap levels is tried backwards by the same warp
// (inverse_search below), which settles the slowly synchronizing families and
// the automata that never synchronize; what is left -- wide both ways -- goes
// to the CTA-wide kernel (k_cta, or k_wide above n = 20) through a list.  Random n = 17..20: 1.7 % of the
// automata pass 1536 subsets, 0.3 % pass 4096.  200K mixed n = 6..20 with 1 %
// Cerny automata: 3.04 ms with every such automaton on the CTA-wide kernel,
// 1.20 ms with the inverse search.
#include <atomic>

#include "common.cuh"

namespace sbfs {
namespace {

constexpr uint32_t kHashLevelCap = 48;         // random n <= 20: at most ~40 levels
constexpr uint32_t kUnsettled = 1u << 31;

template <int CAP_BITS, int MAXN>
struct HashGeom {
    static constexpr int kCap = 1 << CAP_BITS;                  // hash slots per warp
    static constexpr uint32_t kLimit = 3u * (1u << CAP_BITS) / 4u;   // subsets a warp keeps
    // warps per CTA: 2048 slots 75 KB, three CTAs per SM; 4096 slots 29 KB, seven
    static constexpr int kWarps = CAP_BITS <= 11 ? 5 : 1;
    static constexpr int kMaxN = MAXN;
    static constexpr int kChunks = (MAXN + 3) / 4;               // nibble tables
    static constexpr int kEntries = 16 * kChunks;
    static constexpr uint32_t kSubsetMask = (1u << kMaxN) - 1u;
    static constexpr uint32_t kGens = 1u << (32 - kMaxN);        // generation 0 marks never-used slots
};

template <int CAP_BITS, int MAXN>
struct __align__(16) HashWarp {
    using G = HashGeom<CAP_BITS, MAXN>;
    uint64_t table[G::kEntries];
    uint32_t set[G::kCap];
    uint16_t queue[G::kLimit];    // set slot | letter-is-b << 15
    uint16_t parent[G::kLimit];
};

template <int CAP_BITS>
__device__ __forceinline__ uint32_t hash_slot(uint32_t x)
{
    return (x * 0x9E3779B1u) >> (32 - CAP_BITS);
}

// Inserts subset x (generation gen); returns its slot when it was not yet in
// the set, -1 otherwise.
template <int CAP_BITS, int MAXN>
__device__ __forceinline__ int set_insert(uint32_t *set, uint32_t x, uint32_t gen)
{
    constexpr int kCap = 1 << CAP_BITS;
    const uint32_t key = x | (gen << MAXN);
    uint32_t p = hash_slot<CAP_BITS>(x);
    for (int probe = 0; probe < kCap; ++probe) {
        uint32_t v = set[p];
        while ((v >> MAXN) != gen) {   // a slot of an earlier automaton: empty for this one
            const uint32_t prev = atomicCAS(&set[p], v, key);
            if (prev == v) return (int)p;
            v = prev;   // someone else took it: look at what is there now
        }
        if (v == key) return -1;
        p = (p + 1) & (kCap - 1);
    }
    return -1;   // unreachable: the set is never more than ~3/4 full
}

// Entries of the nibble tables from one 64-bit mask pair per state (lane q
// holds state q's, a's mask << 32 | b's), in passes of 32 that every lane takes
// (the shuffles need the whole warp); a last half pass stores lanes 0..15 only.
template <int CAP_BITS, int MAXN>
__device__ __forceinline__ void build_table(HashWarp<CAP_BITS, MAXN> &W, uint64_t mine, int n, int lane)
{
    using G = HashGeom<CAP_BITS, MAXN>;
#pragma unroll
    for (int pass = 0; pass < (G::kEntries + 31) / 32; ++pass) {
        const int e = lane + 32 * pass;
        const int c = min(e >> 4, G::kChunks - 1), v = e & 15;
        uint64_t acc = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint64_t sj = __shfl_sync(kFull, mine, 4 * c + j);
            if (((v >> j) & 1) && 4 * c + j < n) acc |= sj;
        }
        if (e < G::kEntries) W.table[e] = acc;
    }
}

// a's mask << 32 | b's mask of subset x
template <int CAP_BITS, int MAXN>
__device__ __forceinline__ uint64_t lookup(const HashWarp<CAP_BITS, MAXN> &W, uint32_t x)
{
    uint64_t t = W.table[x & 15u];
#pragma unroll
    for (int c = 1; c < HashGeom<CAP_BITS, MAXN>::kChunks; ++c) t |= W.table[16 * c + ((x >> (4 * c)) & 15u)];
    return t;
}

// The generation of the next search; the set is cleared when they wrap.
template <int CAP_BITS, int MAXN>
__device__ __forceinline__ void next_generation(HashWarp<CAP_BITS, MAXN> &W, uint32_t &gen, int lane)
{
    if (++gen == HashGeom<CAP_BITS, MAXN>::kGens) {
        for (int i = lane; i < HashGeom<CAP_BITS, MAXN>::kCap; i += 32) W.set[i] = 0u;
        gen = 1;
        __syncwarp();
    }
}

__device__ __forceinline__ void write_not_synchronizing(const Batch &b, int64_t k, int n)
{
    record_result(b, k, n, kLenNonSync);
    if (b.out_words)
        for (int c = 0; c < b.word_stride; ++c) b.out_words[(size_t)k * b.word_stride + c] = 0ull;
    publish_result(b, k);
}

// The inverse search, for an automaton that the forward search gave up on
// (lane q < n holds a(q) and b(q)).  A word w synchronizes iff w^-1(q) is the
// full set for some state q, and (cw)^-1(q) = c^-1(w^-1(q)): so a breadth-first
// search from the n singletons along preimages reaches the full set first at
// the length of the shortest word, and the parent chain from there spells the
// word from its first letter on.  It runs out without the full set iff the
// automaton is not synchronizing.
//
// The slowly synchronizing families (Cerny automata, a permutation plus one
// merge) have up to 2^n images of the full set but at most n(n-1)+1 preimages
// of singletons: C_20 is settled by 380 sets over 361 levels (tens of
// microseconds in one warp; all 2^20 forward subsets took a 1024-thread CTA
// 1.2 ms).  Their levels hold 1 to n sets; a random automaton whose forward
// search is wide passes n sets in a level at its fifth or sixth (9,000 random
// n = 13..28 with over 1536 images: none was settled before that).  So the
// search stops at the first level wider than n sets, which also keeps every
// level within one step of the warp.
//
// Before giving up, pairs of states settle the wide automata that never
// synchronize: an automaton synchronizes iff every pair of its states is merged
// by some word.  Row q (lane q) collects the states that can be merged with q,
// preimages of the rows of a(q) and b(q), until nothing changes.
//
// Takes a fresh generation; returns the sets this lane expanded, with the top
// bit clear when the automaton is settled and set when it is left to the
// CTA-wide kernel.
template <int CAP_BITS, int MAXN>
__device__ __noinline__ uint32_t inverse_search(const Batch &b, int64_t k, int n, uint32_t av, uint32_t bv,
                                                HashWarp<CAP_BITS, MAXN> &W, uint32_t gen, int lane)
{
    using G = HashGeom<CAP_BITS, MAXN>;
    uint32_t expanded = 0;
    const uint32_t full = (1u << n) - 1u;
    // lane q: the states that a (b) sends to q
    uint64_t inv = 0;
    for (int q = 0; q < n; ++q) {
        const unsigned ia = __ballot_sync(kFull, lane < n && av == (uint32_t)q);
        const unsigned ib = __ballot_sync(kFull, lane < n && bv == (uint32_t)q);
        if (lane == q) inv = ((uint64_t)ia << 32) | ib;
    }
    build_table<CAP_BITS, MAXN>(W, inv, n, lane);
    __syncwarp();
    if (lane < n) W.queue[lane] = (uint16_t)set_insert<CAP_BITS, MAXN>(W.set, 1u << lane, gen);
    __syncwarp();
    uint32_t head = 0, lvl_end = (uint32_t)n, tail = lvl_end, level = 0;
    uint32_t found = 0, found_letter = 0;
    bool hit = false, spent = true;   // spent: no set left to expand
    while (head < lvl_end) {
        const uint32_t idx = head + (uint32_t)lane;
        const bool has = idx < lvl_end;
        uint32_t ya = 0, yb = 0;
        if (has) {
            const uint64_t t = lookup<CAP_BITS, MAXN>(W, W.set[W.queue[idx] & 0x7FFFu] & G::kSubsetMask);
            ya = (uint32_t)(t >> 32);
            yb = (uint32_t)t;
        }
        expanded += has ? 1u : 0u;
        const unsigned hits = __ballot_sync(kFull, ya == full || yb == full);
        if (hits) {
            const int fl = __ffs(hits) - 1;
            found = head + (uint32_t)fl;
            found_letter = (uint32_t)__shfl_sync(kFull, ya == full ? 0 : 1, fl);
            hit = true;
            break;
        }
        const int sa = ya ? set_insert<CAP_BITS, MAXN>(W.set, ya, gen) : -1;
        const int sb = yb ? set_insert<CAP_BITS, MAXN>(W.set, yb, gen) : -1;
        bool fa = sa >= 0, fb = sb >= 0;
        const unsigned ma = __ballot_sync(kFull, fa), mb = __ballot_sync(kFull, fb);
        const uint32_t added = (uint32_t)(__popc(ma) + __popc(mb));
        if (tail + added > min(G::kLimit, lvl_end + (uint32_t)n)) {
            spent = false;
            break;
        }
        const unsigned lt = (1u << lane) - 1u;
        uint32_t p = tail + (uint32_t)(__popc(ma & lt) + __popc(mb & lt));
        if (!SBFS_CHECK(p + (fa ? 1u : 0u) + (fb ? 1u : 0u) <= G::kLimit, b.error)) fa = fb = false;
        if (fa) {
            W.queue[p] = (uint16_t)sa;
            W.parent[p++] = (uint16_t)idx;
        }
        if (fb) {
            W.queue[p] = (uint16_t)(sb | 0x8000);
            W.parent[p] = (uint16_t)idx;
        }
        tail += added;
        head = lvl_end;   // a level is one step: at most n sets
        lvl_end = tail;
        __syncwarp();
        if (head < lvl_end) ++level;
    }
    if (hit) {
        __syncwarp();
        if (lane == 0) {
            record_result(b, k, n, (int32_t)level + 1);
            if (b.out_words) {
                uint64_t *w = b.out_words + (size_t)k * (size_t)b.word_stride;
                uint64_t acc = found_letter;
                int c = 0;
                uint32_t i = found;
                if (level < 64u * (uint32_t)b.word_stride) {
                    for (uint32_t d = 1; d <= level; ++d) {
                        if ((d & 63u) == 0u) {
                            w[c++] = acc;
                            acc = 0ull;
                        }
                        acc |= (uint64_t)(W.queue[i] >> 15) << (d & 63u);
                        i = W.parent[i];
                    }
                    w[c++] = acc;
                }
                for (; c < b.word_stride; ++c) w[c] = 0ull;
            }
            publish_result(b, k);
        }
        __syncwarp();
        return expanded;
    }
    if (!spent) {
        uint32_t row = lane < n ? 1u << lane : 0u;
        while (true) {
            const uint32_t ra = __shfl_sync(kFull, row, (int)av), rb = __shfl_sync(kFull, row, (int)bv);
            const uint32_t grown =
                row | (uint32_t)(lookup<CAP_BITS, MAXN>(W, ra) >> 32) | (uint32_t)lookup<CAP_BITS, MAXN>(W, rb);
            const bool more = lane < n && grown != row;
            if (lane < n) row = grown;
            if (!__any_sync(kFull, more)) break;
        }
        if (__all_sync(kFull, lane >= n || row == full)) return expanded | kUnsettled;
    }
    if (lane == 0) write_not_synchronizing(b, k, n);
    __syncwarp();
    return expanded;
}

template <int CAP_BITS, int MAXN>
__global__ void __launch_bounds__(HashGeom<CAP_BITS, MAXN>::kWarps * 32)
    k_hash(const __grid_constant__ Batch b, int32_t *heavy_list, unsigned long long *heavy_count, unsigned long long *ticket)
{
    using G = HashGeom<CAP_BITS, MAXN>;
    constexpr int kHashCap = G::kCap;
    constexpr uint32_t kHashLimit = G::kLimit;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    HashWarp<CAP_BITS, MAXN> &W = reinterpret_cast<HashWarp<CAP_BITS, MAXN> *>(smem_raw)[warp];
    int64_t count;
    const int32_t *order;
    resolve_work(b, count, order);
    // generation 0 marks never-used slots; each automaton takes the next one
    for (int i = lane; i < kHashCap; i += 32) W.set[i] = 0u;
    __syncwarp();
    uint32_t gen = 0;
    unsigned long long expanded = 0;

    while (true) {
        unsigned long long pos = 0;
        if (lane == 0) pos = atomicAdd(ticket, 1ull);
        pos = __shfl_sync(kFull, pos, 0);
        if (pos >= (unsigned long long)count) break;
        const int64_t k = automaton_at(order, (int64_t)pos);
        const int n = automaton_n(b, k);
        const uint8_t *rec = b.maps + (size_t)k * 2u * (size_t)b.lstride;
        bool bad = n < 1 || n > G::kMaxN || n > b.lstride;
        uint64_t single = 0;
        uint32_t av = 0, bv = 0;
        if (!bad && lane < n) {
            av = rec[lane];
            bv = rec[b.lstride + lane];
            if (av >= (uint32_t)n || bv >= (uint32_t)n)
                bad = true;
            else
                single = ((uint64_t)(1u << av) << 32) | (1u << bv);
        }
        if (__any_sync(kFull, bad)) {
            if (lane == 0) {
                record_result(b, k, n, kLenInvalid);
                if (b.out_words)
                    for (int c = 0; c < b.word_stride; ++c) b.out_words[(size_t)k * b.word_stride + c] = 0ull;
                atomicOr(b.error, kErrInvalid);
                publish_result(b, k);
            }
            continue;
        }
        build_table<CAP_BITS, MAXN>(W, single, n, lane);
        next_generation<CAP_BITS, MAXN>(W, gen, lane);
        const uint32_t full = (1u << n) - 1u;
        if (lane == 0) W.queue[0] = (uint16_t)set_insert<CAP_BITS, MAXN>(W.set, full, gen);
        __syncwarp();
        // n = 1: the visited root is the only singleton, the search generates nothing new
        uint32_t head = 0, lvl_end = n > 1 ? 1u : 0u, tail = lvl_end, level = 0;
        int32_t len = kLenNonSync;
        uint32_t found = 0, found_letter = 0;
        bool heavy = false;
        while (head < lvl_end) {
            const uint32_t idx = head + (uint32_t)lane;
            const bool has = idx < lvl_end;
            uint32_t ya = 0, yb = 0;
            if (has) {
                const uint64_t t = lookup<CAP_BITS, MAXN>(W, W.set[W.queue[idx] & 0x7FFFu] & G::kSubsetMask);
                ya = (uint32_t)(t >> 32);
                yb = (uint32_t)t;
            }
            expanded += has ? 1u : 0u;
            const bool sa = has && is_singleton(ya), sb = has && is_singleton(yb);
            const unsigned smask = __ballot_sync(kFull, sa || sb);
            if (smask) {
                // the first singleton in queue order (lowest lane, a before b)
                const int fl = __ffs(smask) - 1;
                found = head + (uint32_t)fl;
                found_letter = (uint32_t)__shfl_sync(kFull, sa ? 0 : 1, fl);
                len = (int32_t)level + 1;
                break;
            }
            const int sa_slot = has ? set_insert<CAP_BITS, MAXN>(W.set, ya, gen) : -1;
            const int sb_slot = has ? set_insert<CAP_BITS, MAXN>(W.set, yb, gen) : -1;
            bool fa = sa_slot >= 0, fb = sb_slot >= 0;
            const unsigned ma = __ballot_sync(kFull, fa), mb = __ballot_sync(kFull, fb);
            const uint32_t added = (uint32_t)(__popc(ma) + __popc(mb));
            if (tail + added > kHashLimit) {
                heavy = true;
                break;
            }
            const unsigned lt = (1u << lane) - 1u;
            uint32_t p = tail + (uint32_t)(__popc(ma & lt) + __popc(mb & lt));
            if (!SBFS_CHECK(p + (fa ? 1u : 0u) + (fb ? 1u : 0u) <= kHashLimit, b.error)) fa = fb = false;
            if (fa) {
                W.queue[p] = (uint16_t)sa_slot;
                W.parent[p++] = (uint16_t)idx;
            }
            if (fb) {
                W.queue[p] = (uint16_t)(sb_slot | 0x8000);
                W.parent[p] = (uint16_t)idx;
            }
            tail += added;
            head = min(head + 32u, lvl_end);
            __syncwarp();
            if (head == lvl_end && tail > lvl_end) {
                lvl_end = tail;
                if (++level >= kHashLevelCap) {
                    heavy = true;
                    break;
                }
            }
        }
        __syncwarp();
        if (heavy) {
            // a long or wide search: backwards from the singletons, and if that is
            // wide too the CTA-wide kernel takes it from the start
            next_generation<CAP_BITS, MAXN>(W, gen, lane);
            const uint32_t r = inverse_search<CAP_BITS, MAXN>(b, k, n, av, bv, W, gen, lane);
            expanded += r & ~kUnsettled;
            if ((r & kUnsettled) && lane == 0) heavy_list[atomicAdd(heavy_count, 1ull)] = (int32_t)k;
            __syncwarp();
            continue;
        }
        if (lane == 0) {
            record_result(b, k, n, len);
            if (b.out_words) {
                // letters from the root: the entry at depth d + 1 holds letter d
                // (a word here has at most kHashLevelCap <= 64 letters)
                uint64_t w0 = 0;
                if (len > 0) {
                    if (found_letter) w0 |= 1ull << level;
                    uint32_t i = found;
                    for (int d = (int)level - 1; d >= 0; --d) {
                        if (W.queue[i] >> 15) w0 |= 1ull << d;
                        i = W.parent[i];
                    }
                }
                uint64_t *w = b.out_words + (size_t)k * (size_t)b.word_stride;
                w[0] = w0;
                for (int c = 1; c < b.word_stride; ++c) w[c] = 0ull;
            }
            publish_result(b, k);
        }
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) expanded += __shfl_down_sync(kFull, expanded, o);
    if (lane == 0 && b.expanded && expanded) atomicAdd(b.expanded, expanded);
}

// Counting sort of a hand-off list by n, largest first (one CTA): the
// persistent CTA-wide kernel then takes the longest searches first, and the
// short ones fill the SMs that free up (longest-processing-time order).
// With split, the sorted list is also described as two work ranges,
// {0, entries with n >= top_n} and {that, the rest}, so the entries below
// top_n can run in a launch sized for top_n - 1.
__global__ void __launch_bounds__(1024) k_sort_handoff(Batch b, const int32_t *list,
                                                       const unsigned long long *count, int32_t *out,
                                                       int top_n, unsigned long long *split)
{
    __shared__ unsigned int hist[SBFS_MAX_N + 2];
    const int tid = threadIdx.x;
    const int64_t cnt = (int64_t)*count;
    for (int i = tid; i < SBFS_MAX_N + 2; i += blockDim.x) hist[i] = 0u;
    __syncthreads();
    for (int64_t i = tid; i < cnt; i += blockDim.x) {
        const int n = min(max(automaton_n(b, list[i]), 0), SBFS_MAX_N + 1);
        atomicAdd(&hist[n], 1u);
    }
    __syncthreads();
    if (tid == 0) {
        unsigned int off = 0, top = 0;
        for (int n = SBFS_MAX_N + 1; n >= 0; --n) {
            const unsigned int c = hist[n];
            hist[n] = off;
            off += c;
            if (n == top_n) top = off;   // entries with n >= top_n
        }
        if (split) {
            split[0] = 0ull;
            split[1] = top;
            split[2] = top;
            split[3] = (unsigned long long)cnt - top;
        }
    }
    __syncthreads();
    for (int64_t i = tid; i < cnt; i += blockDim.x) {
        const int32_t k = list[i];
        const int n = min(max(automaton_n(b, k), 0), SBFS_MAX_N + 1);
        out[atomicAdd(&hist[n], 1u)] = k;
    }
}

constexpr int kMaxDevices = 16;

int current_device()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    return dev;
}

// The shared-memory cap and the resident CTAs per SM are set and measured once
// per device: the enqueue paths ask on every launch.
template <int CAP_BITS, int MAXN>
struct HashLaunch {
    static size_t smem() { return (size_t)HashGeom<CAP_BITS, MAXN>::kWarps * sizeof(HashWarp<CAP_BITS, MAXN>); }
    static cudaError_t prepare()
    {
        static std::atomic<int> done[kMaxDevices];
        const int dev = current_device();
        const bool cached = dev >= 0 && dev < kMaxDevices;
        if (cached && done[dev].load(std::memory_order_acquire)) return cudaSuccess;
        const cudaError_t e =
            cudaFuncSetAttribute(k_hash<CAP_BITS, MAXN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem());
        if (e == cudaSuccess && cached) done[dev].store(1, std::memory_order_release);
        return e;
    }
    static int per_sm()
    {
        static std::atomic<int> known[kMaxDevices];
        const int dev = current_device();
        const bool cached = dev >= 0 && dev < kMaxDevices;
        if (cached) {
            const int v = known[dev].load(std::memory_order_relaxed);
            if (v > 0) return v;
        }
        if (prepare() != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        int blocks = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_hash<CAP_BITS, MAXN>, HashGeom<CAP_BITS, MAXN>::kWarps * 32,
                                                          smem()) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        if (cached && blocks > 0) known[dev].store(blocks, std::memory_order_relaxed);
        return blocks;
    }
    static cudaError_t launch(int ctas, const Batch &b, int32_t *list, unsigned long long *count,
                              unsigned long long *ticket, cudaStream_t st)
    {
        cudaError_t e = prepare();
        if (e != cudaSuccess) return e;
        k_hash<CAP_BITS, MAXN><<<ctas, HashGeom<CAP_BITS, MAXN>::kWarps * 32, smem(), st>>>(b, list, count, ticket);
        return cudaGetLastError();
    }
};

}  // namespace

// size 1: 2048 hash slots per warp (1536 subsets), size 2: 4096 (3072 subsets);
// max_n: the largest n of the launch's automata (more than 20 states: size 2 only)
int hash_max_ctas_per_sm(int size, int max_n)
{
    if (max_n > 20) return size == 2 ? HashLaunch<12, 28>::per_sm() : 0;
    if (max_n > 16) return size == 2 ? HashLaunch<12, 20>::per_sm() : size == 1 ? HashLaunch<11, 20>::per_sm() : 0;
    return size == 2 ? HashLaunch<12, 16>::per_sm() : size == 1 ? HashLaunch<11, 16>::per_sm() : 0;
}

cudaError_t launch_sort_handoff(const Batch &b, const int32_t *list, const unsigned long long *count, int32_t *out,
                                int top_n, unsigned long long *split, cudaStream_t st)
{
    k_sort_handoff<<<1, 1024, 0, st>>>(b, list, count, out, top_n, split);
    return cudaGetLastError();
}

cudaError_t launch_hash(int size, int max_n, int ctas, const Batch &b, int32_t *heavy_list,
                        unsigned long long *heavy_count, unsigned long long *ticket, cudaStream_t st)
{
    if (ctas < 1 || !heavy_list || !heavy_count || max_n > SBFS_MAX_N) return cudaErrorInvalidValue;
    if (max_n > 20)
        return size == 2 ? HashLaunch<12, 28>::launch(ctas, b, heavy_list, heavy_count, ticket, st)
                         : cudaErrorInvalidValue;
    if (max_n > 16) {
        if (size == 1) return HashLaunch<11, 20>::launch(ctas, b, heavy_list, heavy_count, ticket, st);
        if (size == 2) return HashLaunch<12, 20>::launch(ctas, b, heavy_list, heavy_count, ticket, st);
        return cudaErrorInvalidValue;
    }
    if (size == 1) return HashLaunch<11, 16>::launch(ctas, b, heavy_list, heavy_count, ticket, st);
    if (size == 2) return HashLaunch<12, 16>::launch(ctas, b, heavy_list, heavy_count, ticket, st);
    return cudaErrorInvalidValue;
}

}  // namespace sbfs

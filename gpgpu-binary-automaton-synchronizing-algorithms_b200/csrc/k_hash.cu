// k_hash.cu -- power-set BFS of automata with 13..28 states (size classes 2,
// 3 and 4), one warp per automaton with its visited store, queue and image
// tables in shared memory.
//
// A random automaton of 13..20 states is settled after a few hundred subsets
// over ~11 levels (its shortest word is at most ~36 letters), so neither a
// 2^n-bit bitmap (128 KiB at n = 20) nor a 1024-thread CTA (k_cta.cu) pays for
// itself: the CTA's per-level barriers and round trips dominate.  Per warp:
//   * nibble tables: table[c][v] = (a-image << 32) | b-image of the states
//     4c..4c+3 selected by v, so both images of a subset are 4, 5 or 7 loads
//     (instances for n <= 16, 20 and 28);
//   * the visited store, 4 KB (n <= 16) or 8 KB.  After the first letter every
//     subset lies in the image of a or of b, so with the states relabelled by
//     image 2^rank(a) + 2^rank(b) bits tell them apart (ranks average 0.64 n):
//     a bitmap, one atomicOr per image.  95 % of random n = 20 and nearly all
//     smaller ones fit; the rest use the store as an open-addressed hash set,
//     atomicCAS with linear probing, to three quarters full.  With the hash set
//     for every automaton, whose 32 probe loops a step waits for, 200K n = 16
//     took 1.120 ms against 0.499 ms, 30K n = 20 0.602 against 0.329 ms;
//   * a level-ordered queue, retained for the word (GPGPU/CPU/CPU.cs:203-205):
//     subset, parent index and letter in 32 bits (a separate parent array
//     where they do not fit).
// 10.5 KB per warp for n <= 16 (21 warps per SM), 14.6 KB for n <= 20 (15).
// Sizes above 20 have a 16 KB store and room for 3072 subsets (6 warps per SM),
// of which the forward search takes 1024.
// The warp expands 32 subsets of the current level per step (level-
// synchronous, as GPGPU/CPU/SlimCPUUntweaked.cs:119-184), tests the images
// against the store, and appends the new ones compacted by ballots in queue
// order.  An automaton that needs more subsets than that (or kHashLevelCap
// levels) is tried backwards by the same warp (inverse_search below), which
// settles the slowly synchronizing families and the automata that never
// synchronize; one with a permutation letter and a letter merging at most one
// pair is tried backwards at once.  What is left -- wide both ways -- goes to
// one CTA per automaton (k_mid or k_cta, or k_wide above n = 20) through a list.  Random
// n = 17..20: 1.7 % of the automata pass 1536 subsets, 0.3 % pass 4096.
// 200K mixed n = 6..20 with 1 % Cerny automata: 3.04 ms with every such
// automaton on the CTA-wide kernel, 1.17 ms with the inverse search, 0.67 ms
// with the bitmap store.
#include <atomic>

#include "common.cuh"

namespace sbfs {
namespace {

constexpr uint32_t kHashLevelCap = 48;         // random n <= 20: at most ~40 levels
constexpr uint32_t kUnsettled = 1u << 31;

// SIZE 1: 1536 subsets per warp, SIZE 2: 3072.
template <int MAXN, int SIZE>
struct HashGeom {
    static constexpr uint32_t kLimit = 1536u << (SIZE - 1);      // subsets a warp keeps
    // Subsets the forward search keeps.  Above n = 20 a third of the room, which is
    // the backward search's: a warp takes 60 us per thousand of them, and k_wide
    // settles what is left in 10 to 50.  64 random n = 24 in one call 233 us with
    // 3072, 129 with 1536, 115 with 1024, 102 with 512; 3000 n = 21 298, 183, 178
    // and 210, 3000 n = 28 955, 855, 867 and 903.
    static constexpr uint32_t kForward = MAXN > 20 ? 1024u : kLimit;
    static constexpr int kIdxBits = 10 + SIZE;                   // of a queue index
    // words of the visited store: 2^15 bits for n <= 16, 2^16 for n <= 20 (twice that at SIZE 2)
    static constexpr int kWords = (MAXN <= 16 ? 1024 : 2048) << (SIZE - 1);
    static constexpr uint32_t kBits = 32u * kWords;
    // as a hash set it is filled to three quarters
    static constexpr uint32_t kSetLimit = kLimit < 3u * kWords / 4u ? kLimit : 3u * kWords / 4u;
    static constexpr int kSetShift = 32 - (MAXN <= 16 ? 9 : 10) - SIZE;
    // a queue entry is subset | parent << MAXN | letter-is-b << 31; sizes that
    // leave no room for the parent keep it in an array of its own
    static constexpr bool kPacked = MAXN + kIdxBits + 1 <= 32;
    static constexpr int kChunks = (MAXN + 3) / 4;               // nibble tables
    static constexpr int kEntries = 16 * kChunks;
    static constexpr uint32_t kMask = (1u << MAXN) - 1u;
    // warps per CTA: n <= 16 10.5 KB, three CTAs of seven per SM; n <= 20 14.6 KB,
    // three of five; SIZE 2 single
    static constexpr int kWarps = SIZE == 2 ? 1 : MAXN <= 16 ? 7 : 5;
    static constexpr int kCtas = SIZE == 2 ? 6 : 3;
};

template <int MAXN, int SIZE>
struct __align__(16) HashWarp {
    using G = HashGeom<MAXN, SIZE>;
    uint32_t store[G::kWords];    // visited: bitmap or hash set (0 = free slot)
    uint64_t table[G::kEntries];
    uint32_t queue[G::kLimit];
    uint16_t parent[G::kPacked ? 2 : G::kLimit];

    __device__ __forceinline__ uint32_t subset(uint32_t i) const { return queue[i] & G::kMask; }
    __device__ __forceinline__ uint32_t letter(uint32_t i) const { return queue[i] >> 31; }
    __device__ __forceinline__ uint32_t parent_of(uint32_t i) const
    {
        return G::kPacked ? (queue[i] >> MAXN) & ((1u << G::kIdxBits) - 1u) : parent[i];
    }
    __device__ __forceinline__ void push(uint32_t i, uint32_t x, uint32_t par, uint32_t letter)
    {
        if (G::kPacked) {
            queue[i] = x | (par << (MAXN < 32 ? MAXN : 0)) | (letter << 31);
        } else {
            queue[i] = x | (letter << 31);
            parent[i] = (uint16_t)par;
        }
    }
};

template <int MAXN, int SIZE>
__device__ __forceinline__ uint32_t set_slot(uint32_t x)
{
    return (x * 0x9E3779B1u) >> HashGeom<MAXN, SIZE>::kSetShift;
}

// Inserts subset x into the store as a hash set; false when it was there.
template <int MAXN, int SIZE>
__device__ __forceinline__ bool set_insert(HashWarp<MAXN, SIZE> &W, uint32_t x)
{
    using G = HashGeom<MAXN, SIZE>;
    uint32_t p = set_slot<MAXN, SIZE>(x);
    for (int probe = 0; probe < G::kWords; ++probe) {
        uint32_t v = W.store[p];
        if (v == 0u) {
            v = atomicCAS(&W.store[p], 0u, x);
            if (v == 0u) return true;
        }
        if (v == x) return false;
        p = (p + 1) & (G::kWords - 1);
    }
    return false;   // unreachable: the set is never more than ~3/4 full
}

// Zeroes the store's first `bits` bits (rounded up to 128).
template <int MAXN, int SIZE>
__device__ __forceinline__ void clear_store(HashWarp<MAXN, SIZE> &W, uint32_t bits, int lane)
{
    uint4 *s = reinterpret_cast<uint4 *>(W.store);
    for (uint32_t i = lane; i < (bits + 127u) / 128u; i += 32) s[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Nibble tables of one 64-bit mask pair per state (a's mask << 32 | b's): lane
// q < 32 passes state `label`'s, zero for labels past the last state.  The
// store serves as the staging area.
template <int MAXN, int SIZE>
__device__ __forceinline__ void build_table(HashWarp<MAXN, SIZE> &W, uint64_t mine, int label, int lane)
{
    using G = HashGeom<MAXN, SIZE>;
    uint64_t *stage = reinterpret_cast<uint64_t *>(W.store);
    __syncwarp();
    stage[label] = mine;
    __syncwarp();
#pragma unroll
    for (int pass = 0; pass < (G::kEntries + 31) / 32; ++pass) {
        const int e = lane + 32 * pass;
        const int c = e >> 4, v = e & 15;
        if (e < G::kEntries) {
            uint64_t acc = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if ((v >> j) & 1) acc |= stage[4 * c + j];
            W.table[e] = acc;
        }
    }
    __syncwarp();
}

// a's mask << 32 | b's mask of subset x
template <int MAXN, int SIZE>
__device__ __forceinline__ uint64_t lookup(const HashWarp<MAXN, SIZE> &W, uint32_t x)
{
    uint64_t t = W.table[x & 15u];
#pragma unroll
    for (int c = 1; c < HashGeom<MAXN, SIZE>::kChunks; ++c) t |= W.table[16 * c + ((x >> (4 * c)) & 15u)];
    return t;
}

__device__ __forceinline__ void write_not_synchronizing(const Batch &b, int64_t k, int n)
{
    record_result(b, k, n, kLenNonSync);
    if (b.out_words)
        for (int c = 0; c < b.word_stride; ++c) b.out_words[(size_t)k * b.word_stride + c] = 0ull;
    publish_result(b, k);
}

// The inverse search, for an automaton that the forward search gave up on, or
// that looks slow (lane q < n holds a(q) and b(q)).  A word w synchronizes iff
// w^-1(q) is the full set for some state q, and (cw)^-1(q) = c^-1(w^-1(q)): so a
// breadth-first search from the n singletons along preimages reaches the full
// set first at the length of the shortest word, and the parent chain from there
// spells the word from its first letter on.  It runs out without the full set
// iff the automaton is not synchronizing.
//
// The slowly synchronizing families (Cerny automata, a permutation plus one
// merge) have up to 2^n images of the full set but at most n(n-1)+1 preimages
// of singletons: C_20 is settled by 380 sets over 361 levels (tens of
// microseconds in one warp; all 2^20 forward subsets took a 1024-thread CTA
// 1.2 ms).  Their levels hold 1 to n sets; a random automaton whose forward
// search is wide passes n sets in a level at its fifth or sixth (9,000 random
// n = 13..28 with over 1536 images: none was settled before that).  So the
// search stops at the first level wider than n sets.
//
// Hundreds of levels of one to n sets are a serial chain.  A level of one set
// with one new preimage, found at the first probe (almost every level of a Cerny
// automaton), is run by all lanes alike on the same set: both preimages and both
// probes in registers, one branch, no ballot, shuffle or atomic on the way to the
// next level.  Other levels keep set i in lane i and give every image a lane of
// its own, one hash probe per lane.  C_28 (729 levels): 0.40 ms with every level
// on the lane-per-image form, 0.26 ms with a branch per case on the narrow one,
// 0.17 ms so.  (Looking up the next level's preimages of both while the probes
// run: 0.18 ms; the warp's instructions bound it, not the latencies.)
//
// Before giving up, pairs of states settle the wide automata that never
// synchronize: an automaton synchronizes iff every pair of its states is merged
// by some word.  Row q (lane q) collects the states that can be merged with q,
// preimages of the rows of a(q) and b(q), until nothing changes.
//
// Returns the images this lane looked up, with the top bit clear when the
// automaton is settled and set when it is left to the forward searches.
template <int MAXN, int SIZE>
__device__ __noinline__ uint32_t inverse_search(const Batch &b, int64_t k, int n, uint32_t av, uint32_t bv,
                                                HashWarp<MAXN, SIZE> &W, int lane)
{
    using G = HashGeom<MAXN, SIZE>;
    uint32_t expanded = 0;
    const uint32_t full = (1u << n) - 1u;
    // lane q: the states that a (b) sends to q
    uint64_t inv = 0;
    for (int q = 0; q < n; ++q) {
        const unsigned ia = __ballot_sync(kFull, lane < n && av == (uint32_t)q);
        const unsigned ib = __ballot_sync(kFull, lane < n && bv == (uint32_t)q);
        if (lane == q) inv = ((uint64_t)ia << 32) | ib;
    }
    build_table(W, inv, lane, lane);
    clear_store(W, G::kBits, lane);
    __syncwarp();
    uint32_t front = lane < n ? 1u << lane : 0u;   // set `lane` of the level
    if (front) {
        set_insert(W, front);
        W.push((uint32_t)lane, front, 0u, 0u);
    }
    __syncwarp();
    uint32_t head = 0, width = (uint32_t)n, tail = width, level = 0;
    uint32_t found = 0, found_letter = 0;
    bool hit = false, spent = true;   // spent: no set left to expand
    const uint32_t letter = (uint32_t)lane & 1u;
    while (true) {
        if (width == 1) {
            uint32_t x = __shfl_sync(kFull, front, 0);
            while (true) {
                const uint64_t t = lookup(W, x);
                const uint32_t ya = (uint32_t)(t >> 32), yb = (uint32_t)t;
                const uint32_t pa = set_slot<MAXN, SIZE>(ya), pb = set_slot<MAXN, SIZE>(yb);
                const uint32_t va = W.store[pa], vb = W.store[pb];
                __syncwarp();   // every lane has probed before the set is written
                const bool na = ya != 0u && va == 0u, nb = yb != 0u && vb == 0u && yb != ya;
                const bool sure = (va == 0u || va == ya || ya == 0u) && (vb == 0u || vb == yb || yb == 0u || yb == ya);
                if (!sure || na == nb || ya == full || yb == full || tail >= G::kSetLimit) break;
                x = na ? ya : yb;
                W.store[na ? pa : pb] = x;
                if (SBFS_CHECK(tail < G::kLimit, b.error)) W.push(tail, x, head, na ? 0u : 1u);
                __syncwarp();
                expanded += lane < 2 ? 1u : 0u;
                head = tail++;
                ++level;
            }
            front = x;
        }
        // image j of the level is letter j & 1 of set j >> 1: 32 images per pass, at most two passes
        uint32_t added = 0, next = 0;
        for (uint32_t base = 0; base < 2u * width; base += 32) {
            const uint32_t set = (base + (uint32_t)lane) >> 1;
            const uint32_t x = __shfl_sync(kFull, front, (int)set);
            uint32_t y = 0;
            if (set < width) {
                const uint64_t t = lookup(W, x);
                y = letter ? (uint32_t)t : (uint32_t)(t >> 32);
            }
            expanded += set < width ? 1u : 0u;
            const unsigned hits = __ballot_sync(kFull, y == full);
            if (hits) {
                const int fl = __ffs(hits) - 1;
                found = head + ((base + (uint32_t)fl) >> 1);
                found_letter = (uint32_t)fl & 1u;
                hit = true;
                break;
            }
            const bool fresh = y && set_insert(W, y);
            const unsigned m = __ballot_sync(kFull, fresh);
            if (m) {
                const uint32_t p = tail + added + (uint32_t)__popc(m & ((1u << lane) - 1u));
                if (fresh && p < G::kSetLimit) W.push(p, y, head + set, letter);   // (the limit ends the search)
                if (!(m & (m - 1u))) next = __shfl_sync(kFull, y, __ffs(m) - 1);
                added += (uint32_t)__popc(m);
            }
        }
        if (hit || added == 0) break;
        if (added > (uint32_t)n || tail + added > G::kSetLimit) {
            spent = false;
            break;
        }
        __syncwarp();
        front = added == 1 ? next : lane < (int)added ? W.subset(tail + (uint32_t)lane) : 0u;
        head = tail;
        tail += added;
        width = added;
        ++level;
    }
    __syncwarp();
    if (hit) {
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
                        acc |= (uint64_t)W.letter(i) << (d & 63u);
                        i = W.parent_of(i);
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
            const uint32_t grown = row | (uint32_t)(lookup(W, ra) >> 32) | (uint32_t)lookup(W, rb);
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

// What the forward search of one automaton ends with.
struct Forward {
    bool heavy;              // more subsets or levels than a warp keeps
    int32_t len;
    uint32_t level, found, found_letter;
};

// The warp expands 32 subsets of the current level per step.  BITS: the store
// is a bitmap, subset y at bit y when y < 2^ra and at base + (y >> shift)
// otherwise (a-images always are below 2^ra; see the kernel).
template <int MAXN, int SIZE, bool BITS>
__device__ __forceinline__ Forward forward_search(const Batch &b, int n, HashWarp<MAXN, SIZE> &W, uint32_t low_end,
                                                  uint32_t base, uint32_t shift, int lane,
                                                  unsigned long long &expanded)
{
    using G = HashGeom<MAXN, SIZE>;
    constexpr uint32_t kKeep = BITS || G::kForward < G::kSetLimit ? G::kForward : G::kSetLimit;
    Forward r{false, kLenNonSync, 0u, 0u, 0u};
    // n = 1: the visited root is the only singleton, the search generates nothing new
    uint32_t head = 0, lvl_end = n > 1 ? 1u : 0u, tail = lvl_end, level = 0;
    const unsigned lt = (1u << lane) - 1u;
    while (head < lvl_end) {
        const uint32_t idx = head + (uint32_t)lane;
        const bool has = idx < lvl_end;
        uint32_t ya = 0, yb = 0;
        if (has) {
            const uint64_t t = lookup(W, W.subset(idx));
            ya = (uint32_t)(t >> 32);
            yb = (uint32_t)t;
        }
        expanded += has ? 1u : 0u;
        const bool sa = has && is_singleton(ya), sb = has && is_singleton(yb);
        const unsigned smask = __ballot_sync(kFull, sa || sb);
        if (smask) {
            // the first singleton in queue order (lowest lane, a before b)
            const int fl = __ffs(smask) - 1;
            r.found = head + (uint32_t)fl;
            r.found_letter = (uint32_t)__shfl_sync(kFull, sa ? 0 : 1, fl);
            r.len = (int32_t)level + 1;
            break;
        }
        bool fa = false, fb = false;
        if (has) {
            if (BITS) {
                const uint32_t ib = yb < low_end ? yb : base + (yb >> shift);
                if (SBFS_CHECK(ya < G::kBits && ib < G::kBits, b.error)) {
                    const uint32_t ma = 1u << (ya & 31u), mb = 1u << (ib & 31u);
                    const uint32_t oa = atomicOr(&W.store[ya >> 5], ma);
                    const uint32_t ob = atomicOr(&W.store[ib >> 5], mb);
                    fa = !(oa & ma);
                    fb = !(ob & mb);
                }
            } else {
                fa = set_insert(W, ya);
                fb = set_insert(W, yb);
            }
        }
        const unsigned ma = __ballot_sync(kFull, fa), mb = __ballot_sync(kFull, fb);
        const uint32_t added = (uint32_t)(__popc(ma) + __popc(mb));
        if (tail + added > kKeep) {
            r.heavy = true;
            break;
        }
        uint32_t p = tail + (uint32_t)(__popc(ma & lt) + __popc(mb & lt));
        if (!SBFS_CHECK(p + (fa ? 1u : 0u) + (fb ? 1u : 0u) <= G::kLimit, b.error)) fa = fb = false;
        if (fa) W.push(p++, ya, idx, 0u);
        if (fb) W.push(p, yb, idx, 1u);
        tail += added;
        head = min(head + 32u, lvl_end);
        __syncwarp();
        if (head == lvl_end && tail > lvl_end) {
            lvl_end = tail;
            if (++level >= kHashLevelCap) {
                r.heavy = true;
                break;
            }
        }
    }
    __syncwarp();
    r.level = level;
    return r;
}

template <int MAXN, int SIZE>
__global__ void __launch_bounds__(HashGeom<MAXN, SIZE>::kWarps * 32, HashGeom<MAXN, SIZE>::kCtas)
    k_hash(const __grid_constant__ Batch b, int32_t *heavy_list, unsigned long long *heavy_count, int32_t *wide_list,
           unsigned long long *wide_count, unsigned long long *ticket)
{
    using G = HashGeom<MAXN, SIZE>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    HashWarp<MAXN, SIZE> &W = reinterpret_cast<HashWarp<MAXN, SIZE> *>(smem_raw)[warp];
    int64_t count;
    const int32_t *order;
    resolve_work(b, count, order);
    unsigned long long expanded = 0;

    while (true) {
        unsigned long long pos = 0;
        if (lane == 0) pos = atomicAdd(ticket, 1ull);
        pos = __shfl_sync(kFull, pos, 0);
        if (pos >= (unsigned long long)count) break;
        const int64_t k = automaton_at(order, (int64_t)pos);
        const int n = automaton_n(b, k);
        const uint8_t *rec = b.maps + (size_t)k * 2u * (size_t)b.lstride;
        bool bad = n < 1 || n > MAXN || n > b.lstride;
        uint32_t av = 0, bv = 0;
        if (!bad && lane < n) {
            av = rec[lane];
            bv = rec[b.lstride + lane];
            if (av >= (uint32_t)n || bv >= (uint32_t)n) bad = true;
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
        // New state labels, image of a first: A \ B | A and B | B \ A | the rest, with
        // A = a's image and B = b's.  Every subset but the root lies in A or in B:
        // as a label set it is below 2^ra, or a set of B, whose labels start at
        // |A \ B|: shifted down by that it is below 2^rb.  So 2^ra + 2^rb bits tell
        // all reachable subsets apart (n = 20: about 2^13.5 of 2^20, ranks
        // averaging 12.8).
        const uint32_t A = __reduce_or_sync(kFull, lane < n ? 1u << av : 0u);
        const uint32_t B = __reduce_or_sync(kFull, lane < n ? 1u << bv : 0u);
        const int ra = __popc(A), rb = __popc(B);
        bool tried = false;
        if (ra + rb >= 2 * n - 1 && n > 1) {
            // a permutation and a letter that merges at most one pair: the slow
            // families, whose forward search would be wide
            const uint32_t r = inverse_search(b, k, n, av, bv, W, lane);
            expanded += r & ~kUnsettled;
            if (!(r & kUnsettled)) continue;
            tried = true;
        }
        const uint32_t below = (1u << lane) - 1u;
        const bool in_a = (A >> lane) & 1u, in_b = (B >> lane) & 1u;
        int label = in_a ? (in_b ? __popc(A & ~B) + __popc(A & B & below) : __popc(A & ~B & below))
                         : (in_b ? ra + __popc(B & ~A & below) : __popc(A | B) + __popc(~(A | B) & below));
        if (lane >= n) label = lane;
        const int la = __shfl_sync(kFull, label, (int)av), lb = __shfl_sync(kFull, label, (int)bv);
        build_table(W, lane < n ? ((uint64_t)(1u << la) << 32) | (1u << lb) : 0ull, label, lane);
        const uint32_t full = (1u << n) - 1u;
        uint32_t low_end = 1u << ra, base = low_end, shift = (uint32_t)__popc(A & ~B);
        uint32_t bits = (B & ~A) ? low_end + (1u << rb) : low_end;
        if (bits > 1u << n) {   // a full-rank b beside a smaller a: the plain index is shorter
            base = shift = 0u;
            bits = 1u << n;
        }
        const bool fits = bits <= G::kBits;
        clear_store(W, fits ? bits : G::kBits, lane);
        __syncwarp();
        if (lane == 0) {
            W.push(0u, full, 0u, 0u);
            // the root comes back only through a permutation
            if (!fits) {
                set_insert(W, full);
            } else if (ra == n || rb == n) {
                const uint32_t i = full < low_end ? full : base + (full >> shift);
                W.store[i >> 5] = 1u << (i & 31u);
            }
        }
        __syncwarp();
        const Forward f = fits ? forward_search<MAXN, SIZE, true>(b, n, W, low_end, base, shift, lane, expanded)
                               : forward_search<MAXN, SIZE, false>(b, n, W, 0u, 0u, 0u, lane, expanded);
        if (f.heavy) {
            // a long or wide search: backwards from the singletons, and if that is
            // wide too the CTA-wide kernel takes it from the start
            uint32_t r = kUnsettled;
            if (!tried) {
                r = inverse_search(b, k, n, av, bv, W, lane);
                expanded += r & ~kUnsettled;
            }
            const bool wide = MAXN == 20 && wide_list && bits > kMidBits;
            if ((r & kUnsettled) && lane == 0)
                hand_off(b, wide ? wide_list : heavy_list, wide ? wide_count : heavy_count, k);
            __syncwarp();
            continue;
        }
        if (lane == 0) {
            record_result(b, k, n, f.len);
            if (b.out_words) {
                // letters from the root: the entry at depth d + 1 holds letter d
                // (a word here has at most kHashLevelCap <= 64 letters)
                uint64_t w0 = 0;
                if (f.len > 0) {
                    if (f.found_letter) w0 |= 1ull << f.level;
                    uint32_t i = f.found;
                    for (int d = (int)f.level - 1; d >= 0; --d) {
                        w0 |= (uint64_t)W.letter(i) << d;
                        i = W.parent_of(i);
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
template <int MAXN, int SIZE>
struct HashLaunch {
    static size_t smem() { return (size_t)HashGeom<MAXN, SIZE>::kWarps * sizeof(HashWarp<MAXN, SIZE>); }
    static cudaError_t prepare()
    {
        static std::atomic<int> done[kMaxDevices];
        const int dev = current_device();
        const bool cached = dev >= 0 && dev < kMaxDevices;
        if (cached && done[dev].load(std::memory_order_acquire)) return cudaSuccess;
        const cudaError_t e =
            cudaFuncSetAttribute(k_hash<MAXN, SIZE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem());
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
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_hash<MAXN, SIZE>, HashGeom<MAXN, SIZE>::kWarps * 32,
                                                          smem()) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        if (cached && blocks > 0) known[dev].store(blocks, std::memory_order_relaxed);
        return blocks;
    }
    static cudaError_t launch(int ctas, const Batch &b, int32_t *list, unsigned long long *count, int32_t *wide_list,
                              unsigned long long *wide_count, unsigned long long *ticket, cudaStream_t st)
    {
        cudaError_t e = prepare();
        if (e != cudaSuccess) return e;
        k_hash<MAXN, SIZE><<<ctas, HashGeom<MAXN, SIZE>::kWarps * 32, smem(), st>>>(b, list, count, wide_list,
                                                                                    wide_count, ticket);
        return cudaGetLastError();
    }
};

}  // namespace

// size 1: 1536 subsets per warp and a store of 1024 words (n <= 16) or 2048, size 2:
// twice that; as a hash set three quarters of the store's words.
// max_n: the largest n of the launch's automata (more than 20 states: size 2 only).
// What a warp does not settle goes to heavy_list, or to wide_list (not null where
// max_n is 18..20) if its images need more than kMidBits.
int hash_max_ctas_per_sm(int size, int max_n)
{
    if (max_n > 20) return size == 2 ? HashLaunch<28, 2>::per_sm() : 0;
    if (max_n > 16) return size == 2 ? HashLaunch<20, 2>::per_sm() : size == 1 ? HashLaunch<20, 1>::per_sm() : 0;
    return size == 2 ? HashLaunch<16, 2>::per_sm() : size == 1 ? HashLaunch<16, 1>::per_sm() : 0;
}

cudaError_t launch_hash(int size, int max_n, int ctas, const Batch &b, int32_t *heavy_list,
                        unsigned long long *heavy_count, int32_t *wide_list, unsigned long long *wide_count,
                        unsigned long long *ticket, cudaStream_t st)
{
    if (ctas < 1 || !heavy_list || !heavy_count || max_n > SBFS_MAX_N) return cudaErrorInvalidValue;
    if (max_n > 20)
        return size == 2 ? HashLaunch<28, 2>::launch(ctas, b, heavy_list, heavy_count, nullptr, nullptr, ticket, st)
                         : cudaErrorInvalidValue;
    if (max_n > 16) {
        if (size == 1)
            return HashLaunch<20, 1>::launch(ctas, b, heavy_list, heavy_count, wide_list, wide_count, ticket, st);
        if (size == 2)
            return HashLaunch<20, 2>::launch(ctas, b, heavy_list, heavy_count, wide_list, wide_count, ticket, st);
        return cudaErrorInvalidValue;
    }
    if (size == 1) return HashLaunch<16, 1>::launch(ctas, b, heavy_list, heavy_count, nullptr, nullptr, ticket, st);
    if (size == 2) return HashLaunch<16, 2>::launch(ctas, b, heavy_list, heavy_count, nullptr, nullptr, ticket, st);
    return cudaErrorInvalidValue;
}

}  // namespace sbfs

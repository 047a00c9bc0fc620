// k_lane.cu -- power-set BFS with one automaton per lane (n <= 14).
//
// Each lane runs the sequential BFS of GPGPU/CPU/SlimCPU4bits.cs:214-306 on its
// own automaton: pop subsets, look up both images in its nibble table
// (entry = a-image << 16 | b-image, SlimCPU4bits.cs:122-206), test-and-set them
// in its visited bitmap, append the new ones, advance the level when the
// current level is used up (SlimCPUUntweaked.cs:126-130,160-164), stop at the
// first singleton generated (:151-155).  All 32 lanes of a warp do this in
// lockstep on 32 different automata.
//
// Shared memory is lane-interleaved: element e of lane l's bitmap, table and
// queue lives at [e][l], so every lane-private access of a warp touches 32
// different banks.
//
// Shared memory bounds the resident warps, and those the speed (1M n = 12:
// 0.71 ms at 6 warps per SM, 0.58 at 8, 0.51 at 10 of the same kernel), so the
// bitmap is kept small (n > 8).  After the first letter every subset lies in the
// image of a or of b.  With the states relabelled A \ B, A and B, B \ A, the rest
// (A, B the images), a subset of A is a number below 2^rank(a), and one of B is,
// shifted down by |A \ B|, one below 2^rank(b): 2^rank(a) + 2^rank(b) bits tell
// all of them apart.  Ranks average 0.65 n; 1536 bits serve 98 % of random n = 12
// (512 B of one bit per subset became 192 B, 7 warps per SM became 10), 3072 and
// 6400 bits over 99 % at n = 13 and 14 (4 became 6, 2 became 3).  The other
// automata take bitmaps from a pool of the warp's, in the order in which they came,
// and when that is used up the whole column (bitmap, table, ring) of a lane that
// does not search.  Batches of such automata alone, one permutation and one random
// map: half of the lanes search, 200,000 n = 12 in 0.72 ms and 100,000 n = 13 in
// 0.75 (with the pool alone 2.02 and 4.44, with a bitmap of 2^n bits per lane 0.95
// and 0.99).
// Relabelling changes neither the order of the search nor its words.  1M n = 12
// device-resident: 0.592 -> 0.472 ms; 500K n = 14: 1.158 -> 0.760 ms; a Verify call
// on 2^21 n = 13: 2.25 -> 1.95 ms.
//
// The queue is a ring of R entries holding only the live
// frontier (current level remainder + next level); with words requested each
// entry carries the letters of the word that reaches it (bit NMAX + d =
// letter d, 1 = b), so a word needs no parent pointers or retained history.
//
// Each iteration a lane takes up to kStep (4) subsets of its current level and
// looks up their eight images: more independent work per step hides the
// shared-memory latencies that one warp's dependent chain exposes at 7 warps
// per SM (2 -> 4 subsets: 0.64 -> 0.56 ms per 10^6 automata at n = 12; 6 and 8
// were slower again; at ten warps per SM two take 0.556, three 0.521 and four
// 0.515 ms).  A singleton among them ends the search (no singleton
// is visited before the first one is generated, so it needs no bitmap test).
// Otherwise the eight images are test-and-set with shared-memory atomicOr, issued
// back to back and kept in program order by the hardware for a repeated
// address, and the fresh ones are appended in queue order (first subset's a, b,
// then the second's), as the sequential loop would.
//
// Two rare cases leave the per-lane search: a frontier wider than R, and (with
// words) a word longer than 32 - NMAX letters.  Such an automaton is abandoned
// and appended to the launch's escalation list.  So is, once the batch is
// handed out, the work of a warp with at most `tail_k` lanes still searching.
// A warp that has no lane work left (no new automata, every lane idle) owns
// its whole shared-memory region again and takes escalated automata from that
// list one at a time, solving each with all 32 lanes: a level-synchronous
// search over a linear queue that holds every subset at most once (2^n
// entries, so it cannot overflow), with parent pointers for the word, the
// nibble table in registers read by warp shuffles, and a linear bitmap updated
// with shared-memory atomics.  Claims never wait (see claim_escalated): every
// escalated automaton is solved in the launch that escalated it.
//
// Lanes that finish wait until `refill_k` lanes of the warp are idle; then the
// warp writes their results and loads new automata for all of them in one
// pass, so the per-automaton set-up (record load, table build, bitmap clear)
// runs with many lanes active instead of one.
//
// Instances: NMAX = 8 and 12 for size classes 0 and 1; 13 and 14 for uniform
// batches of that n (a fourth nibble chunk, and words of up to (NMAX - 1)^2 =
// 144 or 169 letters -- three 64-bit words -- in
// the whole-warp search).
#include <algorithm>

#include "common.cuh"

namespace sbfs {
namespace {

// (kLent: waiting, and its column serves its partner's search)
constexpr int kActive = 0, kDone = 1, kEscalate = 2, kIdle = 3, kHeld = 4, kWaiting = 5, kLent = 6;
constexpr int kStep = 4;   // subsets a lane expands per step (their 2 * kStep images are tested together)
// Warps of a launched CTA when `warps` are asked for (n > 8: one, see kOneWarp),
// and CTAs of that many that the registers must allow for
__host__ __device__ constexpr int lane_cta_warps(int nmax, int warps) { return nmax <= 8 ? warps : 1; }
__host__ __device__ constexpr int lane_min_ctas(int nmax) { return nmax <= 8 ? 4 : 11; }
// At n = 13 and 14 fewer warps fit on an SM (six, three), and six subsets per
// step hide more of each warp's latency: 2^21 automata at n = 14 4.83 -> 4.64 ms,
// the n = 13 streamed kernel 2.19 -> 2.09 ms (eight: no better than six; measured
// with four and two warps, one bit per subset and lane)
constexpr int kStepWide = 6;

__host__ __device__ constexpr int low_bit4(int v)
{
    return (v & 1) ? 0 : (v & 2) ? 1 : (v & 4) ? 2 : 3;
}

template <int NMAX>
struct LaneGeom {
    static constexpr int kBitmapWords = (1 << NMAX) / 32;   // whole-warp search: one bit per subset
    // Per-lane search: words of a lane's visited bitmap, and the pool of
    // bitmaps that serves the warp's lanes whose automaton needs more (half of one
    // bit per subset, or a pair of such halves).  The pool takes what the resident
    // warps leave of shared memory (10, 6 and 3 per SM at n = 12, 13 and 14): with
    // one bitmap at n = 12 the automata that need it, the longer searches among
    // them, queued up.
    static constexpr bool kRelabel = NMAX > 8;
    static constexpr int kLaneWords = NMAX <= 8 ? 8 : NMAX <= 12 ? 48 : NMAX == 13 ? 96 : 200;
    static constexpr int kHalfWords = kRelabel ? kBitmapWords / 2 : 0;
    static constexpr int kHalves = NMAX <= 8 ? 0 : NMAX <= 12 ? 6 : NMAX == 13 ? 2 : 8;
    static constexpr int kPoolWords = kHalves * kHalfWords;
    static constexpr uint32_t kAllHalves = (1u << kHalves) - 1u;
    static constexpr uint32_t kBorrowed = 1u << 31;   // beside the halves a lane holds: its partner's column
    // One warp per CTA, so that its region starts at a constant address and every
    // access of a step is a lane's offset plus an immediate (1M n = 12: 0.514 ->
    // 0.490 ms at ten warps per SM).  n <= 8 keeps more warps than that allows.
    static constexpr bool kOneWarp = NMAX > 8;
    // Steps between two looks at the lanes' states while automata are left to hand
    // out.  A look costs three ballots and their branches: 1M n = 12 0.507 ms with
    // one step, 0.471 with two, three or four alike.
    static constexpr int kRounds = NMAX > 8 ? 2 : 1;
    static constexpr int kChunks = (NMAX + 3) / 4;
    static constexpr int kTable = kChunks * 16;
    static constexpr uint32_t kMask = (1u << NMAX) - 1u;
    static constexpr int kWordMax = 32 - NMAX;   // letters an entry can carry
    static constexpr int kWordU64 = ((NMAX - 1) * (NMAX - 1) + 63) / 64;   // words of the whole-warp search
};

template <int NMAX>
__device__ __forceinline__ uint32_t lane_image(const uint32_t *tb, uint32_t x)
{
    uint32_t t = tb[(x & 15u) * 32];
    if (LaneGeom<NMAX>::kChunks > 1) t |= tb[(16 + ((x >> 4) & 15u)) * 32];
    // (x carries a word's letters from bit NMAX on)
    if (LaneGeom<NMAX>::kChunks > 2) t |= tb[(32 + ((x >> 8) & 15u)) * 32];
    if (LaneGeom<NMAX>::kChunks > 3) t |= tb[(48 + ((x >> 12) & ((1u << (NMAX > 12 ? NMAX - 12 : 0)) - 1u))) * 32];
    return t;
}

// Nibble-table entry v of chunk c (a-image << 16 | b-image of the states
// 4c + i for the set bits i of v), read from the record.
template <int NMAX>
__device__ __forceinline__ uint32_t table_entry(const uint8_t *rec, int lstride, int n, int c, int v)
{
    uint32_t t = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int st = 4 * c + i;
        if (((v >> i) & 1) && st < n)
            t |= (1u << (__ldg(rec + st) + 16)) | (1u << __ldg(rec + lstride + st));
    }
    return t;
}

// The lanes beside those of m: 2i for 2i + 1 and 2i + 1 for 2i.
__device__ __forceinline__ unsigned partners(unsigned m)
{
    return ((m & 0x55555555u) << 1) | ((m >> 1) & 0x55555555u);
}

// v << (c & 31)
__device__ __forceinline__ uint32_t shl_wrap(uint32_t v, uint32_t c) { return __funnelshift_l(0u, v, c); }

// The bytes of a word that hold the first `left` of its four states (all when
// left >= 4, none when left <= 0).
__device__ __forceinline__ uint32_t keep_bytes(int left)
{
    return left >= 4 ? ~0u : left <= 0 ? 0u : (1u << (8 * left)) - 1u;
}

// Every byte of w (0..15) replaced by byte w of the table L.
__device__ __forceinline__ uint32_t map_bytes(uint32_t w, const uint32_t (&L)[4])
{
    const uint32_t t = w & 0x07070707u;
    const uint32_t sel = __byte_perm(t | (t >> 4), 0u, 0x4420);
    const uint32_t low = __byte_perm(L[0], L[1], sel), high = __byte_perm(L[2], L[3], sel);
    uint32_t m;   // 0xFF where bit 3 is set (selector bit 3: the sign of the byte, spread)
    asm("prmt.b32 %0, %1, 0, 0xBA98;" : "=r"(m) : "r"(w << 4));
    return (high & m) | (low & ~m);
}

// Four-byte pieces of one map of n states at p (any alignment); bytes past the
// map are whatever follows it.
template <int CHUNKS>
__device__ __forceinline__ void load_map(const uint8_t *p, int n, uint32_t (&w)[CHUNKS])
{
    const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3u);
    const uint32_t *q = reinterpret_cast<const uint32_t *>(p - off);
    uint32_t v[CHUNKS + 1];
#pragma unroll
    for (int c = 0; c <= CHUNKS; ++c) v[c] = 4 * c < n + (int)off ? __ldg(q + c) : 0u;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) w[c] = __funnelshift_r(v[c], v[c + 1], 8u * off);
}

// The same byte by byte, both maps, into words that are zero.
template <int NMAX>
__device__ __forceinline__ void load_bytes(const uint8_t *rec, int lstride, int n, uint32_t (&aw)[(NMAX + 3) / 4],
                                           uint32_t (&bw)[(NMAX + 3) / 4])
{
#pragma unroll
    for (int c = 0; c < (NMAX + 3) / 4; ++c)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (4 * c + j < n) {
                aw[c] |= (uint32_t)__ldg(rec + 4 * c + j) << (8 * j);
                bw[c] |= (uint32_t)__ldg(rec + lstride + 4 * c + j) << (8 * j);
            }
}

// Automaton k's maps, four images per word.  Aligned words whatever the record
// stride: a first or last record whose words would reach outside the batch is
// read byte by byte.
template <int NMAX, bool STREAM>
__device__ __forceinline__ void load_maps(const Batch &b, int64_t k, int n, int64_t count, bool valid,
                                          uint32_t (&aw)[(NMAX + 3) / 4], uint32_t (&bw)[(NMAX + 3) / 4])
{
    constexpr int CH = (NMAX + 3) / 4;
    const uint8_t *rec = b.maps + (size_t)k * 2u * (size_t)b.lstride;
#pragma unroll
    for (int c = 0; c < CH; ++c) aw[c] = bw[c] = 0u;
    if (!valid) return;
    if (NMAX <= 8 && !STREAM) {
        // aligned words or bytes: shorter than words at any alignment (10^6 n = 8
        // 201 -> 195 us; the streamed form would spill)
        if (((reinterpret_cast<uintptr_t>(rec) | (uintptr_t)b.lstride) & 3u) == 0) {
#pragma unroll
            for (int c = 0; c < CH; ++c)
                if (4 * c < n) {
                    aw[c] = __ldg(reinterpret_cast<const uint32_t *>(rec) + c);
                    bw[c] = __ldg(reinterpret_cast<const uint32_t *>(rec + b.lstride) + c);
                }
        } else {
            load_bytes<NMAX>(rec, b.lstride, n, aw, bw);
        }
        return;
    }
    // an order array may point anywhere in the batch: only its own record is known to be there
    const uint8_t *first = b.order ? rec : b.maps;
    const uint8_t *end = b.order ? rec + 2 * b.lstride : b.maps + (size_t)count * 2u * (size_t)b.lstride;
    const uintptr_t lo = reinterpret_cast<uintptr_t>(rec) & ~(uintptr_t)3;
    const uintptr_t hi = (reinterpret_cast<uintptr_t>(rec + b.lstride + n) + 3) & ~(uintptr_t)3;
    if (lo >= reinterpret_cast<uintptr_t>(first) && hi <= reinterpret_cast<uintptr_t>(end)) {
        load_map<CH>(rec, n, aw);
        load_map<CH>(rec + b.lstride, n, bw);
        return;
    }
    load_bytes<NMAX>(rec, b.lstride, n, aw, bw);
}

// Claims the next escalated automaton of the launch for a warp with no lane
// work left, or returns -1.  A claim is one atomicAdd on the claim counter and
// one atomicCAS on the claimed slot, raced against the slot's writer (which
// stores with atomicCAS too): if the slot is still empty (0) the claimer marks it
// abandoned (-1) and stops, and the writer, finding it abandoned, keeps the
// automaton and solves it itself once it runs out of lane work.  Nothing ever
// waits for another warp.
__device__ int64_t claim_escalated(int32_t *list, unsigned long long capacity, unsigned long long *claim,
                                   unsigned long long &slot)
{
    slot = atomicAdd(claim, 1ull);
    if (slot >= capacity) return -1;
    const int32_t prev = atomicCAS(list + slot, 0, -1);
    return (int64_t)prev - 1;   // an empty slot: -1
}

// One automaton (n <= NMAX) solved by the whole warp inside its region of
// `region_words` shared words (>= 2^NMAX / 32 + 2^NMAX).  Queue entry:
// subset | parent index << NMAX | letter << 2*NMAX (letter 1 = b).  `expanded`:
// the subsets this lane expanded; the word is lane 0's.
struct WarpFound {
    int32_t len;
    uint32_t expanded;
    uint64_t w0, w1, w2;
};

template <int NMAX, bool WORDS>
__device__ __forceinline__ WarpFound warp_search(const uint8_t *rec, int lstride, int n, uint32_t *region, int lane,
                                                 int *error)
{
    uint32_t expanded = 0;
    using G = LaneGeom<NMAX>;
    constexpr int BW = G::kBitmapWords;
    uint32_t *bm = region;        // linear bitmap
    uint32_t *q = region + BW;    // linear queue, 2^NMAX entries
    // chunks 0 and 1 in lanes 0-15 / 16-31 of t01, chunk 2 (and 3) likewise in t23
    const uint32_t t01 = table_entry<NMAX>(rec, lstride, n, lane >> 4, lane & 15);
    const uint32_t t23 = G::kChunks > 3   ? table_entry<NMAX>(rec, lstride, n, 2 + (lane >> 4), lane & 15)
                         : G::kChunks > 2 ? table_entry<NMAX>(rec, lstride, n, 2, lane & 15)
                                          : 0u;
    for (int w = lane; w < BW; w += 32) bm[w] = 0u;
    __syncwarp();
    const uint32_t full = (1u << n) - 1u;
    if (lane == 0) {
        bm[full >> 5] = 1u << (full & 31u);
        q[0] = full;
    }
    __syncwarp();
    // n = 1: the visited root is the only singleton (see the per-lane set-up)
    uint32_t head = 0, lvl_end = n > 1 ? 1u : 0u, tail = lvl_end, level = 0;
    int32_t len = kLenNonSync;
    uint32_t found = 0, found_letter = 0;
    while (true) {
        const uint32_t idx = head + (uint32_t)lane;
        const bool has = idx < lvl_end;
        const uint32_t x = has ? (q[idx] & G::kMask) : 0u;
        uint32_t t = __shfl_sync(kFull, t01, (int)(x & 15u)) | __shfl_sync(kFull, t01, 16 + (int)((x >> 4) & 15u));
        if (G::kChunks > 2) t |= __shfl_sync(kFull, t23, (int)((x >> 8) & 15u));
        if (G::kChunks > 3) t |= __shfl_sync(kFull, t23, 16 + (int)((x >> 12) & 15u));
        const uint32_t ya = t >> 16, yb = t & 0xFFFFu;
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
        bool fa = false, fb = false;
        if (has && SBFS_CHECK((ya >> 5) < (uint32_t)BW && (yb >> 5) < (uint32_t)BW, error)) {
            fa = !(atomicOr(&bm[ya >> 5], 1u << (ya & 31u)) & (1u << (ya & 31u)));
            fb = !(atomicOr(&bm[yb >> 5], 1u << (yb & 31u)) & (1u << (yb & 31u)));
        }
        const unsigned ma = __ballot_sync(kFull, fa), mb = __ballot_sync(kFull, fb);
        const unsigned lt = (1u << lane) - 1u;
        uint32_t pos = tail + (uint32_t)(__popc(ma & lt) + __popc(mb & lt));
        const uint32_t par = idx << NMAX;
        // every subset enters the queue at most once: 2^NMAX entries never overflow
        if (fa && SBFS_CHECK(pos < (1u << NMAX), error)) q[pos] = ya | par;
        pos += fa ? 1u : 0u;
        if (fb && SBFS_CHECK(pos < (1u << NMAX), error)) q[pos] = yb | par | (1u << (2 * NMAX));
        tail += (uint32_t)(__popc(ma) + __popc(mb));
        head = min(head + 32u, lvl_end);
        __syncwarp();
        if (head == lvl_end) {
            if (tail == lvl_end) break;   // no new subset: not synchronizing
            lvl_end = tail;
            ++level;
        }
    }
    WarpFound r{len, expanded, 0ull, 0ull, 0ull};
    // at most (NMAX - 1)^2 letters: 2 words at n = 12, 3 at n = 13
    static_assert(G::kWordU64 <= 3, "words of at most 192 letters");
    if (WORDS && lane == 0 && len > 0) {
        // letters from the root: entry at depth d + 1 holds letter d
        auto set = [&](uint32_t d) {
            if (d < 64) r.w0 |= 1ull << d;
            else if (d < 128) r.w1 |= 1ull << (d - 64);
            else if (G::kWordU64 > 2) r.w2 |= 1ull << (d - 128);
        };
        if (found_letter) set(level);
        uint32_t i = found;
        for (int d = (int)level - 1; d >= 0; --d) {
            const uint32_t e = q[i];
            if ((e >> (2 * NMAX)) & 1u) set((uint32_t)d);
            i = (e >> NMAX) & G::kMask;
        }
    }
    return r;
}

// Automaton k searched by the whole warp, and its results.  Returns the subsets
// this lane expanded.
template <int NMAX, bool WORDS, bool STREAM>
__device__ __forceinline__ uint32_t warp_solve_body(const Batch &b, int64_t k, uint32_t *region, int lane,
                                                    const LaneStream &ls, unsigned long long slot)
{
    using G = LaneGeom<NMAX>;
    const int n = automaton_n(b, k);
    const uint8_t *rec = b.maps + (size_t)k * 2u * (size_t)b.lstride;
    const WarpFound r = warp_search<NMAX, WORDS>(rec, b.lstride, n, region, lane, b.error);
    if (lane == 0) {
        record_result(b, k, n, r.len);
        if (WORDS) {
            uint64_t *w = b.out_words + (size_t)k * (size_t)b.word_stride;
            w[0] = r.w0;
            if (b.word_stride > 1) w[1] = r.w1;
            if (G::kWordU64 > 2) {
                if (b.word_stride > 2) w[2] = r.w2;
                for (int c = 3; c < b.word_stride; ++c) w[c] = 0ull;
            } else {
                for (int c = 2; c < b.word_stride; ++c) w[c] = 0ull;
            }
        }
        if (STREAM && ls.escal_out) {
            // streamed batches: the host patches escalated automata from here
            // (if the chunk still had searches out after these results were stored, its
            // copy, which comes after the last of them, takes them along)
            __threadfence();
            const int c = ls.chunk_of(k);
            const bool early = *(volatile unsigned int *)(ls.chunk_done + c) < (unsigned)ls.chunk_size(c, b.count);
            EscalResult e;
            e.k = early ? kEscalInChunk : k;
            e.len = r.len;
            e.pad = 0;
            e.word[0] = r.w0;
            e.word[1] = r.w1;
            e.word[2] = r.w2;
            ls.escal_out[slot] = e;
        }
        publish_result(b, k);
    }
    __syncwarp();
    return r.expanded;
}

// (a call of its own in the streamed kernel, which has two places for it)
template <int NMAX, bool WORDS>
__device__ __noinline__ uint32_t warp_solve_call(const Batch &b, int64_t k, uint32_t *region, int lane,
                                                 const LaneStream &ls, unsigned long long slot)
{
    return warp_solve_body<NMAX, WORDS, true>(b, k, region, lane, ls, slot);
}

template <int NMAX, bool WORDS, bool STREAM>
__device__ __forceinline__ uint32_t warp_solve(const Batch &b, int64_t k, uint32_t *region, int lane,
                                               const LaneStream &ls, unsigned long long slot)
{
    return STREAM ? warp_solve_call<NMAX, WORDS>(b, k, region, lane, ls, slot)
                  : warp_solve_body<NMAX, WORDS, false>(b, k, region, lane, ls, slot);
}

// Words of a warp's shared-memory region: the lanes' bitmaps, tables and rings
// and the pool, or the whole-warp search's bitmap and queue.
template <int NMAX>
__host__ __device__ constexpr size_t region_words(int ring)
{
    using G = LaneGeom<NMAX>;
    const size_t lanes = (size_t)(G::kLaneWords + G::kTable + ring) * 32 + G::kPoolWords;
    const size_t whole = (size_t)G::kBitmapWords + ((size_t)1 << NMAX);
    return lanes > whole ? lanes : whole;
}

// Streamed batches: `add` outcomes of chunk c are written (and fenced); whoever completes the
// chunk tells the host that its lengths and words can be copied out.
__device__ __forceinline__ void tell_chunk(const LaneStream &ls, int64_t c, unsigned add, int64_t count)
{
    if ((int64_t)(atomicAdd(ls.chunk_done + c, add) + add) == ls.chunk_size(c, count)) {
        __threadfence_system();
        *(volatile unsigned int *)(ls.host_flag + c) = 1u;
    }
}

template <int NMAX, bool WORDS, bool STREAM>
__global__ void __launch_bounds__(lane_cta_warps(NMAX, 8) * 32, lane_min_ctas(NMAX))
    k_lane(const __grid_constant__ Batch b, int ring, int refill_k, int tail_k, int32_t *escal_list,
           unsigned long long escal_capacity, unsigned long long *escal_count, unsigned long long *escal_claim,
           unsigned long long *ticket, const __grid_constant__ LaneStream ls)
{
    using G = LaneGeom<NMAX>;
    constexpr int LW = G::kLaneWords;
    constexpr int T = G::kTable;
    extern __shared__ __align__(16) uint32_t smem[];
    const int lane = threadIdx.x & 31;
    const int warp = G::kOneWarp ? 0 : threadIdx.x >> 5;
    uint32_t *base = smem + (size_t)warp * region_words<NMAX>(ring);
    uint32_t *const own = base + lane;           // the lane's bitmap, own[w * 32]
    uint32_t *tb = base + LW * 32 + lane;        // tb[e * 32]
    uint32_t *rq = base + (LW + T) * 32 + lane;  // rq[i * 32]
    uint32_t *const pool = base + (LW + T + ring) * 32;
    const uint32_t rmask = (uint32_t)ring - 1u;

    int64_t count;
    const int32_t *order;
    resolve_work(b, count, order);

    int state = kIdle;
    int64_t k = -1;
    int n = 0;
    uint32_t head = 0, tail = 0, lvl_end = 0, level = 0;
    int32_t res_len = kLenNonSync;
    uint32_t res_word = 0;
    bool more = true;
    unsigned long long expanded = 0;   // whole-warp searches
    uint32_t steps_expanded = 0;       // this lane's own searches
    uint32_t solved = 0;               // lengths it found
    unsigned long long hslot = 0;   // escalation slot of a held automaton
    // The lane's visited bitmap: bit y of subset y below low_end, bit index0 +
    // (y >> shift) of the others (b-images only), word w at bm[w * stride].
    uint32_t *bm = own;
    uint32_t stride = 32, low_end = 1u << NMAX, index0 = 0, shift = 0;
    uint32_t held = 0;              // halves of the pool this lane's bitmap is in
    uint32_t pool_free = G::kAllHalves;   // halves nobody holds (alike in every lane)
    unsigned away = 0;              // lanes that only another's end can start: lent, or without a bitmap
    int enough = refill_k;          // idle lanes that trigger a refill, as a share of those not away
    uint32_t pass = 0, since = 0;   // passes that asked for the pool; the one this lane came in
    uint32_t checks = 0;
    int ready_upto = -1;            // streamed chunks known to be on the device
    unsigned waiting = 0;           // streamed: lanes whose records are not there yet (set at the refill pass)
    // Streamed outcomes that this warp has not told of yet: of the chunk its next
    // ticket is in (`cur`; past the last one once all are handed out) and of the one before
    int cur = 0;
    unsigned own_cur = 0, own_old = 0;

    while (true) {
        // ---- phase: finish waiting lanes, load new automata -----------------
        // no new automata: once at most `tail_k` lanes still search, the warp
        // hands their automata to the whole-warp search instead of finishing
        // them at a few lanes' pace (the launch's tail)
        if (!more && tail_k > 0) {
            const unsigned active = __ballot_sync(kFull, state == kActive);
            if (state == kActive && __popc(active) <= tail_k) state = kEscalate;
        }
        const unsigned not_active = __ballot_sync(kFull, state != kActive);
        // (streamed: lanes that wait for records ask for a look at the chunk flags,
        // one trip to L2, at every eighth check only)
        const unsigned served = not_active & ~(STREAM ? waiting | away : away);
        if (not_active == kFull || (STREAM && waiting && (++checks & 7u) == 0u) ||
            (__popc(served) >= enough && (more || __any_sync(kFull, state == kDone || state == kEscalate)))) {
            const bool outcome = state == kDone || state == kEscalate;
            if (state == kDone) {
                if (STREAM) {
                    record_result(b, k, n, res_len);
                } else {
                    // (counted at the kernel's end: 10^6 n = 5 127 -> 123 us)
                    store_result(b, k, n, res_len);
                    solved += res_len >= 0;
                }
                if (WORDS) {
                    uint64_t *w = b.out_words + (size_t)k * (size_t)b.word_stride;
                    w[0] = res_len > 0 ? (uint64_t)res_word : 0ull;
                    for (int c = 1; c < b.word_stride; ++c) w[c] = 0ull;
                }
                publish_result(b, k);
            }
            const unsigned esc = __ballot_sync(kFull, state == kEscalate);
            if (esc) {
                unsigned long long pos = 0;
                const int leader = __ffs(esc) - 1;
                if (lane == leader) pos = atomicAdd(escal_count, (unsigned long long)__popc(esc));
                pos = __shfl_sync(kFull, pos, leader);
                if (state == kEscalate) {
                    // a slot a drained warp already gave up on: solve this one ourselves later
                    const unsigned long long slot = pos + __popc(esc & ((1u << lane) - 1u));
                    const int32_t prev = SBFS_CHECK(slot < escal_capacity, b.error)
                                             ? atomicCAS(escal_list + slot, 0, (int32_t)k + 1)
                                             : -1;
                    state = prev == 0 ? kIdle : kHeld;
                    hslot = slot;
                }
            }
            if (STREAM && !G::kOneWarp) {
                // n <= 8: told at once (with the counts below the kernel spills: 10^6
                // n = 8 end to end 0.672 ms against 0.657)
                const unsigned om = __ballot_sync(kFull, outcome);
                if (outcome) {
                    __threadfence();   // this lane's results before its count
                    const int c = ls.chunk_of(k);
                    const unsigned grp = __match_any_sync(om, c);
                    if (lane == __ffs(grp) - 1) tell_chunk(ls, c, (unsigned)__popc(grp), count);
                }
            } else if (STREAM) {
                const int c = ls.chunk_of(k);
                own_cur += (unsigned)__popc(__ballot_sync(kFull, outcome && c == cur));
                if (__any_sync(kFull, outcome && c != cur)) {
                    own_old += (unsigned)__popc(__ballot_sync(kFull, outcome && c == cur - 1));
                    // (two chunks and more behind the tickets: told one by one)
                    const bool late = outcome && c < cur - 1;
                    const bool last = own_old && !__any_sync(kFull, c == cur - 1 && (state == kActive || state >= kWaiting));
                    if (__any_sync(kFull, late) || last) {
                        __threadfence();   // every lane's results before the counts
                        __syncwarp();
                        if (late) tell_chunk(ls, c, 1u, count);
                        if (last && lane == 0) tell_chunk(ls, cur - 1, own_old, count);
                        if (last) own_old = 0;
                    }
                }
            }
            if (state == kDone || state == kEscalate) state = kIdle;
            if (G::kRelabel) {
                if (state != kActive) held = 0;
                pool_free = G::kAllHalves & ~__reduce_or_sync(kFull, held);
                const unsigned lent = partners(__ballot_sync(kFull, held & G::kBorrowed));
                if (state == kLent && !((lent >> lane) & 1u)) state = kWaiting;
            }
            const unsigned idle = __ballot_sync(kFull, state == kIdle);
            bool fresh = false;   // the lane just received an automaton
            if (more && idle) {
                unsigned long long got = 0;
                const int leader = __ffs(idle) - 1;
                if (lane == leader) got = atomicAdd(ticket, (unsigned long long)__popc(idle));
                got = __shfl_sync(kFull, got, leader);
                if (got + __popc(idle) >= (unsigned long long)count) more = false;
                if (state == kIdle) {
                    const unsigned long long pos = got + __popc(idle & ((1u << lane) - 1u));
                    if (pos < (unsigned long long)count) {
                        k = automaton_at(order, (int64_t)pos);
                        n = automaton_n(b, k);
                        state = kActive;
                        fresh = true;
                        since = 0;
                    }
                }
                if (STREAM && G::kOneWarp) {
                    const int next = more ? ls.chunk_of((int64_t)(got + __popc(idle))) : ls.chunk_of(count - 1) + 1;
                    if (next != cur) {
                        // The tickets enter a new chunk: what the warp still owes to the
                        // chunk just left is told with its last search there, so a chunk
                        // costs a warp one fence and one atomic, and the chunk is complete
                        // no later for it.  (Told at every pass with an outcome, with the
                        // chunk by division: 2^21 n = 13 end to end 1.66 ms against 1.61,
                        // 500,000 n = 14 0.94 against 0.845, 10^6 n = 12 0.90 against 0.88.)
                        const bool skip = next != cur + 1;   // others took a whole chunk meanwhile
                        const bool done = !__any_sync(kFull, (state == kActive || state >= kWaiting) && ls.chunk_of(k) == cur);
                        if (own_old || (own_cur && (skip || done))) {
                            __threadfence();   // every lane's results before the counts
                            __syncwarp();
                            if (lane == 0 && own_old) tell_chunk(ls, cur - 1, own_old, count);
                            if (lane == 0 && own_cur && (skip || done)) tell_chunk(ls, cur, own_cur, count);
                            if (skip || done) own_cur = 0;
                        }
                        own_old = own_cur;
                        own_cur = 0;
                        cur = next;
                    }
                }
            }
            // every lane that just received an automaton sets it up, and so does one
            // that waited (for the pool, or for its records)
            bool setup = fresh || state == kWaiting;
            if (STREAM) {
                // Streamed batch: the records handed out must have arrived.  A warp with
                // other lanes still searching does not wait for them: stopping those
                // would hold back the results of the chunk before (1M n = 12 end to
                // end: 1.17 ms with every such wait blocking, now that the kernel is
                // faster than the link).
                const int c = setup ? ls.chunk_of(k) : -1;
                // (most passes know already that all chunks handed out are there)
                const int c_last = !G::kOneWarp || cur > ready_upto ? (int)__reduce_max_sync(kFull, (unsigned)(c + 1)) - 1 : -1;
                if (c_last > ready_upto) {
                    const int c_first = (int)__reduce_min_sync(kFull, setup ? (unsigned)c : ~0u);
                    const bool busy = __any_sync(kFull, state == kActive && !fresh);
                    // With nothing to search the warp waits (bounded: wait_polls polls
                    // about 0.2 us apart), solving escalated automata meanwhile
                    for (int polls = 0;;) {
                        if (lane == 0)
                            while (ready_upto < c_last &&
                                   *(volatile const unsigned int *)(ls.chunk_ready + ready_upto + 1))
                                ++ready_upto;
                        ready_upto = __shfl_sync(kFull, ready_upto, 0);
                        if (busy || ready_upto >= c_first) break;
                        if (polls >= ls.wait_polls) {
                            if (lane == 0) atomicOr(b.error, kErrWait);
                            ready_upto = c_last;
                            break;
                        }
                        int64_t e = -1;
                        unsigned long long slot = 0;
                        if (lane == 0 && *(volatile unsigned long long *)escal_claim <
                                             *(volatile unsigned long long *)escal_count)
                            e = claim_escalated(escal_list, escal_capacity, escal_claim, slot);
                        e = __shfl_sync(kFull, e, 0);
                        slot = __shfl_sync(kFull, slot, 0);
                        if (e >= 0) {
                            expanded += warp_solve<NMAX, WORDS, STREAM>(b, e, base, lane, ls, slot);
                        } else {
                            ++polls;
                            __nanosleep(200);
                        }
                    }
                    __threadfence();
                }
                const bool absent = setup && c > ready_upto;
                if (absent) {
                    setup = fresh = false;
                    state = kWaiting;
                }
                waiting = __ballot_sync(kFull, absent);
            }
            if (__any_sync(kFull, setup)) {
                uint32_t words = 0, halves = 0;   // bitmap words, and pool halves they take
                if (setup) {
                    state = kActive;
                    bool bad = (n < 1 || n > NMAX || n > b.lstride);
                    const int nn = bad ? 1 : n;
                    uint32_t aw[G::kChunks], bw[G::kChunks];   // four images each, 15 past the last state
                    load_maps<NMAX, STREAM>(b, k, nn, count, !bad, aw, bw);
                    {
                        uint32_t high = 0;   // top bits: an image that is no state
                        const uint32_t over = (0x80u - (uint32_t)nn) * 0x01010101u;
#pragma unroll
                        for (int c = 0; c < G::kChunks; ++c) {
                            const uint32_t keep = keep_bytes(nn - 4 * c);
                            aw[c] &= keep;
                            bw[c] &= keep;
                            high |= aw[c] | (aw[c] + over) | bw[c] | (bw[c] + over);
                            aw[c] |= 0x0F0F0F0Fu & ~keep;
                            bw[c] |= 0x0F0F0F0Fu & ~keep;
                        }
                        bad |= (high & 0x80808080u) != 0u;
                    }
                    uint32_t ra = 0, rb = 0, a_only = 0;
                    bool b_only = false;
                    if (G::kRelabel) {
                        // bit 2q: q is an image of a, bit 2q + 1: of b
                        uint32_t z = 0;
#pragma unroll
                        for (int c = 0; c < G::kChunks; ++c)
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                z |= shl_wrap(1u, (aw[c] * 2u) >> (8 * j)) | shl_wrap(2u, (bw[c] * 2u) >> (8 * j));
                        z &= (1u << (2 * nn)) - 1u;
                        const uint32_t za = z & 0x55555555u, zb = (z >> 1) & 0x55555555u;
                        ra = (uint32_t)__popc(za);
                        rb = (uint32_t)__popc(zb);
                        a_only = (uint32_t)__popc(za & ~zb);
                        b_only = (zb & ~za) != 0u;
                        // new labels, a byte per state: A \ B | A and B | B \ A | the rest.  One
                        // counter per group, at byte (in A) + 2 * (in B) of `next`
                        uint32_t next = (a_only + rb) | (ra << 16) | (a_only << 24);
                        uint32_t L[4] = {0u, 0u, 0u, 16u << 24};   // 16: the label of image 15, none
#pragma unroll
                        for (int st = 0; st < NMAX; ++st) {
                            const uint32_t at = (st < 2 ? z << (3 - 2 * st) : z >> (2 * st - 3)) & 24u;
                            L[st / 4] = __byte_perm(L[st / 4], next >> at, 0x3210 ^ ((st & 3 ^ 4) << (4 * (st & 3))));
                            next += 1u << at;
                        }
#pragma unroll
                        for (int c = 0; c < G::kChunks; ++c) {
                            const uint32_t la = map_bytes(aw[c], L), lb = map_bytes(bw[c], L);
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (4 * c + j < NMAX)
                                    own[((L[c] >> (8 * j)) & 0xFFu) * 32u] =
                                        shl_wrap(0x10000u, la >> (8 * j)) | (shl_wrap(1u, lb >> (8 * j)) & 0xFFFFu);
                        }
                    }
#pragma unroll
                    for (int c = 0; c < G::kChunks; ++c) {
                        uint32_t s[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int st = 4 * c + j;
                            if (G::kRelabel) {
                                s[j] = st < NMAX ? own[st * 32] : 0u;
                            } else {
                                const uint32_t av = (aw[c] >> (8 * j)) & 15u, bv = (bw[c] >> (8 * j)) & 15u;
                                s[j] = st < nn ? (1u << (av + 16)) | (1u << bv) : 0u;
                            }
                        }
                        // table[c*16 + v] = OR of s[j] over the set bits j of v
                        uint32_t t[16];
                        t[0] = 0u;
#pragma unroll
                        for (int v = 1; v < 16; ++v) t[v] = t[v & (v - 1)] | s[low_bit4(v)];
#pragma unroll
                        for (int v = 0; v < 16; ++v) tb[(c * 16 + v) * 32] = t[v];
                    }
                    if (bad) {
                        // written (and counted) at the next refill pass
                        atomicOr(b.error, kErrInvalid);
                        state = kDone;
                        res_len = kLenInvalid;
                        res_word = 0;
                    } else if (n == 1 || (G::kRelabel && ra + rb == 2u * (uint32_t)n)) {
                        // the root is the only singleton and it is visited, so the
                        // search never generates a new one: not synchronizing, as in
                        // GPGPU/CPU/SlimCPUUntweaked.cs:149-157 (and the singleton-first
                        // test below, which relies on no singleton being visited, is
                        // never reached).  Nor do two permutations generate anything but
                        // the root, and would ask for the largest bitmap to find that out.
                        state = kDone;
                        res_len = kLenNonSync;
                        res_word = 0;
                        steps_expanded += n > 1;
                    } else {
                        uint32_t bits = 1u << n;
                        index0 = shift = 0;
                        low_end = 1u << NMAX;
                        if (G::kRelabel) {
                            const uint32_t need = (1u << ra) + (b_only ? 1u << rb : 0u);
                            if (need < bits) {
                                bits = need;
                                low_end = index0 = 1u << ra;
                                shift = a_only;
                            }
                        }
                        words = (bits + 31u) / 32u;
                        halves = words <= (uint32_t)LW ? 0u : words <= (uint32_t)G::kHalfWords ? 1u : 2u;
                        bm = own;
                        stride = 32;
                    }
                }
                if (G::kRelabel) {
                    // The pool goes to the lanes that need it, in the order in which they
                    // came.  (Out of order, a lane could wait until the end of the
                    // batch: a streamed batch's first chunk was then complete only with
                    // its last.)
                    unsigned want = __ballot_sync(kFull, halves != 0u);
                    if (want) ++pass;
                    if (halves != 0u && since == 0u) since = pass;
                    for (; want; ) {
                        const uint32_t first = __reduce_min_sync(kFull, (want >> lane) & 1u ? since : ~0u);
                        const int l = __ffs(__ballot_sync(kFull, ((want >> lane) & 1u) && since == first)) - 1;
                        const uint32_t pairs = pool_free & (pool_free >> 1) & 0x55555555u;
                        const bool two = __shfl_sync(kFull, halves, l) == 2u;
                        // one half: of a broken pair if there is one
                        const uint32_t lone = pool_free & ~(pairs * 3u);
                        const uint32_t from = two ? pairs : lone ? lone : pool_free;
                        if (!from) break;
                        const int at = __ffs(from) - 1;
                        const uint32_t take = (two ? 3u : 1u) << at;
                        want &= ~(1u << l);
                        pool_free &= ~take;
                        uint32_t *const part = pool + at * G::kHalfWords;
                        for (int w = lane; w < (two ? 2 : 1) * G::kHalfWords; w += 32) part[w] = 0u;
                        __syncwarp();
                        if (lane == l) {
                            bm = part;
                            stride = 1;
                            held = take;
                        }
                    }
                    if (want) {
                        // Batches of permutations and other large ranks need more bitmaps
                        // than the pool has.  A lane that it leaves out takes its partner's
                        // column (bitmap, table and ring: 160, 288 and 520 words at n = 12,
                        // 13 and 14, for 128, 256 and 512) when that lane does not search:
                        // of two left out the one that came first.
                        const bool out = halves != 0u && !held;
                        const uint32_t key = out ? since : state == kActive || state == kDone ? 0u : ~0u;
                        const uint32_t other = __shfl_xor_sync(kFull, key, 1);
                        const bool borrow = out && words <= (uint32_t)(LW + T + ring) &&
                                            (other > since || (other == since && !(lane & 1)));
                        if (out && !borrow) state = kWaiting;
                        if (partners(__ballot_sync(kFull, borrow)) >> lane & 1u) state = state == kWaiting ? kLent : state;
                        __syncwarp();   // every lane is done with its own column
                        if (borrow) {
                            bm = base + (lane ^ 1);
                            held = G::kBorrowed;
                            for (uint32_t w = 0; w < words; ++w) bm[w * 32] = 0u;
                        }
                    }
                    if (halves != 0u) words = 0;
                }
                if (G::kRelabel) {
                    const uint32_t most = __reduce_max_sync(kFull, words);
#pragma unroll 8
                    for (uint32_t w = 0; w < most; ++w)
                        if (setup) own[w * 32] = 0u;
                } else if (setup) {
#pragma unroll
                    for (int w = 0; w < LW; ++w) own[w * 32] = 0u;
                }
                if (setup && state == kActive) {
                    const uint32_t full = (1u << n) - 1u;
                    // the root comes back only through a permutation, and then every
                    // subset keeps its plain index
                    if (index0 == 0) bm[(full >> 5) * (G::kRelabel ? stride : 32u)] = 1u << (full & 31u);
                    rq[0] = full;
                    head = 0;
                    tail = 1;
                    lvl_end = 1;
                    level = 0;
                }
            }
            if (G::kRelabel) {
                // lanes away neither count as idle nor are waited for
                away = __ballot_sync(kFull, state >= kWaiting) & ~(STREAM ? waiting : 0u);
                enough = max(1, refill_k - ((refill_k * __popc(away)) >> 5));
            }
            if (__ballot_sync(kFull, state == kActive) == 0u) {
                // no lane is searching: the region is free for whole-warp searches,
                // first of the automata this warp kept; then, with no new automata
                // either, of escalated ones while any can be claimed.
                unsigned kept = __ballot_sync(kFull, state == kHeld);
                if (G::kRelabel)
                    for (; kept; kept &= kept - 1u) {
                        const int64_t e = __shfl_sync(kFull, k, __ffs(kept) - 1);
                        const unsigned long long slot = __shfl_sync(kFull, hslot, __ffs(kept) - 1);
                        expanded += warp_solve<NMAX, WORDS, STREAM>(b, e, base, lane, ls, slot);
                    }
                if (state == kHeld) state = kIdle;
                // (an outcome decided during set-up -- n = 1, a malformed record -- is
                // written by the next refill pass: that pass comes before leaving)
                const bool last = !more && !__any_sync(kFull, state == kDone || state == kEscalate);
                // (n <= 8: one loop for both.  With two copies of the search 10^6 n = 8
                // took 196 us, not 191, and n = 7 176, not 170; 500,000 n = 14 take
                // 766 with one, 759 with two.)
                while (kept || last) {
                    int64_t e = -1;
                    unsigned long long slot = 0;
                    if (!G::kRelabel && kept) {
                        e = __shfl_sync(kFull, k, __ffs(kept) - 1);
                        slot = __shfl_sync(kFull, hslot, __ffs(kept) - 1);
                        kept &= kept - 1u;
                    } else {
                        if (lane == 0) e = claim_escalated(escal_list, escal_capacity, escal_claim, slot);
                        e = __shfl_sync(kFull, e, 0);
                        slot = __shfl_sync(kFull, slot, 0);
                    }
                    if (e < 0) break;
                    expanded += warp_solve<NMAX, WORDS, STREAM>(b, e, base, lane, ls, slot);
                }
                if (last) break;
                continue;
            }
        }

        // ---- up to kStep expansions per active lane ----------------------------
        // (kRounds of them between two looks at the lanes while new automata are
        // left; in the tail one, so that the few lanes left are seen at once)
#pragma unroll 1
        for (int round = 0; round < G::kRounds; ++round) {
            if (state == kActive && (round == 0 || more)) {
                // a lane with fewer than kStep subsets left in the level expands its
                // first one again in the spare places: those copies' images are
                // already visited by the time they are tested
                constexpr int P = NMAX >= 13 ? kStepWide : kStep;
                const uint32_t take = min(lvl_end - head, (uint32_t)P);
                uint32_t e[P];
#pragma unroll
                for (int i = 0; i < P; ++i)
                    e[i] = (i == 0 || (uint32_t)i < take) ? rq[((head + (uint32_t)i) & rmask) * 32] : e[0];
                head += take;
                steps_expanded += take;
                uint32_t y[2 * P], hi[2 * P];
                // entries carry the word that reaches them: the parent's letters,
                // plus letter `level` = b for the b-images (an entry holds 32 - NMAX
                // letters; at level >= 32 - NMAX a fresh image escalates instead)
                const uint32_t lb = (WORDS && level < (uint32_t)G::kWordMax) ? 1u << (level + NMAX) : 0u;
#pragma unroll
                for (int i = 0; i < P; ++i) {
                    const uint32_t t = lane_image<NMAX>(tb, e[i]);
                    y[2 * i] = t >> 16;
                    y[2 * i + 1] = t & 0xFFFFu;
                    hi[2 * i] = e[i];
                    hi[2 * i + 1] = e[i] | lb;
                }
                // no singleton is ever visited (the search stops at the first one), so
                // a singleton image ends the search without a bitmap test
                bool hit = false;
#pragma unroll
                for (int c = 0; c < 2 * P; ++c) hit |= is_singleton(y[c]);
                if (hit) {
                    int sc = 0;   // the first one in queue order
#pragma unroll
                    for (int c = 2 * P - 1; c >= 0; --c)
                        if (is_singleton(y[c])) sc = c;
                    state = kDone;
                    res_len = (int32_t)level + 1;
                    uint32_t es = e[0];
#pragma unroll
                    for (int i = 1; i < P; ++i)
                        if ((sc >> 1) == i) es = e[i];
                    res_word = WORDS ? ((es >> NMAX) | ((uint32_t)(sc & 1) << level)) : 0u;
                } else {
                    // test-and-set in queue order: a subset met twice in this step is
                    // fresh only the first time (same-address atomics keep program order)
                    uint32_t old[2 * P], at[2 * P];
#pragma unroll
                    for (int c = 0; c < 2 * P; ++c) {
                        // an a-image is always below low_end
                        at[c] = !G::kRelabel || (c & 1) == 0 || y[c] < low_end ? y[c] : index0 + (y[c] >> shift);
                        old[c] = SBFS_CHECK((at[c] >> 5) < (held & G::kBorrowed ? (uint32_t)(LW + T + ring)
                                                        : held               ? (uint32_t)(__popc(held) * G::kHalfWords)
                                                                             : (uint32_t)LW),
                                            b.error)
                                     ? atomicOr(&bm[(at[c] >> 5) * (G::kRelabel ? stride : 32u)], 1u << (at[c] & 31u))
                                     : ~0u;
                    }
                    bool any = false;
#pragma unroll
                    for (int c = 0; c < 2 * P; ++c) {
                        if (!(old[c] & (1u << (at[c] & 31u)))) {
                            rq[(tail & rmask) * 32] = WORDS ? y[c] | (hi[c] & ~G::kMask) : y[c];
                            ++tail;
                            any = true;
                        }
                    }
                    // more live entries than ring slots (the oldest were overwritten), or
                    // a word longer than an entry carries: the whole-warp search takes over
                    if (tail - head > (uint32_t)ring || (WORDS && any && level >= (uint32_t)G::kWordMax)) {
                        state = kEscalate;
                    } else if (head == lvl_end) {
                        if (tail == lvl_end) {
                            state = kDone;
                            res_len = kLenNonSync;
                        } else {
                            lvl_end = tail;
                            ++level;
                        }
                    }
                }
            }
            __syncwarp();
        }
    }
    expanded += steps_expanded;
    for (int o = 16; o; o >>= 1) expanded += __shfl_down_sync(kFull, expanded, o);
    if (lane == 0 && b.expanded) atomicAdd(b.expanded, expanded);
    if (!STREAM) {
        solved = __reduce_add_sync(kFull, solved);
        if (lane == 0 && b.synchronizing && solved) atomicAdd(b.synchronizing, (unsigned long long)solved);
    }
}

template <int NMAX>
size_t smem_for(int warps, int ring)
{
    return (size_t)warps * region_words<NMAX>(ring) * sizeof(uint32_t);
}

template <int NMAX, bool WORDS>
cudaError_t launch_t(int warps, int ring, int refill_k, int tail_k, int ctas, const Batch &b, int32_t *escal_list,
                     unsigned long long escal_capacity, unsigned long long *escal_count,
                     unsigned long long *escal_claim, unsigned long long *ticket, const LaneStream &ls,
                     cudaStream_t st)
{
    // a grid of `ctas` CTAs of `warps` warps, as CTAs of one warp where the kernel wants those
    const int w = lane_cta_warps(NMAX, warps);
    const size_t smem = smem_for<NMAX>(w, ring);
    // the streamed form's bookkeeping is compiled out of the resident-batch kernel
    auto kernel = ls.chunk_done ? k_lane<NMAX, WORDS, true> : k_lane<NMAX, WORDS, false>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
    if (e != cudaSuccess) return e;
    kernel<<<ctas * (warps / w), w * 32, smem, st>>>(b, ring, refill_k, tail_k, escal_list, escal_capacity,
                                                     escal_count, escal_claim, ticket, ls);
    return cudaGetLastError();
}

}  // namespace

// CTAs of `warps` warps that an SM holds (n > 8: groups of that many one-warp CTAs).
int lane_max_ctas_per_sm(int nmax, int warps, int ring)
{
    if (nmax > 14 || warps < 1) return 0;
    const void *k = nmax <= 8    ? (const void *)k_lane<8, true, false>
                    : nmax <= 12 ? (const void *)k_lane<12, true, false>
                    : nmax == 13 ? (const void *)k_lane<13, true, false>
                                 : (const void *)k_lane<14, true, false>;
    const int w = lane_cta_warps(nmax, warps);
    const size_t smem = nmax <= 8    ? smem_for<8>(w, ring)
                        : nmax <= 12 ? smem_for<12>(w, ring)
                        : nmax == 13 ? smem_for<13>(w, ring)
                                     : smem_for<14>(w, ring);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, w * 32, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return blocks * w / warps;
}

// Streamed batches: after the chunk copies, the escalated automata's results
// (solved late, after their chunk may already have been copied) are stored
// straight into the host's mapped output.
__global__ void k_escal_patch(const EscalResult *r, const unsigned long long *count, int32_t *len, uint64_t *words,
                              int ws)
{
    const int64_t n = (int64_t)*count;
    // a store is a packet on the link: 16 bytes of a word at once where they are aligned
    // (10^6 n = 12 end to end 0.880 -> 0.858 ms)
    const bool pairs = (ws & 1) == 0 && (reinterpret_cast<uintptr_t>(words) & 15u) == 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const EscalResult e = r[i];
        if (e.k == kEscalInChunk) continue;
        if (len) len[e.k] = e.len;
        if (words) {
            uint64_t *w = words + (size_t)e.k * (size_t)ws;
            if (pairs)
                for (int j = 0; j < ws; j += 2)
                    *reinterpret_cast<ulonglong2 *>(w + j) =
                        make_ulonglong2(j < 3 ? e.word[j] : 0ull, j + 1 < 3 ? e.word[j + 1] : 0ull);
            else
                for (int j = 0; j < ws; ++j) w[j] = j < 3 ? e.word[j] : 0ull;
        }
    }
}

cudaError_t launch_escal_patch(const EscalResult *r, const unsigned long long *count, int32_t *len, uint64_t *words,
                               int ws, int sm_count, cudaStream_t st)
{
    k_escal_patch<<<2 * sm_count, 256, 0, st>>>(r, count, len, words, ws);
    return cudaGetLastError();
}

cudaError_t launch_lane(int nmax, int warps, int ring, int refill_k, int tail_k, int ctas, const Batch &b,
                        int32_t *escal_list, unsigned long long escal_capacity, unsigned long long *escal_count,
                        unsigned long long *escal_claim, unsigned long long *ticket, const LaneStream &ls,
                        cudaStream_t st)
{
    if ((ring & (ring - 1)) || ring < 8 || warps < 1 || warps > 8 || ctas < 1 || refill_k < 1 || refill_k > 32 ||
        tail_k < 0 || tail_k > 32)
        return cudaErrorInvalidValue;
    if (ls.chunk_done && (ls.chunk_log2 < 5 || ls.chunk_log2 > 30 || b.order || b.range_dev))
        return cudaErrorInvalidValue;
    const bool words = b.out_words != nullptr;
    if (nmax <= 8)
        return words ? launch_t<8, true>(warps, ring, refill_k, tail_k, ctas, b, escal_list, escal_capacity,
                                         escal_count, escal_claim, ticket, ls, st)
                     : launch_t<8, false>(warps, ring, refill_k, tail_k, ctas, b, escal_list, escal_capacity,
                                          escal_count, escal_claim, ticket, ls, st);
    if (nmax <= 12)
        return words ? launch_t<12, true>(warps, ring, refill_k, tail_k, ctas, b, escal_list, escal_capacity,
                                          escal_count, escal_claim, ticket, ls, st)
                     : launch_t<12, false>(warps, ring, refill_k, tail_k, ctas, b, escal_list, escal_capacity,
                                           escal_count, escal_claim, ticket, ls, st);
    if (nmax == 13)
        return words ? launch_t<13, true>(warps, ring, refill_k, tail_k, ctas, b, escal_list, escal_capacity,
                                          escal_count, escal_claim, ticket, ls, st)
                     : launch_t<13, false>(warps, ring, refill_k, tail_k, ctas, b, escal_list, escal_capacity,
                                           escal_count, escal_claim, ticket, ls, st);
    if (nmax == 14)
        return words ? launch_t<14, true>(warps, ring, refill_k, tail_k, ctas, b, escal_list, escal_capacity,
                                          escal_count, escal_claim, ticket, ls, st)
                     : launch_t<14, false>(warps, ring, refill_k, tail_k, ctas, b, escal_list, escal_capacity,
                                           escal_count, escal_claim, ticket, ls, st);
    return cudaErrorInvalidValue;
}

}  // namespace sbfs

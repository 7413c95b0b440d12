// K4: per-partition pilot search; persistent warps, one partition per warp at a time,
// taken from a shared work queue.
//
// Replaces search.comp:31-175 on the bucket-ordered keys and the schedule of K3c.
//
// Order and result follow the reference exactly:
//   * buckets are searched by descending size, and by descending bucket index
//     among equal sizes (sort_sum.comp:156-172, search.comp:145-166);
//   * for each bucket the pilot counter k starts at 0; k is rejected when two
//     keys of the bucket hash to the same slot (search.comp:44-70); otherwise
//     the smallest offset o in [0, ps) whose slots (h_i + o) mod ps are all free
//     is taken (search.comp:72-103 under lockstep execution), the slots are
//     marked, and pilot = o + ps * k (search.comp:122);
//   * pilots are stored bucket-major at pilots[b * partitions + p]
//     (search.comp:170-174); empty buckets get 0.
//
// Work queue: every warp takes the next global partition from one counter, so
// partitions of very different cost (and of different key sets in a batched
// build) spread over the SMs without CTA-level tail imbalance.
//
// Offset search: the occupancy bitmap is kept twice in a row (bits [ps, 2 ps)
// repeat bits [0, ps)), so the 32 slots (h + o) mod ps, o in [w, w + 32), are the
// bits [h + w, h + w + 32) of the doubled bitmap for any slot h < ps and w < ps.
// It is stored as pairs (word i, word i + 1), so that a window that straddles two
// words is one 64-bit load and one funnel shift (two 32-bit loads from a bitmap of single words
// make the search 3.4 % slower: 6.41 against 6.20 ms at 10^8 u64 keys, lambda 7).  Lane L tests offsets [w, w + 32),
// w = w0 + 32 L, by OR-ing the windows of all keys of the bucket; a warp covers
// 1024 offsets per round and the first lane with a free window holds the
// smallest valid offset.  Because w is a multiple of 32, the pair index of a
// window is (h >> 5) + (w >> 5) and its bit shift is h & 31 for every lane.
//
// Buckets of at most 32 keys (nearly all of them) are hashed for 32 / S pilot
// counters at once (S = 4, 8, 16 or 32 lanes per counter) into shared memory, from
// where every lane reads the slots of one counter four at a time (broadcast 128-bit
// loads).  Larger buckets read their keys from the bucket-ordered copy in global
// memory.
#include <algorithm>

#include "kernels.cuh"

namespace phobicb200 {

namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kHsWords = 260;  // packed slots of up to 256 keys, padded to a multiple of 4

// Collision scratch of large buckets: one bit per slot.
__host__ __device__ __forceinline__ uint32_t scr_words(uint32_t cap) { return (cap + 31) / 32 + 1; }
// Pairs of the bitmap of a partition of at most cap slots: for a slot h < ps and lane L in
// round r < ceil(ps / 1024) the offset search reads pair (h >> 5) + L + 32 r, dead lanes
// included, and a mark sets bits below 2 ps; one pair more lies in front, for the mark of
// word 0 as the second word of the pair before it.
__host__ __device__ __forceinline__ uint32_t bitmap_pairs(uint32_t cap) {
    const uint32_t reach = (cap - 1) / 32 + 32 * ((cap + 1023) / 1024), marks = (2 * cap - 1) / 32 + 1;
    return (reach > marks ? reach : marks) + 1;
}

// Per-warp shared memory, in 32-bit words.  Every warp's region starts on a
// 16-byte boundary (its size is rounded up to 4 words):
//   hs    [260]      packed slots (16-byte aligned for the 128-bit slot loads)
//   occ   [2 OP]     pairs of the occupied slots' bitmap (bits [ps, 2 ps) mirror [0, ps))
//   scr   [SW]       collision scratch of large buckets
//   sched [B + 1]    search schedule, in search order: start | bucket << 16; then the end
__host__ __device__ __forceinline__ size_t warp_words(uint32_t B, uint32_t cap) {
    const size_t w = kHsWords + 2 * (size_t)bitmap_pairs(cap) + scr_words(cap) + (size_t)B + 1;
    return (w + 3) & ~size_t(3);
}

struct WarpSmem {
    uint32_t *hs, *scr, *sched;
    uint32_t occ;             // shared-space byte address of pair 0 of the bitmap
    uint32_t occ_lo, occ_hi;  // shared-space byte bounds of the bitmap (checked build)
};

__device__ __forceinline__ WarpSmem carve(uint32_t *w, uint32_t B, uint32_t cap) {
    WarpSmem m;
    m.hs = w;
    m.scr = w + kHsWords + 2 * bitmap_pairs(cap);
    m.sched = m.scr + scr_words(cap);
    m.occ_lo = (uint32_t)__cvta_generic_to_shared(w + kHsWords);
    m.occ = m.occ_lo + 8;
    m.occ_hi = m.occ_lo + 8 * bitmap_pairs(cap);
    return m;
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void red_or(uint32_t addr, uint32_t bit) {
    asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(addr), "r"(bit) : "memory");
}
__device__ __forceinline__ void red_and(uint32_t addr, uint32_t mask) {
    asm volatile("red.shared.and.b32 [%0], %1;" ::"r"(addr), "r"(mask) : "memory");
}

// Byte offset of the pair whose first word holds slot q (the pair before it holds that word
// as its second).
__device__ __forceinline__ uint32_t pair_of(uint32_t q) { return (q >> 5) << 3; }

// Sets slot q and its mirror q + ps, each in the two pairs that hold its word.
__device__ __forceinline__ void mark(uint32_t occ, uint32_t q, uint32_t ps) {
    const uint32_t a = occ + pair_of(q), bit = 1u << (q & 31), m = q + ps;
    const uint32_t b = occ + pair_of(m), mbit = 1u << (m & 31);
    red_or(a, bit);
    red_or(a - 4, bit);
    red_or(b, mbit);
    red_or(b - 4, mbit);
}
__device__ __forceinline__ bool is_taken(uint32_t occ, uint32_t q) {
    uint32_t w;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(occ + pair_of(q)) : "memory");
    return (w >> (q & 31)) & 1u;
}

// A slot h as the offset search reads it: the byte offset of its pair, 8 * (h >> 5),
// shifted left by 5, with the bit position h & 31 in the low bits.  The funnel shift only
// looks at the low 5 bits, so one word serves both uses.
__device__ __forceinline__ uint32_t pack_slot(uint32_t h) { return ((h >> 5) << 8) | (h & 31); }
__device__ __forceinline__ uint32_t unpack_slot(uint32_t v) { return ((v >> 8) << 5) | (v & 31); }

// The 32-bit window of packed slot v, OFF bytes past the pair at `addr`; in the checked build
// the pair must lie inside the bitmap.
template <int OFF>
__device__ __forceinline__ uint32_t window_at(const WarpSmem &ws, uint32_t addr, uint32_t v) {
    if (!PHB_CHECK(addr + OFF >= ws.occ_lo && addr + OFF + 8 <= ws.occ_hi)) return kFullMask;
    uint32_t x, y;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2+%3];" : "=r"(x), "=r"(y) : "r"(addr), "n"(OFF));
    return __funnelshift_r(x, y, v);
}

// What the offset search needs of a partition: the number of rounds of 1024 offsets and, for
// this lane, the offsets of the last round's window that are not below ps.
struct ScanRange {
    uint32_t ps, rounds, last_dead;
    __device__ __forceinline__ static ScanRange make(uint32_t ps, int lane) {
        ScanRange r;
        r.ps = ps;
        r.rounds = (ps + 1023) / 1024;
        const int n = (int)ps - (int)(1024 * (r.rounds - 1)) - 32 * lane;
        r.last_dead = ~__funnelshift_lc(kFullMask, 0u, (uint32_t)max(n, 0));  // n >= 32: none
        return r;
    }
};

// The smallest free offset of a round that starts at offset o0, if any lane's window is open.
__device__ __forceinline__ bool round_result(uint32_t bad, uint32_t o0, uint32_t *o) {
    const uint32_t ball = __ballot_sync(kFullMask, bad != kFullMask);
    if (!ball) return false;
    const int f = __ffs(ball) - 1;
    *o = o0 + 32u * f + __ffs(~__shfl_sync(kFullMask, bad, f)) - 1;
    return true;
}

// Round R of a block of three: the windows of a bucket of at most S = 4 or 8 keys whose packed
// slots are in v and whose pair addresses (this lane's window offset included) are in a.  The
// last two keys of S are skipped when the bucket is that small.
template <int S, int R>
__device__ __forceinline__ uint32_t round_bad(const WarpSmem &ws, const uint32_t (&a)[S], const uint32_t (&v)[S],
                                              bool full, uint32_t bad) {
#pragma unroll
    for (int i = 0; i < S - 2; i++) bad |= window_at<256 * R>(ws, a[i], v[i]);
    if (full) bad |= window_at<256 * R>(ws, a[S - 2], v[S - 2]) | window_at<256 * R>(ws, a[S - 1], v[S - 1]);
    return bad;
}

// Smallest free offset of a bucket of s <= S keys (S = 4 or 8) whose S packed slots start at the
// shared address hs (entries past the bucket repeat a slot: OR is idempotent).  Three rounds at
// constant offsets from each key's pair address cover 3072 offsets; larger partitions repeat
// them.  Dead lanes read inside the padded bitmap (bitmap_pairs) and are masked.
template <int S>
__device__ __forceinline__ uint32_t scan_small(const WarpSmem &ws, uint32_t hs, uint32_t s, const ScanRange &sr,
                                               int lane) {
    const uint32_t lane_sa = ws.occ + 8u * lane;
    uint32_t v[S], a[S];
#pragma unroll
    for (int i = 0; i < S; i += 4) {
        const uint4 x = lds128(hs + 4 * i);
        v[i] = x.x, v[i + 1] = x.y, v[i + 2] = x.z, v[i + 3] = x.w;
    }
#pragma unroll
    for (int i = 0; i < S; i++) a[i] = lane_sa + (v[i] >> 5);
    const bool full = s > S - 2;
    uint32_t o;
    for (uint32_t left = sr.rounds, o0 = 0;;) {
        if (round_result(round_bad<S, 0>(ws, a, v, full, left == 1 ? sr.last_dead : 0u), o0, &o)) return o;
        if (left == 1) return kNone;
        if (round_result(round_bad<S, 1>(ws, a, v, full, left == 2 ? sr.last_dead : 0u), o0 + 1024, &o)) return o;
        if (left == 2) return kNone;
        if (round_result(round_bad<S, 2>(ws, a, v, full, left == 3 ? sr.last_dead : 0u), o0 + 2048, &o)) return o;
        if (left == 3) return kNone;
        left -= 3;
        o0 += 3072;
#pragma unroll
        for (int i = 0; i < S; i++) a[i] += 768;
    }
}

// The same for a bucket of any size: s packed slots at the shared address hs, padded to a
// multiple of 4 with copies of one of them.
__device__ __forceinline__ uint32_t scan_quads(const WarpSmem &ws, uint32_t hs, uint32_t s, const ScanRange &sr,
                                               int lane) {
    uint32_t lane_sa = ws.occ + 8u * lane, o;
    const uint32_t hs_end = hs + 4 * s;
    for (uint32_t r = 1;; r++, lane_sa += 256) {
        uint32_t bad = r == sr.rounds ? sr.last_dead : 0u;
#pragma unroll 2
        for (uint32_t q = hs; q < hs_end; q += 16) {
            const uint4 v = lds128(q);
            bad |= window_at<0>(ws, lane_sa + (v.x >> 5), v.x) | window_at<0>(ws, lane_sa + (v.y >> 5), v.y);
            bad |= window_at<0>(ws, lane_sa + (v.z >> 5), v.z) | window_at<0>(ws, lane_sa + (v.w >> 5), v.w);
        }
        if (round_result(bad, 1024 * (r - 1), &o)) return o;
        if (r == sr.rounds) return kNone;
    }
}

// Whether two keys of a bucket of s <= 32 keys (key `lane` in L) are identical.
// Reached only when a bucket's pilot counter gets to kDupCheckAt, so it is kept
// out of line, away from the instructions of the search loop.
__device__ __noinline__ bool has_duplicate_key(uint2 L, uint32_t s, int lane) {
    bool d = false;
    for (uint32_t t = 0; t + 1 < s; t++) {
        uint32_t x = __shfl_sync(kFullMask, L.x, t), y = __shfl_sync(kFullMask, L.y, t);
        d |= lane < (int)s && lane > (int)t && L.x == x && L.y == y;
    }
    return __any_sync(kFullMask, d);
}

// Two keys of a bucket on one slot reject the pilot counter (search.comp:44-70).  That is
// rare (1 % of the tries of buckets of at most 32 keys at lambda 7), so it is tested only once
// a free offset is found, with the shared-memory atomics that the marks need anyway: two lanes
// on one slot show as a bit that was set already.  __match_any_sync on every try, as before,
// takes 354-378 cycles and occupies an SM's unit for 59-64 cycles per warp (measured alone on a
// B200; atomicOr with its result: 42 and 1.6).  At 10^8 u64 keys (lambda 7, P 2500) the search
// took 7.65 ms with it and 7.17 ms without.

// Marks slot q (and its mirror) of every lane that is `on`, or marks nothing and returns
// false when two of the lanes hold the same slot.  The slots were free before.  Predicated
// instructions: the lanes of a bucket mark without a divergent branch.
__device__ __forceinline__ bool mark_distinct(uint32_t occ, uint32_t q, uint32_t ps, bool on) {
    const uint32_t a = occ + pair_of(q), bit = 1u << (q & 31), m = q + ps;
    const uint32_t b = occ + pair_of(m), mbit = 1u << (m & 31);
    uint32_t old;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\tmov.u32 %0, 0;\n\t"
        "@p atom.shared.or.b32 %0, [%1], %2;\n\t}"
        : "=&r"(old) : "r"(a), "r"(bit), "r"((uint32_t)on) : "memory");
    if (__any_sync(kFullMask, old & bit)) {
        if (on) red_and(a, ~bit);
        __syncwarp();
        return false;
    }
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "@p red.shared.or.b32 [%0+-4], %1;\n\t@p red.shared.or.b32 [%2], %3;\n\t@p red.shared.or.b32 [%2+-4], %3;\n\t}"
        ::"r"(a), "r"(bit), "r"(b), "r"(mbit), "r"((uint32_t)on) : "memory");
    __syncwarp();
    return true;
}

// Whether the slots of the lanes that are `on` are distinct, tested in the warp's own clear
// collision scratch (left clear): for searches that do not mark.
__device__ __forceinline__ bool slots_distinct(uint32_t *scr, uint32_t q, bool on) {
    const uint32_t bit = 1u << (q & 31);
    const uint32_t old = on ? atomicOr(&scr[q >> 5], bit) : 0u;
    const bool hit = __any_sync(kFullMask, on && (old & bit));
    if (on) scr[q >> 5] = 0;
    __syncwarp();
    return !hit;
}

// Lanes per pilot counter for a bucket of s <= 32 keys: 4, 8, 16 or 32.
__device__ __forceinline__ uint32_t counter_lanes(uint32_t s) { return s <= 4 ? 4u : s <= 8 ? 8u : s <= 16 ? 16u : 32u; }
// The key that lane `lane` loads of a bucket of s <= 32 keys: lane t * S + i takes key i, lanes
// past the bucket key 0, whose slots are the padding that the scan expects.
__device__ __forceinline__ uint32_t lane_key(uint32_t s, int lane) {
    const uint32_t i = (uint32_t)lane & (counter_lanes(s) - 1u);
    return i < s ? i : 0u;
}

// A bucket of at most S keys (S = 4, 8, 16 or 32; more than S / 2 of them, or S = 4), L as
// lane_key loads it.  The warp hashes 32 / S pilot counters at once (lane t * S + i holds key i
// under counter k0 + t) into hs and tests them in counter order, so a counter that fails costs
// no new hash.  Same result as trying k = 0, 1, 2, ... one at a time (search.comp:105-124).
// With MARK the slots are marked and *pilot written; without, nothing is marked and the bucket
// pipeline gets the counter, the offset and (lanes < s) the lane's slot in *k_out, *o_out,
// *q_out.
template <int S, bool MARK = true>
__device__ __forceinline__ uint32_t place_batched(const WarpSmem &ws, uint2 L, uint32_t s, const ScanRange &sr,
                                                  FastMod fm, uint32_t k_lim, int lane, uint32_t *pilot,
                                                  uint32_t *k_out = nullptr, uint32_t *o_out = nullptr,
                                                  uint32_t *q_out = nullptr) {
    constexpr uint32_t G = 32 / S;
    const uint32_t hs_sa = (uint32_t)__cvta_generic_to_shared(ws.hs);
    const bool mine = lane < (int)s;
    uint32_t stop = min(k_lim, kDupCheckAt);  // a multiple of G, or k_lim
    for (uint32_t k0 = 0;; k0 += G) {
        if (k0 >= stop) {
            if (k0 >= k_lim) return PHOBIC_ERR_SEARCH_LIMIT;
            if (s > 1 && has_duplicate_key(L, s, lane)) return PHOBIC_ERR_DUPLICATE_KEY;
            stop = k_lim;
        }
        const uint32_t hk = pack_slot(fm.mod(pilot_hash(L.x, L.y, k0 + (uint32_t)lane / S)));
        __syncwarp();
        ws.hs[lane] = hk;
        __syncwarp();
        const uint32_t tries = min(G, k_lim - k0);
#pragma unroll 1
        for (uint32_t u = 0; u < tries; u++) {
            uint32_t o;
            if constexpr (S <= 8) o = scan_small<S>(ws, hs_sa + 4 * S * u, s, sr, lane);
            else o = scan_quads(ws, hs_sa + 4 * S * u, s, sr, lane);
            if (o == kNone) continue;
            uint32_t q = unpack_slot(ws.hs[S * u + (mine ? (uint32_t)lane : 0u)]) + o;
            q = q >= sr.ps ? q - sr.ps : q;
            const bool on = mine && PHB_CHECK(!mine || q < sr.ps);
            if constexpr (MARK) {
                if (!mark_distinct(ws.occ, q, sr.ps, on)) continue;
                *pilot = o + sr.ps * (k0 + u);
            } else {
                if (!slots_distinct(ws.scr, q, on)) continue;
                *k_out = k0 + u;
                *o_out = o;
                *q_out = q;
            }
            return PHOBIC_OK;
        }
    }
}

// place_batched for any bucket of at most 32 keys.
template <bool MARK>
__device__ __forceinline__ uint32_t place_any(const WarpSmem &ws, uint2 L, uint32_t s, const ScanRange &sr, FastMod fm,
                                              uint32_t k_lim, int lane, uint32_t *pilot, uint32_t *k_out = nullptr,
                                              uint32_t *o_out = nullptr, uint32_t *q_out = nullptr) {
    if (s <= 4) return place_batched<4, MARK>(ws, L, s, sr, fm, k_lim, lane, pilot, k_out, o_out, q_out);
    if (s <= 8) return place_batched<8, MARK>(ws, L, s, sr, fm, k_lim, lane, pilot, k_out, o_out, q_out);
    if (s <= 16) return place_batched<16, MARK>(ws, L, s, sr, fm, k_lim, lane, pilot, k_out, o_out, q_out);
    return place_batched<32, MARK>(ws, L, s, sr, fm, k_lim, lane, pilot, k_out, o_out, q_out);
}

// One bucket of more than 32 keys (a few per partition).  Each try hashes chunk by chunk and
// stops at the first chunk that repeats a slot: buckets of 100 to 160 keys are rejected about 37
// times per partition (10^8 u64 keys, lambda 7, P 2500), after 62 keys on average.  The keys are
// read from the bucket-ordered copy on every try: staging them in shared memory takes that much
// from the L1 that the copy and the schedule are read through, and was slower (search 6.18
// against 6.06 ms).
__device__ __forceinline__ uint32_t place_large(const WarpSmem &ws, const uint2 *src, uint32_t s, const ScanRange &sr,
                                                FastMod fm, uint32_t k_lim, int lane, uint32_t *pilot) {
    const uint32_t padded = (s + 3) & ~3u, ps = sr.ps;
    const uint32_t hs_sa = (uint32_t)__cvta_generic_to_shared(ws.hs);
    for (uint32_t k = 0; k < k_lim; k++) {
        if (k == kDupCheckAt) {
            bool d = false;
            for (uint32_t t = 0; t + 1 < s; t++) {
                uint2 kt = src[t];
                for (uint32_t i = lane; i < s; i += 32) d |= i > t && src[i].x == kt.x && src[i].y == kt.y;
            }
            if (__any_sync(kFullMask, d)) return PHOBIC_ERR_DUPLICATE_KEY;
        }
        bool dup = false;
        uint32_t done = 0;  // keys hashed (and marked in the collision scratch)
        for (uint32_t c0 = 0; c0 < s && !dup; c0 += 32) {
            const uint32_t i = c0 + lane;
            bool d = false;
            if (i < s) {
                const uint2 key = src[i];
                const uint32_t h = fm.mod(pilot_hash(key.x, key.y, k));
                ws.hs[i] = pack_slot(h);
                const uint32_t bit = 1u << (h & 31);
                d = PHB_CHECK(h < ps) && (atomicOr(&ws.scr[h >> 5], bit) & bit) != 0;
            }
            dup = __any_sync(kFullMask, d);
            done = c0 + 32;
        }
        for (uint32_t i = lane; i < s && i < done; i += 32) ws.scr[unpack_slot(ws.hs[i]) >> 5] = 0;
        __syncwarp();
        if (dup) continue;
        if (s + lane < padded) ws.hs[s + lane] = ws.hs[0];
        __syncwarp();
        const uint32_t o = scan_quads(ws, hs_sa, s, sr, lane);
        __syncwarp();
        if (o == kNone) continue;
        for (uint32_t i = lane; i < s; i += 32) {
            uint32_t q = unpack_slot(ws.hs[i]) + o;
            q = q >= ps ? q - ps : q;
            if (PHB_CHECK(q < ps)) mark(ws.occ, q, ps);
        }
        __syncwarp();
        *pilot = o + ps * k;
        return PHOBIC_OK;
    }
    return PHOBIC_ERR_SEARCH_LIMIT;
}

// The first SearchArgs words of a partition's search, by `threads` threads of which this is
// number t: the schedule, a clear bitmap (as far as this partition reads it) and a clear
// collision scratch.  w is the start of the group's shared memory.
__device__ __forceinline__ void load_partition(const SearchArgs &a, uint32_t *w, const WarpSmem &ws, uint32_t base,
                                               uint32_t ps, uint32_t nonempty, uint32_t t, uint32_t threads) {
    const uint32_t *sch = reinterpret_cast<const uint32_t *>(a.lowers + base);
#pragma unroll 4
    for (uint32_t i = t; i <= nonempty; i += threads)
        if (PHB_CHECK(i <= a.buckets)) ws.sched[i] = __ldcs(sch + i);
    uint2 *occ = reinterpret_cast<uint2 *>(w + kHsWords);
    const uint32_t pairs = bitmap_pairs(ps);
    for (uint32_t i = t; i < pairs; i += threads) occ[i] = make_uint2(0, 0);
    for (uint32_t i = t; i < scr_words(a.cap); i += threads) ws.scr[i] = 0;
}

// One partition's pilots.
__device__ __forceinline__ uint32_t search_partition(const SearchArgs &a, uint32_t *w, const WarpSmem &ws,
                                                     const SetDesc &d, uint32_t g, uint32_t p, int lane) {
    const uint32_t nonempty = a.part_state[g];
    if (nonempty & kPartSkipped) return nonempty & ~kPartSkipped;
    const uint32_t base = a.G[(size_t)g * a.gstride];
    const uint32_t ps = a.G[(size_t)(g + 1) * a.gstride] - base;
    if (ps == 0) return PHOBIC_OK;
    load_partition(a, w, ws, base, ps, nonempty, (uint32_t)lane, 32);
    __syncwarp();
    uint32_t *pil = d.pilots + p;
    const size_t pstride = d.partitions;
    const uint2 *so = a.sorted + base;

    // Pilot search (search.comp:126-175), next bucket's keys prefetched.
    const FastMod fm = FastMod::make(ps);
    const ScanRange sr = ScanRange::make(ps, lane);
    uint32_t k_lim = 0x80000000u / ps;
    if (k_lim > a.k_max) k_lim = a.k_max;
    // sched[nonempty] holds the end, so a bucket's size is the distance to the next start.
    uint32_t sc = ws.sched[0], sc1 = ws.sched[1];
    uint32_t s_next = (sc1 - sc) & 0xFFFFu;
    uint2 L_next = s_next <= 32 ? so[(sc & 0xFFFFu) + lane_key(s_next, lane)] : make_uint2(0, 0);
    for (uint32_t j = 0; j < nonempty; j++) {
        const uint32_t s = s_next, b = sc >> 16, st = sc & 0xFFFFu;
        const uint2 L = L_next;
        sc = sc1;
        if (j + 1 < nonempty) {
            sc1 = ws.sched[j + 2];
            s_next = (sc1 - sc) & 0xFFFFu;
            if (s_next <= 32) L_next = so[(sc & 0xFFFFu) + lane_key(s_next, lane)];
        }
        uint32_t pilot = 0;
        const uint32_t st_code = s <= 32 ? place_any<true>(ws, L, s, sr, fm, k_lim, lane, &pilot)
                                         : place_large(ws, so + st, s, sr, fm, k_lim, lane, &pilot);
        if (st_code != PHOBIC_OK) return st_code;
        if (lane == 0 && PHB_CHECK(b < a.buckets)) pil[(size_t)b * pstride] = pilot;
    }
    __syncwarp();
    return PHOBIC_OK;
}

// ------------------------------------------------------------------ k-split groups
//
// For builds with far fewer partitions than warp slots (small key sets, where one
// warp per partition leaves most of the GPU idle and each partition's search is
// bound by the latency of its sequential tries), a group of W warps searches one
// partition: in each step, warp w tries pilot counter k0 + w for the current bucket
// (hash, collision test, offset scan over all of [0, ps)).  The step's outcomes are
// exchanged in shared memory and read in k order, so the bucket takes the smallest k
// that has a free offset, with that k's smallest offset: the result of trying
// k = 0, 1, 2, ... one at a time (search.comp:105-124).  Every warp then marks the
// winning slots itself (the marks are idempotent), so no warp reads the bitmap before
// its own copy of the marks is in place.
constexpr uint32_t kTryNone = 0, kTryFound = 1, kTryDup = 2, kTryLimit = 3;

__device__ __forceinline__ void group_bar(uint32_t id, uint32_t threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Per-warp scratch of warps 1..W-1 of a group (warp 0 uses its place in carve()).
__host__ __device__ __forceinline__ size_t group_extra_words(uint32_t cap) {
    return ((size_t)kHsWords + scr_words(cap) + 3) & ~size_t(3);
}
// Exchange words: [2 parities][W] outcomes, the control words (job, nonempty, committed,
// status), and the bucket pipeline's results: [W] (code << 24 | k, offset) pairs and [W][32]
// slots (padded).
__host__ __device__ __forceinline__ size_t group_xch_words(int W) {
    return ((size_t)2 * W + 4 + 2 * (size_t)W + 32 * (size_t)W + 3) & ~size_t(3);
}
__host__ __device__ __forceinline__ size_t group_words(uint32_t B, uint32_t cap, int W) {
    return warp_words(B, cap) + (size_t)(W - 1) * group_extra_words(cap) + group_xch_words(W);
}

// One try of a pilot counter for a bucket of s <= 32 keys, hk holding key `lane`'s slot
// under that counter (lanes past the bucket: a slot of some key): the offset scan and collision
// test of place_batched.  kTryFound with *o, else kTryNone.
__device__ __forceinline__ uint32_t try_small(const WarpSmem &ws, uint32_t s, const ScanRange &sr, uint32_t hk,
                                              int lane, uint32_t *o_out) {
    const bool mine = lane < (int)s;
    __syncwarp();
    ws.hs[lane] = pack_slot(hk);
    __syncwarp();
    const uint32_t hs_sa = (uint32_t)__cvta_generic_to_shared(ws.hs);
    const uint32_t o = s <= 4   ? scan_small<4>(ws, hs_sa, s, sr, lane)
                       : s <= 8 ? scan_small<8>(ws, hs_sa, s, sr, lane)
                                : scan_quads(ws, hs_sa, s, sr, lane);
    if (o == kNone || !slots_distinct(ws.scr, hk, mine && PHB_CHECK(!mine || hk < sr.ps))) return kTryNone;
    *o_out = o;
    return kTryFound;
}

// One try of pilot counter k for a bucket of more than 32 keys read from src: the
// chunked collision test and offset scan of place_large.
__device__ __forceinline__ uint32_t try_large(const WarpSmem &ws, const uint2 *src, uint32_t s, const ScanRange &sr,
                                              FastMod fm, uint32_t k, int lane, uint32_t *o_out) {
    const uint32_t padded = (s + 3) & ~3u;
    const uint32_t hs_sa = (uint32_t)__cvta_generic_to_shared(ws.hs);
    bool dup = false;
    uint32_t done = 0;
    for (uint32_t c0 = 0; c0 < s && !dup; c0 += 32) {
        const uint32_t i = c0 + lane;
        bool d = false;
        if (i < s) {
            const uint2 key = src[i];
            const uint32_t h = fm.mod(pilot_hash(key.x, key.y, k));
            ws.hs[i] = pack_slot(h);
            const uint32_t bit = 1u << (h & 31);
            d = PHB_CHECK(h < sr.ps) && (atomicOr(&ws.scr[h >> 5], bit) & bit) != 0;
        }
        dup = __any_sync(kFullMask, d);
        done = c0 + 32;
    }
    for (uint32_t i = lane; i < s && i < done; i += 32) ws.scr[unpack_slot(ws.hs[i]) >> 5] = 0;
    __syncwarp();
    if (dup) return kTryNone;
    if (s + lane < padded) ws.hs[s + lane] = ws.hs[0];
    __syncwarp();
    const uint32_t o = scan_quads(ws, hs_sa, s, sr, lane);
    __syncwarp();
    if (o == kNone) return kTryNone;
    *o_out = o;
    return kTryFound;
}

// Whether two of the s keys read from src are identical (the check at pilot counter
// kDupCheckAt of place_large).
__device__ __noinline__ bool has_duplicate_key_src(const uint2 *src, uint32_t s, int lane) {
    bool d = false;
    for (uint32_t t = 0; t + 1 < s; t++) {
        const uint2 kt = src[t];
        for (uint32_t i = lane; i < s; i += 32) d |= i > t && src[i].x == kt.x && src[i].y == kt.y;
    }
    return __any_sync(kFullMask, d);
}

// Marks the slots (h_i + o) mod ps of the bucket's keys at pilot counter k.
__device__ __forceinline__ void mark_bucket(const WarpSmem &ws, uint2 L, const uint2 *src, uint32_t s, uint32_t ps,
                                            FastMod fm, uint32_t k, uint32_t o, int lane) {
    if (s <= 32) {
        if (lane < (int)s) {
            uint32_t q = fm.mod(pilot_hash(L.x, L.y, k)) + o;
            q = q >= ps ? q - ps : q;
            if (PHB_CHECK(q < ps)) mark(ws.occ, q, ps);
        }
    } else {
        for (uint32_t i = lane; i < s; i += 32) {
            const uint2 key = src[i];
            uint32_t q = fm.mod(pilot_hash(key.x, key.y, k)) + o;
            q = q >= ps ? q - ps : q;
            if (PHB_CHECK(q < ps)) mark(ws.occ, q, ps);
        }
    }
    __syncwarp();
}

// Group kernel: kSearchWarps / W groups per CTA, each a persistent searcher over the
// partition queue; all W warps of a group search a partition's buckets in k-split steps.
// Small builds leave most SMs idle, so the group kernel is not held to the one-warp
// kernel's 4 CTAs per SM (64 registers): 2 CTAs per SM keep it free of spills.
// Bucket pipeline (PIPE): for buckets of at most 32 keys (the tail of the search order),
// warp w searches bucket j + w completely (smallest k, then smallest o) on the bitmap as it
// stands, without marking.  Warp 0 then commits the W results in order: a result is kept
// while its slots are still free after the results before it were marked.  That keeps the
// sequential answer: the bitmap only gains occupied slots, so a (k, o) valid on the later
// state was valid on the earlier one, and the smallest valid pair on the earlier state, if
// still valid, is the smallest on the later one.  A pilot limit or duplicate keys found on the
// earlier state hold on the later one too.  The first result that conflicts is searched again
// in the next step.
template <int W, bool PIPE>
__global__ void __launch_bounds__(kSearchWarps * 32, 2) k_search_group(SearchArgs a) {
    extern __shared__ __align__(16) uint32_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int grp = warp / W, w = warp % W;
    const uint32_t bar_id = 1 + grp, bar_n = 32 * W;
    uint32_t *gbase = smem + (size_t)grp * group_words(a.buckets, a.cap, W);
    const WarpSmem ws0 = carve(gbase, a.buckets, a.cap);
    WarpSmem ws = ws0;
    if (w > 0) {
        ws.hs = gbase + warp_words(a.buckets, a.cap) + (size_t)(w - 1) * group_extra_words(a.cap);  // own slots
        ws.scr = ws.hs + kHsWords;
    }
    uint32_t *xch = gbase + warp_words(a.buckets, a.cap) + (size_t)(W - 1) * group_extra_words(a.cap);
    uint32_t *ctl = xch + 2 * W;  // [0] job, [1] nonempty, [2] committed, [3] status
    uint32_t *pres = ctl + 4;     // [W] pairs: code << 24 | k, offset
    uint32_t *pslots = pres + 2 * W;  // [W][32] slots of each warp's result
    uint32_t par = 0;
    for (;;) {
        if (w == 0 && lane == 0) ctl[0] = atomicAdd(a.queue, 1u);
        group_bar(bar_id, bar_n);
        const uint32_t g = ctl[0];
        if (g >= a.M) break;
        const uint32_t s_idx = a.nsets == 1 ? 0u : find_set(a.part_base, a.nsets, g);
        const SetDesc &d = a.sets[s_idx];
        const uint32_t p = g - d.part_base;
        // ctl[1] = nonempty buckets, or 0xFFFFFFFF when there is nothing to search.
        if (w == 0 && lane == 0) {
            uint32_t ctl1 = 0xFFFFFFFFu;
            if (!fatal_before_search(*reinterpret_cast<volatile unsigned long long *>(&a.err[s_idx]))) {
                const uint32_t state = a.part_state[g];
                if (!(state & kPartSkipped)) ctl1 = state;
                else if (state != kPartSkipped) report_error(&a.err[s_idx], p, state & ~kPartSkipped);
            }
            if (ctl1 == 0) ctl1 = 0xFFFFFFFFu;
            ctl[1] = ctl1;
        }
        group_bar(bar_id, bar_n);
        const uint32_t nonempty = ctl[1];
        if (nonempty != 0xFFFFFFFFu) {
            const uint32_t base = a.G[(size_t)g * a.gstride];
            const uint32_t ps = a.G[(size_t)(g + 1) * a.gstride] - base;
            const uint2 *so = a.sorted + base;
            uint32_t *pil = d.pilots + p;
            const size_t pstride = d.partitions;
            load_partition(a, gbase, ws0, base, ps, nonempty, (uint32_t)(32 * w + lane), bar_n);
            if (w > 0)
                for (uint32_t i = lane; i < scr_words(a.cap); i += 32) ws.scr[i] = 0;
            group_bar(bar_id, bar_n);
            const FastMod fm = FastMod::make(ps);
            const ScanRange sr = ScanRange::make(ps, lane);
            uint32_t k_lim = 0x80000000u / ps;
            if (k_lim > a.k_max) k_lim = a.k_max;
            uint32_t err = PHOBIC_OK;
            for (uint32_t j = 0; j < nonempty && err == PHOBIC_OK; j++) {
                const uint32_t sc = ws.sched[j];
                const uint32_t b = sc >> 16, st = sc & 0xFFFFu;
                const uint32_t s = (ws.sched[j + 1] - sc) & 0xFFFFu;
                const uint2 *src = so + st;
                if (PIPE && s <= 32) {  // every later bucket is as small (search order: size descending)
                    const uint32_t jw = j + w;
                    if (jw < nonempty) {
                        const uint32_t scw = ws.sched[jw];
                        const uint32_t sw = (ws.sched[jw + 1] - scw) & 0xFFFFu;
                        const uint2 Lw = so[(scw & 0xFFFFu) + lane_key(sw, lane)];
                        uint32_t kk = 0, o = 0, q = 0;
                        const uint32_t st = place_any<false>(ws, Lw, sw, sr, fm, k_lim, lane, nullptr, &kk, &o, &q);
                        const uint32_t code = st == PHOBIC_OK                  ? kTryFound
                                              : st == PHOBIC_ERR_DUPLICATE_KEY ? kTryDup
                                                                               : kTryLimit;
                        if (code == kTryFound && lane < (int)sw) pslots[32 * w + lane] = q;
                        if (lane == 0) {
                            pres[2 * w] = (code << 24) | (kk & 0xFFFFFFu);
                            pres[2 * w + 1] = o;
                        }
                    }
                    group_bar(bar_id, bar_n);
                    if (w == 0) {
                        uint32_t committed = 0, e = PHOBIC_OK;
                        for (uint32_t v = 0; v < (uint32_t)W && j + v < nonempty; v++) {
                            const uint32_t r0 = pres[2 * v], rcode = r0 >> 24;
                            if (rcode != kTryFound) {
                                e = rcode == kTryDup ? PHOBIC_ERR_DUPLICATE_KEY : PHOBIC_ERR_SEARCH_LIMIT;
                                break;
                            }
                            const uint32_t scv = ws.sched[j + v], bv = scv >> 16;
                            const uint32_t sv = (ws.sched[j + v + 1] - scv) & 0xFFFFu;
                            const bool mine = lane < (int)sv;
                            const uint32_t q = mine ? pslots[32 * v + lane] : 0u;
                            const bool on = mine && PHB_CHECK(!mine || q < ps);
                            if (__any_sync(kFullMask, on && is_taken(ws.occ, q))) break;  // searched again next step
                            if (on) mark(ws.occ, q, ps);
                            __syncwarp();
                            if (lane == 0 && PHB_CHECK(bv < a.buckets))
                                pil[(size_t)bv * pstride] = pres[2 * v + 1] + ps * (r0 & 0xFFFFFFu);
                            committed++;
                        }
                        if (lane == 0) {
                            ctl[2] = committed;
                            ctl[3] = e;
                        }
                    }
                    group_bar(bar_id, bar_n);
                    err = ctl[3];
                    j += ctl[2];
                    j--;  // the loop's increment
                    continue;
                }
                const uint2 L = s <= 32 ? src[lane_key(s, lane)] : make_uint2(0, 0);
                for (uint32_t k0 = 0;; k0 += W) {
                    const uint32_t k = k0 + w;
                    uint32_t code = kTryNone, o = 0;
                    if (k >= k_lim) code = kTryLimit;
                    else if (k == kDupCheckAt && s > 1 &&
                             (s <= 32 ? has_duplicate_key(L, s, lane) : has_duplicate_key_src(src, s, lane)))
                        code = kTryDup;
                    else code = s <= 32 ? try_small(ws, s, sr, fm.mod(pilot_hash(L.x, L.y, k)), lane, &o)
                                        : try_large(ws, src, s, sr, fm, k, lane, &o);
                    if (lane == 0) xch[par * W + w] = (code << 16) | (o & 0xFFFFu);
                    group_bar(bar_id, bar_n);
                    uint32_t win = kTryNone << 16, v = 0;
                    for (; v < (uint32_t)W; v++) {
                        win = xch[par * W + v];
                        if ((win >> 16) != kTryNone) break;
                    }
                    par ^= 1u;
                    const uint32_t wcode = win >> 16;
                    if (wcode == kTryNone) continue;
                    if (wcode == kTryFound) {
                        const uint32_t kw = k0 + v, ow = win & 0xFFFFu;
                        mark_bucket(ws, L, src, s, ps, fm, kw, ow, lane);
                        if (w == 0 && lane == 0 && PHB_CHECK(b < a.buckets)) pil[(size_t)b * pstride] = ow + ps * kw;
                    } else {
                        err = wcode == kTryDup ? PHOBIC_ERR_DUPLICATE_KEY : PHOBIC_ERR_SEARCH_LIMIT;
                    }
                    break;
                }
            }
            if (err != PHOBIC_OK && w == 0 && lane == 0) report_error(&a.err[s_idx], p, err);
        }
        // Everyone is done with this partition's tables before the next is fetched.
        group_bar(bar_id, bar_n);
    }
}

}  // namespace

unsigned int check_line_search(bool reset) { return read_check_line(reset); }

size_t search_warp_smem(uint32_t buckets, uint32_t cap) { return 4 * warp_words(buckets, cap); }

// The bound is the shared memory of a warp that also sorted its partition (packed u16 tables of
// bucket sizes and cursors, two of 256 size bins, slots, collision scratch, schedule and
// bitmap); K3c and K4, which share that work, both need less.
bool search_accepts(uint32_t buckets, uint32_t cap) {
    if (cap > 65535 || buckets > 65535) return false;
    const size_t half = (buckets + 1) / 2, reach = (cap - 1) / 32 + 32 * ((cap + 1023) / 1024) + 2,
                 occ = (2 * cap + 31) / 32 + 2;
    const size_t words = std::max(half + 256, (size_t)kHsWords + scr_words(cap)) + half + buckets + std::max(reach, occ);
    return 4 * ((words + 3) & ~size_t(3)) <= kSearchSmemLimit;
}

int search_warps_per_cta(uint32_t buckets, uint32_t cap) {
    if (!search_accepts(buckets, cap)) return 0;
    size_t fit = kSearchSmemLimit / search_warp_smem(buckets, cap);
    return (int)(fit < (size_t)kSearchWarps ? fit : (size_t)kSearchWarps);
}

__global__ void __launch_bounds__(kSearchWarps * 32, kSearchCtasPerSm) k_search(SearchArgs a) {
    extern __shared__ __align__(16) uint32_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *mine = smem + (size_t)warp * warp_words(a.buckets, a.cap);
    const WarpSmem ws = carve(mine, a.buckets, a.cap);
    for (;;) {
        uint32_t g = 0;
        if (lane == 0) g = atomicAdd(a.queue, 1u);
        g = __shfl_sync(kFullMask, g, 0);
        if (g >= a.M) break;
        const uint32_t s = a.nsets == 1 ? 0u : find_set(a.part_base, a.nsets, g);
        if (fatal_before_search(*reinterpret_cast<volatile unsigned long long *>(&a.err[s]))) continue;
        const SetDesc &d = a.sets[s];
        const uint32_t p = g - d.part_base;
        const uint32_t code = search_partition(a, mine, ws, d, g, p, lane);
        if (code != PHOBIC_OK && lane == 0) report_error(&a.err[s], p, code);
    }
}

size_t search_group_smem(uint32_t buckets, uint32_t cap, int W) { return 4 * group_words(buckets, cap, W); }

template <int W, bool PIPE>
static cudaError_t launch_group(const SearchArgs &a, int sm_count, cudaStream_t st) {
    constexpr int groups = kSearchWarps / W;
    const size_t smem = (size_t)groups * search_group_smem(a.buckets, a.cap, W);
    if (smem > kSearchSmemLimit) return cudaErrorInvalidValue;
    cudaError_t e = allow_dynamic_smem(k_search_group<W, PIPE>, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_search_group<W, PIPE>, kSearchWarps * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    const uint64_t want = (a.M + groups - 1) / groups;
    const int grid = (int)std::min<uint64_t>(want, (uint64_t)per_sm * sm_count);
    k_search_group<W, PIPE><<<grid, kSearchWarps * 32, smem, st>>>(a);
    return cudaGetLastError();
}

SearchShape search_shape_for(uint32_t partitions, int sm_count) {
    // Measured on a B200 (the autotuner's ladder, three key sets per size, six parameter
    // sets): bucket pipelines of 8 warps are fastest up to 256 partitions, of 4 warps up to
    // 512, of 2 warps up to 1024; one warp per partition beyond.  A group must fit one wave
    // of the group kernel (2 CTAs of kSearchWarps warps per SM).
    const uint64_t wave = (uint64_t)(sm_count > 0 ? sm_count : 148) * 2 * kSearchWarps;
    SearchShape sh;
    sh.group = 1;
    if ((uint64_t)partitions * 8 <= wave && partitions <= 256) sh = SearchShape{8, true};
    else if ((uint64_t)partitions * 4 <= wave && partitions <= 512) sh = SearchShape{4, true};
    else if ((uint64_t)partitions * 2 <= wave && partitions <= 1024) sh = SearchShape{2, true};
    return sh;
}

cudaError_t launch_search(const SearchArgs &a, int sm_count, cudaStream_t st, SearchShape shape) {
    if (a.M == 0) return cudaSuccess;
    if (shape.group == 0) shape = search_shape_for(a.M, sm_count);
    const int group = shape.group;
    const bool pipeline = shape.pipeline;
    if (group == 2 || group == 4 || group == 8) {
        cudaError_t e;
        if (pipeline)
            e = group == 2 ? launch_group<2, true>(a, sm_count, st)
                : group == 4 ? launch_group<4, true>(a, sm_count, st) : launch_group<8, true>(a, sm_count, st);
        else
            e = group == 2 ? launch_group<2, false>(a, sm_count, st)
                : group == 4 ? launch_group<4, false>(a, sm_count, st) : launch_group<8, false>(a, sm_count, st);
        if (e != cudaErrorInvalidValue) return e;
        cudaGetLastError();  // the group's tables do not fit: one warp per partition
    }
    const int warps = search_warps_per_cta(a.buckets, a.cap);
    if (warps < 1) return cudaErrorInvalidValue;
    const size_t smem = (size_t)warps * search_warp_smem(a.buckets, a.cap);
    cudaError_t e = allow_dynamic_smem(k_search, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_search, warps * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    uint64_t want = (a.M + warps - 1) / warps;
    int grid = (int)std::min<uint64_t>(want, (uint64_t)per_sm * sm_count);
    k_search<<<grid, warps * 32, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace phobicb200

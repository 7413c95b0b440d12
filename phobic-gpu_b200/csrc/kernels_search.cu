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
// loads).  Larger buckets keep their first 32 keys in registers and read the others from
// the bucket-ordered copy in global memory.
//
// Two times in a comment are of two variants measured side by side when the choice was made,
// in a kernel that was otherwise that of its day; the search of 10^8 u64 keys (lambda 7,
// P 2500) now takes 4.96 ms.
#include <algorithm>
#include <type_traits>

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
//   sched [B + 2]    search schedule, in search order: start | bucket << 16; then the end (and
//                    a word that is read past it, unused)
__host__ __device__ __forceinline__ size_t warp_words(uint32_t B, uint32_t cap) {
    const size_t w = kHsWords + 2 * (size_t)bitmap_pairs(cap) + scr_words(cap) + (size_t)B + 2;
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
// The word at addr before `bit` is set in it, where `on` (else 0, and nothing is set).
__device__ __forceinline__ uint32_t atom_or_if(uint32_t addr, uint32_t bit, bool on) {
    uint32_t old;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\tmov.u32 %0, 0;\n\t"
        "@p atom.shared.or.b32 %0, [%1], %2;\n\t}"
        : "=&r"(old) : "r"(addr), "r"(bit), "r"((uint32_t)on) : "memory");
    return old;
}
__device__ __forceinline__ void red_and(uint32_t addr, uint32_t mask) {
    asm volatile("red.shared.and.b32 [%0], %1;" ::"r"(addr), "r"(mask) : "memory");
}

// Byte offset of the pair whose first word holds slot q (the pair before it holds that word
// as its second).
__device__ __forceinline__ uint32_t pair_of(uint32_t q) { return (q >> 5) << 3; }

// The bits of slot q where `on`: its own place (the one that is tested) and, apart from it, the
// second place of its word and both of its mirror q + ps; predicated, without a branch.
__device__ __forceinline__ void mark_own(uint32_t at, uint32_t bit, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p red.shared.or.b32 [%0], %1;\n\t}" ::"r"(at),
                 "r"(bit), "r"((uint32_t)on)
                 : "memory");
}
__device__ __forceinline__ void mark_copies(uint32_t occ, uint32_t q, uint32_t ps, bool on) {
    const uint32_t m = q + ps;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "@p red.shared.or.b32 [%0+-4], %1;\n\t@p red.shared.or.b32 [%2], %3;\n\t@p red.shared.or.b32 [%2+-4], %3;\n\t}"
        ::"r"(occ + pair_of(q)), "r"(1u << (q & 31)), "r"(occ + pair_of(m)), "r"(1u << (m & 31)), "r"((uint32_t)on)
        : "memory");
}
__device__ __forceinline__ void mark(uint32_t occ, uint32_t q, uint32_t ps) {
    mark_own(occ + pair_of(q), 1u << (q & 31), true);
    mark_copies(occ, q, ps, true);
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
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
    uint32_t dead0, dead1;  // the same for rounds 0 and 1: nothing, or last_dead where one is the last
    __device__ __forceinline__ static ScanRange make(uint32_t ps, int lane) {
        ScanRange r;
        r.ps = ps;
        r.rounds = (ps + 1023) / 1024;
        const int n = (int)ps - (int)(1024 * (r.rounds - 1)) - 32 * lane;
        r.last_dead = ~__funnelshift_lc(kFullMask, 0u, (uint32_t)max(n, 0));  // n >= 32: none
        r.dead0 = r.rounds == 1 ? r.last_dead : 0u;
        r.dead1 = r.rounds == 2 ? r.last_dead : 0u;
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
// DENSE: no further keys once the first four have closed every lane's window.
template <int S, int R, bool DENSE = false>
__device__ __forceinline__ uint32_t round_bad(const WarpSmem &ws, const uint32_t (&a)[S], const uint32_t (&v)[S],
                                              bool full, uint32_t bad) {
#pragma unroll
    for (int i = 0; i < S - 2; i++) {
        if (DENSE && i == 4 && __all_sync(kFullMask, bad == kFullMask)) return bad;
        bad |= window_at<256 * R>(ws, a[i], v[i]);
    }
    if (full) bad |= window_at<256 * R>(ws, a[S - 2], v[S - 2]) | window_at<256 * R>(ws, a[S - 1], v[S - 1]);
    return bad;
}

// Smallest free offset of a bucket of s <= S keys (S = 4 or 8) whose S packed slots start at the
// shared address hs (entries past the bucket repeat a slot: OR is idempotent), in a partition of at
// most three rounds, each at a constant offset from the keys' pair addresses.  Dead lanes read
// inside the padded bitmap (bitmap_pairs) and are masked.
// The masks of the rounds are held per partition: chosen in every round, with the loop over blocks
// of rounds below for every partition, the search of 10^8 u64 keys takes 5.49 instead of 5.36 ms.
template <int S, bool DENSE = false>
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
    if (round_result(round_bad<S, 0, DENSE>(ws, a, v, full, sr.dead0), 0, &o)) return o;
    if (sr.rounds == 1) return kNone;
    if (round_result(round_bad<S, 1, DENSE>(ws, a, v, full, sr.dead1), 1024, &o)) return o;
    if (sr.rounds == 2) return kNone;
    return round_result(round_bad<S, 2, DENSE>(ws, a, v, full, sr.last_dead), 2048, &o) ? o : kNone;
}

// The same for a partition of more than three rounds: three at a time (scan_quads, which forms the
// pair addresses in every round, makes the search of P = 4096 7 % slower).
template <int S>
__device__ __forceinline__ uint32_t scan_blocks(const WarpSmem &ws, uint32_t hs, uint32_t s, const ScanRange &sr,
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
template <bool DENSE = false>
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
            if (DENSE && __all_sync(kFullMask, bad == kFullMask)) break;
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
    const uint32_t a = occ + pair_of(q), bit = 1u << (q & 31);
    const uint32_t old = atom_or_if(a, bit, on);
    if (__any_sync(kFullMask, old & bit)) {
        if (on) red_and(a, ~bit);
        __syncwarp();
        return false;
    }
    mark_copies(occ, q, ps, on);
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

// Builds of at most this many keys per partition are searched by the DENSE kernel: their partitions
// need many counters, so what a failing one takes counts.  Search of 2*10^7 keys (lambda 5) at P 128 19.9 ms
// without it, 10.9 with it; at P 256 2.05 and 2.25.
constexpr uint32_t kDenseSlots = 128;
// Slots below which a bucket of S / 2 to S keys meets itself on so many pilot counters (half of them, at
// about three quarters of S keys) that the test comes before the scan: search of 10^6 keys at P 32 77.9 ms
// without, 46.2 with it; limits of twice and half as many slots make 43.8 and 46.2 of it, and 2.42 and 2.34
// of 2.50 ms at 3*10^7 (P 128, lambda 3).
constexpr uint32_t crowded(uint32_t S) { return S * S / 2; }
// The same for the group kernel, whose searches test for it beside their scan: search of 30,000 strings at
// P 64 2.52 ms without, 1.63 with it.  3 S slots for S = 16 and 32 make 176 us of 119 at 3*10^5 keys (P 128,
// lambda 3), 5 S for S = 8, whose counters are also looked at two at a time, 323 of 237 at 1000 (P 32).
constexpr uint32_t crowded_ahead(uint32_t S) { return S == 8 ? 3 * S : 5 * S; }

// Lanes per pilot counter for a bucket of s <= 32 keys: 4, 8, 16 or 32.
__device__ __forceinline__ uint32_t counter_lanes(uint32_t s) { return s <= 4 ? 4u : s <= 8 ? 8u : s <= 16 ? 16u : 32u; }
// The key that lane `lane` loads of a bucket of s <= 32 keys: lane t * S + i takes key i, lanes
// past the bucket key 0, whose slots are the padding that the scan expects.
__device__ __forceinline__ uint32_t lane_key(uint32_t s, int lane) {
    const uint32_t i = (uint32_t)lane & (counter_lanes(s) - 1u);
    return i < s ? i : 0u;
}

// Lanes whose packed slot is also that of another key of their bucket of s <= S keys under the same counter
// (lane t * S + i: key i, counter t), as a vote in which each such pair shows once at least.  S / 2 rotations
// cover all pairs and are in flight together; __match_any_sync takes 360 cycles.
template <int S>
__device__ __forceinline__ uint32_t meeting_lanes(uint32_t hk, uint32_t s, int lane) {
    const bool key = ((uint32_t)lane & (S - 1u)) < s;
    const uint32_t v = key ? hk : 0x80000000u | (uint32_t)lane;  // lanes past the bucket: values of their own
    bool meet = false;
#pragma unroll
    for (int r = 1; r <= S / 2; r++) meet |= v == __shfl_sync(kFullMask, v, lane + r, S);
    return __ballot_sync(kFullMask, meet);
}

// A bucket of at most S keys (S = 4, 8, 16 or 32; more than S / 2 of them, or S = 4), L as
// lane_key loads it.  The warp hashes 32 / S pilot counters at once (lane t * S + i holds key i
// under counter k0 + t) into hs and tests them in counter order, so a counter that fails costs
// no new hash.  Same result as trying k = 0, 1, 2, ... one at a time (search.comp:105-124).
// SMALL: the partition has at most three rounds.  DENSE: of few slots (kDenseSlots).  MEET: the counters
// of a batch that put two keys on one slot are found by one match of all slots and not scanned.
template <int S, bool SMALL, bool DENSE = false, bool MEET = false>
__device__ __forceinline__ uint32_t place_batched(const WarpSmem &ws, uint2 L, uint32_t s, const ScanRange &sr,
                                                  FastMod fm, uint32_t k_lim, int lane, uint32_t *pilot) {
    constexpr uint32_t G = 32 / S;
    const uint32_t hs_sa = (uint32_t)__cvta_generic_to_shared(ws.hs);
    const bool mine = lane < (int)s;
    uint32_t stop = min(k_lim, kDupCheckAt);  // a multiple of G, or k_lim
    uint32_t hk_next = MEET ? pack_slot(fm.mod(pilot_hash(L.x, L.y, (uint32_t)lane / S))) : 0u;
    for (uint32_t k0 = 0;; k0 += G) {
        if (k0 >= stop) {
            if (k0 >= k_lim) return PHOBIC_ERR_SEARCH_LIMIT;
            if (s > 1 && has_duplicate_key(L, s, lane)) return PHOBIC_ERR_DUPLICATE_KEY;
            stop = k_lim;
        }
        const uint32_t hk = MEET ? hk_next : pack_slot(fm.mod(pilot_hash(L.x, L.y, k0 + (uint32_t)lane / S)));
        uint32_t meet = 0;  // lanes whose slot is that of another key under their counter
        if constexpr (MEET) {
            hk_next = pack_slot(fm.mod(pilot_hash(L.x, L.y, k0 + G + (uint32_t)lane / S)));
            meet = meeting_lanes<S>(hk, s, lane);
            if (G == 1 && meet) continue;
        }
        __syncwarp();
        ws.hs[lane] = hk;
        __syncwarp();
        const uint32_t tries = min(G, k_lim - k0);
#pragma unroll 1
        for (uint32_t u = 0; u < tries; u++) {
            if (MEET && (meet >> (S * u)) & (kFullMask >> (32 - S))) continue;
            uint32_t o;
            if constexpr (S <= 8 && SMALL) o = scan_small<S, DENSE>(ws, hs_sa + 4 * S * u, s, sr, lane);
            else if constexpr (S <= 8) o = scan_blocks<S>(ws, hs_sa + 4 * S * u, s, sr, lane);
            else o = scan_quads<DENSE>(ws, hs_sa + 4 * S * u, s, sr, lane);
            if (o == kNone) continue;
            uint32_t q = unpack_slot(ws.hs[S * u + (mine ? (uint32_t)lane : 0u)]) + o;
            q = q >= sr.ps ? q - sr.ps : q;
            if (!mark_distinct(ws.occ, q, sr.ps, mine && PHB_CHECK(!mine || q < sr.ps))) continue;
            *pilot = o + sr.ps * (k0 + u);
            return PHOBIC_OK;
        }
    }
}

// ------------------------------------------------------------------ low-latency search
//
// The group kernel's warps are few, so what counts there is the length of one try's chain, not
// its instructions: all NR rounds of a partition of at most 1024 NR offsets are in flight at
// once, the collision test runs beside them, and the smallest offset comes from one warp-wide
// minimum.

// This lane's windows in all NR rounds (bad[r] bit i: offset 1024 r + 32 lane + i is taken) of a
// bucket of s keys whose packed slots start at the shared address hs, S of them (S = 4 or 8), or
// s padded to a multiple of 4 (S = 16 or 32).  For S = 4 it returns whether two of the keys share
// a slot.
template <int S, int NR>
__device__ __forceinline__ bool all_windows(const WarpSmem &ws, uint32_t hs, uint32_t s, const ScanRange &sr, int lane,
                                            uint32_t (&bad)[NR]) {
    const uint32_t lane_sa = ws.occ + 8u * lane;
#pragma unroll
    for (int r = 0; r < NR; r++) bad[r] = r == NR - 1 ? sr.last_dead : 0u;
    auto quad = [&](uint4 v, bool half) {
        const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
            if (i == 2 && half) break;
            const uint32_t a = lane_sa + (x[i] >> 5), b = lane_sa + (x[i + 1] >> 5);
            bad[0] |= window_at<0>(ws, a, x[i]) | window_at<0>(ws, b, x[i + 1]);
            if constexpr (NR > 1) bad[1] |= window_at<256>(ws, a, x[i]) | window_at<256>(ws, b, x[i + 1]);
            if constexpr (NR > 2) bad[2] |= window_at<512>(ws, a, x[i]) | window_at<512>(ws, b, x[i + 1]);
        }
    };
    if constexpr (S == 4) {
        const uint4 v = lds128(hs);
        quad(v, s <= 2);
        return (s > 1 && v.x == v.y) || (s > 2 && (v.x == v.z || v.y == v.z)) ||
               (s > 3 && (v.x == v.w || v.y == v.w || v.z == v.w));
    } else if constexpr (S == 8) {
        quad(lds128(hs), false);
        quad(lds128(hs + 16), s <= S - 2);
    } else {
        const uint32_t hs_end = hs + 4 * s;
#pragma unroll 2
        for (uint32_t q = hs; q < hs_end; q += 16) quad(lds128(q), false);
    }
    return false;
}

// Which of V counters have an open window, as bits: their buckets' packed slots, S = 4 or 8 of them each,
// start at the shared address hs, in a partition of one round.  All loads of the V counters are in flight together.
template <int S, int V>
__device__ __forceinline__ uint32_t open_counters(const WarpSmem &ws, uint32_t hs, const ScanRange &sr, int lane) {
    const uint32_t lane_sa = ws.occ + 8u * lane;
    uint4 x[V * S / 4];
#pragma unroll
    for (int i = 0; i < V * S / 4; i++) x[i] = lds128(hs + 16 * i);
    uint32_t bad[V];
#pragma unroll
    for (int v = 0; v < V; v++) {
        bad[v] = sr.last_dead;
#pragma unroll
        for (int i = v * S / 4; i < (v + 1) * S / 4; i++) {
            bad[v] |= window_at<0>(ws, lane_sa + (x[i].x >> 5), x[i].x) | window_at<0>(ws, lane_sa + (x[i].y >> 5), x[i].y);
            bad[v] |= window_at<0>(ws, lane_sa + (x[i].z >> 5), x[i].z) | window_at<0>(ws, lane_sa + (x[i].w >> 5), x[i].w);
        }
    }
    uint32_t open = 0;
#pragma unroll
    for (int v = 0; v < V; v++) open |= __any_sync(kFullMask, bad[v] != kFullMask) ? 1u << v : 0u;
    return open;
}

// The warp's smallest free offset in these windows (kNone: none).
template <int NR>
__device__ __forceinline__ uint32_t smallest_offset(const uint32_t (&bad)[NR], int lane) {
    uint32_t open = ~bad[NR - 1], at = 1024u * (NR - 1);  // the lane's first round with a free offset
#pragma unroll
    for (int r = NR - 2; r >= 0; r--) {
        const bool here = bad[r] != kFullMask;
        open = here ? ~bad[r] : open;
        at = here ? 1024u * r : at;
    }
    return __reduce_min_sync(kFullMask, open ? at + 32u * lane + __ffs(open) - 1 : kNone);
}

// A search of the bucket pipeline: pilot counter, offset, the lane's slot under that counter
// before the offset (lanes below the bucket's size), and the windows it was found in.
template <int NR>
struct Seek {
    uint32_t kb, k, o, h;
    uint32_t bad[NR ? NR : 1];
    uint32_t tested, apart;  // seek_crowded: the batch that was tested for keys that meet, its counters without
};

// The search of place_batched as the bucket pipeline runs it: nothing is marked, and it can be
// resumed.  Finds the smallest pilot counter >= k, then the smallest offset, that the bitmap
// allows; kb is the first counter of the batch whose slots hs holds (kNone: none yet), so a
// second call with the same k tests that counter again without a hash.  NR = 0: any number of
// rounds, one after the other.
template <int S, int NR, bool FEW>
__device__ __forceinline__ uint32_t seek_batched(const WarpSmem &ws, uint32_t *hs, uint2 L, uint32_t s,
                                                 const ScanRange &sr, FastMod fm, uint32_t k_lim, int lane, Seek<NR> *f) {
    constexpr uint32_t G = 32 / S;
    const uint32_t hs_sa = (uint32_t)__cvta_generic_to_shared(hs);
    const bool mine = lane < (int)s;
    const uint32_t from = f->k;
#pragma unroll 1
    for (;; ++f->k) {
        if (f->k >= k_lim) return PHOBIC_ERR_SEARCH_LIMIT;
        const uint32_t u = f->k % G;
        if (f->k - u != f->kb) {  // u = 0: a batch is entered at its first counter
            if (f->k == kDupCheckAt && s > 1 && has_duplicate_key(L, s, lane)) return PHOBIC_ERR_DUPLICATE_KEY;
            f->kb = f->k;
            const uint32_t hk = pack_slot(fm.mod(pilot_hash(L.x, L.y, f->k + (uint32_t)lane / S)));
            __syncwarp();
            hs[lane] = hk;
        }
        __syncwarp();
        // One counter has failed: the next ones are looked at V at a time, up to the first with an open window
        // (V divides the batch, and counters past k_lim end the search above).
        if constexpr (FEW && S <= 8) {
            constexpr uint32_t V = 16 / S;
            if (f->k != from && u % V == 0) {
                const uint32_t open = open_counters<S, V>(ws, hs_sa + 4 * S * u, sr, lane);
                if (!(open & 1u)) {
                    f->k += open ? __ffs(open) - 2 : V - 1;
                    continue;
                }
            }
        }
        const uint32_t own = hs[S * u + (mine ? (uint32_t)lane : 0u)];
        bool meet = false;
        if constexpr (NR > 0) meet = all_windows<S, NR>(ws, hs_sa + 4 * S * u, s, sr, lane, f->bad);
        else if constexpr (S <= 8) f->o = scan_blocks<S>(ws, hs_sa + 4 * S * u, s, sr, lane);
        else f->o = scan_quads(ws, hs_sa + 4 * S * u, s, sr, lane);
        f->h = unpack_slot(own);
        if constexpr (S == 4 && NR > 0) {
            f->o = smallest_offset<NR>(f->bad, lane);
        } else {
            // Two keys on one slot: their bits meet in the warp's collision scratch (left clear).
            const bool on = mine && s > 1 && PHB_CHECK(f->h < sr.ps);
            const uint32_t bit = 1u << (f->h & 31), at = (uint32_t)__cvta_generic_to_shared(ws.scr) + 4 * (f->h >> 5);
            const uint32_t old = atom_or_if(at, bit, on) & bit;
            if constexpr (NR > 0) f->o = smallest_offset<NR>(f->bad, lane);
            meet = __any_sync(kFullMask, old);
            if (on) ws.scr[f->h >> 5] = 0;
            __syncwarp();
        }
        if (!meet && f->o != kNone) return PHOBIC_OK;
    }
}
// seek_batched for a bucket that meets itself on most counters, in a partition of few slots: the counters
// of a batch that do are found at once and passed over.
template <int S>
__device__ __forceinline__ uint32_t seek_crowded(const WarpSmem &ws, uint32_t *hs, uint2 L, uint32_t s,
                                                 const ScanRange &sr, FastMod fm, uint32_t k_lim, int lane, Seek<1> *f) {
    constexpr uint32_t G = 32 / S;
    const uint32_t hs_sa = (uint32_t)__cvta_generic_to_shared(hs);
#pragma unroll 1
    for (;; ++f->k) {
        if (f->k >= k_lim) return PHOBIC_ERR_SEARCH_LIMIT;
        uint32_t u = f->k % G;
        if (f->k - u != f->kb) {  // u = 0
            if (f->k == kDupCheckAt && s > 1 && has_duplicate_key(L, s, lane)) return PHOBIC_ERR_DUPLICATE_KEY;
            f->kb = f->k;
            const uint32_t hk = pack_slot(fm.mod(pilot_hash(L.x, L.y, f->k + (uint32_t)lane / S)));
            __syncwarp();
            hs[lane] = hk;
        }
        __syncwarp();
        if (f->tested != f->kb) {
            f->tested = f->kb;
            const uint32_t meet = meeting_lanes<S>(hs[lane], s, lane);
            f->apart = 0;
#pragma unroll
            for (uint32_t t = 0; t < G; t++) f->apart |= (meet >> (S * t)) & (kFullMask >> (32 - S)) ? 0u : 1u << t;
        }
        const uint32_t next = f->apart >> u;
        const uint32_t skip = next ? __ffs(next) - 1 : G - u;
        f->k += skip;
        u += skip;
        if (u == G) {
            --f->k;
            continue;
        }
        if (f->k >= k_lim) return PHOBIC_ERR_SEARCH_LIMIT;
        all_windows<S, 1>(ws, hs_sa + 4 * S * u, s, sr, lane, f->bad);
        if (__all_sync(kFullMask, f->bad[0] == kFullMask)) continue;
        f->o = smallest_offset<1>(f->bad, lane);
        f->h = unpack_slot(hs[S * u + (lane < (int)s ? (uint32_t)lane : 0u)]);
        return PHOBIC_OK;
    }
}
template <int NR, bool FEW>
__device__ __forceinline__ uint32_t seek_any(const WarpSmem &ws, uint32_t *hs, uint2 L, uint32_t s, const ScanRange &sr,
                                             FastMod fm, uint32_t k_lim, int lane, Seek<NR> *f) {
    if constexpr (FEW) {
        if (s > 16 && sr.ps < crowded_ahead(32)) return seek_crowded<32>(ws, hs, L, s, sr, fm, k_lim, lane, f);
        if (s > 8 && s <= 16 && sr.ps < crowded_ahead(16)) return seek_crowded<16>(ws, hs, L, s, sr, fm, k_lim, lane, f);
        if (s > 4 && s <= 8 && sr.ps < crowded_ahead(8)) return seek_crowded<8>(ws, hs, L, s, sr, fm, k_lim, lane, f);
    }
    if (s <= 4) return seek_batched<4, NR, FEW>(ws, hs, L, s, sr, fm, k_lim, lane, f);
    if (s <= 8) return seek_batched<8, NR, FEW>(ws, hs, L, s, sr, fm, k_lim, lane, f);
    if (s <= 16) return seek_batched<16, NR, FEW>(ws, hs, L, s, sr, fm, k_lim, lane, f);
    return seek_batched<32, NR, FEW>(ws, hs, L, s, sr, fm, k_lim, lane, f);
}

// One bucket of more than 32 keys (a few per partition).  Each try hashes chunk by chunk and
// stops at the first chunk that repeats a slot: buckets of 100 to 160 keys are rejected about 37
// times per partition (10^8 u64 keys, lambda 7, P 2500), after 62 keys on average.  In partitions of few
// slots nearly every try ends at the first chunk, after thousands of tries in the worst of them, and the
// build lasts as long as those take: the first chunk's keys are in registers, and its slots under
// the next counter are formed while this counter's are tested.  The other keys are read
// from the bucket-ordered copy on every try: staging them in shared memory takes that much
// from the L1 that the copy and the schedule are read through, and was slower (search 6.18
// against 6.06 ms).
template <bool DENSE>
__device__ __forceinline__ uint32_t place_large(const WarpSmem &ws, const uint2 *src, uint32_t s, const ScanRange &sr,
                                                FastMod fm, uint32_t k_lim, int lane, uint32_t *pilot) {
    const uint32_t padded = (s + 3) & ~3u, ps = sr.ps;
    const uint32_t hs_sa = (uint32_t)__cvta_generic_to_shared(ws.hs);
    // The collision test of one key (its bit in the warp's scratch, clear before).
    auto taken = [&](uint32_t h) {
        const uint32_t bit = 1u << (h & 31);
        return PHB_CHECK(h < ps) && (atomicOr(&ws.scr[h >> 5], bit) & bit) != 0;
    };
    const uint2 key0 = src[lane];
    uint32_t h_next = fm.mod(pilot_hash(key0.x, key0.y, 0u));
    for (uint32_t k = 0; k < k_lim; k++) {
        if (k == kDupCheckAt) {
            bool d = false;
            for (uint32_t t = 0; t + 1 < s; t++) {
                uint2 kt = src[t];
                for (uint32_t i = lane; i < s; i += 32) d |= i > t && src[i].x == kt.x && src[i].y == kt.y;
            }
            if (__any_sync(kFullMask, d)) return PHOBIC_ERR_DUPLICATE_KEY;
        }
        const uint32_t h0 = h_next;
        const bool d0 = taken(h0);
        h_next = fm.mod(pilot_hash(key0.x, key0.y, k + 1));
        if (__any_sync(kFullMask, d0)) {
            if (PHB_CHECK(h0 < ps)) ws.scr[h0 >> 5] = 0;
            __syncwarp();
            continue;
        }
        ws.hs[lane] = pack_slot(h0);
        bool dup = false;
        uint32_t done = 32;  // keys hashed (and marked in the collision scratch)
        for (uint32_t c0 = 32; c0 < s && !dup; c0 += 32) {
            const uint32_t i = c0 + lane;
            bool d = false;
            if (i < s) {
                const uint2 key = src[i];
                const uint32_t h = fm.mod(pilot_hash(key.x, key.y, k));
                ws.hs[i] = pack_slot(h);
                d = taken(h);
            }
            dup = __any_sync(kFullMask, d);
            done = c0 + 32;
        }
        for (uint32_t i = lane; i < s && i < done; i += 32) ws.scr[unpack_slot(ws.hs[i]) >> 5] = 0;
        __syncwarp();
        if (dup) continue;
        if (s + lane < padded) ws.hs[s + lane] = ws.hs[0];
        __syncwarp();
        const uint32_t o = scan_quads<DENSE>(ws, hs_sa, s, sr, lane);
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

// What the search of a partition starts from, brought in by `threads` threads of which this is
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

// The buckets of one key end the search order, and when they begin there are exactly as many free
// slots left as keys.  A single key never collides and every offset to a free slot is valid, so its
// pilot counter is 0 and its offset the distance to the next free slot.  With the free slots in
// registers a key takes one broadcast, one warp minimum and a compare (18 instructions for up to 64
// of them) instead of a search of the bitmap (about 185): the search takes 5.83 against 6.06 ms at
// 10^8 u64 keys (lambda 7, 38 such buckets of 340 per partition), 2.35 against 2.57 ms at 5*10^7
// (lambda 5, 66 of 371), 47 against 72 us for 1000 keys on 8 warps.
constexpr uint32_t kMaxSingles = 128;
constexpr uint32_t kDeadSlot = 0x80000000u;  // farther than any slot from any other

// Number of buckets of one key at the end of the schedule, at most kMaxSingles.
__device__ __forceinline__ uint32_t count_singles(const WarpSmem &ws, uint32_t nonempty, int lane) {
    uint32_t n = 0;
#pragma unroll
    for (uint32_t r = 0; r < kMaxSingles / 32; r++) {
        const uint32_t i = 32 * r + (uint32_t)lane;  // from the end
        bool one = false;
        if (i < nonempty) {
            const uint32_t j = nonempty - 1 - i;
            one = ((ws.sched[j + 1] - ws.sched[j]) & 0xFFFFu) == 1u;
        }
        n += __popc(__ballot_sync(kFullMask, one));
    }
    return n;
}

template <int R>
__device__ __forceinline__ void place_singles_in(const WarpSmem &ws, const uint2 *so, uint32_t first, uint32_t n,
                                                 uint32_t ps, FastMod fm, int lane, uint32_t *pil, size_t pstride) {
    uint32_t slot[R];
#pragma unroll
    for (int r = 0; r < R; r++) slot[r] = 32 * r + lane < (int)n ? ws.hs[32 * r + lane] : kDeadSlot;
    const uint2 *src = so + (ws.sched[first] & 0xFFFFu);
    for (uint32_t c = 0; c < n; c += 32) {
        const uint32_t i = c + (uint32_t)lane;
        const uint2 key = src[i < n ? i : 0];
        const uint32_t h = fm.mod(pilot_hash(key.x, key.y, 0u)), b = ws.sched[first + (i < n ? i : 0)] >> 16;
        uint32_t mine = 0;
        const uint32_t m = min(n - c, 32u);
        for (uint32_t t = 0; t < m; t++) {
            const uint32_t from = __shfl_sync(kFullMask, h, t);
            uint32_t d[R], best = 0xFFFFFFFFu;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint32_t x = slot[r] - from;  // wraps below 0: then the distance is x + ps
                d[r] = min(x, x + ps);
                best = min(best, d[r]);
            }
            const uint32_t o = __reduce_min_sync(kFullMask, best);
#pragma unroll
            for (int r = 0; r < R; r++) slot[r] = d[r] == o ? kDeadSlot : slot[r];
            if (lane == (int)t) mine = o;
        }
        if (i < n) pil[(size_t)b * pstride] = mine;
    }
}

// The last n <= kMaxSingles buckets of the schedule, of one key each, from bucket `first` on.
__device__ __forceinline__ void place_singles(const WarpSmem &ws, const uint2 *so, uint32_t first, uint32_t n,
                                              uint32_t ps, FastMod fm, int lane, uint32_t *pil, size_t pstride) {
    if (n == 0) return;
    // The free slots into hs.
    uint32_t have = 0;
    __syncwarp();
    for (uint32_t w0 = 0; w0 < ps; w0 += 1024) {
        const uint32_t w = w0 + 32u * lane;
        uint32_t open = 0;
        if (w < ps) {
            open = ~lds32(ws.occ + pair_of(w));
            if (ps - w < 32) open &= (1u << (ps - w)) - 1u;
        }
        uint32_t at = __popc(open), incl = at;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(kFullMask, incl, d);
            if (lane >= d) incl += t;
        }
        at = have + incl - at;
        for (; open; open &= open - 1, at++)
            if (PHB_CHECK(at < n)) ws.hs[at] = w + __ffs(open) - 1;
        have += __shfl_sync(kFullMask, incl, 31);
    }
    __syncwarp();
    if (n <= 64) place_singles_in<2>(ws, so, first, n, ps, fm, lane, pil, pstride);
    else place_singles_in<kMaxSingles / 32>(ws, so, first, n, ps, fm, lane, pil, pstride);
    __syncwarp();
}

// Where a partition's search stands: bucket j of the schedule, its entry and the next one, its size
// and (at most 32 keys) its keys as lane_key loads them.
struct Cursor {
    uint32_t j, sc, sc1, s;
    uint2 L;
};
// To the next bucket; past the last one what is read means nothing.
__device__ __forceinline__ void advance(const WarpSmem &ws, Cursor &c) {
    c.j++;
    c.sc = c.sc1;
    c.sc1 = ws.sched[c.j + 1];
    c.s = (c.sc1 - c.sc) & 0xFFFFu;
}

// The buckets of more than S / 2 and at most S keys (S = 4: of at most 4) from c on: the search
// order is by size, so the buckets of a class follow one another.  A loop per class needs no choice
// of the class per bucket and knows the lanes' keys; the next bucket's are loaded during the search.
// One loop for all of them takes 5.83 against 5.51 ms at 10^8 u64 keys (lambda 7), 2.46 against
// 2.29 ms at 5*10^7 (lambda 6).
template <int S, bool SMALL = true, bool DENSE = false, bool MEET = false>
__device__ __forceinline__ uint32_t search_class(const WarpSmem &ws, const uint2 *so, const ScanRange &sr, FastMod fm,
                                                 uint32_t k_lim, uint32_t searched, int lane, Cursor &c, uint32_t *pil,
                                                 size_t pstride) {
    while (c.j < searched && (S == 4 || c.s > S / 2)) {
        const uint32_t s = c.s, b = c.sc >> 16;
        const uint2 L = c.L;
        advance(ws, c);
        if (c.j < searched) {
            const uint32_t i = S == 4 || c.s > S / 2 ? min((uint32_t)lane & (S - 1u), c.s - 1) : lane_key(c.s, lane);
            c.L = so[(c.sc & 0xFFFFu) + i];
        }
        uint32_t pilot = 0;
        const uint32_t code = place_batched<S, SMALL, DENSE, MEET>(ws, L, s, sr, fm, k_lim, lane, &pilot);
        if (code != PHOBIC_OK) return code;
        if (lane == 0) pil[(size_t)b * pstride] = pilot;
    }
    return PHOBIC_OK;
}

// One partition's pilots.
template <bool DENSE>
__device__ __forceinline__ uint32_t search_partition(const SearchArgs &a, uint32_t *w, const WarpSmem &ws,
                                                     const SetDesc &d, uint32_t g, uint32_t p, int lane) {
    const uint32_t nonempty = a.part_state[g];
    if (nonempty & kPartSkipped) return nonempty & ~kPartSkipped;
    const uint32_t base = a.G[g];
    const uint32_t ps = a.G[g + 1] - base;
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
    const uint32_t singles = count_singles(ws, nonempty, lane), searched = nonempty - singles;
    // sched[nonempty] holds the end, so a bucket's size is the distance to the next start.
    Cursor c;
    c.j = 0;
    c.sc = ws.sched[0], c.sc1 = ws.sched[1];
    c.s = (c.sc1 - c.sc) & 0xFFFFu;
    uint32_t code = PHOBIC_OK;
    for (; c.j < searched && c.s > 32 && code == PHOBIC_OK;) {
        const uint32_t s = c.s, b = c.sc >> 16, st = c.sc & 0xFFFFu;
        advance(ws, c);
        uint32_t pilot = 0;
        code = place_large<DENSE>(ws, so + st, s, sr, fm, k_lim, lane, &pilot);
        if (code == PHOBIC_OK && lane == 0 && PHB_CHECK(b < a.buckets)) pil[(size_t)b * pstride] = pilot;
    }
    if (c.j < searched) c.L = so[(c.sc & 0xFFFFu) + lane_key(c.s, lane)];
    // A class whose buckets meet themselves on many counters, in this partition, is searched with MEET.
    auto dense_class = [&](auto size) {
        constexpr int S = decltype(size)::value;
        if (code != PHOBIC_OK) return;
        code = ps < crowded(S) ? search_class<S, true, true, true>(ws, so, sr, fm, k_lim, searched, lane, c, pil, pstride)
                               : search_class<S, true, true>(ws, so, sr, fm, k_lim, searched, lane, c, pil, pstride);
    };
    if constexpr (DENSE) {
        if (sr.rounds <= 3) {
            dense_class(std::integral_constant<int, 32>{});
            dense_class(std::integral_constant<int, 16>{});
            dense_class(std::integral_constant<int, 8>{});
        }
    }
    if (code == PHOBIC_OK) code = search_class<32>(ws, so, sr, fm, k_lim, searched, lane, c, pil, pstride);
    if (code == PHOBIC_OK) code = search_class<16>(ws, so, sr, fm, k_lim, searched, lane, c, pil, pstride);
    if (sr.rounds <= 3) {
        if (code == PHOBIC_OK) code = search_class<8>(ws, so, sr, fm, k_lim, searched, lane, c, pil, pstride);
        if (code == PHOBIC_OK) code = search_class<4>(ws, so, sr, fm, k_lim, searched, lane, c, pil, pstride);
    } else {
        if (code == PHOBIC_OK) code = search_class<8, false>(ws, so, sr, fm, k_lim, searched, lane, c, pil, pstride);
        if (code == PHOBIC_OK) code = search_class<4, false>(ws, so, sr, fm, k_lim, searched, lane, c, pil, pstride);
    }
    if (code != PHOBIC_OK) return code;
    place_singles(ws, so, searched, singles, ps, fm, lane, pil, pstride);
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

// The turn of the bucket pipeline: a hardware barrier per warp that its predecessor arrives at
// and the warp waits on (64 threads).
__device__ __forceinline__ void turn_wait(uint32_t id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void turn_pass(uint32_t id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }

// Per-warp scratch of warps 1..W-1 of a group (warp 0 uses its place in carve()).
__host__ __device__ __forceinline__ size_t group_extra_words(uint32_t cap) {
    return ((size_t)kHsWords + scr_words(cap) + 3) & ~size_t(3);
}
// Exchange words: [2 parities][W] outcomes of the k-split steps and the control words (job,
// nonempty, status; padded).
__host__ __device__ __forceinline__ size_t group_xch_words(int W) { return ((size_t)2 * W + 4 + 3) & ~size_t(3); }
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
    const uint32_t o = s <= 4   ? scan_blocks<4>(ws, hs_sa, s, sr, lane)
                       : s <= 8 ? scan_blocks<8>(ws, hs_sa, s, sr, lane)
                                : scan_quads(ws, hs_sa, s, sr, lane);
    if (o == kNone || !slots_distinct(ws.scr, hk, mine && PHB_CHECK(!mine || hk < sr.ps))) return kTryNone;
    *o_out = o;
    return kTryFound;
}

// Keys i = 32 c + lane of a bucket of at most 32 C keys (zero past its end).
template <int C>
__device__ __forceinline__ void load_keys(uint2 (&key)[C], const uint2 *src, uint32_t s, int lane) {
#pragma unroll
    for (int c = 0; c < C; c++) key[c] = 32 * c + lane < (int)s ? src[32 * c + lane] : make_uint2(0, 0);
}

// One try of pilot counter k for a bucket of more than 32 keys: all chunks are hashed side by side
// (the collision test of place_large, without its early end: here the chain counts).
template <int C>
__device__ __forceinline__ uint32_t try_large(const WarpSmem &ws, const uint2 (&key)[C], uint32_t s, const ScanRange &sr,
                                              FastMod fm, uint32_t k, int lane, uint32_t *o_out) {
    uint32_t h[C], old = 0;
#pragma unroll
    for (int c = 0; c < C; c++) h[c] = fm.mod(pilot_hash(key[c].x, key[c].y, k));
#pragma unroll
    for (int c = 0; c < C; c++)
        if (32 * c + lane < (int)s && PHB_CHECK(h[c] < sr.ps))
            old |= atomicOr(&ws.scr[h[c] >> 5], 1u << (h[c] & 31)) & (1u << (h[c] & 31));
    const bool meet = __any_sync(kFullMask, old);
#pragma unroll
    for (int c = 0; c < C; c++)
        if (32 * c + lane < (int)s && PHB_CHECK(h[c] < sr.ps)) ws.scr[h[c] >> 5] = 0;
    __syncwarp();
    if (meet) return kTryNone;
#pragma unroll
    for (int c = 0; c < C; c++)  // past the end: any slot of the bucket, as padding
        if (32 * c < (int)s) ws.hs[32 * c + lane] = pack_slot(__shfl_sync(kFullMask, h[c], 32 * c + lane < (int)s ? lane : 0));
    __syncwarp();
    const uint32_t hs_sa = (uint32_t)__cvta_generic_to_shared(ws.hs);
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

// One bucket in k-split steps by all W warps of a group; C = 1 for at most 32 keys.  Marks the
// winning slots (every warp: the marks are idempotent).  Returns a status; *pilot when it is OK.
template <int W, int C>
__device__ __forceinline__ uint32_t ksplit_bucket(const WarpSmem &ws, const uint2 *src, uint32_t s, const ScanRange &sr,
                                                  FastMod fm, uint32_t k_lim, uint32_t *xch, uint32_t *par, int w,
                                                  int lane, uint32_t bar_id, uint32_t *pilot) {
    uint2 key[C];
    if constexpr (C == 1) key[0] = src[lane_key(s, lane)];
    else load_keys(key, src, s, lane);
#pragma unroll 1
    for (uint32_t k0 = 0;; k0 += W) {
        const uint32_t k = k0 + w;
        uint32_t code = kTryNone, o = 0;
        if (k >= k_lim) code = kTryLimit;
        else if (k == kDupCheckAt && s > 1 && (C == 1 ? has_duplicate_key(key[0], s, lane) : has_duplicate_key_src(src, s, lane)))
            code = kTryDup;
        else if constexpr (C == 1) code = try_small(ws, s, sr, fm.mod(pilot_hash(key[0].x, key[0].y, k)), lane, &o);
        else code = try_large<C>(ws, key, s, sr, fm, k, lane, &o);
        if (lane == 0) xch[*par * W + w] = (code << 16) | (o & 0xFFFFu);
        group_bar(bar_id, 32 * W);
        uint32_t win = kTryNone << 16, v = 0;
#pragma unroll
        for (int i = W - 1; i >= 0; i--) {
            const uint32_t x = xch[*par * W + i];
            if ((x >> 16) != kTryNone) win = x, v = i;
        }
        *par ^= 1u;
        const uint32_t wcode = win >> 16;
        if (wcode == kTryNone) continue;
        if (wcode != kTryFound) return wcode == kTryDup ? PHOBIC_ERR_DUPLICATE_KEY : PHOBIC_ERR_SEARCH_LIMIT;
        const uint32_t kw = k0 + v, ow = win & 0xFFFFu;
#pragma unroll
        for (int c = 0; c < C; c++) {
            if (32 * c + lane < (int)s) {
                uint32_t q = fm.mod(pilot_hash(key[c].x, key[c].y, kw)) + ow;
                q = q >= sr.ps ? q - sr.ps : q;
                if (PHB_CHECK(q < sr.ps)) mark(ws.occ, q, sr.ps);
            }
        }
        __syncwarp();
        *pilot = ow + sr.ps * kw;
        return PHOBIC_OK;
    }
}

// Partitions of few slots (FEW) have a pipeline of their own: most of the windows that a search saw are stale
// by its turn, and most counters fail.  The same code for all partitions makes the search of 1000 keys
// in one partition 50.2 us instead of 47.5, of 2,000 79.5 instead of 77.9.
constexpr uint32_t kFewSlots = 768;
// FEW: offsets of a bucket's windows that are taken on its turn before the windows are read again (one
// look at the slots and one reduction each; reading them anew takes about three times as long).  In
// partitions of few slots nearly all offsets of the first buckets' windows are gone by their turn: with the windows
// walked to their end the search of 1000 keys takes 189 us at P 256 and 177 at P 128, with 8, 4, 2 and 1
// steps 52, 46, 40 and 36 at P 256 (and up to 4 % more at P 2048, where steps are few, with 1 and 2).
constexpr uint32_t kStaleSteps = 4;

// The bucket pipeline of a group from bucket `first` on (see k_search_group); NR as in
// seek_batched.
template <int W, int NR, bool FEW = false>
__device__ __forceinline__ void pipeline(const WarpSmem &ws, const uint2 *so, const ScanRange &sr, FastMod fm,
                                         uint32_t k_lim, uint32_t first, uint32_t nonempty, int w, int lane,
                                         uint32_t turn_id, uint32_t next_id, volatile uint32_t *status,
                                         uint32_t *pil, size_t pstride) {
    // Ahead of the warp's bucket: the schedule of its third next bucket is read, the keys of the
    // second next one, and the first batch of slots of the next one is hashed, into one half of hs,
    // while the warp's bucket waits for its turn with the other.
    struct Ahead {
        uint32_t sc, s;
        uint2 L;
    } n1{0, 0, make_uint2(0, 0)}, n2 = n1;
    uint32_t sc3 = 0, end3 = 0;
    auto read = [&](uint32_t j) {
        if (j >= nonempty) return;
        sc3 = ws.sched[j];
        end3 = ws.sched[j + 1];
    };
    auto fetch = [&](uint32_t j) {
        if (j >= nonempty) return;
        n2.sc = sc3;
        n2.s = (end3 - sc3) & 0xFFFFu;
        n2.L = so[(sc3 & 0xFFFFu) + lane_key(n2.s, lane)];
    };
    auto hash_first = [&](uint32_t *hs) {
        hs[lane] = pack_slot(fm.mod(pilot_hash(n1.L.x, n1.L.y, (uint32_t)lane / counter_lanes(n1.s))));
    };
    read(first + w);
    fetch(first + w);
    n1 = n2;
    read(first + w + W);
    fetch(first + w + W);
    read(first + w + 2 * W);
    uint32_t half = 0;
    if (first + w < nonempty) hash_first(ws.hs);
#pragma unroll 1
    for (uint32_t j = first + w; j < nonempty; j += W, half ^= 32u) {
        const uint32_t s = n1.s, b = n1.sc >> 16;
        const uint2 L = n1.L;
        n1 = n2;
        fetch(j + 2 * W);
        read(j + 3 * W);
        Seek<NR> f;
        f.kb = f.k = f.o = f.h = 0;
        f.tested = kNone;
        // One lane reads the status, which another warp may be writing: the warp agrees on what it saw.
        uint32_t st = __shfl_sync(kFullMask, lane == 0 ? *status : 0u, 0), q = 0, at = 0, bit = 0;
        bool turn = false, seek = st == PHOBIC_OK, on = false;
        uint32_t gone = 0;
#pragma unroll 1
        for (;;) {
            if (seek) st = seek_any<NR, FEW>(ws, ws.hs + half, L, s, sr, fm, k_lim, lane, &f);
            on = lane < (int)s && st == PHOBIC_OK && PHB_CHECK(f.h < sr.ps && f.o < sr.ps);
            q = f.h + f.o;
            q = q >= sr.ps ? q - sr.ps : q;
            at = on ? ws.occ + pair_of(q) : ws.occ;
            bit = on ? 1u << (q & 31) : 0u;
            if (!turn) {
                if (j + W < nonempty) hash_first(ws.hs + (half ^ 32u));
                if (j > first) turn_wait(turn_id);
                turn = true;
            }
            if (!__any_sync(kFullMask, lds32(at) & bit)) break;
            // An earlier bucket took a slot since: the next free offset of the same windows or, when
            // a few of them were gone too, of the windows as they are now, or the next counter.
            seek = true;
            if constexpr (NR > 0) {
                if (!FEW || ++gone % kStaleSteps != 0) {
#pragma unroll
                    for (int r = 0; r < NR; r++)
                        if (f.o >> 5 == (uint32_t)(32 * r + lane)) f.bad[r] |= 1u << (f.o & 31);
                    f.o = smallest_offset<NR>(f.bad, lane);
                    seek = f.o == kNone;
                    if (seek) ++f.k;
                }
            }
        }
        mark_own(at, bit, on);
        if (st != PHOBIC_OK && lane == 0 && *status == PHOBIC_OK) *status = st;
        __syncwarp();
        if (j + 1 < nonempty) turn_pass(next_id);
        mark_copies(ws.occ, q, sr.ps, on);
        if (st == PHOBIC_OK && lane == 0) pil[(size_t)b * pstride] = f.o + sr.ps * f.k;
    }
}

// Group kernel: kSearchWarps / W groups per CTA, each a persistent searcher over the
// partition queue; all W warps of a group search a partition's buckets in k-split steps.
// Small builds leave most SMs idle, so the group kernel is not held to the one-warp
// kernel's 4 CTAs per SM (64 registers): 2 CTAs per SM keep it free of spills.
// Bucket pipeline (PIPE): the buckets of at most 32 keys (the tail of the search order) go to the
// warps in turn.  A warp searches its bucket (smallest k, then smallest o) on the bitmap as it
// stands, without marking, and then waits for its turn: the arrival of the warp that holds the
// bucket before.  On its turn it tests its slots where the earlier buckets marked them, takes the
// next free offset of the windows it saw (then the next counters) while one of them is taken, marks
// them, and passes the turn on; the
// bitmap's copies of the marks (second words of pairs, mirrors), which only searches read, follow
// after.  That keeps the sequential answer: the bitmap only gains occupied slots, so what was
// rejected stays rejected, a pair that a search found without some marks fails the test, and the
// first pair that passes it is the smallest.  A pilot limit or duplicate keys found on an earlier
// state hold on the later one too; the first bucket in order that fails sets the partition's
// status, and the turns go round without searches from then on.
// From bucket to bucket the chain is a hardware barrier (34 cycles from arrival to wake-up; a
// polled word takes 120), a look at the slots, a vote and one reduction (25 cycles each).
// Against the step pipeline before it (W searches, barrier, commits by one warp up to the first
// conflict, barrier; keys loaded at the start of a step) the search takes 59 against 143 us for
// 1000 keys, 104 against 205 for 98,765 (lambda 6, P 2048), 127 against 264 for 10^6 (lambda 5).
// With 3 CTAs per SM (80 registers, spills) it is 12 to 20 % slower.
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
    uint32_t *ctl = xch + 2 * W;  // [0] job, [1] nonempty, [2] status of the pipeline
    const uint32_t turn_id = 1 + kSearchWarps / W + (uint32_t)warp;  // this warp's turn; group barriers before
    const uint32_t next_id = 1 + kSearchWarps / W + (uint32_t)(grp * W + (w + 1) % W);
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
            ctl[2] = PHOBIC_OK;
        }
        group_bar(bar_id, bar_n);
        const uint32_t nonempty = ctl[1];
        if (nonempty != 0xFFFFFFFFu) {
            const uint32_t base = a.G[g];
            const uint32_t ps = a.G[g + 1] - base;
            const uint2 *so = a.sorted + base;
            uint32_t *pil = d.pilots + p;
            const size_t pstride = d.partitions;
            load_partition(a, gbase, ws0, base, ps, nonempty, (uint32_t)(32 * w + lane), bar_n);
            if (w > 0)
                for (uint32_t i = lane; i < scr_words(a.cap); i += 32) ws.scr[i] = 0;
            // The keys of the large buckets, which come first, into L1 (16 keys a line).
            const uint32_t line = 16 * (uint32_t)(32 * w + lane);
            if (line < ps) asm volatile("{\n\t.reg .b32 t;\n\tld.global.u32 t, [%0];\n\t}" ::"l"(so + line));
            group_bar(bar_id, bar_n);
            const FastMod fm = FastMod::make(ps);
            const ScanRange sr = ScanRange::make(ps, lane);
            uint32_t k_lim = 0x80000000u / ps;
            if (k_lim > a.k_max) k_lim = a.k_max;
            const uint32_t singles = count_singles(ws, nonempty, lane), searched = nonempty - singles;
            uint32_t err = PHOBIC_OK;
            uint32_t j = 0;
            for (; j < searched && err == PHOBIC_OK; j++) {
                const uint32_t sc = ws.sched[j];
                const uint32_t b = sc >> 16, s = (ws.sched[j + 1] - sc) & 0xFFFFu;
                const uint2 *src = so + (sc & 0xFFFFu);
                if (PIPE && s <= 32) break;  // every later bucket is as small (search order: size descending)
                uint32_t pilot = 0;
                if (s <= 32) err = ksplit_bucket<W, 1>(ws, src, s, sr, fm, k_lim, xch, &par, w, lane, bar_id, &pilot);
                else if (s <= 64) err = ksplit_bucket<W, 2>(ws, src, s, sr, fm, k_lim, xch, &par, w, lane, bar_id, &pilot);
                else if (s <= 128) err = ksplit_bucket<W, 4>(ws, src, s, sr, fm, k_lim, xch, &par, w, lane, bar_id, &pilot);
                else err = ksplit_bucket<W, 8>(ws, src, s, sr, fm, k_lim, xch, &par, w, lane, bar_id, &pilot);
                if (err == PHOBIC_OK && w == 0 && lane == 0 && PHB_CHECK(b < a.buckets)) pil[(size_t)b * pstride] = pilot;
            }
            if (PIPE && err == PHOBIC_OK && j < searched) {
                volatile uint32_t *status = ctl + 2;
                if (ps <= kFewSlots) pipeline<W, 1, true>(ws, so, sr, fm, k_lim, j, searched, w, lane, turn_id, next_id, status, pil, pstride);
                else if (sr.rounds == 1) pipeline<W, 1>(ws, so, sr, fm, k_lim, j, searched, w, lane, turn_id, next_id, status, pil, pstride);
                else if (sr.rounds == 2) pipeline<W, 2>(ws, so, sr, fm, k_lim, j, searched, w, lane, turn_id, next_id, status, pil, pstride);
                else if (sr.rounds == 3) pipeline<W, 3>(ws, so, sr, fm, k_lim, j, searched, w, lane, turn_id, next_id, status, pil, pstride);
                else pipeline<W, 0>(ws, so, sr, fm, k_lim, j, searched, w, lane, turn_id, next_id, status, pil, pstride);
                group_bar(bar_id, bar_n);
                err = *status;
            }
            if (err == PHOBIC_OK && w == 0) place_singles(ws, so, searched, singles, ps, fm, lane, pil, pstride);
            if (err != PHOBIC_OK && w == 0 && lane == 0) report_error(&a.err[s_idx], p, err);
        }
        // Everyone is done with this partition's tables before the next is fetched.
        group_bar(bar_id, bar_n);
    }
}

}  // namespace

unsigned int check_line_search(bool reset) { return read_check_line(reset); }

size_t search_warp_smem(uint32_t buckets, uint32_t cap) { return 4 * warp_words(buckets, cap); }

// The rule for what is accepted is the shared memory of a warp that also sorts its partition (packed
// u16 tables of bucket sizes and cursors, two of 256 size bins, slots, collision scratch, schedule
// and bitmap).  K3c without its stage and K4 take more than that where it is far below the limit
// (the bitmap of pairs: 46 KB at 65,535 slots and 1,000 buckets against 32) and less near it (two words a
// bucket each against two and a half), so the last two conditions refuse nothing that the first one
// accepts; they hold the layouts to it.
bool search_accepts(uint32_t buckets, uint32_t cap) {
    if (cap > 65535 || buckets > 65535) return false;
    const size_t half = (buckets + 1) / 2, reach = (cap - 1) / 32 + 32 * ((cap + 1023) / 1024) + 2,
                 occ = (2 * cap + 31) / 32 + 2;
    const size_t words = std::max(half + 256, (size_t)kHsWords + scr_words(cap)) + half + buckets + std::max(reach, occ);
    return 4 * ((words + 3) & ~size_t(3)) <= kSearchSmemLimit && search_warp_smem(buckets, cap) <= kSearchSmemLimit &&
           order_smem(buckets) <= kSearchSmemLimit;
}

int search_warps_per_cta(uint32_t buckets, uint32_t cap) {
    if (!search_accepts(buckets, cap)) return 0;
    size_t fit = kSearchSmemLimit / search_warp_smem(buckets, cap);
    return (int)(fit < (size_t)kSearchWarps ? fit : (size_t)kSearchWarps);
}

template <bool DENSE>
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
        const uint32_t code = search_partition<DENSE>(a, mine, ws, d, g, p, lane);
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

SearchShape search_shape_for(uint32_t partitions, uint32_t partition_size, uint32_t buckets, int sm_count) {
    // Measured on a B200 (the autotuner's ladder, three key sets per size, seven parameter sets,
    // build ms): bucket pipelines of 8 warps take 0.89 to 0.99 of the time of 4 warps up to 256
    // partitions (at most two per SM) and 0.96 to 1.4 above; 4 warps win up to 2048 partitions
    // (0.54-1.16 against 0.63-1.60 ms on one warp).  At 4096 they are level with one warp per
    // partition where few pilot counters fail (average bucket of 6 keys and less: 0.97-1.18 against
    // 0.83-1.02 ms) and still ahead where many do (7 and more: 1.30-2.04 against 1.33-2.40 ms).
    SearchShape sh;
    sh.group = 1;
    const uint64_t sms = sm_count > 0 ? sm_count : 148;
    const bool retries = (uint64_t)partition_size * 2 >= (uint64_t)buckets * 13;
    if (partitions <= 256 && partitions <= 2 * sms) sh = SearchShape{8, true};
    else if (partitions <= (retries ? 30 : 18) * sms) sh = SearchShape{4, true};  // 4440 or 2664 on 148 SMs
    return sh;
}

cudaError_t launch_search(const SearchArgs &a, int sm_count, cudaStream_t st, SearchShape shape) {
    if (a.M == 0) return cudaSuccess;
    if (shape.group == 0) shape = search_shape_for(a.M, a.partition_size, a.buckets, sm_count);
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
    auto *kernel = a.partition_size <= kDenseSlots ? k_search<true> : k_search<false>;
    cudaError_t e = allow_dynamic_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, warps * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    uint64_t want = (a.M + warps - 1) / warps;
    int grid = (int)std::min<uint64_t>(want, (uint64_t)per_sm * sm_count);
    kernel<<<grid, warps * 32, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace phobicb200

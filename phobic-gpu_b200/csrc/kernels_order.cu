// K3c: the bucket order of every partition; one CTA per partition.
//
// Replaces bucket_sizes.comp:21-35 (bucket sizes), sort_sum.comp:141-226 (descending-size
// order, in-partition offsets) and the part of redistribute_keys.comp:21-53 that brings the
// keys of a partition into that order.  For every partition it leaves
//   sorted[base ..)        the lower pairs, bucket after bucket in search order
//   schedule               start | bucket << 16 of every nonempty bucket in search order, then
//                          the end; it takes the place of the partition's own (read) records
//                          in `lowers`, whose 8 bytes per key always hold it
//   part_state[g]          the number of nonempty buckets, or a status for the search to report
// and pilot 0 for the empty buckets.
//
// 10 bytes are read and 8 + 4 / lambda written per key.  The histogram's atomics return each key's
// rank in its bucket, so the order of a partition is one shared-memory scatter of 16-bit indexes,
// and the keys, copied to shared memory asynchronously meanwhile, leave in coalesced 16-byte
// stores.  Before, every warp of the search sorted its own partition (a histogram pass, a second
// pass with a 32-way scattered store per step, a serial size order, all with one warp's loads in
// flight): 1.48 ms of the 6.97 ms of that search at 10^8 u64 keys (lambda 7, P 2500), 0.60 of
// 3.12 ms at 5*10^7 keys (lambda 6, P 2048).  This kernel takes 0.52 and 0.24 ms (instruction
// issue 61 %, DRAM 41 %); with 3, 5 or 6 CTAs per SM instead of 4 it is 8, 8 and 25 % slower.
#include <algorithm>
#include <cmath>

#include "kernels.cuh"

namespace phobicb200 {

namespace {

constexpr int kOrderThreads = 256;
constexpr int kOrderItems = 16;
constexpr int kOrderCtas = 4;  // per SM: 64 registers per thread
constexpr uint32_t kSizeBins = kMaxBucket;  // bin 256 - size

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint32_t t = __shfl_up_sync(kFullMask, v, d);
        if (lane >= d) v += t;
    }
    return v;
}

// Packed u16 tables (no entry may exceed 0xFFFF).
__device__ __forceinline__ uint32_t half_get(const uint32_t *w, uint32_t b) { return (w[b >> 1] >> ((b & 1) << 4)) & 0xFFFFu; }
__device__ __forceinline__ void half_add(uint32_t *w, uint32_t b, uint32_t v) { atomicAdd(&w[b >> 1], v << ((b & 1) << 4)); }

// Lanes holding the same BITS-bit value: one vote per bit, all in flight together (nine votes
// take an SM about 15 cycles, __match_any_sync 60).
template <int BITS>
__device__ __forceinline__ uint32_t same_value_lanes(uint32_t v) {
    uint32_t same = kFullMask;
#pragma unroll
    for (int b = 0; b < BITS; b++) {
        const bool on = (v >> b) & 1u;
        const uint32_t set = __ballot_sync(kFullMask, on);
        same &= on ? set : ~set;
    }
    return same;
}

// Search order of the buckets whose sizes are in cnt, by one warp: exclusive prefixes over the
// size bins of buckets and keys (sort_sum.comp:184-215), then within a bin the higher bucket
// index first (sort_sum.comp:156).  Fills sched, replaces cnt by the starts and returns the
// number of nonempty buckets.
__device__ __forceinline__ uint32_t order_buckets(uint32_t *cnt, uint32_t *sched, uint32_t *binPos, uint32_t *binKey,
                                                  uint32_t B, uint32_t ps, int lane) {
    uint32_t c[8], loc = 0, lock = 0;  // lane L owns bins 8L .. 8L+7
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const uint32_t bin = 8 * lane + j;
        c[j] = half_get(binPos, bin);
        loc += c[j];
        lock += c[j] * (kSizeBins - bin);
    }
    const uint32_t inc = warp_incl_scan(loc, lane), inck = warp_incl_scan(lock, lane);
    const uint32_t nonempty = __shfl_sync(kFullMask, inc, 31);
    uint32_t ex = inc - loc, exk = inck - lock;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        const uint32_t bin = 8 * lane + j;
        const uint32_t ex1 = ex + c[j], exk1 = exk + c[j] * (kSizeBins - bin);
        binPos[bin >> 1] = ex | (ex1 << 16);
        binKey[bin >> 1] = exk | (exk1 << 16);
        ex = ex1 + c[j + 1];
        exk = exk1 + c[j + 1] * (kSizeBins - bin - 1);
    }
    __syncwarp();
    for (uint32_t c0 = 0; c0 < B; c0 += 32) {
        const int bi = (int)B - 1 - (int)(c0 + lane);
        const uint32_t s = bi >= 0 ? cnt[bi] : 0u;
        const uint32_t peers = same_value_lanes<9>(s);
        const uint32_t r = __popc(peers & lanemask_lt());
        const uint32_t bin = kSizeBins - s;
        if (s) {
            const uint32_t j = half_get(binPos, bin) + r, st = half_get(binKey, bin) + r * s;
            if (PHB_CHECK(j < B && st + s <= ps)) {
                sched[j] = st | ((uint32_t)bi << 16);
                cnt[bi] = st;
            }
        }
        __syncwarp();
        if (s && lane == __ffs(peers) - 1) {
            half_add(binPos, bin, __popc(peers));
            half_add(binKey, bin, __popc(peers) * s);
        }
        __syncwarp();
    }
    if (lane == 0) sched[nonempty] = ps;
    return nonempty;
}

// Number of buckets up to which every thread orders two buckets (order_parallel); above, one warp
// orders them 32 at a time (order_buckets).
constexpr uint32_t kOrderParallel = 2 * kOrderThreads;
static_assert(2 * kOrderThreads / 32 == 16, "a size's counts per 32 buckets are one 16-byte row");

// Shared memory, in words: the size tables, the partition's keys as they came, their order
// (u16, one more for the parity of the output), bucket sizes (then starts), the schedule, and the
// two parities of the CTA's partition.
//   parallel   rows u8[257][16] (buckets of a size per 32 buckets), first u32[256] (packed starts
//              of a size bin), sums u32[8]
//   one warp   binPos u16[256], binKey u16[256]
constexpr uint32_t kInfoWords = 8;
__host__ __device__ __forceinline__ uint32_t table_words(uint32_t B) {
    return B <= kOrderParallel ? 257 * 4 + 256 + 8 : 256;
}
__host__ __device__ __forceinline__ size_t order_words(uint32_t B, uint32_t stage_keys) {
    return table_words(B) + 2 * (size_t)stage_keys + (stage_keys ? stage_keys / 2 + 1 : 0) + 2 * (size_t)B + 1 +
           2 * kInfoWords;
}

__device__ __forceinline__ void copy_async8(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Sum of the bytes of a row below byte w (w <= 16).
__device__ __forceinline__ uint32_t row_sum(uint4 r, uint32_t w) {
    uint32_t t = 0;
    const uint32_t v[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) {
        const uint32_t n = w > 4 * q ? min(w - 4 * q, 4u) : 0u;
        t = __dp4a(v[q] & ~__funnelshift_lc(0u, kFullMask, 8 * n), 0x01010101u, t);
    }
    return t;
}

// Search order of at most kOrderParallel buckets, two per thread: the order of order_buckets.
// Slot t + 256 h of thread t holds bucket B - 1 - slot, so a bucket's rank in its size is the
// number of equal sizes in the 32-slot groups before (rows) and in the lanes before.  Returns
// false, without an order, when a bucket is too large; *nonempty_out is set by thread 255 only.
__device__ __forceinline__ bool order_parallel(const SearchArgs &a, uint32_t g, uint32_t *cnt, uint32_t *sched,
                                               uint32_t *tables, uint32_t *pil, uint32_t pstride, uint32_t ps,
                                               uint32_t *nonempty_out) {
    const uint32_t B = a.buckets, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint8_t *rows = reinterpret_cast<uint8_t *>(tables);
    uint32_t *first = tables + 257 * 4, *sums = first + 256;
    bool over = false;
    uint32_t v[2], before[2];
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
        const uint32_t slot = tid + kOrderThreads * h, bi = B - 1 - slot;
        v[h] = before[h] = 0;
        if (kOrderThreads * h >= B) continue;
        const uint32_t s = slot < B ? cnt[bi] : 0u;
        if (slot < B) {
            if (a.debug_sizes) a.debug_sizes[(size_t)g * B + bi] = s;
            if (s == 0) pil[(size_t)bi * pstride] = 0;
        }
        if (s > kMaxBucket) over = true;
        else v[h] = s;
        const uint32_t peers = same_value_lanes<9>(v[h]);
        before[h] = __popc(peers & lanemask_lt());
        if (v[h] && before[h] == 0) rows[16 * v[h] + warp + 8 * h] = (uint8_t)__popc(peers);
    }
    if (__syncthreads_or(over)) return false;
    // Starts of the size bins, largest size first: buckets in the low half, keys in the high.
    const uint32_t size = 256 - tid;
    const uint32_t c = row_sum(*reinterpret_cast<const uint4 *>(rows + 16 * size), 16);
    const uint32_t total = c | ((c * size) << 16);
    uint32_t incl = warp_incl_scan(total, (int)lane);
    if (lane == 31) sums[warp] = incl;
    __syncthreads();
    for (uint32_t w = 0; w < warp; w++) incl += sums[w];
    first[tid] = incl - total;
    if (tid == 255) {
        *nonempty_out = incl & 0xFFFFu;
        sched[incl & 0xFFFFu] = ps;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
        if (!v[h]) continue;
        const uint32_t bi = B - 1 - (tid + kOrderThreads * h);
        const uint32_t f = first[256 - v[h]];
        const uint32_t r = row_sum(*reinterpret_cast<const uint4 *>(rows + 16 * v[h]), warp + 8 * h) + before[h];
        const uint32_t j = (f & 0xFFFFu) + r, st = (f >> 16) + r * v[h];
        if (PHB_CHECK(j < B && st + v[h] <= ps)) {
            sched[j] = st | (bi << 16);
            cnt[bi] = st;
        }
    }
    return true;
}

// Looks a partition up, by one thread, so that those who order it agree on what becomes of it:
// {base, size, state, -, pilots, partitions}.
__device__ __forceinline__ void look_up(const SearchArgs &a, uint32_t g, uint32_t *in) {
    const uint32_t s_idx = a.nsets == 1 ? 0u : find_set(a.part_base, a.nsets, g);
    const SetDesc &d = a.sets[s_idx];
    const uint32_t p = g - d.part_base;
    const uint32_t base = a.G[g], end = a.G[g + 1];
    const uint32_t ps = end - base;
    // The size check comes first and looks at every partition, also of a set that failed before
    // (only a scan that timed out leaves no offsets to check): the error word then holds the
    // lowest oversized partition, whichever CTA comes to its own first.
    const unsigned long long e = *reinterpret_cast<volatile unsigned long long *>(&a.err[s_idx]);
    uint32_t state = 0;
    if (e != kNoError && (uint32_t)e == PHOBIC_ERR_TIMEOUT) {
        state = kPartSkipped;
    } else if (ps > a.cap) {
        report_error(&a.err[s_idx], p, PHOBIC_ERR_PARTITION_OVERFLOW);
        state = kPartSkipped;
    } else if (fatal_before_search(e)) {
        state = kPartSkipped;
    } else {
        if (d.part_off) {
            const uint32_t g0 = a.G[d.part_base];
            d.part_off[p] = base - g0;
            if (p + 1 == d.partitions) d.part_off[p + 1] = end - g0;
        }
        if (!PHB_CHECK(base + ps <= a.G[a.M])) {
            state = kPartSkipped;
        } else if (a.part_state[g] != end) {
            // K3 placed exactly the keys K1 counted, unless the keys changed in between.
            state = kPartSkipped | PHOBIC_ERR_KEYS_CHANGED;
        }
    }
    if (state) a.part_state[g] = state;
    const unsigned long long pil = reinterpret_cast<unsigned long long>(d.pilots + p);
    in[0] = base, in[1] = ps, in[2] = state, in[4] = (uint32_t)pil, in[5] = (uint32_t)(pil >> 32);
    in[6] = d.partitions;
}

}  // namespace

__global__ void __launch_bounds__(kOrderThreads, kOrderCtas) k_order(SearchArgs a, uint32_t stage_keys) {
    extern __shared__ __align__(16) uint32_t smem[];
    const uint32_t B = a.buckets, tid = threadIdx.x;
    uint32_t *tables = smem;
    uint2 *raw = reinterpret_cast<uint2 *>(tables + table_words(B));  // table_words is even
    uint16_t *perm = reinterpret_cast<uint16_t *>(raw + stage_keys);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(raw + stage_keys) + (stage_keys ? stage_keys / 2 + 1 : 0);
    uint32_t *sched = cnt + B;
    uint32_t *info = sched + B + 1;  // {base, size, state, nonempty, pilots, partitions} by parity
    const bool parallel = B <= kOrderParallel;

    uint32_t par = 0;
    if (tid == 0 && blockIdx.x < a.M) look_up(a, blockIdx.x, info);
    for (uint32_t g = blockIdx.x; g < a.M; g += gridDim.x, par ^= kInfoWords) {
        for (uint32_t i = tid; i < B; i += kOrderThreads) cnt[i] = 0;
        for (uint32_t i = tid; i < table_words(B); i += kOrderThreads) tables[i] = 0;
        __syncthreads();
        const uint32_t *in = info + par;
        const uint32_t base = in[0], ps = in[1], state = in[2];
        const bool staged = ps <= stage_keys;
        uint32_t *pil = reinterpret_cast<uint32_t *>((unsigned long long)in[4] | (unsigned long long)in[5] << 32);
        const uint32_t pstride = in[6];
        const uint16_t *bk = a.bkt + base;
        const uint2 *lo = a.lowers + base;
        uint32_t br[kOrderItems];  // bucket, then bucket | rank << 16
        if (!state && staged) {
            // All loads of the partition in flight together: the bucket ids to registers, the
            // lower pairs to shared memory, where they are needed last.
#pragma unroll
            for (int j = 0; j < kOrderItems; j++) {
                const uint32_t i = j * kOrderThreads + tid;
                br[j] = i < ps ? __ldcs(bk + i) : 0u;
            }
#pragma unroll
            for (int j = 0; j < kOrderItems; j++) {
                const uint32_t i = j * kOrderThreads + tid;
                if (i < ps) copy_async8(raw + i, lo + i);
            }
        }
        // The next partition is looked up meanwhile.
        if (tid == kOrderThreads - 1 && g + gridDim.x < a.M) look_up(a, g + gridDim.x, info + (par ^ kInfoWords));
        if (state) continue;

        // Bucket sizes (bucket_sizes.comp:21-35).  Ids >= B never come from K3 for keys that K1
        // counted; the clamp keeps a stale record (keys changed during the build) in the tables.
        if (staged) {
#pragma unroll
            for (int j = 0; j < kOrderItems; j++) {
                const uint32_t i = j * kOrderThreads + tid;
                if (i >= ps) continue;
                const uint32_t b = min(br[j], B - 1);
                (void)PHB_CHECK(b == br[j]);
                br[j] = b | (atomicAdd(&cnt[b], 1u) << 16);
            }
        } else {
            for (uint32_t i = tid; i < ps; i += kOrderThreads) {
                const uint32_t b = min((uint32_t)bk[i], B - 1);
                if (PHB_CHECK(b == bk[i])) atomicAdd(&cnt[b], 1u);
            }
        }
        __syncthreads();

        // Search order (sort_sum.comp:56-58,156-215); empty buckets get pilot 0.
        bool ok;
        if (parallel) {
            ok = order_parallel(a, g, cnt, sched, tables, pil, pstride, ps, &info[par + 3]);
        } else {
            bool over = false;
            for (uint32_t b = tid; b < B; b += kOrderThreads) {
                const uint32_t s = cnt[b];
                if (a.debug_sizes) a.debug_sizes[(size_t)g * B + b] = s;
                if (s > kMaxBucket) over = true;
                else if (s && PHB_CHECK(s <= kSizeBins)) half_add(tables, kSizeBins - s, 1);
                else pil[(size_t)b * pstride] = 0;
            }
            ok = !__syncthreads_or(over);
            if (ok && tid < 32) {
                const uint32_t nonempty = order_buckets(cnt, sched, tables, tables + 128, B, ps, (int)tid);
                if (tid == 0) info[par + 3] = nonempty;
            }
        }
        if (!ok) {
            copy_async_wait();
            if (tid == 0) a.part_state[g] = kPartSkipped | PHOBIC_ERR_BUCKET_OVERFLOW;
            continue;
        }
        __syncthreads();

        // Keys into bucket order (redistribute_keys.comp:21-53, inside the partition).
        const uint32_t nonempty = in[3];
        uint2 *so = a.sorted + base;
        if (staged) {
            const uint32_t odd = base & 1;  // pairs of output keys start on 16 bytes
#pragma unroll
            for (int j = 0; j < kOrderItems; j++) {
                const uint32_t i = j * kOrderThreads + tid;
                if (i >= ps) continue;
                const uint32_t pos = cnt[br[j] & 0xFFFFu] + (br[j] >> 16);
                if (PHB_CHECK(pos < ps)) perm[pos + odd] = (uint16_t)i;
            }
            copy_async_wait();
            __syncthreads();
            const uint32_t end = ps + odd;
#pragma unroll 4
            for (uint32_t q = 2 * tid; q < end; q += 2 * kOrderThreads) {
                const uint32_t two = *reinterpret_cast<const uint32_t *>(perm + q);
                const bool first = q >= odd, second = q + 1 < end;
                uint2 x = make_uint2(0, 0), y = x;
                if (first) x = raw[two & 0xFFFFu];
                if (second) y = raw[two >> 16];
                if (first && second) {
                    *reinterpret_cast<uint4 *>(so + (q - odd)) = make_uint4(x.x, x.y, y.x, y.y);
                } else if (first) {
                    so[q - odd] = x;
                } else if (second) {
                    so[q + 1 - odd] = y;
                }
            }
        } else {
            for (uint32_t i = tid; i < ps; i += kOrderThreads) {
                const uint32_t pos = atomicAdd(&cnt[min((uint32_t)bk[i], B - 1)], 1u);
                if (PHB_CHECK(pos < ps)) so[pos] = lo[i];
            }
            __syncthreads();
        }
        // The partition's records have been read by every thread: their place takes the schedule.
        uint32_t *sch = reinterpret_cast<uint32_t *>(const_cast<uint2 *>(lo));
        for (uint32_t i = tid; i <= nonempty; i += kOrderThreads)
            if (ps && PHB_CHECK(i < 2 * ps)) sch[i] = sched[i];
        if (tid == 0) a.part_state[g] = nonempty;
    }
}

// ------------------------------------------------------------------ small partitions
//
// The same for partitions of few keys, one warp each: with so little to do in a partition, k_order's seven
// barriers and its tables for 256 sizes are what takes the time, with 4 partitions in flight per SM.  Keys and
// bucket ids of a partition of at most 32 ITEMS keys are in registers, and leave in bucket order through
// shared memory.  3*10^7 keys: at P 64 0.96 ms of bucket order and partition passes instead of 4.1, at P 128
// 0.78 instead of 2.3, at P 256 0.69 instead of 1.4, at P 512 0.62 instead of 0.92; larger partitions would
// not fit the registers.
constexpr int kWarpOrderThreads = 128;
constexpr uint32_t kWarpOrderKeys = 512, kWarpOrderBuckets = 512;
__host__ __device__ __forceinline__ size_t warp_order_words(uint32_t B, uint32_t stage_keys) {
    return (2 * (size_t)stage_keys + 256 + 2 * (size_t)B + 1 + 2 * kInfoWords + 1) & ~size_t(1);
}

template <int ITEMS>
__global__ void __launch_bounds__(kWarpOrderThreads) k_order_warp(SearchArgs a) {
    extern __shared__ __align__(16) uint32_t smem[];
    constexpr uint32_t kStage = 32 * ITEMS;
    const uint32_t B = a.buckets, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t warps = gridDim.x * (kWarpOrderThreads / 32);
    uint2 *raw = reinterpret_cast<uint2 *>(smem + warp * warp_order_words(B, kStage));
    uint32_t *tables = reinterpret_cast<uint32_t *>(raw + kStage);
    uint32_t *cnt = tables + 256;
    uint32_t *sched = cnt + B;
    uint32_t *info = sched + B + 1;

    uint32_t g = blockIdx.x * (kWarpOrderThreads / 32) + warp, par = 0;
    if (lane == 0 && g < a.M) look_up(a, g, info);
    for (; g < a.M; g += warps, par ^= kInfoWords) {
        for (uint32_t i = lane; i < B; i += 32) cnt[i] = 0;
        for (uint32_t i = lane; i < 256; i += 32) tables[i] = 0;
        __syncwarp();
        const uint32_t *in = info + par;
        const uint32_t base = in[0], ps = in[1], state = in[2];
        uint32_t *pil = reinterpret_cast<uint32_t *>((unsigned long long)in[4] | (unsigned long long)in[5] << 32);
        const uint32_t pstride = in[6];
        const bool staged = ps <= kStage;
        const uint16_t *bk = a.bkt + base;
        const uint2 *lo = a.lowers + base;
        uint2 key[ITEMS];
        uint32_t br[ITEMS];  // bucket, then bucket | rank << 16
        if (!state && staged) {
#pragma unroll
            for (int j = 0; j < ITEMS; j++) {
                const uint32_t i = 32 * j + lane;
                br[j] = i < ps ? __ldcs(bk + i) : 0u;
                key[j] = i < ps ? __ldcs(lo + i) : make_uint2(0, 0);
            }
        }
        if (lane == 31 && g + warps < a.M) look_up(a, g + warps, info + (par ^ kInfoWords));
        if (state) continue;

        if (staged) {
#pragma unroll
            for (int j = 0; j < ITEMS; j++) {
                if (32 * j + lane >= ps) continue;
                const uint32_t b = min(br[j], B - 1);
                (void)PHB_CHECK(b == br[j]);
                br[j] = b | (atomicAdd(&cnt[b], 1u) << 16);
            }
        } else {
            for (uint32_t i = lane; i < ps; i += 32) {
                const uint32_t b = min((uint32_t)bk[i], B - 1);
                if (PHB_CHECK(b == bk[i])) atomicAdd(&cnt[b], 1u);
            }
        }
        __syncwarp();
        bool over = false;
        for (uint32_t b = lane; b < B; b += 32) {
            const uint32_t s = cnt[b];
            if (a.debug_sizes) a.debug_sizes[(size_t)g * B + b] = s;
            if (s > kMaxBucket) over = true;
            else if (s && PHB_CHECK(s <= kSizeBins)) half_add(tables, kSizeBins - s, 1);
            else pil[(size_t)b * pstride] = 0;
        }
        if (__any_sync(kFullMask, over)) {
            if (lane == 0) a.part_state[g] = kPartSkipped | PHOBIC_ERR_BUCKET_OVERFLOW;
            continue;
        }
        __syncwarp();
        const uint32_t nonempty = order_buckets(cnt, sched, tables, tables + 128, B, ps, (int)lane);
        __syncwarp();

        uint2 *so = a.sorted + base;
        if (staged) {
#pragma unroll
            for (int j = 0; j < ITEMS; j++) {
                if (32 * j + lane >= ps) continue;
                const uint32_t pos = cnt[br[j] & 0xFFFFu] + (br[j] >> 16);
                if (PHB_CHECK(pos < ps)) raw[pos] = key[j];
            }
            __syncwarp();
            for (uint32_t i = lane; i < ps; i += 32) so[i] = raw[i];
        } else {
            for (uint32_t i = lane; i < ps; i += 32) {
                const uint32_t pos = atomicAdd(&cnt[min((uint32_t)bk[i], B - 1)], 1u);
                if (PHB_CHECK(pos < ps)) so[pos] = lo[i];
            }
            __syncwarp();
        }
        uint32_t *sch = reinterpret_cast<uint32_t *>(const_cast<uint2 *>(lo));
        for (uint32_t i = lane; i <= nonempty; i += 32)
            if (ps && PHB_CHECK(i < 2 * ps)) sch[i] = sched[i];
        if (lane == 0) a.part_state[g] = nonempty;
        __syncwarp();
    }
}

template <int ITEMS>
static cudaError_t launch_order_warp(const SearchArgs &a, int sm_count, cudaStream_t st) {
    constexpr int warps = kWarpOrderThreads / 32;
    const size_t smem = 4 * warps * warp_order_words(a.buckets, 32 * ITEMS);
    cudaError_t e = allow_dynamic_smem(k_order_warp<ITEMS>, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_order_warp<ITEMS>, kWarpOrderThreads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    const int grid = (int)std::min<uint64_t>((a.M + warps - 1) / warps, (uint64_t)per_sm * (sm_count > 0 ? sm_count : 148));
    k_order_warp<ITEMS><<<grid, kWarpOrderThreads, smem, st>>>(a);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ small builds
//
// A build of one set of at most kGatherMaxKeys fixed-size keys in at most one partition per SM needs
// no passes between the keys and their order: the CTA of a partition reads and hashes all of the
// set's keys, keeps its own (lower pair, bucket, rank in the bucket) in shared memory, counts the
// keys of the partitions before it, which is its offset, and orders its keys as k_order does.  One
// launch takes the place of K1, the scan, both partition passes and K3c; every CTA hashes every key,
// which up to this size costs less than the launches (stage times with their events, us: 1000 keys
// 19 against 39, 10,000 keys 37 against 45, 16,384 keys 47 against 44).
// The CTAs read the keys at different times.  The last one to finish checks that they saw the same
// keys: every partition ends where the next one begins, and the sum over the keys that were taken
// (key_sum) is the sum over all keys as the first CTA read them.  The sum is what tells two keys
// that trade partitions during the build, which leave every count as it was.  If not, the build
// reports that the keys changed (every store is in bounds all the same: no CTA finds more than n
// keys).  A change that no CTA saw, or that every CTA saw, gives a function of the keys as read.
__host__ __device__ __forceinline__ size_t gather_words(uint32_t B, uint32_t stage_keys) {
    return order_words(B, stage_keys) + stage_keys;
}

// One key in the sum: all four words, so mixed that keys which differ in a pattern don't cancel.
__device__ __forceinline__ unsigned long long key_sum(const Key4 &k) {
    return xxh3::fold64(((uint64_t)k.lower1 << 32 | k.lower2) ^ 0x9E3779B97F4A7C15ull,
                        ((uint64_t)k.partitioner << 32 | k.bucketer) ^ 0xD1B54A32D192ED03ull);
}

// CHANGE (tests, u64 keys): every CTA but the first reads key change_index as changed by change_mask.
template <int KIND, bool CHANGE = false>
__global__ void __launch_bounds__(kOrderThreads) k_gather(MapArgs m, SearchArgs a, uint32_t *G, uint32_t *ends,
                                                         uint32_t *ticket, uint32_t stage_keys, uint32_t change_index,
                                                         uint64_t change_mask) {
    extern __shared__ __align__(16) uint32_t smem[];
    const uint32_t B = a.buckets, tid = threadIdx.x, lane = tid & 31, n = (uint32_t)m.total_keys, p = blockIdx.x;
    uint32_t *tables = smem;
    uint2 *raw = reinterpret_cast<uint2 *>(tables + table_words(B));
    uint16_t *perm = reinterpret_cast<uint16_t *>(raw + stage_keys);
    uint32_t *br = reinterpret_cast<uint32_t *>(raw + stage_keys) + stage_keys / 2 + 1;  // bucket | rank << 16
    uint32_t *cnt = br + stage_keys;
    uint32_t *sched = cnt + B;
    uint32_t *info = sched + B + 1;  // {keys taken, keys of partitions before, -, nonempty, sum of the keys taken}
    unsigned long long *taken = reinterpret_cast<unsigned long long *>((reinterpret_cast<uintptr_t>(info + 4) + 7) & ~uintptr_t(7));
    unsigned long long *sum_all = reinterpret_cast<unsigned long long *>(ticket + 2);
    const SetDesc &d = a.sets[0];
    uint32_t *pil = d.pilots + p;
    for (uint32_t i = tid; i < B; i += kOrderThreads) cnt[i] = 0;
    for (uint32_t i = tid; i < table_words(B); i += kOrderThreads) tables[i] = 0;
    if (tid < kInfoWords) info[tid] = 0;
    __syncthreads();

    constexpr int U = 4;  // keys per thread and round, their loads in flight together
    uint32_t before = 0;
    unsigned long long sum = 0;  // of the keys taken; in the first CTA less all keys, its own cancelling
    bool bad = false;
    for (uint32_t i0 = 0; i0 < n; i0 += U * kOrderThreads) {
        Key4 k[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t i = i0 + u * kOrderThreads + tid;
            if constexpr (CHANGE) {
                const uint64_t v = __ldg(static_cast<const unsigned long long *>(d.data) + (i < n ? i : 0));
                k[u] = key_from_hash(xxh3::hash_u64(p && i == change_index ? v ^ change_mask : v));
            } else {
                k[u] = load_key<KIND>(d.data, nullptr, i < n ? i : 0);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool valid = i0 + u * kOrderThreads + tid < n;
            const uint32_t gp = partition_of(k[u].partitioner, a.M);
            const bool mine = valid && gp == p;
            before += valid && gp < p;
            if (p == 0 && valid && !mine) sum -= key_sum(k[u]);
            const uint32_t ball = __ballot_sync(kFullMask, mine);
            if (!ball) continue;
            uint32_t at = 0;
            if (lane == (uint32_t)__ffs(ball) - 1) at = atomicAdd(&info[0], (uint32_t)__popc(ball));
            at = __shfl_sync(kFullMask, at, __ffs(ball) - 1) + __popc(ball & lanemask_lt());
            if (!mine) continue;
            if (p) sum += key_sum(k[u]);
            const uint32_t b = bucket_of(k[u].bucketer, m.fulcs);
            bad |= b >= B;
            if (at < stage_keys) {  // more only where the partition exceeds the search's capacity
                const uint32_t bb = min(b, B - 1);
                raw[at] = make_uint2(k[u].lower1, k[u].lower2);
                br[at] = bb | (atomicAdd(&cnt[bb], 1u) << 16);
            }
        }
    }
    before = __reduce_add_sync(kFullMask, before);
    for (int x = 16; x; x >>= 1) sum += __shfl_xor_sync(kFullMask, sum, x);
    if (lane == 0) {
        if (before) atomicAdd(&info[1], before);
        atomicAdd(taken, sum);
    }
    if (bad) report_error(&a.err[0], 0, PHOBIC_ERR_INVALID);
    __syncthreads();

    const uint32_t ps = info[0], base = info[1];
    if (tid == 0) {
        G[p] = base;
        ends[p] = base + ps;
        if (p + 1 == a.M) G[a.M] = n;
        if (d.part_off) {
            d.part_off[p] = base;
            if (p + 1 == a.M) d.part_off[a.M] = n;
        }
    }
    uint32_t state = kPartSkipped;
    if (ps > a.cap) {
        if (tid == 0) report_error(&a.err[0], p, PHOBIC_ERR_PARTITION_OVERFLOW);
    } else {
        bool ok;
        if (B <= kOrderParallel) {
            ok = order_parallel(a, p, cnt, sched, tables, pil, d.partitions, ps, &info[3]);
        } else {
            bool over = false;
            for (uint32_t b = tid; b < B; b += kOrderThreads) {
                const uint32_t s = cnt[b];
                if (s > kMaxBucket) over = true;
                else if (s && PHB_CHECK(s <= kSizeBins)) half_add(tables, kSizeBins - s, 1);
                else pil[(size_t)b * d.partitions] = 0;
            }
            ok = !__syncthreads_or(over);
            if (ok && tid < 32) {
                const uint32_t nonempty = order_buckets(cnt, sched, tables, tables + 128, B, ps, (int)tid);
                if (tid == 0) info[3] = nonempty;
            }
        }
        __syncthreads();
        if (!ok) {
            state = kPartSkipped | PHOBIC_ERR_BUCKET_OVERFLOW;
        } else {
            state = info[3];
            for (uint32_t i = tid; i < ps; i += kOrderThreads) {
                const uint32_t pos = cnt[br[i] & 0xFFFFu] + (br[i] >> 16);
                if (PHB_CHECK(pos < ps)) perm[pos] = (uint16_t)i;
            }
            __syncthreads();
            if (PHB_CHECK(base + ps <= n)) {
                uint2 *so = a.sorted + base;
                for (uint32_t i = tid; i < ps; i += kOrderThreads) so[i] = raw[perm[i]];
                uint32_t *sch = reinterpret_cast<uint32_t *>(const_cast<uint2 *>(a.lowers + base));
                for (uint32_t i = tid; i <= state; i += kOrderThreads)
                    if (ps && PHB_CHECK(i < 2 * ps)) sch[i] = sched[i];
            }
        }
    }
    if (tid == 0) {
        a.part_state[p] = state;
        atomicAdd(sum_all, *taken);
        __threadfence();
        if (atomicAdd(ticket, 1u) == a.M - 1) {
            __threadfence();
            const volatile uint32_t *g = G, *e = ends;
            bool same = g[0] == 0 && *reinterpret_cast<volatile unsigned long long *>(sum_all) == 0;
            for (uint32_t q = 0; q < a.M; q++) same &= e[q] == (q + 1 < a.M ? g[q + 1] : n);
            if (!same)
                for (uint32_t q = 0; q < a.M; q++) a.part_state[q] = kPartSkipped | PHOBIC_ERR_KEYS_CHANGED;
        }
    }
}

// The shared memory of k_gather for a build, or 0 when the build takes the general path.
static size_t gather_smem(uint64_t n, uint64_t M, uint32_t B, uint32_t cap, uint32_t *stage_keys) {
    *stage_keys = (uint32_t)((std::min<uint64_t>(n, cap) + 1) & ~1ull);
    const size_t smem = 4 * gather_words(B, *stage_keys);
    return n && n <= kGatherMaxKeys && M <= kGatherMaxPartitions && smem <= kSearchSmemLimit ? smem : 0;
}

bool gather_fits(int kind, uint64_t n, uint64_t M, uint32_t B, uint32_t cap) {
    uint32_t stage = 0;
    return kind != PHOBIC_KEYS_STRINGS && gather_smem(n, M, B, cap, &stage) != 0;
}

template <int KIND, bool CHANGE = false>
static cudaError_t launch_gather_kind(const MapArgs &m, const SearchArgs &a, uint32_t *G, uint32_t *ends,
                                      uint32_t *ticket, cudaStream_t st, uint32_t index = 0, uint64_t mask = 0) {
    uint32_t stage = 0;
    const size_t smem = gather_smem(m.total_keys, a.M, a.buckets, a.cap, &stage);
    const cudaError_t e = allow_dynamic_smem(k_gather<KIND, CHANGE>, smem);
    if (e != cudaSuccess) return e;
    k_gather<KIND, CHANGE><<<a.M, kOrderThreads, smem, st>>>(m, a, G, ends, ticket, stage, index, mask);
    return cudaGetLastError();
}

cudaError_t launch_gather(int kind, const MapArgs &m, const SearchArgs &a, uint32_t *G, uint32_t *ends, uint32_t *ticket,
                          cudaStream_t st, uint64_t change_index, uint64_t change_mask) {
    if (change_mask)  // u64 keys (take_key_change)
        return launch_gather_kind<PHOBIC_KEYS_U64, true>(m, a, G, ends, ticket, st, (uint32_t)change_index, change_mask);
    switch (kind) {
    case PHOBIC_KEYS_U64: return launch_gather_kind<PHOBIC_KEYS_U64>(m, a, G, ends, ticket, st);
    case PHOBIC_KEYS_BYTES16: return launch_gather_kind<PHOBIC_KEYS_BYTES16>(m, a, G, ends, ticket, st);
    default: return launch_gather_kind<PHOBIC_KEYS_PREHASHED>(m, a, G, ends, ticket, st);
    }
}

size_t order_smem(uint32_t buckets) { return 4 * order_words(buckets, 0); }

unsigned int check_line_order(bool reset) { return read_check_line(reset); }

cudaError_t launch_order(const SearchArgs &a, int sm_count, cudaStream_t st) {
    if (a.M == 0) return cudaSuccess;
    // Partitions of up to 4096 keys (16 per thread) are staged; larger ones, or bucket counts that
    // leave no room for the stage, scatter in global memory.  A partition's size is binomial with
    // a mean of at most P, so the stage need not hold the search's whole capacity: eight standard
    // deviations above P leave room for kOrderCtas CTAs per SM.
    const double slack = 8.0 * std::sqrt((double)a.partition_size);
    const uint64_t want = std::min<uint64_t>((uint64_t)a.partition_size + (uint64_t)slack, a.cap);
    if (a.partition_size <= kWarpOrderKeys && a.buckets <= kWarpOrderBuckets) {
        if (want <= 128) return launch_order_warp<4>(a, sm_count, st);
        if (want <= 256) return launch_order_warp<8>(a, sm_count, st);
        if (want <= 512) return launch_order_warp<16>(a, sm_count, st);
        return launch_order_warp<24>(a, sm_count, st);
    }
    uint32_t stage_keys = (uint32_t)std::min<uint64_t>((want + 1) & ~1ull, kOrderThreads * kOrderItems);
    if (4 * order_words(a.buckets, stage_keys) > kSearchSmemLimit) stage_keys = 0;
    const size_t smem = 4 * order_words(a.buckets, stage_keys);
    cudaError_t e = allow_dynamic_smem(k_order, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_order, kOrderThreads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    const int grid = (int)std::min<uint64_t>(a.M, (uint64_t)per_sm * (sm_count > 0 ? sm_count : 148));
    k_order<<<grid, kOrderThreads, smem, st>>>(a, stage_keys);
    return cudaGetLastError();
}

}  // namespace phobicb200

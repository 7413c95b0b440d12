// Encoding of a build's result on the device, for the encoders made of compact
// vectors: interleaved_encoder<compact> and mono_encoder<compact> pilots
// (include/encoders/pilotEncoders/interleaved_encoder.hpp:8-15, mono_encoders.hpp),
// diff_partition_encoder<compact> and direct_partition_encoder<compact> offsets
// (include/encoders/partitionOffsetEnocders/*.hpp, base/linear_diff_encoder.hpp:15-28).
// This is Mphf::setData (include/phobicGpu/mphf.hpp:65-75) without the host pass
// over the pilots.
//
// Every compact vector is written as the host encoders serialise it, in visit
// order: size, width, mask (u64 each), then its words as a vector (u64 count,
// count = ceil(size * width / 64) + 1, then the words).  Value i occupies bits
// [i w, i w + w) of the little-endian word array; width = bit length of the
// largest value, at least 1 (compact_vector.hpp build).  The bytes equal
// phobic_encode's for the same arrays.
//
//   k_colmax     per column (an interleaved column of `partitions` pilots, or the
//                one mono column of all pilots): largest value; and the largest
//                partition-offset code (zig-zag difference to i * P, or the offset
//                itself)
//   k_table      widths and byte offsets of all columns (one CTA)
//   k_pack       one thread per output word of every column; writes the headers,
//                unless the output does not fit (the host then packs into a stage)
//
// A column's words depend only on its values and width, so all columns are
// written by one launch from the table.  The widths are known on the device only: with
// the table made there, the call waits for the device once, at its end.  At 10^8 keys
// (57 MB of pilots) the call took 132 us with the table made on the host between the
// maxima and the packing (three copies, a wait, one copy), and takes 97 us.
#include <algorithm>
#include <cstring>
#include <vector>

#include "engine.hpp"
#include "kernels.cuh"

namespace phobicb200 {

namespace {

constexpr int kEncThreads = 256;
constexpr int kMaxLoads = 8;  // loads in flight per thread of k_colmax

// One compact vector of the output.
struct EncColumn {
    const uint32_t *vals;  // pilot column (null: the partition-offset codes)
    uint64_t n;            // values
    uint64_t out;          // byte offset of its header in the output
    uint32_t width;
    uint32_t pad;
};

// Code of partition offset i (linear_diff_encoder.hpp:15-28 for diff, the value itself for direct).
__device__ __forceinline__ uint64_t offset_code(const uint32_t *off, uint64_t i, uint32_t psize, bool diff) {
    const uint64_t v = off[i];
    if (!diff) return v;
    const int64_t d = (int64_t)v - (int64_t)(i * psize);
    const uint64_t a = (uint64_t)(d < 0 ? -d : d);
    return (a << 1) | (uint64_t)(d > 0);
}

__device__ __forceinline__ uint64_t words_for(uint64_t bits) { return (bits + 63) / 64; }

// Largest value of column blockIdx.x, per CTA chunk, into maxes[x] (atomicMax); the last
// blockIdx.x: largest partition-offset code into *code_max.
__global__ void __launch_bounds__(kEncThreads) k_colmax(const uint32_t *pilots, uint64_t per_col, uint32_t cols,
                                                        uint32_t *maxes, const uint32_t *off, uint64_t noff,
                                                        uint32_t psize, int diff, unsigned long long *code_max) {
    const uint64_t first = (uint64_t)blockIdx.y * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.y * blockDim.x;
    if (blockIdx.x == cols) {
        unsigned long long m = 0;
        for (uint64_t i = first; i < noff; i += step) m = max(m, (unsigned long long)offset_code(off, i, psize, diff != 0));
        for (int d = 16; d; d >>= 1) m = max(m, __shfl_xor_sync(kFullMask, m, d));
        if ((threadIdx.x & 31) == 0 && m) atomicMax(code_max, m);
        return;
    }
    const uint32_t *v = pilots + (uint64_t)blockIdx.x * per_col;
    uint32_t m = 0;
    for (uint64_t i = first; i < per_col; i += kMaxLoads * step) {  // the loads of a round in flight together
        uint32_t x[kMaxLoads];
#pragma unroll
        for (int j = 0; j < kMaxLoads; j++) x[j] = i + j * step < per_col ? __ldg(v + i + j * step) : 0u;
#pragma unroll
        for (int j = 0; j < kMaxLoads; j++) m = max(m, x[j]);
    }
    m = __reduce_max_sync(kFullMask, m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(&maxes[blockIdx.x], m);
}

// Bytes of a compact vector of n values of width w: size, width, mask, count, words.
__host__ __device__ __forceinline__ uint64_t vector_bytes(uint64_t n, uint32_t w) { return 32 + 8 * ((n * w + 63) / 64 + 1); }

// The column table in visit order (pilot columns, then the offsets) from the maxima; info[0] = the
// size of the output, info[1] = keys.  One CTA: each thread takes the columns tid + 256 k, a chunk
// of 256 columns at a time.
__global__ void __launch_bounds__(kEncThreads) k_table(const uint32_t *maxes, const unsigned long long *code_max,
                                                       const uint32_t *pilots, uint64_t per_col, uint32_t cols,
                                                       const uint32_t *off, uint64_t noff, EncColumn *table,
                                                       unsigned long long *info) {
    __shared__ unsigned long long sums[kEncThreads / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long at = 0;
    for (uint32_t c0 = 0; c0 <= cols; c0 += kEncThreads) {
        const uint32_t c = c0 + tid;
        EncColumn e{nullptr, 0, 0, 0, 0};
        unsigned long long bytes = 0;
        if (c <= cols) {
            const unsigned long long m = c < cols ? maxes[c] : *code_max;
            e.vals = c < cols ? pilots + (uint64_t)c * per_col : nullptr;
            e.n = c < cols ? per_col : noff;
            e.width = m ? 64 - __clzll((long long)m) : 1;
            bytes = vector_bytes(e.n, e.width);
        }
        unsigned long long incl = bytes;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long t = __shfl_up_sync(kFullMask, incl, d);
            if (lane >= (uint32_t)d) incl += t;
        }
        if (lane == 31) sums[warp] = incl;
        __syncthreads();
        unsigned long long total = 0;
        for (uint32_t v = 0; v < kEncThreads / 32; v++) {
            if (v < warp) incl += sums[v];
            total += sums[v];
        }
        if (c <= cols) {
            e.out = at + incl - bytes;
            table[c] = e;
        }
        at += total;
        __syncthreads();
    }
    if (tid == 0) {
        info[0] = at;
        info[1] = off[noff - 1];
    }
}

// Word t of column blockIdx.x / per_col (t = index among the vector's words, the
// column's CTAs striding over them; the header's four u64 are written by t = 0).
// Words past ceil(n w / 64) are zero.  Nothing is written when the output exceeds `room`.
__global__ void __launch_bounds__(kEncThreads) k_pack(const EncColumn *cols, uint32_t per_col, const uint32_t *off,
                                                      uint32_t psize, int diff, uint8_t *out,
                                                      const unsigned long long *info, uint64_t room) {
    if (info[0] > room) return;
    const EncColumn c = cols[blockIdx.x / per_col];
    const uint64_t chunk = blockIdx.x % per_col;
    const uint32_t w = c.width;
    const uint64_t bits_used = c.n * w;
    const uint64_t words = words_for(bits_used) + 1;
    uint64_t *hdr = reinterpret_cast<uint64_t *>(out + c.out);
    uint64_t *bits = hdr + 4;
    const bool narrow = bits_used + 64 < 0xFFFFFFFFull;  // bit positions fit 32 bits: a 64-bit division costs four times as much
    for (uint64_t t = chunk * blockDim.x + threadIdx.x; t < words; t += (uint64_t)per_col * blockDim.x) {
        if (t == 0) {
            hdr[0] = c.n;
            hdr[1] = w;
            hdr[2] = w == 64 ? ~0ull : (1ull << w) - 1;
            hdr[3] = words;
        }
        const uint64_t lo = 64 * t;  // first bit of this word
        uint64_t word = 0;
        if (lo < bits_used) {
            uint64_t i = narrow ? (uint32_t)lo / w : lo / w;
            // Value i may begin before the word; the following ones begin inside it.
            int32_t pos = (int32_t)(i * w - lo);
            for (; pos < 64 && i < c.n; i++, pos += (int32_t)w) {
                const uint64_t v = c.vals ? (uint64_t)__ldg(c.vals + i) : offset_code(off, i, psize, diff != 0);
                word |= pos >= 0 ? v << pos : v >> -pos;
            }
        }
        bits[t] = word;
    }
}

}  // namespace

phobic_status run_encode_gpu(Worker &w, DeviceArena &out_arena, int pilot_encoder, int offset_encoder,
                             const phobic_result *built, uint32_t partitions, const phobic_params *params,
                             uint8_t *out, size_t cap, int out_on_device, size_t *size, double *bits_per_key,
                             std::string *err) {
    if (!built || !params || !size || (pilot_encoder != 0 && pilot_encoder != 3) ||
        (offset_encoder != 0 && offset_encoder != 1) || params->buckets == 0 || params->partition_size == 0) {
        if (err) *err = "phobic_encode_gpu: unsupported encoder or missing argument";
        return PHOBIC_ERR_INVALID;
    }
    const uint64_t B = params->buckets, P = partitions;
    const uint64_t npil = B * P, noff = P + 1;
    const bool mono = pilot_encoder == 3;
    const uint32_t cols = mono ? 1u : (uint32_t)B;
    PHB_TRY(cudaSetDevice(w.device), "cudaSetDevice");
    phobic_status st = settle(w, err);
    if (st != PHOBIC_OK) return st;
    PHB_TRY(w.pinned.reserve(4096), "pinned");
    cudaStream_t s = w.stream;

    // Inputs on the device; {size, keys, largest offset code} and the columns' maxima, side by side; the
    // column table.
    const size_t info_bytes = align256(24), max_bytes = align256(4 * (size_t)cols);
    const size_t need = align256(4 * npil) + align256(4 * noff) + info_bytes + max_bytes +
                        align256(sizeof(EncColumn) * (cols + 1)) + 4096;
    w.arena.reset();
    PHB_TRY(w.arena.reserve(need), "device arena");
    const uint32_t *d_pil = built->pilots, *d_off = built->partition_offsets;
    if (!built->on_device) {
        uint32_t *a = static_cast<uint32_t *>(w.arena.take(4 * npil));
        uint32_t *b = static_cast<uint32_t *>(w.arena.take(4 * noff));
        if (npil) PHB_TRY(cudaMemcpyAsync(a, built->pilots, 4 * npil, cudaMemcpyHostToDevice, s), "H2D pilots");
        PHB_TRY(cudaMemcpyAsync(b, built->partition_offsets, 4 * noff, cudaMemcpyHostToDevice, s), "H2D offsets");
        d_pil = a, d_off = b;
    }
    unsigned long long *d_info = static_cast<unsigned long long *>(w.arena.take(info_bytes + max_bytes));
    unsigned long long *d_cmax = d_info + 2;
    uint32_t *d_max = reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(d_info) + info_bytes);
    EncColumn *d_cols = static_cast<EncColumn *>(w.arena.take(sizeof(EncColumn) * (cols + 1)));
    PHB_TRY(cudaMemsetAsync(d_info, 0, info_bytes + max_bytes, s), "memset");
    const uint64_t per_col = mono ? npil : P;
    const uint32_t psize = params->partition_size;
    const int diff = offset_encoder == 0;
    const uint32_t gy = (uint32_t)std::max<uint64_t>(
        1, std::min<uint64_t>((std::max(per_col, noff) + kEncThreads * kMaxLoads - 1) / (kEncThreads * kMaxLoads),
                              mono ? (uint64_t)w.sm_count * 8 : 64));
    k_colmax<<<dim3(cols + 1, gy), kEncThreads, 0, s>>>(d_pil, per_col, cols, d_max, d_off, noff, psize, diff, d_cmax);
    PHB_TRY(cudaGetLastError(), "k_colmax");
    k_table<<<1, kEncThreads, 0, s>>>(d_max, d_cmax, d_pil, per_col, cols, d_off, noff, d_cols, d_info);
    PHB_TRY(cudaGetLastError(), "k_table");
    // The widths are not known here: CTAs for columns of up to 32-bit values (they stride over more).
    const uint64_t max_words = (std::max(per_col, noff) + 1) / 2 + 2;
    const uint64_t per = std::min<uint64_t>((max_words + kEncThreads - 1) / kEncThreads,
                                            std::max<uint64_t>(1, (uint64_t)w.sm_count * 16 / (cols + 1)));
    auto pack = [&](uint8_t *to, uint64_t room) {
        k_pack<<<(uint32_t)(per * (cols + 1)), kEncThreads, 0, s>>>(d_cols, (uint32_t)per, d_off, psize, diff, to, d_info,
                                                                    room);
        return cudaGetLastError();
    };
    // The kernel stores 8-byte words: only a device destination that is 8-byte aligned and large
    // enough is written directly.
    const bool direct = out && out_on_device && !(reinterpret_cast<uintptr_t>(out) & 7);
    if (direct) PHB_TRY(pack(out, cap), "k_pack");
    unsigned long long *h_info = static_cast<unsigned long long *>(w.pinned.data());
    PHB_TRY(cudaMemcpyAsync(h_info, d_info, 16, cudaMemcpyDeviceToHost, s), "D2H size");
    PHB_TRY(cudaEventRecord(w.ev[7], s), "event");
    if ((st = wait_event(w.ev[7], w.timeout_ms, err)) != PHOBIC_OK) return st;
    w.unsettled = false;
    const uint64_t total = h_info[0], n = h_info[1];
    *size = total;
    // getBitsPerKey (mphf.hpp:88-91): encoder bits (8 per serialised byte), fulcrums and partition count.
    if (bits_per_key) *bits_per_key = n ? (double)(float(total * 8 + 32 * (uint64_t)kFulcrums + 32 * P) / float(n)) : 0.0;
    if (!out || (direct && total <= cap)) return PHOBIC_OK;

    w.unsettled = true;
    PHB_TRY(out_arena.reserve(total), "device output");
    out_arena.reset();
    uint8_t *d_out = static_cast<uint8_t *>(out_arena.take(total));
    PHB_TRY(pack(d_out, total), "k_pack");
    const size_t ncopy = std::min<size_t>(cap, total);
    if (ncopy)
        PHB_TRY(cudaMemcpyAsync(out, d_out, ncopy, out_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, s),
                "copy out");
    PHB_TRY(cudaEventRecord(w.ev[7], s), "event");
    if ((st = wait_event(w.ev[7], w.timeout_ms, err)) == PHOBIC_OK) w.unsettled = false;
    return st;
}

}  // namespace phobicb200

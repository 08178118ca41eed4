// Encode-side kernels.  Two families:
//  * the two per-stream operators of the reference (character / word output, one thread per
//    stream, reference src/kernel.cu:590-610 and :767-811), kept for operator compatibility;
//  * the whole-layer two-pass encoder that writes the device format directly from the BF16
//    weight: one thread per stream, 64 consecutive threads per record, so that the BF16 reads
//    (2 columns per thread, 256 B per record and block) and the interleaved word stores
//    (64 words per record row) are coalesced.
#pragma once

#include "bhi_common.cuh"

namespace bhi {

// ---- operator-compatible per-stream encoders ------------------------------------------------------
__global__ void huffman_encode_chars_kernel(const uint8_t *__restrict__ data, int streams, int n,
                                            const uint8_t *__restrict__ lut, uint8_t *__restrict__ out,
                                            int32_t *__restrict__ out_len) {
    __shared__ uint8_t codes[256 * 32];
    for (int i = threadIdx.x; i < 256 * 32; i += blockDim.x) codes[i] = lut[i];
    __syncthreads();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= streams) return;
    const uint8_t *src = data + static_cast<int64_t>(t) * n;
    uint8_t *dst = out + static_cast<int64_t>(t) * n * 32;
    int32_t cnt = 0;
    for (int i = 0; i < n; i++) {
        const uint8_t *c = codes + 32 * src[i];
        for (int j = 0; j < 32 && c[j] != 0; j++) dst[cnt++] = c[j];
    }
    out_len[t] = cnt;
}

// One entry of an rANS encoding model.  A state is below freq << 32 <= 2^47 when it is divided (models have at most 15 bits),
// so its quotient by freq is the high half of (2 * state) * inv with inv = ceil(2^63 / freq): the excess
// inv * freq - 2^63 is below freq <= 2^15 and 2^47 * 2^15 < 2^63, so no quotient is off by one.  (A 64-bit division in its place
// lies on the serial chain of every stream: size and emit pass over a 12288 x 4096 layer took 279 and 287 us with it, 81 and 95 us
// with the product; the whole-layer encoder's form of it is below.)
struct AnsModel {
    uint64_t inv[256];
    uint32_t freq[256], cum[256];
};

__device__ __forceinline__ void load_model(AnsModel &t, const uint32_t *freq, const uint32_t *cum) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        const uint32_t f = freq[i];
        t.freq[i] = f;
        t.cum[i] = cum[i];
        t.inv[i] = f ? ((1ull << 63) + f - 1u) / f : 0ull;
    }
}

// Probability precision of a model: its frequencies sum to 2^bits (cum[255] + freq[255] is that sum).
__device__ __forceinline__ uint32_t ans_model_bits(const AnsModel &t) {
    const uint32_t total = t.cum[255] + t.freq[255];
    return total ? 31u - static_cast<uint32_t>(__clz(total)) : kAnsBitsMin;
}

// rANS step shared by all encoders: emits renormalisation words through `put(word)`.  A symbol that the model does not
// hold (frequency 0) has no code; it leaves the state alone.
template <class Put>
__device__ __forceinline__ void ans_push(uint64_t &state, const AnsModel &t, uint32_t sym, uint32_t bits, Put &&put) {
    const uint32_t f = t.freq[sym];
    if (f == 0u) return;
    if ((state >> 32) >= f) {                      // once is enough: the state is below 2^(32 + bits) and f >= 1
        put(static_cast<uint32_t>(state));
        state >>= 32;
    }
    const uint32_t q = static_cast<uint32_t>(__umul64hi(state << 1, t.inv[sym]));
    const uint32_t r = static_cast<uint32_t>(state) - q * f;
    state = (static_cast<uint64_t>(q) << bits) + r + t.cum[sym];
}

__global__ void ans_encode_words_kernel(const uint8_t *__restrict__ data, int streams, int n,
                                        const uint32_t *__restrict__ freq, const uint32_t *__restrict__ cum,
                                        uint32_t *__restrict__ out, int32_t *__restrict__ out_len) {
    __shared__ AnsModel model;
    load_model(model, freq, cum);
    __syncthreads();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= streams) return;
    const uint8_t *src = data + static_cast<int64_t>(t) * n;
    uint32_t *dst = out + static_cast<int64_t>(t) * n * 8;
    const uint32_t bits = ans_model_bits(model);
    uint64_t state = 1ull << bits;
    int32_t cnt = 0;
    auto put = [&](uint32_t w) { dst[cnt++] = w; };
    for (int i = n - 1; i >= 0; i--) ans_push(state, model, src[i], bits, put);
    while (state > 0) { put(static_cast<uint32_t>(state)); state >>= 32; }
    for (int i = 0; i < cnt / 2; i++) {
        const uint32_t a = dst[i];
        dst[i] = dst[cnt - 1 - i];
        dst[cnt - 1 - i] = a;
    }
    out_len[t] = cnt;
}

// ---- whole-layer encoder ---------------------------------------------------------------------------
constexpr int kEncThreads = 256;                 // 4 records per block
constexpr int kEncRecords = kEncThreads / 64;
constexpr int kEncAhead = 4;                     // blocks of a record that are loaded together

struct EncGeom {
    const uint16_t *W;     // [M, K]
    int M, K, S, Nc;
};

// thread -> (record, stream); returns false past the end
__device__ __forceinline__ bool enc_locate(const EncGeom &g, int64_t &rec, int &k, int &m, int &st) {
    rec = static_cast<int64_t>(blockIdx.x) * kEncRecords + (threadIdx.x >> 6);
    st = threadIdx.x & 63;
    if (rec >= static_cast<int64_t>(g.S) * g.M) return false;
    k = static_cast<int>(rec / g.M);
    m = static_cast<int>(rec - static_cast<int64_t>(k) * g.M);
    return true;
}

// the two BF16 values (as one u32) a stream owns in block `blk` of its record
__device__ __forceinline__ uint32_t enc_pair(const EncGeom &g, int k, int m, int st, int blk) {
    const uint16_t *p = g.W + static_cast<int64_t>(m) * g.K + static_cast<int64_t>(k) * g.Nc + blk * 128 + 2 * st;
    return __ldg(reinterpret_cast<const uint32_t *>(p));
}
__device__ __forceinline__ uint32_t exp_lo(uint32_t pair) { return (pair >> 7) & 0xFF; }
__device__ __forceinline__ uint32_t exp_hi(uint32_t pair) { return (pair >> 23) & 0xFF; }

// max over the 64 threads of a record (two warps) -> every thread of the record gets it
__device__ __forceinline__ uint32_t record_max(uint32_t v, uint32_t *scratch /*[kEncThreads/32]*/) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) scratch[w] = v;
    __syncthreads();
    return max(scratch[w & ~1], scratch[w | 1]);
}

__global__ void __launch_bounds__(kEncThreads)
huffman_size_kernel(EncGeom g, const uint8_t *__restrict__ code_len, int32_t *__restrict__ words_per_row) {
    __shared__ uint8_t len[256];
    __shared__ uint32_t scratch[kEncThreads / 32];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) len[i] = code_len[i];
    __syncthreads();
    int64_t rec; int k, m, st;
    const bool live = enc_locate(g, rec, k, m, st);
    uint32_t bits = 0;
    if (live)
        for (int blk = 0; blk < (g.Nc >> 7); blk++) {
            const uint32_t p = enc_pair(g, k, m, st, blk);
            bits += len[exp_lo(p)] + len[exp_hi(p)];
        }
    const uint32_t worst = record_max(bits, scratch);
    if (live && st == 0) words_per_row[rec] = static_cast<int32_t>(((worst + 7) / 8 + 3) / 4);
}

__device__ __forceinline__ void store_rem(uint8_t *rem_row, int st, int blk, uint32_t pair) {
    // stream st = h*32 + lane owns bytes blk*128 + lane*4 + h*2 + {0,1} (reference functional.py:184)
    const uint32_t lo = ((pair >> 8) & 0x80) | (pair & 0x7F);
    const uint32_t hi = ((pair >> 24) & 0x80) | ((pair >> 16) & 0x7F);
    *reinterpret_cast<uint16_t *>(rem_row + blk * 128 + (st & 31) * 4 + (st >> 5) * 2) = static_cast<uint16_t>(lo | (hi << 8));
}

// The coded words of every record.  What bounds it is the work per symbol (12288 x 4096: 43 us, of which HBM 19; with one table of
// codes and one of lengths 62), so the table has a copy for each lane: the 32 lookups of a warp always hit 32 different banks, and
// their address is the exponent where it stands in the weight (128 bytes per entry).  Codes of at most 16 bits, which all but the
// reference's own builder make, stand with their lengths in one word and are joined in pairs.  Blocks stay for several records, as
// the copies take a while to write.
constexpr int kEncBlocksPerSm = 6;               // 33 KB of shared memory each

__global__ void __launch_bounds__(kEncThreads, kEncBlocksPerSm)
huffman_emit_kernel(EncGeom g, const uint8_t *__restrict__ code_len, const uint32_t *__restrict__ code_val,
                    const int32_t *__restrict__ offsets, uint8_t *rem, uint32_t *__restrict__ exp) {
    __shared__ uint32_t table[256 * 32];
    __shared__ uint8_t len[256];
    static_assert(kEncThreads == 256, "a thread writes one symbol's copies");
    const uint32_t my_len = code_len[threadIdx.x], my_val = code_val[threadIdx.x];
    len[threadIdx.x] = static_cast<uint8_t>(my_len);
    const bool pairs = !__syncthreads_or(my_len > 16u);
    for (int i = 0; i < 32; i++) table[threadIdx.x * 32 + ((i + threadIdx.x) & 31)] = pairs ? my_val | my_len << 16 : my_val;
    __syncthreads();
    const uint8_t *mine = reinterpret_cast<const uint8_t *>(table) + 4 * (threadIdx.x & 31);
    auto entry = [&](uint32_t at) { return *reinterpret_cast<const uint32_t *>(mine + at); };
    const int nblk = g.Nc >> 7, st = threadIdx.x & 63;
    const int64_t records = static_cast<int64_t>(g.S) * g.M;
    for (int64_t rec = static_cast<int64_t>(blockIdx.x) * kEncRecords + (threadIdx.x >> 6); rec < records; rec += static_cast<int64_t>(gridDim.x) * kEncRecords) {
        const int k = static_cast<int>(rec / g.M), m = static_cast<int>(rec - static_cast<int64_t>(k) * g.M);
        uint8_t *rem_row = rem ? rem + rec * g.Nc : nullptr;
        uint32_t *out = exp + static_cast<uint32_t>(offsets[rec]) + st;
        uint64_t acc = 0;
        uint32_t have = 0;
        auto append = [&](uint32_t bits, uint32_t n) {                 // n <= 32
            acc |= static_cast<uint64_t>(bits) << have;
            have += n;
            if (have >= 32u) {
                *out = static_cast<uint32_t>(acc);
                out += kStreamsPerRecord;
                acc >>= 32;
                have -= 32u;
            }
        };
        for (int blk = 0; blk < nblk; blk += kEncAhead) {
            uint32_t p[kEncAhead];
#pragma unroll
            for (int i = 0; i < kEncAhead; i++) p[i] = blk + i < nblk ? enc_pair(g, k, m, st, blk + i) : 0u;
#pragma unroll
            for (int i = 0; i < kEncAhead; i++) {
                if (blk + i < nblk) {
                    if (rem_row) store_rem(rem_row, st, blk + i, p[i]);
                    const uint32_t e0 = entry(p[i] & 0x7F80u), e1 = entry((p[i] >> 16) & 0x7F80u);
                    if (pairs) {
                        append((e0 & 0xFFFFu) | (e1 & 0xFFFFu) << (e0 >> 16), (e0 >> 16) + (e1 >> 16));
                    } else {
                        append(e0, len[exp_lo(p[i])]);
                        append(e1, len[exp_hi(p[i])]);
                    }
                }
            }
        }
        if (have > 0) *out = static_cast<uint32_t>(acc);
    }
}

// rANS over one stream of a record, symbols last to first; `put` sees words in emission order.  Bound by the integer work of a
// step and its chain: 12288 x 4096 73 us in the size pass and 86 in the emit pass (79 and 92 with one model for all lanes and a
// 64-bit product).  The model has a copy for each lane (96 KB, two blocks of 512 threads per SM, which stay for several records):
// the lookups of a warp hit 32 different banks.
constexpr int kAnsEncThreads = 512;
constexpr int kAnsEncRecords = kAnsEncThreads / 64;
constexpr int kAnsEncBytes = 256 * 32 * 12;

struct AnsLaneModel {
    const uint2 *inv;          // [256][32], this lane's column
    const uint32_t *fc;        // freq | cum << 16, the same
    uint32_t bits;
};

__device__ __forceinline__ AnsLaneModel load_lane_model(uint8_t *smem, const uint32_t *freq, const uint32_t *cum) {
    uint2 *inv = reinterpret_cast<uint2 *>(smem);
    uint32_t *fc = reinterpret_cast<uint32_t *>(smem + 256 * 32 * 8);
    const uint32_t s = threadIdx.x & 255u, first = (threadIdx.x >> 8) * 16u;       // two threads per symbol
    const uint32_t f = freq[s], c = cum[s];
    const uint64_t v = f ? ((1ull << 63) + f - 1u) / f : 0ull;                     // see AnsModel
    for (uint32_t i = 0; i < 16u; i++) {
        const uint32_t at = 32u * s + ((first + i + s) & 31u);
        inv[at] = make_uint2(static_cast<uint32_t>(v), static_cast<uint32_t>(v >> 32));
        fc[at] = f | c << 16;
    }
    const uint32_t total = cum[255] + freq[255];
    __syncthreads();
    return {inv + (threadIdx.x & 31), fc + (threadIdx.x & 31), total ? 31u - static_cast<uint32_t>(__clz(total)) : kAnsBitsMin};
}

template <class Put>
__device__ __forceinline__ void ans_encode_record_stream(const EncGeom &g, int k, int m, int st, const AnsLaneModel &t, Put &&put) {
    // As ans_push, word by word: the state's high word is below f <= 2^15 once it is renormalised, which leaves four products of
    // the quotient's long multiplication and no carries; r + cum fills the bits below q << bits.
    uint32_t lo = 1u << t.bits, hi = 0u;
    auto push = [&](uint32_t sym) {
        const uint32_t w = t.fc[32u * sym], f = w & 0xFFFFu;
        if (f == 0u) return;
        const uint2 v = t.inv[32u * sym];
        if (hi >= f) {
            put(lo);
            lo = hi;
            hi = 0u;
        }
        const uint64_t mid = static_cast<uint64_t>(hi) * v.x + (static_cast<uint64_t>(lo) * v.y + __umulhi(lo, v.x));
        const uint32_t top = hi * v.y + static_cast<uint32_t>(mid >> 32);
        const uint32_t q = __funnelshift_l(static_cast<uint32_t>(mid), top, 1);
        lo = q * ((1u << t.bits) - f) + (lo + (w >> 16));              // q 2^bits + (lo - q f) + cum
        hi = q >> (32u - t.bits);
    };
    for (int last = (g.Nc >> 7) - 1; last >= 0; last -= kEncAhead) {
        uint32_t p[kEncAhead];
#pragma unroll
        for (int i = 0; i < kEncAhead; i++) p[i] = last >= i ? enc_pair(g, k, m, st, last - i) : 0u;
#pragma unroll
        for (int i = 0; i < kEncAhead; i++) {
            if (last >= i) {
                push(exp_hi(p[i]));
                push(exp_lo(p[i]));
            }
        }
    }
    if (lo | hi) put(lo);
    if (hi) put(hi);
}

__global__ void __launch_bounds__(kAnsEncThreads, 2)
ans_size_kernel(EncGeom g, const uint32_t *__restrict__ freq, const uint32_t *__restrict__ cum,
                int32_t *__restrict__ words_per_row, uint8_t *__restrict__ stream_words) {
    extern __shared__ __align__(16) uint8_t enc_smem[];
    __shared__ uint32_t worst_of[kAnsEncThreads / 32];
    const AnsLaneModel model = load_lane_model(enc_smem, freq, cum);
    const int st = threadIdx.x & 63, warp = threadIdx.x >> 5;
    const int64_t records = static_cast<int64_t>(g.S) * g.M;
    for (int64_t first = static_cast<int64_t>(blockIdx.x) * kAnsEncRecords; first < records; first += static_cast<int64_t>(gridDim.x) * kAnsEncRecords) {
        const int64_t rec = first + (threadIdx.x >> 6);
        uint32_t cnt = 0;
        if (rec < records) {
            const int k = static_cast<int>(rec / g.M), m = static_cast<int>(rec - static_cast<int64_t>(k) * g.M);
            ans_encode_record_stream(g, k, m, st, model, [&](uint32_t) { cnt++; });
            stream_words[rec * 64 + st] = static_cast<uint8_t>(cnt);
        }
        const uint32_t worst = __reduce_max_sync(0xFFFFFFFFu, cnt);
        if ((threadIdx.x & 31) == 0) worst_of[warp] = worst;
        __syncthreads();
        if (rec < records && st == 0) words_per_row[rec] = static_cast<int32_t>(max(worst_of[warp], worst_of[warp + 1]));
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kAnsEncThreads, 2)
ans_emit_kernel(EncGeom g, const uint32_t *__restrict__ freq, const uint32_t *__restrict__ cum,
                const int32_t *__restrict__ offsets, const uint8_t *__restrict__ stream_words,
                uint8_t *rem, uint32_t *__restrict__ exp) {
    extern __shared__ __align__(16) uint8_t enc_smem[];
    const AnsLaneModel model = load_lane_model(enc_smem, freq, cum);
    const int st = threadIdx.x & 63;
    const int64_t records = static_cast<int64_t>(g.S) * g.M;
    for (int64_t rec = static_cast<int64_t>(blockIdx.x) * kAnsEncRecords + (threadIdx.x >> 6); rec < records;
         rec += static_cast<int64_t>(gridDim.x) * kAnsEncRecords) {
        const int k = static_cast<int>(rec / g.M), m = static_cast<int>(rec - static_cast<int64_t>(k) * g.M);
        if (rem) {
            uint8_t *rem_row = rem + rec * g.Nc;
            for (int blk = 0; blk < (g.Nc >> 7); blk++) store_rem(rem_row, st, blk, enc_pair(g, k, m, st, blk));
        }
        // the j-th emitted word is the (cnt-1-j)-th word the decoder reads
        uint32_t *out = exp + static_cast<uint32_t>(offsets[rec]) + st;
        int at = static_cast<int>(stream_words[rec * 64 + st]) - 1;
        ans_encode_record_stream(g, k, m, st, model, [&](uint32_t w) {
            if (at >= 0) out[static_cast<int64_t>(at) * kStreamsPerRecord] = w;
            at--;
        });
    }
}

// ---- sign/mantissa plane and exponent histogram ----------------------------------------------------------------------
// One pass over a slab of rows: both results need every weight and neither needs a code table, so the weight is read
// once for both, and slabs of a weight that is still on its way from the host are taken as they arrive.  Bound by HBM
// (3 bytes per weight) and the shared-memory adds: 49 us at 12288 x 4096, 24 us without the plane.  A warp takes four consecutive
// 128-column blocks at a time: two 128-byte loads and one 128-byte store per block, eight loads in flight per lane.  Counts go to
// a column of the block's table that belongs to the lane: the 32 adds of a warp always hit 32 different banks, however few
// exponents occur.
constexpr int kSplitThreads = 256;
constexpr int kSplitUnroll = 4;

__global__ void __launch_bounds__(kSplitThreads)
split_histogram_kernel(const uint32_t *__restrict__ W, int rows, int row0, int M, int kblocks, int nblk, uint8_t *rem,
                       unsigned long long *hist) {
    __shared__ uint32_t counts[256 * 32];
    for (int i = threadIdx.x; i < 256 * 32; i += kSplitThreads) counts[i] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t total = static_cast<int64_t>(rows) * kblocks;
    const int64_t warp = static_cast<int64_t>(blockIdx.x) * (kSplitThreads / 32) + (threadIdx.x >> 5);
    const int64_t step = static_cast<int64_t>(gridDim.x) * (kSplitThreads / 32) * kSplitUnroll;
    uint32_t *mine = counts + lane;
    for (int64_t g0 = warp * kSplitUnroll; g0 < total; g0 += step) {
        uint32_t a[kSplitUnroll], b[kSplitUnroll];
#pragma unroll
        for (int j = 0; j < kSplitUnroll; j++) {
            if (g0 + j < total) {
                a[j] = __ldg(W + (g0 + j) * 64 + lane);
                b[j] = __ldg(W + (g0 + j) * 64 + 32 + lane);
            }
        }
        int m = static_cast<int>(g0 / kblocks);
        int kb = static_cast<int>(g0 - static_cast<int64_t>(m) * kblocks);
#pragma unroll
        for (int j = 0; j < kSplitUnroll; j++) {
            if (g0 + j < total) {
                if (hist) {
                    atomicAdd(mine + 32 * exp_lo(a[j]), 1u);
                    atomicAdd(mine + 32 * exp_hi(a[j]), 1u);
                    atomicAdd(mine + 32 * exp_lo(b[j]), 1u);
                    atomicAdd(mine + 32 * exp_hi(b[j]), 1u);
                }
                if (rem) {
                    const int k = kb / nblk, blk = kb - k * nblk;
                    // bytes (lo, hi) of each pair: sign in bit 7, mantissa below
                    const uint32_t sa = (a[j] & 0x007F007Fu) | ((a[j] >> 8) & 0x00800080u);
                    const uint32_t sb = (b[j] & 0x007F007Fu) | ((b[j] >> 8) & 0x00800080u);
                    uint32_t *dst = reinterpret_cast<uint32_t *>(
                        rem + (((static_cast<int64_t>(k) * M + row0 + m) * nblk + blk) << 7));
                    dst[lane] = prmt(sa, sb, 0x6420u);
                }
                if (++kb == kblocks) {
                    kb = 0;
                    m++;
                }
            }
        }
    }
    if (hist) {
        __syncthreads();
        uint32_t n = 0;
#pragma unroll 8
        for (int i = 0; i < 32; i++) n += counts[threadIdx.x * 32 + ((threadIdx.x + i) & 31)];
        if (n) atomicAdd(hist + threadIdx.x, static_cast<unsigned long long>(n));
    }
}

// ---- code tables of a layer, from its histogram --------------------------------------------------------------------------
// The same tables as the host's builders make, on the device: the host would have to wait for the histogram, build, and send
// the tables back before the size pass can start (two codes: 0.45 ms of a conversion of 0.9 ms).  One block each; what bounds
// it is a chain of a few hundred dependent steps.  Histograms that these kernels do not serve (more symbols than the limit
// allows, a frequency that its field cannot hold) set `status` and leave tables of zeros, or with that frequency cut off in the
// decode table: the size pass reads them before anybody has looked at the status.  The host builds the tables after all (for more
// than 64 exponents in 13 ms, beside which that pass does not show: 4096 x 4096 14.8 ms with and without it).
constexpr int kTableThreads = 256;
constexpr int kLimitMax = 8;

// exclusive sum over the block's 256 values
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t *scratch /*[8]*/) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t run = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, run, o);
        if (lane >= o) run += up;
    }
    __syncthreads();
    if (lane == 31) scratch[warp] = run;
    __syncthreads();
    for (int w = 0; w < warp; w++) run += scratch[w];
    return run - v;
}

// Optimal prefix code with no length above `limit` (package-merge) in canonical order.  A level's list is the leaves merged
// with the packages (pairs) of the level before, leaves first where weights are equal.  Every level holds the leaves in their
// own order, so a leaf's length is the number of levels whose chosen prefix reaches it: 2 n - 2 items of the last level, and
// of each level before, two for each package chosen after it.
__global__ void __launch_bounds__(kTableThreads)
huffman_limit_tables_kernel(const long long *__restrict__ hist, int limit, uint8_t *lut1, uint8_t *lut2, uint8_t *lut3, uint8_t *lut4,
                            uint8_t *code_lengths, uint32_t *code_values, int64_t *status) {
    constexpr int kMax = 1 << kLimitMax;
    __shared__ long long weight[kMax], list[2 * kMax], packages[kMax];
    __shared__ uint8_t sym[kMax], used[256], isleaf[2 * kMax], len_of[256];          // sym: by rank, used: in order
    __shared__ uint16_t leaves_before[kLimitMax][2 * kMax + 1];        // of each level, among its first i items
    __shared__ uint32_t scratch[8], value_of[256];
    const int tid = threadIdx.x;
    const long long mine = hist[tid];
    const uint32_t at = block_scan(mine > 0 ? 1u : 0u, scratch);
    const int n = __syncthreads_count(mine > 0);
    if (tid == 0) *status = n > (1 << limit) || n == 0;
    if (n > (1 << limit) || n == 0) {
        lut1[tid] = lut2[tid] = lut3[tid] = lut4[tid] = code_lengths[tid] = 0;
        code_values[tid] = 0u;
        return;
    }
    len_of[tid] = 0;
    value_of[tid] = 0u;
    if (mine > 0) {
        used[at] = static_cast<uint8_t>(tid);
        list[at] = mine;                                               // (the counts, for the ranks below)
    }
    __syncthreads();
    // leaves by (weight, symbol)
    if (mine > 0) {
        int rank = 0;
        for (int i = 0; i < n; i++) rank += list[i] < mine || (list[i] == mine && i < static_cast<int>(at));
        weight[rank] = mine;
        sym[rank] = static_cast<uint8_t>(tid);
    }
    __syncthreads();
    // levels
    int items = n;
    if (tid < n) {
        list[tid] = weight[tid];
        leaves_before[0][tid + 1] = static_cast<uint16_t>(tid + 1);
    }
    if (tid < limit) leaves_before[tid][0] = 0;
    __syncthreads();
    for (int level = 1; level < limit; level++) {
        const int pairs = items / 2;
        if (tid < pairs) packages[tid] = list[2 * tid] + list[2 * tid + 1];
        __syncthreads();
        if (tid < n) {
            int lo = 0, hi = pairs;                                    // packages lighter than this leaf
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (packages[mid] < weight[tid]) lo = mid + 1;
                else hi = mid;
            }
            list[tid + lo] = weight[tid];
            isleaf[tid + lo] = 1;
        }
        if (tid < pairs) {
            int lo = 0, hi = n;                                        // leaves no heavier than this package
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (weight[mid] <= packages[tid]) lo = mid + 1;
                else hi = mid;
            }
            list[tid + lo] = packages[tid];
            isleaf[tid + lo] = 0;
        }
        items = n + pairs;
        __syncthreads();
        const uint32_t a = 2 * tid < items ? isleaf[2 * tid] : 0u, b = 2 * tid + 1 < items ? isleaf[2 * tid + 1] : 0u;
        const uint32_t before = block_scan(a + b, scratch);
        if (2 * tid < items) leaves_before[level][2 * tid + 1] = static_cast<uint16_t>(before + a);
        if (2 * tid + 1 < items) leaves_before[level][2 * tid + 2] = static_cast<uint16_t>(before + a + b);
        __syncthreads();
    }
    if (tid < n) {
        int chosen = 2 * n - 2, length = n == 1 ? 1 : 0;
        for (int level = limit - 1; level >= 0; level--) {
            const int leaves = leaves_before[level][chosen];
            length += tid < leaves;
            chosen = 2 * (chosen - leaves);
        }
        len_of[sym[tid]] = static_cast<uint8_t>(length);
    }
    __syncthreads();
    // canonical codes: by (length, symbol); a code is the number of leaves of the full tree to its left
    const int length = len_of[tid];
    if (length > 0) {
        uint32_t code = 0;
        for (int i = 0; i < n; i++) {
            const int s = used[i], l = len_of[s];
            if (l < length || (l == length && s < tid)) code += 1u << (kLimitMax - l);
        }
        value_of[tid] = __brev(code >> (kLimitMax - length)) >> (32 - length);
    }
    __syncthreads();
    int found = 255;
    for (int i = 0; i < n; i++) {
        const int s = used[i];
        if ((tid & ((1 << len_of[s]) - 1)) == static_cast<int>(value_of[s])) found = s;
    }
    lut1[tid] = static_cast<uint8_t>(found);
    lut2[tid] = lut3[tid] = lut4[tid] = 255;
    code_lengths[tid] = static_cast<uint8_t>(length);
    code_values[tid] = value_of[tid];
}

// rANS model: counts scaled to a sum of 2^bits (rounded half to even, at least 1), the difference handed out or taken back unit
// by unit over the symbols in the order of their rounding errors.
__global__ void __launch_bounds__(kTableThreads)
ans_tables_kernel(const long long *__restrict__ hist, int bits, uint32_t *freq, uint32_t *cum, uint32_t *lut, int64_t *status) {
    __shared__ double err[256];
    __shared__ int scaled[256], order[256];
    __shared__ uint32_t scratch[8];
    __shared__ unsigned long long total;
    __shared__ int have;
    const int tid = threadIdx.x, target = 1 << bits;
    const long long mine = hist[tid];
    if (tid == 0) {
        total = 0ull;
        have = 0;
    }
    __syncthreads();
    atomicAdd(&total, static_cast<unsigned long long>(mine));
    __syncthreads();
    const int at = static_cast<int>(block_scan(mine > 0 ? 1u : 0u, scratch));
    const int n = __syncthreads_count(mine > 0);
    int q = 0;
    double e = 0.0;
    if (mine > 0) {
        const double exact = static_cast<double>(mine * target) / static_cast<double>(total);
        q = max(static_cast<int>(rint(exact)), 1);
        e = exact - q;
    }
    if (mine > 0) {
        err[at] = e;
        atomicAdd(&have, q);
    }
    scaled[tid] = q;
    __syncthreads();
    const bool small = have < target;
    if (mine > 0) {                                                    // largest underestimate first, or largest overestimate
        int rank = 0;
        for (int i = 0; i < n; i++)
            if (i != at) rank += small ? err[i] > e || (err[i] == e && i > at) : err[i] < e || (err[i] == e && i < at);
        order[rank] = tid;
    }
    __syncthreads();
    if (tid == 0) {
        int rest = target - have;
        if (n > 0 && n <= target) {
            for (int i = 0; rest > 0; i = i + 1 == n ? 0 : i + 1) {
                scaled[order[i]]++;
                rest--;
            }
            for (int i = 0; rest < 0; i = i + 1 == n ? 0 : i + 1) {
                if (scaled[order[i]] > 1) {
                    scaled[order[i]]--;
                    rest++;
                }
            }
        }
        have = target - rest;
    }
    __syncthreads();
    const uint32_t f = scaled[tid];
    const int wide = __syncthreads_count(f > 0xFFFu);
    if (tid == 0) *status = wide > 0 || have != target;
    if (have != target) {
        freq[tid] = cum[tid] = 0u;
        for (int slot = tid; slot < target; slot += kTableThreads) lut[slot] = 0u;
        return;
    }
    const uint32_t c = block_scan(f, scratch);
    freq[tid] = f;
    cum[tid] = c;
    order[tid] = static_cast<int>(c);
    __syncthreads();
    for (int slot = tid; slot < target; slot += kTableThreads) {
        int lo = 0, hi = 256;                                          // the last symbol whose slots start here or before
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (order[mid] <= slot) lo = mid;
            else hi = mid;
        }
        lut[slot] = (static_cast<uint32_t>(lo) << 24) | ((static_cast<uint32_t>(scaled[lo]) & 0xFFFu) << 12) | static_cast<uint32_t>(slot - order[lo]);
    }
}

// ---- record offsets --------------------------------------------------------------------------------------------------
// Exclusive sum of the record sizes (64 words per record row; 64 more after every slab of `slab` rows and after the last
// row of a chunk), in storage order.  One block: a layer has some thousand records, and the launch waits for the size
// pass anyway.  offsets are exact modulo 2^32; total[0] is the whole sum, which the caller has to hold below 2^31.
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 8;

__global__ void __launch_bounds__(kScanThreads)
record_offsets_kernel(const int32_t *__restrict__ words_per_row, int64_t records, int M, int slab, int32_t *__restrict__ offsets,
                      int64_t *__restrict__ total) {
    __shared__ int64_t warp_sums[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t base = 0;
    for (int64_t tile = 0; tile < records; tile += kScanThreads * kScanItems) {
        const int64_t first = tile + static_cast<int64_t>(threadIdx.x) * kScanItems;
        int64_t size[kScanItems], sum = 0;
        int m = static_cast<int>(first % M);
#pragma unroll
        for (int i = 0; i < kScanItems; i++) {
            size[i] = 0;
            if (first + i < records) {
                const int pad = (m % slab == slab - 1 || m == M - 1) ? 64 : 0;
                size[i] = static_cast<int64_t>(words_per_row[first + i]) * 64 + pad;
            }
            sum += size[i];
            if (++m == M) m = 0;
        }
        int64_t scan = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t up = __shfl_up_sync(0xFFFFFFFFu, scan, o);
            if (lane >= o) scan += up;
        }
        if (lane == 31) warp_sums[warp] = scan;
        __syncthreads();
        int64_t before = 0, all = 0;
        for (int w = 0; w < kScanThreads / 32; w++) {
            const int64_t s = warp_sums[w];
            if (w < warp) before += s;
            all += s;
        }
        int64_t at = base + before + scan - sum;
#pragma unroll
        for (int i = 0; i < kScanItems; i++) {
            if (first + i < records) offsets[first + i] = static_cast<int32_t>(at);
            at += size[i];
        }
        base += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = base;
}

}  // namespace bhi

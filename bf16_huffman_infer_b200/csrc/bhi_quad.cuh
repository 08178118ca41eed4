// Decoders of four weight rows at a time over records staged in a ring (see bhi_tileq.cuh, which uses them).
//
// A *quad* is four consecutive weight rows.  Lane (r = lane/8, s = (lane/4)%2, t = lane%4) of a warp runs the two streams
// sigma = 8j + 4s + t and sigma + 32 of row r, j being the warp's pass; records are shifted by 32 bytes against each other,
// so the 32 lanes read 32 different banks.  A Huffman stream is a bit cursor; one 32-bit window fetched under it serves two
// lookups of the folded pair table (two blocks, four symbols).  Windows a 12-bit index cannot resolve as two symbols are
// flagged in the entry; the warp then re-decodes those streams symbol by symbol.  rANS decoding follows the reference's
// state update, refills from the ring.
#pragma once

#include "bhi_staged.cuh"

namespace bhi {

constexpr int kQuadGroups = 8;                                 // warp groups per CTA, one quad each at a time
constexpr int kQuadCtrlBytes = 1024;                           // mbarriers
constexpr uint32_t kQuadRingWant = 59u * 256u;                 // per group: two units of four 7-row records
constexpr uint32_t kEntFlags = kEntSingle | kEntExact;

struct QuadGeom {
    uint32_t lut_bytes;        // fast table region (copies * one table)
    uint32_t copy_shift;       // log2(bytes between consecutive table entries) = 2 + log2(copies)
    uint32_t index_mask;       // table index bits, already at their place in a biased window
    uint32_t ring_off;
    uint32_t ring_bytes;       // per group
};

__device__ __forceinline__ uint32_t lds32(const uint8_t *smem, uint32_t a) { return *reinterpret_cast<const uint32_t *>(smem + a); }

// barrier among the warps of one group: hardware barrier group + 1 (0 is the CTA-wide one).  Literal
// barrier numbers, so that the kernel reserves nine barriers and not all sixteen.
__device__ __forceinline__ void group_barrier(int group, int threads) {
#define BHI_GROUP_BAR(g) \
    case g: asm volatile("bar.sync " #g " + 1, %0;" ::"r"(threads) : "memory"); break;
    switch (group) {
        BHI_GROUP_BAR(0) BHI_GROUP_BAR(1) BHI_GROUP_BAR(2) BHI_GROUP_BAR(3)
        BHI_GROUP_BAR(4) BHI_GROUP_BAR(5) BHI_GROUP_BAR(6) BHI_GROUP_BAR(7)
    }
#undef BHI_GROUP_BAR
}

// ---- Huffman, symbol by symbol (rare windows) --------------------------------------------------------
// Decodes the next four symbols of one stream with first-symbol lookups (and the exact cascade for
// codes longer than the table index).  `p` is the true bit cursor.  Returns the two entry words
// {block A, block B} with the exponents at bits 7..14 and 23..30.  Inlined: as a call it cost a
// quarter more on tables where a few percent of the windows need it.
__device__ __forceinline__ uint2 quad_huff_slow(uint32_t p, uint32_t off, uint32_t plim, uint32_t copy_shift, uint32_t lut_bytes,
                                             uint32_t *p_out) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const HuffTables &t = *reinterpret_cast<const HuffTables *>(smem + lut_bytes);
    uint32_t sym[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t a = ((p >> 5) << 8) + off;
        const uint32_t win = __funnelshift_r(lds32(smem, a), lds32(smem, a + 256), p);
        const uint32_t e = lds32(smem, (win & (kPairEntries - 1)) << copy_shift);
        uint32_t s = (e >> 7) & 0xFFu, l = (e >> 16) & 15u;
        if (e & kEntExact) {
            s = huff_cascade(t, win);
            l = t.len[s];
        }
        sym[i] = s;
        p = min(p + l, plim);
    }
    *p_out = p;
    return make_uint2((sym[0] << 7) | (sym[1] << 23), (sym[2] << 7) | (sym[3] << 23));
}

// Per-lane decoder state over the group's ring.  Interface shared by both coders:
//   open(base, sigma4, rows)  - record of this lane's row at byte `base`, `rows` word rows long
//   two<kChecked>(eA0, eA1, eB0, eB1) - entry words of the next two blocks (streams sigma, sigma+32)
//   clamp()
struct QuadCtx {
    const uint8_t *smem;
    Consts k;
    uint32_t copy_off, index_mask, bias, copy_shift, lut_bytes;
};

struct QuadHuff {
    uint32_t p0, p1, plim, off;          // cursors run `bias` bits behind the stream position
    __device__ __forceinline__ void open(const QuadCtx &c, uint32_t base, uint32_t sigma4, uint32_t rows) {
        off = (base & 255u) + sigma4;
        p0 = p1 = (base >> 8) * 32u - c.bias;
        plim = p0 + 32u * (rows + 1u);
    }
    static __device__ __forceinline__ uint32_t window(const QuadCtx &c, uint32_t p, uint32_t o) {
        const uint32_t a = umad(p & ~31u, c.k.eight, o);
        return __funnelshift_r(lds32(c.smem, a), lds32(c.smem, a + 256u), p);
    }
    static __device__ __forceinline__ uint32_t lookup(const QuadCtx &c, uint32_t win) {
        return lds32(c.smem, (win & c.index_mask) | c.copy_off);
    }
    template <bool kChecked>
    __device__ __forceinline__ void two(const QuadCtx &c, uint32_t &eA0, uint32_t &eA1, uint32_t &eB0, uint32_t &eB1) {
        const uint32_t q0 = p0, q1 = p1;
        const uint32_t w0 = window(c, p0, off);
        const uint32_t w1 = window(c, p1, off + 128u);
        eA0 = lookup(c, w0);
        eA1 = lookup(c, w1);
        eB0 = lookup(c, __funnelshift_r(w0, 0u, eA0));       // shift count = low five bits = bits used by A
        eB1 = lookup(c, __funnelshift_r(w1, 0u, eA1));
        p0 += (eA0 + eB0) & 31u;
        p1 += (eA1 + eB1) & 31u;
        if (kChecked) {
            if ((eA0 | eB0 | eA1 | eB1) & kEntFlags) {
                if ((eA0 | eB0) & kEntFlags) {
                    uint32_t p;
                    const uint2 f = quad_huff_slow(q0 + c.bias, off, plim + c.bias, c.copy_shift, c.lut_bytes, &p);
                    eA0 = f.x;
                    eB0 = f.y;
                    p0 = p - c.bias;
                }
                if ((eA1 | eB1) & kEntFlags) {
                    uint32_t p;
                    const uint2 f = quad_huff_slow(q1 + c.bias, off + 128u, plim + c.bias, c.copy_shift, c.lut_bytes, &p);
                    eA1 = f.x;
                    eB1 = f.y;
                    p1 = p - c.bias;
                }
            }
        }
    }
    __device__ __forceinline__ void clamp() {
        p0 = min(p0, plim);
        p1 = min(p1, plim);
    }
};

struct QuadAnsLane {
    uint32_t lo, hi, nx;
    __device__ __forceinline__ uint32_t symbol(const QuadCtx &c, uint32_t alim) {
        if (hi == 0 && lo <= c.k.ans_mask) {
            hi = lo;
            lo = lds32(c.smem, nx);
            nx = min(nx + 256u, alim);
        }
        const uint32_t e = lds32(c.smem, ((lo << c.copy_shift) & c.index_mask) | c.copy_off);
        const uint32_t shifted = __funnelshift_r(lo, hi, c.k.ans_bits);
        const uint64_t next = static_cast<uint64_t>((e >> 12) & 0xFFFu) * shifted + (e & 0xFFFu);
        lo = static_cast<uint32_t>(next);
        hi = static_cast<uint32_t>(next >> 32);
        return e >> 24;
    }
};

struct QuadAns {
    QuadAnsLane a0, a1;
    uint32_t alim;
    __device__ __forceinline__ void open(const QuadCtx &c, uint32_t base, uint32_t sigma4, uint32_t rows) {
        const uint32_t p = base + sigma4;
        a0.lo = lds32(c.smem, p);
        a1.lo = lds32(c.smem, p + 128u);
        a0.hi = a1.hi = 0;
        a0.nx = p + 256u;
        a1.nx = p + 128u + 256u;
        alim = p + rows * 256u;
    }
    template <bool>
    __device__ __forceinline__ void two(const QuadCtx &c, uint32_t &eA0, uint32_t &eA1, uint32_t &eB0, uint32_t &eB1) {
        const uint32_t s00 = a0.symbol(c, alim), s10 = a1.symbol(c, alim + 128u);
        const uint32_t s01 = a0.symbol(c, alim), s11 = a1.symbol(c, alim + 128u);
        const uint32_t s02 = a0.symbol(c, alim), s12 = a1.symbol(c, alim + 128u);
        const uint32_t s03 = a0.symbol(c, alim), s13 = a1.symbol(c, alim + 128u);
        eA0 = (s00 << 7) | (s01 << 23);
        eA1 = (s10 << 7) | (s11 << 23);
        eB0 = (s02 << 7) | (s03 << 23);
        eB1 = (s12 << 7) | (s13 << 23);
    }
    __device__ __forceinline__ void clamp() {}
};

template <class Codec> struct QuadOf;
template <> struct QuadOf<HuffCodec> { using type = QuadHuff; };
template <> struct QuadOf<AnsCodec> { using type = QuadAns; };

struct QuadUnit {
    int qi, k;              // quad index inside the CTA, chunk
    int rec;                // this lane's row: record index (chunk * M + row)
    uint32_t off;           // this lane's row: first exponent word
    uint32_t bytes;         // this lane's row: staged bytes
    uint32_t rows;          // word rows of the longest of the four records
    uint32_t base;          // byte offset of the unit in shared memory
    bool valid, staged;
    __device__ __forceinline__ uint32_t stride() const { return rows * 256u + 32u; }      // bytes between the four records
    __device__ __forceinline__ uint32_t foot() const { return rows * 1024u + 128u; }      // bytes of the unit in the ring
};

}  // namespace bhi

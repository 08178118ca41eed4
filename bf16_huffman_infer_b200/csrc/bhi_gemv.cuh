// Fused decode + product for 1..32 rows of X, and decode to a dense matrix (sm_100a).
//
// What bounds it.  Not HBM: an SM runs out of issue slots (half of them on the half-rate integer pipe) and shared-memory
// wavefronts before the compressed bytes run out.  The layout spends both sparingly: table lookups without bank conflicts,
// one X fragment for eight weight rows, no staging work in registers.
//
// Work mapping.  A *unit* is up to eight consecutive weight rows (two quads) of one K-chunk; a group of four warps works on
// a unit.  Warp j of the group (its *pass*) decodes streams 8j..8j+7 and 32+8j..32+8j+7 of all eight rows: lane
// (r = lane/8, s = (lane/4)%2, t = lane%4) runs streams sigma = 8j + 4s + t and sigma + 32 of row r of either quad, four
// streams in all.  Per 128-column block a lane rebuilds two bf16x2 words per quad, exactly the B fragment of one
// mma.sync.m16n8k16 whose eight columns n = lane/4 are (row r, half s); the sixteen A rows are (half s, batch row b),
// b = 0..7, the same for both quads.  The products of mismatched halves (c1, c2) are discarded and c0 + c3 of lane (b, t)
// is the dot product of batch row b with weight row t of the quad.  The cost of a launch hardly depends on the batch up to
// eight rows; every eight more cost one more product per block and quad, none of the decoding.
//
// Memory.  The records of a unit are brought into the group's ring by bulk async copies on one mbarrier, one unit ahead,
// each record shifted by 32 bytes against the previous one, so that the 32 lanes of a warp (4 rows x 8 streams) read 32
// different banks.  Sign/mantissa rows pass through shared memory too, in chunks of four blocks copied asynchronously by
// the warp that reads them: as loads into registers they took a quarter of the register file and stalled every warp
// (151936 x 4096, four rows: 312 us, as copies 276 us).  X lies in shared memory row by row, padded by 16 bytes, where one
// ldmatrix yields a fragment; it comes by bulk copy, whole if it fits, else through a ring of four-block segments that all
// groups read in step.
//
// Results: the four warps of a group add their partial sums through shared memory in pass order (deterministic).
// Row-sharded layers stage their results and store them into every rank's output with coalesced peer stores at the end
// of the kernel (see ExchangeSink for the protocol).
#pragma once

#include "bhi_staged.cuh"

namespace bhi {

constexpr int kGemvWarps = 4;                 // warps of a group
constexpr int kRG = 4;                        // blocks per chunk of the sign/mantissa rows, and per segment of the X ring
constexpr uint32_t kRemChunk = 1024;          // bytes of a chunk: four blocks, eight rows, 32 bytes of a pass
constexpr uint32_t kXSegCols = 128 * kRG;
constexpr uint32_t kXPad = 16;                // bytes between rows of X: eight rows of a fragment lie on different banks
constexpr int kXSlotsMax = 4;                 // most segments of the X ring
constexpr int kGemvCtrlBytes = 512;           // mbarriers, unit descriptors
constexpr uint32_t kTableAt = 1024;           // where dynamic shared memory starts in the CTA's window (the system's share lies below)

struct GemvGeom {
    uint32_t exact_off, part_off, ys_off, rem_off, ring_off, x_off;
    uint32_t ring_bytes;       // per group
    uint32_t x_pitch;          // bytes between rows of X
    uint32_t x_slot;           // bytes of a segment of the X ring
    int x_slots;               // segments of the ring; 0 = all of X is resident
    int batch;
    int max_quads;             // of a unit: 2, or 1 when records are long
};

// Values the compiler must not see: multiply-adds by them stay on the FMA pipe.
struct GemvConsts {
    uint32_t ans_bits, ans_mask, freq_mask;
    uint32_t eight, entry;     // entry = bytes of one rANS table entry's copies
};

// Shared memory by its 32-bit address.  Written as instructions because address arithmetic on pointers cost an addition
// per load.  Tables do not change while they are read; what does (see keep_order, lds_now) keeps its place.
template <uint32_t kOffset>
__device__ __forceinline__ uint32_t lds_table(uint32_t a) {
    uint32_t v;
    asm("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(kOffset));
    return v;
}
template <uint32_t kOffset>
__device__ __forceinline__ uint32_t lds_now(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(kOffset));
    return v;
}
template <uint32_t kOffset>
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&v)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4+%5];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a), "n"(kOffset) : "memory");
}
// 16 bytes, or (bytes = 0) zeros without reading the source
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void *src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// barrier among the warps of one group: hardware barrier group + 1 (0 is the CTA-wide one).  Literal barrier numbers, so
// that the kernel reserves as many as it uses.
__device__ __forceinline__ void gemv_group_barrier(int group) {
    switch (group) {
        case 0: asm volatile("bar.sync 1, 128;" ::: "memory"); break;
        case 1: asm volatile("bar.sync 2, 128;" ::: "memory"); break;
        case 2: asm volatile("bar.sync 3, 128;" ::: "memory"); break;
        default: asm volatile("bar.sync 4, 128;" ::: "memory"); break;
    }
}

struct GemvCtx {
    const HuffTables *exact;
    GemvConsts k;
    uint32_t lane_table;       // this lane's byte offset inside a table entry
};

// Decoders of one quad's two streams of a lane.  Interface:
//   source(prepared)      the table as a region of the prepared blob, or null: fill() builds it (whole CTA)
//   usable(exact tables)  whether the table serves this layer; else its records are decoded from global memory
//   open(base, rows)      record at byte `base` (+ the stream's offset inside a word row), `rows` word rows long
//   step(ctx, dec, e)     exponent words of the next two blocks of n quads: e[quad][block][stream half]
//   clamp()               once per four blocks: a corrupt stream cannot leave the CTA's shared memory

// The 32-bit window under a cursor: word rows are 256 bytes apart.
__device__ __forceinline__ uint32_t ring_window(const GemvCtx &c, uint32_t p, uint32_t off) {
    const uint32_t a = umad(p & ~31u, c.k.eight, off);
    return __funnelshift_r(lds_table<0>(a), lds_table<256>(a), p);
}
// Ring words change between records.  Their loads are free to move among each other, but what they depend on passes
// through here, after the wait for the record's copies, so they cannot move before it.
__device__ __forceinline__ void keep_order(uint32_t &a, uint32_t &b) { asm volatile("" : "+r"(a), "+r"(b)::"memory"); }

// Huffman codes of at most 6 bits, symbol by symbol, in tables that hold one copy per lane: entry v of lane l lies at
// 128 v + 4 l, so the 32 lanes always hit 32 different banks.  The cursor runs seven bits behind the stream position, which
// puts the index into its place for that stride: a lookup is one logic instruction and one load.  An entry's low five bits
// are the code's length; the hardware shift takes exactly those five bits as its count, so one window serves four symbols.
// First and second symbol of a block have tables of their own, s << 7 | n and s << 23 | n: the SUM of two entries is the
// block's exponent word, with the bits the two used below it.  Twice the lookups of a table of symbol pairs, but one
// wavefront each instead of about 3.5 (151936 x 4096, four rows: 276 us, with a 12-bit pair table 320).
struct GemvSingle {
    using Codec = HuffCodec;
    static constexpr uint32_t kSecond = 64 * 128;          // byte offset of the second symbol's table
    static constexpr uint32_t kTableBytes = kSingleBytes;
    static constexpr uint32_t kMask = 63u << 7;
    uint32_t p0, p1, plim, off;
    static __device__ __forceinline__ const uint8_t *source(const uint8_t *prepared) { return prepared + kPreparedSingle; }
    static __device__ __forceinline__ void fill(uint8_t *, const HuffTables &, const HuffArgs &, const GemvConsts &, int, int) {}
    static __device__ __forceinline__ bool usable(const HuffTables &t) { return *reinterpret_cast<const uint32_t *>(&t + 1) == 0u; }
    __device__ __forceinline__ void open(uint32_t base, uint32_t rows) {
        off = base & 255u;
        p0 = p1 = (base >> 8) * 32u - 7u;
        plim = p0 + 32u * (rows + 1u);
        keep_order(p0, p1);
    }
    static __device__ __forceinline__ void blocks(const GemvCtx &c, uint32_t &p, uint32_t o, uint32_t &eA, uint32_t &eB) {
        auto at = [&](uint32_t w) { return (w & kMask) | c.lane_table; };
        uint32_t w = ring_window(c, p, o);
        const uint32_t e0 = lds_table<kTableAt>(at(w));
        w = __funnelshift_r(w, 0u, e0);
        const uint32_t e1 = lds_table<kTableAt + kSecond>(at(w));
        w = __funnelshift_r(w, 0u, e1);
        const uint32_t e2 = lds_table<kTableAt>(at(w));
        w = __funnelshift_r(w, 0u, e2);
        const uint32_t e3 = lds_table<kTableAt + kSecond>(at(w));
        eA = e0 + e1;
        eB = e2 + e3;
        p += (eA + eB) & 31u;                              // at most 24 bits
    }
    template <int n>
    static __device__ __forceinline__ void step(const GemvCtx &c, GemvSingle (&d)[n], uint32_t (&e)[n][2][2]) {
#pragma unroll
        for (int q = 0; q < n; q++) {
            blocks(c, d[q].p0, d[q].off, e[q][0][0], e[q][1][0]);
            blocks(c, d[q].p1, d[q].off + 128u, e[q][0][1], e[q][1][1]);
        }
    }
    __device__ __forceinline__ void clamp() {
        p0 = min(p0, plim);
        p1 = min(p1, plim);
    }
};

// Any Huffman code of the format, by pairs of symbols: a window's low kBits bits (the cursor runs two bits behind, which
// scales them by the entry's four bytes) yield two symbols, already in place, and the bits they used, so one window serves
// two blocks.  Windows that kBits do not resolve are flagged: 0.15 % of those of the escape-byte code at 14 bits, 0.22 % at
// 13, and up to 0.5 and 1 % of the reference's where its repair loop has lengthened the frequent codes.  14 bits are 7 %
// faster than 13 where the 64 KB of their table leave room for X beside it.
template <int kBits>
struct GemvPair {
    using Codec = HuffCodec;
    static constexpr uint32_t kTableBytes = 4u << kBits;
    static constexpr uint32_t kMask = ((1u << kBits) - 1u) << 2;
    static constexpr uint32_t kFlags = kEntSingle | kEntExact;
    uint32_t p0, p1, plim, off;
    static __device__ __forceinline__ const uint8_t *source(const uint8_t *prepared) {
        return prepared == nullptr ? nullptr : prepared + (kBits == kWideBits ? kPreparedWide : kBits == kWidestBits ? kPreparedWidest : 0);
    }
    static __device__ __forceinline__ void fill(uint8_t *table, const HuffTables &t, const HuffArgs &, const GemvConsts &, int tid, int threads) {
        for (int v = tid; v < (1 << kBits); v += threads) reinterpret_cast<uint32_t *>(table)[v] = pair_entry<kBits>(t, v);
    }
    static __device__ __forceinline__ bool usable(const HuffTables &) { return true; }
    __device__ __forceinline__ void open(uint32_t base, uint32_t rows) {
        off = base & 255u;
        p0 = p1 = (base >> 8) * 32u - 2u;
        plim = p0 + 32u * (rows + 1u);
        keep_order(p0, p1);
    }
    static __device__ __forceinline__ uint32_t lookup(uint32_t w) { return lds_table<kTableAt>(w & kMask); }
    // A flagged entry `e` at cursor p: the second symbol takes a lookup of its own, a code longer than the index the exact
    // tables.  Advances p; the entry returned has the two symbols and no bits.
    static __device__ __forceinline__ uint32_t resolve(const GemvCtx &c, uint32_t e, uint32_t &p, uint32_t o, uint32_t limit) {
        uint32_t bits = e & 15u;
        if (e & kEntExact) {
            const uint2 f = huff_exact_symbol(ring_window(c, p + 2u, o), c.exact);
            e = f.x << 7;
            bits = f.y;
        }
        p = min(p + bits, limit);
        const uint32_t f = lookup(ring_window(c, p, o));
        uint32_t s = f >> 7;
        bits = (f >> 16) & 15u;
        if (f & kEntExact) {
            const uint2 x = huff_exact_symbol(ring_window(c, p + 2u, o), c.exact);
            s = x.x;
            bits = x.y;
        }
        p = min(p + bits, limit);
        return (e & 0x7F80u) | (s << 23);
    }
    // The flagged entries of one block, stream by stream, in one piece of code for all streams of a lane: copies of it for
    // each would not fit the instruction cache.  blk = 0: w gets the window of the next block.
    template <int blk, int n>
    static __device__ __forceinline__ void resolve_block(const GemvCtx &c, GemvPair (&d)[n], uint32_t (&e)[n][2][2], uint32_t (&w)[n][2]) {
        uint32_t flags = 0u;
#pragma unroll
        for (int q = 0; q < n; q++) flags |= e[q][blk][0] | e[q][blk][1];
        if (flags & kFlags) {
            uint32_t todo = 0u;
#pragma unroll
            for (int z = 0; z < 2 * n; z++) todo |= (e[z >> 1][blk][z & 1] & kFlags) ? 1u << z : 0u;
#pragma unroll 1
            do {
                const int z = __ffs(todo) - 1;
                todo &= todo - 1u;
                uint32_t p = 0u, o = 0u, limit = 0u, entry = 0u;
#pragma unroll
                for (int y = 0; y < 2 * n; y++)
                    if (y == z) {
                        p = ((y & 1) ? d[y >> 1].p1 : d[y >> 1].p0) + (blk == 1 ? e[y >> 1][0][y & 1] & 31u : 0u);
                        o = d[y >> 1].off + ((y & 1) ? 128u : 0u);
                        limit = d[y >> 1].plim;
                        entry = e[y >> 1][blk][y & 1];
                    }
                entry = resolve(c, entry, p, o, limit);
                const uint32_t next = blk == 0 ? ring_window(c, p, o) : 0u;
#pragma unroll
                for (int y = 0; y < 2 * n; y++)
                    if (y == z) {
                        e[y >> 1][blk][y & 1] = entry;
                        if (blk == 0) w[y >> 1][y & 1] = next;
                        else e[y >> 1][0][y & 1] &= ~31u;
                        if (y & 1) d[y >> 1].p1 = p;
                        else d[y >> 1].p0 = p;
                    }
            } while (todo);
        }
    }
    template <int n>
    static __device__ __forceinline__ void step(const GemvCtx &c, GemvPair (&d)[n], uint32_t (&e)[n][2][2]) {
        uint32_t w[n][2];
#pragma unroll
        for (int q = 0; q < n; q++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                w[q][h] = ring_window(c, h ? d[q].p1 : d[q].p0, d[q].off + 128u * h);
                e[q][0][h] = lookup(w[q][h]);
            }
        resolve_block<0>(c, d, e, w);
#pragma unroll
        for (int q = 0; q < n; q++)
#pragma unroll
            for (int h = 0; h < 2; h++) e[q][1][h] = lookup(__funnelshift_r(w[q][h], 0u, e[q][0][h]));
        resolve_block<1>(c, d, e, w);
#pragma unroll
        for (int q = 0; q < n; q++) {
            d[q].p0 += (e[q][0][0] + e[q][1][0]) & 31u;
            d[q].p1 += (e[q][0][1] + e[q][1][1]) & 31u;
        }
    }
    __device__ __forceinline__ void clamp() {
        p0 = min(p0, plim);
        p1 = min(p1, plim);
    }
};

// rANS.  A table entry is the 64-bit addend of the state update, {word 0: slot - cum, word 1: symbol << 24 |
// freq << bits}: freq * (state >> bits) + entry is the next state, with the symbol (and the frequency, which nobody reads
// there) above the state's own 32 + bits bits, where the next step's funnel shift never looks.
// As many copies of the table as fill its place; a 64-bit load is served in two halves of 16 lanes, so 16 copies are free
// of conflicts.
//   k8 = true   8 bits: 32 copies, so that the entry stride is 256 bytes and the address one byte permutation of the state
//               and the lane's offset
//   k8 = false  any precision, half the space
template <bool k8>
struct GemvAns {
    using Codec = AnsCodec;
    static constexpr uint32_t kTableBytes = k8 ? 64 * 1024 : 32 * 1024;
    struct Stream {
        uint32_t lo, hi, nx;
    };
    Stream a0, a1;
    uint32_t alim;
    static __device__ __forceinline__ const uint8_t *source(const uint8_t *) { return nullptr; }
    static __device__ __forceinline__ void fill(uint8_t *table, const AnsTables &, const AnsArgs &a, const GemvConsts &k, int tid, int threads) {
        auto entry = [&](uint32_t v) {
            const uint32_t w = __ldg(a.lut + v);
            return make_uint2(w & 0xFFFu, (w & 0xFF000000u) | (((w >> 12) & 0xFFFu) << k.ans_bits));
        };
        if (k8) {
            // half an entry (16 copies) per thread, each lane starting at another 16 bytes of it: no bank conflicts
            for (uint32_t i = tid; i < 512u; i += threads) {
                const uint2 e = entry(i >> 1);
#pragma unroll
                for (uint32_t j = 0; j < 8u; j++)
                    reinterpret_cast<uint4 *>(table)[8u * i + ((j + tid) & 7u)] = make_uint4(e.x, e.y, e.x, e.y);
            }
        } else {
            for (uint32_t i = tid; i < kTableBytes / 8; i += threads) reinterpret_cast<uint2 *>(table)[i] = entry(i >> (12u - k.ans_bits));
        }
    }
    static __device__ __forceinline__ bool usable(const AnsTables &) { return true; }
    __device__ __forceinline__ void open(uint32_t base, uint32_t rows) {
        a0.nx = base + 256u;
        a1.nx = base + 384u;
        alim = base + rows * 256u;
        keep_order(a0.nx, a1.nx);
        a0.lo = lds_now<0>(base);
        a1.lo = lds_now<128>(base);
        a0.hi = a1.hi = 0u;
    }
    // Decodes one symbol; returns a word with the symbol in its top byte.  A state below 2^bits, the condition for a refill,
    // is one whose shifted value is zero; the refill goes straight into that value and the low word.  (As inline assembly
    // with predicates the same steps spilled 400 bytes.)
    static __device__ __forceinline__ uint32_t symbol(const GemvCtx &c, Stream &a) {
        const uint32_t bits = k8 ? 8u : c.k.ans_bits;
        uint32_t upper = __funnelshift_r(a.lo, a.hi, bits);
        if (upper == 0u) {
            const uint32_t w = lds_table<0>(a.nx);
            a.nx += 256u;
            upper = __funnelshift_r(w, a.lo, bits);
            a.lo = w;
        }
        const uint32_t at = k8 ? prmt(a.lo, c.lane_table, 0x5504u) : umad(a.lo & c.k.ans_mask, c.k.entry, c.lane_table);
        uint32_t e0, e1;
        asm("ld.shared.v2.u32 {%0, %1}, [%2+%3];" : "=r"(e0), "=r"(e1) : "r"(at), "n"(kTableAt));
        const uint32_t freq = k8 ? prmt(e1, 0u, 0x4421u) : (e1 >> c.k.ans_bits) & c.k.freq_mask;
        const uint64_t next = static_cast<uint64_t>(freq) * upper + ((static_cast<uint64_t>(e1) << 32) | e0);
        a.lo = static_cast<uint32_t>(next);
        a.hi = static_cast<uint32_t>(next >> 32);
        return a.hi;
    }
    template <int n>
    static __device__ __forceinline__ void step(const GemvCtx &c, GemvAns (&d)[n], uint32_t (&e)[n][2][2]) {
#pragma unroll
        for (int blk = 0; blk < 2; blk++) {
            uint32_t s[2][n][2];
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int q = 0; q < n; q++) {
                    s[i][q][0] = symbol(c, d[q].a0);
                    s[i][q][1] = symbol(c, d[q].a1);
                }
#pragma unroll
            for (int q = 0; q < n; q++)
#pragma unroll
                for (int h = 0; h < 2; h++)
                    e[q][blk][h] = prmt(s[0][q][h], s[1][q][h], 0x7632u) >> 1;     // from bits 8..15 and 24..31 to the exponents' places
        }
    }
    __device__ __forceinline__ void clamp() {
        a0.nx = min(a0.nx, alim);
        a1.nx = min(a1.nx, alim + 128u);
    }
};

// Records that are not staged (too long for the ring, not in storage order, not whole rows): the same interface over
// guarded loads from global memory, with the exact tables.  Few registers rather than speed.
struct GlobalRecord {
    const uint32_t *exp;
    uint32_t limit, at;        // words of the buffer; first word of the lane's first stream
    __device__ __forceinline__ uint32_t word(uint32_t row, uint32_t half) const {
        const uint64_t i = static_cast<uint64_t>(at) + 32u * half + static_cast<uint64_t>(kStreamsPerRecord) * row;
        return i < limit ? __ldg(exp + i) : 0u;
    }
};

struct DirectHuff {
    GlobalRecord src;
    const HuffTables *tab;
    uint32_t p[2];
    __device__ __forceinline__ void open(const GlobalRecord &g, const HuffTables *t) {
        src = g;
        tab = t;
        p[0] = p[1] = 0u;
    }
    __device__ __forceinline__ uint32_t symbol(int half) {
        const uint32_t at = p[half], row = at >> 5;
        const uint32_t s = huff_cascade(*tab, __funnelshift_r(src.word(row, half), src.word(row + 1u, half), at));
        p[half] = at + tab->len[s];
        return s;
    }
};

struct DirectAns {
    GlobalRecord src;
    const AnsTables *tab;
    uint32_t lo[2], hi[2], row[2];
    __device__ __forceinline__ void open(const GlobalRecord &g, const AnsTables *t) {
        src = g;
        tab = t;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            lo[h] = src.word(0u, h);
            hi[h] = 0u;
            row[h] = 1u;
        }
    }
    __device__ __forceinline__ uint32_t symbol(int half) {
        uint64_t state = static_cast<uint64_t>(hi[half]) << 32 | lo[half];
        if (state < (1ull << tab->bits)) state = (state << 32) | src.word(row[half]++, half);
        const uint32_t e = __ldg(tab->lut + (static_cast<uint32_t>(state) & ((1u << tab->bits) - 1u)));
        state = static_cast<uint64_t>((e >> 12) & 0xFFFu) * (state >> tab->bits) + (e & 0xFFFu);
        lo[half] = static_cast<uint32_t>(state);
        hi[half] = static_cast<uint32_t>(state >> 32);
        return e >> 24;
    }
};

template <class C>
struct GemvDirect : std::conditional<std::is_same<C, HuffCodec>::value, DirectHuff, DirectAns>::type {
    template <int n>
    static __device__ __forceinline__ void step(const GemvCtx &, GemvDirect (&d)[n], uint32_t (&e)[n][2][2]) {
#pragma unroll
        for (int q = 0; q < n; q++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t s0 = 0u, s1 = 0u, s2 = 0u, s3 = 0u;
#pragma unroll 1
                for (int i = 0; i < 4; i++) {
                    s0 = s1;
                    s1 = s2;
                    s2 = s3;
                    s3 = d[q].symbol(h);
                }
                e[q][0][h] = (s0 << 7) | (s1 << 23);
                e[q][1][h] = (s2 << 7) | (s3 << 23);
            }
    }
    __device__ __forceinline__ void clamp() {}
};

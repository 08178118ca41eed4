// Fused decode + product for 1..32 rows of X, and decode to a dense matrix (sm_100a).
//
// What bounds it.  Not HBM: an SM runs out of integer work (the half-rate pipe takes half of the issue slots) and of shared-memory
// wavefronts before the compressed bytes run out; with all sixteen warps in the loop both are four fifths full and more, so that
// work taken out of either counts and waits taken out do not.  The layout spends both sparingly: table lookups without bank
// conflicts, one X fragment for eight weight rows, no staging work in registers.
//
// Work mapping.  A *unit* is up to eight consecutive weight rows (two quads) of one K-chunk; a group of four warps works on
// a unit.  Warp j of the group (its *pass*) decodes streams 8j..8j+7 and 32+8j..32+8j+7 of all eight rows: lane
// (r = lane/8, s = (lane/4)%2, t = lane%4) runs streams sigma = 8j + 4s + t and sigma + 32 of row r of either quad, four
// streams in all.  Per 128-column block a lane rebuilds two bf16x2 words per quad.  Up to four rows of X (kFew) they are the A
// fragment of one mma.sync.m16n8k16 for both quads: sixteen rows (row r and half s of either quad), X the eight columns (half s,
// X row b).  More rows: a quad's two words are the B fragment of a product of its own, eight columns n = lane/4 that are (row r,
// half s); the sixteen A rows are (half s, X row b), b = 0..7, the same for both quads.  Either way the products of unequal
// halves are discarded, and the sum over s of the others is the dot product of X row b with row r of the quad.  Every eight
// rows of X more cost one more product per block and quad, none of the decoding.
//
// Memory.  The records of a unit are brought into the group's ring by bulk async copies on one mbarrier, one unit ahead,
// each record shifted by 32 bytes against the previous one, so that the 32 lanes of a warp (4 rows x 8 streams) read 32
// different banks.  Sign/mantissa rows pass through shared memory too, in chunks of four blocks copied asynchronously by
// the warp that reads them: as loads into registers they took a quarter of the register file and stalled every warp
// (151936 x 4096, four rows: 312 us, as copies 276 us).  X lies in shared memory row by row, padded by 16 bytes (few rows: 32),
// where one ldmatrix yields a fragment; it comes by bulk copy, whole if it fits, else through a ring of four-block segments that all
// groups read in step.
//
// Results: the four warps of a group add their partial sums through shared memory in pass order (deterministic).
// Row-sharded layers stage their results and store them into every rank's output with coalesced peer stores at the end
// of the kernel (see PeerSet for the protocol); where a CTA has too many rows for that, above a million rows per launch, the
// lanes that hold the results store them.
#pragma once

#include "bhi_launch.cuh"
#include "bhi_staged.cuh"

namespace bhi {

constexpr int kGemvWarps = 4;                 // warps of a group
constexpr int kRG = 4;                        // blocks per chunk of the sign/mantissa rows, and per segment of the X ring
constexpr uint32_t kRemChunk = 1024;          // bytes of a chunk: four blocks, eight rows, 32 bytes of a pass
constexpr uint32_t kXSegCols = 128 * kRG;
constexpr int kFewRows = 4;                    // most rows of X that can be the eight B columns of a product, twice
constexpr uint32_t kXPad = 16;                // bytes between rows of X (twice that for few rows): what one wavefront reads lies on different banks
constexpr int kXSlotsMax = 4;                 // most segments of the X ring
constexpr int kGemvCtrlBytes = 512;           // mbarriers, unit descriptors
constexpr uint32_t kTableAt = 1024;           // where dynamic shared memory starts in the CTA's window (the system's share lies below)

struct GemvGeom {
    uint32_t exact_off, part_off, ys_off, rem_off, ring_off, x_off;
    uint32_t ring_bytes;       // per group
    uint32_t ring_early;       // ... of which two units fill so much that the second's copies start before the first is read
    uint32_t pair_rows;        // longest record, in word rows, of a unit of two quads that the ring takes
    uint32_t x_pitch;          // bytes between rows of X
    uint32_t x_slot;           // bytes of a segment of the X ring
    int x_slots;               // segments of the ring; 0 = all of X is resident
    int batch;
    int max_quads;             // of a unit: 2, or 1 when all records are long
    int split;                 // the groups of a CTA share its quads and divide the chunks among them
    uint32_t acc_off;          // ... whose sums meet here
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
template <uint32_t kOffset>
__device__ __forceinline__ void ldmatrix_x2(uint32_t (&v)[2], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2+%3];" : "=r"(v[0]), "=r"(v[1]) : "r"(a), "n"(kOffset) : "memory");
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
// A cursor that is moved by whole table entries: the address of the word row it stands in, and the bit.  Only the low seven bits
// of `bit` count, the symbols of the entries may stand above them.  No step is longer than a row, so the row changes when bit 5
// does.  Two integer instructions per four symbols less than a cursor in bits alone (49152 x 4096: 93.6 us with that, 92.7 so);
// pair tables, whose flagged entries move a cursor in parts, gained nothing (6144 x 2048, reference tables: 16.9 and 17.1 us).
struct Cursor {
    uint32_t at, bit;
    __device__ __forceinline__ uint32_t window() const { return __funnelshift_r(lds_table<0>(at), lds_table<256>(at), bit); }
    __device__ __forceinline__ void step(const GemvCtx &c, uint32_t next) {
        at = umad((next ^ bit) & 32u, c.k.eight, at);
        bit = next;
    }
};
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
    static constexpr bool kRans = false;
    static constexpr uint32_t kSecond = 64 * 128;          // byte offset of the second symbol's table
    static constexpr uint32_t kTableBytes = kSingleBytes;
    static constexpr uint32_t kMask = 63u << 7;
    Cursor s0, s1;
    uint32_t limit;
    static __device__ __forceinline__ const uint8_t *source(const uint8_t *prepared) { return prepared + kPreparedSingle; }
    static __device__ __forceinline__ void fill(uint8_t *, const HuffTables &, const HuffArgs &, const GemvConsts &, int, int) {}
    static __device__ __forceinline__ bool usable(const HuffTables &t) { return prepared_longest(reinterpret_cast<const uint8_t *>(&t)) <= 6u; }
    __device__ __forceinline__ void open(uint32_t base, uint32_t rows) {
        s0 = {base - 256u, 32u - 7u};
        s1 = {base - 128u, 32u - 7u};
        limit = base + 256u * rows;
        keep_order(s0.at, s1.at);
    }
    static __device__ __forceinline__ void blocks(const GemvCtx &c, Cursor &s, uint32_t &eA, uint32_t &eB) {
        auto at = [&](uint32_t w) { return (w & kMask) | c.lane_table; };
        uint32_t w = s.window();
        const uint32_t e0 = lds_table<kTableAt>(at(w));
        w = __funnelshift_r(w, 0u, e0);
        const uint32_t e1 = lds_table<kTableAt + kSecond>(at(w));
        w = __funnelshift_r(w, 0u, e1);
        const uint32_t e2 = lds_table<kTableAt>(at(w));
        w = __funnelshift_r(w, 0u, e2);
        const uint32_t e3 = lds_table<kTableAt + kSecond>(at(w));
        eA = e0 + e1;
        eB = e2 + e3;
        s.step(c, s.bit + eA + eB);                        // at most 24 bits
    }
    template <int n>
    static __device__ __forceinline__ void step(const GemvCtx &c, GemvSingle (&d)[n], uint32_t (&e)[n][2][2]) {
#pragma unroll
        for (int q = 0; q < n; q++) {
            blocks(c, d[q].s0, e[q][0][0], e[q][1][0]);
            blocks(c, d[q].s1, e[q][0][1], e[q][1][1]);
        }
    }
    __device__ __forceinline__ void clamp() {
        s0.at = min(s0.at, limit);
        s1.at = min(s1.at, limit + 128u);
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
    static constexpr bool kRans = false;
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
    // With the window (`whole`: all of its 32 bits count), which still holds the second code where the first was resolved.
    template <bool whole>
    static __device__ __forceinline__ uint32_t resolve(const GemvCtx &c, uint32_t e, uint32_t window, uint32_t &p, uint32_t o, uint32_t limit) {
        uint32_t bits = e & 15u;
        if (e & kEntExact) {
            const uint2 f = huff_exact_symbol(ring_window(c, p + 2u, o), c.exact);
            e = f.x << 7;
            bits = f.y;
            p = min(p + bits, limit);
            window = ring_window(c, p, o);
        } else {
            p = min(p + bits, limit);
            window = whole ? __funnelshift_r(window, 0u, bits) : ring_window(c, p, o);
        }
        const uint32_t f = lookup(window);
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
    // each would not fit the instruction cache.  blk = 0: w gets the window of the next block.  Every instruction here counts: a
    // quarter to a half of the blocks have a flagged entry in some lane (flags gathered by bytes, the first block's second code
    // taken from the window that is here: 12288 x 4096 escape 33.4 us, so 32.9; reference tables 32.3, 31.9).
    template <int blk, int n>
    static __device__ __forceinline__ void resolve_block(const GemvCtx &c, GemvPair (&d)[n], uint32_t (&e)[n][2][2], uint32_t (&w)[n][2]) {
        uint32_t flags = 0u;
#pragma unroll
        for (int q = 0; q < n; q++) flags |= e[q][blk][0] | e[q][blk][1];
        if (flags & kFlags) {
            // one byte per stream, with one flag at most
            uint32_t todo = prmt(e[0][blk][0], e[0][blk][1], 0x0040u) & (kFlags | kFlags << 8);
            if (n > 1) todo |= prmt(e[n - 1][blk][0], e[n - 1][blk][1], 0x4000u) & (kFlags << 16 | kFlags << 24);
#pragma unroll 1
            do {
                const int z = (__ffs(todo) - 1) >> 3;
                todo &= todo - 1u;
                uint32_t p = 0u, o = 0u, limit = 0u, entry = 0u, window = 0u;
#pragma unroll
                for (int y = 0; y < 2 * n; y++)
                    if (y == z) {
                        p = ((y & 1) ? d[y >> 1].p1 : d[y >> 1].p0) + (blk == 1 ? e[y >> 1][0][y & 1] & 31u : 0u);
                        o = d[y >> 1].off + ((y & 1) ? 128u : 0u);
                        limit = d[y >> 1].plim;
                        entry = e[y >> 1][blk][y & 1];
                        if (blk == 0) window = w[y >> 1][y & 1];
                    }
                entry = resolve<blk == 0>(c, entry, window, p, o, limit);
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
//   k8 = true   8 bits in 64 KB: 32 copies, so that the entry stride is 256 bytes and the address one byte permutation of
//               the state and the lane's offset
//   k8 = false  any precision, in 64 KB or, where X needs the room, 32
template <bool k8, uint32_t kBytes>
struct GemvAns {
    using Codec = AnsCodec;
    static constexpr bool kRans = true;
    static constexpr uint32_t kTableBytes = kBytes;
    static_assert(!k8 || kBytes == 64 * 1024, "the address permutation needs a stride of 256 bytes");
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
        // 128 bytes of copies per thread and turn, written 16 bytes at a time, each lane starting at another 16 of them: no
        // bank conflicts.  An entry that has fewer copies than that shares the 128 bytes with its neighbours.
        const uint32_t copies_log2 = (kBytes == 64 * 1024 ? 13u : 12u) - k.ans_bits;
#pragma unroll
        for (uint32_t i = tid; i < kBytes / 128u; i += threads) {
            if (copies_log2 >= 4u) {
                const uint2 e = entry(i >> (copies_log2 - 4u));
#pragma unroll
                for (uint32_t j = 0; j < 8u; j++)
                    reinterpret_cast<uint4 *>(table)[8u * i + ((j + tid) & 7u)] = make_uint4(e.x, e.y, e.x, e.y);
            } else {
                uint2 lo[8], hi[8];
#pragma unroll
                for (uint32_t j = 0; j < 8u; j++) {
                    const uint32_t at = 16u * i + 2u * ((j + tid) & 7u);
                    lo[j] = entry(at >> copies_log2);
                    hi[j] = entry((at + 1u) >> copies_log2);
                }
#pragma unroll
                for (uint32_t j = 0; j < 8u; j++)
                    reinterpret_cast<uint4 *>(table)[8u * i + ((j + tid) & 7u)] = make_uint4(lo[j].x, lo[j].y, hi[j].x, hi[j].y);
            }
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

// A part of an X row into shared memory: by the calling thread as a bulk copy on `bar`, or (unaligned source) by the whole
// warp with plain stores.
__device__ __forceinline__ void copy_x_row(uint32_t dst, const uint16_t *src, uint32_t bytes, uint32_t bar, bool bulk, int lane) {
    if (bulk) {
        bulk_copy_g2s(dst, src, bytes, bar);
    } else {
        for (uint32_t i = 4u * lane; i < bytes; i += 256u) {           // (two at a time; a block of columns is 256 bytes)
            const uint32_t *p = reinterpret_cast<const uint32_t *>(src) + (i >> 2);
            const uint32_t v = load_written(p), w = load_written(p + 32);
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + i), "r"(v) : "memory");
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + i + 128u), "r"(w) : "memory");
        }
    }
}

// How many sets the quads [quad_lo, quad_hi) make (whole warp): pairs, but two of a pair that has, in any chunk, a record of
// more than `most` words.
__device__ __forceinline__ int count_sets(const int32_t *offsets, int S, int M, uint32_t exp_words, int quad_lo, int quad_hi, uint32_t most) {
    int sets = (quad_hi - quad_lo + 1) >> 1;
    for (int q0 = quad_lo; q0 + 1 < quad_hi; q0 += 64) {
        const int q = q0 + 2 * static_cast<int>(threadIdx.x & 31);
        bool longer = false;
        for (int k = 0; k < S && q + 1 < quad_hi; k++) {
            const int rec = k * M + 4 * q, last = k * M + M;
            uint32_t at[9];
#pragma unroll
            for (int i = 0; i < 9; i++) {
                const int m = min(rec + i, last);
                at[i] = m < S * M ? static_cast<uint32_t>(__ldg(offsets + m)) : exp_words;
            }
#pragma unroll
            for (int i = 0; i < 8; i++) longer |= at[i + 1] > at[i] && at[i + 1] - at[i] > most;
        }
        sets += __popc(__ballot_sync(0xFFFFFFFFu, longer));
    }
    return sets;
}

// Sixteen warps and one more have 96 registers each (five warps share a quarter of the register file).  With the register shift the
// one more is a warpgroup, of which one warp works: it gives registers back, so that the sixteen can have 112 (640 x 96 at the launch
// = 512 x 112 + 128 x 32).  Without it / with it, in us:
//   pair tables, up to eight rows        4096 x 12288 39.9/39.1   12288 x 8192 73.2/71.6   8192 x 28672 167.9/164.0   (escape, 8 rows)
//   ... 16, 24, 32 rows                  12288 x 4096  47.2/45.0   49.3/46.2   61.5/55.5
//   ... 25 rows, some CTA with six       3000 x 14336  64.1/69.2   3584 x 18944  88.2/97.8   3630 x 7680  38.8/41.8: two groups have a pair of
//       quads of several long chunks     quads and two a single one, in step.  These do without, but with at most five quads or from seven on
//                                        2600 x 14336  61.9/59.7   4300 x 14336, 32 rows, 73.2/68.3, with one chunk 3584 x 4096  22.1/21.4,
//                                        with short ones or rows 3630 x 9856 (11 blocks)  89.4/81.4   4096 x 6144, 32 rows, 34.0/31.9
//   rANS, up to eight rows               512 x 16256  27.6/28.9   1024 x 8192  18.6/19.3   4096 x 12288  50.7/50.5: without.  Single quads
//                                        are decoded slower with the shift's registers, pairs of them faster
//   ... 9 to 16 rows                     2300 x 4096 (a quad for each group)  14.9/15.0   2600 x 8576 (units of one quad)  41.2/43.0: without;
//                                        2400 x 4096  18.5/16.9   12288 x 4096  58.2/54.9
//   ... 24, 32 rows                      12288 x 4096  64.6/61.6   73.5/67.2   (but 4096 x 12288, 32 rows, of such different scales, log-normal with
//                                        sigma 0.8, that records are decoded from global memory, 234/248)
//   limit6, 24 rows                      3584 x 4096  15.4/16.0   4096 x 12288  40.4/41.6   50000 x 2560  98.4/95.1: without
//   ... 32 rows                          12288 x 4096  50.9/48.5
template <class Dec, int NB, int NG, bool kRing>
constexpr bool kShiftsRegisters = kRing && NG == 4 && (std::is_same<Dec, GemvSingle>::value ? NB > 3 : !Dec::kRans || NB > 1);
// ... and whether there is a kernel without the shift beside it
template <class Dec, int NB>
constexpr bool kShiftsOrNot = Dec::kRans ? NB == 2 : NB == 4 && !std::is_same<Dec, GemvSingle>::value;
// The launch has to hold what both sides have in the end: setmaxnreg waits without limit for registers that are not there.  The
// compiler's count may be below the launch bounds', so each such kernel's is looked at before its first launch.
constexpr int kShiftAtLaunch = 96, kShiftUp = 112, kShiftDown = 32;
static_assert(kShiftAtLaunch * (512 + 128) >= kShiftUp * 512 + kShiftDown * 128, "more registers than the launch brings");
template <bool kRing, bool kShift>
constexpr int kRingThreads = !kRing ? 0 : kShift ? 128 : 32;

// NB = groups of eight X rows (0: no product, the dense matrix is written instead).  NG = groups of four warps per CTA.
// Two: two CTAs share an SM, so the next kernel's CTAs start as this one's leave.  Four: one CTA per SM, for launches whose
// X or tables two CTAs could not both hold.  kRing: X passes through a ring that one more warp fills and all groups read in
// step.  (20 warps of 96 registers instead of 16 gain nothing: it is pipes that are short, not warps.)
// kHalf: two groups, and no more CTAs than SMs, so that half of each SM is the next kernel's: it has its tables and records by
// the time this one ends.  For launches so small that latencies, not the pipes, set their time (see kHalfUnits).
// kFew: at most four rows of X.  The weights are then the sixteen A rows (row r and half s of either quad) and X the eight B
// columns (half s, X row b): one product instead of two serves both quads of a block, and a fragment of X takes two wavefronts
// of shared memory instead of four.  Of the products those of equal halves count, (r, s) x (s, b); their sum over s is the
// result.  (One row: 49152 x 4096 limit6 92.9 us, so 90.1, rANS 150.4, 146.2; 12288 x 4096 escape 34.6, 34.0.)
// kShard: a layer whose rows are shared among ranks (1: results staged, 2: stored one by one).  An argument of the template,
// because code that a launch does not run costs it time all the same: each part taken out of the kernel made launches of small
// layers 0.1 to 0.2 us shorter (2048 x 2048, limit6: 6.0 us with all three in one kernel, 5.8 so).
// kShift: see kShiftsRegisters.
// (The ring forms of two groups have an SM to themselves, but bounds for one CTA, and up to 168 registers, made them slower:
// 8192 x 16256 of 120 exponents, escape, 417.4 us, so 419.1; row-sharded, whose 96 registers spill 16 to 40 bytes, 427.5, 430.1.)
template <class Dec, int NB, int NG, bool kRing, int kShard, bool kHalf, bool kFew, bool kShift>
__global__ void __launch_bounds__(NG * kGemvWarps * 32 + kRingThreads<kRing, kShift>, NG == 2 ? 2 : 1)
gemv_kernel(Layer L, typename Dec::Codec::Args targs, const uint8_t *prepared, const uint16_t *X, const uint16_t *bias, uint16_t *Y,
            PeerSet peers, GemvGeom G, GemvConsts kc) {
    extern __shared__ __align__(1024) uint8_t smem[];
    using Codec = typename Dec::Codec;
    using Tables = typename Codec::Tables;
    constexpr bool kHuff = std::is_same<Codec, HuffCodec>::value;
    constexpr int kThreads = NG * kGemvWarps * 32;                     // without the warp that fills the X ring
    constexpr int kAcc = NB > 0 ? NB : 1;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = warp / kGemvWarps, wig = warp % kGemvWarps;      // warp inside the group = its pass
    const int r = lane >> 3, t = lane & 3, gq = lane >> 2;
    // Dense: no product ties rows together, so a warp takes whole rows (two of the eight, or one of four) and lane l the
    // streams l and l + 32: its stores are whole 128-byte lines.
    const uint32_t sigma4 = NB > 0 ? 4u * (8 * wig + (lane & 7)) : 4u * lane;      // byte offset of the lane's stream inside a word row
    auto row_of = [&](int q, int n, int row) { return NB > 0 ? 4 * q + row : n * wig + q; };       // row of a unit of n quads
    constexpr bool exchange = NB == 1 && kShard > 0;
    const int B = G.batch;

    Tables &tab = *reinterpret_cast<Tables *>(smem + G.exact_off);
    uint8_t *ctrl = smem + G.exact_off + kExactBytes;
    const uint32_t smem_base = smem_addr(smem);
    const uint32_t ctrl_at = smem_addr(ctrl);
    const uint32_t bar0 = ctrl_at + 16u * group;                       // record copies: two slots per group
    const uint32_t table_bar = ctrl_at + 80u, x_bar = ctrl_at + 88u;
    const uint32_t x_full = ctrl_at + 96u, x_empty = x_full + 8u * kXSlotsMax;      // X ring: filled, read by all warps
    volatile uint32_t *posted = reinterpret_cast<volatile uint32_t *>(ctrl + 256) + 8 * group;     // [slot]{word rows, base, staged, quads}
    float *part = reinterpret_cast<float *>(smem + G.part_off) + group * (kGemvWarps * 64 * kAcc);
    uint16_t *ys = reinterpret_cast<uint16_t *>(smem + G.ys_off);
    const uint32_t xs = smem_base + G.x_off;
    const uint32_t rem_at = smem_base + G.rem_off + warp * (kRemChunk * 2u);
    const uint32_t ring = G.ring_off + group * G.ring_bytes;

    GemvCtx ctx;
    ctx.exact = reinterpret_cast<const HuffTables *>(&tab);
    ctx.k = kc;
    // (through a shuffle, which cannot be computed anew: without it the compiler put that into every lookup of the limit6 form
    // for few rows, 4 instructions more per 128 weights)
    ctx.lane_table = __shfl_sync(0xFFFFFFFFu, kHuff ? 4u * lane : (8u * lane) & (kc.entry - 1u), lane);

    // Quads are dealt to the groups of the grid in equal contiguous ranges; a group takes them two at a time.
    const int nquads = (L.M + 3) >> 2;
    auto deal = [&](int g) { return static_cast<int>(static_cast<int64_t>(nquads) * g / (static_cast<int>(gridDim.x) * NG)); };
    const bool split = !kRing && NB <= 1 && G.split;
    const int cta_lo = deal(blockIdx.x * NG), cta_hi = deal(blockIdx.x * NG + NG);
    const int k_lo = split ? L.S * group / NG : 0, k_hi = split ? L.S * (group + 1) / NG : L.S;
    const int quad_lo = !split ? deal(blockIdx.x * NG + group) : k_lo < k_hi ? cta_lo : cta_hi;
    const int quad_hi = !split ? deal(blockIdx.x * NG + group + 1) : cta_hi;
    const int row_lo = 4 * cta_lo;                                     // rows of the CTA
    const int rows_cta = min(4 * cta_hi, L.M) - row_lo;
    float *acc = reinterpret_cast<float *>(smem + G.acc_off);          // [quad of the CTA][group][lane]
    const int nblk = L.Nc >> 7;
    const int chunks = (nblk + kRG - 1) / kRG;                         // of a record

    pdl_launch_dependents();
    if (tid == 0) {
        for (uint32_t i = 0; i < 2u * NG; i++) mbar_init(ctrl_at + 8u * i, 1);
        mbar_init(table_bar, 1);
        mbar_init(x_bar, kHalf ? NG * kGemvWarps : 1);
        for (uint32_t i = 0; kRing && i < kXSlotsMax; i++) {
            mbar_init(x_full + 8u * i, 1);
            mbar_init(x_empty + 8u * i, NG * kGemvWarps);
        }
        mbar_fence_init();
        if (kHuff && prepared != nullptr) {
            mbar_expect_tx(table_bar, Dec::kTableBytes + kExactBytes);
            bulk_copy_g2s(smem_base, Dec::source(prepared), Dec::kTableBytes, table_bar);
            bulk_copy_g2s(smem_base + G.exact_off, prepared + kPairEntries * 4, kExactBytes, table_bar);
        }
    }
    __syncthreads();

    // Segments of X that pass through the ring: every unit reads those of its chunk, in order.  The groups post how many sets
    // of quads they have.
    volatile uint32_t *all_sets = reinterpret_cast<volatile uint32_t *>(ctrl + 384);
    auto x_segments = [&]() {
        uint32_t sets = 0u;
        for (int g = 0; g < NG; g++) sets = max(sets, all_sets[g]);
        return static_cast<int>(sets) * L.S * chunks;
    };
    // ---- the warp that fills the X ring.  (With the readers filling it between their chunks, the last reader of a segment
    // its next one, the refill lay on the slowest warp and cost half as much again as the decoding.)
    if (kRing && warp >= NG * kGemvWarps) {
        if constexpr (kShift) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kShiftDown));
        __syncthreads();                                               // the readers' barrier before their loop
        if (warp > NG * kGemvWarps) {
            if (exchange) __syncthreads();                             // exchange_finish's
            return;
        }
        pdl_wait();
        const bool bulk = (reinterpret_cast<uintptr_t>(X) & 15u) == 0u;
        const int x_total = x_segments();
        int slot = 0, k = 0, ch = 0;
        uint32_t phase = 1u;                                           // nobody has to have read the first lap's places
        for (int i = 0; i < x_total; i++) {
            const uint32_t bar = x_full + 8u * slot;
            if (!mbar_wait_bounded(x_empty + 8u * slot, phase)) {
                if (lane == 0) atomicExch(&g_staged_status, 3);
                break;
            }
            const uint32_t bytes = 2u * min(kXSegCols, static_cast<uint32_t>(L.Nc) - ch * kXSegCols);
            const uint16_t *src = X + static_cast<int64_t>(k) * L.Nc + ch * kXSegCols;
            if (bulk) {
                if (lane == 0) mbar_expect_tx(bar, bytes * B);
                __syncwarp();
            }
            for (int b = bulk ? lane : 0; b < B; b += bulk ? 32 : 1)
                copy_x_row(xs + slot * G.x_slot + b * G.x_pitch, src + static_cast<int64_t>(b) * L.S * L.Nc, bytes, bar, bulk, lane);
            __syncwarp();
            if (!bulk && lane == 0) mbar_arrive(bar);
            if (++ch == chunks) {
                ch = 0;
                if (++k == L.S) k = 0;
            }
            if (++slot == G.x_slots) {
                slot = 0;
                phase ^= 1u;
            }
        }
        if (exchange) __syncthreads();                                 // exchange_finish's
        return;
    }

    if constexpr (kShift) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kShiftUp));
    // ---- units ---------------------------------------------------------------------------------------------------------
    // A set is a pair of quads, or one quad: the last of an odd number, and both of a pair that has, in any chunk, a record
    // longer than the ring takes beside seven of that length.  For each set, the chunks in order.  The group's first warp
    // knows where the records of the next unit lie (its lanes 0..7 hold one row each; of a set's first unit the others hold
    // the same rows in the three chunks after), decides how many quads the set has, places the records in the ring, starts
    // their copies and posts {word rows, base, staged, quads} for the others; the offsets it needs are requested one unit
    // ahead of that.  Until then a pair counts as whole.
    struct Place {
        int quad, k, n;
    };
    const uint32_t exp_words = static_cast<uint32_t>(L.exp_words);
    auto after = [&](const Place &u) {
        Place v{u.quad, u.k + 1, u.n};
        if (v.k == k_hi) {
            v.k = k_lo;
            v.quad += u.n;
            v.n = G.max_quads == 1 || ((v.quad - quad_lo) & 1) ? 1 : min(2, quad_hi - v.quad);
        }
        return v;
    };
    const bool leader = wig == 0;
    auto row_in_layer = [&](const Place &u, int row) { return min(4 * u.quad + (row < 4 * u.n ? row : 0), L.M - 1); };      // row 0..7 of the unit
    auto record_of = [&](const Place &u, int row) { return u.k * L.M + row_in_layer(u, row); };
    uint32_t off = 0u, end = 0u;                                       // leader: first and last exponent word
    auto load_span = [&](int rec) {
        off = static_cast<uint32_t>(__ldg(L.offsets + rec));
        end = rec + 1 < L.S * L.M ? static_cast<uint32_t>(__ldg(L.offsets + rec + 1)) : exp_words;
    };
    auto request = [&](const Place &u) {
        if (leader && u.quad < quad_hi) load_span(min(u.k + (u.k == k_lo ? lane >> 3 : 0), k_hi - 1) * L.M + row_in_layer(u, lane & 7));
    };
    uint32_t words = 0u, at = 0u, foot = 0u, base = 0u;                // leader: the unit being placed
    bool staged = false;
    auto place = [&](Place &u, int slot) {
        at = off;
        words = end - off;                                             // in storage order, whole word rows, inside the buffer
        const bool fits = words - 1u < (1u << 16) && ((words & 63u) | (off & 3u)) == 0u && off < end && end <= exp_words;
        if (u.n == 2 && u.k == k_lo) {
            bool longer = off < end && words > 64u * G.pair_rows;
            for (int k = k_lo + 4 + (lane >> 3); k < k_hi; k += 4) {   // a layer of more than four chunks
                load_span(k * L.M + row_in_layer(u, lane & 7));
                longer |= off < end && end - off > 64u * G.pair_rows;
            }
            if (__any_sync(0xFFFFFFFFu, longer)) u.n = 1;
        }
        uint32_t rows = fits && lane < 4 * u.n ? words >> 6 : 0u;
        rows = __reduce_max_sync(0xFFFFFFFFu, rows);
        foot = (4u * u.n * (rows * 256u + 32u) + 255u) & ~255u;
        staged = __all_sync(0xFFFFFFFFu, fits || lane >= 4 * u.n) && foot <= G.ring_bytes;
        base = slot == 0 ? ring : ring + G.ring_bytes - foot;
        if (lane == 0) {
            posted[4 * slot] = rows;
            posted[4 * slot + 1] = base;
            posted[4 * slot + 2] = staged ? 1u : 0u;
            posted[4 * slot + 3] = u.n;
        }
    };
    auto start_copies = [&](const Place &u, int slot) {
        const uint32_t bar = bar0 + 8u * slot;
        const int n = u.n;
        const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, lane < 4 * n ? words * 4u : 0u);
        const uint32_t rows = __reduce_max_sync(0xFFFFFFFFu, lane < 4 * n ? words >> 6 : 0u);
        if (lane == 0) mbar_expect_tx(bar, total);
        __syncwarp();
        if (lane < 4 * n) {
            bulk_copy_g2s(smem_base + base + lane * (rows * 256u + 32u), L.exp + at, words * 4u, bar);
            prefetch_l2(L.rem + static_cast<int64_t>(record_of(u, lane)) * L.Nc, static_cast<uint32_t>(L.Nc));
        }
    };

    // A lane's share of the copies that bring a chunk of its warp's sign/mantissa rows: 16 bytes of block lane / 8 of the
    // chunk, row (lane / 2) % 4 of each quad (dense: of each of the warp's rows).
    const uint8_t *rem[2];
    auto rem_rows = [&](const Place &u) {
#pragma unroll
        for (int q = 0; q < 2; q++)
            rem[q] = L.rem + static_cast<int64_t>(record_of(u, row_of(q, u.n, (lane >> 1) & 3))) * L.Nc + (lane >> 3) * 128 +
                     (NB > 0 ? wig * 32 + (lane & 1) * 16 : (lane & 7) * 16);
    };
    // A row's 32 bytes of a block are two rows of an 8 x 8 matrix, whose words the lanes want as ldmatrix deals them: one
    // instruction for two blocks of both quads instead of four loads.  Lane i supplies row i % 8 of matrix i / 8.
    // (49152 x 4096, limit6, one row 89.1 us, so 87.2; 12288 x 4096, eight rows 29.9, 29.1; rANS 144.2, 145.3, so not there, nor
    // for limit6 of 24 rows, whose registers are short: 4096 x 4096 16.0, so 16.3.)
    constexpr bool kRemMatrix = kHuff && !(NB == 3 && std::is_same<Dec, GemvSingle>::value), kFewPairs = kFew && !kHuff;
    const uint32_t rem_lane = kRemMatrix ? 16u * (lane & 7) + 128u * ((lane >> 3) & 1) + 512u * (lane >> 4) : 4u * lane;
    uint32_t half = 0u;                                                // half of the warp's buffer that holds the current chunk
    auto fetch = [&](int n, int blk, uint32_t to) {
        const uint32_t bytes = blk + (lane >> 3) < nblk ? 16u : 0u, dst = rem_at + to + 16u * lane;
        cp_async_16(dst, rem[0] + (bytes ? blk * 128 : -(lane >> 3) * 128), bytes);
        if (n > 1) cp_async_16(dst + 512u, rem[1] + (bytes ? blk * 128 : -(lane >> 3) * 128), bytes);
    };

    // How many quads the set of unit u has, now that it is known.  Dense, a warp's rows depend on it: those of the first chunk
    // are fetched once more if it was taken for a pair.
    auto settle = [&](Place &u, int n) {
        if (NB == 0 && n != u.n) {
            u.n = n;
            cp_async_wait();
            rem_rows(u);
            fetch(n, 0, half);
        }
        u.n = n;
    };

    Place cur{quad_lo, k_lo, min(G.max_quads, quad_hi - quad_lo)};
    request(cur);
    if (cur.quad < quad_hi) {
        rem_rows(cur);
        fetch(cur.n, 0, 0u);
        if (leader) {
            Place placed = cur;
            place(placed, 0);
            if (staged) start_copies(placed, 0);
            settle(cur, placed.n);
        }
    }
    Place nxt = after(cur);
    request(nxt);
    if (kRing && leader) {                                             // for the warp that fills the X ring
        const int sets = G.max_quads == 2 ? count_sets(L.offsets, L.S, L.M, exp_words, quad_lo, quad_hi, 64u * G.pair_rows) : max(quad_hi - quad_lo, 0);
        if (lane == 0) all_sets[group] = sets;
    }
    uint32_t prev_foot = staged ? foot : 0u;                           // leader: ring bytes of the unit being decoded

    // The table's place is a constant in the loads.  Where shared memory starts elsewhere records are decoded directly: right,
    // but several times as slow, so the status says so.
    bool usable = smem_base == kTableAt;
    if (!usable && tid == 0) atomicExch(&g_staged_status, 10);
    if (kHuff && prepared != nullptr) {
        if (!mbar_wait_bounded(table_bar, 0u) && tid == 0) atomicExch(&g_staged_status, 2);
        usable = usable && Dec::usable(*reinterpret_cast<const Tables *>(&tab));
    } else {
        load_tables(tab, targs, tid, kThreads);
        asm volatile("bar.sync 5, %0;" ::"n"(kThreads) : "memory");
        Dec::fill(smem, tab, targs, kc, tid, kThreads);
    }

    // Everything above read weights only.  X (and Y) belong to the previous kernel in the stream.
    if (!kHalf) pdl_wait();
    uint32_t launch_no = 0;
    if (exchange) {
        launch_no = *reinterpret_cast<const volatile uint32_t *>(peers.launches) + 1u;
        if (blockIdx.x == 0 && tid < peers.world) red_release_sys_add(pick(peers.ready, tid), 1u);
        // results that are not staged are stored from the first set on: see the end for those that are
        if (kShard == 2 && tid == 0 && !counter_wait_bounded(pick(peers.ready, peers.rank), launch_no * peers.world)) atomicExch(&g_staged_status, 8);
    }
    if (NB > 0 && !kRing && !kHalf) {
        const bool bulk = (reinterpret_cast<uintptr_t>(X) & 15u) == 0u;
        const uint32_t bytes = static_cast<uint32_t>(L.S) * L.Nc * 2u;
        if (tid == 0 && bulk) mbar_expect_tx(x_bar, bytes * B);
        if (bulk) __syncwarp();
        for (int b = bulk ? tid : warp; b < B; b += bulk ? kThreads : NG * kGemvWarps)
            copy_x_row(xs + b * G.x_pitch, X + static_cast<int64_t>(b) * L.S * L.Nc, bytes, x_bar, bulk, lane);
        if (!bulk && tid == 0) mbar_arrive(x_bar);
    }
    __syncthreads();
    if (NB > 0 && !kRing && !kHalf && !mbar_wait_bounded(x_bar, 0u) && tid == 0) atomicExch(&g_staged_status, 3);

    // Beside the previous kernel: its end is waited for, and X fetched, when the records of the first unit are here and those
    // of the second on their way.
    bool x_asked = false;
    auto ask_for_x = [&]() {
        x_asked = true;
        pdl_wait();
        const bool bulk = (reinterpret_cast<uintptr_t>(X) & 15u) == 0u;
        const uint32_t bytes = static_cast<uint32_t>(L.S) * L.Nc * 2u;
        if (bulk && tid == 0) mbar_expect_tx_only(x_bar, bytes * B);
        __syncwarp();
        if (!bulk || warp == 0)
            for (int b = bulk ? lane : warp; b < B; b += bulk ? 32 : NG * kGemvWarps)
                copy_x_row(xs + b * G.x_pitch, X + static_cast<int64_t>(b) * L.S * L.Nc, bytes, x_bar, bulk, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(x_bar);
    };

    // ---- decode and multiply -------------------------------------------------------------------------------------------
    float c[2][kAcc][4];
    auto clear = [&]() {
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
            for (int g = 0; g < kAcc; g++) c[q][g][0] = c[q][g][1] = c[q][g][2] = c[q][g][3] = 0.f;
    };
    clear();
    // ldmatrix: lane i supplies the address of row i % 8 of matrix i / 8: pairs 8j.., 8j + 4.., 32 + 8j.., 32 + 8j + 4.. of a
    // block.  Rows past the batch repeat the last one; their products are never read.  Few rows: rows 0..3 of pairs 8j.. and 0..3 of
    // pairs 8j + 4.., the same of pairs 32 + 8j.., and for rANS both again of the next block (49152 x 4096 144.2 us, so
    // 142.7; limit6 86.9, 87.8, so not there).
    uint32_t x_row[kAcc];
#pragma unroll
    for (int g = 0; g < kAcc; g++)
        x_row[g] = kFew ? xs + min(lane & 3, max(B, 1) - 1) * G.x_pitch + 32u * wig + 16u * ((lane >> 2) & 1) + 128u * (kFewPairs ? lane >> 3 : (lane >> 3) & 1)
                        : xs + min(8 * g + (lane & 7), max(B, 1) - 1) * G.x_pitch + 32u * wig + 16u * ((lane >> 3) & 1) + 128u * (lane >> 4);
    const int x_total = kRing ? x_segments() : 0;
    int x_slot = 0, x_seg = 0;
    uint32_t x_phase = 0u;
    auto x_wait = [&]() {
        if (kRing && !mbar_wait_bounded(x_full + 8u * x_slot, x_phase) && lane == 0) atomicExch(&g_staged_status, 3);
    };
    auto x_done = [&]() {
        if (kRing) {
            __syncwarp();
            if (lane == 0) mbar_arrive(x_empty + 8u * x_slot);
            x_seg++;
            if (++x_slot == G.x_slots) {
                x_slot = 0;
                x_phase ^= 1u;
            }
        }
    };

    auto keep = [&](int b, int row, float v) {                          // a result of a row-sharded layer
        if (kShard != 2) {
            ys[b * rows_cta + (row - row_lo)] = f32_to_bf16_rn(v);
        } else {
#pragma unroll 1
            for (int q = 0; q < peers.world; q++) pick(peers.y, q)[static_cast<int64_t>(b) * peers.m_total + peers.row_base + row] = f32_to_bf16_rn(v);
        }
    };

    uint32_t phases = 0u;
    int slot = 0;
    if (cur.quad < quad_hi && !leader) {
        settle(cur, posted[3]);
        nxt = after(cur);
    }
    while (cur.quad < quad_hi) {
        const uint32_t rows = posted[4 * slot], ubase = posted[4 * slot + 1];
        const bool is_staged = posted[4 * slot + 2] != 0u && usable;
        bool late = false;                    // leader: the next unit's copies have to wait for this one's space
        if (leader && nxt.quad < quad_hi) {
            place(nxt, slot ^ 1);
            late = staged && prev_foot + foot > G.ring_early;
            if (staged && !late) start_copies(nxt, slot ^ 1);
            prev_foot = staged ? foot : 0u;
        }
        request(after(nxt));
        if (kHalf && !x_asked) {
            if (is_staged && !mbar_wait_bounded(bar0 + 8u * slot, (phases >> slot) & 1u) && lane == 0) atomicExch(&g_staged_status, 1);
            ask_for_x();
            if (!mbar_wait_bounded(x_bar, 0u) && lane == 0) atomicExch(&g_staged_status, 3);
        }

        // the unit with n quads, by decoders of type D
        auto run = [&](auto quads, auto &dec) {
            constexpr int n = decltype(quads)::value;
            using D = typename std::remove_reference<decltype(dec[0])>::type;
            uint32_t *out[2] = {nullptr, nullptr};
            bool live[2] = {false, false};
            if (NB == 0) {
#pragma unroll
                for (int q = 0; q < n; q++) {
                    const int m = 4 * cur.quad + row_of(q, n, r);
                    live[q] = m < L.M;
                    out[q] = reinterpret_cast<uint32_t *>(Y) + (((static_cast<int64_t>(m) * L.S + cur.k) * L.Nc) >> 1) + (sigma4 >> 2);
                }
            }
            uint32_t xo = kRing ? 0u : static_cast<uint32_t>(cur.k * nblk) * 256u;
            auto pair = [&](auto which, uint32_t rw, uint32_t xa, bool both) {
                constexpr uint32_t j = decltype(which)::value;          // 0 or 2: block of the chunk
                uint32_t e[n][2][2], rems[4];                           // sign/mantissa words: [quad][block]
                if constexpr (!kRemMatrix) {
                } else if constexpr (n > 1) {
                    ldmatrix_x4<j * 128u>(rems, rw);
                } else {
                    ldmatrix_x2<j * 128u>(*reinterpret_cast<uint32_t (*)[2]>(rems), rw);
                }
                D::step(ctx, dec, e);
                uint32_t few[4];
                if constexpr (kFewPairs) ldmatrix_x4<j * 256u>(few, x_row[0] + xa);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    if (i == 0 || both) {
                        uint32_t w0[n], w1[n];
#pragma unroll
                        for (int q = 0; q < n; q++) {
                            const uint32_t w = kRemMatrix ? rems[2 * q + i] : q == 0 ? (i == 0 ? lds_now<j * 128u>(rw) : lds_now<j * 128u + 128u>(rw))
                                                      : (i == 0 ? lds_now<j * 128u + 512u>(rw) : lds_now<j * 128u + 640u>(rw));
                            w0[q] = bitselect(prmt(w, 0u, 0x1100u), e[q][i][0], kRemMask);
                            w1[q] = bitselect(prmt(w, 0u, 0x3322u), e[q][i][1], kRemMask);
                        }
                        if constexpr (kFew) {
                            uint32_t f[2];
                            if constexpr (kFewPairs) {
                                f[0] = few[2 * i];
                                f[1] = few[2 * i + 1];
                            } else if (i == 0) {
                                ldmatrix_x2<j * 256u>(f, x_row[0] + xa);
                            } else {
                                ldmatrix_x2<j * 256u + 256u>(f, x_row[0] + xa);
                            }
                            mma_bf16_16x8x16(c[0][0], w0[0], n > 1 ? w0[n - 1] : 0u, w1[0], n > 1 ? w1[n - 1] : 0u, f[0], f[1]);
                        } else if constexpr (NB > 0) {
#pragma unroll
                            for (int g = 0; g < kAcc; g++) {
                                uint32_t f[4];
                                if (i == 0) ldmatrix_x4<j * 256u>(f, x_row[g] + xa);
                                else ldmatrix_x4<j * 256u + 256u>(f, x_row[g] + xa);
#pragma unroll
                                for (int q = 0; q < n; q++) mma_bf16_16x8x16(c[q][g], f[0], f[1], f[2], f[3], w0[q], w1[q]);
                            }
                        } else {
#pragma unroll
                            for (int q = 0; q < n; q++) {
                                if (live[q]) {
                                    out[q][(j + i) * 64u] = w0[q];
                                    out[q][(j + i) * 64u + 32u] = w1[q];
                                }
                            }
                        }
                    }
                }
            };
            // Chunks of four blocks.  While one is used the next (the next unit's first, at the end) is copied into the other
            // half of the warp's buffer.
#pragma unroll 1
            for (int blk = 0; blk < nblk; blk += kRG) {
                cp_async_wait();
                __syncwarp();                 // the chunk is here for every lane, and the other half is read out
                if (blk + kRG < nblk) {
                    fetch(n, blk + kRG, half ^ kRemChunk);
                } else if (nxt.quad < quad_hi) {
                    rem_rows(nxt);
                    fetch(nxt.n, 0, half ^ kRemChunk);
                }
                x_wait();
                const uint32_t rw = rem_at + half + rem_lane, xa = kRing ? x_slot * G.x_slot : xo;
                const int left = nblk - blk;
                using J0 = std::integral_constant<uint32_t, 0>;
                using J2 = std::integral_constant<uint32_t, 2>;
                if (left >= kRG) {
                    pair(J0{}, rw, xa, true);
                    pair(J2{}, rw, xa, true);
                } else {
                    pair(J0{}, rw, xa, left > 1);
                    if (left > 2) pair(J2{}, rw, xa, false);
                }
#pragma unroll
                for (int q = 0; q < n; q++) {
                    dec[q].clamp();
                    if (NB == 0) out[q] += kRG * 64;
                }
                half ^= kRemChunk;
                xo += kRG * 256u;
                x_done();
            }
        };
        auto dispatch = [&](auto quads) {
            constexpr int n = decltype(quads)::value;
            if (is_staged) {
                const bool arrived = mbar_wait_bounded(bar0 + 8u * slot, (phases >> slot) & 1u);
                phases ^= 1u << slot;
                if (!arrived && lane == 0) atomicExch(&g_staged_status, 1);
                Dec dec[n];
#pragma unroll
                for (int q = 0; q < n; q++) dec[q].open(smem_base + ubase + row_of(q, n, r) * (rows * 256u + 32u) + sigma4, rows);
                run(quads, dec);
            } else {
                if (posted[4 * slot + 2] != 0u) {          // its copies were started all the same
                    if (!mbar_wait_bounded(bar0 + 8u * slot, (phases >> slot) & 1u) && lane == 0) atomicExch(&g_staged_status, 1);
                    phases ^= 1u << slot;
                }
                GemvDirect<Codec> dec[n];
#pragma unroll
                for (int q = 0; q < n; q++) {
                    const uint32_t first = static_cast<uint32_t>(__ldg(L.offsets + record_of(cur, row_of(q, n, r))));
                    dec[q].open(GlobalRecord{L.exp, exp_words, first + (sigma4 >> 2)}, &tab);
                }
                run(quads, dec);
            }
        };
        const int n = cur.n;
        if (n == 2) dispatch(std::integral_constant<int, 2>{});
        else dispatch(std::integral_constant<int, 1>{});

        const bool set_done = cur.k == k_hi - 1;
        if (NB > 0 && set_done) {
            gemv_group_barrier(group);        // the previous set's partial sums have been read
#pragma unroll
            for (int q = 0; q < 2; q++) {
                if constexpr (kFew) {         // row r of the quad and X rows 2 (t % 2) and the next, of half s where the columns are that half's
                    if ((t >> 1) == (gq & 1)) {
                        float *pp = part + (wig * 2 + q) * 32 + 16 * (gq & 1) + 8 * (t & 1) + r;
                        pp[0] = c[0][0][2 * q];
                        pp[4] = c[0][0][2 * q + 1];
                    }
                } else {
#pragma unroll
                    for (int g = 0; g < kAcc; g++) part[((wig * 2 + q) * kAcc + g) * 32 + lane] = c[q][g][0] + c[q][g][3];
                }
            }
            clear();
        }
        gemv_group_barrier(group);            // the unit's ring space is free; partial sums and the next unit's place are visible
        if (late) start_copies(nxt, slot ^ 1);
        if (NB > 0 && set_done) {
            for (int z = wig ^ 2; z < n * kAcc; z += kGemvWarps) {      // warp z % 4 ^ 2, the leader last, finishes (quad, eight X rows) z
                const int q = z / kAcc, g = z % kAcc;
                const float *pp = part + (q * kAcc + g) * 32 + (kFew ? lane & 15 : lane);
                float v = kFew ? pp[0] + pp[16] : pp[0];
#pragma unroll
                for (int w = 1; w < kGemvWarps; w++) v += kFew ? pp[w * 64 * kAcc] + pp[w * 64 * kAcc + 16] : pp[w * 64 * kAcc];
                const int row = 4 * (cur.quad + q) + t, b = 8 * g + gq;
                if (split) {
                    acc[((cur.quad + q - cta_lo) * NG + group) * 32 + lane] = v;
                } else if (b < B && row < L.M) {
                    if (exchange) keep(b, row, v);
                    else if (B <= BHI_MAX_BATCH) Y[static_cast<int64_t>(b) * L.M + row] = finish_value(v, bias, row);
                    else Y[static_cast<int64_t>(b) * L.M + row] =
                        f32_to_bf16_rn(bias ? v + __uint_as_float(static_cast<uint32_t>(load_written(bias + row)) << 16) : v);
                }
            }
        }
        if (nxt.quad < quad_hi && !leader) settle(nxt, posted[4 * (slot ^ 1) + 3]);
        cur = nxt;
        nxt = after(nxt);
        slot ^= 1;
    }

    if (kHalf && !x_asked) ask_for_x();       // a group without units copies its share of an unaligned X
    if (NB == 1 && split) {                   // the groups' sums, in the order of their chunks
        asm volatile("bar.sync 5, %0;" ::"n"(kThreads) : "memory");
        for (int i = warp; i < cta_hi - cta_lo; i += NG * kGemvWarps) {
            float v = 0.f;
#pragma unroll
            for (int g = 0; g < NG; g++)
                if (L.S * g / NG < L.S * (g + 1) / NG) v += acc[(i * NG + g) * 32 + lane];
            const int row = 4 * (cta_lo + i) + t;
            if (gq < B && row < L.M) {
                if (exchange) keep(gq, row, v);
                else Y[static_cast<int64_t>(gq) * L.M + row] = finish_value(v, bias, row);
            }
        }
    }
    if (kRing) {                              // groups with fewer units see the segments through, so that the others get theirs
        while (x_seg < x_total) {
            x_wait();
            x_done();
        }
    }
    if (exchange) {
        // one thread asks whether every peer's buffer may be overwritten (an acquire at system scope); the barrier that
        // makes the staged results visible hands its answer to the others
        if (kShard != 2) {
            if (tid == 0 && !counter_wait_bounded(pick(peers.ready, peers.rank), launch_no * peers.world)) atomicExch(&g_staged_status, 8);
            asm volatile("bar.sync 5, %0;" ::"n"(kThreads) : "memory");
            for (int i = tid; i < B * rows_cta; i += kThreads) {
                const int b = i / rows_cta, rr = i - b * rows_cta;
                const uint16_t v = ys[i];
                const int64_t to = static_cast<int64_t>(b) * peers.m_total + peers.row_base + row_lo + rr;
#pragma unroll
                for (int q = 0; q < kMaxPeers; q++)
                    if (q < peers.world) peers.y[q][to] = v;
            }
        }
        exchange_finish(peers, launch_no);
    }
}

// ---- host side -------------------------------------------------------------------------------------
int gemv_groups();      // 0 = by the forms below, else 2 or 4 groups only: see bhi_set_quad_warps

enum class GemvX { none, resident, ring };

// One way to lay a launch out: how many groups, how many CTAs share an SM, how many quads a unit has, how many quarters of
// a unit the record ring holds, where X is.
struct GemvForm {
    int groups, per_sm, quads, quarters;
    GemvX x;
};

static uint32_t mean_rows(const Layer &L) {      // word rows of a record
    const int64_t per_row = 64 * static_cast<int64_t>(L.S) * L.M;
    return static_cast<uint32_t>((L.exp_words + per_row * 15 / 16) / per_row);
}

// Shared-memory plan of a form; false when it does not fit.  The record ring is sized by the average record, so that it takes a
// unit whose longest is a word row and an eighth longer (a word row where it has room for one unit only), and grows into what
// the form leaves.  Rows of a layer whose scales differ have records of different lengths: a pair of quads that does not fit
// together comes quad by quad, and a quad that does not fit alone is decoded from global memory, several times as slow.
// (4096 x 12288, rANS, one row of X, row scales log-normal with sigma 0.35: 177 us without the growth and the quads, 42 with
// them, as with equal rows; 12288 x 4096, limit6, four rows: 76 and 30.)
static bool gemv_plan(const Layer &L, int B, uint32_t table_bytes, int acc_groups, bool few, const GemvForm &f, int grid,
                      bool stage_results, GemvGeom &G, uint32_t &smem_bytes) {
    auto up = [](uint64_t v) { return static_cast<uint32_t>((v + 255u) & ~static_cast<uint64_t>(255u)); };
    const uint32_t cap = f.per_sm == 2 ? kSmemMax / 2 - 512 : kSmemMax;
    const uint32_t rows = mean_rows(L);
    const int nquads = (L.M + 3) / 4, nq = (nquads + grid - 1) / grid + 1;                         // most quads of a CTA
    // Few quads and several chunks: a group would take the chunks of its quad or two one after the other while others have
    // none.  The groups of a CTA share its quads instead and divide the chunks, where that shortens the longest group's
    // work by a tenth (a unit of one quad takes six tenths of one of two).
    auto sets = [&](int quads) { return f.quads == 2 ? quads / 2 * 10 + quads % 2 * 6 : quads * 6; };
    const int group_quads = (nquads + grid * f.groups - 1) / (grid * f.groups), cta_quads = (nquads + grid - 1) / grid;
    G.split = f.x != GemvX::ring && L.S > 1 && acc_groups <= 1 &&
              10 * ((L.S + f.groups - 1) / f.groups) * sets(cta_quads) <= 9 * L.S * sets(group_quads);
    // table | exact tables, barriers | partial sums | staged results | split sums | sign/mantissa chunks | record rings | X (their slack)
    G.exact_off = up(table_bytes);
    G.part_off = G.exact_off + kExactBytes + kGemvCtrlBytes;
    G.ys_off = G.part_off + up(static_cast<uint64_t>(f.groups) * kGemvWarps * 64 * 4 * acc_groups);
    G.acc_off = G.ys_off + (stage_results ? up(static_cast<uint64_t>(B) * 4 * nq * 2) : 0u);
    G.rem_off = G.acc_off + (G.split && acc_groups ? up(static_cast<uint64_t>(nq) * f.groups * 128) : 0u);
    G.ring_off = G.rem_off + f.groups * kGemvWarps * 2u * kRemChunk;
    auto unit = [&](uint64_t r) { return 4ull * f.quads * (r * 256u + 32u); };
    const uint64_t spare = f.quarters > 4 ? 1u + rows / 8u : 1u;
    const uint64_t wanted = unit(rows) * f.quarters / 4u, longest = f.quarters ? unit(rows + spare) : 0u;
    G.ring_bytes = up(wanted > longest ? wanted : longest);
    const uint64_t x_off = static_cast<uint64_t>(G.ring_off) + static_cast<uint64_t>(f.groups) * G.ring_bytes;
    if (x_off + kSlackBytes > cap) return false;
    G.x_off = static_cast<uint32_t>(x_off);
    uint64_t x_bytes = 0;
    G.x_slots = 0;
    G.x_pitch = G.x_slot = 0;
    if (f.x == GemvX::resident) {
        const uint64_t pitch = static_cast<uint64_t>(L.S) * L.Nc * 2u + (few ? 2u : 1u) * kXPad;
        x_bytes = pitch * B + (few ? 256u : 0u);                       // two blocks are read together, the last one's neighbour too
        G.x_pitch = static_cast<uint32_t>(pitch);
    } else if (f.x == GemvX::ring) {
        G.x_pitch = 2u * kXSegCols + kXPad;
        G.x_slot = G.x_pitch * B;
        G.x_slots = kXSlotsMax;
        while (G.x_slots > 2 && x_off + static_cast<uint64_t>(G.x_slots) * G.x_slot > cap) G.x_slots--;
        x_bytes = static_cast<uint64_t>(G.x_slots) * G.x_slot;
    }
    if (x_bytes < kSlackBytes) x_bytes = kSlackBytes;
    if (x_off + x_bytes > cap) return false;
    // What is left goes to the rings, for units of longer records; copies start as early as in the ring that was asked for
    // (two units of all the space in flight at once cost 2 to 4 % where the form means them to take turns).
    G.ring_early = G.ring_bytes;
    if (f.quarters) G.ring_bytes += ((cap - static_cast<uint32_t>(x_off + x_bytes)) / f.groups) & ~255u;
    G.x_off += f.groups * (G.ring_bytes - G.ring_early);
    G.pair_rows = G.ring_bytes < 256u ? 0u : (G.ring_bytes / 8u - 32u) / 256u;
    smem_bytes = static_cast<uint32_t>(G.x_off + x_bytes);
    G.batch = B;
    G.max_quads = f.quads;
    return true;
}

template <class Dec, int NB, int NG, bool kRing, int kShard, bool kHalf, bool kFew, bool kShift = kShiftsRegisters<Dec, NB, NG, kRing>>
static int gemv_start_as(const Layer &L, const typename Dec::Codec::Args &targs, const uint8_t *prepared, const uint16_t *X,
                      const uint16_t *bias, uint16_t *Y, const PeerSet *peers, int grid, const GemvGeom &G, uint32_t smem_bytes,
                      cudaStream_t st) {
    auto kernel = gemv_kernel<Dec, NB, NG, kRing, kShard, kHalf, kFew, kShift>;
    if (int rc = staged_prepare(kernel, kSmemMax, kShift ? kShiftAtLaunch : 0)) return rc;
    PeerSet ps{};
    if (peers) ps = *peers;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NG * kGemvWarps * 32 + kRingThreads<kRing, kShift>);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap_launches() ? 1 : 0;
    const uint32_t bits = ans_bits_of(targs);
    const GemvConsts k{bits, (1u << bits) - 1u, bits == 12u ? 0xFFFu : (2u << bits) - 1u, 8u, Dec::kTableBytes >> bits};
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, L, targs, prepared, X, bias, Y, ps, G, k);
    return e == cudaSuccess ? BHI_OK : cuda_fail(e, "gemv kernel launch");
}

template <class Dec, int NB, int NG, bool kRing>
static int gemv_start(const Layer &L, const typename Dec::Codec::Args &targs, const uint8_t *prepared, const uint16_t *X,
                      const uint16_t *bias, uint16_t *Y, const PeerSet *peers, bool direct, bool few, bool shift, int grid, const GemvGeom &G,
                      uint32_t smem_bytes, cudaStream_t st) {
    if constexpr (kRing && NG == 4 && kShiftsOrNot<Dec, NB>)
        if (!shift) return gemv_start_as<Dec, NB, NG, kRing, 0, false, false, false>(L, targs, prepared, X, bias, Y, peers, grid, G, smem_bytes, st);
    if constexpr (NB == 1) {
        if constexpr (kRing) {
            if (direct) return gemv_start_as<Dec, NB, NG, kRing, 2, false, false>(L, targs, prepared, X, bias, Y, peers, grid, G, smem_bytes, st);
        }
        if (peers) return gemv_start_as<Dec, NB, NG, kRing, 1, false, false>(L, targs, prepared, X, bias, Y, peers, grid, G, smem_bytes, st);
        if constexpr (!kRing) {
            if (few) return gemv_start_as<Dec, NB, NG, kRing, 0, false, true>(L, targs, prepared, X, bias, Y, peers, grid, G, smem_bytes, st);
        }
    }
    return gemv_start_as<Dec, NB, NG, kRing, 0, false, false>(L, targs, prepared, X, bias, Y, peers, grid, G, smem_bytes, st);
}

// The first form that fits, best first.  Measured on 12288 x 4096, limit6, in us where each fits with one, four, eight rows:
//   two CTAs per SM, X resident, two units in the ring   25.8
//   same, 1.25 units (the next unit's copies wait for this one's space; the other groups work on)   26.2 / 26.7
//   one CTA of twice the groups (one copy of table and X for all), X resident   27.2 / 27.6; 1.25 units 28.1 / 28.7 / 28.9
//   same, room for one unit only, where X stays resident just so (3584 x 18944, two rows: rANS 70.5 against 79.9 with X
//   through the ring, which also bars dividing the chunks; tables of the reference's builder 50.6 against 69.2)
//   same, X through the ring   30.9 / 31.4 / 31.9
//   units of four rows, for long records   35.7
// The last form stages no record at all.
template <class Dec, int NB, bool kLast>
static int gemv_launch_dec(const Layer &L, const typename Dec::Codec::Args &targs, const uint8_t *prepared, const uint16_t *X,
                           const uint16_t *bias, uint16_t *Y, const PeerSet *peers, int B, cudaStream_t st) {
    constexpr GemvX kFew = NB == 0 ? GemvX::none : GemvX::resident, kMany = NB == 0 ? GemvX::none : GemvX::ring;
    const GemvForm forms[] = {{2, 2, 2, 8, kFew}, {2, 2, 2, 5, kFew}, {4, 1, 2, 8, kFew}, {4, 1, 2, 5, kFew}, {4, 1, 2, 4, kFew},
                              {4, 1, 2, 8, kMany}, {4, 1, 2, 5, kMany}, {4, 1, 1, 5, kFew}, {4, 1, 1, 5, kMany}, {2, 1, 1, 5, kMany},
                              {2, 1, 1, 0, kMany}};
    const int nquads = (L.M + 3) / 4, only = gemv_groups();
    for (int direct = 0; direct <= (kLast && peers != nullptr ? 1 : 0); direct++) {
        for (const GemvForm &f : forms) {
            if (only && f.groups != only) continue;
            if (!kLast && (f.quads < 2 || f.x == GemvX::ring)) break;
            if (peers != nullptr && !direct && f.quarters == 0) continue;           // staged records before staged results
            if (direct && f.x != GemvX::ring) continue;                            // so many rows that X hardly counts
            if (NB > 1 && (f.x == GemvX::resident || f.groups == 2)) continue;     // more than eight rows hardly ever fit
            int grid = sm_count() * f.per_sm;
            if (grid > nquads) grid = nquads;
            GemvGeom G{};
            uint32_t smem_bytes = 0;
            const bool sixes = f.quads == 2 && nquads > 5 * grid && nquads < 7 * grid;       // some CTA has six quads
            const bool long_chunks = L.S > 1 && L.Nc >= 12 * 128 && L.S * L.Nc >= 54 * 128;
            const bool shift = !kShiftsOrNot<Dec, NB> || (Dec::kRans ? f.quads == 2 && nquads > 4 * grid : !(sixes && long_chunks));
            const bool few = NB == 1 && B <= kFewRows && peers == nullptr && f.x == GemvX::resident;
            if (!gemv_plan(L, B, Dec::kTableBytes, NB, few, f, grid, peers != nullptr && !direct, G, smem_bytes)) continue;
            if (f.x == GemvX::ring) {
                if constexpr (NB > 0 && kLast) {
                    if constexpr (NB == 1) {
                        if (f.groups == 2) return gemv_start<Dec, NB, 2, true>(L, targs, prepared, X, bias, Y, peers, direct, few, shift, grid, G, smem_bytes, st);
                    }
                    return gemv_start<Dec, NB, 4, true>(L, targs, prepared, X, bias, Y, peers, direct, few, shift, grid, G, smem_bytes, st);
                }
            } else {
                if constexpr (NB <= 1) {
                    if (f.groups == 2) return gemv_start<Dec, NB, 2, false>(L, targs, prepared, X, bias, Y, peers, direct, few, shift, grid, G, smem_bytes, st);
                    return gemv_start<Dec, NB, 4, false>(L, targs, prepared, X, bias, Y, peers, direct, few, shift, grid, G, smem_bytes, st);
                }
            }
        }
    }
    return kStagedDeclined;
}

// The kHalf launch of a small layer, in half an SM's shared memory.  Where a group has pairs of quads, their ring has to have room for
// rows that differ in scale, as the other forms' have: pairs that do not fit come quad by quad, each waiting for its records.  (Rows
// log-normal with sigma 0.6, other forms / half an SM with less room than this: limit6, four rows, 1200 x 4096  7.3/9.6, 2300 x 4096
// 8.4/10.1; sigma 0.35, rANS of 12 bits, two rows, 1200 x 4096  12.1/14.7.)  rANS has no longest code, so its rows differ more.
template <class Dec>
static int gemv_launch_half(const Layer &L, const typename Dec::Codec::Args &targs, const uint8_t *prepared, const uint16_t *X,
                            const uint16_t *bias, uint16_t *Y, int B, cudaStream_t st) {
    const int nquads = (L.M + 3) / 4, grid = nquads < sm_count() ? nquads : sm_count();
    for (int quarters = 8; quarters >= 4; quarters -= 4) {             // two units in the ring, or the one that most groups have
        GemvGeom G{};
        uint32_t smem_bytes = 0;
        if (!gemv_plan(L, B, Dec::kTableBytes, 1, B <= kFewRows, GemvForm{2, 2, 2, quarters, GemvX::resident}, grid, false, G, smem_bytes)) continue;
        const int cta_quads = (nquads + grid - 1) / grid;
        const uint32_t rows = mean_rows(L), room = Dec::kRans ? 2u * rows - 1u : rows + rows / 2u + 1u;
        if ((G.split ? cta_quads : (cta_quads + 1) / 2) < 2 || G.pair_rows >= room)
            return B <= kFewRows ? gemv_start_as<Dec, 1, 2, false, 0, true, true>(L, targs, prepared, X, bias, Y, nullptr, grid, G, smem_bytes, st)
                                 : gemv_start_as<Dec, 1, 2, false, 0, true, false>(L, targs, prepared, X, bias, Y, nullptr, grid, G, smem_bytes, st);
    }
    return kStagedDeclined;
}

// Layers of up to this many quads per SM, counting each of their chunks, take half of each SM: a unit of two quads, or two of
// one, for each of an SM's two groups.  Other forms / half an SM, in us, one row of X but where a count stands: back to back in a graph, and
// with an elementwise kernel before each launch (after which nothing can start early; what comes before a launch is not known here):
//   limit6         512 x 2048  3.9/3.5, 6.6/6.7   1024 x 4096  6.3/5.4, 8.8/9.2   2048 x 2048  5.6/4.2, 8.0/8.0   eight rows  6.0/4.5, 8.4/8.4
//                  2368 x 4096  8.2/6.7, 10.5/11.0   1024 x 6144 (two chunks)  6.4/5.5, 8.9/9.2
//                  beyond the line  4096 x 2048  7.3/7.7   2048 x 6144  9.1/10.3   4096 x 4096  11.2/12.7
//   rANS, 8 bits   512 x 3584  7.5/6.7, 10.2/10.1   1024 x 4096  9.2/8.0, 11.5/11.9   2048 x 2048  7.6/6.7, 10.5/10.7   four rows  7.9/6.8, 10.3/10.8
//   rANS, 12 bits  1024 x 4096  10.3/8.9, 13.5/13.1   2048 x 2048  9.1/8.0, 12.1/12.1   1180 x 6144  11.6/10.6   700 x 6144  10.1/10.4
// 8-bit rANS has the larger table in the other forms and fills half an SM's pipes sooner than an SM's.  It takes the form for one chunk
// (425 x 7168  7.9/8.8) with more quads than half the SMs (300 x 3584  6.7/6.3; 256 x 3584  6.1/6.3, 128 x 4096  6.5/6.9) and up to
// kHalfAnsCols columns of quads per SM (two rows, beyond it, 1536 x 4096  10.2/9.7, 12.7/13.8   2368 x 4096  11.9/11.1, 14.3/15.6).
// Without launch overlap no next kernel comes early, half of each SM would stand empty and the form is not taken (1024 x 4096 limit6
// 7.9/8.3, 2368 x 4096 limit6 9.4/10.2, rANS 13.4/14.7).
// More than two chunks are divided among four groups instead (512 x 18944: 9.1/12.9, 512 x 12288: 11.1/10.5).  Pair tables of
// 14 bits leave no room beside themselves and of 13 gain only where a group has one quad at most and often not then
// (1024 x 1024 escape 4.2/3.8, 1024 x 4096 8.2/8.1, 512 x 2048 reference 6.0/6.3, 2048 x 2048 8.4/9.7), so they stay out.
constexpr int kHalfUnits = 4, kHalfChunks = 2, kHalfAnsCols = 4 * 2048;

// kLast: no other decoder is tried after this one, so it takes the less favourable forms too.  kMore: more than eight rows.
template <class Dec, bool kLast, bool kMore>
static int gemv_launch_rows(const Layer &L, const typename Dec::Codec::Args &targs, const uint8_t *prepared, const uint16_t *X,
                            const uint16_t *bias, uint16_t *Y, const PeerSet *peers, int B, cudaStream_t st) {
    if (B == 0) return gemv_launch_dec<Dec, 0, kLast>(L, targs, prepared, X, bias, Y, peers, B, st);
    if (B <= 8) return gemv_launch_dec<Dec, 1, kLast>(L, targs, prepared, X, bias, Y, peers, B, st);
    if constexpr (kMore) {
        if (B <= 16) return gemv_launch_dec<Dec, 2, kLast>(L, targs, prepared, X, bias, Y, peers, B, st);
        if (B <= 24) return gemv_launch_dec<Dec, 3, kLast>(L, targs, prepared, X, bias, Y, peers, B, st);
        return gemv_launch_dec<Dec, 4, kLast>(L, targs, prepared, X, bias, Y, peers, B, st);
    }
    return kStagedDeclined;
}

// Each eight rows more cost one product per decoded word, and their accumulators registers (see kShiftsRegisters).  Here / by way
// of the dense matrix and a library GEMM, in us, graph-replayed from HBM, at 16, 24 and 32 rows:
//                12288 x 4096                        4096 x 12288                       50000 x 2560
//   limit6       33.9/53.0  41.7/53.2  47.5/53.1     33.5/57.1  40.7/57.3  46.8/57.3    82.3/129  97.2/130  115/130
//   escape       43.4/56.3  47.2/56.5  56.2/56.6     44.3/60.6  48.8/61.0  61.4/60.9    101/133   114/133  133/133
//   rANS, 8 bit  55.1/61.8  60.8/62.1  66.9/62.1     54.4/66.6  60.1/66.8  65.6/66.9    136/151   149/152  165/152
// (1024 x 4096: limit6 9.8/16.8, 11.8/15.2, 13.7/15.3; escape 10.7/18.7, 12.5/17.1, 14.4/17.2; rANS 11.5/19.2, 13.2/17.6, 15.5/17.8.)
// Only rANS would be served faster by the dense matrix, from 25 rows on (pair tables alike there).  It is not: with so few rows the
// library divides the columns among its blocks and adds their sums as BF16, up to 1.5 % of the results' rms off, where the sums here
// stay in 32 bits (0.2 %, the rounding of the result).
constexpr int kGemvMaxRows = 32;

// B rows of X (0: the dense matrix into Y).  pair_complete: the caller knows that no code of the prepared table is longer
// than 6 bits; only a tuning hint, the kernel reads from the table header whether it is so.
// The larger table first, where it leaves room for the favourable forms, although its CTAs then have an SM to themselves; one
// row of X, in us, with the larger / only the smaller table:
//                           1024 x 4096   4096 x 4096   12288 x 4096   4096 x 12288   5120 x 5120
//   pair table, 14 / 13 bits    8.4 / 8.8   14.7 / 16.1    34.9 / 37.1    35.5 / 37.7   25.4 / 23.5   (escape)
//   rANS, 8 bits, 64 / 32 KB    9.4 / 9.2   17.1 / 19.4    43.3 / 50.0    42.5 / 52.5   30.0 / 30.9
template <class Codec>
int gemv_launch(const Layer &L, const typename Codec::Args &targs, const uint8_t *prepared, const uint16_t *X,
                       const uint16_t *bias, uint16_t *Y, const PeerSet *peers, int B, bool pair_complete, cudaStream_t st) {
    if (!staged_shape_ok(L) || !aligned(prepared, 16) || B > kGemvMaxRows) return kStagedDeclined;
    if (static_cast<int64_t>(L.S) * L.M >= (1ll << 31) || L.exp_words >= (1ll << 32)) return kStagedDeclined;
    const bool half = overlap_launches() && B >= 1 && B <= 8 && peers == nullptr && gemv_groups() == 0 && L.S <= kHalfChunks &&
                      L.S * ((L.M + 3ll) / 4) <= static_cast<int64_t>(kHalfUnits) * sm_count();
    if constexpr (std::is_same<Codec, HuffCodec>::value) {
        if (half && pair_complete) {
            const int rc = gemv_launch_half<GemvSingle>(L, targs, prepared, X, bias, Y, B, st);
            if (rc != kStagedDeclined) return rc;
        }
        if (prepared == nullptr) return gemv_launch_rows<GemvPair<kPairBits>, true, false>(L, targs, prepared, X, bias, Y, peers, B, st);
        if (pair_complete) return gemv_launch_rows<GemvSingle, true, true>(L, targs, prepared, X, bias, Y, peers, B, st);
        const int rc = gemv_launch_rows<GemvPair<kWidestBits>, false, false>(L, targs, prepared, X, bias, Y, peers, B, st);
        if (rc != kStagedDeclined) return rc;
        return gemv_launch_rows<GemvPair<kWideBits>, true, true>(L, targs, prepared, X, bias, Y, peers, B, st);
    } else {
        // (a finer model on a layer of at most a quad per group: filling the larger table costs more than its conflicts)
        int rc = kStagedDeclined;
        const int64_t nquads = (L.M + 3ll) / 4;
        const bool half_ans = half && (targs.bits > 8 || (L.S == 1 && 2 * nquads > sm_count() && nquads * L.Nc <= static_cast<int64_t>(kHalfAnsCols) * sm_count()));
        if (half_ans && targs.bits == 8) rc = gemv_launch_half<GemvAns<true, 64 * 1024>>(L, targs, prepared, X, bias, Y, B, st);
        if (half_ans && rc == kStagedDeclined) rc = gemv_launch_half<GemvAns<false, 32 * 1024>>(L, targs, prepared, X, bias, Y, B, st);
        if (rc != kStagedDeclined) return rc;
        if (targs.bits == 8) rc = gemv_launch_rows<GemvAns<true, 64 * 1024>, false, false>(L, targs, prepared, X, bias, Y, peers, B, st);
        else if (L.M > 16 * sm_count()) rc = gemv_launch_rows<GemvAns<false, 64 * 1024>, false, false>(L, targs, prepared, X, bias, Y, peers, B, st);
        if (rc != kStagedDeclined) return rc;
        return gemv_launch_rows<GemvAns<false, 32 * 1024>, true, true>(L, targs, prepared, X, bias, Y, peers, B, st);
    }
}

}  // namespace bhi

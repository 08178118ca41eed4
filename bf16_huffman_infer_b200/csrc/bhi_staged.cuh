// What the decode-side kernels share (sm_100a): shared-memory constants, PTX wrappers, folded Huffman tables, the counters
// of row-sharded layers, and the host side's launch helpers.
//
// Every wait on an mbarrier is bounded; on expiry the warp records a status code in a device word (bhi_debug_status), skips
// the record and carries on: a lost copy cannot hang the GPU.  Cursors are clamped once per group of blocks, so corrupt
// tables or data cannot walk a read out of the CTA's shared memory.
#pragma once

#include <mutex>
#include <type_traits>
#include <unordered_map>

#include "bhi_common.cuh"

namespace bhi {

constexpr int kStagedDeclined = -1;

constexpr int kPairBits = 12;
constexpr int kPairEntries = 1 << kPairBits;
constexpr int kCopies = 4;                     // bank-interleaved copies of the fast table (lane & 3 picks one)
constexpr int kLutBytes = kPairEntries * 4 * kCopies;   // 64 KB (Huffman pair table; rANS uses the first 4 KB)
constexpr int kExactBytes = 2048;              // table-exact copies for rare windows / direct records
constexpr int kCtrlBytes = 1024;               // mbarriers (2 per warp) + row counter
constexpr int kSlackBytes = 2048;              // readable space above the last ring
constexpr int kSmemMax = 227 * 1024;
constexpr int kRingMax = 8192;
constexpr uint32_t kSpinLimit = 1u << 22;

// pair-table entry fields
constexpr uint32_t kEntBits = 0xFu;            // bits 0..3: stream bits consumed (bit 4 stays zero: the word is also a shift count)
constexpr uint32_t kEntSingle = 0x20u;         // only the first symbol is resolved
constexpr uint32_t kEntExact = 0x40u;          // nothing resolved: use the exact tables
constexpr uint32_t kRemMask = 0x807F807Fu;     // sign + mantissa bits of a bf16x2 word; the rest is exponent

// Multipliers handed to the kernel at launch.  Integer multiply-add runs on the FMA pipe, plain
// shifts/adds on the (half-rate, saturated) integer pipe; because the compiler cannot see these
// values it has to keep the multiply-add form.
struct Consts {
    uint32_t ans_bits, ans_mask;             // rANS: probability precision of the layer's table and 2^bits - 1
    uint32_t eight, entry;                   // entry = bytes between consecutive fast-table entries (4 * copies)
};

// A prepared-table blob (Huffman): one copy of the folded pair table, the exact tables, the single-symbol tables with one
// copy per lane (codes of at most 6 bits), two pair tables with a wider index.
constexpr int kSingleBytes = 2 * 64 * 128;
constexpr int kWideBits = 13, kWidestBits = 14;
constexpr int kPreparedSingle = kPairEntries * 4 + kExactBytes;
constexpr int kPreparedWide = kPreparedSingle + kSingleBytes;
constexpr int kPreparedWidest = kPreparedWide + (4 << kWideBits);
constexpr int kPreparedBytes = kPreparedWidest + (4 << kWidestBits);

static_assert(sizeof(HuffTables) + 8 <= kExactBytes && sizeof(AnsTables) <= kExactBytes, "exact tables do not fit");
static_assert((4 << kAnsBitsMax) * kCopies <= kLutBytes, "the largest rANS table does not fit the fast-table region");

// 0 = fine; otherwise the last failure code.  Each source file of kernels has one of its own, which its take_status is for.
static __device__ int g_staged_status = 0;

// reads and clears this source file's
static cudaError_t take_status(int *out) {
    const int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(out, g_staged_status, sizeof(int));
    return e == cudaSuccess ? cudaMemcpyToSymbol(g_staged_status, &zero, sizeof(int)) : e;
}

// ---- PTX wrappers ----------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// announces bytes without arriving
__device__ __forceinline__ void mbar_expect_tx_only(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// global -> this CTA's shared memory; both addresses 16-byte aligned, size a multiple of 16
__device__ __forceinline__ void bulk_copy_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// Programmatic dependent launch: let the next kernel in the stream start its weight-only prologue
// while this one is still running, and wait for the previous kernel's results before touching them.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kSpinLimit; i++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void mma_bf16_16x8x16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                                 uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---- row-sharded GEMV whose epilogue is the all-gather ------------------------------------------------
// Every rank computes the rows [row_base, row_base + M) of Y [B, M_total] and needs all of it.  Instead
// of a collective after the kernel, the CTA stores its finished dot products straight into the Y buffer
// of every rank (plain stores to peer-mapped pointers over NVLink, every thread to all ranks in turn).
// Four counter words per layer and rank make that safe without any other kernel:
//   ready  - each rank adds 1 on every peer when its launch may be written to (its earlier consumers of
//            Y are done: the add comes after the wait for the previous kernel in the stream); a warp
//            checks its own copy (>= world * launch number) before its first remote store;
//   arrive (local) - every CTA adds 1 after its stores; the CTA that brings it to the grid size is the last
//            one of this launch on this GPU and puts it back to zero;
//   done   - that last CTA adds 1 on every peer (release at system scope, cumulative over all CTAs'
//            stores through the arrive counter) and then waits until its own copy shows
//            world * launch number, so whatever runs next on the stream sees the whole of Y.  One
//            system-scope signal per peer and launch, whatever the grids of the ranks are;
//   launches (local) - how often this layer has run; written by the one waiting thread at the end.
// launches and arrive are two consecutive words (PeerSet::launches points at the first).
// Both waits are bounded; on expiry the status word is set (8 = peers not ready, 9 = peers not done)
// and the kernel carries on.
constexpr int kMaxPeers = BHI_MAX_PEERS;

struct PeerSet {
    uint16_t *y[kMaxPeers];
    uint32_t *ready[kMaxPeers];
    uint32_t *done[kMaxPeers];
    uint32_t *launches;
    int world, rank, row_base, m_total;
};

__device__ __forceinline__ void red_release_sys_add(uint32_t *p, uint32_t v) {
    asm volatile("red.release.sys.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_relaxed_sys_add(uint32_t *p, uint32_t v) {
    asm volatile("red.relaxed.sys.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// waits until the counter has reached `target` (wrap-safe); false when a second has passed without it
constexpr uint64_t kPeerWaitNs = 1000ull * 1000ull * 1000ull;
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t ld_relaxed_sys(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool counter_wait_bounded(const uint32_t *p, uint32_t target) {
    if (static_cast<int32_t>(ld_acquire_sys(p) - target) >= 0) return true;
    const uint64_t t0 = global_ns();
    for (uint32_t i = 0; i < kSpinLimit; i++) {            // the iteration bound is a second line of defence
        if (static_cast<int32_t>(ld_relaxed_sys(p) - target) >= 0) {
            asm volatile("fence.acq_rel.sys;" ::: "memory");
            return true;
        }
        if ((i & 15u) == 15u && global_ns() - t0 > kPeerWaitNs) return false;
        __nanosleep(40);
    }
    return false;
}

// a[i] without indexing the array by a register (that would move the whole kernel-parameter struct to
// local memory, accumulators included)
template <class T>
__device__ __forceinline__ T pick(T const (&a)[kMaxPeers], int i) {
    T v = a[0];
#pragma unroll
    for (int r = 1; r < kMaxPeers; r++)
        if (i == r) v = a[r];
    return v;
}

__device__ __forceinline__ uint32_t atom_add_acq_rel_gpu(uint32_t *p, uint32_t v) {
    uint32_t old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// End of an exchange kernel (every thread of the CTA calls it after its stores to the peers).
__device__ __forceinline__ void exchange_finish(const PeerSet &peers, uint32_t launch_no) {
    // The barrier orders every warp's stores before thread 0; its release is cumulative over them, and the
    // last CTA's acquire of the arrive counter, then its release at system scope, carry them to the peers.
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t before = atom_add_acq_rel_gpu(peers.launches + 1, 1u);
        if (before + 1u == gridDim.x) {
            // last CTA of this launch.  The arrival counter goes back to zero for the next launch of the layer,
            // whatever grid that one uses (its CTAs arrive only after this whole grid has completed).
            *reinterpret_cast<volatile uint32_t *>(peers.launches + 1) = 0u;
            // one system-scope fence, then a relaxed add per peer: a release per peer would be a fence per peer, one after
            // the other (7 us more per launch on 8 GPUs than on 4)
            asm volatile("fence.acq_rel.sys;" ::: "memory");
#pragma unroll
            for (int q = 0; q < kMaxPeers; q++)
                if (q < peers.world) red_relaxed_sys_add(peers.done[q], 1u);
            if (!counter_wait_bounded(pick(peers.done, peers.rank), launch_no * peers.world)) atomicExch(&g_staged_status, 9);
            *peers.launches = launch_no;
            __threadfence();
        }
    }
}

// ---- Huffman: folded pair table ---------------------------------------------------------------------
__device__ __forceinline__ uint32_t umad(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// (a & mask) | (b & ~mask) in one logic instruction
__device__ __forceinline__ uint32_t bitselect(uint32_t a, uint32_t b, uint32_t mask) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xE4;" : "=r"(d) : "r"(a), "r"(b), "r"(mask));
    return d;
}

// Resolve one symbol from `known` valid low bits of `v` (other bits zero).  Returns its length, 0
// if the known bits do not determine it.
__device__ __forceinline__ uint32_t resolve_symbol(const HuffTables &t, uint32_t v, uint32_t known, uint32_t &sym) {
    sym = t.lut[0][v & 0xFF];
    if (sym != 255) {
        const uint32_t n = t.len[sym];
        return (n >= 1 && n <= 8 && n <= known) ? n : 0;
    }
    if (known <= 8) return 0;
    sym = t.lut[1][(v >> 8) & 0xFF];
    if (sym == 255) return 0;
    const uint32_t n = t.len[sym];
    return (n >= 9 && n <= known) ? n : 0;
}

// entry: bits 0..3 stream bits consumed, bit 5 single, bit 6 exact, bits 7..14 first exponent,
// bits 16..19 length of the first symbol, bits 23..30 second exponent
template <int kBits = kPairBits>
__device__ __forceinline__ uint32_t pair_entry(const HuffTables &t, uint32_t v) {
    uint32_t s0, s1;
    const uint32_t l0 = resolve_symbol(t, v, kBits, s0);
    if (!l0) return kEntExact;
    const uint32_t l1 = resolve_symbol(t, v >> l0, kBits - l0, s1);
    return l1 ? ((s0 << 7) | (s1 << 23) | (l0 << 16) | (l0 + l1)) : ((s0 << 7) | (l0 << 16) | l0 | kEntSingle);
}

// Where the kCopies copies of entry v live (word index of copy 0): interleaved, so copy c only ever
// touches banks congruent to c mod kCopies.  (Picking the bank from the top index bits instead was
// measured slower: two more integer instructions per lookup cost more than the conflicts they save.)
__device__ __forceinline__ uint32_t pair_slot(uint32_t v) { return v * kCopies; }

__device__ __forceinline__ void build_pair_table(uint32_t *dst, const HuffTables &t, int tid, int nthreads) {
    for (int v = tid; v < kPairEntries; v += nthreads) {
        const uint32_t e = pair_entry(t, v);
        *reinterpret_cast<uint4 *>(dst + pair_slot(v)) = make_uint4(e, e, e, e);
    }
}

// this lane's copy of entry (win & 0xFFF): see pair_slot
__device__ __forceinline__ uint32_t pair_lookup(const uint8_t *smem, const Consts &k, uint32_t win, uint32_t copy_off) {
    return *reinterpret_cast<const uint32_t *>(smem + umad(win & (kPairEntries - 1), k.entry, copy_off));
}

// A code longer than the table index: resolve one symbol with the exact four-table cascade.
// Returns {symbol, length}.  Out of line on purpose: it is rare and must not bloat the loop.
static __device__ __noinline__ uint2 huff_exact_symbol(uint32_t win, const HuffTables *t) {
    const uint32_t s = huff_cascade(*t, win);
    return make_uint2(s, t->len[s]);
}

__device__ __forceinline__ void build_fast_table(uint32_t *fast, const HuffTables &t, int tid, int n) { build_pair_table(fast, t, tid, n); }
__device__ __forceinline__ void build_fast_table(uint32_t *fast, const AnsTables &t, int tid, int n) {
    for (int i = tid; i < (1 << t.bits); i += n) {
        const uint32_t e = __ldg(t.lut + i);
        *reinterpret_cast<uint4 *>(fast + i * kCopies) = make_uint4(e, e, e, e);
    }
}

// ---- host side -------------------------------------------------------------------------------------
bool overlap_launches();     // process-wide switch, see bhi_set_launch_overlap

template <class K>
static int staged_prepare(K kernel, int bytes = kSmemMax, int registers = 0) {
    // Opt in to the large dynamic shared-memory carve-out once per device and kernel.  Keyed by the
    // kernel's address: instantiations that differ only in a non-type argument share their pointer type.
    static std::mutex mu;
    static std::unordered_map<const void *, uint64_t> done;      // kernel -> bit per device
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BHI_ERR_CUDA;
    const void *key = reinterpret_cast<const void *>(kernel);
    std::lock_guard<std::mutex> lock(mu);
    uint64_t &bits = done[key];
    if (!(bits >> dev & 1u)) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(shared memory)");
        if (registers) {                           // as many per thread as the kernel's register shift counts on
            cudaFuncAttributes a;
            e = cudaFuncGetAttributes(&a, kernel);
            if (e != cudaSuccess) return cuda_fail(e, "cudaFuncGetAttributes");
            if (a.numRegs < registers) return fail(BHI_ERR_CUDA, "kernel was compiled with fewer registers than it shifts between its warps");
        }
        bits |= 1ull << dev;
    }
    return BHI_OK;
}

static bool staged_shape_ok(const Layer &L) { return aligned(L.rem, 16) && aligned(L.exp, 16); }


// number of flagged entries of the folded table (0 = every 12-bit window resolves two symbols)
__device__ __forceinline__ uint32_t prepared_flagged(const uint8_t *exact_region) {
    return *reinterpret_cast<const uint32_t *>(exact_region + sizeof(HuffTables));
}

// length of the longest code
__device__ __forceinline__ uint32_t prepared_longest(const uint8_t *exact_region) {
    return *reinterpret_cast<const uint32_t *>(exact_region + sizeof(HuffTables) + 4);
}

// blob = folded pair table (one copy), exact tables with two words behind them (how many folded entries do not resolve two
// symbols, and the length of the longest code; a code of a single symbol is one bit long and leaves half the entries
// unresolved), single-symbol tables, wide pair tables.  The first block makes the first two, the others share the rest.
static __global__ void __launch_bounds__(1024) huffman_prepare_kernel(HuffArgs targs, uint8_t *blob) {
    __shared__ HuffTables tab;
    __shared__ uint32_t flagged, longest;
    if (threadIdx.x == 0) flagged = longest = 0u;
    load_tables(tab, targs, threadIdx.x, blockDim.x);
    __syncthreads();
    if (blockIdx.x > 0) {
        const int first = (blockIdx.x - 1) * blockDim.x + threadIdx.x, step = (gridDim.x - 1) * blockDim.x;
        for (int i = first; i < kSingleBytes / 4; i += step) {
            const uint32_t s = tab.lut[0][(i >> 5) & 63], n = tab.len[s];
            reinterpret_cast<uint32_t *>(blob + kPreparedSingle)[i] = (s << (i < kSingleBytes / 8 ? 7 : 23)) | (n & 31u);
        }
        for (int v = first; v < (1 << kWideBits); v += step)
            reinterpret_cast<uint32_t *>(blob + kPreparedWide)[v] = pair_entry<kWideBits>(tab, v);
        for (int v = first; v < (1 << kWidestBits); v += step)
            reinterpret_cast<uint32_t *>(blob + kPreparedWidest)[v] = pair_entry<kWidestBits>(tab, v);
        return;
    }
    uint32_t mine = 0;
    for (int v = threadIdx.x; v < kPairEntries; v += blockDim.x) {
        const uint32_t e = pair_entry(tab, v);
        reinterpret_cast<uint32_t *>(blob)[v] = e;
        mine += (e & (kEntSingle | kEntExact)) ? 1u : 0u;
    }
    if (mine) atomicAdd(&flagged, mine);
    if (threadIdx.x < 256) atomicMax(&longest, static_cast<uint32_t>(tab.len[threadIdx.x]));
    __syncthreads();
    uint32_t *dst = reinterpret_cast<uint32_t *>(blob + kPairEntries * 4);
    const uint32_t *src = reinterpret_cast<const uint32_t *>(&tab);
    constexpr int kTabWords = static_cast<int>(sizeof(HuffTables) / 4);
    for (int i = threadIdx.x; i < kExactBytes / 4; i += blockDim.x)
        dst[i] = i < kTabWords ? src[i] : (i == kTabWords ? flagged : i == kTabWords + 1 ? longest : 0u);
}

}  // namespace bhi

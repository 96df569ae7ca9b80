// Large-segment kernel of the varlen blocked GEMM on the 5th-generation tensor
// cores: TMA-fed tcgen05.mma with the accumulator in tensor memory.
//
// A persistent CTA (one per SM) walks a static list of work items, an item being a 128-row block of one segment of one head
// (or one 256-column chunk of it).  An item's columns are taken in chunks: 128 wide, or 256 wide in the variant for plain
// scores of long contractions (WIDE), which want the widest instruction.  Roles:
//   warp 0     producer: one lane issues 3-D tiled TMA loads (k, row, head) of a 128 x 64 tile of the first operand and a
//              chunk x 64 tile of the second into a ring of 128-byte-swizzled stages;
//   warp 1     MMA: one lane issues tcgen05.mma (M = 128, K = 16 per instruction) into the next of four 128-column (two
//              256-column) accumulators;
//   last warp  planner: one lane reads the work items ahead of everybody and hands them out through a ring in shared
//              memory (a role that fetched its own would wait for that load at every item);
//   the others groups of four epilogue warps, four groups (two when WIDE); a warp owns 32 rows (the accumulator lanes it may
//              read), a thread one row.  Plain scores: groups take chunks in turn.  Softmax: two groups share an item, its
//              chunks in turn, and meet once to combine the row statistics; the other two have the next item.  So some
//              groups take exponentials while others store or wait for products: with all warps on one item, in step
//              through maximum, exponentials and stores, the special-function unit was busy a quarter of the time.
// A thread reads its row 32 columns at a time (tcgen05.ld), applies the epilogue and writes packed words into its warp's
// strip (32 rows x 128 16-bit or 64 fp32 columns) at the position the row has in global memory modulo one 32-bit word; then
// the warp writes the strip out as row pieces of 256 contiguous bytes, two fully coalesced 128-byte word stores each, with
// odd first and last elements as 16-bit stores.  Wide contiguous row pieces matter: the same data written as 128-byte pieces
// with element-wise ragged edges runs at little more than half the rate.
//
// Epilogues.  Scores: scale and round.  Softmax with N <= 512: the whole row stays in tensor memory; pass 1 takes the
// exponentials against a running reference (the first piece's maximum; moved, with what was written rescaled, only when a
// piece exceeds it by 2^32) and writes them back as fp32 while summing, pass 2 normalises and stores, so the exponential is
// evaluated once per element and the scores never leave the SM.  Softmax with N > 512: the products are computed twice -- a
// first sweep keeps only (reference, sum) per row, a second recomputes each chunk and stores normalised probabilities; the
// second sweep of an item alternates chunk by chunk with the first sweep of the next, all four groups taking chunks of both.
//
// Large batches of short contractions, plain or with rows beyond 512 columns, run on the kernel of independent streams instead
// (blk_scores_umma.cu; the second of the following then takes 757).
//
// Measured against one item at a time with 8 arithmetic and 4 store warps: scores + softmax of 1024 segments of 64..512 rows,
// 16 heads, K = 128: 2054 -> 1532 us; of 512 segments of 16..2048 rows, 4 heads, K = 64 (two sweeps): 872 -> 897 us
// sustained; 2048 products of at most 256 x 256, fp32 out: 57.3 -> 55.5 us; 64 products of 1024..2048 rows and columns,
// K 1024..4096: 845 -> 835 us sustained.  Without its stores the first takes 1230 us, and one sweep and two run at the same
// 2.1-2.3 TB/s: what bounds the softmax is the latency of a chunk through loads, products and registers, then the write rate
// of misaligned rows (4 TB/s alone).  The long contractions (tensor pipe active 66 % in a single launch) move 48 KB from L2
// per 128 x 256 x 64 step, 11 TB/s, half of what that path can do.
//
// Rows of the operand views past the end of a segment belong to its neighbour (or are zero-filled past the end of the
// buffer); they only reach accumulator rows/columns the epilogue never stores, and columns >= N are masked before any row
// reduction.  A warp none of whose rows exist only hands its accumulators back.
//
// Every wait on an mbarrier is bounded: when the bound is hit the kernel records a status code, all roles leave their
// loops, tensor memory is released and the kernel returns.
//
// Replaces upstream sparseBlockedHGEMM_half / _bf16 with the 128 x 128 x 16
// WMMA tile (csrc/cuda/spBlkGEMM.cu:424-817, :866-868) and, fused, the softmax
// kernels (csrc/cuda/spBlkSoftmax.cu:88-269).
#include <cuda.h>

#include <mutex>

#include "blk_device.cuh"
#include "blk_kernels.h"
#include "blk_umma_items.cuh"
#include "blk_umma_ptx.cuh"

namespace {

constexpr int UM_BM = BLK_UMMA_BM;      // 128 rows per work item
constexpr int UM_BK = 64;               // k elements per shared-memory stage (one 128-byte swizzle row)
constexpr int UM_A_BYTES = UM_BM * UM_BK * 2;  // 16 KB
constexpr int UM_PW = 64;                             // 32-bit words of a staged row piece (128 x 16-bit, 64 x fp32)
// Strip row pitch in words: odd, so that the 32 row-owning lanes of a store (same word, consecutive rows) hit 32
// different banks; a row holds UM_PW words plus the half word an odd first element pushes past the end.
constexpr int UM_STRIP_PITCHW = UM_PW + 1;
constexpr int UM_STRIP_BYTES = 32 * UM_STRIP_PITCHW * 4;  // one per warp of the groups
constexpr float UM_LAZY = 32.f;                       // exponent slack before a softmax reference moves
constexpr uint32_t UM_ITEMS = 8;                      // ring of item records

template <bool WIDE>
struct UL {
    static constexpr int GROUPS = WIDE ? 2 : 4;       // of four epilogue warps
    static constexpr int THREADS = 96 + 128 * GROUPS;
    static constexpr int BN = WIDE ? 256 : 128;       // columns of a chunk = of an accumulator
    static constexpr uint32_t NBUF = 512 / BN;
    static constexpr int STAGES = 3;
    static constexpr int STAGE_BYTES = UM_A_BYTES + BN * UM_BK * 2;
    static constexpr int STRIP_OFF = STAGES * STAGE_BYTES;
    static constexpr int BAR_OFF = STRIP_OFF + 4 * GROUPS * UM_STRIP_BYTES;
    static constexpr int SMEM_BYTES = BAR_OFF + 464 + (int)UM_ITEMS * 64;
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

// A work item as the roles see it, in shared memory.
struct __align__(16) Work {
    int64_t cbase;   // element of the output where the item's rows start (head, segment and row block included)
    int32_t rows, N; // rows of the block | first quarter that holds them << 8; columns of the segment
    int32_t ch0, nchunks;  // chunks [ch0, ch0 + nchunks)
    int32_t sweeps;
    int32_t pair;    // chunks of the next item's first sweep, which alternates with this one's second (0: it does not)
    int32_t rowA, rowB, K, views;
    int32_t head;
    int32_t valid;   // 0: nothing follows
    int32_t next_rows, next_N;  // of the item this one pairs with
};
static_assert(sizeof(Work) == 64, "Work is written as four 16-byte vectors");

template <bool SOFT, bool WIDE>
__device__ __forceinline__ void publish(const BlkUmmaParams& p, Work* dst, const BlkUmmaItem& it, int head, uint32_t n,
                                        bool valid, const BlkUmmaItem& nx, bool nx_valid) {
    constexpr int BN = UL<WIDE>::BN;
    Work w{};
    if (valid) {
        w.rows = item_rows(it, n);
        w.cbase = (int64_t)head * p.Dout + it.offC + (int64_t)it.tm * UM_BM * it.N;
        w.N = it.N;
        w.ch0 = it.ch0 * (256 / BN);  // (the plan counts chunks of 256 columns)
        w.nchunks = (it.N + BN - 1) / BN - w.ch0;
        if (it.nch) w.nchunks = min(w.nchunks, it.nch * (256 / BN));
        w.sweeps = SOFT && it.N > 512 ? 2 : 1;
        w.pair = w.sweeps == 2 && nx_valid && nx.N > 512 ? (nx.N + BN - 1) / BN : 0;
        w.rowA = it.rowA - 32 * (w.rows >> 8);
        w.rowB = it.rowB;
        w.K = it.K;
        w.views = it.views;
        w.head = head;
        w.valid = 1;
        w.next_rows = item_rows(nx, n + 1u);
        w.next_N = nx.N;
    }
    *dst = w;
}

// The chunks of item n in the order in which they are loaded, multiplied and consumed: its first sweep (unless that ran
// alongside the item before), then the storing chunks, each followed by a first-sweep chunk of the next item when the two
// pair up.  f(next, ch, first): chunk ch of this item or the next, in its first sweep or storing; false stops.
template <typename F>
__device__ __forceinline__ void chunk_order(int ch0, int nchunks, int sweeps, int pair, bool pre, F f) {
    const int first = sweeps == 2 && !pre ? nchunks : 0;
    const int rest = pair ? 2 * max(nchunks, pair) : nchunks;
#pragma unroll 1
    for (int i = 0; i < first + rest; ++i) {
        const int t = i - first;
        const bool nx = pair && t >= 0 && (t & 1);
        const int ch = t < 0 ? i : pair ? t >> 1 : t;
        if (t >= 0 && ch >= (nx ? pair : nchunks)) continue;  // the other item has more chunks
        if (!f(nx, t < 0 || nx ? ch : ch0 + ch, t < 0 || nx)) return;
    }
}

// Predicated global stores as single instructions (no branch around them).
__device__ __forceinline__ void stg_b32_if(void* p, uint32_t v, bool ok) {
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n @q st.global.b32 [%0], %1;\n}\n" ::"l"(p), "r"(v), "r"((int)ok)
                 : "memory");
}
__device__ __forceinline__ void stg_b16_if(void* p, uint32_t v, bool ok) {
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n @q st.global.b16 [%0], %1;\n}\n" ::"l"(p), "h"((uint16_t)v),
                 "r"((int)ok)
                 : "memory");
}
__device__ __forceinline__ uint32_t lds_b32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(v) : "r"(addr));
    return v;
}

// A warp writes the piece in its strip to the output: element g0 is the first of its first row, row k starts N elements
// further each; `rows` rows of pcols columns exist.  halves: some row starts or ends on half a word.
template <bool OUT32>
__device__ __forceinline__ void store_strip(uint32_t strip, void* out, int64_t g0, int N, int pcols, int rows, bool halves,
                                            int lane) {
    constexpr int BATCH = 8;  // rows whose words are in registers at a time
    // lane l carries words l and l + 32 of a row: two stores of 128 contiguous bytes per row
    const uint32_t rbase = strip + 4u * lane;
    uint32_t v[BATCH][2];
    auto fetch = [&](int kb) {
#pragma unroll
        for (int k = 0; k < BATCH; ++k)
#pragma unroll
            for (int i = 0; i < 2; ++i) v[k][i] = lds_b32(rbase + (uint32_t)(kb + k) * (UM_STRIP_PITCHW * 4) + 128u * i);
    };
    if (rows == 32 && pcols == (OUT32 ? UM_PW : 2 * UM_PW)) {
        // A whole piece (the common case), with as few instructions per row as it takes.  Rows go by twos: row 2 j starts j * two
        // words past the word of g0, as far into its first word as g0 (`even`), and row 2 j + 1 starts `one` words further and is
        // `odd` elements into its word.  (A row may have 2^30 columns: nothing but a row's own length fits 32 bits.)  Words 1..63
        // of a row are whole; word 0 is whole when the row starts on an even element (its upper half goes out below
        // otherwise, and so does the lower half of word 64).
        const uint32_t even = OUT32 ? 0u : (uint32_t)(g0 & 1), one = OUT32 ? (uint32_t)N : (even + (uint32_t)N) >> 1;
        const uint32_t odd = OUT32 ? 0u : (even + (uint32_t)N) & 1u;
        const int64_t two = OUT32 ? 2 * (int64_t)N : N;
        uint32_t* w0 = static_cast<uint32_t*>(out) + (OUT32 ? g0 : g0 >> 1) + lane;
#pragma unroll 1
        for (int kb = 0; kb < 32; kb += BATCH) {
            fetch(kb);
#pragma unroll
            for (int k = 0; k < BATCH; ++k) {
                uint32_t* wp = w0 + (k & 1 ? one : 0u);
                if (OUT32) asm volatile("st.global.b32 [%0], %1;\n" ::"l"(wp), "r"(v[k][0]) : "memory");
                else stg_b32_if(wp, v[k][0], lane >= (int)(k & 1 ? odd : even));
                asm volatile("st.global.b32 [%0], %1;\n" ::"l"(wp + 32), "r"(v[k][1]) : "memory");
                if (k & 1) w0 += two;
            }
        }
    } else {
#pragma unroll 1
        for (int kb = 0; kb < rows; kb += BATCH) {
            fetch(kb);
#pragma unroll
            for (int k = 0; k < BATCH; ++k) {
                const int64_t gr = g0 + (int64_t)(kb + k) * N;
                const int pr = OUT32 ? 0 : (int)(gr & 1);
                // whole words of the piece: [pr, (pr + pcols) / 2) for 16-bit elements, [0, pcols) for fp32
                const int wl = kb + k < rows ? (OUT32 ? pcols : (pr + pcols) >> 1) : 0;
                uint32_t* wp = static_cast<uint32_t*>(out) + (OUT32 ? gr : gr >> 1) + lane;
#pragma unroll
                for (int i = 0; i < 2; ++i) stg_b32_if(wp + 32 * i, v[k][i], lane + 32 * i >= pr && lane + 32 * i < wl);
            }
        }
    }
    if (!OUT32 && halves) {
        // half words at the ends: lane k the odd first element of row k, then the last element of row k when the
        // piece ends on half a word
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const bool tail = t != 0;
            const int64_t gr = g0 + (int64_t)lane * N;
            const int pr = (int)(gr & 1);
            const int endh = pr + pcols;                 // half words [pr, endh) of the row's words are the piece
            const int wi = tail ? (endh >> 1) : 0;       // word that is only half inside the piece
            const bool need = lane < rows && (tail ? (endh & 1) != 0 : pr != 0);
            const uint32_t word = lds_b32(strip + (uint32_t)lane * (UM_STRIP_PITCHW * 4) + 4u * (need ? wi : 0));
            unsigned char* dst = static_cast<unsigned char*>(out) + (gr - pr) * 2 + 4 * (int64_t)wi + (tail ? 0 : 2);
            stg_b16_if(dst, tail ? (word & 0xffffu) : (word >> 16), need);
        }
    }
}

template <typename Tag, bool OUT32, bool SOFT, bool WIDE>
__global__ void __launch_bounds__(UL<WIDE>::THREADS, 1)
blk_gemm_umma_kernel(const BlkUmmaParams p, const __grid_constant__ UmMaps maps) {
    static_assert(!(SOFT && WIDE), "the fused softmax keeps up to four 128-column chunks of a row");
    using L = UL<WIDE>;
    constexpr int BN = L::BN;
    constexpr uint32_t GROUPS = L::GROUPS;
    constexpr uint32_t NBUF = L::NBUF;
    extern __shared__ __align__(1024) unsigned char um_smem_raw[];  // the swizzled tiles need a 1024-byte aligned base
    unsigned char* smem = um_smem_raw;
    if (blk_smem_u32(smem) & 1023u) {  // cannot happen with the alignment above; checked because the swizzle relies on it
        if (threadIdx.x == 0) atomicCAS(p.status, 0, 9);
        return;
    }
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
    // [0..] stage full, [4..] stage empty, [8..] accumulator free, [12 + 4 g + i] chunk i mod 4 of group g ready,
    // [28..] item record written, [36..] read by all, [44 + 4 (g / 2) + q] rendezvous of quarter q's warps of two groups,
    // [52 + q] of all groups
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 56);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 57);
    Work* const ring = reinterpret_cast<Work*>(bars + 58);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_u32 = blk_smem_u32(smem);
    const uint32_t bar0 = blk_smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (4 + s); };
    auto tempty_bar = [&](uint32_t b) { return bar0 + 8u * (8u + b); };
    auto ready_bar = [&](uint32_t g, uint32_t k) { return bar0 + 8u * (12u + 4u * g + (k & 3u)); };
    auto item_full = [&](uint32_t n) { return bar0 + 8u * (28u + n % UM_ITEMS); };
    auto item_empty = [&](uint32_t n) { return bar0 + 8u * (36u + n % UM_ITEMS); };
    // The group that takes a chunk.  Scores: in turn.  Softmax of a resident row: two groups per item, in turn within it.
    // Two sweeps: in turn, shifted by one every four chunks, so that a group gets first-sweep and storing chunks alternately
    // (a storing chunk takes half as long again; two groups with the one kind and two with the other waited for each other
    // a quarter of the time).
    auto group_of = [&](uint32_t slot, uint32_t n, int ch, int sweeps) {
        if (!SOFT) return slot % GROUPS;
        return sweeps == 2 ? (slot + (slot >> 2)) & 3u : 2u * (n & 1u) + (((uint32_t)ch + (n >> 1)) & 1u);
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < 4; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
            mbar_init(tempty_bar(s), 4);  // the warps of the group that consumed the chunk
        }
        for (uint32_t i = 0; i < 16; ++i) mbar_init(ready_bar(i >> 2, i), 1);
        for (uint32_t i = 0; i < 12; ++i) mbar_init(bar0 + 8u * (44u + i), i < 8 ? 2 : 4);
        for (uint32_t i = 0; i < UM_ITEMS; ++i) {
            mbar_init(item_full(i), 1);
            mbar_init(item_empty(i), 2 + 4 * GROUPS);  // producer, MMA, the groups
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(blk_smem_u32(tmem_slot)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    blk_grid_ready();
    blk_grid_wait();
    const uint32_t lim = p.spin_limit ? p.spin_limit : BLK_UMMA_SPIN_LIMIT;
    auto item_wait = [&](uint32_t n) { return mbar_wait(item_full(n), (n / UM_ITEMS) & 1u, abort_flag, 11, lim); };

    if (warp == 0) {
        // ---------------- producer (one lane) ----------------
        if (elect_one() && !p.stall) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true, pre = false;
#pragma unroll 1
            for (uint32_t n = 0; ok; ++n) {
                if (!item_wait(n)) break;
                const Work& wk = ring[n % UM_ITEMS];
                if (!wk.valid) break;
                const int pair = wk.pair;
                if (pair && !item_wait(n + 1u)) break;
                chunk_order(wk.ch0, wk.nchunks, wk.sweeps, pair, pre, [&](bool next, int ch, bool) -> bool {
                    const Work& k = ring[(next ? n + 1u : n) % UM_ITEMS];
                    // coordinates (k, row, head), or (k, head, row) for a token-major operand
                    const int rA = k.rowA, rB = k.rowB + ch * BN, hd = k.head, K = k.K;
                    const CUtensorMap *mapA = &maps.a[k.views & 255], *mapB = &maps.b[k.views >> 8];
#pragma unroll 1
                    for (int kk = 0; kk < K; kk += UM_BK) {
                        if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, 1, lim)) { ok = false; return false; }
                        const uint32_t sA = smem_u32 + stage * L::STAGE_BYTES, sB = sA + UM_A_BYTES;
                        mbar_expect_tx(full_bar(stage), L::STAGE_BYTES);
                        tma_load_3d(sA, mapA, full_bar(stage), kk, p.head_firstA ? hd : rA, p.head_firstA ? rA : hd);
                        tma_load_3d(sB, mapB, full_bar(stage), kk, p.head_firstB ? hd : rB, p.head_firstB ? rB : hd);
                        if (++stage == L::STAGES) { stage = 0; phase ^= 1u; }
                    }
                    return true;
                });
                pre = pair != 0;
                mbar_arrive(item_empty(n));
            }
        }
    } else if (warp == 2 + 4 * (int)GROUPS) {
        // ---------------- planner (one lane): the records of the items ----------------
        if (elect_one() && !p.stall) {
            BlkUmmaItem it{}, nx{};  // records n and n + 1
            int head = 0, nhead = 0;
            bool have = fetch_item(p, 0, gridDim.x, blockIdx.x, it, head),
                 nhave = have && fetch_item(p, 1, gridDim.x, blockIdx.x, nx, nhead);
#pragma unroll 1
            for (uint32_t n = 0;; ++n) {
                if (!mbar_wait(item_empty(n), ((n / UM_ITEMS) & 1u) ^ 1u, abort_flag, 12, lim)) break;
                publish<SOFT, WIDE>(p, ring + n % UM_ITEMS, it, head, n, have, nx, nhave);
                mbar_arrive(item_full(n));  // release: the record is visible to whoever sees the phase end
                if (!have) break;
                it = nx;
                head = nhead;
                have = nhave;
                if (nhave) nhave = fetch_item(p, n + 2u, gridDim.x, blockIdx.x, nx, nhead);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issue (one lane) ----------------
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0, slot = 0, counts = 0;  // chunks so far; of the groups, modulo 4, a byte each
            bool ok = true, pre = false;
            const uint32_t idesc0 = instr_desc(p.bf16, 0, SOFT && p.scale < 0.f);
#pragma unroll 1
            for (uint32_t n = 0; ok; ++n) {
                if (!item_wait(n)) break;
                const Work& wk = ring[n % UM_ITEMS];
                const int ch0 = wk.ch0, nchunks = wk.nchunks, sweeps = wk.sweeps, pair = wk.pair, N = wk.N, K = wk.K;
                if (!wk.valid) break;
                int N2 = 0, K2 = 0;
                if (pair) {
                    if (!item_wait(n + 1u)) break;
                    N2 = ring[(n + 1u) % UM_ITEMS].N;
                    K2 = ring[(n + 1u) % UM_ITEMS].K;
                }
                mbar_arrive(item_empty(n));
                chunk_order(ch0, nchunks, sweeps, pair, pre, [&](bool next, int ch, bool) -> bool {
                    // the chunk's products into the next accumulator
                    const uint32_t buf = slot % NBUF, grp = group_of(slot, n, ch, sweeps);
                    const uint32_t ready = ready_bar(grp, counts >> (8u * grp));
                    const int ncols = min((next ? N2 : N) - ch * BN, BN);
                    const uint32_t idesc = idesc0 | ((uint32_t)((ncols + 15) >> 4) << 18);  // columns in units of 16
                    const uint32_t d_tmem = tmem_base + buf * (uint32_t)BN;
                    if (!mbar_wait(tempty_bar(buf), ((slot / NBUF) & 1u) ^ 1u, abort_flag, 2, lim)) { ok = false; return false; }
#pragma unroll 1
                    for (int krem = next ? K2 : K, kb = 0; krem > 0; krem -= UM_BK, ++kb) {
                        const uint32_t sA = smem_u32 + stage * L::STAGE_BYTES;
                        const uint64_t da = smem_desc_sw128(sA), db = smem_desc_sw128(sA + UM_A_BYTES);
                        if (!mbar_wait(full_bar(stage), phase, abort_flag, 3, lim)) { ok = false; return false; }
                        tc_fence_after();
                        // steps of 16 along k in this block: all four, or as many as reach the end of a short last block
                        // (the tensor map fills what lies past K with zeros)
                        if (krem > UM_BK - 16) {
#pragma unroll
                            for (int j = 0; j < UM_BK / 16; ++j)
                                tc_mma_f16(d_tmem, da + (uint64_t)(2 * j), db + (uint64_t)(2 * j), idesc, j ? 1u : (uint32_t)kb);
                        } else {
#pragma unroll 1
                            for (int j = 0; 16 * j < krem; ++j)
                                tc_mma_f16(d_tmem, da + (uint64_t)(2 * j), db + (uint64_t)(2 * j), idesc, (uint32_t)(kb | j));
                        }
                        tc_commit(empty_bar(stage));  // stage reusable once these products have read it
                        if (++stage == L::STAGES) { stage = 0; phase ^= 1u; }
                    }
                    tc_commit(ready);
                    ++slot;
                    counts = (counts + (1u << (8u * grp))) & 0x03030303u;
                    return true;
                });
                pre = pair != 0;
            }
        }
    } else {
        // ---------------- epilogue: groups of four warps ----------------
        const int q = warp & 3;
        const uint32_t grp = (uint32_t)(warp - 2) >> 2;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        const uint32_t strip = smem_u32 + L::STRIP_OFF + (uint32_t)(warp - 2) * UM_STRIP_BYTES;
        const uint32_t srow = strip + (uint32_t)lane * (UM_STRIP_PITCHW * 4);
        const float sl = SOFT ? fabsf(p.scale) * BLK_LOG2E : p.scale;  // a negative softmax scale is applied by the MMA (negated A)
        const float2 sl2 = make_float2(sl, sl);
        constexpr int PC = OUT32 ? UM_PW : 2 * UM_PW;  // columns of a staged piece
        uint32_t slot = 0, mychunks = 0, meetings = 0, assemblies = 0;
        bool ok = true, pre = false;

        auto chunk_wait = [&]() -> bool {
            const bool good = mbar_wait(ready_bar(grp, mychunks), (mychunks >> 2) & 1u, abort_flag, 4, lim);
            ++mychunks;
            tc_fence_after();
            return good;
        };
        auto release = [&](uint32_t buf) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty_bar(buf));
        };
        // f(values, unit) for the 32-column units of [col, col + 32 units) of the accumulators; loaded() after the last load.
        // (Four warps per scheduler hide a load's latency; a second buffer of values would not fit their registers.)
        auto each_unit = [&](uint32_t col, int units, auto f, auto loaded) {
#pragma unroll 1
            for (int u = 0; u < units; ++u) {
                uint32_t r[32];
                tc_ld32_nowait(col + 32u * u, r);
                tc_ld_wait(r);
                if (u == units - 1) loaded();
                f(r, u);
            }
        };
        // Columns [c0, c0 + cols) of this warp's rows (the first starts at element cbase), from accumulator columns col on,
        // through xform (two values at a time) to the output; loaded() after the last load.
        auto put = [&](uint32_t col, int c0, int cols, int64_t cbase, int rows, int N, bool anyodd, auto xform, auto loaded) {
#pragma unroll 1
            for (int pc = 0; pc < cols; pc += PC) {
                const int pcols = min(PC, cols - pc);
                const int64_t g0 = cbase + c0 + pc;
                const uint32_t par = OUT32 ? 0u : (uint32_t)((g0 + (int64_t)lane * N) & 1);
                uint32_t prev = 0;
                each_unit(col + (uint32_t)pc, (pcols + 31) >> 5,
                          [&](const uint32_t (&r)[32], int u) {
                              if constexpr (OUT32) {
#pragma unroll
                                  for (int i = 0; i < 32; i += 2) {
                                      const float2 v = xform(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])));
                                      blk_sts_f32(srow + 128u * u + 4 * i, v.x);
                                      blk_sts_f32(srow + 128u * u + 4 * i + 4, v.y);
                                  }
                              } else {
                                  uint32_t w[16];
#pragma unroll
                                  for (int i = 0; i < 16; ++i) {
                                      const float2 v = xform(make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])));
                                      w[i] = BlkCvt<Tag>::pack2(v.x, v.y);
                                  }
                                  const uint32_t a = srow + 64u * u;
                                  if (!anyodd) {
#pragma unroll
                                      for (int i = 0; i < 16; ++i) blk_sts_b32(a + 4 * i, w[i]);
                                  } else {
                                      // a row that starts on an odd element is shifted by half a word
#pragma unroll
                                      for (int i = 0; i < 16; ++i) {
                                          blk_sts_b32(a + 4 * i, __funnelshift_l(prev, w[i], par * 16u));
                                          prev = w[i];
                                      }
                                  }
                              }
                          },
                          [&]() { if (pc + PC >= cols) loaded(); });
                if (!OUT32 && anyodd) blk_sts_b32(srow + 64u * (uint32_t)((pcols + 31) >> 5), prev >> 16);
                __syncwarp();
                store_strip<OUT32>(strip, p.C, g0, N, pcols, rows, anyodd || (pcols & 1), lane);
                __syncwarp();
            }
        };
        auto mask_unit = [](uint32_t (&r)[32], int lim_) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (i >= lim_) r[i] = 0xff800000u;  // -inf
        };
        // Softmax, running over the units of a row that this warp has: reference and sum of exp2((x - reference) sl).
        float ref = -INFINITY, sum = 0.f, off = 0.f;
        // Rendezvous with the warps of the other groups that share the item's rows (the other of a pair, or all four):
        // mbarriers, bounded like every wait.
        auto meet = [&](bool all) -> bool {
            const uint32_t bar = bar0 + 8u * (all ? 52u + (uint32_t)q : 44u + 4u * (grp >> 1) + (uint32_t)q);
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
            return mbar_wait(bar, (all ? assemblies++ : meetings++) & 1u, abort_flag, 8, lim);
        };
        // Reference and sum of the whole row, through the strips (free at that time); false when another gave up.
        auto combine = [&](bool all, float& m, float& l) -> bool {
            const uint32_t base = strip - (all ? grp : grp & 1u) * (4u * UM_STRIP_BYTES) + 8u * lane;
            blk_sts_f32x2(strip + 8u * lane, ref, sum);
            if (!meet(all)) return false;
            float r[4], t[4];
            m = -INFINITY;
#pragma unroll
            for (uint32_t g = 0; g < 4; ++g) {
                const uint32_t at = base + (all || g < 2 ? g : 0u) * (4u * UM_STRIP_BYTES);
                r[g] = __uint_as_float(lds_b32(at));
                t[g] = __uint_as_float(lds_b32(at + 4));
                m = fmaxf(m, r[g]);
            }
            l = 0.f;
#pragma unroll
            for (uint32_t g = 0; g < 4; ++g)
                if ((all || g < 2) && r[g] != -INFINITY) l += t[g] * blk_exp2((r[g] - m) * sl);
            return meet(all);  // everybody has read: the strips may be written
        };
        // New reference for a unit; true when some row's has moved (f: what its earlier exponentials are to be multiplied by)
        auto unit_ref = [&](const uint32_t (&r)[32], float& f) -> bool {
            float m4[4] = {ref, __uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2])};
#pragma unroll
            for (int i = 0; i < 32; i += 8)
#pragma unroll
                for (int e = 0; e < 4; ++e) m4[e] = blk_max3(m4[e], __uint_as_float(r[i + 2 * e]), __uint_as_float(r[i + 2 * e + 1]));
            const float m = fmaxf(blk_max3(m4[0], m4[1], m4[2]), m4[3]);
            const bool move = (m - ref) * sl > UM_LAZY;  // always at the first unit (ref = -inf)
            if (!__any_sync(0xffffffffu, move)) return false;
            f = move ? blk_exp2((ref - m) * sl) : 1.f;
            if (move) ref = m;
            return true;
        };
        // exponentials of a unit in place, added to the sum
        auto unit_exp = [&](uint32_t (&r)[32]) {
            const float nm = ref == -INFINITY ? 0.f : -ref * sl;
            const float2 nm2 = make_float2(nm, nm);
            float2 s2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
                float2 t = blk_fma2(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), sl2, nm2);
                t.x = blk_exp2(t.x);
                t.y = blk_exp2(t.y);
                s2[(i >> 1) & 1] = blk_add2(s2[(i >> 1) & 1], t);
                r[i] = __float_as_uint(t.x);
                r[i + 1] = __float_as_uint(t.y);
            }
            sum += (s2[0].x + s2[0].y) + (s2[1].x + s2[1].y);
        };

#pragma unroll 1
        for (uint32_t n = 0; ok; ++n) {
            if (!item_wait(n)) break;
            const Work& wk = ring[n % UM_ITEMS];
            const int rec_rows = wk.rows, N = wk.N, ch0 = wk.ch0, nchunks = wk.nchunks, sweeps = wk.sweeps, pair = wk.pair;
            const int next_rows = wk.next_rows, next_N = wk.next_N, valid = wk.valid;
            const int r0 = (q - (rec_rows >> 8)) * 32;  // row of the block that this warp's first lane holds
            const int64_t cbase = wk.cbase + (int64_t)r0 * N;
            __syncwarp();
            if (lane == 0) mbar_arrive(item_empty(n));
            if (!valid) break;
            const int rows = min((rec_rows & 255) - r0, 32);
            const bool here = r0 >= 0 && rows > 0;  // some of this warp's rows exist
            // 16-bit rows that start on an odd element need the half-word shift while staging (chunks and pieces start
            // on even columns, so a row's parity is the same for all of them)
            const bool anyodd = !OUT32 && __any_sync(0xffffffffu, (int)((cbase + (int64_t)lane * N) & 1));
            if constexpr (SOFT) {
                if (sweeps == 1) {
                    if ((n & 1u) == grp >> 1) {
                        // the whole row resident: chunk k in accumulator (slot + k) mod NBUF; this warp has every other one
                        const int k0 = (int)((grp ^ (n >> 1)) & 1u);
                        ref = -INFINITY;
                        sum = 0.f;
#pragma unroll 1
                        for (int k = k0; k < nchunks; k += 2) {
                            if (!chunk_wait()) { ok = false; break; }
                            const uint32_t buf = (slot + (uint32_t)k) % NBUF;
                            if (!here) { release(buf); continue; }
                            const int cols = min(N - k * BN, BN);
                            const uint32_t col = lane_addr + buf * (uint32_t)BN;
                            each_unit(col, (cols + 31) >> 5,
                                      [&](uint32_t (&r)[32], int u) {
                                          if (32 * u + 32 > cols) mask_unit(r, cols - 32 * u);
                                          float f;
                                          if (unit_ref(r, f) && (k > k0 || u)) {
                                              // a reference moved far: what this warp has written is rescaled
                                              sum *= f;
#pragma unroll 1
                                              for (int c = k0 * BN; c < k * BN + 32 * u; c += 16) {
                                                  if (((c / BN) ^ k0) & 1) continue;  // the other warp's chunk
                                                  uint32_t o[16];
                                                  const uint32_t at = lane_addr + ((slot + (uint32_t)(c / BN)) % NBUF) * (uint32_t)BN + (uint32_t)(c % BN);
                                                  tc_wait_st();
                                                  tc_ld16(at, o);
#pragma unroll
                                                  for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
                                                  tc_st16(at, o);
                                              }
                                          }
                                          unit_exp(r);
                                          tc_st32(col + 32u * u, r);
                                      },
                                      []() {});
                        }
                        if (!ok) break;
                        if (here && nchunks > k0) {
                            tc_wait_st();
                            float m = ref, l = sum;
                            if (nchunks > 1 && !combine(false, m, l)) { ok = false; break; }
                            const float inv = __frcp_rn(l) * (nchunks > 1 ? blk_exp2((ref - m) * sl) : 1.f);
                            const float2 inv2 = make_float2(inv, inv);
#pragma unroll 1
                            for (int k = k0; k < nchunks; k += 2) {
                                const uint32_t buf = (slot + (uint32_t)k) % NBUF;
                                put(lane_addr + buf * (uint32_t)BN, k * BN, min(N - k * BN, BN), cbase, rows, N, anyodd,
                                    [&](float2 v) { return blk_mul2(v, inv2); }, [&]() { release(buf); });
                            }
                        }
                    }
                    slot += (uint32_t)nchunks;
                } else {
                    // first sweep of this item (unless it ran alongside the item before), then its storing chunks
                    // alternating with the first sweep of the next item
                    const int nr0 = (q - (next_rows >> 8)) * 32;
                    const bool next_here = nr0 >= 0 && nr0 < (next_rows & 255);
                    bool fresh = !pre;  // the first sweep of this item is still to be finished
                    if (fresh) {
                        ref = -INFINITY;
                        sum = 0.f;
                    }
                    auto statistics = [&]() -> bool {
                        // exp2(x sl + off) = exp2((x - m) sl) / l: no multiply after the exponential
                        float m, l;
                        if (!combine(true, m, l)) return false;
                        off = -m * sl - __log2f(l);
                        return true;
                    };
                    float off_now = off;
                    chunk_order(ch0, nchunks, sweeps, pair, pre, [&](bool next, int ch, bool first) -> bool {
                        if (fresh && !(first && !next)) {
                            fresh = false;
                            if (here && !statistics()) { ok = false; return false; }
                            off_now = off;
                        }
                        if (!fresh && next && ch == 0) {
                            ref = -INFINITY;
                            sum = 0.f;
                        }
                        const uint32_t buf = slot % NBUF, owner = group_of(slot, n, ch, 2);
                        ++slot;
                        if (owner != grp) return true;
                        if (!chunk_wait()) { ok = false; return false; }
                        const int cols = min((next ? next_N : N) - ch * BN, BN);
                        const uint32_t col = lane_addr + buf * (uint32_t)BN;
                        if (!(next ? next_here : here)) { release(buf); return true; }
                        if (first) {
                            each_unit(col, (cols + 31) >> 5,
                                      [&](uint32_t (&r)[32], int u) {
                                          if (32 * u + 32 > cols) mask_unit(r, cols - 32 * u);
                                          float f;
                                          if (unit_ref(r, f)) sum *= f;
                                          unit_exp(r);
                                      },
                                      [&]() { release(buf); });
                        } else {
                            const float2 off2 = make_float2(off_now, off_now);
                            put(col, ch * BN, cols, cbase, rows, N, anyodd,
                                [&](float2 v) {
                                    const float2 t = blk_fma2(v, sl2, off2);
                                    return make_float2(blk_exp2(t.x), blk_exp2(t.y));
                                },
                                [&]() { release(buf); });
                        }
                        return true;
                    });
                    if (ok && pair && next_here && !statistics()) ok = false;
                    pre = pair != 0;
                }
            } else {
#pragma unroll 1
                for (int k = 0; k < nchunks; ++k, ++slot) {
                    if (slot % GROUPS != grp) continue;
                    const uint32_t buf = slot % NBUF;
                    const int c0 = (ch0 + k) * BN;
                    if (!chunk_wait()) { ok = false; break; }
                    if (!here) { release(buf); continue; }
                    put(lane_addr + buf * (uint32_t)BN, c0, min(N - c0, BN), cbase, rows, N, anyodd,
                        [&](float2 v) { return blk_mul2(v, sl2); }, [&]() { release(buf); });
                }
            }
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    wait_report(abort_flag, p.status);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512));
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    return fn;
}

template <typename Tag, bool OUT32, bool SOFT, bool WIDE>
cudaError_t launch(const BlkUmmaParams& p, const UmMaps& maps, int sms, cudaStream_t st) {
    auto kern = blk_gemm_umma_kernel<Tag, OUT32, SOFT, WIDE>;
    cudaError_t e = blk_func_smem(reinterpret_cast<const void*>(kern), UL<WIDE>::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const int64_t total = (int64_t)p.num_items * p.H;
    const dim3 grid((unsigned)(total < sms ? total : sms)), block(UL<WIDE>::THREADS);
    return blk_launch(total <= (WIDE ? 4 : 24) * (int64_t)sms, kern, grid, block, UL<WIDE>::SMEM_BYTES, st, p, maps);
}

}  // namespace

// Encoded maps are remembered: a map depends only on the arguments below (never on the memory it describes), and a
// plan is run many times on the same buffers, so the driver's encoder is called once per distinct view.
namespace {
struct MapKey {
    const void* base; int64_t K, H, rows, row_stride, head_stride; int bf16, box_k, box_rows;
    bool operator==(const MapKey& o) const {
        return base == o.base && K == o.K && H == o.H && rows == o.rows && row_stride == o.row_stride &&
               head_stride == o.head_stride && bf16 == o.bf16 && box_k == o.box_k && box_rows == o.box_rows;
    }
};
struct MapSlot { MapKey key; CUtensorMap map; int head_first; uint64_t stamp; bool used; };
constexpr int MAP_SLOTS = 64;
MapSlot g_map_slots[MAP_SLOTS];
uint64_t g_map_clock = 0;
std::mutex g_map_mu;
}  // namespace

bool blk_make_row_map(CUtensorMap_st* map, const void* base, int bf16, int64_t K, int64_t H, const BlkOperandLayout& lay,
                      int box_k, int box_rows, int* head_first) {
    EncodeTiledFn fn = encode_fn();
    if (!fn || lay.rows <= 0 || H <= 0) return false;
    if (lay.row_stride % 8 || lay.head_stride % 8 || lay.row_stride < K) return false;  // 16-byte strides
    const MapKey key{base, K, H, lay.rows, lay.row_stride, lay.head_stride, bf16, box_k, box_rows};
    {
        std::lock_guard<std::mutex> g(g_map_mu);
        for (MapSlot& sl : g_map_slots)
            if (sl.used && sl.key == key) {
                sl.stamp = ++g_map_clock;
                *map = sl.map;
                *head_first = sl.head_first;
                return true;
            }
    }
    const bool hf = lay.head_stride < lay.row_stride;  // token-major: heads are the closer dimension
    *head_first = hf ? 1 : 0;
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)(hf ? H : lay.rows), (cuuint64_t)(hf ? lay.rows : H)};
    const cuuint64_t strides[2] = {(cuuint64_t)(hf ? lay.head_stride : lay.row_stride) * 2,
                                   (cuuint64_t)(hf ? lay.row_stride : lay.head_stride) * 2};
    const cuuint32_t box[3] = {(cuuint32_t)box_k, (cuuint32_t)(hf ? 1 : box_rows), (cuuint32_t)(hf ? box_rows : 1)};
    const cuuint32_t estr[3] = {1, 1, 1};
    auto encode = [&]() {
        return fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims,
                  strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    if (!encode()) {
        // The encoder needs a current context, and a thread that has made no other runtime call yet (an autograd worker)
        // has none: selecting its device again makes the primary context current.
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess || !encode()) return false;
    }
    std::lock_guard<std::mutex> g(g_map_mu);
    MapSlot* victim = &g_map_slots[0];
    for (MapSlot& sl : g_map_slots) {
        if (!sl.used) { victim = &sl; break; }
        if (sl.stamp < victim->stamp) victim = &sl;
    }
    victim->key = key;
    victim->map = *map;
    victim->head_first = *head_first;
    victim->stamp = ++g_map_clock;
    victim->used = true;
    return true;
}

// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) once per kernel and device instead of before every launch.
cudaError_t blk_func_smem(const void* kern, int bytes) {
    constexpr int SLOTS = 256;
    static struct { const void* kern; int dev; } done[SLOTS];
    static int ndone = 0;
    static std::mutex mu;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> g(mu);
        for (int i = 0; i < ndone; ++i)
            if (done[i].kern == kern && done[i].dev == dev) return cudaSuccess;
    }
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> g(mu);
    if (ndone < SLOTS) { done[ndone].kern = kern; done[ndone].dev = dev; ++ndone; }
    return cudaSuccess;
}

// The maps of a launch are remembered as a set under everything they depend on (buffers, strip lengths, views,
// layouts): a plan is run many times on a few sets of buffers, and encoding up to 48 maps costs more than the launch.
namespace {
struct LaunchKey {
    const void *a, *b;
    int64_t Da, Db, H;
    int na, nb, bf16, ga, gb, box_a, box_b;
    BlkOperandLayout layA, layB;
    BlkUmmaView va[BLK_UMMA_VIEWS], vb[BLK_UMMA_VIEWS];
};
struct LaunchSlot { LaunchKey key; UmMaps maps; int hfA, hfB; uint64_t stamp; bool used; };
constexpr int LAUNCH_SLOTS = 8;
LaunchSlot g_launch_slots[LAUNCH_SLOTS];
uint64_t g_launch_clock = 0;
std::mutex g_launch_mu;
bool same_key(const LaunchKey& x, const LaunchKey& y) {
    if (x.a != y.a || x.b != y.b || x.Da != y.Da || x.Db != y.Db || x.H != y.H || x.na != y.na || x.nb != y.nb ||
        x.bf16 != y.bf16 || x.box_a != y.box_a || x.box_b != y.box_b || x.ga != y.ga || x.gb != y.gb)
        return false;
    auto lay_eq = [](const BlkOperandLayout& p, const BlkOperandLayout& q) {
        return p.rows == q.rows && p.row_stride == q.row_stride && p.head_stride == q.head_stride;
    };
    if ((x.ga && !lay_eq(x.layA, y.layA)) || (x.gb && !lay_eq(x.layB, y.layB))) return false;
    for (int i = 0; i < x.na; ++i)
        if (x.va[i].K != y.va[i].K || x.va[i].residue != y.va[i].residue) return false;
    for (int i = 0; i < x.nb; ++i)
        if (x.vb[i].K != y.vb[i].K || x.vb[i].residue != y.vb[i].residue) return false;
    return true;
}
}  // namespace

bool blk_umma_maps(BlkUmmaParams& p, const BlkUmmaOperand& A, const BlkUmmaOperand& B, int box_a, int box_b, UmMaps& maps) {
    if (A.num_views < 1 || B.num_views < 1 || A.num_views > BLK_UMMA_VIEWS || B.num_views > BLK_UMMA_VIEWS) return false;
    static thread_local LaunchKey key;   // kilobytes: not on the stack of a caller's thread
    key.a = A.base; key.b = B.base; key.Da = A.D; key.Db = B.D; key.H = p.H;
    key.na = A.num_views; key.nb = B.num_views; key.bf16 = p.bf16;
    key.box_a = box_a; key.box_b = box_b;
    key.ga = A.given != nullptr; key.gb = B.given != nullptr;
    if (A.given) key.layA = *A.given;
    if (B.given) key.layB = *B.given;
    for (int i = 0; i < A.num_views; ++i) key.va[i] = A.views[i];
    for (int i = 0; i < B.num_views; ++i) key.vb[i] = B.views[i];
    {
        std::lock_guard<std::mutex> g(g_launch_mu);
        for (LaunchSlot& sl : g_launch_slots)
            if (sl.used && same_key(sl.key, key)) {
                sl.stamp = ++g_launch_clock;
                maps = sl.maps;
                p.head_firstA = sl.hfA;
                p.head_firstB = sl.hfB;
                return true;
            }
    }
    // every view of an operand has the same order of its strides, so the same order of coordinates
    auto encode = [&](const BlkUmmaOperand& op, CUtensorMap* out, int box_rows, int* head_first) {
        if (op.given && (op.num_views != 1 || op.views[0].residue != 0)) return false;
        for (int v = 0; v < op.num_views; ++v) {
            const BlkUmmaView& vw = op.views[v];
            const BlkOperandLayout lay = op.given ? *op.given : BlkOperandLayout{(op.D - vw.residue) / vw.K, vw.K, op.D};
            int hf = 0;
            if (!blk_make_row_map(&out[v], static_cast<const unsigned char*>(op.base) + 2 * vw.residue, p.bf16, vw.K, p.H, lay,
                                  64, box_rows, &hf))
                return false;
            if (v > 0 && hf != *head_first) return false;
            *head_first = hf;
        }
        return true;
    };
    if (!encode(A, maps.a, box_a, &p.head_firstA) || !encode(B, maps.b, box_b, &p.head_firstB)) return false;
    std::lock_guard<std::mutex> g(g_launch_mu);
    LaunchSlot* victim = &g_launch_slots[0];
    for (LaunchSlot& sl : g_launch_slots) {
        if (!sl.used) { victim = &sl; break; }
        if (sl.stamp < victim->stamp) victim = &sl;
    }
    victim->key = key;
    victim->maps = maps;
    victim->hfA = p.head_firstA;
    victim->hfB = p.head_firstB;
    victim->stamp = ++g_launch_clock;
    victim->used = true;
    return true;
}

cudaError_t blk_launch_gemm_umma(const BlkUmmaParams& p_in, const BlkUmmaOperand& A, const BlkUmmaOperand& B, int sms,
                                 cudaStream_t st) {
    if ((int64_t)p_in.num_items * p_in.H == 0) return cudaSuccess;
    BlkUmmaParams p = p_in;
    static thread_local UmMaps maps;
    if (!blk_umma_maps(p, A, B, UM_BM, p.wide ? UL<true>::BN : UL<false>::BN, maps)) return cudaErrorInvalidValue;
    auto run = [&](auto tag) {
        typedef decltype(tag) Tag;
        if (p.epi == BLK_EPI_SOFTMAX)
            return p.out_f32 ? launch<Tag, true, true, false>(p, maps, sms, st) : launch<Tag, false, true, false>(p, maps, sms, st);
        if (p.wide) return p.out_f32 ? launch<Tag, true, false, true>(p, maps, sms, st) : launch<Tag, false, false, true>(p, maps, sms, st);
        return p.out_f32 ? launch<Tag, true, false, false>(p, maps, sms, st) : launch<Tag, false, false, false>(p, maps, sms, st);
    };
    return p.bf16 ? run(BlkBf16Tag{}) : run(BlkHalfTag{});
}

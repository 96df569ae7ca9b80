// Fused attention for segments of any length on the 5th-generation tensor cores:
// out_s = softmax(scale * Q_s K_s^T) V_s per segment and head, head dimension 64 or
// 128, without the probabilities ever leaving the SM.
//
// A persistent CTA (one per SM, 20 warps) walks a static list of work items.  An item is
// up to two 128-row query blocks of one head, stream A and stream B: two blocks of one
// segment, which share every key and value tile, or the odd last blocks of two segments
// with tiles of their own.  A stream sweeps its keys and values in tiles of 64 rows with
// two score buffers in tensor memory, so that the softmax warps find the next scores ready
// whenever they are done with a tile, and two streams put two independent warps on every
// scheduler: neither the chain Q K^T -> softmax -> P V of a tile nor a warp's own latencies
// are waited for.  Roles:
//   warps 0, 1   producers: a lane each issues tiled TMA loads (128-byte swizzle) of the query
//                blocks and key tiles, of the value tiles, into rings;
//   warps 2, 3   scores of stream A, of stream B: S = Q K^T of a tile into the buffer whose
//                probabilities (two tiles back) P V has read;
//   warps 16, 17 products with the values of stream A, of stream B: O += P V.  P is read from
//                tensor memory (first operand [tmem], two 16-bit elements per column, row =
//                lane), V as loaded, i.e. MN-major.  The warps of a pair see every tile of their
//                ring: a tile is free when both have let go of it, and each sees all phases of
//                the ring's barriers;
//   warps 4-7, 8-11  softmax of stream A, of stream B: a thread owns one row of 64 scores, so
//                no row statistics are exchanged.  Online softmax with a lazy reference: the
//                running maximum is only moved (and O rescaled in tensor memory) when the new
//                one exceeds it by more than 8 in the exponent, so P <= 2^8 and the rescale is
//                rare.  P, rounded to the input type, overwrites the scores;
//   warps 12-15  output: wait for a block's last P V and its row sums, read O, divide, store
//                the rows (and the logarithm of the row sums when a backward pass will want
//                them), hand the accumulator back;
//   warp 18      planner: the items' records, a ring of them in shared memory (warp 19 only
//                completes the warpgroup for the trade of registers).
//
// Tensor memory at d = 128 is full: 2 streams x (2 x 64 columns of scores + 128 of result).
// Tiles of 128 rows would leave room for one score buffer per stream only; measured, that
// left the softmax warps waiting 2400 of every 5600 cycles.
//
// Bound by no single pipe in short runs (208 segments of 64..512 rows, 16 heads, d = 128: tensor
// pipe active 44 %, special-function unit 48 %, issue slots 43 %, DRAM 52 %; the softmax warps
// wait for their loads from tensor memory and for products), and by the power limit in long
// ones: 1088 such segments take 1220 us alone and 1390-1490 us sustained at 1.35-1.4 GHz.
//
// Rows of the tiles past the end of a segment belong to its neighbour (or are zero
// past the end of the buffer): extra query rows are never stored, extra key columns
// are masked before the row maximum, and the value rows between the end of a segment
// and the next multiple of 16 are cleared in shared memory before P V.
//
// Every wait is bounded: when the bound is hit the kernel records a status code, all
// roles leave their loops, tensor memory is released and the kernel returns.
//
// Upstream has no fused operator; this replaces the chain blockGEMM -> blockSoftmax ->
// blockGEMM(P, V) of its two operators (blockedAttention/apply.py:6-41) for the
// attention use they are built for.
#include <cuda.h>

#include "blk_device.cuh"
#include "blk_kernels.h"
#include "blk_umma_ptx.cuh"

namespace {

constexpr int FA_BN = 64;                  // key / value rows per tile
constexpr int FA_THREADS = 32 * 20;         // launched with 96 registers each; see FA_REGS
// Registers per thread after the warpgroups have traded: 2 x 128 x 144 (softmax) + 3 x 128 x 64 = the 640 x 96 of the launch.
constexpr int FA_REGS_SOFTMAX = 144, FA_REGS_OTHER = 64;
constexpr int FA_QB_BYTES = 128 * 128;     // 128 rows of one 64-column block: 16 KB
constexpr int FA_TB_BYTES = FA_BN * 128;   // the same of a key / value tile
constexpr int FA_S_COL = 0;                // tensor-memory columns: two score buffers of stream A at 0, of stream B at 128,
constexpr int FA_O_COL = 256;              // results at 256 and 384
constexpr float FA_LAZY = 8.f;             // exponent slack before the running maximum moves

template <int D>
struct FL {
    static constexpr int NB = D / 64;                     // 64-column blocks of an operand row
    static constexpr uint32_t LOG_NS = D == 64 ? 3 : 2, NS = 1u << LOG_NS;  // slots of the key ring, and of the value ring
    static constexpr uint32_t NQ = 3;                                     // slots of the query ring
    static constexpr int Q_BYTES = NB * FA_QB_BYTES;      // a query block
    static constexpr int TILE_BYTES = NB * FA_TB_BYTES;   // a key or value tile
    static constexpr int K_OFF = NQ * Q_BYTES;
    static constexpr int V_OFF = K_OFF + NS * TILE_BYTES;
    static constexpr int LSUM_OFF = V_OFF + NS * TILE_BYTES;
    static constexpr int LSUM_BYTES = 2 * 2 * 128 * 4;    // per stream: row sums, row references
    static constexpr int ITEM_OFF = LSUM_OFF + LSUM_BYTES;
    static constexpr int BAR_OFF = ITEM_OFF + 4 * 64;
    static constexpr int SMEM_BYTES = BAR_OFF + 544;
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

// A work item as the roles read it from shared memory (a ring of FA_ITEMS of them, filled by the planner warp): the
// roles keep few registers and do no arithmetic that is the same for all of them.
struct FaItem {
    int4 side[2];  // per stream: keys N, tiles T (0: no such block), steps of the item = larger T, shared tiles
    int4 rows;     // rowQ, rowKV of stream A, of stream B
    int4 misc;     // query rows M of A (0: nothing follows), of B, head, tiles of B
};
constexpr int FA_ITEMS = 4;
constexpr int FA_ITEM_READERS = 18;  // 2 producers, 4 MMA warps, 8 softmax warps, 4 output warps

// What a role needs to walk the items.
struct FaRing {
    const unsigned char* items;
    uint32_t bar;  // item_full[FA_ITEMS], item_empty[FA_ITEMS]
    volatile int* abort_flag;
};

// A walk of stream x over the tiles of a CTA.  Step j of an item is tile j of both streams; the tiles of a ring are
// numbered by step: one per step when the streams share them, else two, stream A's first (also where one of the two
// streams has no such tile any more: its number is passed over without a load).
struct FaWalk {
    int x, j, steps, rem;    // rem: keys of stream x left from this step on
    uint32_t item, n, q;     // item: items begun; n: number of the step's first tile; q: of the item's first query block
    bool shared, two;
    __device__ __forceinline__ explicit FaWalk(int x_) : x(x_), j(0), steps(0), rem(0), item(0), n(0), q(0), shared(false), two(false) {}
    // To the next item: all lanes of the warp call; false at the end.  The rest of the item's record goes to rows and misc.
    __device__ __forceinline__ bool begin(const FaRing& r, int4* rows, int4* misc) {
        const uint32_t s = item % FA_ITEMS;
        if (!mbar_wait(r.bar + 8u * s, (item / FA_ITEMS) & 1u, r.abort_flag, 18)) return false;
        const FaItem* it = reinterpret_cast<const FaItem*>(r.items) + s;
        const int4 mine = it->side[x], m = it->misc;
        if (rows) *rows = it->rows;
        if (misc) *misc = m;
        if (item > 0) q += two ? 2u : 1u;
        rem = mine.y ? mine.x : 0;
        steps = mine.z;
        shared = mine.w != 0;
        two = m.y != 0;
        j = 0;
        ++item;
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(r.bar + 8u * (FA_ITEMS + s));
        return m.x != 0;
    }
    // To the next step (called before every step, the first one too).
    __device__ __forceinline__ bool step(const FaRing& r, int4* rows = nullptr, int4* misc = nullptr) {
        if (j == steps) return begin(r, rows, misc);
        return true;
    }
    __device__ __forceinline__ void done() {
        n += shared ? 1u : 2u;
        rem -= FA_BN;
        ++j;
    }
    __device__ __forceinline__ uint32_t tile() const { return n + (shared ? 0u : (uint32_t)x); }
    __device__ __forceinline__ uint32_t other() const { return n + 1u - (uint32_t)x; }
    __device__ __forceinline__ bool mine() const { return rem > 0; }
    __device__ __forceinline__ bool last() const { return rem <= FA_BN; }
    __device__ __forceinline__ int ncols() const { return min(rem, FA_BN); }
};

template <typename Tag, int D>
__global__ void __launch_bounds__(FA_THREADS, 1)
blk_attn_umma_kernel(const BlkFlashParams p, const __grid_constant__ CUtensorMap mapQ,
                     const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV) {
    using L = FL<D>;
    constexpr uint32_t NS = L::NS, LOG_NS = L::LOG_NS, NQ = L::NQ;
    extern __shared__ __align__(1024) unsigned char fa_smem_raw[];
    unsigned char* smem = fa_smem_raw;
    if (blk_smem_u32(smem) & 1023u) {  // the swizzled tiles rely on a 1024-byte aligned base
        if (threadIdx.x == 0) atomicCAS(p.status, 0, 29);
        return;
    }
    volatile float* lsum = reinterpret_cast<volatile float*>(smem + L::LSUM_OFF);  // [stream][sum, reference][row]
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 66);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 67);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_u32 = blk_smem_u32(smem);
    const uint32_t bar0 = blk_smem_u32(bars);
    auto o_ready = [&](int x) { return bar0 + 8u * (0 + x); };
    auto o_free = [&](int x) { return bar0 + 8u * (2 + x); };
    auto l_ready = [&](int x) { return bar0 + 8u * (4 + x); };
    auto pv_done = [&](int x, uint32_t b) { return bar0 + 8u * (54 + 2 * x + b); };
    auto s_full = [&](int x, uint32_t b) { return bar0 + 8u * (8 + 2 * x + b); };  // per stream and score buffer
    auto p_full = [&](int x, uint32_t b) { return bar0 + 8u * (12 + 2 * x + b); };
    auto q_full = [&](uint32_t s) { return bar0 + 8u * (16 + s); };
    auto q_empty = [&](uint32_t s) { return bar0 + 8u * (19 + s); };
    auto k_full = [&](uint32_t s) { return bar0 + 8u * (22 + s); };
    auto k_empty = [&](uint32_t s) { return bar0 + 8u * (30 + s); };
    auto v_full = [&](uint32_t s) { return bar0 + 8u * (38 + s); };
    auto v_empty = [&](uint32_t s) { return bar0 + 8u * (46 + s); };
    const FaRing ring{smem + L::ITEM_OFF, bar0 + 8u * 58, abort_flag};  // item_full, item_empty: barriers 58 to 65
    auto sQ = [&](uint32_t s) { return smem_u32 + s * L::Q_BYTES; };
    auto sK = [&](uint32_t s) { return smem_u32 + L::K_OFF + s * L::TILE_BYTES; };
    auto sV = [&](uint32_t s) { return smem_u32 + L::V_OFF + s * L::TILE_BYTES; };

    if (threadIdx.x == 0) {
        for (int x = 0; x < 2; ++x) {
            mbar_init(o_ready(x), 1);
            mbar_init(o_free(x), 4);
            mbar_init(l_ready(x), 4);
            for (uint32_t b = 0; b < 2; ++b) {
                mbar_init(s_full(x, b), 1);
                mbar_init(p_full(x, b), 4);
                mbar_init(pv_done(x, b), 1);
            }
        }
        for (uint32_t s = 0; s < NQ; ++s) {
            mbar_init(q_full(s), 1);
            mbar_init(q_empty(s), 1);
        }
        for (uint32_t s = 0; s < NS; ++s) {  // a tile is let go by both MMA warps
            mbar_init(k_full(s), 1);
            mbar_init(k_empty(s), 2);
            mbar_init(v_full(s), 1);
            mbar_init(v_empty(s), 2);
        }
        for (uint32_t s = 0; s < FA_ITEMS; ++s) {
            mbar_init(ring.bar + 8u * s, 1);
            mbar_init(ring.bar + 8u * (FA_ITEMS + s), FA_ITEM_READERS);
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

    // (the trade of registers is between whole warpgroups)
    if (warp >= 4 && warp < 12) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(FA_REGS_SOFTMAX));
        // ---------------- softmax: warps 4..7 stream A, 8..11 stream B ----------------
        const int q = warp & 3, x = (warp - 4) >> 2;
        const int row = q * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        const uint32_t ocol = lane_addr + (uint32_t)(FA_O_COL + 128 * x);
        const float sl = fabsf(p.scale) * BLK_LOG2E;  // a negative scale is applied by the MMA (negated Q)
        uint32_t g = 0, itc = 0;
        bool ok = true;
        uint32_t ra[32], rb[32];
        FaWalk wk(x);
#pragma unroll 1
        while (ok && wk.begin(ring, nullptr, nullptr)) {
            if (!wk.mine()) continue;
            const int N = wk.rem, T = (N + FA_BN - 1) / FA_BN;
            float m_run = -INFINITY, l_run = 0.f;
#pragma unroll 1
            for (int j = 0; j < T; ++j, ++g) {
                const uint32_t scol = lane_addr + (uint32_t)(FA_S_COL + 128 * x) + FA_BN * (g & 1u);
                if (!mbar_wait(s_full(x, g & 1u), (g >> 1) & 1u, abort_flag, 30)) { ok = false; break; }
                tc_fence_after();
                tc_ld32_nowait(scol, ra);
                tc_ld32_nowait(scol + 32, rb);
                tc_ld_wait(ra);
                tc_ld_wait(rb);
                const int ncols = N - j * FA_BN;
                if (ncols < FA_BN) {  // columns past the end of the segment
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        if (i >= ncols) ra[i] = 0xff800000u;  // -inf
                        if (32 + i >= ncols) rb[i] = 0xff800000u;
                    }
                }
                float m4[4] = {m_run, __uint_as_float(ra[0]), __uint_as_float(rb[0]), __uint_as_float(rb[1])};
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    m4[0] = blk_max3(m4[0], __uint_as_float(ra[i]), __uint_as_float(ra[i + 1]));
                    m4[1] = blk_max3(m4[1], __uint_as_float(ra[i + 2]), __uint_as_float(ra[i + 3]));
                    m4[2] = blk_max3(m4[2], __uint_as_float(rb[i]), __uint_as_float(rb[i + 1]));
                    m4[3] = blk_max3(m4[3], __uint_as_float(rb[i + 2]), __uint_as_float(rb[i + 3]));
                }
                const float m_new = fmaxf(blk_max3(m4[0], m4[1], m4[2]), m4[3]);
                const bool move = (m_new - m_run) * sl > FA_LAZY;  // always at the first tile (m_run = -inf)
                float f = 1.f;
                if (move) {
                    f = blk_exp2((m_run - m_new) * sl);
                    m_run = m_new;
                }
                const float nm = -m_run * sl;
                const float2 sl2 = make_float2(sl, sl), nm2 = make_float2(nm, nm);
                float2 s2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
                uint32_t pk[32];
#pragma unroll
                for (int i = 0; i < 64; i += 2) {
                    const uint32_t u0 = i < 32 ? ra[i & 31] : rb[i & 31], u1 = i < 32 ? ra[(i + 1) & 31] : rb[(i + 1) & 31];
                    float2 t = blk_fma2(make_float2(__uint_as_float(u0), __uint_as_float(u1)), sl2, nm2);
                    t.x = blk_exp2(t.x);
                    t.y = blk_exp2(t.y);
                    s2[(i >> 1) & 1] = blk_add2(s2[(i >> 1) & 1], t);
                    pk[i >> 1] = BlkCvt<Tag>::pack2(t.x, t.y);
                }
                l_run = l_run * f + ((s2[0].x + s2[0].y) + (s2[1].x + s2[1].y));
                tc_st32(scol, pk);
                if (j > 0 && __any_sync(0xffffffffu, move)) {
                    // a row's reference moved: rescale O, at rest once P V of the previous tile is done
                    if (!mbar_wait(pv_done(x, (g - 1u) & 1u), ((g - 1u) >> 1) & 1u, abort_flag, 31)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 0; c < D; c += 32) {
                        tc_ld32(ocol + c, ra);
#pragma unroll
                        for (int i = 0; i < 32; ++i) ra[i] = __float_as_uint(__uint_as_float(ra[i]) * f);
                        tc_st32(ocol + c, ra);
                    }
                }
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full(x, g & 1u));
            }
            if (!ok) break;
            // row sums to the output warps; the slot is free once they have stored this stream's previous block
            if (!mbar_wait(o_free(x), (itc & 1u) ^ 1u, abort_flag, 33)) break;
            lsum[(2 * x) * 128 + row] = l_run;
            lsum[(2 * x + 1) * 128 + row] = m_run * sl;
            __syncwarp();
            if (lane == 0) mbar_arrive(l_ready(x));
            ++itc;
        }
    } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(FA_REGS_OTHER));
    if (warp < 2) {
        // ---------------- producers: warp 0 queries and keys, warp 1 values ----------------
        const bool keys = warp == 0;
        const CUtensorMap* map = keys ? &mapK : &mapV;
        const int hf = keys ? p.head_firstK : p.head_firstV;
        int4 rows, misc;
        FaWalk wk(0);
        bool ok = true;
#pragma unroll 1
        while (ok && wk.step(ring, &rows, &misc)) {
            const int head = misc.z;
            if (keys && wk.j == 0) {
#pragma unroll 1
                for (uint32_t i = 0; ok && i < (wk.two ? 2u : 1u); ++i) {
                    const uint32_t n = wk.q + i, slot = n % NQ;
                    if (!(ok = mbar_wait(q_empty(slot), ((n / NQ) & 1u) ^ 1u, abort_flag, 21))) break;
                    const int row = i ? rows.z : rows.x;
                    if (elect_one()) {
                        mbar_expect_tx(q_full(slot), L::Q_BYTES);
#pragma unroll
                        for (int b = 0; b < L::NB; ++b)  // coordinates (k, row, head), or (k, head, row) for a token-major operand
                            tma_load_3d(sQ(slot) + b * FA_QB_BYTES, &mapQ, q_full(slot), 64 * b, p.head_firstQ ? head : row,
                                        p.head_firstQ ? row : head);
                    }
                    __syncwarp();
                }
            }
#pragma unroll 1
            for (int i = 0; ok && i < (wk.shared ? 1 : 2); ++i) {
                const uint32_t n = wk.n + (uint32_t)i, slot = n & (NS - 1u);
                const uint32_t full = keys ? k_full(slot) : v_full(slot), dst = keys ? sK(slot) : sV(slot);
                if (!(ok = mbar_wait(keys ? k_empty(slot) : v_empty(slot), ((n >> LOG_NS) & 1u) ^ 1u, abort_flag, 22))) break;
                const int row = (i ? rows.w : rows.y) + wk.j * FA_BN;
                const bool there = i ? wk.j < misc.w : wk.mine();
                if (elect_one()) {
                    if (there) {
                        mbar_expect_tx(full, L::TILE_BYTES);
#pragma unroll
                        for (int b = 0; b < L::NB; ++b)
                            tma_load_3d(dst + b * FA_TB_BYTES, map, full, 64 * b, hf ? head : row, hf ? row : head);
                    } else {
                        mbar_arrive(full);  // this stream is done with the item
                    }
                }
                __syncwarp();
            }
            wk.done();
        }
    } else if (warp == 2 || warp == 3) {
        // ---------------- scores: warp 2 stream A, warp 3 stream B ----------------
        const int x = warp - 2;
        const uint32_t idesc_qk = instr_desc(p.bf16, 0, p.scale < 0.f);
        const uint32_t s_tmem = tmem_base + (uint32_t)(FA_S_COL + 128 * x);
        FaWalk wk(x);
        uint64_t desc_q = 0;
        uint32_t q_slot = 0, g = 0;  // g: tiles of this stream so far
#pragma unroll 1
        while (wk.step(ring)) {
            const uint32_t n = wk.tile(), slot = n & (NS - 1u);
            if (!mbar_wait(k_full(slot), (n >> LOG_NS) & 1u, abort_flag, 24)) break;
            if (wk.mine()) {
                if (wk.j == 0) {
                    // (waited for behind the item's first key tile, which is loaded later: the slot's previous use is over)
                    const uint32_t qn = wk.q + (uint32_t)x;
                    q_slot = qn % NQ;
                    if (!mbar_wait(q_full(q_slot), (qn / NQ) & 1u, abort_flag, 23)) break;
                    desc_q = smem_desc_sw128(sQ(q_slot));
                }
                // S = Q K^T into score buffer g & 1, whose probabilities (tile g - 2) P V has read
                const uint32_t idesc = idesc_qk | ((uint32_t)((wk.ncols() + 15) >> 4) << 18);  // columns in units of 16
                const uint32_t d_tmem = s_tmem + FA_BN * (g & 1u);
                const uint64_t db0 = smem_desc_sw128(sK(slot));
                if (g >= 2u && !mbar_wait(pv_done(x, g & 1u), ((g >> 1) & 1u) ^ 1u, abort_flag, 20)) break;
                tc_fence_after();
                if (elect_one()) {
                    // descriptors of the k-th step: the start-address field (16-byte units) moves by 2 per 32 bytes
                    // inside a 64-column block, and by the block's size per block
#pragma unroll
                    for (int k = 0; k < D / 16; ++k)
                        tc_mma_f16(d_tmem, desc_q + (uint64_t)((k >> 2) * (FA_QB_BYTES >> 4) + 2 * (k & 3)),
                                   db0 + (uint64_t)((k >> 2) * (FA_TB_BYTES >> 4) + 2 * (k & 3)), idesc, k != 0);
                    tc_commit(s_full(x, g & 1u));
                    tc_commit(k_empty(slot));                     // key tile reusable
                    if (wk.last()) tc_commit(q_empty(q_slot));    // the query block is free once these products have read it
                }
                __syncwarp();
                ++g;
            } else if (lane == 0) {
                mbar_arrive(k_empty(slot));
            }
            if (!wk.shared) {
                const uint32_t m = wk.other(), os = m & (NS - 1u);
                if (!mbar_wait(k_full(os), (m >> LOG_NS) & 1u, abort_flag, 25)) break;
                if (lane == 0) mbar_arrive(k_empty(os));
            }
            wk.done();
        }
    } else if (warp == 16 || warp == 17) {
        // ---------------- products with the values: warp 16 stream A, warp 17 stream B ----------------
        const int x = warp - 16;
        const uint32_t idesc_pv = instr_desc(p.bf16, D, 0, 1);
        const uint32_t s_tmem = tmem_base + (uint32_t)(FA_S_COL + 128 * x), o_tmem = tmem_base + (uint32_t)(FA_O_COL + 128 * x);
        FaWalk wk(x);
        uint32_t o_par = 1u, g = 0;
#pragma unroll 1
        while (wk.step(ring)) {
            const uint32_t n = wk.tile(), slot = n & (NS - 1u);
            if (!mbar_wait(v_full(slot), (n >> LOG_NS) & 1u, abort_flag, 27)) break;
            if (wk.mine()) {
                const int ncols = wk.ncols();
                if (ncols & 15) {
                    // value rows past the end of the segment (with a shared tile both warps write the same zeros)
#pragma unroll 1
                    for (int i = lane; i < (16 - (ncols & 15)) * L::NB * 8; i += 32) {  // 16-byte pieces
                        const int rr = i / (L::NB * 8), rem = i % (L::NB * 8);
                        tc_sts_v4(sV(slot) + (rem >> 3) * FA_TB_BYTES + (ncols + rr) * 128 + (rem & 7) * 16, 0u, 0u, 0u, 0u);
                    }
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // generic-proxy writes before the MMA's reads
                    __syncwarp();
                }
                if (wk.j == 0) {
                    if (!mbar_wait(o_free(x), o_par, abort_flag, 19)) break;
                    o_par ^= 1u;
                }
                const uint64_t db0 = smem_desc_sw128_mn(sV(slot), FA_TB_BYTES);
                const uint32_t a_tmem = s_tmem + FA_BN * (g & 1u);
                if (!mbar_wait(p_full(x, g & 1u), (g >> 1) & 1u, abort_flag, 26)) break;
                tc_fence_after();
                // O += P V; 16 probabilities of a row are 8 columns; 16 value rows are 2048 bytes
                if (elect_one()) {
                    if (ncols > FA_BN - 16) {
#pragma unroll
                        for (int k = 0; k < FA_BN / 16; ++k)
                            tc_mma_f16_ts(o_tmem, a_tmem + 8u * k, db0 + (uint64_t)(128 * k), idesc_pv, k ? 1u : (uint32_t)wk.j);
                    } else {
#pragma unroll 1
                        for (int k = 0; 16 * k < ncols; ++k)
                            tc_mma_f16_ts(o_tmem, a_tmem + 8u * k, db0 + (uint64_t)(128 * k), idesc_pv, (uint32_t)(wk.j | k));
                    }
                    tc_commit(pv_done(x, g & 1u));                    // the score buffer is free, O at rest until the next P V
                    tc_commit(v_empty(slot));                 // value tile reusable
                    if (wk.last()) tc_commit(o_ready(x));     // the block's result is complete
                }
                __syncwarp();
                ++g;
            } else if (lane == 0) {
                mbar_arrive(v_empty(slot));
            }
            if (!wk.shared) {
                const uint32_t m = wk.other(), os = m & (NS - 1u);
                if (!mbar_wait(v_full(os), (m >> LOG_NS) & 1u, abort_flag, 28)) break;
                if (lane == 0) mbar_arrive(v_empty(os));
            }
            wk.done();
        }
    } else if (warp == 18) {
        // ---------------- planner: the records of the items ----------------
        const uint32_t total = (uint32_t)p.num_pairs * (uint32_t)p.H;
        bool more = true;
#pragma unroll 1
        for (uint32_t i = 0; more; ++i) {
            // odd rounds run through the CTAs backwards: with the items sorted by cost no CTA always gets the heaviest
            const uint32_t n = i * gridDim.x + ((i & 1u) ? gridDim.x - 1u - blockIdx.x : blockIdx.x), s = i % FA_ITEMS;
            more = n < total;
            int4 a = make_int4(0, 0, 0, 0), b = a;
            uint32_t q = 0;
            if (more) {
                q = n / (uint32_t)p.H;
                const int4* src = reinterpret_cast<const int4*>(p.pairs + q);
                a = blk_ld_table(src);
                b = blk_ld_table(src + 1);
            }
            if (!mbar_wait(ring.bar + 8u * (FA_ITEMS + s), ((i / FA_ITEMS) & 1u) ^ 1u, abort_flag, 17)) break;
            if (lane == 0) {
                const int Ta = more ? (a.w + FA_BN - 1) / FA_BN : 0, Tb = b.z > 0 ? (b.w + FA_BN - 1) / FA_BN : 0;
                const int shared = b.z > 0 && a.y == b.y, steps = max(Ta, Tb);
                FaItem* it = reinterpret_cast<FaItem*>(smem + L::ITEM_OFF) + s;
                it->side[0] = make_int4(a.w, Ta, steps, shared);
                it->side[1] = make_int4(b.w, Tb, steps, shared);
                it->rows = make_int4(a.x, a.y, b.x, b.y);
                it->misc = make_int4(a.z, b.z, (int)(n - q * (uint32_t)p.H), Tb);
                mbar_arrive(ring.bar + 8u * s);  // release: the record is visible to whoever sees the phase end
            }
            __syncwarp();
        }
    } else if (warp >= 12 && warp < 16) {
        // ---------------- output: warps 12..15 ----------------
        const int q = warp & 3;
        const int row = q * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        uint32_t par = 0;  // per stream, parity of the next waits
        uint32_t r[32];
        int4 rows, misc;
        bool ok = true;
        FaWalk wk(0);
#pragma unroll 1
        while (ok && wk.begin(ring, &rows, &misc)) {
#pragma unroll 1
            for (int x = 0; x < 2; ++x) {
                const int M = x ? misc.y : misc.x, row0 = x ? rows.z : rows.x, head = misc.z;
                if (M == 0) continue;
                if (!mbar_wait(l_ready(x), (par >> x) & 1u, abort_flag, 35)) { ok = false; break; }
                const float lrow = lsum[(2 * x) * 128 + row], mref = lsum[(2 * x + 1) * 128 + row];
                if (!mbar_wait(o_ready(x), (par >> x) & 1u, abort_flag, 36)) { ok = false; break; }
                par ^= 1u << x;
                tc_fence_after();
                const float inv = __frcp_rn(lrow);
                const bool mine = row < M;
                // a thread stores its row, 64 bytes at a time
                uint16_t* orow = reinterpret_cast<uint16_t*>(p.out) + (int64_t)head * p.out_head_stride +
                                 (int64_t)(row0 + row) * p.out_row_stride;
                if (p.lse && mine) p.lse[(int64_t)head * p.layQ.rows + row0 + row] = mref + __log2f(lrow);
#pragma unroll 1
                for (int c = 0; c < D; c += 32) {
                    tc_ld32(lane_addr + (uint32_t)(FA_O_COL + 128 * x + c), r);
#pragma unroll
                    for (int i = 0; i < 32; i += 2)
                        r[i >> 1] = BlkCvt<Tag>::pack2(__uint_as_float(r[i]) * inv, __uint_as_float(r[i + 1]) * inv);
                    if (mine) blk_stg64(orow + c, r);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(o_free(x));  // accumulator and row-sum slot reusable
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

template <typename Tag, int D>
cudaError_t launch(const BlkFlashParams& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, int sms,
                   cudaStream_t st) {
    auto kern = blk_attn_umma_kernel<Tag, D>;
    cudaError_t e = blk_func_smem(reinterpret_cast<const void*>(kern), FL<D>::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const int64_t total = (int64_t)p.num_pairs * p.H;
    const dim3 grid((unsigned)(total < sms ? total : sms)), block(FA_THREADS);
    return blk_launch(total <= 12 * (int64_t)sms, kern, grid, block, FL<D>::SMEM_BYTES, st, p, mq, mk, mv);
}

}  // namespace

cudaError_t blk_launch_attn_umma(const BlkFlashParams& p_in, const void* q, const void* k, const void* v, int sms,
                                 cudaStream_t st) {
    if ((int64_t)p_in.num_pairs * p_in.H == 0) return cudaSuccess;
    if (p_in.D != 64 && p_in.D != 128) return cudaErrorInvalidValue;
    BlkFlashParams p = p_in;
    CUtensorMap mq, mk, mv;
    if (!blk_make_row_map(&mq, q, p.bf16, p.D, p.H, p.layQ, 64, BLK_FLASH_BM, &p.head_firstQ) ||
        !blk_make_row_map(&mk, k, p.bf16, p.D, p.H, p.layK, 64, FA_BN, &p.head_firstK) ||
        !blk_make_row_map(&mv, v, p.bf16, p.D, p.H, p.layV, 64, FA_BN, &p.head_firstV))
        return cudaErrorInvalidValue;
    if (p.D == 64) return p.bf16 ? launch<BlkBf16Tag, 64>(p, mq, mk, mv, sms, st) : launch<BlkHalfTag, 64>(p, mq, mk, mv, sms, st);
    return p.bf16 ? launch<BlkBf16Tag, 128>(p, mq, mk, mv, sms, st) : launch<BlkHalfTag, 128>(p, mq, mk, mv, sms, st);
}

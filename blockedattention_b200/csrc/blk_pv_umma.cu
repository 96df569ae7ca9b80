// Second product of blocked attention on the 5th-generation tensor cores:
// out_s (M x D) = scale * A_s (M x K) B_s (K x D) per segment and head, where the rows of
// the first operand have an arbitrary length K and start at arbitrary 2-byte
// offsets (a block of probabilities P_s of a packed (M_s, N_s) score buffer, K =
// N_s) and the second operand is stored (K, D) with D = 64 or 128 (the values V_s
// of a segment: upstream's transpose2 = true).
//
// The rows of P cannot be fetched by tiled TMA (a tensor map needs 16-byte aligned row
// pitches; a packed score block has whatever pitch its segment has), so they take
// another road into the tensor core: one bulk copy a row brings the aligned 16-byte
// vectors that hold a tile's part of it to shared memory, loader warps shift the rows
// into place in registers and store them into tensor memory, from where tcgen05.mma
// takes them as its first operand ([tmem], 16-bit elements, two per column, row =
// lane).  A first operand stored (K, M) -- a gradient block in a backward pass -- is
// copied the same way and read across its rows.  The values are fetched by tiled TMA
// exactly as they lie (MN-major second operand, 128-byte swizzle).
// Bound by memory and by the rate of the row copies (about 13 cycles each, and the issuing warps wait for it): 1024
// segments of 64..512 rows and columns, 16 heads, D = 128 take 1050-1085 us (1197 with a copy for every 128 columns of a
// row, rows re-aligned by selects over whole vectors and rows past a block cleared; 1333 with vector loads by the lane that
// owns a row, 32 cache lines an instruction; 1709 with 8-byte asynchronous copies); the product of a gradient block of a
// long-tailed batch, D = 64, 105 (118), the transposed one, that the staged mma.sync kernel did in 350 us, 127.
//
// A persistent CTA (one per SM, 22 warps) walks a static list of work items, an
// item being a 128-row block of the first operand of one segment of one head; it
// sweeps the contraction index in tiles of 256 (a transposed first operand: 128).  Roles:
//   warp 0      producer: one lane issues the TMA loads of the values, 128 rows a stage;
//   warp 1      MMA: one lane issues O += P V for each tile, P from one of two
//               128-column (four 64-column) buffers in tensor memory, O in one of two
//               accumulators (items alternate); tcgen05.commit frees the value stages and
//               the P buffer and, after an item's last tile, hands O to the output warps;
//   warps 2-17  loaders, a group of eight (four) per P buffer, so the copies of all
//               buffers' tiles are in flight: a lane issues the copy of one row, the next
//               tile's as soon as this one has left shared memory;
//   warps 18-21 output: read O, scale, round and store the rows (a row of the result is
//               D contiguous, 16-byte aligned elements).
//
// Columns of a tile between the end of a row (K) and the next multiple of 16 become
// zeros, and the value rows there are cleared in shared memory; rows past the end of
// the block (M) are never stored.  So nothing outside the segment reaches a result.
// Every wait is bounded: when the bound is hit the kernel records a status code,
// all roles leave their loops, tensor memory is released and the kernel returns.
//
// Replaces upstream sparseBlockedHGEMM_half / _bf16 with transpose2 = true
// (csrc/cuda/spBlkGEMM.cu:424-817) for the product it is used for after the
// softmax, blockGEMM(P, V, ..., transpose2=True) (blockedAttention/apply.py:6-25).
#include <cuda.h>

#include "blk_device.cuh"
#include "blk_kernels.h"
#include "blk_umma_ptx.cuh"

namespace {

static_assert(BLK_UMMA_BM == 128, "a work item is a block of 128 rows: one accumulator lane per row");
constexpr int PV_UNIT = 128;         // value rows of a stage, contraction elements that a loader warp brings in of a tile
constexpr int PV_LOADERS = 16;       // loader warps
constexpr int PV_OUT_WARPS = 4;
constexpr int PV_THREADS = 64 + 32 * (PV_LOADERS + PV_OUT_WARPS);
constexpr int PV_BLOCK_BYTES = 128 * 128;  // 128 value rows of one 64-column block: 16 KB
constexpr int PV_O_COL = 256;              // tensor-memory columns of the two result accumulators: 256 and 384

// TA: the first operand is stored (K, M).
template <int D, bool TA>
struct PVL {
    static constexpr int BK = TA ? 128 : 256;               // contraction elements per tile
    static constexpr int PARTS = BK / PV_UNIT;              // loader warps of a group and lane quarter, value stages of a tile
    static constexpr int GROUPS = 4 / PARTS;                // groups of loader warps, one per tensor-memory buffer of the first
                                                            // operand (BK / 2 columns each, below the result accumulators at column 256)
    // a row of a tile in shared memory: its vectors of 16 bytes and one more (an odd number, see row_slot)
    static constexpr int ROW_BYTES = 2 * (TA ? 128 : BK) + 16;
    static constexpr int STRIP_BYTES = 128 * ROW_BYTES;     // per group
    static constexpr int NB = D / 64;                       // 64-column blocks of a value row
    static constexpr int VS = D == 64 ? 5 : 2;              // value ring
    static constexpr int OPER_BYTES = NB * PV_BLOCK_BYTES;  // a 128 x D stage
    static constexpr int V_OFF = 0;
    static constexpr int STRIP_OFF = VS * OPER_BYTES;
    static constexpr int BAR_OFF = STRIP_OFF + GROUPS * STRIP_BYTES;
    static constexpr int SMEM_BYTES = BAR_OFF + 512;
    static_assert(VS <= 6, "barrier slots");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

struct PvWork {
    BlkPvItem it;
    int head;
};

__device__ __forceinline__ bool pv_work(const BlkPvParams& p, uint32_t w, PvWork& wk) {
    const uint32_t total = (uint32_t)p.num_items * (uint32_t)p.H;
    if (w >= total) return false;
    const uint32_t item = w / (uint32_t)p.H;
    wk.head = (int)(w - item * (uint32_t)p.H);
    wk.it = p.items[item];
    return true;
}

// The items of a CTA in order, the record of the next one always on its way.
struct PvItems {
    PvWork nx;
    uint32_t w;
    bool has;
    __device__ __forceinline__ explicit PvItems(const BlkPvParams& p) : w(blockIdx.x) { has = pv_work(p, w, nx); }
    __device__ __forceinline__ bool next(const BlkPvParams& p, PvWork& wk) {
        if (!has) return false;
        wk = nx;
        w += gridDim.x;
        has = pv_work(p, w, nx);
        return true;
    }
};

// A walk over the tiles of one loader group: every GROUPS-th tile of the CTA.
template <int BK>
struct PvTiles {
    PvItems items;
    PvWork wk;
    int j;
    uint32_t g;   // tile of the CTA
    uint32_t u0;  // value stages before this item
    bool valid;
    __device__ __forceinline__ PvTiles(const BlkPvParams& p, uint32_t grp) : items(p), j(0), g(0), u0(0) {
        valid = items.next(p, wk);
        seek(p, grp);
    }
    __device__ __forceinline__ void seek(const BlkPvParams& p, uint32_t to) {  // to tile number `to` of the CTA
#pragma unroll 1
        while (valid) {
            const uint32_t left = (uint32_t)((wk.it.K + BK - 1) / BK - j);
            if (g + left > to) break;
            g += left;
            u0 += (uint32_t)((wk.it.K + PV_UNIT - 1) / PV_UNIT);
            j = 0;
            valid = items.next(p, wk);
        }
        j += (int)(to - g);
        g = to;
    }
};

// Where a warp's strip keeps row r of its 32: the lanes, each reading the same word of its row, counted from the word that the
// row starts in -- (a + r K) / 2 modulo 4 words into the strip's row -- hit 32 banks for every K that is not a multiple of 4.
__device__ __forceinline__ uint32_t row_slot(uint32_t r, int K) {
    return K & 1 ? (r & 1u) + 2u * (r >> 3) + 8u * ((r >> 1) & 3u) : (r >> 2) + 8u * (r & 3u);
}

template <typename Tag, int D, bool TA>
__global__ void __launch_bounds__(PV_THREADS, 1)
blk_pv_umma_kernel(const BlkPvParams p, const __grid_constant__ CUtensorMap mapV) {
    using L = PVL<D, TA>;
    constexpr int VS = L::VS, BK = L::BK, GROUPS = L::GROUPS, PARTS = L::PARTS, ROW_BYTES = L::ROW_BYTES;
    extern __shared__ __align__(1024) unsigned char pv_smem_raw[];
    unsigned char* smem = pv_smem_raw;
    if (blk_smem_u32(smem) & 1023u) {  // the swizzled tiles rely on a 1024-byte aligned base
        if (threadIdx.x == 0) atomicCAS(p.status, 0, 49);
        return;
    }
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
    // barriers: 0.. p_full[4], 4.. p_free[4], 8.. o_ready[2], 10.. o_free[2], 12.. v_full[VS], 18.. v_empty[VS],
    // 24.. rows_in[16], 40.. rows_out[16]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 56);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 57);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_u32 = blk_smem_u32(smem);
    const uint32_t bar0 = blk_smem_u32(bars);
    auto p_full = [&](int b) { return bar0 + 8u * (0 + b); };
    auto p_free = [&](int b) { return bar0 + 8u * (4 + b); };
    auto o_ready = [&](int b) { return bar0 + 8u * (8 + b); };
    auto o_free = [&](int b) { return bar0 + 8u * (10 + b); };
    auto v_full = [&](int s) { return bar0 + 8u * (12 + s); };
    auto v_empty = [&](int s) { return bar0 + 8u * (18 + s); };
    // per group and quarter of its rows; a transposed operand, whose rows everybody reads: the group's first
    auto rows_in = [&](int w) { return bar0 + 8u * (24 + w); };
    auto rows_out = [&](int w) { return bar0 + 8u * (40 + w); };
    auto sV = [&](int s) { return smem_u32 + L::V_OFF + s * L::OPER_BYTES; };

    if (threadIdx.x == 0) {
        for (int b = 0; b < GROUPS; ++b) {
            mbar_init(p_full(b), 4 * PARTS);
            mbar_init(p_free(b), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(o_ready(b), 1);
            mbar_init(o_free(b), PV_OUT_WARPS);
        }
        for (int s = 0; s < VS; ++s) {
            mbar_init(v_full(s), 1);
            mbar_init(v_empty(s), 1);
        }
        for (int w = 0; w < 4 * GROUPS; ++w) {
            mbar_init(rows_in(w), TA ? 4 : PARTS);
            mbar_init(rows_out(w), TA ? 4 : PARTS);
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

    if (warp == 0) {
        // ---------------- producer: value tiles ----------------
        if (elect_one()) {
            uint32_t g = 0;
            PvItems items(p);
            PvWork wk;
            bool ok = true;
#pragma unroll 1
            while (ok && items.next(p, wk)) {
#pragma unroll 1
                for (int k = 0; k < wk.it.K; k += PV_UNIT, ++g) {
                    const int vs = (int)(g % VS);
                    if (!mbar_wait(v_empty(vs), ((g / VS) & 1u) ^ 1u, abort_flag, 41)) { ok = false; break; }
                    mbar_expect_tx(v_full(vs), L::OPER_BYTES);
                    const int row = wk.it.rowB + k;
#pragma unroll
                    for (int b = 0; b < L::NB; ++b)  // coordinates (column, row, head)
                        tma_load_3d(sV(vs) + b * PV_BLOCK_BYTES, &mapV, v_full(vs), 64 * b, row, wk.head);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issue ----------------
        if (elect_one()) {
            const uint32_t idesc = instr_desc(p.bf16, D, 0, 1);  // second operand MN-major
            uint32_t g = 0, u = 0, itc = 0;  // tiles, value stages, items so far
            PvItems items(p);
            PvWork wk;
            bool ok = true;
#pragma unroll 1
            for (; ok && items.next(p, wk); ++itc) {
                const int ob = (int)(itc & 1u);
                if (!mbar_wait(o_free(ob), ((itc >> 1) & 1u) ^ 1u, abort_flag, 42)) break;
#pragma unroll 1
                for (int k0 = 0; ok && k0 < wk.it.K; k0 += BK, ++g) {
                    const int buf = (int)(g % GROUPS);
                    if (!mbar_wait(p_full(buf), (g / GROUPS) & 1u, abort_flag, 43)) { ok = false; break; }
                    const uint32_t d_tmem = tmem_base + (uint32_t)(PV_O_COL + 128 * ob);
#pragma unroll 1
                    for (int part = 0; part < PARTS && k0 + part * PV_UNIT < wk.it.K; ++part, ++u) {
                        const int vs = (int)(u % VS), k1 = k0 + part * PV_UNIT;
                        if (!mbar_wait(v_full(vs), (u / VS) & 1u, abort_flag, 44)) { ok = false; break; }
                        tc_fence_after();
                        const int ksteps = (min(wk.it.K - k1, PV_UNIT) + 15) >> 4;
                        const uint32_t a_tmem = tmem_base + (uint32_t)(buf * (BK / 2) + part * (PV_UNIT / 2));
                        const uint64_t db0 = smem_desc_sw128_mn(sV(vs), PV_BLOCK_BYTES);
#pragma unroll
                        for (int k = 0; k < PV_UNIT / 16; ++k)  // 16 elements of a row are 8 columns; 16 value rows are 2048 bytes
                            if (k < ksteps) tc_mma_f16_ts(d_tmem, a_tmem + 8u * k, db0 + (uint64_t)(128 * k), idesc, (k1 | k) != 0);
                        tc_commit(v_empty(vs));  // value stage reusable
                    }
                    tc_commit(p_free(buf));                                  // first-operand buffer reusable
                    if (k0 + BK >= wk.it.K) tc_commit(o_ready(ob));         // the item's result is complete
                }
            }
        }
    } else if (warp < 2 + PV_LOADERS) {
        // ---------------- loaders: warps 2..17, group grp fills buffer grp (every GROUPS-th tile) ----------------
        const int grp = (warp - 2) / (4 * PARTS), part = ((warp - 2) >> 2) % PARTS;
        const int q = warp & 3;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        const unsigned char* A = reinterpret_cast<const unsigned char*>(p.A);
        const uint32_t strip = smem_u32 + L::STRIP_OFF + (uint32_t)grp * L::STRIP_BYTES;
        const uint32_t bar_rows = rows_in(4 * grp + (TA ? 0 : q)), bar_read = rows_out(4 * grp + (TA ? 0 : q));
        // byte address, from the start of the operand, of the first element of row r of a tile as it lies in memory
        auto addr_of = [&](const PvTiles<BK>& t, int r) {
            const int64_t e = (int64_t)t.wk.head * p.Dm1 + t.wk.it.offA;
            return TA ? 2 * (e + (int64_t)(t.j * BK + r) * t.wk.it.pitch) : 2 * (e + (int64_t)r * t.wk.it.K + t.j * BK);
        };
        // a lane copies a row, of the 32 / PARTS of its warp: the aligned 16-byte vectors that hold its elements
        auto copy = [&](const PvTiles<BK>& t) {
            const int rq = part * (32 / PARTS) + lane % (32 / PARTS), r = q * 32 + rq;  // of its quarter, of the block
            const int kk = min(t.wk.it.K - t.j * BK, BK), mm = min(t.wk.it.M, 128);
            const int64_t b = addr_of(t, r);
            const int sh = (int)(b & 15);
            const uint32_t bytes = lane < 32 / PARTS && r < (TA ? kk : mm) ? (uint32_t)((sh + 2 * (TA ? mm : kk) + 15) & ~15) : 0u;
            const uint32_t sum = __reduce_add_sync(0xffffffffu, bytes);
            if (lane == 0) mbar_expect_tx(bar_rows, sum);
            __syncwarp();
            if (bytes)
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                                 strip + (TA ? (uint32_t)r : (uint32_t)(q * 32) + row_slot((uint32_t)rq, t.wk.it.K)) * ROW_BYTES),
                             "l"(A + (b - sh)), "r"(bytes), "r"(bar_rows)
                             : "memory");
        };
        uint32_t round = 0;
        PvTiles<BK> cur(p, (uint32_t)grp);
        if (cur.valid) copy(cur);
#pragma unroll 1
        while (cur.valid) {
            const uint32_t g = cur.g;
            const int ncols = min(cur.wk.it.K - cur.j * BK, BK);  // of the tile
            // the value stage that holds its last rows
            const uint32_t vu = cur.u0 + (uint32_t)(cur.j * PARTS + (ncols - 1) / PV_UNIT);
            bool ok = mbar_wait(bar_rows, round & 1u, abort_flag, 48);
            ++round;
#pragma unroll
            for (int h = 0; h < 2; ++h) {  // 64 elements of this warp's part of the row at a time, two per word
                const int c0 = part * PV_UNIT + 64 * h;
                const int nv = min(ncols - c0, 64);  // of these that exist
                uint32_t pk[32];
                if (nv <= 0) {
                } else if constexpr (TA) {
                    // element (k, this lane's row): neighbouring lanes read neighbouring elements of row k
                    // (the rows' first bytes repeat modulo 16 after eight rows)
                    const uint32_t src = strip + (uint32_t)(64 * h) * ROW_BYTES + 2u * (q * 32 + lane);
                    const uint32_t b = (uint32_t)addr_of(cur, 0), step = 2u * (uint32_t)cur.wk.it.pitch;
                    uint32_t at[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) at[i] = src + ((b + i * step) & 15u);
#pragma unroll
                    for (int i = 0; i < 64; i += 2) {
                        uint32_t lo, hi;
                        asm volatile("ld.shared.u16 %0, [%1];\n" : "=r"(lo) : "r"(at[i & 7] + i * ROW_BYTES));
                        asm volatile("ld.shared.u16 %0, [%1];\n" : "=r"(hi) : "r"(at[(i + 1) & 7] + (i + 1) * ROW_BYTES));
                        pk[i >> 1] = __byte_perm(lo, hi, 0x5410);
                    }
                } else {
                    const uint32_t sh = (uint32_t)addr_of(cur, q * 32 + lane) & 15u;  // bytes before the row's first element
                    const uint32_t src = strip + (uint32_t)(q * 32) * ROW_BYTES + row_slot(lane, cur.wk.it.K) * ROW_BYTES + 2u * c0;
                    if (!__any_sync(0xffffffffu, (int)sh)) {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n"
                                         : "=r"(pk[4 * i]), "=r"(pk[4 * i + 1]), "=r"(pk[4 * i + 2]), "=r"(pk[4 * i + 3])
                                         : "r"(src + 16u * i));
                    } else {
                        // word by word from the word the row starts in; a start on an odd element is shifted out
                        uint32_t v[33];
#pragma unroll
                        for (int i = 0; i < 33; ++i) asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(v[i]) : "r"(src + (sh & 12u) + 4u * i));
                        if (__any_sync(0xffffffffu, (int)(sh & 2u))) {
                            const uint32_t hs = (sh & 2u) * 8u;
#pragma unroll
                            for (int i = 0; i < 32; ++i) pk[i] = __funnelshift_r(v[i], v[i + 1], hs);
                        } else {
#pragma unroll
                            for (int i = 0; i < 32; ++i) pk[i] = v[i];
                        }
                    }
                }
                if (nv > 0 && nv < 64 && (nv & 15)) {
                    // elements between the end of the row and the next multiple of 16 meet value rows that are zero, and must not
                    // be what such a product is not zero for.  (Rows past the end of the block may be anything: nobody reads
                    // what they give.)
                    asm volatile("");  // (a branch: as selects this would cost every tile)
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        if (2 * i >= nv) pk[i] = 0u;
                        else if (2 * i + 1 >= nv) pk[i] &= 0xffffu;
                    }
                }
                if (h == 0) {
                    ok = ok && mbar_wait(p_free(grp), ((g / GROUPS) & 1u) ^ 1u, abort_flag, 45);
                    tc_fence_after();
                } else {
                    cur.seek(p, g + GROUPS);
                    // the rows have been read: by the warps of this quarter, or (a transposed operand) by all of the group
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_read);
                    ok = ok && mbar_wait(bar_read, (round & 1u) ^ 1u, abort_flag, 39);
                    if (ok && cur.valid) copy(cur);
                }
                if (nv > 0) tc_st32(lane_addr + (uint32_t)(grp * (BK / 2) + c0 / 2), pk);
            }
            if (!ok) break;
            tc_wait_st();
            if (ncols & 15) {
                // last tile of the row: clear the value rows between its end and the next multiple of 16
                // (what was in that stage before must have been multiplied, or the parity of an older load would pass for this one's.
                // The tile GROUPS back is over; a short ring needs more than that)
                constexpr uint32_t BACK = PARTS == 1 ? VS : 1;
                if (VS < GROUPS * PARTS && g >= BACK &&
                    !mbar_wait(p_free((int)((g - BACK) % GROUPS)), ((g - BACK) / GROUPS) & 1u, abort_flag, 40))
                    break;
                const int vs = (int)(vu % VS), last = (ncols - 1) % PV_UNIT + 1;  // rows of the stage that exist
                if (!mbar_wait(v_full(vs), (vu / VS) & 1u, abort_flag, 46)) break;
                const int nz = (16 - (ncols & 15)) * L::NB * 8;  // 16-byte pieces to clear
#pragma unroll 1
                for (int t = (part * 4 + q) * 32 + lane; t < nz; t += 128 * PARTS) {
                    const int rr = t / (L::NB * 8), rem = t % (L::NB * 8);
                    tc_sts_v4(sV(vs) + (rem >> 3) * PV_BLOCK_BYTES + (last + rr) * 128 + (rem & 7) * 16, 0u, 0u, 0u, 0u);
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // generic-proxy writes before the MMA's reads
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full(grp));
        }
    } else {
        // ---------------- output: the last four warps ----------------
        const int q = warp & 3;
        const int row = q * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        uint32_t itc = 0;
        PvItems items(p);
        PvWork wk;
        uint32_t r[32];
#pragma unroll 1
        for (; items.next(p, wk); ++itc) {
            const int ob = (int)(itc & 1u);
            if (!mbar_wait(o_ready(ob), (itc >> 1) & 1u, abort_flag, 47)) break;
            tc_fence_after();
            // a thread stores its row, 64 bytes at a time
            uint16_t* orow = reinterpret_cast<uint16_t*>(p.C) + (int64_t)wk.head * p.Dout + wk.it.offC + (int64_t)row * D;
#pragma unroll 1
            for (int c = 0; c < D; c += 32) {
                tc_ld32(lane_addr + (uint32_t)(PV_O_COL + 128 * ob + c), r);
#pragma unroll
                for (int i = 0; i < 32; i += 2)
                    r[i >> 1] = BlkCvt<Tag>::pack2(__uint_as_float(r[i]) * p.scale, __uint_as_float(r[i + 1]) * p.scale);
                if (row < wk.it.M) blk_stg64(orow + c, r);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(o_free(ob));  // result accumulator reusable
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

template <typename Tag, int D, bool TA>
cudaError_t launch(const BlkPvParams& p, const CUtensorMap& mv, int sms, cudaStream_t st) {
    auto kern = blk_pv_umma_kernel<Tag, D, TA>;
    cudaError_t e = blk_func_smem(reinterpret_cast<const void*>(kern), PVL<D, TA>::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const int64_t total = (int64_t)p.num_items * p.H;
    const dim3 grid((unsigned)(total < sms ? total : sms)), block(PV_THREADS);
    return blk_launch(total <= 12 * (int64_t)sms, kern, grid, block, PVL<D, TA>::SMEM_BYTES, st, p, mv);
}

}  // namespace

cudaError_t blk_launch_pv_umma(const BlkPvParams& p, const void* V, int sms, cudaStream_t st) {
    if ((int64_t)p.num_items * p.H == 0) return cudaSuccess;
    if (p.D != 64 && p.D != 128) return cudaErrorInvalidValue;
    CUtensorMap mv;
    int head_first = 0;
    const BlkOperandLayout lay{p.Dm2 / p.D, p.D, p.Dm2};  // the values as a (rows, D) matrix per head strip
    if (!blk_make_row_map(&mv, V, p.bf16, p.D, p.H, lay, 64, PV_UNIT, &head_first) || head_first) return cudaErrorInvalidValue;
    auto run = [&](auto tag) {
        typedef decltype(tag) Tag;
        if (p.D == 64) return p.ta ? launch<Tag, 64, true>(p, mv, sms, st) : launch<Tag, 64, false>(p, mv, sms, st);
        return p.ta ? launch<Tag, 128, true>(p, mv, sms, st) : launch<Tag, 128, false>(p, mv, sms, st);
    };
    return p.bf16 ? run(BlkBf16Tag{}) : run(BlkHalfTag{});
}

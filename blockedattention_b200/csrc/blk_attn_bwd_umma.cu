// Backward of the fused attention for segments of any length on the 5th-generation tensor cores, head dimension 64 or
// 128.  With P = softmax(scale Q K^T) recomputed from the saved row logarithms, dP = dO V^T and
// dS = P (dP - rowsum(dO O)):
//     dV = P^T dO      dK = scale dS^T Q      dQ = scale dS K
// Two launches of one kernel, which differ in what a CTA keeps and what it sweeps:
//     <QUERIES>  a 128-row query block with its dO stays, keys and values pass:  S = Q K^T, dP = dO V^T, dQ += dS K
//     <KEYS>     a 128-row key block with its values stays, queries and dO pass: S^T = K Q^T, dP^T = V dO^T,
//                dV += P^T dO, dK += dS^T Q
// Either way every operand is used as it lies: the first operand of the accumulating products (P^T, dS^T, dS) is what the
// softmax threads have in their rows and goes back to tensor memory as 16-bit elements ([tmem] operand), the second is a
// passing tile, MN-major.  Seven products instead of the five of a one-pass kernel, but no atomics and no fp32 workspace
// for dQ (adding a segment's key blocks into it would move more bytes than the two products cost time for segments of
// 64..512 rows), and results that do not depend on the order of the CTAs.
//
// A persistent CTA (one per SM, 16 warps) walks a static list of items (resident block, head), longest sweeps first:
//   warp 0      producer: resident blocks (two slots) and passing tiles of 64 rows (a ring of stages);
//   warp 1      S and dP products of a tile, into one of two pairs of 64-column buffers in tensor memory;
//   warp 2      accumulating products of a tile; clears the tile rows between the end of a segment and the next multiple
//               of 16 first;
//   warp 3      planner: item records in shared memory; <KEYS>: row logarithms and sums of the passing queries;
//   warps 4-11  softmax: warps 4-7 take the even tiles, 8-11 the odd ones; a thread owns one row of 64 columns and meets
//               nobody;
//   warps 12-15 output; <QUERIES>: also rowsum(dO O) of the next item, kept for the <KEYS> launch.
// Bound by the products and the chain of a tile through the roles -- scores, exponentials, dP, dS, product -- with two pairs
// of buffers to overlap it: at d = 128 the products of a tile occupy the tensor pipe for 1280 cycles (<KEYS>) and 1024
// (<QUERIES>; S and dP run at two thirds of the rate with 64 columns, but 128-column tiles would leave room for one pair) of
// the 2120 and 1740 that it takes, and softmax warps wait for scores two fifths and a third of their time.  256 segments of
// 64..512 rows, 16 heads: 620 and 484 us.  (<QUERIES> 609 with rowsum(dO O) made by the lane that owns a row, dO from the
// resident block, four loads of O at a time: softmax warps waited two fifths of their time for it.)
//
// rowsum(dO O) takes O as the forward pass rounded it, where a chain of operators has rowsum(P dP) of its own rounded P.
// 2-norm errors of dQ against 64 bits, 300 rows, d = 64, bf16: 2.4e-3 (the chain: 3.3e-3) for scores of deviation 1, 5.4e-3
// (4.2e-3) for 8 and 7.1e-3 (5.0e-3) for 32, where a row's probability sits on one key and dS is what is left of a
// difference.
//
// Rows past the end of a segment belong to its neighbour: as resident rows they are computed and not stored, as passing
// rows they get P = dS = 0.  Every wait is bounded, as in the forward kernel.
//
// Upstream differentiates the chain blockGEMM -> blockSoftmax -> blockGEMM operator by operator
// (csrc/sparseBlockedAttention.cpp:52-72, :103-114), with P, dP and dS in memory.
#include <cuda.h>

#include "blk_device.cuh"
#include "blk_kernels.h"
#include "blk_umma_ptx.cuh"

namespace {

constexpr int BW_BN = 64;              // rows of a passing tile
constexpr int BW_THREADS = 32 * 16;    // launched with 128 registers each: 2 x 128 x 168 + 2 x 128 x 88 after the trade
constexpr int BW_REGS_SOFTMAX = 168, BW_REGS_OTHER = 88;
constexpr int BW_RB_BYTES = 128 * 128;    // 64-column block of a resident block
constexpr int BW_TB_BYTES = BW_BN * 128;  // 64-column block of a tile
constexpr int BW_S_COL = 0, BW_DP_COL = 128, BW_ACC_COL = 256;  // tensor memory: S 2 x 64, dP 2 x 64, accumulators 2 x 128
constexpr uint32_t BW_ITEMS = 8;
constexpr uint32_t BW_AHEAD = 6;       // the planner publishes this many items ahead of its own walk

struct BwItem {
    int4 a;  // first resident row, first passing row, passing rows, tiles
    int4 b;  // resident rows, head, valid (0: nothing follows)
};

template <int D>
struct BL {
    static constexpr int NB = D / 64;
    static constexpr uint32_t NS = D == 64 ? 6 : 3;          // stages (a tile of each passing operand)
    static constexpr int R_BYTES = NB * BW_RB_BYTES;         // one resident block
    static constexpr int T_BYTES = NB * BW_TB_BYTES;         // one passing tile
    static constexpr int T_OFF = 4 * R_BYTES;                // two slots x two resident operands
    static constexpr int AUX_OFF = T_OFF + (int)NS * 2 * T_BYTES;
    static constexpr int AUX_BYTES = (int)NS * 512 > 2048 ? (int)NS * 512 : 2048;  // <KEYS>: per stage 64 + 64 floats; <QUERIES>: 2 x (128 + 128)
    static constexpr int ITEM_OFF = AUX_OFF + AUX_BYTES;
    static constexpr int BAR_OFF = ITEM_OFF + (int)BW_ITEMS * 32;
    static constexpr int SMEM_BYTES = BAR_OFF + 512;
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

enum BwMode { QUERIES, KEYS };

template <typename Tag, int D, BwMode MODE>
__global__ void __launch_bounds__(BW_THREADS, 1)
blk_attn_bwd_umma_kernel(const BlkFlashBwdParams p, const __grid_constant__ CUtensorMap mapR1,
                         const __grid_constant__ CUtensorMap mapR2, const __grid_constant__ CUtensorMap mapT1,
                         const __grid_constant__ CUtensorMap mapT2) {
    using L = BL<D>;
    constexpr uint32_t NS = L::NS;
    constexpr int NB = L::NB;
    extern __shared__ __align__(1024) unsigned char bw_smem_raw[];
    unsigned char* smem = bw_smem_raw;
    if (blk_smem_u32(smem) & 1023u) {  // the swizzled tiles rely on a 1024-byte aligned base
        if (threadIdx.x == 0) atomicCAS(p.status, 0, 59);
        return;
    }
    volatile float* aux = reinterpret_cast<volatile float*>(smem + L::AUX_OFF);
    const BwItem* items = reinterpret_cast<const BwItem*>(smem + L::ITEM_OFF);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 62);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 63);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_u32 = blk_smem_u32(smem);
    const uint32_t bar0 = blk_smem_u32(bars);
    auto r_full = [&](uint32_t i) { return bar0 + 8u * (0 + i); };
    auto r_empty = [&](uint32_t i) { return bar0 + 8u * (2 + i); };
    auto s_full = [&](uint32_t b) { return bar0 + 8u * (4 + b); };
    auto dp_full = [&](uint32_t b) { return bar0 + 8u * (6 + b); };
    auto p_full = [&](uint32_t b) { return bar0 + 8u * (8 + b); };
    auto ds_full = [&](uint32_t b) { return bar0 + 8u * (10 + b); };
    auto b_free = [&](uint32_t b) { return bar0 + 8u * (12 + b); };
    auto o_ready = [&](uint32_t i) { return bar0 + 8u * (14 + i); };
    auto o_free = [&](uint32_t i) { return bar0 + 8u * (16 + i); };
    auto rowv_full = [&](uint32_t i) { return bar0 + 8u * (18 + i); };   // <QUERIES>: row values of an item
    auto rowv_empty = [&](uint32_t i) { return bar0 + 8u * (20 + i); };
    auto t_full = [&](uint32_t s) { return bar0 + 8u * (22 + s); };
    auto t_empty = [&](uint32_t s) { return bar0 + 8u * (28 + s); };
    auto aux_full = [&](uint32_t s) { return bar0 + 8u * (34 + s); };    // <KEYS>: row values of a tile
    auto item_full = [&](uint32_t i) { return bar0 + 8u * (40 + i); };
    auto item_empty = [&](uint32_t i) { return bar0 + 8u * (48 + i); };
    auto sR = [&](uint32_t slot, int op) { return smem_u32 + (2u * slot + (uint32_t)op) * L::R_BYTES; };
    auto sT = [&](uint32_t s, int op) { return smem_u32 + L::T_OFF + (2u * s + (uint32_t)op) * L::T_BYTES; };

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < 2; ++i) {
            mbar_init(r_full(i), 1);
            mbar_init(r_empty(i), 1);
            mbar_init(s_full(i), 1);
            mbar_init(dp_full(i), 1);
            mbar_init(p_full(i), 4);
            mbar_init(ds_full(i), 4);
            mbar_init(b_free(i), 1);
            mbar_init(o_ready(i), 1);
            mbar_init(o_free(i), 4);
            mbar_init(rowv_full(i), 4);
            mbar_init(rowv_empty(i), 8);
        }
        for (uint32_t s = 0; s < NS; ++s) {
            mbar_init(t_full(s), 1);
            mbar_init(t_empty(s), 1);
            mbar_init(aux_full(s), 1);
        }
        for (uint32_t i = 0; i < BW_ITEMS; ++i) {
            mbar_init(item_full(i), 1);
            mbar_init(item_empty(i), 16);
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

    uint32_t item = 0;  // items begun by this warp
    int4 ia, ib;
    // To the next item (all lanes of the warp call); false at the end.
    auto begin = [&]() -> bool {
        const uint32_t s = item % BW_ITEMS;
        if (!mbar_wait(item_full(s), (item / BW_ITEMS) & 1u, abort_flag, 50)) return false;
        ia = items[s].a;
        ib = items[s].b;
        ++item;
        __syncwarp();
        if (lane == 0) mbar_arrive(item_empty(s));
        return ib.z != 0;
    };

    // (the trade of registers is between whole warpgroups)
    if (warp >= 4 && warp < 12) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(BW_REGS_SOFTMAX));
        // ---------------- softmax: warps 4..7 even tiles, 8..11 odd tiles ----------------
        const int q = warp & 3;
        const uint32_t b = (uint32_t)(warp - 4) >> 2;  // the parity this warp takes, and its buffer
        const int row = q * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        const uint32_t scol = lane_addr + BW_S_COL + BW_BN * b, dcol = lane_addr + BW_DP_COL + BW_BN * b;
        const float sl = fabsf(p.scale) * BLK_LOG2E;  // a negative scale is applied by the MMA (negated first operand)
        const float2 sl2 = make_float2(sl, sl);
        uint32_t g = 0;  // tiles of the CTA so far
        bool ok = true;
        uint32_t ra[32], rb[32];
#pragma unroll 1
        while (ok && begin()) {
            const int n = ia.z, T = ia.w;
            float nlse = 0.f, ndelta = 0.f;  // <QUERIES>: negated row values
            if constexpr (MODE == QUERIES) {
                const uint32_t i = (item - 1u) & 1u;
                if (!mbar_wait(rowv_full(i), ((item - 1u) >> 1) & 1u, abort_flag, 51)) break;
                nlse = aux[256 * i + row];
                ndelta = aux[256 * i + 128 + row];
                __syncwarp();
                if (lane == 0) mbar_arrive(rowv_empty(i));
            }
#pragma unroll 1
            for (int j = 0; j < T; ++j, ++g) {
                if ((g & 1u) != b) continue;
                const int ncols = n - j * BW_BN;
                const uint32_t par = (g >> 1) & 1u;
                if (!mbar_wait(s_full(b), par, abort_flag, 52)) { ok = false; break; }
                tc_fence_after();
                tc_ld32_nowait(scol, ra);
                tc_ld32_nowait(scol + 32, rb);
                // <KEYS>: values of the tile's 64 query rows (waited for behind the scores: the stage's previous use is over)
                const volatile float* tv = aux + 128 * (g % NS);
                if (MODE == KEYS && !mbar_wait(aux_full(g % NS), (g / NS) & 1u, abort_flag, 53)) { ok = false; break; }
                tc_ld_wait(ra);
                tc_ld_wait(rb);
                auto vals4 = [&](int i) {  // four column values, one 16-byte shared load
                    float4 v;
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                                 : "r"(blk_smem_u32(const_cast<const float*>(tv)) + 4u * i));
                    return v;
                };
                // P over the scores, in registers
                auto probs = [&](uint32_t (&r)[32], int c0) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        float4 l = make_float4(nlse, nlse, nlse, nlse);
                        if constexpr (MODE == KEYS) l = vals4(c0 + i);
                        const float2 x = blk_fma2(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), sl2, make_float2(l.x, l.y));
                        const float2 y = blk_fma2(make_float2(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])), sl2, make_float2(l.z, l.w));
                        r[i] = __float_as_uint(blk_exp2(x.x));
                        r[i + 1] = __float_as_uint(blk_exp2(x.y));
                        r[i + 2] = __float_as_uint(blk_exp2(y.x));
                        r[i + 3] = __float_as_uint(blk_exp2(y.y));
                    }
                };
                probs(ra, 0);
                probs(rb, 32);
                if (ncols < BW_BN) {  // columns past the end of the segment
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        if (i >= ncols) ra[i] = 0u;
                        if (32 + i >= ncols) rb[i] = 0u;
                    }
                }
                if constexpr (MODE == KEYS) {
                    uint32_t pk[32];
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        pk[i >> 1] = BlkCvt<Tag>::pack2(__uint_as_float(ra[i]), __uint_as_float(ra[i + 1]));
                        pk[16 + (i >> 1)] = BlkCvt<Tag>::pack2(__uint_as_float(rb[i]), __uint_as_float(rb[i + 1]));
                    }
                    tc_st32(scol, pk);
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(p_full(b));
                }
                if (!mbar_wait(dp_full(b), par, abort_flag, 54)) { ok = false; break; }
                tc_fence_after();
                // dS = P (dP - delta), half by half; the first half is stored over columns already read
                auto dscores = [&](const uint32_t (&r)[32], int c0) {
                    uint32_t d[32], pk[16];
                    tc_ld32_nowait(dcol + c0, d);
                    tc_ld_wait(d);
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        float4 e = make_float4(ndelta, ndelta, ndelta, ndelta);
                        if constexpr (MODE == KEYS) e = vals4(64 + c0 + i);
                        const float2 x = blk_add2(make_float2(__uint_as_float(d[i]), __uint_as_float(d[i + 1])), make_float2(e.x, e.y));
                        const float2 y = blk_add2(make_float2(__uint_as_float(d[i + 2]), __uint_as_float(d[i + 3])), make_float2(e.z, e.w));
                        float s0 = x.x * __uint_as_float(r[i]), s1 = x.y * __uint_as_float(r[i + 1]);
                        float s2 = y.x * __uint_as_float(r[i + 2]), s3 = y.y * __uint_as_float(r[i + 3]);
                        if (c0 + i + 3 >= ncols) {  // (dP may be anything there)
                            s0 = c0 + i < ncols ? s0 : 0.f;
                            s1 = c0 + i + 1 < ncols ? s1 : 0.f;
                            s2 = c0 + i + 2 < ncols ? s2 : 0.f;
                            s3 = 0.f;
                        }
                        pk[i >> 1] = BlkCvt<Tag>::pack2(s0, s1);
                        pk[(i >> 1) + 1] = BlkCvt<Tag>::pack2(s2, s3);
                    }
                    tc_st16(dcol + (c0 >> 1), pk);
                };
                dscores(ra, 0);
                dscores(rb, 32);
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(ds_full(b));
            }
        }
    } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(BW_REGS_OTHER));
    if (warp == 0) {
        // ---------------- producer ----------------
        uint32_t g = 0;
        bool ok = true;
        const int hr = p.head_firstR, ht = p.head_firstT;
#pragma unroll 1
        while (ok && begin()) {
            const int head = ib.y;
            const uint32_t slot = (item - 1u) & 1u;
            if (!mbar_wait(r_empty(slot), (((item - 1u) >> 1) & 1u) ^ 1u, abort_flag, 55)) break;
            if (elect_one()) {
                mbar_expect_tx(r_full(slot), 2 * L::R_BYTES);
#pragma unroll
                for (int c = 0; c < NB; ++c) {  // coordinates (k, row, head), or (k, head, row) for a token-major operand
                    tma_load_3d(sR(slot, 0) + c * BW_RB_BYTES, &mapR1, r_full(slot), 64 * c, hr ? head : ia.x, hr ? ia.x : head);
                    tma_load_3d(sR(slot, 1) + c * BW_RB_BYTES, &mapR2, r_full(slot), 64 * c, hr ? head : ia.x, hr ? ia.x : head);
                }
            }
            __syncwarp();
#pragma unroll 1
            for (int j = 0; j < ia.w; ++j, ++g) {
                const uint32_t s = g % NS;
                if (!mbar_wait(t_empty(s), ((g / NS) & 1u) ^ 1u, abort_flag, 56)) { ok = false; break; }
                const int row = ia.y + j * BW_BN;
                if (elect_one()) {
                    mbar_expect_tx(t_full(s), 2 * L::T_BYTES);
#pragma unroll
                    for (int c = 0; c < NB; ++c) {
                        tma_load_3d(sT(s, 0) + c * BW_TB_BYTES, &mapT1, t_full(s), 64 * c, ht ? head : row, ht ? row : head);
                        tma_load_3d(sT(s, 1) + c * BW_TB_BYTES, &mapT2, t_full(s), 64 * c, ht ? head : row, ht ? row : head);
                    }
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // ---------------- S and dP ----------------
        const uint32_t idesc_s = instr_desc(p.bf16, 0, p.scale < 0.f), idesc_dp = instr_desc(p.bf16, 0, 0);
        uint32_t g = 0;
        bool ok = true;
#pragma unroll 1
        while (ok && begin()) {
            const uint32_t slot = (item - 1u) & 1u;
            if (!mbar_wait(r_full(slot), ((item - 1u) >> 1) & 1u, abort_flag, 57)) break;
            const uint64_t dr0 = smem_desc_sw128(sR(slot, 0)), dr1 = smem_desc_sw128(sR(slot, 1));
            int rem = ia.z;
#pragma unroll 1
            for (int j = 0; j < ia.w; ++j, ++g, rem -= BW_BN) {
                const uint32_t s = g % NS, b = g & 1u;
                const uint32_t cols = (uint32_t)((min(rem, BW_BN) + 15) >> 4) << 18;  // columns in units of 16
                const uint64_t dt0 = smem_desc_sw128(sT(s, 0)), dt1 = smem_desc_sw128(sT(s, 1));
                if (!mbar_wait(t_full(s), (g / NS) & 1u, abort_flag, 58)) { ok = false; break; }
                if (!mbar_wait(b_free(b), ((g >> 1) & 1u) ^ 1u, abort_flag, 60)) { ok = false; break; }
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < D / 16; ++k)
                        tc_mma_f16(tmem_base + BW_S_COL + BW_BN * b, dr0 + (uint64_t)((k >> 2) * (BW_RB_BYTES >> 4) + 2 * (k & 3)),
                                   dt0 + (uint64_t)((k >> 2) * (BW_TB_BYTES >> 4) + 2 * (k & 3)), idesc_s | cols, k != 0);
                    tc_commit(s_full(b));
#pragma unroll
                    for (int k = 0; k < D / 16; ++k)
                        tc_mma_f16(tmem_base + BW_DP_COL + BW_BN * b, dr1 + (uint64_t)((k >> 2) * (BW_RB_BYTES >> 4) + 2 * (k & 3)),
                                   dt1 + (uint64_t)((k >> 2) * (BW_TB_BYTES >> 4) + 2 * (k & 3)), idesc_dp | cols, k != 0);
                    tc_commit(dp_full(b));
                    if (j == ia.w - 1) tc_commit(r_empty(slot));
                }
                __syncwarp();
            }
        }
    } else if (warp == 2) {
        // ---------------- accumulating products ----------------
        const uint32_t idesc = instr_desc(p.bf16, D, 0, 1);  // second operand MN-major
        uint32_t g = 0;
        bool ok = true;
        // acc += [tmem a] x tile rows
        auto accumulate = [&](uint32_t acc, uint32_t a_col, uint32_t tile, int ncols, int j) {
            const uint64_t db = smem_desc_sw128_mn(tile, BW_TB_BYTES);
            const uint32_t d_tmem = tmem_base + BW_ACC_COL + 128u * acc, a_tmem = tmem_base + a_col;
            if (ncols > BW_BN - 16) {
#pragma unroll
                for (int k = 0; k < BW_BN / 16; ++k)
                    tc_mma_f16_ts(d_tmem, a_tmem + 8u * k, db + (uint64_t)(128 * k), idesc, k ? 1u : (uint32_t)j);
            } else {
#pragma unroll 1
                for (int k = 0; 16 * k < ncols; ++k)
                    tc_mma_f16_ts(d_tmem, a_tmem + 8u * k, db + (uint64_t)(128 * k), idesc, (uint32_t)(j | k));
            }
        };
#pragma unroll 1
        while (ok && begin()) {
            const uint32_t k0 = item - 1u;
            const uint32_t acc1 = MODE == KEYS ? 1u : k0 & 1u;                                   // of dS x first tile operand
            const uint32_t par = (MODE == KEYS ? k0 & 1u : (k0 >> 1) & 1u) ^ 1u;                 // its accumulator is free
            int rem = ia.z;
#pragma unroll 1
            for (int j = 0; j < ia.w; ++j, ++g, rem -= BW_BN) {
                const uint32_t s = g % NS, b = g & 1u, bpar = (g >> 1) & 1u;
                const int ncols = min(rem, BW_BN);
                const bool last = j == ia.w - 1;
                if (!mbar_wait(t_full(s), (g / NS) & 1u, abort_flag, 61)) { ok = false; break; }
                if (ncols & 15) {
                    const int per = (16 - (ncols & 15)) * NB * 8;  // 16-byte pieces of one tile
#pragma unroll 1
                    for (int i = lane; i < (MODE == KEYS ? 2 : 1) * per; i += 32) {
                        const int op = i >= per, e = i - op * per;
                        const int rr = e / (NB * 8), c = e % (NB * 8);
                        tc_sts_v4(sT(s, op) + (c >> 3) * BW_TB_BYTES + (ncols + rr) * 128 + (c & 7) * 16, 0u, 0u, 0u, 0u);
                    }
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // generic-proxy writes before the MMA's reads
                    __syncwarp();
                }
                if constexpr (MODE == KEYS) {
                    if (j == 0 && !mbar_wait(o_free(0), par, abort_flag, 62)) { ok = false; break; }
                    if (!mbar_wait(p_full(b), bpar, abort_flag, 63)) { ok = false; break; }
                    tc_fence_after();
                    if (elect_one()) {
                        accumulate(0u, BW_S_COL + BW_BN * b, sT(s, 1), ncols, j);  // dV += P^T dO
                        if (last) tc_commit(o_ready(0));
                    }
                    __syncwarp();
                }
                if (j == 0 && !mbar_wait(o_free(acc1), par, abort_flag, 64)) { ok = false; break; }
                if (!mbar_wait(ds_full(b), bpar, abort_flag, 65)) { ok = false; break; }
                tc_fence_after();
                if (elect_one()) {
                    accumulate(acc1, BW_DP_COL + BW_BN * b, sT(s, 0), ncols, j);   // dK += dS^T Q, or dQ += dS K
                    tc_commit(b_free(b));
                    tc_commit(t_empty(s));
                    if (last) tc_commit(o_ready(acc1));
                }
                __syncwarp();
            }
        }
    } else if (warp == 3) {
        // ---------------- planner; <KEYS>: row values of the passing queries ----------------
        const uint32_t total = (uint32_t)p.num_items * (uint32_t)p.H;
        uint32_t pub = 0, g = 0;
        bool more = true, ok = true;
#pragma unroll 1
        for (uint32_t k = 0; ok; ++k) {
#pragma unroll 1
            while (more && pub < k + BW_AHEAD) {
                // odd rounds run through the CTAs backwards: with the items sorted by cost no CTA always gets the heaviest
                const uint32_t n = pub * gridDim.x + ((pub & 1u) ? gridDim.x - 1u - blockIdx.x : blockIdx.x), s = pub % BW_ITEMS;
                more = n < total;
                int4 f = make_int4(0, 0, 0, 0);  // first resident row, first passing row, resident rows, passing rows
                uint32_t q = 0;
                if (more) {
                    q = n / (uint32_t)p.H;
                    f = blk_ld_table(reinterpret_cast<const int4*>(p.items + q));
                }
                if (!mbar_wait(item_empty(s), ((pub / BW_ITEMS) & 1u) ^ 1u, abort_flag, 66)) { ok = false; break; }
                if (lane == 0) {
                    BwItem* it = reinterpret_cast<BwItem*>(smem + L::ITEM_OFF) + s;
                    it->a = make_int4(f.x, f.y, f.w, (f.w + BW_BN - 1) / BW_BN);
                    it->b = make_int4(f.z, (int)(n - q * (uint32_t)p.H), more ? 1 : 0, 0);
                    mbar_arrive(item_full(s));  // release: the record is visible to whoever sees the phase end
                }
                __syncwarp();
                ++pub;
            }
            if (!ok || !begin()) break;
            if constexpr (MODE == KEYS) {
                const int64_t base = (int64_t)ib.y * p.rows_q + ia.y;
#pragma unroll 1
                for (int j = 0; j < ia.w; ++j, ++g) {
                    const uint32_t s = g % NS;
                    if (!mbar_wait(t_empty(s), ((g / NS) & 1u) ^ 1u, abort_flag, 67)) { ok = false; break; }
#pragma unroll
                    for (int r = lane; r < BW_BN; r += 32) {
                        const int at = j * BW_BN + r;
                        aux[128 * s + r] = at < ia.z ? -p.lse[base + at] : 0.f;
                        aux[128 * s + 64 + r] = at < ia.z ? -p.delta[base + at] : 0.f;
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(aux_full(s));
                }
            }
        }
    } else {
        // ---------------- output: warps 12..15 ----------------
        const int q = warp & 3;
        const int row = q * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        // a thread stores its row of an accumulator, 64 bytes at a time
        auto store = [&](uint32_t acc, void* base, int64_t r, bool mine, float f) {
            uint32_t v[32];
            uint16_t* orow = reinterpret_cast<uint16_t*>(base) + r * D;
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < D; c += 32) {
                tc_ld32(lane_addr + BW_ACC_COL + 128u * acc + (uint32_t)c, v);
#pragma unroll
                for (int i = 0; i < 32; i += 2)
                    v[i >> 1] = BlkCvt<Tag>::pack2(__uint_as_float(v[i]) * f, __uint_as_float(v[i + 1]) * f);
                if (mine) blk_stg64(orow + c, v);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(o_free(acc));
        };
        bool have = false;
        int64_t prow = 0;     // this thread's row of the item to be stored
        bool pmine = false;
        uint32_t k = 0;       // that item
#pragma unroll 1
        while (true) {
            const bool more = begin();
            const int64_t r = more ? (int64_t)ib.y * p.rows_r + ia.x + row : 0;
            const bool mine = more && row < ib.x;
            if (MODE == QUERIES && more) {
                // Row values of the item: saved logarithm, rowsum(dO O).  Both from global memory, so that they need not wait for
                // the item's operands; eight lanes a row, everything of 16 rows on its way at a time.
                const uint32_t i = item - 1u, slot = i & 1u;
                const float l = mine ? p.lse[r] : 0.f;
                const int64_t r0 = r - lane + (lane >> 3);  // row lane / 8 of this warp's; then every fourth
                const int left = ib.x - q * 32 - (lane >> 3);
                const uint4* o0 = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.o) + r0 * D) + (lane & 7);
                const uint4* g0 = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.g) + r0 * D) + (lane & 7);
                float d[8];
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint4 ov[4][NB], gv[4][NB];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int c = 0; c < NB; ++c) {
                            const int row4 = 4 * (4 * half + k);
                            ov[k][c] = gv[k][c] = make_uint4(0u, 0u, 0u, 0u);
                            if (row4 < left) {
                                ov[k][c] = o0[row4 * D / 8 + 8 * c];
                                gv[k][c] = g0[row4 * D / 8 + 8 * c];
                            }
                        }
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        float d0 = 0.f, d1 = 0.f;
#pragma unroll
                        for (int c = 0; c < NB; ++c) {
                            const uint32_t ow[4] = {ov[k][c].x, ov[k][c].y, ov[k][c].z, ov[k][c].w}, gw[4] = {gv[k][c].x, gv[k][c].y, gv[k][c].z, gv[k][c].w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                d0 = fmaf(BlkCvt<Tag>::unpack1((uint16_t)ow[e]), BlkCvt<Tag>::unpack1((uint16_t)gw[e]), d0);
                                d1 = fmaf(BlkCvt<Tag>::unpack1((uint16_t)(ow[e] >> 16)), BlkCvt<Tag>::unpack1((uint16_t)(gw[e] >> 16)), d1);
                            }
                        }
                        d[4 * half + k] = d0 + d1;
                    }
                }
#pragma unroll
                for (int k = 0; k < 8; ++k)
#pragma unroll
                    for (int x = 4; x; x >>= 1) d[k] += __shfl_xor_sync(0xffffffffu, d[k], x);
                if (!mbar_wait(rowv_empty(slot), ((i >> 1) & 1u) ^ 1u, abort_flag, 69)) break;
                aux[256 * slot + row] = -l;
                if (!(lane & 7)) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) aux[256 * slot + 128 + q * 32 + 4 * k + (lane >> 3)] = -d[k];
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(rowv_full(slot));
                if (mine) p.delta[r] = -aux[256 * slot + 128 + row];
            }
            if (have) {
                if constexpr (MODE == QUERIES) {
                    if (!mbar_wait(o_ready(k & 1u), (k >> 1) & 1u, abort_flag, 70)) break;
                    store(k & 1u, p.out1, prow, pmine, p.scale);
                } else {
                    if (!mbar_wait(o_ready(0), k & 1u, abort_flag, 71)) break;
                    store(0, p.out0, prow, pmine, 1.f);
                    if (!mbar_wait(o_ready(1), k & 1u, abort_flag, 72)) break;
                    store(1, p.out1, prow, pmine, p.scale);
                }
            }
            if (!more) break;
            prow = r;
            pmine = mine;
            k = item - 1u;
            have = true;
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

template <typename Tag, int D, BwMode MODE>
cudaError_t launch(const BlkFlashBwdParams& p, const CUtensorMap* maps, int sms, cudaStream_t st) {
    auto kern = blk_attn_bwd_umma_kernel<Tag, D, MODE>;
    cudaError_t e = blk_func_smem(reinterpret_cast<const void*>(kern), BL<D>::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const int64_t total = (int64_t)p.num_items * p.H;
    const dim3 grid((unsigned)(total < sms ? total : sms)), block(BW_THREADS);
    return blk_launch(total <= 12 * (int64_t)sms, kern, grid, block, BL<D>::SMEM_BYTES, st, p, maps[0], maps[1], maps[2], maps[3]);
}

}  // namespace

cudaError_t blk_launch_attn_bwd_umma(const BlkFlashBwdParams& p_in, int keys, const void* const* tensors,
                                     const BlkOperandLayout& layR, const BlkOperandLayout& layT, int sms, cudaStream_t st) {
    if ((int64_t)p_in.num_items * p_in.H == 0) return cudaSuccess;
    if (p_in.D != 64 && p_in.D != 128) return cudaErrorInvalidValue;
    BlkFlashBwdParams p = p_in;
    p.g = tensors[1];
    CUtensorMap maps[4];
    for (int i = 0; i < 4; ++i)
        if (!blk_make_row_map(&maps[i], tensors[i], p.bf16, p.D, p.H, i < 2 ? layR : layT, 64, i < 2 ? 128 : BW_BN,
                              i < 2 ? &p.head_firstR : &p.head_firstT))
            return cudaErrorInvalidValue;
    if (p.D == 64) {
        if (p.bf16)
            return keys ? launch<BlkBf16Tag, 64, KEYS>(p, maps, sms, st) : launch<BlkBf16Tag, 64, QUERIES>(p, maps, sms, st);
        return keys ? launch<BlkHalfTag, 64, KEYS>(p, maps, sms, st) : launch<BlkHalfTag, 64, QUERIES>(p, maps, sms, st);
    }
    if (p.bf16)
        return keys ? launch<BlkBf16Tag, 128, KEYS>(p, maps, sms, st) : launch<BlkBf16Tag, 128, QUERIES>(p, maps, sms, st);
    return keys ? launch<BlkHalfTag, 128, KEYS>(p, maps, sms, st) : launch<BlkHalfTag, 128, QUERIES>(p, maps, sms, st);
}

// Scores of large segments, with or without their softmax, on the 5th-generation tensor cores: independent streams.
//
// A persistent CTA (one per SM) runs S streams side by side: S = 4 for contractions of up to 64, 3 for up to 128.  A stream
// walks its own static list of items, an item being a 128-row block of one segment of one head, and takes an item's columns in
// tiles of 64: once for plain scores, twice for the softmax, where the first sweep keeps a reference and a sum per row and the
// second computes the products again, normalises and stores.  A stream has
//   a producer warp  one lane issues the TMA loads: the item's block of the first operand, which stays for the item, and the
//                    tiles of the second into a ring of 64 x 64 units; it also hands the item's record to the others;
//   an MMA warp      one lane issues tcgen05.mma (M = 128, N = 64) into the next of two 64-column accumulators;
//   four epilogue warps, a thread owning a row (one lane of tensor memory): nobody else ever needs to know about it.
// A tile is one piece of a row on its way out: 128 bytes (fp32: two), staged in the warp's strip at the position it has within
// a 32-byte sector of the output, and written by the warp as whole sectors, eight lanes a row.  What does not fill a sector at the
// end of a piece goes in front of the next one, and the sector that a row ends and the next one begins in is put together
// when the row ends: a warp's 32 rows are contiguous, so of all its sectors only the first and the last are written in part.
// That is what the rate hangs on.  Rows of 4094 bytes written by 148 CTAs in pieces of 128 bytes: 3.1 TB/s where a piece
// starts on any 16 bytes, 2.6 as words from any 4 bytes on (256-byte pieces), 4.8 to 5.7 where it starts on a sector;
// rows of 578 bytes 2.3 to 3.1, 1.8 and 4.5 to 5.6.
//
// Why streams: with all epilogue warps of the CTA taking chunks of one or two items in turn, a third of their time
// went into waiting for products (a resident row takes up to all of the tensor memory, and the item behind it waits for it to
// be stored), a fifth into stepping over the chunks of others and a twentieth into meeting to combine row statistics.
// A stream's warps meet nobody, its two accumulators are free again as soon as they are in registers, and
// four streams are in different phases of an item, so one's exponentials overlap another's stores.  The price is a second
// exponential per element for rows that tensor memory could hold (129..512 columns; up to two tiles stay in the accumulators
// between the sweeps), so the other kernel keeps those.
//
// Measured, us, the other kernel -> this one: plain bf16 scores of 128 segments of 16..2048 rows, 4 heads, K = 64: 168 -> 121 (3.7
// of the 4.8 TB/s that such rows can be written at); their softmax for 512 segments: 898 -> 757 (743 with the logarithm of
// a row's sum in the exponent instead of a division, see below).  What bounds the softmax: exponentials (two per element, the unit
// 65 % busy in a single launch), 58 % of the issue slots, the shared-memory path; of 810 us, when that was its time, 676 were left without
// exponentials and 674 without stores.  Bulk copies from the strips in place of the stores: 917, they queue in front of the operands' copies.
//
// Every wait on an mbarrier is bounded: when the bound is hit the kernel records a status code, all roles leave their
// loops, tensor memory is released and the kernel returns.  Rows past the end of a segment belong to its neighbour (or are
// zero-filled past the end of the buffer); they only reach accumulator rows and columns that are never stored, and columns
// >= N are masked before any row reduction.
//
// Replaces upstream sparseBlockedHGEMM_half / _bf16 with the 128 x 128 x 16 WMMA tile (csrc/cuda/spBlkGEMM.cu:424-817,
// :866-868) and, fused, the softmax kernels (csrc/cuda/spBlkSoftmax.cu:88-269).
#include <cuda.h>

#include "blk_device.cuh"
#include "blk_kernels.h"
#include "blk_umma_items.cuh"
#include "blk_umma_ptx.cuh"

namespace {

constexpr int SS_BN = 64;               // columns of a tile = of an accumulator
constexpr int SS_BK = 64;               // k elements of a unit (one 128-byte swizzle row)
constexpr int SS_A_BYTES = 128 * SS_BK * 2;
constexpr int SS_UNIT = SS_BN * SS_BK * 2;
constexpr int SS_BOX = 64;              // rows of a copy
constexpr float SS_LAZY = 32.f;         // exponent slack before a softmax reference moves
// Strip of an epilogue warp: 32 row pieces of 128 bytes and the sector that a first element inside a sector pushes past the
// end, and for each row the sector that it begins in.
constexpr int SS_PITCH = 160;
constexpr uint64_t SS_NEAR = 0xffffffffull / 32;  // rows of so many bytes: 31 of them and a sector are within 32 bits
constexpr int SS_HEADS = 32 * SS_PITCH;
constexpr int SS_STRIP_BYTES = SS_HEADS + 32 * 32;

template <int KB>  // 64-element blocks of the contraction
struct SL {
    static constexpr int S = KB == 1 ? 4 : 3;
    static constexpr int THREADS = 32 * (4 * S + 8);
    // registers of a thread: 80 (96) at launch; the warpgroups of producers and MMA warps give to those of the epilogues
    static constexpr int REGS_EPI = KB == 1 ? 104 : 120, REGS_OTHER = KB == 1 ? 32 : 56, REGS = KB == 1 ? 80 : 96;
    static_assert(128 * S * REGS_EPI + 256 * REGS_OTHER <= THREADS * REGS, "the shares of the warpgroups");
    static constexpr uint32_t UNITS = 2;  // ring of a stream
    static constexpr int STREAM_BYTES = KB * SS_A_BYTES + (int)UNITS * SS_UNIT;
    static constexpr int STRIP_OFF = S * STREAM_BYTES;
    static constexpr int BAR_OFF = STRIP_OFF + 4 * S * SS_STRIP_BYTES;  // 16 barriers a stream
    static constexpr int REC_OFF = BAR_OFF + S * 128 + 16;              // two records a stream
    static constexpr int SMEM_BYTES = REC_OFF + S * 128;
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};

// An item as the roles of its stream see it, in shared memory.
struct __align__(16) Rec {
    int64_t cbase;   // element of the output where the item's rows start (head, segment and row block included)
    int32_t rows;    // rows of the block | first quarter that holds them << 8
    int32_t N, K;
    int32_t valid;   // 0: nothing follows
    int32_t pad[2];
};
static_assert(sizeof(Rec) == 32, "two records of a stream in 64 bytes");

// Predicated global stores as single instructions (no branch around them).
__device__ __forceinline__ void stg_v4(uint64_t p, const uint4& v) {
    asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void stg_v4_if(uint64_t p, const uint4& v, bool ok) {
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %5, 0;\n @q st.global.v4.b32 [%0], {%1, %2, %3, %4};\n}\n"
                 ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"((int)ok) : "memory");
}
__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// Where a strip keeps row r.  A row's words start at the word its first element has within a sector of the output,
// (a + r N) mod 8 words, and a slot adds 8 banks: the order of the slots is such that the 32 lanes, each storing the same word
// of its row, hit 32 banks (16-bit elements: any N that is not a multiple of 4; fp32: any odd N).
__device__ __forceinline__ uint32_t strip_slot(uint32_t r, bool odd16) {
    return odd16 ? (r & 1u) + 2u * (r >> 4) + 4u * ((r >> 1) & 7u) : (r >> 3) + 4u * (r & 7u);
}

// A warp writes the piece in its strip to the output: sectors 0..3 of each of its rows' pieces, those of them that lie
// within columns [lo, hi) of the piece.  r0: address of row lane / 8 at the piece's first column;
// pitch: bytes of a row.  A lane has half a sector, eight lanes the 128 bytes of a row.
template <int E>
__device__ __forceinline__ void store_sectors(uint32_t strip, uint64_t r0, uint32_t pitch, int lo, int hi, int rows, bool odd16, int lane) {
    constexpr int SE = 32 / E;
    const uint32_t j = (uint32_t)lane >> 3, v = (uint32_t)lane & 7u;
    const uint32_t from = strip + (odd16 ? (j & 1u) + 4u * (j >> 1) : 4u * j) * SS_PITCH + 16u * v;
    const uint32_t o1 = (odd16 ? 8u : 16u) * SS_PITCH, o2 = (odd16 ? 16u : 1u) * SS_PITCH;  // slots of rows r + 4, r + 8 less that of r
    const uint64_t step = 4ull * pitch, voff = 16u * v;
#pragma unroll 1
    for (int t = 0; t < rows; t += 16) {
        uint4 w[4];
        const uint32_t at = from + (uint32_t)t * (SS_PITCH / 8);
        w[0] = lds_v4(at);
        w[1] = lds_v4(at + o1);
        w[2] = lds_v4(at + o2);
        w[3] = lds_v4(at + o1 + o2);
#pragma unroll
        for (int i = 0; i < 4; ++i, r0 += step) {
            const int x = SE * (int)(v >> 1) - (int)(((uint32_t)r0 & 31u) / E);  // first column of the sector
            stg_v4_if((r0 & ~31ull) + voff, w[i], x >= lo && x + SE <= hi && t + 4 * i + (int)j < rows);
        }
    }
}
// The same for the whole piece of 32 rows of at most SS_NEAR bytes: the lane's part of row lane / 8 + 4 i goes `goes[i]` bytes past
// origin.
__device__ __forceinline__ void store_sectors_all(uint32_t from, uint32_t o1, uint32_t o2, uint64_t origin, const uint32_t (&goes)[8]) {
#pragma unroll
    for (int t = 0; t < 8; t += 4) {
        uint4 w[4];
        const uint32_t at = from + (uint32_t)t * (SS_PITCH / 2);
        w[0] = lds_v4(at);
        w[1] = lds_v4(at + o1);
        w[2] = lds_v4(at + o2);
        w[3] = lds_v4(at + o1 + o2);
#pragma unroll
        for (int i = 0; i < 4; ++i) stg_v4(origin + goes[t + i], w[i]);
    }
}
// Element i of a strip row (32-byte aligned base `from`), to p.
template <int E>
__device__ __forceinline__ void store_element(uint64_t p, uint32_t from, bool ok) {
    if constexpr (E == 4) {
        uint32_t v;
        asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(v) : "r"(from));
        asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n @q st.global.b32 [%0], %1;\n}\n" ::"l"(p), "r"(v), "r"((int)ok) : "memory");
    } else {
        uint16_t v;
        asm volatile("ld.shared.b16 %0, [%1];\n" : "=h"(v) : "r"(from));
        asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %2, 0;\n @q st.global.b16 [%0], %1;\n}\n" ::"l"(p), "h"(v), "r"((int)ok) : "memory");
    }
}
// The sector in which a row ends (its first n bytes, at `end` in shared memory) and the next row begins (`begin`), to p.
__device__ __forceinline__ void store_joint(uint64_t p, uint32_t end, uint32_t begin, uint32_t n, bool ok) {
#pragma unroll
    for (uint32_t h = 0; h < 32; h += 16) {
        const uint4 x = lds_v4(end + h), y = lds_v4(begin + h);
        auto pick = [&](uint32_t a, uint32_t b, uint32_t at) {  // bytes [at, at + 4) of the sector
            return n >= at + 4 ? a : n > at ? __byte_perm(a, b, 0x7610) : b;  // (an end inside a word leaves half of it)
        };
        stg_v4_if(p + h, make_uint4(pick(x.x, y.x, h), pick(x.y, y.y, h + 4), pick(x.z, y.z, h + 8), pick(x.w, y.w, h + 12)), ok);
    }
}

template <typename Tag, bool OUT32, bool SOFT, int KB>
__global__ void __launch_bounds__(SL<KB>::THREADS, 1)
blk_scores_umma_kernel(const BlkUmmaParams p, const __grid_constant__ UmMaps maps) {
    using L = SL<KB>;
    constexpr int S = L::S;
    extern __shared__ __align__(1024) unsigned char ss_smem_raw[];  // the swizzled tiles need a 1024-byte aligned base
    unsigned char* smem = ss_smem_raw;
    if (blk_smem_u32(smem) & 1023u) {  // cannot happen with the alignment above; checked because the swizzle relies on it
        if (threadIdx.x == 0) atomicCAS(p.status, 0, 9);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t smem_u32 = blk_smem_u32(smem);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::BAR_OFF + S * 128);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    // The stream of this warp: epilogue warps 0..4S-1, then producers and MMA warps (with S = 3 two warps have nothing to do).
    const bool epi = warp < 4 * S;
    const int s = epi ? warp >> 2 : (warp - 4 * S) & 3;
    const uint32_t bar0 = smem_u32 + L::BAR_OFF + 128u * (uint32_t)s;
    auto b_full = [&](uint32_t u) { return bar0 + 8u * (u % L::UNITS); };
    auto b_empty = [&](uint32_t u) { return bar0 + 8u * (3u + u % L::UNITS); };
    const uint32_t a_full = bar0 + 48u, a_empty = bar0 + 56u;
    auto acc_full = [&](uint32_t t) { return bar0 + 64u + 8u * (t & 1u); };
    auto acc_empty = [&](uint32_t t) { return bar0 + 80u + 8u * (t & 1u); };
    auto rec_full = [&](uint32_t n) { return bar0 + 96u + 8u * (n & 1u); };
    auto rec_empty = [&](uint32_t n) { return bar0 + 112u + 8u * (n & 1u); };
    Rec* const recs = reinterpret_cast<Rec*>(smem + L::REC_OFF) + 2 * s;
    const uint32_t sA = smem_u32 + (uint32_t)(s * L::STREAM_BYTES);
    auto sB = [&](uint32_t u) { return sA + (uint32_t)(KB * SS_A_BYTES) + u % L::UNITS * SS_UNIT; };

    if (threadIdx.x == 0) {
        for (int t = 0; t < S; ++t) {
            const uint32_t b = smem_u32 + L::BAR_OFF + 128u * (uint32_t)t;
            for (uint32_t i = 0; i < 16; ++i) mbar_init(b + 8u * i, i < 10 ? 1u : i < 12 ? 4u : i < 14 ? 1u : 5u);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 4 * S) {
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
    const uint32_t tmem_s = tmem_base + 128u * (uint32_t)s;  // the stream's two accumulators
    const uint32_t lim = p.spin_limit ? p.spin_limit : BLK_UMMA_SPIN_LIMIT;
    // Whether an item's tiles stay in the accumulators between the sweeps of its softmax.
    auto stays = [](int N) { return SOFT && N <= 2 * SS_BN; };

    if (!epi) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(L::REGS_OTHER));
        const bool producer = warp - 4 * S < 4;
        if (s < S && elect_one()) {
            if (producer) {
                // ---------------- producer ----------------
                if (!p.stall) {
                    // item n of the stream: all streams of the grid take items in turn, odd rounds backwards, so that with the
                    // items sorted by cost no stream always gets the heaviest of a round
                    const uint32_t G = gridDim.x * (uint32_t)S, g = blockIdx.x + (uint32_t)s * gridDim.x;
                    BlkUmmaItem it{}, nx{};
                    int head = 0, nhead = 0;
                    bool have = fetch_item(p, 0, G, g, it, head), ok = true;
                    uint32_t u = 0;
#pragma unroll 1
                    for (uint32_t n = 0; ok; ++n) {
                        const bool nhave = have && fetch_item(p, n + 1u, G, g, nx, nhead);
                        if (!mbar_wait(rec_empty(n), ((n >> 1) & 1u) ^ 1u, abort_flag, 12, lim)) break;
                        const int rec_rows = item_rows(it, n + (uint32_t)s);
                        Rec r{};
                        if (have) {
                            r.cbase = (int64_t)head * p.Dout + it.offC + (int64_t)it.tm * 128 * it.N;
                            r.rows = rec_rows;
                            r.N = it.N;
                            r.K = it.K;
                            r.valid = 1;
                        }
                        recs[n & 1u] = r;
                        mbar_arrive(rec_full(n));  // release: the record is visible to whoever sees the phase end
                        if (!have) break;
                        const int K = it.K, N = it.N, kbs = (K + SS_BK - 1) / SS_BK, tiles = (N + SS_BN - 1) / SS_BN;
                        const int total = SOFT && !stays(N) ? 2 * tiles : tiles;
                        const int a0 = 32 * (rec_rows >> 8), a1 = a0 + (rec_rows & 255), rA = it.rowA - a0;
                        const CUtensorMap *mapA = &maps.a[it.views & 255], *mapB = &maps.b[it.views >> 8];
                        // coordinates (k, row, head), or (k, head, row) for a token-major operand
                        int j = 0;
#pragma unroll 1
                        for (int t = 0; ok && t < total; ++t) {
                            const int rB = it.rowB + j * SS_BN;
                            if (++j == tiles) j = 0;
#pragma unroll 1
                            for (int kb = 0; kb < kbs; ++kb, ++u) {
                                if (!mbar_wait(b_empty(u), ((u / L::UNITS) & 1u) ^ 1u, abort_flag, 1, lim)) { ok = false; break; }
                                mbar_expect_tx(b_full(u), SS_UNIT);
                                tma_load_3d(sB(u), mapB, b_full(u), kb * SS_BK, p.head_firstB ? head : rB, p.head_firstB ? rB : head);
                            }
                            if (t == 0 && ok) {
                                // the block of the first operand, behind the first tile: its place is free later
                                if (!mbar_wait(a_empty, (n & 1u) ^ 1u, abort_flag, 2, lim)) { ok = false; break; }
                                const int b0 = a0 / SS_BOX, b1 = (a1 + SS_BOX - 1) / SS_BOX;
                                mbar_expect_tx(a_full, (uint32_t)(kbs * (b1 - b0)) * (SS_BOX * 128));
#pragma unroll 1
                                for (int kb = 0; kb < kbs; ++kb)
#pragma unroll 1
                                    for (int b = b0; b < b1; ++b)
                                        tma_load_3d(sA + kb * SS_A_BYTES + b * (SS_BOX * 128), mapA, a_full, kb * SS_BK,
                                                    p.head_firstA ? head : rA + b * SS_BOX, p.head_firstA ? rA + b * SS_BOX : head);
                            }
                        }
                        it = nx;
                        head = nhead;
                        have = nhave;
                    }
                }
            } else {
                // ---------------- MMA issue ----------------
                const uint32_t idesc0 = instr_desc(p.bf16, 0, SOFT && p.scale < 0.f);
                uint32_t u = 0, acc = 0;  // units, accumulators so far
                bool ok = true;
#pragma unroll 1
                for (uint32_t n = 0; ok; ++n) {
                    if (!mbar_wait(rec_full(n), (n >> 1) & 1u, abort_flag, 11, lim)) break;
                    const Rec& r = recs[n & 1u];
                    const int N = r.N, K = r.K, valid = r.valid;
                    mbar_arrive(rec_empty(n));
                    if (!valid) break;
                    const int tiles = (N + SS_BN - 1) / SS_BN, total = SOFT && !stays(N) ? 2 * tiles : tiles;
                    if (!mbar_wait(a_full, n & 1u, abort_flag, 3, lim)) break;
                    int left = N;
#pragma unroll 1
                    for (int t = 0; t < total; ++t, ++acc) {
                        const uint32_t idesc = idesc0 | ((uint32_t)((min(left, SS_BN) + 15) >> 4) << 18);  // columns in units of 16
                        left -= SS_BN;
                        if (left <= 0) left = N;
                        const uint32_t d_tmem = tmem_s + (uint32_t)SS_BN * (acc & 1u);
                        if (!mbar_wait(acc_empty(acc), ((acc >> 1) & 1u) ^ 1u, abort_flag, 4, lim)) { ok = false; break; }
#pragma unroll 1
                        for (int krem = K, kb = 0; krem > 0; krem -= SS_BK, ++kb, ++u) {
                            const uint64_t da = smem_desc_sw128(sA + kb * SS_A_BYTES), db = smem_desc_sw128(sB(u));
                            if (!mbar_wait(b_full(u), (u / L::UNITS) & 1u, abort_flag, 5, lim)) { ok = false; break; }
                            tc_fence_after();
                            // steps of 16 along k in this block: all four, or as many as reach the end of a short last block
                            // (the tensor map fills what lies past K with zeros)
                            if (krem > SS_BK - 16) {
#pragma unroll
                                for (int i = 0; i < SS_BK / 16; ++i)
                                    tc_mma_f16(d_tmem, da + (uint64_t)(2 * i), db + (uint64_t)(2 * i), idesc, i ? 1u : (uint32_t)kb);
                            } else {
#pragma unroll 1
                                for (int i = 0; 16 * i < krem; ++i)
                                    tc_mma_f16(d_tmem, da + (uint64_t)(2 * i), db + (uint64_t)(2 * i), idesc, (uint32_t)(kb | i));
                            }
                            tc_commit(b_empty(u));  // the unit is reusable once these products have read it
                        }
                        if (!ok) break;
                        tc_commit(acc_full(acc));
                        if (t == total - 1) tc_commit(a_empty);
                    }
                }
            }
        }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(L::REGS_EPI));
        // ---------------- epilogue ----------------
        constexpr int E = OUT32 ? 4 : 2, PC = 128 / E, SE = 32 / E;  // bytes of an element, columns of a piece, elements of a sector
        const int q = warp & 3;
        const uint32_t lane_addr = tmem_s + ((uint32_t)(q * 32) << 16);
        const uint32_t strip = smem_u32 + L::STRIP_OFF + (uint32_t)warp * SS_STRIP_BYTES;
        const float sl = SOFT ? fabsf(p.scale) * BLK_LOG2E : p.scale;  // a negative softmax scale is applied by the MMA (negated A)
        const float2 sl2 = make_float2(sl, sl);
        uint32_t acc = 0;  // accumulators so far
        bool ok = true;
        uint32_t ra[32], rb[32];  // a tile's columns of this thread's row

        auto acc_wait = [&](uint32_t t) -> bool {
            const bool good = mbar_wait(acc_full(t), (t >> 1) & 1u, abort_flag, 6, lim);
            tc_fence_after();
            return good;
        };
        auto acc_release = [&](uint32_t t) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(t));
        };
        auto load = [&](uint32_t t) {
            tc_ld32_nowait(lane_addr + (uint32_t)SS_BN * (t & 1u), ra);
            tc_ld32_nowait(lane_addr + (uint32_t)SS_BN * (t & 1u) + 32u, rb);
            tc_ld_wait(ra);
            tc_ld_wait(rb);
        };

#pragma unroll 1
        for (uint32_t n = 0; ok; ++n) {
            if (!mbar_wait(rec_full(n), (n >> 1) & 1u, abort_flag, 11, lim)) break;
            const Rec& r = recs[n & 1u];
            const int N = r.N, rec_rows = r.rows, valid = r.valid;
            const int r0 = (q - (rec_rows >> 8)) * 32;  // row of the block that this warp's first lane holds
            const uint64_t base = reinterpret_cast<uint64_t>(p.C) + (uint64_t)((r.cbase + (int64_t)r0 * N) * E);
            __syncwarp();
            if (lane == 0) mbar_arrive(rec_empty(n));
            if (!valid) break;
            const int rows = min((rec_rows & 255) - r0, 32);
            const int tiles = (N + SS_BN - 1) / SS_BN;
            const bool here = r0 >= 0 && rows > 0, stay = stays(N);
            if (!here) {  // none of this warp's rows exist: it only hands the accumulators back
                for (int t = SOFT && !stay ? 2 * tiles : tiles; t > 0; --t, ++acc) {
                    if (!acc_wait(acc)) { ok = false; break; }
                    acc_release(acc);
                }
                continue;
            }
            float2 off2 = make_float2(0.f, 0.f), inv2 = off2;
            if constexpr (SOFT) {
                // first sweep: reference and sum of exp2((x - reference) sl)
                float ref = -INFINITY, sum = 0.f;
                int cols = N;
#pragma unroll 1
                for (int t = 0; t < tiles; ++t, cols -= SS_BN) {
                    if (!acc_wait(acc + (uint32_t)t)) { ok = false; break; }
                    load(acc + (uint32_t)t);
                    if (!stay) acc_release(acc + (uint32_t)t);
                    if (cols < SS_BN) {  // (a branch: as selects this would cost every tile 64 instructions)
                        asm volatile("");
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            if (i >= cols) ra[i] = 0xff800000u;  // -inf
                            if (32 + i >= cols) rb[i] = 0xff800000u;
                        }
                    }
                    float m4[4] = {ref, __uint_as_float(ra[0]), __uint_as_float(ra[1]), __uint_as_float(ra[2])};
#pragma unroll
                    for (int i = 0; i < 32; i += 8)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            m4[e] = blk_max3(m4[e], __uint_as_float(ra[i + 2 * e]), __uint_as_float(ra[i + 2 * e + 1]));
                            m4[e] = blk_max3(m4[e], __uint_as_float(rb[i + 2 * e]), __uint_as_float(rb[i + 2 * e + 1]));
                        }
                    const float m = fmaxf(blk_max3(m4[0], m4[1], m4[2]), m4[3]);
                    if ((m - ref) * sl > SS_LAZY) {  // always at the first tile (ref = -inf)
                        if (t) sum *= blk_exp2((ref - m) * sl);
                        ref = m;
                    }
                    const float nm = ref == -INFINITY ? 0.f : -ref * sl;
                    const float2 nm2 = make_float2(nm, nm);
                    float2 s2[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float2 x = blk_fma2(make_float2(__uint_as_float(ra[i]), __uint_as_float(ra[i + 1])), sl2, nm2);
                        float2 y = blk_fma2(make_float2(__uint_as_float(rb[i]), __uint_as_float(rb[i + 1])), sl2, nm2);
                        x.x = blk_exp2(x.x);
                        x.y = blk_exp2(x.y);
                        y.x = blk_exp2(y.x);
                        y.y = blk_exp2(y.y);
                        s2[i & 2] = blk_add2(s2[i & 2], x);
                        s2[(i & 2) + 1] = blk_add2(s2[(i & 2) + 1], y);
                    }
                    const float2 sa = blk_add2(blk_add2(s2[0], s2[1]), blk_add2(s2[2], s2[3]));
                    sum += sa.x + sa.y;
                }
                if (!ok) break;
                if (!stay) acc += (uint32_t)tiles;
                // exp2(x sl + off) / sum with the offset that the sum was made with: its rounding, which is that of the scores' own
                // size, is the same for both and cancels.  (With the sum's logarithm in the offset it does not: up to 7e-4 of a
                // probability for scores of 20000, more than the rounding of a half.  A choice between the two by the size of the
                // offset took as long as the division always.)
                const float off = ref == -INFINITY ? 0.f : -ref * sl, inv = __frcp_rn(sum);
                inv2 = make_float2(inv, inv);
                off2 = make_float2(off, off);
            }
            // the storing sweep
            const uint64_t pitch = (uint64_t)N * E;
            uint64_t own = base + (uint64_t)lane * pitch;                  // this lane's row ...
            uint64_t quarter = base + (uint64_t)(lane >> 3) * pitch;       // ... and row lane / 8, at the piece's first column
            // where this lane's halves of sectors go: in the first row, and the bytes from there to rows lane / 8 + 4 i, which fit 32
            // bits for rows that are not longer than SS_NEAR (others take the general way out; offsets counted in sectors, for rows
            // of any length, took 714.5 us for the softmax of 512 segments of 16..2048 rows where this takes 710.5)
            const bool near = pitch <= SS_NEAR;
            uint64_t origin = (base & ~31ull) + 16u * ((uint32_t)lane & 7u);
            uint32_t goes[8];
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) goes[i] = ((uint32_t)base & 31u) + ((uint32_t)(lane >> 3) + 4u * i) * (uint32_t)pitch & ~31u;
            const uint32_t phase = (uint32_t)own & 31u;                    // how far into a sector the row starts
            const bool odd16 = !OUT32 && (N & 1);
            const bool anyodd = !OUT32 && __any_sync(0xffffffffu, (int)(phase & 2u));
            const bool shifted = __any_sync(0xffffffffu, (int)phase);
            const bool vectors = !__any_sync(0xffffffffu, (int)(phase & 15u));
            const uint32_t srow = strip + strip_slot((uint32_t)lane, odd16) * SS_PITCH, swords = srow + (phase & 28u);
            const uint32_t heads = strip + SS_HEADS, par = (phase & 2u) << 3;
            // this lane's part of a whole piece in the strip
            const uint32_t lj = (uint32_t)lane >> 3;
            const uint32_t from = strip + (odd16 ? (lj & 1u) + 4u * (lj >> 1) : 4u * lj) * SS_PITCH + 16u * ((uint32_t)lane & 7u);
            const uint32_t o1 = (odd16 ? 8u : 16u) * SS_PITCH, o2 = (odd16 ? 16u : 1u) * SS_PITCH;
            uint32_t prev = 0;
            uint32_t rest[8];  // the last words of a piece
            auto xform = [&](float2 v) {
                if constexpr (!SOFT) return blk_mul2(v, sl2);
                const float2 t = blk_fma2(v, sl2, off2);
                return blk_mul2(make_float2(blk_exp2(t.x), blk_exp2(t.y)), inv2);
            };
            // 32 columns (16 words, fp32: 32) to words at of the strip row
            auto stage = [&](const uint32_t (&v)[32], uint32_t at) {
                uint32_t w[OUT32 ? 32 : 16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float2 y = xform(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])));
                    if constexpr (OUT32) {
                        w[2 * i] = __float_as_uint(y.x);
                        w[2 * i + 1] = __float_as_uint(y.y);
                    } else {
                        w[i] = BlkCvt<Tag>::pack2(y.x, y.y);
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) rest[i] = w[(OUT32 ? 24 : 8) + i];
                if (vectors) {
#pragma unroll
                    for (int i = 0; i < (OUT32 ? 32 : 16); i += 4) tc_sts_v4(at + 4 * i, w[i], w[i + 1], w[i + 2], w[i + 3]);
                } else if (OUT32 || !anyodd) {
#pragma unroll
                    for (int i = 0; i < (OUT32 ? 32 : 16); ++i) blk_sts_b32(at + 4 * i, w[i]);
                } else {
                    // a row that starts on an odd element is shifted by half a word
#pragma unroll
                    for (int i = 0; i < (OUT32 ? 0 : 16); ++i) {
                        const uint32_t x = __funnelshift_l(prev, w[i], par);
                        blk_sts_b32(at + 4 * i, x);
                        prev = w[i];
                        if (i >= 8) rest[i - 8] = x;
                    }
                }
            };
            // the staged piece, cols columns of it, goes out
            auto flush = [&](int cols, bool first, bool last) {
                __syncwarp();
                if (N < SE) {  // several rows in a sector: element by element, in the order of the output
#pragma unroll 1
                    for (int i = lane; i < rows * N; i += 32) {
                        const int k = i / N;
                        const uint64_t at = base + (uint64_t)i * E;
                        store_element<E>(at, strip + strip_slot((uint32_t)k, odd16) * SS_PITCH + ((uint32_t)(base + (uint64_t)k * pitch) & 31u) + (uint32_t)((i - k * N) * E), true);
                    }
                    __syncwarp();
                    return;
                }
                if (near && rows == 32 && cols >= PC && !(first && shifted))
                    store_sectors_all(from, o1, o2, origin, goes);
                else
                    store_sectors<E>(strip, quarter, (uint32_t)pitch, first ? 0 : -SE, cols, rows, odd16, lane);
                if (shifted) {
                    if (first) {  // the sector a row begins in waits for the end of the row before; the first row's has none
                        const uint4 x = lds_v4(srow), y = lds_v4(srow + 16u);
                        tc_sts_v4(heads + 32u * lane, x.x, x.y, x.z, x.w);
                        tc_sts_v4(heads + 32u * lane + 16u, y.x, y.y, y.z, y.w);
                        const int a0 = (int)((uint32_t)base & 31u) / E;
                        __syncwarp();
                        if (a0) store_element<E>((base & ~31ull) + (uint64_t)(lane * E), heads + (uint32_t)(lane * E) % 32u, lane >= a0 && lane < SE);
                    }
                    if (last) {
                        const uint32_t end = phase + (uint32_t)(cols * E), n = end & 31u;  // the row's end in the strip
                        store_joint(own - phase + (end & ~31u), srow + (end & ~31u), heads + 32u * min(lane + 1, 31), n, n && lane < rows - 1);
                        // the last row's end
                        const uint64_t at = own + (uint64_t)(cols * E);
                        const uint32_t nl = __shfl_sync(0xffffffffu, n, rows - 1), from = __shfl_sync(0xffffffffu, srow + (end & ~31u), rows - 1);
                        const uint64_t to = __shfl_sync(0xffffffffu, at, rows - 1) & ~31ull;
                        if (nl) store_element<E>(to + (uint64_t)(lane * E), from + (uint32_t)(lane * E) % 32u, lane * E < (int)nl);
                    }
                    __syncwarp();
                    if (!last) {  // what does not fill a sector yet goes in front of the next piece
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (8u - (uint32_t)i <= (phase >> 2)) blk_sts_b32(swords + 4 * i - 32, rest[i]);
                    }
                } else {
                    __syncwarp();
                }
                own += 128u;
                quarter += 128u;
                origin += 128u;
            };
            int cols = N;
#pragma unroll 1
            for (int t = 0; t < tiles; ++t, ++acc, cols -= SS_BN) {
                if (!(SOFT && stay) && !acc_wait(acc)) { ok = false; break; }
                load(acc);
                acc_release(acc);
                if constexpr (OUT32) {
                    stage(ra, swords);
                    flush(min(cols, PC), t == 0, cols <= PC);
                    if (cols > PC) {
                        stage(rb, swords);
                        flush(min(cols - PC, PC), false, cols <= 2 * PC);
                    }
                } else {
                    stage(ra, swords);
                    if (cols > 32) stage(rb, swords + 64u);
                    if (anyodd && cols <= SS_BN) blk_sts_b32(swords + (cols > 32 ? 128u : 64u), prev >> 16);
                    flush(min(cols, PC), t == 0, cols <= PC);
                }
            }
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before();
    __syncthreads();
    wait_report(abort_flag, p.status);
    if (warp == 4 * S) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512));
    }
}

template <typename Tag, bool OUT32, bool SOFT, int KB>
cudaError_t launch(const BlkUmmaParams& p, const UmMaps& maps, int sms, cudaStream_t st) {
    using L = SL<KB>;
    auto kern = blk_scores_umma_kernel<Tag, OUT32, SOFT, KB>;
    cudaError_t e = blk_func_smem(reinterpret_cast<const void*>(kern), L::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const int64_t total = (int64_t)p.num_items * p.H;
    const dim3 grid((unsigned)(total < sms ? total : sms)), block(L::THREADS);
    return blk_launch(total <= 24 * (int64_t)sms, kern, grid, block, L::SMEM_BYTES, st, p, maps);
}

}  // namespace

cudaError_t blk_launch_scores_umma(const BlkUmmaParams& p_in, const BlkUmmaOperand& A, const BlkUmmaOperand& B, int sms,
                                   cudaStream_t st) {
    BlkUmmaParams p = p_in;
    static thread_local UmMaps maps;  // kilobytes: not on the stack of a caller's thread
    if (!blk_umma_maps(p, A, B, SS_BOX, SS_BOX, maps)) return cudaErrorInvalidValue;
    int64_t K = 0;
    for (int i = 0; i < A.num_views; ++i) K = A.views[i].K > K ? A.views[i].K : K;
    if (K > (p.epi == BLK_EPI_SOFTMAX ? BLK_STREAM_MAXK / 2 : BLK_STREAM_MAXK)) return cudaErrorInvalidValue;
    auto run = [&](auto tag) {
        typedef decltype(tag) Tag;
        if (K <= SS_BK) {
            if (p.epi == BLK_EPI_SOFTMAX) return p.out_f32 ? launch<Tag, true, true, 1>(p, maps, sms, st) : launch<Tag, false, true, 1>(p, maps, sms, st);
            return p.out_f32 ? launch<Tag, true, false, 1>(p, maps, sms, st) : launch<Tag, false, false, 1>(p, maps, sms, st);
        }
        return p.out_f32 ? launch<Tag, true, false, 2>(p, maps, sms, st) : launch<Tag, false, false, 2>(p, maps, sms, st);
    };
    return p.bf16 ? run(BlkBf16Tag{}) : run(BlkHalfTag{});
}

// Backward of the fused attention for segments of at most 64 query and 64 key rows, head dimension 64 or 128: one CTA per
// (segment, head), everything in shared memory and registers.
//
// Such a segment is a few 16-row blocks: a 128-row tcgen05 tile would be mostly padding (25 rows on average in a molecular
// batch), so the products run on mma.sync m16n8k16, whose work grows in steps of 16 rows.  The kernel is bound by memory
// (q, k, v, dO in, dQ, dK, dV out); what hides the latency is many small CTAs per SM: 2 warps and 23 KB for segments of at
// most 32 rows at d = 64 (nine CTAs per SM), 4 warps for up to 64 rows.
//
//   phase 1  a warp per 16-row block of the queries: S = Q K^T and dP = dO V^T in registers, the softmax and
//            rowsum(P dP) over whole rows (no saved statistics needed), dS = P (dP - rowsum), dQ = scale dS K;
//            P and dS, rounded to the input type, go to shared memory
//   phase 2  a warp per 16-row block of the keys and output: dV = P^T dO, dK = scale dS^T Q (transposing ldmatrix loads)
//
// Rows past the end of a segment are zero-filled while loading (cp.async with a short source), so they add nothing.
// Upstream differentiates the chain blockGEMM -> blockSoftmax -> blockGEMM operator by operator
// (csrc/sparseBlockedAttention.cpp:52-72, :103-114).
#include "blk_device.cuh"
#include "blk_kernels.h"

namespace {

template <int D, int R>
struct SB {
    static constexpr int PITCH = D * 2 + 16;        // bytes; an odd number of 16-byte units: ldmatrix rows hit different banks
    static constexpr int PPITCH = R * 2 + 16;
    static constexpr int OPER = R * PITCH;          // one operand
    static constexpr int P_OFF = 4 * OPER, S_OFF = P_OFF + R * PPITCH;
    static constexpr int SMEM = S_OFF + R * PPITCH;
    static constexpr int WARPS = R / 16;
};

template <typename Tag>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    blk_mma16816<Tag>(d, a[0], a[1], a[2], a[3], b0, b1);
}
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// Rows g and g + 8 of a 16 x D accumulator, times f, to base (row pitch D): two neighbouring 8-column tiles are traded
// between neighbouring lanes so that a row's 16 columns leave as four 8-byte stores, a whole 32-byte sector.
template <typename Tag, int D>
__device__ __forceinline__ void store_rows(uint16_t* base, const float (&o)[D / 8][4], float f, int rows, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const bool odd = t & 1;
#pragma unroll
    for (int j = 0; j < D / 8; j += 2)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t lo = BlkCvt<Tag>::pack2(o[j][2 * h] * f, o[j][2 * h + 1] * f);
            const uint32_t hi = BlkCvt<Tag>::pack2(o[j + 1][2 * h] * f, o[j + 1][2 * h + 1] * f);
            const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
            // even lanes: columns 2 t .. 2 t + 3 of tile j; odd lanes: columns 2 t - 2 .. 2 t + 1 of tile j + 1
            const uint2 v = odd ? make_uint2(got, hi) : make_uint2(lo, got);
            const int row = g + 8 * h, col = 8 * (j + (odd ? 1 : 0)) + 2 * (t & 2);
            if (row < rows) *reinterpret_cast<uint2*>(base + (int64_t)row * D + col) = v;
        }
}

template <typename Tag, int D, int R>
__global__ void __launch_bounds__(SB<D, R>::WARPS * 32)
blk_attn_bwd_small_kernel(const BlkAttnBwdSmallParams p) {
    using L = SB<D, R>;
    extern __shared__ __align__(128) unsigned char sb_smem[];
    const uint32_t sm = blk_smem_u32(sb_smem);
    const uint32_t sQ = sm, sK = sm + L::OPER, sV = sm + 2 * L::OPER, sG = sm + 3 * L::OPER, sP = sm + L::P_OFF, sS = sm + L::S_OFF;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t unit = blockIdx.x, item = unit / (uint32_t)p.H;
    const int head = (int)(unit - item * (uint32_t)p.H);
    const BlkFlashItem it = p.items[item];
    blk_grid_wait();
    const int M = it.M, N = it.N, Mb = (M + 15) >> 4, Nb = (N + 15) >> 4;
    const int64_t offQ = ((int64_t)head * p.rows_q + it.rowQ) * D, offK = ((int64_t)head * p.rows_kv + it.rowKV) * D;

    // ---- operands: 16-byte pieces, rows up to the next multiple of 16 (zeros past the end) ----
    constexpr int CH = D / 8;
    for (int i = tid; i < Mb * 16 * CH; i += L::WARPS * 32) {
        const int r = i / CH, c = i % CH;
        const int64_t src = offQ + (int64_t)(r < M ? r : 0) * D + c * 8;
        cp16(sQ + r * L::PITCH + c * 16, p.q + src, r < M);
        cp16(sG + r * L::PITCH + c * 16, p.g + src, r < M);
    }
    for (int i = tid; i < Nb * 16 * CH; i += L::WARPS * 32) {
        const int r = i / CH, c = i % CH;
        const int64_t src = offK + (int64_t)(r < N ? r : 0) * D + c * 8;
        cp16(sK + r * L::PITCH + c * 16, p.k + src, r < N);
        cp16(sV + r * L::PITCH + c * 16, p.v + src, r < N);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();

    const int g = lane >> 2, t = lane & 3;
    // lane addresses inside a 16 x 16 tile: first operand (and B with trans: rows of the contraction), second operand
    const int la_row = lane & 15, la_col = (lane >> 4) * 8;                                    // A[m][k]; x4: m lo/hi, then k hi
    const int lb_row = (lane & 7) + ((lane >> 4) & 1) * 8, lb_col = ((lane >> 3) & 1) * 8;      // B[n][k]; x4: k lo/hi of tile 0, of tile 1
    const int lt_row = (lane & 7) + ((lane >> 3) & 1) * 8, lt_col = ((lane >> 4) & 1) * 8;      // B[k][n] transposed
    const int lp_row = (lane & 7) + ((lane >> 4) & 1) * 8, lp_col = ((lane >> 3) & 1) * 8;      // A[k][m] transposed

    // ---- phase 1 ----
    if (warp < Mb) {
        const int r0 = warp * 16;
        float s[R / 8][4], dp[R / 8][4];
#pragma unroll
        for (int j = 0; j < R / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[j][e] = dp[j][e] = 0.f;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
            uint32_t a[4], c[4];
            blk_ldmatrix_x4(a, sQ + (r0 + la_row) * L::PITCH + (ks * 16 + la_col) * 2);
            blk_ldmatrix_x4(c, sG + (r0 + la_row) * L::PITCH + (ks * 16 + la_col) * 2);
#pragma unroll
            for (int jp = 0; jp < R / 16; ++jp)
                if (jp < Nb) {
                    uint32_t b[4];
                    blk_ldmatrix_x4(b, sK + (jp * 16 + lb_row) * L::PITCH + (ks * 16 + lb_col) * 2);
                    mma16816<Tag>(s[2 * jp], a, b[0], b[1]);
                    mma16816<Tag>(s[2 * jp + 1], a, b[2], b[3]);
                    blk_ldmatrix_x4(b, sV + (jp * 16 + lb_row) * L::PITCH + (ks * 16 + lb_col) * 2);
                    mma16816<Tag>(dp[2 * jp], c, b[0], b[1]);
                    mma16816<Tag>(dp[2 * jp + 1], c, b[2], b[3]);
                }
        }
        const float sl = p.scale * BLK_LOG2E;
        float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
        for (int j = 0; j < R / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s[j][e] = 8 * j + 2 * t + (e & 1) < N ? s[j][e] * sl : -INFINITY;
                if (e < 2) m0 = fmaxf(m0, s[j][e]);
                else m1 = fmaxf(m1, s[j][e]);
            }
        m0 = blk_quad_max(m0);
        m1 = blk_quad_max(m1);
        float l0 = 0.f, l1 = 0.f;
#pragma unroll
        for (int j = 0; j < R / 8; ++j) {
            s[j][0] = blk_exp2(s[j][0] - m0); s[j][1] = blk_exp2(s[j][1] - m0);
            s[j][2] = blk_exp2(s[j][2] - m1); s[j][3] = blk_exp2(s[j][3] - m1);
            l0 += s[j][0] + s[j][1];
            l1 += s[j][2] + s[j][3];
        }
        const float i0 = __frcp_rn(blk_quad_sum(l0)), i1 = __frcp_rn(blk_quad_sum(l1));
        float d0 = 0.f, d1 = 0.f;
#pragma unroll
        for (int j = 0; j < R / 8; ++j) {
            s[j][0] *= i0; s[j][1] *= i0; s[j][2] *= i1; s[j][3] *= i1;
            d0 += s[j][0] * dp[j][0] + s[j][1] * dp[j][1];
            d1 += s[j][2] * dp[j][2] + s[j][3] * dp[j][3];
        }
        d0 = blk_quad_sum(d0);
        d1 = blk_quad_sum(d1);
        uint32_t ds[R / 8][2];
#pragma unroll
        for (int j = 0; j < R / 8; ++j) {
            ds[j][0] = BlkCvt<Tag>::pack2(s[j][0] * (dp[j][0] - d0), s[j][1] * (dp[j][1] - d0));
            ds[j][1] = BlkCvt<Tag>::pack2(s[j][2] * (dp[j][2] - d1), s[j][3] * (dp[j][3] - d1));
            if (j < 2 * Nb) {
                const uint32_t at = (uint32_t)((r0 + g) * L::PPITCH + (8 * j + 2 * t) * 2);
                blk_sts_b32(sP + at, BlkCvt<Tag>::pack2(s[j][0], s[j][1]));
                blk_sts_b32(sP + at + 8 * L::PPITCH, BlkCvt<Tag>::pack2(s[j][2], s[j][3]));
                blk_sts_b32(sS + at, ds[j][0]);
                blk_sts_b32(sS + at + 8 * L::PPITCH, ds[j][1]);
            }
        }
        float o[D / 8][4];
#pragma unroll
        for (int j = 0; j < D / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
#pragma unroll
        for (int kk = 0; kk < R / 16; ++kk)
            if (kk < Nb) {
                const uint32_t a[4] = {ds[2 * kk][0], ds[2 * kk][1], ds[2 * kk + 1][0], ds[2 * kk + 1][1]};
#pragma unroll
                for (int n = 0; n < D / 16; ++n) {
                    uint32_t b[4];
                    blk_ldmatrix_x4_trans(b, sK + (kk * 16 + lt_row) * L::PITCH + (n * 16 + lt_col) * 2);
                    mma16816<Tag>(o[2 * n], a, b[0], b[1]);
                    mma16816<Tag>(o[2 * n + 1], a, b[2], b[3]);
                }
            }
        store_rows<Tag, D>(p.dq + offQ + (int64_t)r0 * D, o, p.scale, M - r0, lane);
    }
    __syncthreads();

    // ---- phase 2: jobs (key block, output) ----
    for (int job = warp; job < 2 * Nb; job += L::WARPS) {
        const bool keys = job >= Nb;  // dK, else dV
        const int n0 = (keys ? job - Nb : job) * 16;
        const uint32_t sA = keys ? sS : sP, sB = keys ? sQ : sG;
        float o[D / 8][4];
#pragma unroll
        for (int j = 0; j < D / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
#pragma unroll
        for (int kk = 0; kk < R / 16; ++kk)
            if (kk < Mb) {
                uint32_t a[4];
                blk_ldmatrix_x4_trans(a, sA + (kk * 16 + lp_row) * L::PPITCH + (n0 + lp_col) * 2);
#pragma unroll
                for (int n = 0; n < D / 16; ++n) {
                    uint32_t b[4];
                    blk_ldmatrix_x4_trans(b, sB + (kk * 16 + lt_row) * L::PITCH + (n * 16 + lt_col) * 2);
                    mma16816<Tag>(o[2 * n], a, b[0], b[1]);
                    mma16816<Tag>(o[2 * n + 1], a, b[2], b[3]);
                }
            }
        store_rows<Tag, D>((keys ? p.dk : p.dv) + offK + (int64_t)n0 * D, o, keys ? p.scale : 1.f, N - n0, lane);
    }
}

template <typename Tag, int D, int R>
cudaError_t launch(const BlkAttnBwdSmallParams& p, cudaStream_t st) {
    auto kern = blk_attn_bwd_small_kernel<Tag, D, R>;
    cudaError_t e = blk_func_smem(reinterpret_cast<const void*>(kern), SB<D, R>::SMEM);
    if (e != cudaSuccess) return e;
    return blk_launch(true, kern, (unsigned)((int64_t)p.num_items * p.H), SB<D, R>::WARPS * 32, SB<D, R>::SMEM, st, p);
}

}  // namespace

cudaError_t blk_launch_attn_bwd_small(const BlkAttnBwdSmallParams& p, int D, int rows, int bf16, cudaStream_t st) {
    if ((int64_t)p.num_items * p.H == 0) return cudaSuccess;
    if ((D != 64 && D != 128) || (rows != 32 && rows != 64)) return cudaErrorInvalidValue;
    if (bf16) {
        if (D == 64) return rows == 32 ? launch<BlkBf16Tag, 64, 32>(p, st) : launch<BlkBf16Tag, 64, 64>(p, st);
        return rows == 32 ? launch<BlkBf16Tag, 128, 32>(p, st) : launch<BlkBf16Tag, 128, 64>(p, st);
    }
    if (D == 64) return rows == 32 ? launch<BlkHalfTag, 64, 32>(p, st) : launch<BlkHalfTag, 64, 64>(p, st);
    return rows == 32 ? launch<BlkHalfTag, 128, 32>(p, st) : launch<BlkHalfTag, 128, 64>(p, st);
}

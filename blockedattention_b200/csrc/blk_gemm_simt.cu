// fp32 path of the varlen blocked GEMM on the CUDA cores: fp32 in, fp32 accumulate in the order of k, fp32 out, either
// operand transposed, any alignment.
//
// A block of 16 x 16 threads has a tile of 128 x 128 (TM = 8: segments of several such tiles) or 64 x 64 (TM = 4), a thread TM x
// TM results of it: rows in runs of four, so that an LDS.128 brings four of the first operand, columns 16 apart, so that
// half a warp stores 64 contiguous bytes.  Steps of 16 along k, double-buffered in shared memory: the next step's operands are
// on their way to registers while this one's products are made, one barrier a step.  Rows of a multiple of four elements that
// start on 16 bytes are loaded as vectors.  Products two at a time (fma.rn.f32x2: the pairs are the rows of a run).
//
// Bound by the FMA units for long contractions (65 % active, a quarter of it for what tiles have past the ends of a segment).
// us, before (64 x 64 tiles for everything, single-buffered, loaded element by element) -> now: 36 products of 256..621 rows
// and columns over 1160, 4 heads, 2465 -> 2025; 27 of 256..882 over 3128 1960 -> 1625; scores of 1146 segments of 1..496 rows with
// their softmax and gradients, K = 64, 1714 -> 1527.
//
// Replaces upstream sparseBlockedGEMM<float,...> (csrc/cuda/spBlkGEMM.cu:120-271).
#include "blk_device.cuh"
#include "blk_kernels.h"

namespace {

constexpr int SBK = 16, SNT = 256;

// This thread's share of a (16 TM rows of the logical operand) x (16 k) tile, by way of registers to s[k][row].  The logical
// operand is (R, K) row-major, or stored (K, R) when TR.
template <int TM, bool TR>
struct Share {
    static constexpr int B = 16 * TM, PITCH = B + 4;
    float v[TM];
    // vec: rows (TR: columns of the stored operand) are a multiple of four elements and start on 16 bytes
    __device__ __forceinline__ void load(const float* g, int R, int K, int r0, int k0, int tid, bool vec) {
        if (vec) {
#pragma unroll
            for (int i = 0; i < TM / 4; ++i) {
                const int r = r0 + (TR ? tid % (B / 4) * 4 : tid / 4 + 64 * i), k = k0 + (TR ? tid / (B / 4) + 1024 / B * i : tid % 4 * 4);
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < R && k < K) x = *reinterpret_cast<const float4*>(g + (TR ? (int64_t)k * R + r : (int64_t)r * K + k));
                v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const int r = r0 + (TR ? tid % B : tid / 16 + 16 * i), k = k0 + (TR ? tid / B + SNT / B * i : tid % 16);
                v[i] = r < R && k < K ? g[TR ? (int64_t)k * R + r : (int64_t)r * K + k] : 0.f;
            }
        }
    }
    __device__ __forceinline__ void store(float (*s)[PITCH], int tid, bool vec) const {
        if (vec) {
#pragma unroll
            for (int i = 0; i < TM / 4; ++i) {
                if (TR) {
                    *reinterpret_cast<float4*>(&s[tid / (B / 4) + 1024 / B * i][tid % (B / 4) * 4]) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[tid % 4 * 4 + e][tid / 4 + 64 * i] = v[4 * i + e];
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < TM; ++i) s[TR ? tid / B + SNT / B * i : tid % 16][TR ? tid % B : tid / 16 + 16 * i] = v[i];
        }
    }
};

template <int TM, bool TA, bool TB>
__global__ void __launch_bounds__(SNT, TM == 8 ? 2 : 4) blk_gemm_simt_kernel(const BlkSimtParams p) {
    constexpr int B = 16 * TM;
    typedef Share<TM, TA> ShA;
    typedef Share<TM, TB> ShB;
    __shared__ __align__(16) float sA[2][SBK][ShA::PITCH];
    __shared__ __align__(16) float sB[2][SBK][ShB::PITCH];
    const int tid = threadIdx.x;
    const int64_t bid = blockIdx.x;
    const int head = (int)(bid / p.num_items);
    const BlkTileItem it = p.items[bid % p.num_items];
    const BlkSeg sd = p.segs[it.seg];
    blk_grid_wait();
    const int64_t baseA = (int64_t)head * p.Dm1 + sd.offA, baseB = (int64_t)head * p.Dm2 + sd.offB;
    const float* gA = p.A + baseA;
    const float* gB = p.B + baseB;
    float* gC = p.C + (int64_t)head * p.Dout + sd.offC;
    const int M = sd.M, N = sd.N, K = sd.K;
    const int m0 = it.tm * B, n0 = it.tn * B;
    const bool vecA = ((baseA | (TA ? M : K)) & 3) == 0, vecB = ((baseB | (TB ? N : K)) & 3) == 0;
    const int ty = tid / 16, tx = tid % 16;  // rows ty * 4 + 64 h + (0..3), columns tx + 16 j

    float2 acc[TM / 2][TM];
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TM; ++j) acc[i][j] = make_float2(0.f, 0.f);

    ShA a;
    ShB b;
    a.load(gA, M, K, m0, 0, tid, vecA);
    b.load(gB, N, K, n0, 0, tid, vecB);
    a.store(sA[0], tid, vecA);
    b.store(sB[0], tid, vecB);
    if (SBK < K) {
        a.load(gA, M, K, m0, SBK, tid, vecA);
        b.load(gB, N, K, n0, SBK, tid, vecB);
    }
    __syncthreads();
    int buf = 0;
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += SBK, buf ^= 1) {
#pragma unroll
        for (int k = 0; k < SBK; ++k) {
            float2 x[TM / 2];
#pragma unroll
            for (int h = 0; h < TM / 4; ++h) {
                const float4 q = *reinterpret_cast<const float4*>(&sA[buf][k][ty * 4 + 64 * h]);
                x[2 * h] = make_float2(q.x, q.y);
                x[2 * h + 1] = make_float2(q.z, q.w);
            }
#pragma unroll
            for (int j = 0; j < TM; ++j) {
                const float y = sB[buf][k][tx + 16 * j];
#pragma unroll
                for (int i = 0; i < TM / 2; ++i) acc[i][j] = blk_fma2(x[i], make_float2(y, y), acc[i][j]);
            }
        }
        if (k0 + SBK < K) {
            a.store(sA[buf ^ 1], tid, vecA);
            b.store(sB[buf ^ 1], tid, vecB);
            // on their way across the barrier (a plain load does not move ahead of it by itself; us, loads behind the barrier ->
            // here: 6 training steps' products of 16..1699 rows, 8 heads, 78.4 -> 74.4, chains of 438 segments 47.1 -> 45.3)
            if (k0 + 2 * SBK < K) {
                a.load(gA, M, K, m0, k0 + 2 * SBK, tid, vecA);
                b.load(gB, N, K, n0, k0 + 2 * SBK, tid, vecB);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int r = m0 + ty * 4 + 64 * (i >> 1) + 2 * (i & 1) + e;
            if (r < M) {
                float* row = gC + (int64_t)r * N + n0 + tx;
#pragma unroll
                for (int j = 0; j < TM; ++j)
                    if (n0 + tx + 16 * j < N) row[16 * j] = (e ? acc[i][j].y : acc[i][j].x) * p.scale;
            }
        }
}

template <int TM>
cudaError_t launch(const BlkSimtParams& p, cudaStream_t st) {
    const int64_t blocks = (int64_t)p.num_items * p.H;
    if (blocks == 0) return cudaSuccess;
    const dim3 grid((unsigned)blocks), block(SNT);
    auto run = [&](auto kern) { return blk_launch(grid.x <= BLK_EARLY_GRID, kern, grid, block, 0, st, p); };
    if (!p.ta && !p.tb) return run(blk_gemm_simt_kernel<TM, false, false>);
    if (!p.ta && p.tb) return run(blk_gemm_simt_kernel<TM, false, true>);
    if (p.ta && !p.tb) return run(blk_gemm_simt_kernel<TM, true, false>);
    return run(blk_gemm_simt_kernel<TM, true, true>);
}

}  // namespace

cudaError_t blk_launch_gemm_simt(const BlkSimtParams& p, int big, cudaStream_t st) { return big ? launch<8>(p, st) : launch<4>(p, st); }

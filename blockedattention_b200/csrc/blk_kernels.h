// Kernel parameter blocks and launcher prototypes (internal).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "blk_internal.h"

// Where the rows of one 16-bit operand live: element (head h, row r, k) is at base[r * row_stride +
// h * head_stride + k].  Packed head-major strips: row_stride = K, head_stride = elements per strip;
// token-major [rows, H, K]: row_stride = H * K, head_stride = K.
struct BlkOperandLayout {
    int64_t rows;         // rows per head
    int64_t row_stride;   // elements
    int64_t head_stride;  // elements
};

struct BlkGemmParams {
    const uint16_t* A;
    const uint16_t* B;
    void* C;
    const BlkSeg* segs;
    const BlkTileItem* items;
    const BlkTileRec* recs;  // items[i] and its segment side by side
    int64_t Dm1, Dm2, Dout;
    int num_items;
    int H;
    int out_f32;
    int epi;
    float scale;
};

struct BlkSimtParams {
    const float* A;
    const float* B;
    float* C;
    const BlkSeg* segs;
    const BlkTileItem* items;
    int64_t Dm1, Dm2, Dout;
    int num_items;
    int H;
    int ta, tb;
    float scale;
};

struct BlkSmallParams {
    const uint16_t* A;
    const uint16_t* B;
    void* C;
    const BlkSmallItem* items;
    int64_t Dm1, Dm2, Dout;
    int num_items;
    int H;
    int out_f32;
    int epi;
    float scale;
};

struct BlkUmmaParams {
    void* C;
    const BlkUmmaItem* items;
    int64_t Dout;
    int num_items;
    int H;
    int bf16;
    int out_f32;
    int epi;
    float scale;
    int* status;
    int head_firstA, head_firstB;  // coordinate order of the operands' tensor maps
    int wide;                      // scores only, items of single 256-column chunks (long contractions)
    // Test hook for the bounded waits: stall != 0 makes the producer role issue no copies at all (nothing is ever
    // in flight), so the first wait for operands runs out after spin_limit polls (0: the normal limit), the kernel
    // records BLK_ERR_TIMEOUT's status code and returns.
    int stall;
    uint32_t spin_limit;
};

struct BlkPvParams {
    const void* A;  // first operand: rows of K elements at arbitrary 2-byte offsets
    void* C;
    const BlkPvItem* items;
    int64_t Dm1, Dm2, Dout;
    int num_items;
    int H;
    int D;  // columns of the second operand and of the result: 64 or 128
    int ta; // the first operand is stored (K, M)
    int bf16;
    float scale;
    int* status;
};

struct BlkPackParams {
    const uint16_t* A;
    const uint16_t* B;
    void* C;
    const BlkPack* packs;
    const BlkPackBlock* blocks;
    int64_t Dm1, Dm2, Dout;
    int num_packs;
    int H;
    int epi;
    float scale;
    int* status;
    BlkOperandLayout layA, layB;   // where the operands' rows are (filled by the caller)
    int head_firstA, head_firstB;  // coordinate order of the tensor maps (filled by the launcher)
    // attention variant (V != null): C receives softmax(scale A B^T) V, 64 columns per first-operand row
    const uint16_t* V;
    BlkOperandLayout layV;
    int head_firstV;
    int64_t out_row_stride, out_head_stride;  // elements; result row r of head h at C[h * head_stride + r * row_stride]
};

struct BlkFlashParams {
    void* out;
    float* lse;                 // [head][query row] base-2 logarithm of the row sums (reference included); null: not wanted
    const BlkFlashPair* pairs;
    int num_pairs;
    int H;
    int D;  // head dimension: 64 or 128
    int bf16;
    float scale;
    int* status;
    BlkOperandLayout layQ, layK, layV;
    int head_firstQ, head_firstK, head_firstV;  // coordinate order of the tensor maps (filled by the launcher)
    int64_t out_row_stride, out_head_stride;    // elements; result row r of head h at out[h * head_stride + r * row_stride]
};

// One launch of the backward of the attention kernel (see blk_attn_bwd_umma.cu).  items: first resident row, first
// passing row, resident rows from there on, passing rows.
struct BlkFlashBwdParams {
    const BlkFlashItem* items;
    int num_items;
    int H;
    int D;
    int bf16;
    float scale;
    int* status;
    const void* o;     // forward result (query launch)
    const void* g;     // its gradient (query launch; filled by the launcher)
    const float* lse;  // [head][query row] as the forward kernel leaves it
    float* delta;      // [head][query row] rowsum(dO O): written by the query launch, read by the key launch
    void* out0;        // dV (key launch)
    void* out1;        // dQ or dK
    int64_t rows_q;    // query rows per head
    int64_t rows_r;    // rows per head of the resident operands
    int head_firstR, head_firstT;  // coordinate order of the tensor maps (filled by the launcher)
};

// The backward of segments of at most 64 x 64 (blk_attn_bwd_small.cu); packed head-major strips.
struct BlkAttnBwdSmallParams {
    const uint16_t *q, *k, *v, *g;  // g: gradient of the result
    uint16_t *dq, *dk, *dv;
    const BlkFlashItem* items;      // rowQ, rowKV, M, N of a segment
    int num_items;
    int H;
    int64_t rows_q, rows_kv;        // rows per head
    float scale;
};

struct BlkSmxParams {
    const void* src;
    void* dst;
    const BlkSmxChunk* chunks;
    int64_t D;
    int num_chunks;
    int H;
    float scale;
};

// Grids of one-shot blocks up to which blk_launch is asked for an early start.  What it saves is the same 2 us a launch on both sides
// of the line as long as blocks are alike: products of 60 rows and columns over 100 on the staged kernel 8.2 -> 6.4 us for 296 blocks,
// 10.3 -> 7.5 for 444, 22.4 -> 19.6 for 1184, 39.1 -> 37.4 for 2368; fp32 ones of 64 over 64 9.9 -> 7.2, 12.2 -> 9.3, 24.6 -> 21.8,
// 47.4 -> 45.3.  Several waves of unlike blocks lose up to an eighth (385 products of 256..1216 rows on the staged kernel
// 5238 -> 5880 us): the line is low for their sake.
constexpr unsigned BLK_EARLY_GRID = 296;

// Launches a kernel that waits by itself for the one in front of it (blk_grid_wait): its start -- the launch, barriers, tensor
// memory -- overlaps the end of that one.  Passes one after the other, us: 32 fp32 products and softmaxes of at most 32 x 32 x 32 (two
// launches) 12.3 -> 8.7, attention of 16 graphs 8.2 -> 6.0, forward and backward of 1024 graphs (three launches) 84.5 -> 79.1.
// early = false: an ordinary launch.  Persistent kernels of the tensor cores ask for that beyond a number of items per SM that is a
// launch of 45 us for short items and 200 to 450 for long ones: the 2 us that are saved are below 2 % there, and blocks that come
// one by one where an SM is free lie on the chip in no order, so that neighbours in the list of items, which read the same
// operands, may no longer share a part of the L2 (64 products of 1024..2048 rows and columns, long contractions: 839 -> 850 and
// 865 us).  Ordinary -> early at the lines, items of segments of 256 and of 1024 rows: attention, 12 items an SM, 95.0 -> 93.5 us and
// 234 -> 230; with its backward 231 -> 230 and 564 -> 559; P V, 12, 46.4 -> 45.8 and 126 -> 122; plain scores, 24, streams 90.8 -> 88.9
// and 332 -> 330, grouped 82.3 -> 80.4 and 279 -> 274; softmax, 24, streams 123.5 -> 121.5 and 462 -> 460, grouped 92.5 -> 89.1 and
// 439 -> 435; long contractions of 1024 and 4096, 4, 51.8 -> 51.4 and 181 -> 179.  Four times as many items: all within 1.8 % either
// way, less than their runs differ by.
template <typename... P>
inline cudaError_t blk_launch(bool early, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const P&... args) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
    if (e != cudaSuccess) cudaGetLastError();  // reported here and not again by whoever looks next
    return e;
}

// Tensor map (128-byte swizzle) over such an operand, boxes of box_k x box_rows of one head.  The dimension
// with the smaller stride comes second: *head_first = 0 means coordinates (k, row, head), 1 means (k, head, row).
// False when the driver's encoder is unavailable or rejects the view.  Defined in blk_gemm_umma.cu.
struct CUtensorMap_st;
bool blk_make_row_map(CUtensorMap_st* map, const void* base, int bf16, int64_t K, int64_t H, const BlkOperandLayout& lay,
                      int box_k, int box_rows, int* head_first);

// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) once per kernel and device.  Defined in blk_gemm_umma.cu.
cudaError_t blk_func_smem(const void* kern, int bytes);

cudaError_t blk_launch_gemm_tile(const BlkGemmParams& p, int dtype_in, int ta, int tb, cudaStream_t st);
// Pipelined softmax kernels (blk_softmax_pipe.cu).  Forward: in0 = src, in1 unused; backward: in0 = forward
// result, in1 = its gradient (out may alias in1).
struct BlkSmxPipeParams {
    const void* in0;
    const void* in1;
    void* out;
    const BlkSmxWindow* windows;
    const BlkSmxChunk* pieces;
    int64_t D;
    int num_windows;
    int H;
    float scale;
    int* status;
};
cudaError_t blk_launch_softmax_pipe(const BlkSmxPipeParams& p, int dtype, int backward, int sms, cudaStream_t st);
// big: the items are tiles of 128 x 128, not 64 x 64.
cudaError_t blk_launch_gemm_simt(const BlkSimtParams& p, int big, cudaStream_t st);
cudaError_t blk_launch_scores_small(const BlkSmallParams& p, int dtype_in, int K, int bucket, int sms,
                                    cudaStream_t st);
// An operand of the tcgen05 GEMM kernel: the buffer, the length of a head strip, and the views the plan's items refer
// to.  given != nullptr (strided operands): the one view, which starts at the buffer, has this layout instead of the
// packed one.
struct BlkUmmaOperand {
    const void* base;
    int64_t D;
    const BlkUmmaView* views;
    int num_views;
    const BlkOperandLayout* given;
};
cudaError_t blk_launch_gemm_umma(const BlkUmmaParams& p, const BlkUmmaOperand& A, const BlkUmmaOperand& B, int sms,
                                 cudaStream_t st);
// The same for contractions of at most BLK_STREAM_MAXK: independent streams of items (blk_scores_umma.cu).
cudaError_t blk_launch_scores_umma(const BlkUmmaParams& p, const BlkUmmaOperand& A, const BlkUmmaOperand& B, int sms,
                                   cudaStream_t st);
cudaError_t blk_launch_pv_umma(const BlkPvParams& p, const void* V, int sms, cudaStream_t st);
cudaError_t blk_launch_attn_umma(const BlkFlashParams& p, const void* q, const void* k, const void* v, int sms,
                                 cudaStream_t st);
// keys = 0: tensors Q, dO (resident), K, V (passing); keys = 1: K, V (resident), Q, dO (passing).
cudaError_t blk_launch_attn_bwd_umma(const BlkFlashBwdParams& p, int keys, const void* const* tensors,
                                     const BlkOperandLayout& layR, const BlkOperandLayout& layT, int sms, cudaStream_t st);
// rows: 32 or 64, the most a segment of the list has of either kind.
cudaError_t blk_launch_attn_bwd_small(const BlkAttnBwdSmallParams& p, int D, int rows, int bf16, cudaStream_t st);
cudaError_t blk_launch_scores_pipe(const BlkPackParams& p, int dtype_in, int sms, cudaStream_t st);
cudaError_t blk_launch_softmax(const BlkSmxParams& p, int dtype, cudaStream_t st);

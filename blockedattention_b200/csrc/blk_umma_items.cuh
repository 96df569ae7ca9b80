// What the two tcgen05 GEMM kernels share: the tensor maps of a launch and how work items are read.
#pragma once
#include <cuda.h>

#include "blk_device.cuh"
#include "blk_kernels.h"

// The tensor maps of the operands' views (BlkUmmaView), passed as one kernel parameter.
struct UmMaps {
    CUtensorMap a[BLK_UMMA_VIEWS];
    CUtensorMap b[BLK_UMMA_VIEWS];
};
// Encodes (or finds) the maps of a launch, boxes of box_a and box_b rows, and sets the order of coordinates in p.
bool blk_umma_maps(BlkUmmaParams& p, const BlkUmmaOperand& A, const BlkUmmaOperand& B, int box_a, int box_b, UmMaps& maps);

namespace {

// Item n of walker g of G, from global memory.  Odd rounds run through the walkers backwards, so that with the items sorted by
// cost no walker always gets the heaviest of a round.  Only the last round can point past the end, so a walker that gets
// nothing there has nothing left either.
__device__ __forceinline__ bool fetch_item(const BlkUmmaParams& p, uint32_t n, uint32_t G, uint32_t g, BlkUmmaItem& it, int& head) {
    const uint32_t w = n * G + ((n & 1u) ? G - 1u - g : g);
    if (w >= (uint32_t)p.num_items * (uint32_t)p.H) return false;
    const uint32_t item = w / (uint32_t)p.H;
    head = (int)(w - item * (uint32_t)p.H);
    const int4* src = reinterpret_cast<const int4*>(p.items + item);
    int4* dst = reinterpret_cast<int4*>(&it);
#pragma unroll
    for (int i = 0; i < 3; ++i) dst[i] = blk_ld_table(src + i);
    return true;
}
// Rows of an item's block.  A block that fills less than four quarters of the accumulator lanes is put into other
// quarters from item to item (its operand rows are loaded that much earlier): a quarter is one scheduler's warps.
__device__ __forceinline__ int item_rows(const BlkUmmaItem& it, uint32_t n) {
    const int rows = min(it.M - it.tm * BLK_UMMA_BM, BLK_UMMA_BM);
    const uint32_t slack = 4u - (uint32_t)((rows + 31) >> 5);
    return rows | (int)((n % (slack + 1u)) << 8);
}

}  // namespace

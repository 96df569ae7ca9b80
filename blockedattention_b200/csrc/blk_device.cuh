// Device-side helpers shared by the kernels of libblkattn (sm_100a).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "blk_internal.h"

#define BLK_LOG2E 1.4426950408889634f

// 16-bit storage type used for both fp16 and bf16 buffers; the tag types pick
// the arithmetic.
struct BlkHalfTag {};
struct BlkBf16Tag {};

template <typename Tag> struct BlkCvt;
template <> struct BlkCvt<BlkHalfTag> {
    static __device__ __forceinline__ uint32_t pack2(float a, float b) {
        __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<uint32_t*>(&h);
    }
    static __device__ __forceinline__ uint16_t pack1(float a) {
        __half h = __float2half_rn(a);
        return *reinterpret_cast<uint16_t*>(&h);
    }
    static __device__ __forceinline__ float unpack1(uint16_t v) {
        return __half2float(*reinterpret_cast<__half*>(&v));
    }
};
template <> struct BlkCvt<BlkBf16Tag> {
    static __device__ __forceinline__ uint32_t pack2(float a, float b) {
        __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<uint32_t*>(&h);
    }
    static __device__ __forceinline__ uint16_t pack1(float a) {
        __nv_bfloat16 h = __float2bfloat16_rn(a);
        return *reinterpret_cast<uint16_t*>(&h);
    }
    static __device__ __forceinline__ float unpack1(uint16_t v) {
        return __uint_as_float(((uint32_t)v) << 16);
    }
};

// D(16x8,f32) += A(16x16) * B(16x8); A row-major fragment, B column fragment.
template <typename Tag>
__device__ __forceinline__ void blk_mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void blk_mma16816<BlkHalfTag>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                         uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void blk_mma16816<BlkBf16Tag>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                         uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A kernel may be resident before the one in front of it in the stream has finished (blk_launch).  Before its first access to
// memory that another kernel writes or reads it waits for that one (and, as every kernel does, for all before it); work tables of
// a plan are there before any launch and may be read earlier.  blk_grid_ready lets the next kernel of the stream come: to be called
// when the block holds all it will ever need of its SM (tensor memory), or the next one's blocks could take what it waits for.
__device__ __forceinline__ void blk_grid_ready() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
// Kernels with several blocks on an SM never call it: their blocks let the next kernel come by ending.  Blocks of the next one that
// come while these are still there settle where there happens to be room, several on one SM.  Announced from the start by grids
// of at most a block per SM, us against this: 148 products of 60 rows and columns over 2001 on the staged kernel 90.5 -> 63.2
// (one after the other 65.5), its fused softmax for 9 segments of 1000 123.7 -> 97.3 (99.6); nothing gained over 33 to 1001
// either (3.6 to 33 us, both the same within 0.3).
__device__ __forceinline__ void blk_grid_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

__device__ __forceinline__ uint32_t blk_smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void blk_ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void blk_ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

__device__ __forceinline__ float blk_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

// Two fp32 operations in one instruction (packed forms of sm_100): a * b + c and a + b, element by element.
__device__ __forceinline__ float2 blk_fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n .reg .b64 a, b, c, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n mov.b64 c, {%6, %7};\n"
        " fma.rn.f32x2 d, a, b, c;\n mov.b64 {%0, %1}, d;\n}\n"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 blk_add2(float2 a, float2 b) {
    float2 d;
    asm("{\n .reg .b64 a, b, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n add.rn.f32x2 d, a, b;\n"
        " mov.b64 {%0, %1}, d;\n}\n"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

__device__ __forceinline__ float2 blk_mul2(float2 a, float2 b) {
    float2 d;
    asm("{\n .reg .b64 a, b, d;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %5};\n mul.rn.f32x2 d, a, b;\n"
        " mov.b64 {%0, %1}, d;\n}\n"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// max(a, b, c) in one instruction (three-input maximum of sm_100).
__device__ __forceinline__ float blk_max3(float a, float b, float c) {
    float y;
    asm("max.f32 %0, %1, %2, %3;\n" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}
// 16-byte global load that does not allocate in L1 (data touched once).  Not a
// read-only (.nc) load: the softmax may run in place.
__device__ __forceinline__ uint4 blk_ldg_stream16(const void* p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
// Shared-memory stores through 32-bit shared-window addresses.
__device__ __forceinline__ void blk_sts_b32(uint32_t addr, uint32_t v) {
    asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(addr), "r"(v));
}
__device__ __forceinline__ void blk_sts_b16(uint32_t addr, uint32_t v) {
    asm volatile("st.shared.b16 [%0], %1;\n" ::"r"(addr), "h"((uint16_t)v));
}
__device__ __forceinline__ void blk_sts_f32(uint32_t addr, float v) {
    asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(addr), "f"(v));
}
__device__ __forceinline__ void blk_sts_f32x2(uint32_t addr, float x, float y) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};\n" ::"r"(addr), "f"(x), "f"(y));
}

// 64 contiguous bytes of a lane, to 16-byte aligned memory.  As whole 32-byte sectors where it lies on them: two 16-byte stores
// to a sector, each of them 16 bytes for every row of a warp, pass through the memory system as two partial writes, at half
// the rate.
__device__ __forceinline__ void blk_stg64(void* p, const uint32_t* w) {
    if (!(reinterpret_cast<uintptr_t>(p) & 31u)) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(static_cast<char*>(p) + 32 * i), "r"(w[8 * i]),
                         "r"(w[8 * i + 1]), "r"(w[8 * i + 2]), "r"(w[8 * i + 3]), "r"(w[8 * i + 4]), "r"(w[8 * i + 5]), "r"(w[8 * i + 6]),
                         "r"(w[8 * i + 7])
                         : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) static_cast<uint4*>(p)[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
    }
}

// Loads of what another kernel may have written are plain ones.  Loads through the read-only path (__ldg) ask for memory that
// nobody writes as long as the kernel runs, and a kernel runs from before the one in front of it has finished (blk_launch); the
// compiler may also move them ahead of blk_grid_wait.  They are for the work tables of a plan alone, here:
__device__ __forceinline__ int4 blk_ld_table(const int4* p) { return __ldg(p); }

__device__ __forceinline__ float blk_quad_max(float v) {
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
    v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
    return v;
}
__device__ __forceinline__ float blk_quad_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
}

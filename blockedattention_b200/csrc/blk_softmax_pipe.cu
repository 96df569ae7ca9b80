// Pipelined varlen row softmax, forward and backward, over a packed (H, D) buffer.
//
// The host groups consecutive row pieces (blk_softmax.cu's chunks) whose bytes are contiguous in memory into
// windows of at most 12 KB -- many small segments, or a few rows of a wide one.  A persistent CTA walks windows
// w = blockIdx.x, + gridDim.x, ... of the (window, head) list through a ring of shared-memory stages:
//   * one warp copies: it fetches windows ahead with bulk asynchronous copies (cp.async.bulk, completion on the
//     stage's mbarrier) of the 16-byte aligned range that covers them, and when the computing warps are done with
//     a window writes it back with a bulk store of the aligned vectors that lie wholly inside it, a few lanes
//     storing the ragged edge elements;
//   * the other warps do the row arithmetic out of shared memory (fp32, base-2 exponent, one rounding).  Work is
//     dealt out in units -- a long row, four short ones to eight lanes each, 32 very short ones to a lane each --
//     in turn through all windows of the CTA, so no warp waits for another inside a window.  A long row is read
//     and written as 16-byte vectors between its first and last 16-byte boundary (the few elements outside go one
//     per lane).
// A row longer than a window is streamed from global memory by all computing warps.
// Every barrier wait is bounded and reports through the status word.
//
// Bound by the instructions it issues and their latency, with memory close behind (in the profiler, 512 segments of 16..2048
// rows and columns, 4 heads, bf16: 734 us, issue slots 63 %, special-function unit 64 %, DRAM 62 %; the copies alone 650; the
// backward of a quarter of it 197, DRAM 76 %, its copies alone 187).  A spilled register in a row loop costs more than any
// parallelism: with 28 warps of 64 registers the loops over a row's vectors stay rolled, and rows of short segments are
// functions of their own.  Against the form with two stages, all warps of a CTA meeting twice a window, the call takes
// 856 -> 771 us sustained, a quarter of it 200 -> 167 forward and 223 -> 199 backward (a fifth of the instructions were the
// counting of units in windows of one piece until those were told apart).
//
// Forward: out = softmax_rows(scale * src); replaces upstream sparseBlockedSoftmax_warp / _block
// (csrc/cuda/spBlkSoftmax.cu:88-138, :182-269).  Backward: grad_src = scale * (grad_out - rowsum(out *
// grad_out)) * out; replaces sparseBlockedSoftmaxBackward_warp / _block (:140-180, :271-332).
#include "blk_device.cuh"
#include "blk_kernels.h"

namespace {

// Warps that compute in a CTA, CTAs on an SM and shared-memory stages of a CTA: 16 windows of an SM are in flight or in
// work (backward, with two inputs a window: 8).
template <bool BWD>
struct SpShape {
    static constexpr int NW = BWD ? 9 : 7;
    static constexpr int CTAS = BWD ? 2 : 4;
    static constexpr int STAGES = 4;
    static constexpr int THREADS = 32 * (NW + 1);
};
constexpr int SP_WIN = BLK_SMX_WINDOW_BYTES;
constexpr int SP_BUF = SP_WIN + 32;  // a window plus the slack of its 16-byte aligned cover
constexpr uint32_t SP_SPIN_LIMIT = 1u << 22;

// Element types: E, scalar conversion, and the 16-byte vector of VE elements.
template <typename Tag>
struct SpIO16;
template <>
struct SpIO16<BlkHalfTag> {
    typedef uint16_t E;
    static constexpr int VE = 8;
    static __device__ __forceinline__ float ld(E v) { return BlkCvt<BlkHalfTag>::unpack1(v); }
    static __device__ __forceinline__ E st(float v) { return BlkCvt<BlkHalfTag>::pack1(v); }
    static __device__ __forceinline__ void unpack(const uint4& q, float2 (&f)[4]) {
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[i] = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        }
    }
    static __device__ __forceinline__ uint4 pack(const float2 (&f)[4]) {
        return make_uint4(BlkCvt<BlkHalfTag>::pack2(f[0].x, f[0].y), BlkCvt<BlkHalfTag>::pack2(f[1].x, f[1].y),
                          BlkCvt<BlkHalfTag>::pack2(f[2].x, f[2].y), BlkCvt<BlkHalfTag>::pack2(f[3].x, f[3].y));
    }
    // running extreme (maximum, or minimum for a negative scale) of a row, taken on the packed pairs as they lie in
    // memory: one instruction per two elements and no conversion; none: elements that scale to minus infinity
    template <bool NEG> static __device__ __forceinline__ uint32_t none() { return NEG ? 0x7c007c00u : 0xfc00fc00u; }
    template <bool NEG> static __device__ __forceinline__ E none1() { return (E)none<NEG>(); }
    typedef uint32_t X;
    template <bool NEG> static __device__ __forceinline__ X xinit() { return none<NEG>(); }
    template <bool NEG> static __device__ __forceinline__ X xacc(X a, const uint4& q) {
        X r;
        if (NEG) asm("{\n .reg .b32 t, u;\n min.f16x2 t, %1, %2;\n min.f16x2 u, %3, %4;\n min.f16x2 t, t, u;\n min.f16x2 %0, t, %5;\n}\n" : "=r"(r) : "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w), "r"(a));
        else asm("{\n .reg .b32 t, u;\n max.f16x2 t, %1, %2;\n max.f16x2 u, %3, %4;\n max.f16x2 t, t, u;\n max.f16x2 %0, t, %5;\n}\n" : "=r"(r) : "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w), "r"(a));
        return r;
    }
    template <bool NEG> static __device__ __forceinline__ float xfin(X a) {
        const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&a));
        return NEG ? fminf(t.x, t.y) : fmaxf(t.x, t.y);
    }
};
template <>
struct SpIO16<BlkBf16Tag> {
    typedef uint16_t E;
    static constexpr int VE = 8;
    static __device__ __forceinline__ float ld(E v) { return BlkCvt<BlkBf16Tag>::unpack1(v); }
    static __device__ __forceinline__ E st(float v) { return BlkCvt<BlkBf16Tag>::pack1(v); }
    static __device__ __forceinline__ void unpack(const uint4& q, float2 (&f)[4]) {
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
        }
    }
    static __device__ __forceinline__ uint4 pack(const float2 (&f)[4]) {
        return make_uint4(BlkCvt<BlkBf16Tag>::pack2(f[0].x, f[0].y), BlkCvt<BlkBf16Tag>::pack2(f[1].x, f[1].y),
                          BlkCvt<BlkBf16Tag>::pack2(f[2].x, f[2].y), BlkCvt<BlkBf16Tag>::pack2(f[3].x, f[3].y));
    }
    template <bool NEG> static __device__ __forceinline__ uint32_t none() { return NEG ? 0x7f807f80u : 0xff80ff80u; }
    template <bool NEG> static __device__ __forceinline__ E none1() { return (E)none<NEG>(); }
    typedef uint32_t X;
    template <bool NEG> static __device__ __forceinline__ X xinit() { return none<NEG>(); }
    template <bool NEG> static __device__ __forceinline__ X xacc(X a, const uint4& q) {
        X r;
        if (NEG) asm("{\n .reg .b32 t, u;\n min.bf16x2 t, %1, %2;\n min.bf16x2 u, %3, %4;\n min.bf16x2 t, t, u;\n min.bf16x2 %0, t, %5;\n}\n" : "=r"(r) : "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w), "r"(a));
        else asm("{\n .reg .b32 t, u;\n max.bf16x2 t, %1, %2;\n max.bf16x2 u, %3, %4;\n max.bf16x2 t, t, u;\n max.bf16x2 %0, t, %5;\n}\n" : "=r"(r) : "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w), "r"(a));
        return r;
    }
    template <bool NEG> static __device__ __forceinline__ float xfin(X a) {
        const float lo = __uint_as_float(a << 16), hi = __uint_as_float(a & 0xffff0000u);
        return NEG ? fminf(lo, hi) : fmaxf(lo, hi);
    }
};
struct SpIO32 {
    typedef float E;
    static constexpr int VE = 4;
    static __device__ __forceinline__ float ld(E v) { return v; }
    static __device__ __forceinline__ E st(float v) { return v; }
    static __device__ __forceinline__ void unpack(const uint4& q, float2 (&f)[2]) {
        f[0] = make_float2(__uint_as_float(q.x), __uint_as_float(q.y));
        f[1] = make_float2(__uint_as_float(q.z), __uint_as_float(q.w));
    }
    static __device__ __forceinline__ uint4 pack(const float2 (&f)[2]) {
        return make_uint4(__float_as_uint(f[0].x), __float_as_uint(f[0].y), __float_as_uint(f[1].x), __float_as_uint(f[1].y));
    }
    template <bool NEG> static __device__ __forceinline__ uint32_t none() { return NEG ? 0x7f800000u : 0xff800000u; }
    template <bool NEG> static __device__ __forceinline__ E none1() { return __uint_as_float(none<NEG>()); }
    typedef float X;
    template <bool NEG> static __device__ __forceinline__ X xinit() { return none1<NEG>(); }
    template <bool NEG> static __device__ __forceinline__ X xacc(X a, const uint4& q) {
        const float x = __uint_as_float(q.x), y = __uint_as_float(q.y), z = __uint_as_float(q.z), w = __uint_as_float(q.w);
        return NEG ? fminf(fminf(a, x), fminf(fminf(y, z), w)) : fmaxf(fmaxf(a, x), fmaxf(fmaxf(y, z), w));
    }
    template <bool NEG> static __device__ __forceinline__ float xfin(X a) { return a; }
};

__device__ __forceinline__ float sp_max(float v, int G) {
    for (int o = G >> 1; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float sp_sum(float v, int G) {
    for (int o = G >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void sp_bar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void sp_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool sp_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred q;\n mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n selp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool sp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
#pragma unroll 1
    for (uint32_t i = 0; !sp_try(bar, parity); ++i) {
        if (*abort_flag) return false;
        if (i >= SP_SPIN_LIMIT) {
            *abort_flag = 1;
            return false;
        }
        __nanosleep(40);
    }
    return true;
}
__device__ __forceinline__ void sp_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// contiguous bulk copies (16-byte aligned addresses and size)
__device__ __forceinline__ void sp_bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void sp_bulk_s2g(void* dst, uint32_t src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void sp_bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
// all bulk stores of this thread but the last have finished reading shared memory
__device__ __forceinline__ void sp_bulk_wait_read1() { asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory"); }
// ... and have completed
__device__ __forceinline__ void sp_bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }

// ---- row arithmetic on a piece that sits in shared memory ---------------------------------------------------

// A row of at least 8 vectors' worth of columns, one warp per row: the row starts at an arbitrary element of
// shared memory, so it is split into the elements before the first 16-byte boundary (at most VE - 1, one per
// lane 0..7), whole 16-byte vectors (lane l takes vectors l, l + 32, ...) and the elements after the last
// whole vector (one per lane 8..15).
template <typename IO>
struct RowSplit {
    uint32_t row, body;  // shared-memory addresses
    int nv;              // whole vectors
    int xi;              // this lane's extra element, or -1
    __device__ __forceinline__ RowSplit(uint32_t r, int cols, int lane) : row(r) {
        constexpr int ES = (int)sizeof(typename IO::E);
        const int h = (int)((16u - (r & 15u)) & 15u) / ES;
        nv = (cols - h) / IO::VE;
        const int tail = cols - h - nv * IO::VE;
        body = r + (uint32_t)(h * ES);
        xi = -1;
        if (lane < 8) {
            if (lane < h) xi = lane;
        } else if (lane < 16) {
            if (lane - 8 < tail) xi = h + nv * IO::VE + lane - 8;
        }
    }
};
// elements and 16-byte vectors of a shared-memory buffer
__device__ __forceinline__ void sp_lds(uint16_t& v, uint32_t a) { asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(a)); }
__device__ __forceinline__ void sp_lds(float& v, uint32_t a) { asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(v) : "r"(a)); }
__device__ __forceinline__ void sp_sts(uint32_t a, uint16_t v) { asm volatile("st.shared.u16 [%0], %1;\n" ::"r"(a), "h"(v) : "memory"); }
__device__ __forceinline__ void sp_sts(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(a), "f"(v) : "memory"); }
template <typename IO>
__device__ __forceinline__ float sp_ld(uint32_t row, int i) {
    typename IO::E v;
    sp_lds(v, row + (uint32_t)(i * (int)sizeof(typename IO::E)));
    return IO::ld(v);
}
// ... or the value that stands for no element
template <typename IO, bool NEG>
__device__ __forceinline__ float sp_ld_if(bool there, uint32_t row, int i) {
    typename IO::E v = IO::template none1<NEG>();
    if (there) sp_lds(v, row + (uint32_t)(i * (int)sizeof(typename IO::E)));
    return IO::ld(v);
}
template <typename IO>
__device__ __forceinline__ void sp_st(uint32_t row, int i, float v) {
    sp_sts(row + (uint32_t)(i * (int)sizeof(typename IO::E)), IO::st(v));
}
__device__ __forceinline__ uint4 sp_ldv(uint32_t body, int vi) {
    uint4 q;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
                 : "r"(body + 16u * (uint32_t)vi));
    return q;
}
__device__ __forceinline__ void sp_stv(uint32_t body, int vi, const uint4& q) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(body + 16u * (uint32_t)vi), "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w)
                 : "memory");
}

// Every forward row is exp2(y) over its sum with y = (x - m) * sl, m the largest x of the row, or the smallest (NEG: the
// kernel for negative scales).  The difference is taken before the product, so that y is rounded relative to itself: with
// x * sl rounded first it is off by half a unit of m * sl (fp32 rows, measured against 64 bits: 5e-6 of the result for scores
// around 200, 4e-4 around 20000; this form: below 1.3e-7 for both), and rows masked throughout with a type's lowest value
// stay finite.  (x - m overflows only where a row spans more than the largest number; y is then minus infinity, which is
// right for any scale above 1e-37.)
__device__ __forceinline__ void sp_exp2(float2& f) {
    f.x = blk_exp2(f.x);
    f.y = blk_exp2(f.y);
}
// the value that stands for no element, and the larger of two in the order of x * sl
template <bool NEG> __device__ __forceinline__ float sp_none() { return NEG ? INFINITY : -INFINITY; }
template <bool NEG> __device__ __forceinline__ float sp_top(float a, float b) { return NEG ? fminf(a, b) : fmaxf(a, b); }
template <bool NEG> __device__ __forceinline__ float sp_top3(float a, float b, float c) {
    return NEG ? -blk_max3(-a, -b, -c) : blk_max3(a, b, c);
}
template <bool NEG> __device__ __forceinline__ float sp_tops(float v, int G) {  // over G lanes
    return NEG ? -sp_max(-v, G) : sp_max(v, G);
}
// exp2(y) of a row's elements in place, and their sum
template <int N>
__device__ __forceinline__ float sp_exps(float2 (&v)[N], float m, float sl) {
    const float2 nm = make_float2(-m, -m), sl2 = make_float2(sl, sl);
    float2 sum = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        v[i] = blk_mul2(blk_add2(v[i], nm), sl2);
        sp_exp2(v[i]);
        sum = blk_add2(sum, v[i]);
    }
    return sum.x + sum.y;
}
// f(vi) for this lane's vectors; kept rolled, see the note on registers at the head of the file
template <typename F>
__device__ __forceinline__ void sp_each(int nv, int lane, F f) {
#pragma unroll 1
    for (int vi = lane; vi < nv; vi += 32) f(vi);
}
template <typename IO, bool NEG>
__device__ __forceinline__ float sp_extreme(uint32_t body, int nv, int lane) {
    typename IO::X ex = IO::template xinit<NEG>();
    sp_each(nv, lane, [&](int vi) { ex = IO::template xacc<NEG>(ex, sp_ldv(body, vi)); });
    return IO::template xfin<NEG>(ex);
}

// forward, at most 32 EPV whole vectors per row and a scale that is not zero: values kept in registers, one exponential
// per element.  Lanes without a vector hold elements that scale to minus infinity.
template <typename IO, bool NEG, int EPV, int NW>
__device__ __forceinline__ void fwd_rows_vec(uint32_t piece, int rows, int cols, float sl, int r0, int lane) {
    constexpr int VP = IO::VE / 2;
    const float2 sl2 = make_float2(sl, sl);
    const uint32_t none = IO::template none<NEG>();
#pragma unroll 1
    for (int r = r0; r < rows; r += NW) {
        const RowSplit<IO> rs(piece + (uint32_t)(r * cols * (int)sizeof(typename IO::E)), cols, lane);
        float x = sp_ld_if<IO, NEG>(rs.xi >= 0, rs.row, rs.xi);
        float2 v[EPV][VP];
        float m = x;
#pragma unroll
        for (int i = 0; i < EPV; ++i) {
            uint4 q = make_uint4(none, none, none, none);
            if (lane + 32 * i < rs.nv) q = sp_ldv(rs.body, lane + 32 * i);
            IO::unpack(q, v[i]);
#pragma unroll
            for (int e = 0; e < VP; ++e) m = sp_top3<NEG>(m, v[i][e].x, v[i][e].y);
        }
        m = sp_tops<NEG>(m, 32);
        x = blk_exp2((x - m) * sl);
        const float2 nm = make_float2(-m, -m);
        float2 sum = make_float2(x, 0.f);
#pragma unroll
        for (int i = 0; i < EPV; ++i)
#pragma unroll
            for (int e = 0; e < VP; ++e) {
                v[i][e] = blk_mul2(blk_add2(v[i][e], nm), sl2);
                sp_exp2(v[i][e]);
                sum = blk_add2(sum, v[i][e]);
            }
        const float inv = 1.f / sp_sum(sum.x + sum.y, 32);
        const float2 inv2 = make_float2(inv, inv);
#pragma unroll
        for (int i = 0; i < EPV; ++i) {
#pragma unroll
            for (int e = 0; e < VP; ++e) v[i][e] = blk_mul2(v[i][e], inv2);
            if (lane + 32 * i < rs.nv) sp_stv(rs.body, lane + 32 * i, IO::pack(v[i]));
        }
        if (rs.xi >= 0) sp_st<IO>(rs.row, rs.xi, x * inv);
    }
}
// forward, any column count that fits the window: three passes over the row, exponential evaluated twice.  NEAR, for rows
// whose |m * sl| is at most sp_near: y = x * sl - m * sl in one fused operation.  The rounding of m * sl is then the same
// for the whole row and cancels; for 16-bit elements, whose third pass takes the logarithm of the sum off as well instead
// of multiplying by its inverse, it does not, but is at most 2^-18, a hundredth of the result's own.
template <typename IO> __device__ __forceinline__ float sp_near() { return IO::VE == 8 ? 64.f : 1048576.f; }
template <typename IO, bool NEAR>
__device__ __forceinline__ void fwd_row_streamed(const RowSplit<IO>& rs, float x, float m, float sl, int lane) {
    constexpr int VP = IO::VE / 2;
    constexpr bool FOLD = NEAR && IO::VE == 8;
    const float2 sl2 = make_float2(sl, sl);
    float2 off = make_float2(NEAR ? -m * sl : -m, NEAR ? -m * sl : -m);
    auto exps = [&](int vi, float2 (&f)[VP]) {
        IO::unpack(sp_ldv(rs.body, vi), f);
#pragma unroll
        for (int e = 0; e < VP; ++e) {
            f[e] = NEAR ? blk_fma2(f[e], sl2, off) : blk_mul2(blk_add2(f[e], off), sl2);
            sp_exp2(f[e]);
        }
    };
    auto extra = [&]() { return rs.xi >= 0 ? blk_exp2(NEAR ? fmaf(x, sl, off.x) : (x - m) * sl) : 0.f; };
    float2 sum = make_float2(extra(), 0.f);
    sp_each(rs.nv, lane, [&](int vi) {
        float2 f[VP];
        exps(vi, f);
#pragma unroll
        for (int e = 0; e < VP; ++e) sum = blk_add2(sum, f[e]);
    });
    const float total = sp_sum(sum.x + sum.y, 32);
    float2 inv2 = make_float2(1.f, 1.f);
    if (FOLD) off.x = off.y = off.x - __log2f(total);
    else inv2.x = inv2.y = 1.f / total;
    sp_each(rs.nv, lane, [&](int vi) {
        float2 f[VP];
        exps(vi, f);
        if (!FOLD) {
#pragma unroll
            for (int e = 0; e < VP; ++e) f[e] = blk_mul2(f[e], inv2);
        }
        sp_stv(rs.body, vi, IO::pack(f));
    });
    if (rs.xi >= 0) sp_st<IO>(rs.row, rs.xi, extra() * inv2.x);
}
// (out of line: the loops of the usual rows stay close together, 1.5 % of the 16-bit long rows)
template <typename IO>
__device__ __noinline__ void fwd_row_far(RowSplit<IO> rs, float x, float m, float sl, int lane) {
    fwd_row_streamed<IO, false>(rs, x, m, sl, lane);
}
template <typename IO, bool NEG, int NW>
__device__ __forceinline__ void fwd_rows_vec_streamed(uint32_t piece, int rows, int cols, float sl, int r0, int lane) {
#pragma unroll 1
    for (int r = r0; r < rows; r += NW) {
        const RowSplit<IO> rs(piece + (uint32_t)(r * cols * (int)sizeof(typename IO::E)), cols, lane);
        const float x = sp_ld_if<IO, NEG>(rs.xi >= 0, rs.row, rs.xi);
        const float m = sp_tops<NEG>(sp_top<NEG>(x, sp_extreme<IO, NEG>(rs.body, rs.nv, lane)), 32);
        if (fabsf(m * sl) <= sp_near<IO>()) fwd_row_streamed<IO, true>(rs, x, m, sl, lane);
        else fwd_row_far<IO>(rs, x, m, sl, lane);
    }
}
// backward over whole vectors, two passes (dot product, then the result over the gradient)
template <typename IO, int NW>
__device__ __forceinline__ void bwd_rows_vec(uint32_t ppiece, uint32_t gpiece, int rows, int cols,
                                             float scale, int r0, int lane) {
    constexpr int VP = IO::VE / 2;
    const float2 scale2 = make_float2(scale, scale);
#pragma unroll 1
    for (int r = r0; r < rows; r += NW) {
        RowSplit<IO> rs(gpiece + (uint32_t)(r * cols * (int)sizeof(typename IO::E)), cols, lane);  // both rows sit at the same offset of their buffers
        const uint32_t prow = ppiece + (uint32_t)(r * cols * (int)sizeof(typename IO::E));
        const uint32_t pbody = prow + (rs.body - rs.row);
        float px = 0.f, gx = 0.f;
        if (rs.xi >= 0) {
            px = sp_ld<IO>(prow, rs.xi);
            gx = sp_ld<IO>(rs.row, rs.xi);
        }
        float2 dot2 = make_float2(px * gx, 0.f);
        sp_each(rs.nv, lane, [&](int vi) {
            float2 pf[VP], gf[VP];
            IO::unpack(sp_ldv(pbody, vi), pf);
            IO::unpack(sp_ldv(rs.body, vi), gf);
#pragma unroll
            for (int e = 0; e < VP; ++e) dot2 = blk_fma2(pf[e], gf[e], dot2);
        });
        const float dot = sp_sum(dot2.x + dot2.y, 32);
        const float2 ndot = make_float2(-dot, -dot);
        sp_each(rs.nv, lane, [&](int vi) {
            float2 pf[VP], gf[VP];
            IO::unpack(sp_ldv(pbody, vi), pf);
            IO::unpack(sp_ldv(rs.body, vi), gf);
#pragma unroll
            for (int e = 0; e < VP; ++e) gf[e] = blk_mul2(blk_mul2(blk_add2(gf[e], ndot), pf[e]), scale2);
            sp_stv(rs.body, vi, IO::pack(gf));
        });
        if (rs.xi >= 0) sp_st<IO>(rs.row, rs.xi, (gx - dot) * px * scale);
    }
}

// Short rows (fewer columns than eight vectors).  Up to 16 columns: one lane per row, no shuffle.  More: eight lanes per
// row, which keeps the row in registers and every warp busy when a window is one long piece of short rows.
constexpr int SP_LANE_COLS = 16;
template <typename IO, bool NEG>
__device__ __noinline__ void fwd_rows_lane(uint32_t piece, int rows, int cols, float sl, int r, int lane) {
    r += lane;
    if (r >= rows) return;
    const uint32_t row = piece + (uint32_t)(r * cols * (int)sizeof(typename IO::E));
    float2 v[SP_LANE_COLS / 2];
    float m = sp_none<NEG>();
#pragma unroll
    for (int c = 0; c < SP_LANE_COLS / 2; ++c) {
        v[c] = make_float2(sp_ld_if<IO, NEG>(2 * c < cols, row, 2 * c), sp_ld_if<IO, NEG>(2 * c + 1 < cols, row, 2 * c + 1));
        m = sp_top3<NEG>(m, v[c].x, v[c].y);
    }
    const float inv = 1.f / sp_exps(v, m, sl);
#pragma unroll
    for (int c = 0; c < SP_LANE_COLS / 2; ++c) {
        if (2 * c < cols) sp_st<IO>(row, 2 * c, v[c].x * inv);
        if (2 * c + 1 < cols) sp_st<IO>(row, 2 * c + 1, v[c].y * inv);
    }
}
template <typename IO, bool NEG>
__device__ __noinline__ void fwd_rows_group(uint32_t piece, int rows, int cols, float sl, int r, int lane) {
    r += lane >> 3;
    const int l = lane & 7;
    const uint32_t row = piece + (uint32_t)(r * cols * (int)sizeof(typename IO::E));
    const int have = r < rows ? cols - l : 0;  // this lane's elements are l, l + 8, ...
    float2 v[IO::VE / 2];
    float m = sp_none<NEG>();
#pragma unroll
    for (int i = 0; i < IO::VE / 2; ++i) {
        v[i] = make_float2(sp_ld_if<IO, NEG>(16 * i < have, row, l + 16 * i), sp_ld_if<IO, NEG>(16 * i + 8 < have, row, l + 16 * i + 8));
        m = sp_top3<NEG>(m, v[i].x, v[i].y);
    }
    m = sp_tops<NEG>(m, 8);
    const float inv = 1.f / sp_sum(sp_exps(v, m, sl), 8);
#pragma unroll
    for (int i = 0; i < IO::VE / 2; ++i) {
        if (16 * i < have) sp_st<IO>(row, l + 16 * i, v[i].x * inv);
        if (16 * i + 8 < have) sp_st<IO>(row, l + 16 * i + 8, v[i].y * inv);
    }
}
// row r by a lane, for a scale of zero: the above keep elements past a row's end out by an infinite y
template <typename IO>
__device__ __noinline__ void fwd_row_zero_scale(uint32_t piece, int cols, int r) {
    const uint32_t row = piece + (uint32_t)(r * cols * (int)sizeof(typename IO::E));
    float sum = 0.f;
#pragma unroll 1
    for (int c = 0; c < cols; ++c) sum += blk_exp2(sp_ld<IO>(row, c) * 0.f);
#pragma unroll 1
    for (int c = 0; c < cols; ++c) sp_st<IO>(row, c, blk_exp2(sp_ld<IO>(row, c) * 0.f) / sum);
}
template <typename IO>
__device__ __forceinline__ void bwd_rows_lane(uint32_t ppiece, uint32_t gpiece, int rows, int cols,
                                              float scale, int r, int lane) {
    r += lane;
    if (r >= rows) return;
    const uint32_t prow = ppiece + (uint32_t)(r * cols * (int)sizeof(typename IO::E));
    const uint32_t grow = gpiece + (uint32_t)(r * cols * (int)sizeof(typename IO::E));
    float dot = 0.f;
    for (int c = 0; c < cols; ++c) dot = fmaf(sp_ld<IO>(prow, c), sp_ld<IO>(grow, c), dot);
    for (int c = 0; c < cols; ++c) sp_st<IO>(grow, c, (sp_ld<IO>(grow, c) - dot) * sp_ld<IO>(prow, c) * scale);
}
template <typename IO>
__device__ __forceinline__ void bwd_rows_group(uint32_t ppiece, uint32_t gpiece, int rows, int cols,
                                               float scale, int r, int lane) {
    r += lane >> 3;
    const int l = lane & 7;
    const uint32_t prow = ppiece + (uint32_t)(r * cols * (int)sizeof(typename IO::E));
    const uint32_t grow = gpiece + (uint32_t)(r * cols * (int)sizeof(typename IO::E));
    float pv[IO::VE], gv[IO::VE];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < IO::VE; ++i) {
        const bool in = r < rows && l + 8 * i < cols;
        pv[i] = in ? sp_ld<IO>(prow, l + 8 * i) : 0.f;
        gv[i] = in ? sp_ld<IO>(grow, l + 8 * i) : 0.f;
        dot = fmaf(pv[i], gv[i], dot);
    }
    dot = sp_sum(dot, 8);
#pragma unroll
    for (int i = 0; i < IO::VE; ++i)
        if (r < rows && l + 8 * i < cols) sp_st<IO>(grow, l + 8 * i, (gv[i] - dot) * pv[i] * scale);
}

// Rows of a unit of short rows, the amount of work that goes to one warp.
__device__ __forceinline__ int sp_unit_rows(int cols) { return cols <= SP_LANE_COLS ? 32 : 4; }

// One piece: this warp's units -- rows, or groups of short rows -- are u, u + NW, ...
template <typename IO, bool NEG, int NW>
__device__ __forceinline__ void fwd_piece(uint32_t srow, int rows, int cols, float sl, int u, int lane) {
    constexpr int VE = IO::VE;
    if (cols < 8 * VE) {
        const int ur = sp_unit_rows(cols);
#pragma unroll 1
        for (int r = u * ur; r < rows; r += NW * ur) {
            if (!NEG && sl == 0.f) {
                if (lane < ur && r + lane < rows) fwd_row_zero_scale<IO>(srow, cols, r + lane);
            } else if (cols <= SP_LANE_COLS) {
                fwd_rows_lane<IO, NEG>(srow, rows, cols, sl, r, lane);
            } else {
                fwd_rows_group<IO, NEG>(srow, rows, cols, sl, r, lane);
            }
        }
        return;
    }
    const int nvmax = cols / VE;  // whole vectors of a row never exceed this
    if (nvmax > 64 || (!NEG && sl == 0.f)) fwd_rows_vec_streamed<IO, NEG, NW>(srow, rows, cols, sl, u, lane);
    else if (nvmax <= 32) fwd_rows_vec<IO, NEG, 1, NW>(srow, rows, cols, sl, u, lane);
    else fwd_rows_vec<IO, NEG, 2, NW>(srow, rows, cols, sl, u, lane);
}
template <typename IO, int NW>
__device__ __forceinline__ void bwd_piece(uint32_t prow0, uint32_t grow0, int rows, int cols, float scale,
                                          int u, int lane) {
    if (cols >= 8 * IO::VE) {
        bwd_rows_vec<IO, NW>(prow0, grow0, rows, cols, scale, u, lane);
        return;
    }
    const int ur = sp_unit_rows(cols);
#pragma unroll 1
    for (int r = u * ur; r < rows; r += NW * ur) {
        if (cols <= SP_LANE_COLS) bwd_rows_lane<IO>(prow0, grow0, rows, cols, scale, r, lane);
        else bwd_rows_group<IO>(prow0, grow0, rows, cols, scale, r, lane);
    }
}

template <int NW>
__device__ __forceinline__ void sp_compute_sync() {  // among the computing warps
    asm volatile("bar.sync 1, %0;\n" ::"n"(32 * NW) : "memory");
}
template <int NW>
__device__ __forceinline__ float sp_cta_reduce(float v, bool is_max, float* red, int warp, int lane) {
    v = is_max ? sp_max(v, 32) : sp_sum(v, 32);
    sp_compute_sync<NW>();  // red may still be read from the previous reduction
    if (lane == 0) red[warp] = v;
    sp_compute_sync<NW>();
    float r = red[0];
#pragma unroll
    for (int w = 1; w < NW; ++w) r = is_max ? fmaxf(r, red[w]) : r + red[w];
    return r;
}

// forward, one row longer than a window, from and to global memory by all computing warps (out of line, like fwd_row_far)
template <typename IO, bool NEG, int NW>
__device__ __noinline__ void fwd_wide_row(const typename IO::E* src, typename IO::E* dst, int cols, float sl, float* red, int tid) {
    constexpr int NT = 32 * NW;
    constexpr float SIGN = NEG ? -1.f : 1.f;
    const int warp = tid >> 5, lane = tid & 31;
    float m = -INFINITY;
    for (int c = tid; c < cols; c += NT) m = fmaxf(m, SIGN * IO::ld(src[c]));
    m = SIGN * sp_cta_reduce<NW>(m, true, red, warp, lane);
    auto normalise = [&](auto y) {
        float sum = 0.f;
        for (int c = tid; c < cols; c += NT) sum += blk_exp2(y(IO::ld(src[c])));
        sum = sp_cta_reduce<NW>(sum, false, red, warp, lane);
        const float inv = 1.f / sum;
        for (int c = tid; c < cols; c += NT) dst[c] = IO::st(blk_exp2(y(IO::ld(src[c]))) * inv);
    };
    const float mx = m * sl;
    if (fabsf(mx) <= sp_near<SpIO32>()) normalise([&](float x) { return fmaf(x, sl, -mx); });
    else normalise([&](float x) { return (x - m) * sl; });
}

// A window in its stage.
struct SpWin {
    int64_t e0;   // its first element in the buffers
    int64_t off;  // ... inside the head strip
    int nbytes, npieces, first_piece;
};

// The (window, head) list of a CTA: window index and head of entry blockIdx.x, + gridDim.x, ...
struct SpWalk {
    int idx, head, didx, dhead;
    bool has;
    __device__ __forceinline__ explicit SpWalk(const BlkSmxPipeParams& p) {
        head = (int)(blockIdx.x / (unsigned)p.num_windows);
        idx = (int)(blockIdx.x - (unsigned)head * (unsigned)p.num_windows);
        dhead = (int)(gridDim.x / (unsigned)p.num_windows);
        didx = (int)(gridDim.x - (unsigned)dhead * (unsigned)p.num_windows);
        has = head < p.H;
    }
    __device__ __forceinline__ void step(const BlkSmxPipeParams& p) {
        idx += didx;
        head += dhead;
        if (idx >= p.num_windows) {
            idx -= p.num_windows;
            ++head;
        }
        has = head < p.H;
    }
    __device__ __forceinline__ SpWin load(const BlkSmxPipeParams& p) const {
        const BlkSmxWindow w = p.windows[idx];
        return SpWin{(int64_t)head * p.D + w.off, w.off, w.nbytes, w.npieces, w.first_piece};
    }
};

// BWD = false: in0 = src, result = softmax (NEG: of a negative scale); BWD = true: in0 = forward result, in1 = its gradient.
template <typename IO, bool BWD, bool NEG>
__global__ void __launch_bounds__(SpShape<BWD>::THREADS, SpShape<BWD>::CTAS) blk_softmax_pipe_kernel(const BlkSmxPipeParams p) {
    typedef typename IO::E E;
    constexpr int ES = (int)sizeof(E);
    constexpr int NIN = BWD ? 2 : 1;
    constexpr int NW = SpShape<BWD>::NW, ST = SpShape<BWD>::STAGES;
    extern __shared__ __align__(128) unsigned char sp_smem[];  // [stages][NIN][SP_BUF]
    __shared__ __align__(8) uint64_t bars[2 * ST];             // full[stage], done[stage]
    __shared__ float red[NW];
    __shared__ SpWin wins[ST];
    __shared__ __align__(16) BlkSmxChunk recs[ST][BLK_SMX_WINDOW_PIECES];  // the windows' piece records, per stage
    __shared__ volatile int abort_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bar0 = blk_smem_u32(bars);
    auto full = [&](int st) { return bar0 + 8u * st; };
    auto done = [&](int st) { return bar0 + 8u * (ST + st); };
    auto buf = [&](int st, int in) { return sp_smem + (st * NIN + in) * SP_BUF; };
    if (tid == 0) {
        for (int i = 0; i < ST; ++i) {
            sp_bar_init(full(i), 1);
            sp_bar_init(done(i), NW);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    blk_grid_wait();

    const E* g0 = reinterpret_cast<const E*>(p.in0);
    const E* g1 = reinterpret_cast<const E*>(p.in1);
    E* gd = reinterpret_cast<E*>(p.out);

    if (warp == NW) {
        // ---------------- the copying warp ----------------
        SpWalk next(p);   // the next window to fetch
        SpWin rec = {};
        if (next.has) rec = next.load(p);
        // lane 0: start the copies of the next window into stage st (none for a row longer than a window)
        auto issue = [&](int st) {
            wins[st] = rec;
            const bool fits = rec.nbytes <= SP_WIN;
            const int64_t a = rec.e0 * ES;  // byte offset of the window in each buffer
            const int mis = (int)(a & 15);
            const uint32_t bytes = fits ? (uint32_t)((mis + rec.nbytes + 15) & ~15) : 0u;
            const uint32_t rbytes = fits ? (uint32_t)rec.npieces * (uint32_t)sizeof(BlkSmxChunk) : 0u;
            sp_expect_tx(full(st), NIN * bytes + rbytes);
            if (fits) {
                sp_bulk_g2s(blk_smem_u32(recs[st]), p.pieces + rec.first_piece, rbytes, full(st));
                sp_bulk_g2s(blk_smem_u32(buf(st, 0)), reinterpret_cast<const unsigned char*>(g0) + (a - mis), bytes, full(st));
                if (BWD)
                    sp_bulk_g2s(blk_smem_u32(buf(st, 1)), reinterpret_cast<const unsigned char*>(g1) + (a - mis), bytes, full(st));
            }
            next.step(p);
            if (next.has) rec = next.load(p);
        };
        if (lane == 0) {
#pragma unroll 1
            for (int i = 0; i < ST && next.has; ++i) issue(i);
        }
        SpWalk cur(p);
#pragma unroll 1
        for (uint32_t k = 0; cur.has; cur.step(p), ++k) {
            const int st = (int)(k % ST);
            if (!__all_sync(0xffffffffu, sp_wait(done(st), (k / ST) & 1u, &abort_flag) && !abort_flag)) break;
            const int64_t e0 = wins[st].e0;
            const int nbytes = wins[st].nbytes;
            if (nbytes <= SP_WIN) {
                // aligned vectors wholly inside the window: one bulk store; ragged edges: single elements
                const int mis = (int)((e0 * ES) & 15);
                unsigned char* res = buf(st, BWD ? 1 : 0);  // the buffer that holds the result
                const int span = mis + nbytes;
                const int lo = mis ? 16 : 0, hi = span & ~15;
                unsigned char* dst_al = reinterpret_cast<unsigned char*>(gd) + (e0 * ES - mis);
                if (lane == 0 && hi > lo) sp_bulk_s2g(dst_al + lo, blk_smem_u32(res + lo), (uint32_t)(hi - lo));
                // head edge: bytes [mis, min(lo, span)); tail edge: bytes [max(hi, lo), span)  (hi >= lo or the window is tiny)
                const int h_end = lo < span ? lo : span;
                const int b = mis + lane * ES;
                if (lane < 16 / ES && b < h_end) *reinterpret_cast<E*>(dst_al + b) = *reinterpret_cast<const E*>(res + b);
                const int t0 = hi > h_end ? hi : h_end;
                const int bt = t0 + (lane - 16) * ES;
                if (lane >= 16 && lane < 16 + 16 / ES && bt < span)
                    *reinterpret_cast<E*>(dst_al + bt) = *reinterpret_cast<const E*>(res + bt);
            }
            __syncwarp();
            if (lane == 0) {
                sp_bulk_commit();
                // the stage of the window before this one is free once its bulk store is done with shared memory
                if (k > 0 && next.has) {
                    sp_bulk_wait_read1();
                    issue((int)((k - 1) % ST));
                }
            }
        }
        if (lane == 0) sp_bulk_wait_all();
    } else {
        // ---------------- computing warps ----------------
        const float sl = BWD ? p.scale : p.scale * BLK_LOG2E;
        constexpr int LONG = 8 * IO::VE;  // rows of at least this many columns take a warp each
        int turn = warp;                  // the unit of the next window, counted from its first, that is this warp's
        bool ok = true;
        SpWalk cur(p);
#pragma unroll 1
        for (uint32_t k = 0; cur.has; cur.step(p), ++k) {
            const int st = (int)(k % ST);
            ok = __all_sync(0xffffffffu, ok && sp_wait(full(st), (k / ST) & 1u, &abort_flag));
            const SpWin win = ok ? wins[st] : cur.load(p);
            if (win.nbytes > SP_WIN) {
                // one row longer than a window: streamed from global memory by all computing warps
                const int cols = p.pieces[win.first_piece].cols;
                const int64_t e0 = win.e0;
                constexpr int NT = 32 * NW;
                if (!BWD) {
                    fwd_wide_row<IO, NEG, NW>(g0 + e0, gd + e0, cols, sl, red, tid);
                } else {
                    float dot = 0.f;
                    for (int c = tid; c < cols; c += NT) dot += IO::ld(g0[e0 + c]) * IO::ld(g1[e0 + c]);
                    dot = sp_cta_reduce<NW>(dot, false, red, warp, lane);
                    for (int c = tid; c < cols; c += NT)
                        gd[e0 + c] = IO::st((IO::ld(g1[e0 + c]) - dot) * IO::ld(g0[e0 + c]) * sl);
                }
            } else if (ok) {
                const int mis = (int)((win.e0 * ES) & 15);
                const uint32_t r0 = blk_smem_u32(buf(st, BWD ? 1 : 0)) + mis, p0 = blk_smem_u32(buf(st, 0)) + mis;
                auto piece = [&](int pi, int first) {
                    const BlkSmxChunk pc = recs[st][pi];
                    const uint32_t eo = (uint32_t)(pc.off - win.off) * ES;
                    if (BWD) bwd_piece<IO, NW>(p0 + eo, r0 + eo, pc.rows, pc.cols, sl, first, lane);
                    else fwd_piece<IO, NEG, NW>(r0 + eo, pc.rows, pc.cols, sl, first, lane);
                };
                auto units_of = [&](int pi) {
                    const BlkSmxChunk pc = recs[st][pi];
                    if (pc.cols >= LONG) return (int)pc.rows;
                    const int ur = sp_unit_rows(pc.cols);
                    return (int)(pc.rows + ur - 1) / ur;
                };
                // The window's units -- a row of a piece of long rows, a group of short ones -- go to the warps in turn, from
                // window to window.  A lane counts those of one piece; a warp then visits the pieces that hold one of its
                // own.  (A window of one piece, the usual one of wide segments, needs no counting.)
                if (win.npieces == 1) {
                    const int n = units_of(0);
                    if (turn < n) piece(0, turn);
                    turn += (n > turn ? (n - turn + NW - 1) / NW * NW : 0) - n;
                } else {
#pragma unroll 1
                    for (int base = 0; base < win.npieces; base += 32) {
                        const int units = base + lane < win.npieces ? units_of(base + lane) : 0;
                        int incl = units;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const int v = __shfl_up_sync(0xffffffffu, incl, o);
                            if (lane >= o) incl += v;
                        }
                        const int excl = incl - units;
                        // this warp's first unit of the piece: the smallest turn + i NW >= excl
                        const int first = turn + (excl > turn ? (excl - turn + NW - 1) / NW * NW : 0) - excl;
                        uint32_t mine = __ballot_sync(0xffffffffu, first < units);
                        while (mine) {
                            const int src = __ffs(mine) - 1;
                            mine &= mine - 1;
                            piece(base + src, __shfl_sync(0xffffffffu, first, src));
                        }
                        const int n = __shfl_sync(0xffffffffu, incl, 31);
                        turn += (n > turn ? (n - turn + NW - 1) / NW * NW : 0) - n;
                    }
                }
            }
            // results (generic-proxy writes) must be visible to the bulk store (async proxy)
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) sp_arrive(done(st));
        }
    }
    __syncthreads();
    if (tid == 0 && abort_flag) {
        atomicCAS(p.status, 0, 21);
        for (int i = 0; i < 64; ++i) __nanosleep(1000);  // copies in flight land before the CTA's memory is released
    }
}

}  // namespace

cudaError_t blk_launch_softmax_pipe(const BlkSmxPipeParams& p, int dtype, int backward, int sms, cudaStream_t st) {
    const int64_t total = (int64_t)p.num_windows * p.H;
    if (total == 0) return cudaSuccess;
    auto go = [&](auto kern, int nin, auto shape) -> cudaError_t {
        typedef decltype(shape) S;
        const int smem = S::STAGES * nin * SP_BUF;
        cudaError_t e = blk_func_smem(reinterpret_cast<const void*>(kern), smem);
        if (e != cudaSuccess) return e;
        const int64_t resident = (int64_t)sms * S::CTAS;
        const dim3 grid((unsigned)(total < resident ? total : resident)), block(S::THREADS);
        // (an early start up to about 100 us: blocks that come one by one take a hundredth longer (778 -> 785 us for the scores of 512
        // segments of 16..2048 rows, 4 heads); it saves 2 of 45)
        return blk_launch(total <= 32 * resident, kern, grid, block, smem, st, p);
    };
    auto forward = [&](auto io) {
        typedef decltype(io) IO;
        return p.scale < 0.f ? go(blk_softmax_pipe_kernel<IO, false, true>, 1, SpShape<false>{})
                             : go(blk_softmax_pipe_kernel<IO, false, false>, 1, SpShape<false>{});
    };
    if (!backward)
        return dtype == BLK_F16 ? forward(SpIO16<BlkHalfTag>{}) : dtype == BLK_BF16 ? forward(SpIO16<BlkBf16Tag>{}) : forward(SpIO32{});
    if (dtype == BLK_F16) return go(blk_softmax_pipe_kernel<SpIO16<BlkHalfTag>, true, false>, 2, SpShape<true>{});
    if (dtype == BLK_BF16) return go(blk_softmax_pipe_kernel<SpIO16<BlkBf16Tag>, true, false>, 2, SpShape<true>{});
    return go(blk_softmax_pipe_kernel<SpIO32, true, false>, 2, SpShape<true>{});
}

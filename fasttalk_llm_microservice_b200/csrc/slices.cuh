// fp32 operands on the fp16 tensor cores without losing fp32 accuracy: every number as three fp16 slices.
//
// tcgen05 adds exact products into fp32 accumulators but cuts off what lies below the accumulator's last bit (toward zero, measured: sums of
// 128 products of random bf16 numbers are 7e-8 too small on average, of 2048 products 1.7e-6).  So the first slice is a whole number of
// at most 2^kSliceBits in units of a power of two that a whole row (or tile) shares: sums of products of first slices are whole numbers below
// 2^24 and hence exact, in whatever order they are added.  The remainder, at most half a unit, is an fp16 number (11 bits) and the
// remainder of that another one.  Of the nine products of two triples six are taken: first x first into one accumulator, the five others
// (2^-10 and less of it, so that their cut-off bits do not matter) into a second one; the two meet in an ordinary rounded fp32 addition.
// What is left out is below 2^-22 of a unit squared.  Against 64 bits a contraction of 128 comes out as near as with fused fp32
// multiply-adds in order, or nearer.
#pragma once
#include "common.cuh"

namespace ft {

constexpr int kSliceBits = 10;
constexpr float kSliceMagic = 12582912.f;               // 1.5 * 2^23: x + magic - magic is x rounded to a whole number

__device__ __forceinline__ unsigned warp_umax(unsigned v) { return __reduce_max_sync(0xffffffffu, v); }
// Bit patterns of |x| order as the numbers do, infinities and NaN above all of them.
__device__ __forceinline__ unsigned abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }
constexpr int kSliceMinExp = -100;                      // rows below 2^-100 share its unit
// 1 / unit and unit of numbers whose largest has these bits (finite, below 2^80)
__device__ __forceinline__ int slice_exp(unsigned top) { return max((int)(top >> 23) - 127, kSliceMinExp); }
__device__ __forceinline__ float slice_inv(unsigned top) { return __uint_as_float((unsigned)(127 + kSliceBits - 1 - slice_exp(top)) << 23); }
__device__ __forceinline__ float slice_unit(unsigned top) { return __uint_as_float((unsigned)(127 + slice_exp(top) - (kSliceBits - 1)) << 23); }

__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
    __half2 t = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&t);
}
// Two fp32 numbers ride in each f32x2: half the instructions.
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// the largest size of three, NaN if one of them is
__device__ __forceinline__ float top3(float a, float b, float c) {
    float r;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
template <int N>
__device__ __forceinline__ float top_of(const f32x2* x, float m = 0.f) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float u, v;
        unpack2(x[i], u, v);
        m = top3(m, u, v);
    }
    return m;
}
// One slice of N pairs as packed fp16; x becomes the remainder.  slice_first: x comes in numbers, leaves in units.
template <int N>
__device__ __forceinline__ void slice_first(f32x2* x, float inv, uint32_t* out) {
    const f32x2 i2 = pack2(inv, inv), up = pack2(kSliceMagic, kSliceMagic), down = pack2(-kSliceMagic, -kSliceMagic), minus = pack2(-1.f, -1.f);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const f32x2 y = mul2(x[i], i2), h = add2(add2(y, up), down);      // the product with a power of two is exact
        float u, v;
        unpack2(h, u, v);
        out[i] = pack_f16(u, v);
        x[i] = fma2(h, minus, y);
    }
}
template <int N>
__device__ __forceinline__ void slice_next(f32x2* x, uint32_t* out) {
    const f32x2 minus = pack2(-1.f, -1.f);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float u, v;
        unpack2(x[i], u, v);
        out[i] = pack_f16(u, v);
        const float2 m = __half22float2(*reinterpret_cast<__half2*>(&out[i]));
        x[i] = fma2(pack2(m.x, m.y), minus, x[i]);
    }
}
template <int N>
__device__ __forceinline__ void slice_last(const f32x2* x, uint32_t* out) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float u, v;
        unpack2(x[i], u, v);
        out[i] = pack_f16(u, v);
    }
}
// four numbers -> 8 bytes of each slice, `plane` bytes apart; eight -> 16
__device__ __forceinline__ void slice4(f32x2* x, float inv, uint8_t* at, int plane) {
    uint32_t w[2];
    slice_first<2>(x, inv, w);
    *reinterpret_cast<uint2*>(at) = make_uint2(w[0], w[1]);
    slice_next<2>(x, w);
    *reinterpret_cast<uint2*>(at + plane) = make_uint2(w[0], w[1]);
    slice_last<2>(x, w);
    *reinterpret_cast<uint2*>(at + 2 * plane) = make_uint2(w[0], w[1]);
}
__device__ __forceinline__ void slice8(f32x2* x, float inv, uint8_t* at, int plane) {
    uint32_t w[4];
    slice_first<4>(x, inv, w);
    *reinterpret_cast<uint4*>(at) = make_uint4(w[0], w[1], w[2], w[3]);
    slice_next<4>(x, w);
    *reinterpret_cast<uint4*>(at + plane) = make_uint4(w[0], w[1], w[2], w[3]);
    slice_last<4>(x, w);
    *reinterpret_cast<uint4*>(at + 2 * plane) = make_uint4(w[0], w[1], w[2], w[3]);
}
// 32 lanes x 8 columns
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
                 "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// 16 numbers of a row as three slices, PITCH columns apart
template <int PITCH>
__device__ __forceinline__ void slices_to_tmem(f32x2* x, float inv, uint32_t at) {
    uint32_t w[8];
    slice_first<8>(x, inv, w);
    tmem_st8(at, w);
    slice_next<8>(x, w);
    tmem_st8(at + PITCH, w);
    slice_last<8>(x, w);
    tmem_st8(at + 2 * PITCH, w);
}
// The products beside first x first, smallest first: (slice of A, slice of B)
constexpr int kSlicePairs = 5;
__host__ __device__ constexpr int slice_a(int p) { return (0x10012 >> (4 * p)) & 0xf; }      // 2 1 0 0 1 read from the low digit: 2, 1, 0, 0, 1
__host__ __device__ constexpr int slice_b(int p) { return (0x01210 >> (4 * p)) & 0xf; }      // 0, 1, 2, 1, 0

}  // namespace ft

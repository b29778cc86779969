// fp32 operands on the bf16 tensor cores without losing fp32 accuracy: every number as three bf16 slices.
//
// A slice has fp32's exponents, so a number is its three slices whatever stands beside it: no unit is shared, and nothing is lost of a small number in a row
// or column of large ones, or beside a large one that a mask hides.  The first slice has kFirstBits bits of the number, the second eight bits of the
// remainder, the third all that is left (24 bits in all, exact down to 2^-110 or so, where the third slice runs out of exponents).
//
// Why the first slice is short: tcgen05 adds exact products into fp32 accumulators but cuts off what lies below the accumulator's last bit, toward zero.
// First slices of eight bits have products of 16, whose ends are cut off in one product of eight, and sums of 128 products of random numbers came out 7e-8 too
// small on average; products of six and six bits are cut off in one of a hundred.  Of the nine products of two triples eight are taken: first x
// first into one accumulator, the seven others (2^-6 and less of it, so that their cut-off bits do not matter) into a second one; the two
// meet in an ordinary rounded fp32 addition.  The product left out, third x third, is below 2^-29 of the numbers' own product.  (First slices of eight bits and six products
// took 118 instead of 132 us in window attention of 2313 tokens, and results were up to a quarter further from 64 bits.)
#pragma once
#include "common.cuh"

namespace ft {

constexpr int kFirstBits = 6;

// Bit patterns of |x| order as the numbers do, infinities and NaN above all of them.
__device__ __forceinline__ unsigned abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }
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
// One slice of N pairs as packed bf16; x becomes the remainder (exact).
template <int N>
__device__ __forceinline__ void slice_first(f32x2* x, uint32_t* out) {
    constexpr uint32_t keep = ~0u << (24 - kFirstBits), half = 1u << (23 - kFirstBits);
    const f32x2 minus = pack2(-1.f, -1.f);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float u, v;
        unpack2(x[i], u, v);
        const uint32_t a = (__float_as_uint(u) + half) & keep, b = (__float_as_uint(v) + half) & keep;      // rounded by size
        out[i] = __byte_perm(a, b, 0x7632);
        x[i] = fma2(pack2(__uint_as_float(a), __uint_as_float(b)), minus, x[i]);
    }
}
template <int N>
__device__ __forceinline__ void slice_next(f32x2* x, uint32_t* out) {
    const f32x2 minus = pack2(-1.f, -1.f);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float u, v;
        unpack2(x[i], u, v);
        out[i] = pack_bf16(u, v);
        x[i] = fma2(pack2(bf16_lo(out[i]), bf16_hi(out[i])), minus, x[i]);
    }
}
template <int N>
__device__ __forceinline__ void slice_last(const f32x2* x, uint32_t* out) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float u, v;
        unpack2(x[i], u, v);
        out[i] = pack_bf16(u, v);
    }
}
// four numbers -> 8 bytes of each slice, `plane` bytes apart; eight -> 16
__device__ __forceinline__ void slice4(f32x2* x, uint8_t* at, int plane) {
    uint32_t w[2];
    slice_first<2>(x, w);
    *reinterpret_cast<uint2*>(at) = make_uint2(w[0], w[1]);
    slice_next<2>(x, w);
    *reinterpret_cast<uint2*>(at + plane) = make_uint2(w[0], w[1]);
    slice_last<2>(x, w);
    *reinterpret_cast<uint2*>(at + 2 * plane) = make_uint2(w[0], w[1]);
}
__device__ __forceinline__ void slice8(f32x2* x, uint8_t* at, int plane) {
    uint32_t w[4];
    slice_first<4>(x, w);
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
__device__ __forceinline__ void slices_to_tmem(f32x2* x, uint32_t at) {
    uint32_t w[8];
    slice_first<8>(x, w);
    tmem_st8(at, w);
    slice_next<8>(x, w);
    tmem_st8(at + PITCH, w);
    slice_last<8>(x, w);
    tmem_st8(at + 2 * PITCH, w);
}
// What tcgen05 cuts off a sum of first slices is 0.75 of its last place on average over sums of random numbers, and more where all have one sign: three eighths of 2^-24
// of the sum given back leave no mean error in the former, and less in the latter.  m: first x first, r: the other products.
constexpr float kCutBack = 0.375f / 16777216.f;
__device__ __forceinline__ f32x2 rest_of(f32x2 m, f32x2 r) { return fma2(add2(m, r), pack2(kCutBack, kCutBack), r); }
__device__ __forceinline__ float rest_of(float m, float r) { return __fmaf_rn(m + r, kCutBack, r); }
// The products beside first x first, smallest first: (slice of A, slice of B)
constexpr int kSlicePairs = 7;
__host__ __device__ constexpr int slice_a(int p) { return (0x1001212 >> (4 * p)) & 0xf; }      // read from the low digit: 2, 1, 2, 1, 0, 0, 1
__host__ __device__ constexpr int slice_b(int p) { return (0x0121021 >> (4 * p)) & 0xf; }      // 1, 2, 0, 1, 2, 1, 0
// Instruction descriptor of their products; mn: B is an MN-major tile
__host__ __device__ constexpr uint32_t slice_idesc(int M, int N, bool mn = false) { return umma_idesc_bf16(M, N) | (mn ? 1u << 16 : 0u); }

}  // namespace ft

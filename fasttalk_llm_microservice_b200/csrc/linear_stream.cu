// Projections of a few rows on the CUDA cores (decode steps of a few sessions, the experts of a step of few pairs), fp32 activations times
// bf16 weights.  The weights' way from memory is all that counts: a CTA brings NC weight rows of one problem whole into shared memory with
// bulk copies, all of them on the way from the start, needs no registers for them, and takes the problem's rows past them four at a time, so
// that a second group of rows reads nothing again.  A warp holds eight weight rows' sums of four rows over its share of K and reads the rows'
// numbers straight into registers while the weights land.
//
// The kernel by rows (layered.cu: a warp per four columns, 16 bytes of each on the way, rows staged first) took 30.8 and 25 us for the 32 pairs of 16
// sessions over 16 experts of 1024 x 2048 and of 2048 x 1024 (58 MB of weights each, 9 us at the copy rate); this one takes 19 each.
//
// The wait for the weights has a limit; a CTA whose wait runs out marks `err`, leaves NaN and ends.
#include "common.cuh"
#include "ft_internal.h"

namespace ft {
namespace {

constexpr int LS_WARPS = 8, LS_ROWS = 4, LS_STEP = 256;      // a step: 8 channels of K per lane
constexpr int LS_MAX_BYTES = 100 * 1024;                     // of weights: two CTAs per SM

// 32 sums per lane over the lanes of a warp: lane l ends with that of index l
__device__ __forceinline__ float transpose_sum(float (&v)[32], int lane) {
#pragma unroll
    for (int half = 16; half >= 1; half >>= 1) {
        const bool up = (lane & half) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float give = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
        }
    }
    return v[0];
}

template <bool PAIR, int NC>
__global__ void __launch_bounds__(LS_WARPS * 32) linear_stream_kernel(LinearArgs a, int* err) {
    pdl_wait();
    constexpr int HALVES = NC / 8;                           // groups of eight weight rows
    extern __shared__ __align__(128) uint8_t ls_w[];
    __shared__ float red[LS_WARPS][32];
    __shared__ uint64_t full;
    __shared__ volatile int dead;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, p = blockIdx.y, n0 = blockIdx.x * NC;
    int r0 = 0, r1 = a.M;
    if (a.seg) { r0 = a.seg[p]; r1 = a.seg[p + 1]; }
    if (r1 <= r0) return;
    const int rows_w = min(NC, a.N - n0), row_bytes = a.K * 2;
    if (tid == 0) {
        mbar_init(&full, 1);
        fence_mbar_init();
        dead = 0;
        mbar_expect_tx(&full, (uint32_t)(rows_w * row_bytes));
    }
    __syncthreads();
    if (tid < rows_w)
        tma_bulk_g2s(ls_w + (size_t)tid * row_bytes, a.W + (size_t)p * a.w_stride + (size_t)(n0 + tid) * a.ldw, row_bytes, &full, policy_evict_first());
    const float* A = a.A + (size_t)p * a.a_col_stride;
    float* C = a.C + (size_t)p * a.c_col_stride;
    const int half = warp % HALVES, k_first = warp / HALVES * LS_STEP + lane * 8;
    constexpr int K_NEXT = LS_WARPS / HALVES * LS_STEP;
    const uint8_t* wt = ls_w + (size_t)half * 8 * row_bytes;
    bool ok = true;
    for (int rb = r0; rb < r1; rb += LS_ROWS) {
        const int nr = min(LS_ROWS, r1 - rb);
        const float* src[LS_ROWS];
#pragma unroll
        for (int i = 0; i < LS_ROWS; ++i) {
            const int r = rb + min(i, nr - 1);
            src[i] = A + (size_t)(a.a_rows ? a.a_rows[r] : r) * a.lda;
        }
        float acc[32];                                       // [weight row of eight][row of four]
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = 0.f;
        for (int k = k_first; k < a.K; k += K_NEXT) {
            float x[LS_ROWS][8];
#pragma unroll
            for (int i = 0; i < LS_ROWS; ++i) {
                if (i >= nr) break;
                *reinterpret_cast<float4*>(x[i]) = *reinterpret_cast<const float4*>(src[i] + k);
                *reinterpret_cast<float4*>(x[i] + 4) = *reinterpret_cast<const float4*>(src[i] + k + 4);
            }
            if (ok) ok = mbar_wait_limited(&full, 0, &dead);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const uint4 t = *reinterpret_cast<const uint4*>(wt + (size_t)c * row_bytes + k * 2);      // (rows beyond N: never written out)
                const float w[8] = {bf16_lo(t.x), bf16_hi(t.x), bf16_lo(t.y), bf16_hi(t.y), bf16_lo(t.z), bf16_hi(t.z), bf16_lo(t.w), bf16_hi(t.w)};
#pragma unroll
                for (int i = 0; i < LS_ROWS; ++i) {
                    if (i >= nr) break;
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[c * LS_ROWS + i] = fmaf(x[i][e], w[e], acc[c * LS_ROWS + i]);
                }
            }
        }
        if (ok) ok = mbar_wait_limited(&full, 0, &dead);     // a warp without a step of its own
        red[warp][lane] = transpose_sum(acc, lane);
        ok = __syncthreads_and(ok);
        // thread (output, row): the warps' sums of one weight row, or of a pair's two
        constexpr int OUT = PAIR ? NC / 2 : NC;
        const int j = tid / LS_ROWS, i = tid % LS_ROWS;
        if (tid < OUT * LS_ROWS && i < nr) {
            auto total = [&](int c) {
                float s = 0.f;
#pragma unroll
                for (int q = 0; q < LS_WARPS / HALVES; ++q) s += red[q * HALVES + c / 8][c % 8 * LS_ROWS + i];
                return s;
            };
            const int col = (PAIR ? n0 / 2 : n0) + j;
            if (col < (PAIR ? a.N / 2 : a.N)) {
                float v;
                if (PAIR) {
                    v = glu_value(a.glu, total(2 * j), total(2 * j + 1), col);
                } else {
                    v = total(j);
                    if (a.epi == LIN_SOFTCAP) v = a.cap * tanhf(v / a.cap);
                    else if (a.epi == LIN_RELU2) { v = fmaxf(v, 0.f); v *= v; }
                    if (a.gate) v *= 1.f / (1.f + expf(-a.gate[(size_t)(rb + i) * a.ldg + (size_t)p * a.c_col_stride + col]));
                }
                if (!ok) v = __int_as_float(0x7fc00000);
                if (a.C16) a.C16[(size_t)(rb + i) * a.ldc + (size_t)p * a.c_col_stride + col] = __float2bfloat16_rn(v * a.c16_scale);
                else C[(size_t)(rb + i) * a.ldc + col] = v;
            }
        }
        __syncthreads();
    }
    if (!ok && tid == 0) {                                   // the results are NaN; the CTA's copies may still be on their way into its memory
        if (err) *err = 1;
        for (int i = 0; i < kWaitLimit && !mbar_try_wait(&full, 0); ++i) {}
    }
}

int weight_rows(int K) { return (size_t)16 * K * 2 <= LS_MAX_BYTES ? 16 : (size_t)8 * K * 2 <= LS_MAX_BYTES ? 8 : 0; }

template <bool PAIR, int NC>
int launch(const LinearArgs& a, int* err, cudaStream_t stream) {
    static PerDeviceFlag attr;
    if (!attr.done()) {
        FT_CHECK_CUDA(cudaFuncSetAttribute(linear_stream_kernel<PAIR, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, LS_MAX_BYTES));
        attr.mark();
    }
    launch_after(linear_stream_kernel<PAIR, NC>, dim3((a.N + NC - 1) / NC, a.P), LS_WARPS * 32, (size_t)NC * a.K * 2, stream, a, err);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace

// Rows and weights on 16 bytes, K long enough that a warp has a whole step.
bool linear_stream_ok(const LinearArgs& a) {
    return a.K >= 512 && weight_rows(a.K) > 0 && (a.K & 7) == 0 && (a.ldw & 7) == 0 && (a.lda & 3) == 0 && (a.a_col_stride & 3) == 0 && (a.w_stride & 7) == 0 &&
           ((uintptr_t)a.A & 15) == 0 && ((uintptr_t)a.W & 15) == 0;
}
long long linear_stream_ctas(const LinearArgs& a) { return (long long)a.P * ((a.N + weight_rows(a.K) - 1) / weight_rows(a.K)); }
int launch_linear_stream(const LinearArgs& a, int* err, cudaStream_t stream) {
    FT_REQUIRE(linear_stream_ok(a) && a.P <= 65535, "linear (few rows): K %d, row strides %d and %d do not fit", a.K, a.lda, a.ldw);
    const bool pair = a.epi == LIN_SWIGLU_PAIR;
    if (weight_rows(a.K) == 16) return pair ? launch<true, 16>(a, err, stream) : launch<false, 16>(a, err, stream);
    return pair ? launch<true, 8>(a, err, stream) : launch<false, 8>(a, err, stream);
}

}  // namespace ft

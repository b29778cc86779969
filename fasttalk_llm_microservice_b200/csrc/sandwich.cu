// The joint of the sandwich layer form (FT_LAYER_SANDWICH): the ONE kernel between two GEMM chains of a layer, one CTA per row.
// It gathers the sublayer's result (the scaled sum of up to two branch results, or the experts' rows plus a dense or shared
// result and its bias), norms it, adds it to the stream, and norms the stream for what reads it next, writing the bf16 planes as
// well — or, ahead of a pass over looped layers, lays the stream down beside the embedding output.  A step's first joint
// fills the stream from the embedding table.  Everything is fp32; the embedding table is bf16.
#include "common.cuh"
#include "ft_internal.h"
#include "rows.cuh"

namespace ft {
namespace {

// V: columns per thread and pass (4 when the width is a multiple of four and every row starts on 16 bytes)
template <int V>
__device__ __forceinline__ void put_row(float* f32, void* hi, void* lo, size_t at, const float (&v)[V]) {
    st_cols<V>(f32 + at, v);
    if (hi) st_planes<V>((__nv_bfloat16*)hi + at, (__nv_bfloat16*)lo + at, v);
}

template <int V>
__global__ void __launch_bounds__(256) sandwich_joint_kernel(SandwichArgs a) {
    pdl_wait();
    __shared__ float red[33];
    extern __shared__ __align__(16) float row[];          // [W]: the sublayer's result, then the new row of the stream
    const int t = blockIdx.x, W = a.W;
    const bool sub = a.y0 || a.y1 || a.top > 0;
    float* xr = a.x + (size_t)t * W;
    float r1 = 0.f;
    if (sub) {
        float ss = 0.f;
        for (int c = threadIdx.x * V; c < W; c += blockDim.x * V) {
            float y[V], v[V];
#pragma unroll
            for (int i = 0; i < V; ++i) y[i] = 0.f;
            for (int k = 0; k < a.top; ++k) {
                ld_cols<V>(v, a.eout + (size_t)a.slot_pos[(size_t)t * a.top + k] * W + c);
                const float wk = a.wt[(size_t)t * a.top + k];
#pragma unroll
                for (int i = 0; i < V; ++i) y[i] = fmaf(wk, v[i], y[i]);
            }
            if (a.y0) {
                ld_cols<V>(v, a.y0 + (size_t)t * W + c);
#pragma unroll
                for (int i = 0; i < V; ++i) y[i] = fmaf(a.s0, v[i], y[i]);
            }
            if (a.b0) {
                ld_cols<V>(v, a.b0 + c);
#pragma unroll
                for (int i = 0; i < V; ++i) y[i] += v[i];
            }
            if (a.y1) {
                ld_cols<V>(v, a.y1 + (size_t)t * W + c);
#pragma unroll
                for (int i = 0; i < V; ++i) y[i] = fmaf(a.s1, v[i], y[i]);
            }
            st_cols<V>(row + c, y);
#pragma unroll
            for (int i = 0; i < V; ++i) ss = fmaf(y[i], y[i], ss);
        }
        r1 = 1.f / sqrtf(cta_total(ss, red) / (float)W + a.eps);
    }
    const __nv_bfloat16* emb = a.tokens ? (const __nv_bfloat16*)a.embed + (size_t)a.tokens[t] * W : nullptr;
    float s2 = 0.f;
    for (int c = threadIdx.x * V; c < W; c += blockDim.x * V) {
        float x[V];
        if (emb) {
            ld_cols_bf16<V>(x, emb + c);
#pragma unroll
            for (int i = 0; i < V; ++i) x[i] *= a.embed_scale;
        } else {
            ld_cols<V>(x, xr + c);
        }
        if (sub) {
            float y[V], w[V];
            ld_cols<V>(y, row + c);
            ld_cols<V>(w, a.post_w + c);
#pragma unroll
            for (int i = 0; i < V; ++i) x[i] += y[i] * r1 * w[i];
        }
        if (sub || emb) st_cols<V>(xr + c, x);
        if (a.cat_x) put_row<V>(a.cat, a.cat_hi, a.cat_lo, (size_t)t * 2 * W + c, x);
        if (a.cat_x0) put_row<V>(a.cat, a.cat_hi, a.cat_lo, (size_t)t * 2 * W + W + c, x);
        st_cols<V>(row + c, x);
#pragma unroll
        for (int i = 0; i < V; ++i) s2 = fmaf(x[i], x[i], s2);
    }
    if (!a.next_w) return;
    const float r2 = 1.f / sqrtf(cta_total(s2, red) / (float)W + a.eps);
    for (int c = threadIdx.x * V; c < W; c += blockDim.x * V) {
        float x[V], w[V];
        ld_cols<V>(x, row + c);
        ld_cols<V>(w, a.next_w + c);
#pragma unroll
        for (int i = 0; i < V; ++i) x[i] = x[i] * r2 * w[i];
        put_row<V>(a.hn, a.hi, a.lo, (size_t)t * W + c, x);
    }
}

// The same with a row's numbers in registers, N passes of them: every load is on the way before the first sum, two barriers in all.
template <int N>
__global__ void __launch_bounds__(256) sandwich_joint_regs_kernel(SandwichArgs a) {
    pdl_wait();
    __shared__ float red[2][8];
    const int t = blockIdx.x, W = a.W, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool sub = a.y0 || a.y1 || a.top > 0;
    float* xr = a.x + (size_t)t * W;
    const __nv_bfloat16* emb = a.tokens ? (const __nv_bfloat16*)a.embed + (size_t)a.tokens[t] * W : nullptr;
    float x[N][4], y[N][4], w1[N][4], w2[N][4];
    auto total = [&](float v, float* r) {
        v = warp_sum(v);
        if (lane == 0) r[warp] = v;
        __syncthreads();
        return ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
    };
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const int c = (n * 256 + threadIdx.x) * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i) x[n][i] = y[n][i] = w1[n][i] = w2[n][i] = 0.f;
        if (c >= W) continue;
        if (emb) {
            ld_cols_bf16<4>(x[n], emb + c);
#pragma unroll
            for (int i = 0; i < 4; ++i) x[n][i] *= a.embed_scale;
        } else {
            ld_cols<4>(x[n], xr + c);
        }
        if (sub) ld_cols<4>(w1[n], a.post_w + c);
        if (a.next_w) ld_cols<4>(w2[n], a.next_w + c);
        float v[4];
        for (int k = 0; k < a.top; ++k) {
            ld_cols<4>(v, a.eout + (size_t)a.slot_pos[(size_t)t * a.top + k] * W + c);
            const float wk = a.wt[(size_t)t * a.top + k];
#pragma unroll
            for (int i = 0; i < 4; ++i) y[n][i] = fmaf(wk, v[i], y[n][i]);
        }
        if (a.y0) {
            ld_cols<4>(v, a.y0 + (size_t)t * W + c);
#pragma unroll
            for (int i = 0; i < 4; ++i) y[n][i] = fmaf(a.s0, v[i], y[n][i]);
        }
        if (a.b0) {
            ld_cols<4>(v, a.b0 + c);
#pragma unroll
            for (int i = 0; i < 4; ++i) y[n][i] += v[i];
        }
        if (a.y1) {
            ld_cols<4>(v, a.y1 + (size_t)t * W + c);
#pragma unroll
            for (int i = 0; i < 4; ++i) y[n][i] = fmaf(a.s1, v[i], y[n][i]);
        }
    }
    if (sub) {
        float ss = 0.f;
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) ss = fmaf(y[n][i], y[n][i], ss);
        const float r1 = 1.f / sqrtf(total(ss, red[0]) / (float)W + a.eps);
#pragma unroll
        for (int n = 0; n < N; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) x[n][i] += y[n][i] * r1 * w1[n][i];
    }
    float s2 = 0.f;
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const int c = (n * 256 + threadIdx.x) * 4;
        if (c >= W) continue;
        if (sub || emb) st_cols<4>(xr + c, x[n]);
        if (a.cat_x) put_row<4>(a.cat, a.cat_hi, a.cat_lo, (size_t)t * 2 * W + c, x[n]);
        if (a.cat_x0) put_row<4>(a.cat, a.cat_hi, a.cat_lo, (size_t)t * 2 * W + W + c, x[n]);
#pragma unroll
        for (int i = 0; i < 4; ++i) s2 = fmaf(x[n][i], x[n][i], s2);
    }
    if (!a.next_w) return;
    const float r2 = 1.f / sqrtf(total(s2, red[1]) / (float)W + a.eps);
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const int c = (n * 256 + threadIdx.x) * 4;
        if (c >= W) continue;
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = x[n][i] * r2 * w2[n][i];
        put_row<4>(a.hn, a.hi, a.lo, (size_t)t * W + c, v);
    }
}

}  // namespace

int launch_sandwich_joint(const SandwichArgs& a, int T, cudaStream_t stream) {
    const bool sub = a.y0 || a.y1 || a.top > 0;
    FT_REQUIRE(a.x && (!sub || a.post_w) && (!a.next_w || a.hn) && (a.next_w || a.cat_x) && (!(a.cat_x || a.cat_x0) || a.cat) &&
                   (!a.tokens || a.embed) && (!a.cat_x0 || a.tokens) && (a.top == 0 || (a.eout && a.wt && a.slot_pos)),
               "sandwich joint: missing operands");
    const size_t smem = (size_t)a.W * 4;
    FT_REQUIRE(smem <= 160 * 1024, "sandwich joint: width %d is too large", a.W);
    auto al = [](const void* p, size_t n) { return ((uintptr_t)p & (n - 1)) == 0; };
    const bool v4 = a.W % 4 == 0 && al(a.x, 16) && al(a.hn, 16) && al(a.y0, 16) && al(a.y1, 16) && al(a.b0, 16) && al(a.eout, 16) &&
                    al(a.post_w, 16) && al(a.next_w, 16) && al(a.cat, 16) && al(a.embed, 8) && al(a.hi, 8) && al(a.lo, 8) && al(a.cat_hi, 8) &&
                    al(a.cat_lo, 8);
    if (smem > 48 * 1024) {
        static PerDeviceFlag attr;
        if (!attr.done()) {
            FT_CHECK_CUDA(cudaFuncSetAttribute(sandwich_joint_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
            FT_CHECK_CUDA(cudaFuncSetAttribute(sandwich_joint_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
            attr.mark();
        }
    }
    // Few rows: up to 4096 columns in registers (16 rows of 2048: 4.1 us, through shared memory 5.4).  All joints of a step of two layers, shared memory / registers, by rows: 512 columns
    // 16: 15.2 / 12.2, 296: 16.3 / 13.2; 2048 columns 20.2 / 16.3, 22.9 / 18.4; 4096 columns 28.3 / 22.4, 32.7 / 27.7: ahead at every size up to two rows per SM.  Many rows want
    // the other kernel's occupancy (2313 rows of 2048: 16.2 us, in registers 18.4); between the two nothing was measured.
    const bool regs = v4 && T <= 2 * device_sms();
    if (regs && a.W <= 1024) launch_after(sandwich_joint_regs_kernel<1>, T, 256, 0, stream, a);
    else if (regs && a.W <= 2048) launch_after(sandwich_joint_regs_kernel<2>, T, 256, 0, stream, a);
    else if (regs && a.W <= 4096) launch_after(sandwich_joint_regs_kernel<4>, T, 256, 0, stream, a);
    else if (v4) launch_after(sandwich_joint_kernel<4>, T, 256, smem, stream, a);
    else launch_after(sandwich_joint_kernel<1>, T, 256, smem, stream, a);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace ft

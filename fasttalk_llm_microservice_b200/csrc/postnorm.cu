// Kernels of the post-norm layer form (FT_LAYER_POSTNORM) and the staging of latent window attention.  Everything fp32.
//
//   embedding            x = embed[token] * scale, also kept as X_0 of the depth history
//   input convolution    what a sublayer reads: hn = x + conv(x), a causal convolution over time per coordinate whose
//                        inputs before the step's first row come from the slot's ring of stream rows
//   post norm            x += rms(y) * gain for a sublayer's result y (one or two branch results with their biases), fused
//                        with what follows it: the ring's new rows, and either the next sublayer's input convolution or, at a
//                        layer's end, the weighted sum over depth (the new row is X_k, the stream becomes sum_j w_j X_j)
//   row norms            the model's last norm over the wanted rows; a run of columns normed to a place (latents)
#include "common.cuh"
#include "ft_internal.h"

namespace ft {

namespace {
__device__ __forceinline__ float block_sum(float v, float* red) {      // red: >= 33 floats of shared memory
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (wid == 0) {
        float t = lane < nw ? red[lane] : 0.f;
        t = warp_sum(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}
__device__ __forceinline__ void planes_put(__nv_bfloat16* hi, __nv_bfloat16* lo, size_t i, float v) {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    hi[i] = h;
    lo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
}
}  // namespace

__global__ void __launch_bounds__(256)
embed_scale_kernel(const int* __restrict__ tokens, const __nv_bfloat16* __restrict__ embed, float scale, float* __restrict__ x,
                   float* __restrict__ hist, int W) {
    pdl_wait();
    const int t = blockIdx.x;
    const __nv_bfloat16* e = embed + (size_t)tokens[t] * W;
    for (int c = threadIdx.x; c < W; c += blockDim.x) {
        const float v = __bfloat162float(e[c]) * scale;
        x[(size_t)t * W + c] = v;
        if (hist) hist[(size_t)t * W + c] = v;
    }
}
int launch_embed_scale(const int* tokens, const void* embed, float scale, float* x, float* hist, int T, int W, cudaStream_t stream) {
    launch_after(embed_scale_kernel, T, 256, 0, stream, tokens, (const __nv_bfloat16*)embed, scale, x, hist, W);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

// ------------------------------------------------------------------ input convolution
// The rows a convolution needs from before the step live in the session's slot as a ring over positions: the stream row of
// position p (as the sublayer saw it) sits in ring[p % (taps - 1)].  The ring is READ by the kernel that forms the
// sublayer's input and WRITTEN by the post-norm kernel that follows the sublayer (it still holds the rows the sublayer read):
// two launches in stream order, so a step never reads a ring entry that it has already replaced.
constexpr int kCanonMaxTaps = 17;
// A CTA takes TB tokens of 256 columns, a thread one column.  Up to four taps whose inputs are all rows of this step and of one
// request are read once for the block (2313 tokens of 2048 columns, one CTA per token: 31 us; now 15 us).
template <int TB>
__global__ void __launch_bounds__(256) canon_kernel(CanonArgs a, int T) {
    pdl_wait();
    const int t0 = blockIdx.x * TB, nt = min(TB, T - t0), W = a.W, taps = a.taps, keep = taps - 1;
    const int c = blockIdx.y * 256 + threadIdx.x;
    if (c >= W) return;
    __nv_bfloat16 *hi = (__nv_bfloat16*)a.hi, *lo = (__nv_bfloat16*)a.lo;
    auto put = [&](int t, float s) {
        a.hn[(size_t)t * W + c] = s;
        if (hi) planes_put(hi, lo, (size_t)t * W + c, s);
    };
    bool inside = TB > 1 && nt == TB && a.w && taps <= 4;
    if (inside) {
        const int req = a.seq_rows[t0];
        inside = a.seq_rows[t0 + TB - 1] == req && t0 - a.req_start[req] >= 3;
    }
    if (inside) {
        float w[4], v[TB + 3];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = i >= 4 - taps ? a.w[(size_t)c * taps + i - (4 - taps)] : 0.f;
        const float* row = a.x + (size_t)(t0 - 3) * W + c;
#pragma unroll
        for (int i = 0; i < TB + 3; ++i) v[i] = row[(size_t)i * (unsigned)W];
#pragma unroll
        for (int i = 0; i < TB; ++i) {
            float acc = 0.f;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k >= 4 - taps) acc = fmaf(w[k], v[i + k], acc);      // (a row out of reach may hold an infinity: no zero tap)
            put(t0 + i, v[i + 3] + acc);
        }
        return;
    }
    for (int t = t0; t < t0 + nt; ++t) {
        const int req = a.seq_rows[t];
        const int r = t - a.req_start[req];              // index inside this step's portion
        const int pos0 = a.req_pos0[req];
        const float* ring = a.state + (size_t)a.req_slot[req] * a.slot_stride + a.tail_off;      // [taps - 1][W]
        float s = a.x[(size_t)t * W + c];
        if (a.w) {
            float acc = 0.f;
            for (int i = 0; i < taps; ++i) {
                const int back = taps - 1 - i;
                float v;
                if (r - back >= 0) v = a.x[(size_t)(t - back) * W + c];
                else if (pos0 + r - back >= 0) v = ring[(size_t)((pos0 + r - back) % keep) * W + c];
                else v = 0.f;
                acc = fmaf(a.w[(size_t)c * taps + i], v, acc);
            }
            s += acc;
        }
        put(t, s);
    }
}
// The same for blocks of eight tokens, rows on 16 bytes and four taps: a thread takes four columns, so that a warp asks for 512 bytes of each of
// eleven rows at once (one column per thread: 14.0 us for 2313 tokens of 2048 columns; now 12.1 us, the bytes take 8.7).
__global__ void __launch_bounds__(128) canon_rows_kernel(CanonArgs a, int T) {
    pdl_wait();
    constexpr int TB = 8;
    const int t0 = blockIdx.x * TB, nt = min(TB, T - t0), W = a.W;
    const int c = (blockIdx.y * 128 + threadIdx.x) * 4;
    if (c >= W) return;
    __nv_bfloat16 *hi = (__nv_bfloat16*)a.hi, *lo = (__nv_bfloat16*)a.lo;
    auto put = [&](int t, float4 s) {
        store_f4(a.hn + (size_t)t * W + c, s);
        if (hi) {
            const uint32_t h0 = pack_bf16(s.x, s.y), h1 = pack_bf16(s.z, s.w);
            *reinterpret_cast<uint2*>(hi + (size_t)t * W + c) = make_uint2(h0, h1);
            *reinterpret_cast<uint2*>(lo + (size_t)t * W + c) =
                make_uint2(pack_bf16(s.x - bf16_lo(h0), s.y - bf16_hi(h0)), pack_bf16(s.z - bf16_lo(h1), s.w - bf16_hi(h1)));
        }
    };
    auto plus = [](float4 x, float4 y) { return make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w); };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 w[4];
    load_taps4(a.w + (size_t)c * 4, w);
    const int first = a.seq_rows[t0];
    if (nt == TB && a.seq_rows[t0 + TB - 1] == first && t0 - a.req_start[first] >= 3) {
        float4 v[TB + 3];
        const float* row = a.x + (size_t)(t0 - 3) * W + c;
#pragma unroll
        for (int i = 0; i < TB + 3; ++i) v[i] = load_f4(row + (size_t)i * (unsigned)W);
#pragma unroll
        for (int i = 0; i < TB; ++i) {
            float4 acc = zero;
#pragma unroll
            for (int k = 0; k < 4; ++k) acc = fma_f4(w[k], v[i + k], acc);
            put(t0 + i, plus(v[i + 3], acc));
        }
        return;
    }
    for (int t = t0; t < t0 + nt; ++t) {
        const int req = a.seq_rows[t], r = t - a.req_start[req], pos0 = a.req_pos0[req];
        const float* ring = a.state + (size_t)a.req_slot[req] * a.slot_stride + a.tail_off;      // [3][W]
        float4 acc = zero;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int back = 3 - i;
            const float4 v = r - back >= 0 ? load_f4(a.x + (size_t)(t - back) * W + c)
                                           : pos0 + r - back >= 0 ? load_f4(ring + (size_t)((pos0 + r - back) % 3) * W + c) : zero;
            acc = fma_f4(w[i], v, acc);
        }
        put(t, plus(load_f4(a.x + (size_t)t * W + c), acc));
    }
}
int launch_canon(const CanonArgs& a, int T, cudaStream_t stream) {
    FT_REQUIRE(a.x && a.hn && a.W >= 1, "input convolution: missing operands");
    FT_REQUIRE(!a.w || (a.taps >= 1 && a.taps <= kCanonMaxTaps && a.state), "input convolution: %d taps are beyond %d", a.taps,
               kCanonMaxTaps);
    const int cols = (a.W + 255) / 256;
    const uintptr_t all = (uintptr_t)a.x | (uintptr_t)a.w | (uintptr_t)a.hn | (uintptr_t)a.hi | (uintptr_t)a.lo | (uintptr_t)a.state | (uintptr_t)(a.slot_stride * 4) |
                          (uintptr_t)(a.tail_off * 4);
    if (T > 64 && a.w && a.taps == 4 && a.W % 4 == 0 && (all & 15) == 0) launch_after(canon_rows_kernel, dim3((T + 7) / 8, (a.W / 4 + 127) / 128), 128, 0, stream, a, T);
    else if (T > 64) launch_after(canon_kernel<8>, dim3((T + 7) / 8, cols), 256, 0, stream, a, T);
    else launch_after(canon_kernel<1>, dim3(T, cols), 256, 0, stream, a, T);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

// ------------------------------------------------------------------ post norm, the sum over depth, the next input
// One kernel per sublayer joint, one CTA per row t:
//   (1) the row the sublayer read goes into its ring when it is among the last taps - 1 of its sequence in this step;
//   (2) v = x[t] + rms(y[t]) * post_w;
//   (3) at a layer's end: hist[k][t] = v and the stream becomes sum_j depth_w[j] hist[j][t];
//   (4) otherwise, with cw: the NEXT sublayer's input hn[t] = v + sum_i cw[:, i] v[t - taps + 1 + i].  The earlier rows of
//       the step are formed again from their own x and y (a row's norm needs nothing but that row), rows before the step
//       come from the next sublayer's ring.  The new rows go to x_out, a buffer of its own, since the CTAs of the following
//       rows read the old x[t].
__device__ __forceinline__ float post_y(const PostNormArgs& a, size_t i, int c) {
    float y = a.y0[i] + (a.b0 ? a.b0[c] : 0.f);
    if (a.y1) y = a.s0 * y + a.s1 * (a.y1[i] + (a.b1 ? a.b1[c] : 0.f));
    else if (a.s0 != 1.f) y *= a.s0;
    return y;
}
__global__ void __launch_bounds__(256) postnorm_kernel(PostNormArgs a) {
    pdl_wait();
    __shared__ float red[33];
    extern __shared__ float sm[];
    const int t = blockIdx.x, W = a.W;
    float* row = sm;                                  // [W] y of the row at hand
    float* acc = sm + W;                              // [W] the convolution's sum (only with cw)
    int r = 0, pos0 = 0, n = 1;
    float* slot = nullptr;
    if (a.seq_rows) {
        const int req = a.seq_rows[t];
        r = t - a.req_start[req];
        n = a.req_start[req + 1] - a.req_start[req];
        pos0 = a.req_pos0[req];
        slot = a.state + (size_t)a.req_slot[req] * a.slot_stride;
    }
    const int keep = a.taps - 1;
    if (a.save_off >= 0 && keep > 0 && r >= n - keep) {
        float* ring = slot + a.save_off + (size_t)((pos0 + r) % keep) * W;
        for (int c = threadIdx.x; c < W; c += blockDim.x) ring[c] = a.x[(size_t)t * W + c];
    }
    const int first = a.cw ? keep : 0;                // how many earlier rows are formed again
    if (a.cw)
        for (int c = threadIdx.x; c < W; c += blockDim.x) acc[c] = 0.f;
    for (int b = first; b >= 0; --b) {
        const int rb = r - b;                         // uniform over the CTA
        const float* cwb = a.cw ? a.cw + (a.taps - 1 - b) : nullptr;
        if (rb < 0) {
            if (pos0 + rb < 0) continue;
            const float* ring = slot + a.read_off + (size_t)((pos0 + rb) % keep) * W;
            for (int c = threadIdx.x; c < W; c += blockDim.x) acc[c] = fmaf(cwb[(size_t)c * a.taps], ring[c], acc[c]);
            continue;
        }
        const size_t base = (size_t)(t - b) * W;
        float ss = 0.f;
        for (int c = threadIdx.x; c < W; c += blockDim.x) {
            const float y = post_y(a, base + c, c);
            row[c] = y;
            ss += y * y;
        }
        ss = block_sum(ss, red);
        const float rs = 1.f / sqrtf(ss / (float)W + a.eps);
        if (b > 0) {
            for (int c = threadIdx.x; c < W; c += blockDim.x)
                acc[c] = fmaf(cwb[(size_t)c * a.taps], a.x[base + c] + row[c] * rs * a.post_w[c], acc[c]);
            continue;
        }
        __nv_bfloat16 *hi = (__nv_bfloat16*)a.hi, *lo = (__nv_bfloat16*)a.lo;
        for (int c = threadIdx.x; c < W; c += blockDim.x) {
            float v = a.x[base + c] + row[c] * rs * a.post_w[c];
            if (a.hist) {
                a.hist[((size_t)a.k * a.t_stride + t) * W + c] = v;
                if (a.depth_w) {
                    v *= a.depth_w[a.k];
                    for (int j = a.k - 1; j >= 0; --j) v = fmaf(a.depth_w[j], a.hist[((size_t)j * a.t_stride + t) * W + c], v);
                }
            }
            a.x_out[base + c] = v;
            if (a.cw) {
                const float h = v + fmaf(cwb[(size_t)c * a.taps], v, acc[c]);
                a.hn[base + c] = h;
                if (hi) planes_put(hi, lo, base + c, h);
            }
        }
    }
}
// The same without the next input, rows of whole 16-byte groups: NV groups of four columns per thread stay in registers between the
// sum and the result (one column at a time through shared memory: 41 us for 2313 rows of 2048, the mean of a layer's two joints; now 17 us).
template <int NV>
__global__ void __launch_bounds__(256) postnorm_rows_kernel(PostNormArgs a) {
    pdl_wait();
    __shared__ float red[33];
    const int t = blockIdx.x, n4 = a.W >> 2;
    int r = 0, pos0 = 0, n = 1;
    float* slot = nullptr;
    if (a.seq_rows) {
        const int req = a.seq_rows[t];
        r = t - a.req_start[req];
        n = a.req_start[req + 1] - a.req_start[req];
        pos0 = a.req_pos0[req];
        slot = a.state + (size_t)a.req_slot[req] * a.slot_stride;
    }
    const int keep = a.taps - 1;
    float* ring = a.save_off >= 0 && keep > 0 && r >= n - keep ? slot + a.save_off + (size_t)((pos0 + r) % keep) * a.W : nullptr;
    auto at = [&](const float* p, size_t row, int c) { return reinterpret_cast<const float4*>(p + row * a.W)[c]; };
    float4 x[NV], y[NV];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = threadIdx.x + 256 * i;
        if (c >= n4) continue;
        x[i] = at(a.x, t, c);
        float4 v = at(a.y0, t, c);
        if (a.b0) { const float4 b = at(a.b0, 0, c); v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w; }
        if (a.y1) {
            float4 u = at(a.y1, t, c);
            if (a.b1) { const float4 b = at(a.b1, 0, c); u.x += b.x; u.y += b.y; u.z += b.z; u.w += b.w; }
            v.x = a.s0 * v.x + a.s1 * u.x; v.y = a.s0 * v.y + a.s1 * u.y; v.z = a.s0 * v.z + a.s1 * u.z; v.w = a.s0 * v.w + a.s1 * u.w;
        } else if (a.s0 != 1.f) {
            v.x *= a.s0; v.y *= a.s0; v.z *= a.s0; v.w *= a.s0;
        }
        y[i] = v;
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        if (ring) *reinterpret_cast<float4*>(ring + 4 * c) = x[i];
    }
    ss = block_sum(ss, red);
    const float rs = 1.f / sqrtf(ss / (float)a.W + a.eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = threadIdx.x + 256 * i;
        if (c >= n4) continue;
        const float4 w = at(a.post_w, 0, c);
        float4 v = make_float4(x[i].x + y[i].x * rs * w.x, x[i].y + y[i].y * rs * w.y, x[i].z + y[i].z * rs * w.z, x[i].w + y[i].w * rs * w.w);
        if (a.hist) {
            reinterpret_cast<float4*>(a.hist + ((size_t)a.k * a.t_stride + t) * a.W)[c] = v;
            if (a.depth_w) {
                const float d = a.depth_w[a.k];
                v.x *= d; v.y *= d; v.z *= d; v.w *= d;
                for (int j = a.k - 1; j >= 0; --j) {
                    const float4 h = at(a.hist, (size_t)j * a.t_stride + t, c);
                    const float e = a.depth_w[j];
                    v.x = fmaf(e, h.x, v.x); v.y = fmaf(e, h.y, v.y); v.z = fmaf(e, h.z, v.z); v.w = fmaf(e, h.w, v.w);
                }
            }
        }
        reinterpret_cast<float4*>(a.x_out + (size_t)t * a.W)[c] = v;
    }
}
int launch_postnorm(const PostNormArgs& a, int T, cudaStream_t stream) {
    FT_REQUIRE(a.x && a.x_out && a.y0 && a.post_w && a.W >= 1, "post norm: missing operands");
    FT_REQUIRE(!a.cw || (a.x_out != a.x && a.hn && !a.hist && a.taps >= 1 && a.taps <= kCanonMaxTaps && (a.taps == 1 || a.seq_rows)),
               "post norm: the fused input convolution needs a second stream buffer and the step's rows");
    FT_REQUIRE(a.save_off < 0 || a.taps <= 1 || a.seq_rows, "post norm: saving rows needs the step's rows");
    // rows on 16 bytes: every row of every operand then is (a slot's ring too)
    const uintptr_t all = (uintptr_t)a.x | (uintptr_t)a.x_out | (uintptr_t)a.y0 | (uintptr_t)a.y1 | (uintptr_t)a.b0 | (uintptr_t)a.b1 | (uintptr_t)a.post_w |
                          (uintptr_t)a.hist | (a.save_off >= 0 ? (uintptr_t)a.state | (uintptr_t)(a.slot_stride * 4) | (uintptr_t)(a.save_off * 4) : 0);
    if (!a.cw && a.W % 4 == 0 && a.W <= 8192 && (all & 15) == 0) {
        if (a.W <= 1024) launch_after(postnorm_rows_kernel<1>, T, 256, 0, stream, a);
        else if (a.W <= 2048) launch_after(postnorm_rows_kernel<2>, T, 256, 0, stream, a);
        else if (a.W <= 4096) launch_after(postnorm_rows_kernel<4>, T, 256, 0, stream, a);
        else launch_after(postnorm_rows_kernel<8>, T, 256, 0, stream, a);
    } else {
        launch_after(postnorm_kernel, T, 256, (size_t)a.W * 8, stream, a);
    }
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

// ------------------------------------------------------------------ row norms
__global__ void __launch_bounds__(256)
rms_rows_kernel(const float* __restrict__ x, const int* __restrict__ rows, const float* __restrict__ w, float gain,
                float* __restrict__ out, int W, float eps) {
    pdl_wait();
    __shared__ float red[33];
    const float* src = x + (size_t)(rows ? rows[blockIdx.x] : blockIdx.x) * W;
    float ss = 0.f;
    for (int c = threadIdx.x; c < W; c += blockDim.x) ss += src[c] * src[c];
    ss = block_sum(ss, red);
    const float r = 1.f / sqrtf(ss / (float)W + eps);
    for (int c = threadIdx.x; c < W; c += blockDim.x) out[(size_t)blockIdx.x * W + c] = src[c] * r * (w ? w[c] : gain);
}
int launch_rms_rows(const float* x, const int* rows, const float* w, float gain, float* out, int n, int W, float eps,
                    cudaStream_t stream) {
    launch_after(rms_rows_kernel, n, 256, 0, stream, x, rows, w, gain, out, W, eps);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

__global__ void __launch_bounds__(128)
rms_cols_kernel(const float* __restrict__ src, int lds, int src_off, const float* __restrict__ w, float* __restrict__ dst, int ldd,
                int dst_off, int n, float eps) {
    pdl_wait();
    __shared__ float red[33];
    const float* s = src + (size_t)blockIdx.x * lds + src_off;
    float* d = dst + (size_t)blockIdx.x * ldd + dst_off;
    float ss = 0.f;
    for (int c = threadIdx.x; c < n; c += blockDim.x) ss += s[c] * s[c];
    ss = block_sum(ss, red);
    const float r = 1.f / sqrtf(ss / (float)n + eps);
    for (int c = threadIdx.x; c < n; c += blockDim.x) d[c] = s[c] * r * w[c];
}
int launch_rms_cols(const float* src, int lds, int src_off, const float* w, float* dst, int ldd, int dst_off, int n, float eps,
                    int T, cudaStream_t stream) {
    launch_after(rms_cols_kernel, T, 128, 0, stream, src, lds, src_off, w, dst, ldd, dst_off, n, eps);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

// Latent window attention, per token: from the query projection q [heads][dim plain | rot] and the layer's projection
// (kv_rank latent columns, then rot columns of the shared key part at o_k) to the staging row the window-attention kernels read:
//   [heads x (rot query part | folded plain query, written by the caller's GEMM)] [rot key part | normed latent]
__global__ void __launch_bounds__(128)
latent_stage_kernel(const float* __restrict__ q, int heads, int dim, int rot, const float* __restrict__ proj, int ldp, int o_k,
                    int rank, const float* __restrict__ w, float eps, float* __restrict__ stage, int lds) {
    pdl_wait();
    __shared__ float red[33];
    const int t = blockIdx.x, kd = rot + rank;
    float* st = stage + (size_t)t * lds;
    const float* qr = q + (size_t)t * heads * (dim + rot);
    for (int i = threadIdx.x; i < heads * rot; i += blockDim.x) {
        const int h = i / rot, c = i - h * rot;
        st[(size_t)h * kd + c] = qr[(size_t)h * (dim + rot) + dim + c];
    }
    const float* pr = proj + (size_t)t * ldp + o_k;
    float* key = st + (size_t)heads * kd;
    for (int c = threadIdx.x; c < rot; c += blockDim.x) key[c] = pr[rank + c];
    float ss = 0.f;
    for (int c = threadIdx.x; c < rank; c += blockDim.x) ss += pr[c] * pr[c];
    ss = block_sum(ss, red);
    const float r = 1.f / sqrtf(ss / (float)rank + eps);
    for (int c = threadIdx.x; c < rank; c += blockDim.x) {
        const float v = pr[c] * r * w[c];
        key[rot + c] = v;
    }
}
int launch_latent_stage(const float* q, int heads, int dim, int rot, const float* proj, int ldp, int o_k, int rank, const float* w,
                        float eps, float* stage, int lds, int T, cudaStream_t stream) {
    launch_after(latent_stage_kernel, T, 128, 0, stream, q, heads, dim, rot, proj, ldp, o_k, rank, w, eps, stage, lds);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace ft

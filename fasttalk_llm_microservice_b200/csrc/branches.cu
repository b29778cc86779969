// Kernels of the branch mixers (ft_branch_desc).  Everything here is
// fp32: positions and angles, scores and softmax, norms, gates, decays and the recurrent state; the projections that feed
// these kernels come from the linear / tensor-core GEMMs of the layered family.
//
//   window attention     biases + rotary pairs, rotated keys and values into the paged cache; one CTA per (token, head),
//                        its warps take key blocks of the window in turn (one key per lane for the scores, one value column
//                        per lane for the sum), online softmax, merged through shared memory; prompt portions on a tiled
//                        kernel.  Options, each off by default: queries and keys divided by their root mean square, a bias
//                        by distance, first positions that stay visible beyond the window, a sink in the softmax denominator,
//                        values mixed with those an earlier layer kept for the step, values that are columns of the keys, a
//                        temperature that grows with the position, an element-wise gate on the result
//   scalar-decay rule    S <- a_t S + b_t k_t v_t^T, o_t = S^T q_t for a request's tokens in order; one CTA per (request,
//                        head, block of value columns), LPC lanes share a column and hold a run of key channels of its
//                        state in registers.  Decay attention, the gated matrix memory and the state-space mixer all run
//                        on it; they differ in how a, b, q, k, v are prepared and in the read-out that follows
//   preparation          SiLU in place; rotation of q and k in place; gate pre-activations and the running-maximum scan of the matrix memory; short causal
//                        convolution over a step's rows and the slot's tail, step sizes and decays of the state space
//   read-out             normaliser, skip, gates and group-wise RMS norm, one CTA per (token, norm group)
#include "common.cuh"
#include "ft_internal.h"

#include <algorithm>

namespace ft {

__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

__device__ __forceinline__ float cta_sum(float v, float* red) {      // red: >= 33 floats of shared memory
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

// ------------------------------------------------------------------ elementwise preparation
// x[t][c0 .. c0 + n) <- silu(x) in place, rows of stride ld; V columns (16 bytes or one) per thread
template <int V>
__global__ void __launch_bounds__(256) silu_cols_kernel(float* __restrict__ x, int ld, int c0, int n) {
    pdl_wait();
    const int c = (blockIdx.y * 256 + threadIdx.x) * V;
    if (c >= n) return;
    float* r = x + (size_t)blockIdx.x * ld + c0 + c;
    if (V == 4) {
        float4 v = *reinterpret_cast<float4*>(r);
        v = make_float4(silu_f(v.x), silu_f(v.y), silu_f(v.z), silu_f(v.w));
        *reinterpret_cast<float4*>(r) = v;
    } else {
        *r = silu_f(*r);
    }
}
int launch_silu_cols(float* x, int ld, int c0, int n, int T, cudaStream_t stream) {
    const bool v4 = ld % 4 == 0 && c0 % 4 == 0 && n % 4 == 0 && ((uintptr_t)x & 15) == 0;
    const int per = 256 * (v4 ? 4 : 1);
    const dim3 grid(T, (n + per - 1) / per);
    if (v4) launch_after(silu_cols_kernel<4>, grid, 256, 0, stream, x, ld, c0, n);
    else launch_after(silu_cols_kernel<1>, grid, 256, 0, stream, x, ld, c0, n);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}
__global__ void turn_qk_kernel(TurnArgs a) {
    pdl_wait();
    const int t = blockIdx.x, half = a.rot_dims >> 1, per = half + a.dim - a.rot_dims;      // pairs, then single coordinates of a head
    const float pos = (float)a.positions[t];
    for (int i = threadIdx.x; i < (a.heads + a.kv_heads) * per; i += blockDim.x) {
        const int hh = i / per, j = i % per;
        const bool isq = hh < a.heads;
        if (isq && j >= half) continue;                       // a query's other coordinates stay
        float* x = a.proj + (size_t)t * a.ldp + (isq ? a.o_q + hh * a.dim : a.o_k + (hh - a.heads) * a.dim);
        const float s = isq ? 1.f : a.k_scale;
        if (j >= half) { x[a.rot_dims + j - half] *= s; continue; }
        float sn, cs;
        sincosf(pos * a.rot_freq[j], &sn, &cs);
        float* p = x + (a.rot_half ? j : 2 * j);
        float* q = x + (a.rot_half ? j + half : 2 * j + 1);
        const float u = *p, v = *q;
        *p = (u * cs - v * sn) * s;
        *q = (v * cs + u * sn) * s;
    }
}
int launch_turn_qk(const TurnArgs& a, int T, cudaStream_t stream) {
    FT_REQUIRE(a.rot_dims >= 0 && a.rot_dims <= a.dim && (a.rot_dims & 1) == 0 && (a.rot_dims == 0 || a.rot_freq),
               "rotation: bad sizes (dim %d, rotated %d)", a.dim, a.rot_dims);
    launch_after(turn_qk_kernel, T, 256, 0, stream, a);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}
// ab[t][h] = (decay[h], 1)
__global__ void const_decay_kernel(const float* __restrict__ decay, float* __restrict__ ab, int heads, int n) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { ab[2 * (size_t)i] = decay[i % heads]; ab[2 * (size_t)i + 1] = 1.f; }
}
int launch_const_decay(const float* decay, float* ab, int heads, int T, cudaStream_t stream) {
    const int n = T * heads;
    launch_after(const_decay_kernel, (n + 255) / 256, 256, 0, stream, decay, ab, heads, n);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

// ------------------------------------------------------------------ window attention
// Token t: q = proj[o_q ..] + bias, rotated, -> q_out; k = proj[o_k ..] + bias: the rotated key and the value (the key before
// rotation, or proj[o_v ..]) -> the cache row of its position: [kv_heads * dim keys | kv_heads * vdim values].
// One coordinate of a query or key head after bias, norm factor, gain and rotation.  idx: its place in the projection's run of
// heads; c: its place inside the head; gi0: where the head's gains start in `gain` (the same for all heads, or per head).
// The cosines and sines of the position's pairs (times the magnitude) are formed once per CTA: trig[pair], trig[pairs + pair].
struct RotSpec { const float* trig; int dims, half_layout; };
__device__ __forceinline__ float rotated(const float* __restrict__ src, const float* __restrict__ bias, const float* __restrict__ gain,
                                         int gi0, int idx, int c, const RotSpec& r, float sc) {
    float me = (src[idx] + (bias ? bias[idx] : 0.f)) * sc;
    if (gain) me *= gain[gi0 + c];
    if (c >= r.dims) return me;
    const int half = r.dims >> 1;
    // partner and turning direction: (2i, 2i+1) pairs, or (i, i + dims / 2)
    const bool second = r.half_layout ? c >= half : (c & 1);
    const int oc = r.half_layout ? (second ? c - half : c + half) : (second ? c - 1 : c + 1);
    const int other = idx + (oc - c);
    float ot = (src[other] + (bias ? bias[other] : 0.f)) * sc;
    if (gain) ot *= gain[gi0 + oc];
    const int pair = r.half_layout ? (second ? c - half : c) : (c >> 1);
    const float cs = r.trig[pair], sn = r.trig[half + pair];
    return second ? me * cs + ot * sn : me * cs - ot * sn;
}
// CTA (token x, part y): the heads whose number is y modulo the parts — a step of few tokens is cut by heads so that more than a CTA
// per token runs (one root mean square over all heads, qk_norm 2, keeps to one part).
__global__ void __launch_bounds__(128) window_write_kernel(WindowArgs a) {
    pdl_wait();
    extern __shared__ float inv[];             // qk_norm: 1 / rms of every query head, then of every key head; then the pairs' trig
    const int t = blockIdx.x, part = blockIdx.y, parts = gridDim.y;
    const float* pr = a.proj + (size_t)t * a.ldp;
    const int p = a.positions[t];
    const float pos = (float)p;
    float* trig = inv + (a.qk_norm ? a.H + a.G : 0);
    for (int i = threadIdx.x; i < a.rot_dims >> 1; i += blockDim.x) {
        float sn, cs;
        sincosf(pos * a.rot_freq[i], &sn, &cs);
        trig[i] = cs * a.rot_mag;
        trig[(a.rot_dims >> 1) + i] = sn * a.rot_mag;
    }
    const int nq = a.H * a.dim, nk = a.G * a.dim, nv = a.G * a.vdim;
    const int nkh = a.no_kv ? 0 : a.G;            // key heads this layer forms itself
    if (a.qk_norm == 2) {
        // one root mean square over all heads of q, one over all heads of k
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        if (wid < 2 && (wid == 0 || nkh > 0)) {
            const float* src = pr + (wid == 0 ? a.o_q : a.o_k);
            const float* bias = wid == 0 ? a.q_bias : a.k_bias;
            const int n = wid == 0 ? nq : nk;
            float ss = 0.f;
            for (int d = lane; d < n; d += 32) {
                const float v = src[d] + (bias ? bias[d] : 0.f);
                ss = fmaf(v, v, ss);
            }
            ss = warp_sum(ss);
            const float r = 1.f / sqrtf(ss / (float)n + a.eps);
            for (int hh = lane; hh < (wid == 0 ? a.H : a.G); hh += 32) inv[(wid == 0 ? 0 : a.H) + hh] = r;
        }
        __syncthreads();
    } else if (a.qk_norm) {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
        for (int hh = wid; hh < a.H + nkh; hh += nw) {
            const bool isq = hh < a.H;
            if ((isq ? hh : hh - a.H) % parts != part) continue;
            const float* src = pr + (isq ? a.o_q + hh * a.dim : a.o_k + (hh - a.H) * a.dim);
            const float* bias = isq ? (a.q_bias ? a.q_bias + hh * a.dim : nullptr) : (a.k_bias ? a.k_bias + (hh - a.H) * a.dim : nullptr);
            float ss = 0.f;
            for (int d = lane; d < a.dim; d += 32) {
                const float v = src[d] + (bias ? bias[d] : 0.f);
                ss = fmaf(v, v, ss);
            }
            ss = warp_sum(ss);
            if (lane == 0) inv[hh] = 1.f / sqrtf(ss / (float)a.dim + a.eps);
        }
        __syncthreads();
    }
    __syncthreads();
    const RotSpec rs = {trig, a.rot_dims, a.rot_half};
    const float qt = a.temp_every > 0 ? fmaf(a.temp_coef, logf((float)((p + 1) / a.temp_every + 1)), 1.f) : 1.f;
    const bool wide = a.qk_norm == 2;             // gains per (head, coordinate) instead of per coordinate
    // element e of this part's heads: head part + parts * (e / size), coordinate e % size
    const int qh = (a.H - part + parts - 1) / parts, kh = (a.G - part + parts - 1) / parts;
    for (int e = threadIdx.x; e < qh * a.dim; e += blockDim.x) {
        const int c = e % a.dim, hh = part + parts * (e / a.dim), i = hh * a.dim + c;
        a.q_out[(size_t)t * nq + i] = qt * rotated(pr + a.o_q, a.q_bias, a.q_gain, wide ? i - c : 0, i, c, rs, a.qk_norm ? inv[hh] : 1.f);
    }
    if (a.no_kv) return;
    const int* pt = a.page_table + (size_t)a.seq_rows[t] * a.max_pages;
    const bool alias = a.v_in_key >= 0;                // the values are columns of the keys: the row holds the keys only
    float* row = a.cache + ((size_t)pt[p >> 6] * 64 + (p & 63)) * (size_t)(alias ? nk : nk + nv);
    for (int e = threadIdx.x; e < kh * a.dim; e += blockDim.x) {
        const int c = e % a.dim, hh = part + parts * (e / a.dim), i = hh * a.dim + c;
        row[i] = rotated(pr + a.o_k, a.k_bias, a.k_gain, wide ? i - c : 0, i, c, rs, a.qk_norm ? inv[a.H + hh] : 1.f);
    }
    const float lam = a.v_role == 2 ? a.v_mix[0] : 0.f;
    for (int e = threadIdx.x; e < (alias ? 0 : kh * a.vdim); e += blockDim.x) {
        const int i = (part + parts * (e / a.vdim)) * a.vdim + e % a.vdim;
        float v = a.o_v >= 0 ? pr[a.o_v + i] + (a.v_bias ? a.v_bias[i] : 0.f) : pr[a.o_k + i] + (a.k_bias ? a.k_bias[i] : 0.f);
        if (a.v_role == 1) a.v_first[(size_t)t * nv + i] = v;
        else if (a.v_role == 2) v = (1.f - lam) * v + lam * a.v_first[(size_t)t * nv + i];
        row[nk + i] = v;
    }
}
// The same for heads of 16 * 2^n channels (up to 128) whose rows lie on 16 bytes, without a norm over all heads: a group of dim / 4 lanes takes a head, four channels
// a lane, which stay in registers between the norm and the rotation (one channel per thread, two passes: 36 us for 2313 tokens of 16 + 4 + 4
// heads of 128; now 15.6 us, the bytes take 9).  The heads of a token are dealt out to the groups of `gridDim.y` CTAs.
__global__ void __launch_bounds__(128) window_write_rows_kernel(WindowArgs a, int lanes) {
    pdl_wait();
    extern __shared__ float trig[];
    const int t = blockIdx.x, p = a.positions[t], half = a.rot_dims >> 1;
    const float* pr = a.proj + (size_t)t * a.ldp;
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
        float sn, cs;
        sincosf((float)p * a.rot_freq[i], &sn, &cs);
        trig[i] = cs * a.rot_mag;
        trig[half + i] = sn * a.rot_mag;
    }
    const int nq = a.H * a.dim, nk = a.G * a.dim, nv = a.G * a.vdim;
    const bool alias = a.v_in_key >= 0;
    const int n_qk = a.H + (a.no_kv ? 0 : a.G), step = gridDim.y * 128 / lanes;
    float* row = nullptr;
    if (!a.no_kv) {
        const int page = a.page_table[(size_t)a.seq_rows[t] * a.max_pages + (p >> 6)];
        row = a.cache + ((size_t)page * 64 + (p & 63)) * (size_t)(alias ? nk : nk + nv);
    }
    const float qt = a.temp_every > 0 ? fmaf(a.temp_coef, logf((float)((p + 1) / a.temp_every + 1)), 1.f) : 1.f;
    auto plus = [](float4 x, const float* b) {
        const float4 y = load_f4(b);
        return make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
    };
    const int c = (threadIdx.x & (lanes - 1)) * 4, group = (blockIdx.y * 128 + threadIdx.x) / lanes;
    // rotation: four channels' own cosines, and sines with the sign of their partners'
    const bool turns = c < a.rot_dims, second = a.rot_half && c >= half;
    const int oc = second ? c - half : c + half;
    __syncthreads();
    float4 cs = make_float4(1.f, 1.f, 1.f, 1.f), sn = make_float4(0.f, 0.f, 0.f, 0.f);
    if (turns && a.rot_half) {
        const int i0 = second ? c - half : c;
        const float f = second ? 1.f : -1.f;
        cs = make_float4(trig[i0], trig[i0 + 1], trig[i0 + 2], trig[i0 + 3]);
        sn = make_float4(f * trig[half + i0], f * trig[half + i0 + 1], f * trig[half + i0 + 2], f * trig[half + i0 + 3]);
    } else if (turns) {
        const int i0 = c >> 1;
        cs = make_float4(trig[i0], trig[i0], trig[i0 + 1], trig[i0 + 1]);
        sn = make_float4(-trig[half + i0], trig[half + i0], -trig[half + i0 + 1], trig[half + i0 + 1]);
    }
    for (int u0 = group - (int)(threadIdx.x & 31) / lanes; u0 < n_qk; u0 += step) {      // the warp's first head: whole warps stay together for the sums
        const int u = u0 + (int)(threadIdx.x & 31) / lanes;
        const bool live = u < n_qk, isq = u < a.H;
        const int h = !live ? 0 : isq ? u : u - a.H;
        const float* src = pr + (isq || !live ? a.o_q : a.o_k) + h * a.dim;
        const float* bias = isq || !live ? a.q_bias : a.k_bias;
        const float* gain = isq || !live ? a.q_gain : a.k_gain;
        float4 x = load_f4(src + c), y = make_float4(0.f, 0.f, 0.f, 0.f);
        if (bias) x = plus(x, bias + h * a.dim + c);
        if (turns && a.rot_half) {
            y = load_f4(src + oc);
            if (bias) y = plus(y, bias + h * a.dim + oc);
        }
        float f = 1.f;
        if (a.qk_norm) {
            float ss = x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
            for (int o = lanes >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            f = 1.f / sqrtf(ss / (float)a.dim + a.eps);
        }
        x = make_float4(x.x * f, x.y * f, x.z * f, x.w * f);
        y = make_float4(y.x * f, y.y * f, y.z * f, y.w * f);
        if (gain) {
            const float4 g = load_f4(gain + c);
            x = make_float4(x.x * g.x, x.y * g.y, x.z * g.z, x.w * g.w);
            if (turns && a.rot_half) {
                const float4 o = load_f4(gain + oc);
                y = make_float4(y.x * o.x, y.y * o.y, y.z * o.z, y.w * o.w);
            }
        }
        if (turns) {
            if (!a.rot_half) y = make_float4(x.y, x.x, x.w, x.z);
            x = make_float4(x.x * cs.x + y.x * sn.x, x.y * cs.y + y.y * sn.y, x.z * cs.z + y.z * sn.z, x.w * cs.w + y.w * sn.w);
        }
        if (!live) continue;
        if (isq) store_f4(a.q_out + (size_t)t * nq + h * a.dim + c, make_float4(qt * x.x, qt * x.y, qt * x.z, qt * x.w));
        else store_f4(row + h * a.dim + c, x);
    }
    if (a.no_kv || alias) return;
    const float lam = a.v_role == 2 ? a.v_mix[0] : 0.f;
    for (int i = (blockIdx.y * 128 + threadIdx.x) * 4; i < nv; i += gridDim.y * 512) {
        float4 v = load_f4(pr + (a.o_v >= 0 ? a.o_v : a.o_k) + i);
        const float* bias = a.o_v >= 0 ? a.v_bias : a.k_bias;
        if (bias) v = plus(v, bias + i);
        if (a.v_role == 1) {
            store_f4(a.v_first + (size_t)t * nv + i, v);
        } else if (a.v_role == 2) {
            const float4 w = load_f4(a.v_first + (size_t)t * nv + i);
            v = make_float4((1.f - lam) * v.x + lam * w.x, (1.f - lam) * v.y + lam * w.y, (1.f - lam) * v.z + lam * w.z, (1.f - lam) * v.w + lam * w.w);
        }
        store_f4(row + nk + i, v);
    }
}

// 16-byte asynchronous copy global -> shared of which only the first src_bytes (0 or 16) are read, the rest filled with zeros
__device__ __forceinline__ void cp_async16_zfill(float* dst_smem, const float* src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst_smem)), "l"(src), "r"(src_bytes) : "memory");
}

constexpr int kWinWarps = 4;
template <int VPL, bool VEC>
__global__ void __launch_bounds__(kWinWarps * 32) window_attn_kernel(WindowArgs a) {
    pdl_wait();
    extern __shared__ float sh[];
    float* sq = sh;                                    // [dim]
    float* sm = sq + ((a.dim + 3) & ~3);               // [warps] running maxima
    float* sl = sm + kWinWarps;                        // [warps] running sums
    float* sacc = sl + kWinWarps;                      // [warps][vdim]
    const int h = blockIdx.y, t = blockIdx.x;      // tokens along x: a step may hold more rows than y allows
    const int g = h / (a.H / a.G);
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = a.positions[t];
    const int lo = a.window > 0 ? (a.chunked ? p - p % a.window : max(0, p - a.window + 1)) : 0;
    const int nf = min(a.keep_first, lo);              // kept first positions that lie before the window
    const int n = nf + p - lo + 1;                     // key idx < nf: position idx; otherwise position lo + idx - nf
    const int* pt = a.page_table + (size_t)a.seq_rows[t] * a.max_pages;
    const bool alias = a.v_in_key >= 0;
    const size_t rowsz = (size_t)a.G * (alias ? a.dim : a.dim + a.vdim);
    const size_t v_at = alias ? (size_t)g * a.dim + a.v_in_key : (size_t)a.G * a.dim + (size_t)g * a.vdim;
    for (int c = threadIdx.x; c < a.dim; c += blockDim.x) sq[c] = a.q_out[((size_t)t * a.H + h) * a.dim + c];
    __syncthreads();
    float m = -INFINITY, l = 0.f, acc[VPL];
#pragma unroll
    for (int i = 0; i < VPL; ++i) acc[i] = 0.f;
    for (int b0 = wid * 32; b0 < n; b0 += kWinWarps * 32) {
        const int idx = b0 + lane;
        const int j = idx < nf ? idx : lo + idx - nf;
        const bool valid = idx < n;
        const int jj = valid ? j : p;
        const long long base = ((long long)pt[jj >> 6] * 64 + (jj & 63)) * (long long)rowsz;
        const float* kr = a.cache + base + (size_t)g * a.dim;
        float s = 0.f;
        if (VEC) {
#pragma unroll 8
            for (int c = 0; c < a.dim; c += 4) {
                const float4 kv = *reinterpret_cast<const float4*>(kr + c);
                const float4 qv = *reinterpret_cast<const float4*>(sq + c);
                s = fmaf(qv.x, kv.x, s); s = fmaf(qv.y, kv.y, s); s = fmaf(qv.z, kv.z, s); s = fmaf(qv.w, kv.w, s);
            }
        } else {
            for (int c = 0; c < a.dim; ++c) s = fmaf(sq[c], kr[c], s);
        }
        s *= a.scale;
        if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
        if (a.rel) s += a.rel[(size_t)min(p - jj, a.rel_n - 1) * a.H + h];
        if (!valid) s = -INFINITY;
        const float m_new = fmaxf(m, warp_max(s));
        const float corr = expf(m - m_new);            // 0 on the first block (m = -inf)
        const float pj = valid ? expf(s - m_new) : 0.f;
        l = l * corr + warp_sum(pj);
#pragma unroll
        for (int i = 0; i < VPL; ++i) acc[i] *= corr;
        m = m_new;
        // all 32 keys of the block, four at a time so that their value loads are in flight together; a lane beyond the block's
        // end holds weight 0 and the (valid) row of position p
        for (int x0 = 0; x0 < 32; x0 += 4) {
            if (x0 >= n - b0) break;
            float px[4];
            const float* vr[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                px[u] = __shfl_sync(0xffffffffu, pj, x0 + u);
                const long long bx = __shfl_sync(0xffffffffu, base, x0 + u);
                vr[u] = a.cache + bx + v_at;
            }
            float vv[4][VPL];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int i = 0; i < VPL; ++i) {
                    const int c = lane + 32 * i;
                    vv[u][i] = c < a.vdim ? vr[u][c] : 0.f;
                }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int i = 0; i < VPL; ++i) acc[i] = fmaf(px[u], vv[u][i], acc[i]);
        }
    }
    if (lane == 0) { sm[wid] = m; sl[wid] = l; }
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
        const int c = lane + 32 * i;
        if (c < a.vdim) sacc[(size_t)wid * a.vdim + c] = acc[i];
    }
    __syncthreads();
    float mm = sm[0];
    for (int w = 1; w < kWinWarps; ++w) mm = fmaxf(mm, sm[w]);
    float den = 0.f;
    if (a.sink) {
        mm = fmaxf(mm, a.sink[h]);
        den = expf(a.sink[h] - mm);
    }
    for (int w = 0; w < kWinWarps; ++w) den += sl[w] * expf(sm[w] - mm);
    for (int c = threadIdx.x; c < a.vdim; c += blockDim.x) {
        float num = 0.f;
        for (int w = 0; w < kWinWarps; ++w) num += sacc[(size_t)w * a.vdim + c] * expf(sm[w] - mm);
        float r = num / den;
        if (a.gate) r *= sigmoid_f(a.gate[(size_t)t * a.ldg + h * a.vdim + c]);
        a.out[((size_t)t * a.H + h) * a.vdim + c] = r;
    }
}

// The same for heads of up to 128 channels, up to four query heads per key head: one CTA per (token, key head), so that a key and a value row is read once for the
// group and by neighbouring lanes.  A warp takes KEYS keys at a time, all of their rows copied to its part of shared memory at once, the next ones' while it
// works: scores by eight lanes a key, the softmax by a lane a key, the sums by four channels a lane.  Bound by the chain of a round of WARPS * KEYS keys: copies that
// set out one step ahead, sums and maxima over lanes (3.8 us for 128 keys with four query heads, 2.2 with one).  Eight warps of 16 keys are the shortest chain while
// every CTA runs at once; beyond that four of eight, of which four to eight times as many fit an SM.
constexpr int step_ctas(int grp, int warps) { return warps == 8 ? (grp == 1 ? 3 : grp == 2 ? 2 : 1) : (grp == 1 ? 8 : grp == 2 ? 5 : 3); }      // that an SM's registers hold
template <int GRP, int WARPS, int KEYS>
__global__ void __launch_bounds__(WARPS * 32, step_ctas(GRP, WARPS)) window_step_kernel(WindowArgs a) {
    pdl_wait();
    extern __shared__ __align__(16) float kv[];        // a warp's keys and values: [KEYS][dim], [KEYS][vdim]; at the end its sums [GRP][vdim]
    __shared__ __align__(16) float ps[WARPS][KEYS][GRP];       // scores, then probabilities of a warp's keys
    __shared__ float sm[WARPS][GRP], sl[WARPS][GRP];
    const int t = blockIdx.x, g = blockIdx.y, grp = a.H / a.G, h0 = g * grp;
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane & 7;
    const int p = a.positions[t];
    const int* pt = a.page_table + (size_t)a.seq_rows[t] * a.max_pages;
    const int lo = a.window > 0 ? (a.chunked ? p - p % a.window : max(0, p - a.window + 1)) : 0;
    const int nf = min(a.keep_first, lo);              // kept first positions that lie before the window
    const int n = nf + p - lo + 1;                     // key idx < nf: position idx; otherwise position lo + idx - nf
    const bool alias = a.v_in_key >= 0;
    const size_t rowsz = (size_t)a.G * (alias ? a.dim : a.dim + a.vdim);
    const float* k_at = a.cache + (size_t)g * a.dim;
    const float* v_at = a.cache + (alias ? (size_t)g * a.dim + a.v_in_key : (size_t)a.G * a.dim + (size_t)g * a.vdim);
    float* ks = kv + (size_t)wid * KEYS * (a.dim + a.vdim);
    float* vs = ks + KEYS * a.dim;
    constexpr int STEP = WARPS * KEYS;
    // the place of key b0 + lane % KEYS (behind the last one: of position p, whose weight is then 0)
    auto place = [&](int b0) {
        const int idx = b0 + (lane & (KEYS - 1)), j = idx < n ? (idx < nf ? idx : lo + idx - nf) : p;
        return pt[j >> 6] * 64 + (j & 63);
    };
    auto copy = [&](int row, const float* from, float* to, int width) {
        const uint32_t dst = smem_u32(to) + lane * 16;
#pragma unroll 4
        for (int key = 0; key < KEYS; ++key) {
            const int r = __shfl_sync(0xffffffffu, row, key);
            if (4 * lane < width)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + key * width * 4), "l"(from + (size_t)r * rowsz + 4 * lane) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int b0 = wid * KEYS;
    if (b0 < n) {
        const int row = place(b0);
        copy(row, k_at, ks, a.dim);
        copy(row, v_at, vs, a.vdim);
    }
    float4 q[GRP][4];
#pragma unroll
    for (int h = 0; h < GRP; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c = sub * 4 + 32 * i;
            q[h][i] = h < grp && c < a.dim ? load_f4(a.q_out + ((size_t)t * a.H + h0 + h) * a.dim + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    float m[GRP], l[GRP];
    float4 acc[GRP];
#pragma unroll
    for (int h = 0; h < GRP; ++h) {
        m[h] = -INFINITY;
        l[h] = 0.f;
        acc[h] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int c_out = lane * 4;
    for (; b0 < n; b0 += STEP) {
        const int idx = b0 + (lane & (KEYS - 1)), j = idx < nf ? idx : lo + idx - nf;      // every KEYS lanes hold the same keys
        const bool valid = idx < n, more = b0 + STEP < n;
        const int row = more ? place(b0 + STEP) : 0;
        asm volatile("cp.async.wait_group 1;" ::: "memory");     // the keys (the values are the group behind them)
        __syncwarp();
#pragma unroll
        for (int it = 0; it < KEYS / 4; ++it) {
            const int key = 4 * it + (lane >> 3);
            float s[GRP];
#pragma unroll
            for (int h = 0; h < GRP; ++h) s[h] = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int c = sub * 4 + 32 * i;
                if (c >= a.dim) continue;
                const float4 k = load_f4(ks + key * a.dim + c);
#pragma unroll
                for (int h = 0; h < GRP; ++h) s[h] = fmaf(q[h][i].x, k.x, fmaf(q[h][i].y, k.y, fmaf(q[h][i].z, k.z, fmaf(q[h][i].w, k.w, s[h]))));
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                for (int h = 0; h < GRP; ++h) s[h] += __shfl_xor_sync(0xffffffffu, s[h], o);
            if (sub == 0)
#pragma unroll
                for (int h = 0; h < GRP; ++h) ps[wid][key][h] = s[h];
        }
        __syncwarp();
        if (more) copy(row, k_at, ks, a.dim);
        float s[GRP], top[GRP], sum[GRP], corr[GRP];
#pragma unroll
        for (int h = 0; h < GRP; ++h) s[h] = ps[wid][lane & (KEYS - 1)][h] * a.scale;
        if (a.softcap > 0.f)
#pragma unroll
            for (int h = 0; h < GRP; ++h) s[h] = a.softcap * tanhf(s[h] / a.softcap);
#pragma unroll
        for (int h = 0; h < GRP; ++h) {
            if (a.rel && valid && h < grp) s[h] += a.rel[(size_t)min(p - j, a.rel_n - 1) * a.H + h0 + h];
            if (!valid || h >= grp) s[h] = -INFINITY;
            top[h] = s[h];
        }
#pragma unroll
        for (int o = KEYS / 2; o > 0; o >>= 1)
#pragma unroll
            for (int h = 0; h < GRP; ++h) top[h] = fmaxf(top[h], __shfl_xor_sync(0xffffffffu, top[h], o));
#pragma unroll
        for (int h = 0; h < GRP; ++h) {
            const float m_new = fmaxf(m[h], top[h]), base = m_new == -INFINITY ? 0.f : m_new;      // (scores may all be -inf so far: their weights are 0)
            corr[h] = h < grp ? expf(m[h] - base) : 0.f;         // 0 on the first block (m = -inf)
            sum[h] = valid && h < grp ? expf(s[h] - base) : 0.f;
            m[h] = m_new;
            ps[wid][lane & (KEYS - 1)][h] = sum[h];
        }
#pragma unroll
        for (int o = KEYS / 2; o > 0; o >>= 1)
#pragma unroll
            for (int h = 0; h < GRP; ++h) sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], o);
#pragma unroll
        for (int h = 0; h < GRP; ++h) {
            l[h] = l[h] * corr[h] + sum[h];
            acc[h] = make_float4(acc[h].x * corr[h], acc[h].y * corr[h], acc[h].z * corr[h], acc[h].w * corr[h]);
        }
        if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        if (c_out < a.vdim)
#pragma unroll
            for (int u = 0; u < KEYS; ++u) {
                const float4 v = load_f4(vs + u * a.vdim + c_out);
#pragma unroll
                for (int h = 0; h < GRP; ++h) {
                    const float w = ps[wid][u][h];
                    acc[h] = make_float4(fmaf(w, v.x, acc[h].x), fmaf(w, v.y, acc[h].y), fmaf(w, v.z, acc[h].z), fmaf(w, v.w, acc[h].w));
                }
            }
        __syncwarp();
        if (more) copy(row, v_at, vs, a.vdim);
    }
    if (lane == 0)
#pragma unroll
        for (int h = 0; h < GRP; ++h) {
            sm[wid][h] = m[h];
            sl[wid][h] = l[h];
        }
    if (c_out < a.vdim)
#pragma unroll
        for (int h = 0; h < GRP; ++h) store_f4(ks + h * a.vdim + c_out, acc[h]);        // (all copies have landed; four rows fit the warp's part)
    __syncthreads();
    for (int i = threadIdx.x; i < grp * a.vdim; i += WARPS * 32) {
        const int h = i / a.vdim, c = i % a.vdim;
        float mm = sm[0][h];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) mm = fmaxf(mm, sm[w][h]);
        float den = 0.f, num = 0.f;
        if (a.sink) {
            mm = fmaxf(mm, a.sink[h0 + h]);
            den = expf(a.sink[h0 + h] - mm);
        }
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float f = expf(sm[w][h] - mm);
            den += sl[w][h] * f;
            num += kv[(size_t)w * KEYS * (a.dim + a.vdim) + h * a.vdim + c] * f;
        }
        float r = num / den;
        if (a.gate) r *= sigmoid_f(a.gate[(size_t)t * a.ldg + (h0 + h) * a.vdim + c]);
        a.out[((size_t)t * a.H + h0 + h) * a.vdim + c] = r;
    }
}

// Prompt portions: one CTA per (key head, run of QT consecutive tokens of one request), QT = 64 / (query heads per key head),
// so that up to 64 query rows — the tokens of the run times the query heads of the group — share every key and value row
// that is brought into shared memory.  Keys are taken 32 at a time from the first one the run's first token sees to the
// run's last position: S = Q K^T (each thread 2 rows x 4 keys, keys interleaved by 8 so that the 16-byte reads of a warp fall
// into different banks), cap, per-row window mask, online softmax (a row's 8 threads are neighbouring lanes), P to shared
// memory, O = O * corr + P V (each warp 8 rows, each lane 4 value columns per 128).  All of it in fp32.
constexpr int WT_ROWS = 64, WT_KEYS = 32, WT_THREADS = 256;
template <int VK>
__global__ void __launch_bounds__(WT_THREADS) window_tile_kernel(WindowArgs a, WindowTiles tm, int QT, int subs) {
    pdl_wait();
    extern __shared__ __align__(16) float wsh[];
    const bool alias = a.v_in_key >= 0;       // the values are columns v_in_key.. of the key rows: no value tile of their own
    const int ldq = a.dim + 4, ldv = alias ? ldq : a.vdim, ldp = WT_KEYS + 1;
    const int kvf = WT_KEYS * ldq + (alias ? 0 : WT_KEYS * ldv);      // floats of one staged key (+ value) tile
    float* Qs = wsh;                          // [64][dim + 4]
    float* KV = Qs + WT_ROWS * ldq;           // two tiles of [32][dim + 4] keys (+ [32][vdim] values): one in use, one arriving
    float* Ps = KV + 2 * kvf;                 // [64][33]
    float* cr = Ps + WT_ROWS * ldp;           // [64] rescale of a row's sums in this tile; at the end the row's softmax sum
    const int tile = blockIdx.x / subs, sub = blockIdx.x % subs, g = blockIdx.y, tid = threadIdx.x;
    const int j = tm.tile_req[tile];
    const int q0 = tm.tile_q0[tile] + sub * QT;
    const int n_j = tm.req_q_start[j + 1] - tm.req_q_start[j];
    if (sub * QT >= 64 || q0 >= n_j) return;
    const int ntok = min(QT, min(n_j - q0, 64 - sub * QT));
    const int row_base = tm.req_q_start[j] + q0, p_first = tm.req_pos0[j] + q0;
    const int* pt = a.page_table + (size_t)tm.req_slot[j] * a.max_pages;
    const int grp = a.H / a.G, rows_used = ntok * grp;
    const size_t rowsz = (size_t)a.G * (alias ? a.dim : a.dim + a.vdim);
    const int d4n = a.dim >> 2, v4n = alias ? 0 : a.vdim >> 2;
    for (int i = tid; i < WT_ROWS * d4n; i += WT_THREADS) {
        const int r = i / d4n, d4 = i - r * d4n;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows_used)
            v = *reinterpret_cast<const float4*>(a.q_out + ((size_t)(row_base + r / grp) * a.H + g * grp + r % grp) * a.dim + 4 * d4);
        *reinterpret_cast<float4*>(Qs + r * ldq + 4 * d4) = v;
    }
    const int lo = a.window > 0 ? (a.chunked ? p_first - p_first % a.window : max(0, p_first - a.window + 1)) : 0, hi = p_first + ntok - 1;
    const int ry = tid >> 3, cx = tid & 7;            // scores: rows 2 ry, 2 ry + 1; keys cx, cx + 8, cx + 16, cx + 24 of the tile
    const int oy = tid >> 5, ox = tid & 31;           // sums: rows 8 oy .. 8 oy + 7; columns 4 ox .. 4 ox + 3 (+ 128)
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    int pr[2];
    bool rv[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) { rv[i] = 2 * ry + i < rows_used; pr[i] = p_first + (2 * ry + i) / grp; }
    f32x2 acc[8][VK][2];                              // value columns (4 ox, + 1) and (+ 2, + 3) of 8 rows, per 128 columns
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int k = 0; k < VK; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c) acc[r][k][c] = 0ull;
    // The key tiles of this CTA in order: first those of the kept first positions that lie before the window (keys below nf),
    // then those of the window up to the run's last position.  Tile it + 1 is copied asynchronously while tile it is used.
    const int nf = min(a.keep_first, lo);
    const int n0 = (nf + WT_KEYS - 1) / WT_KEYS, nt = n0 + (hi - lo) / WT_KEYS + 1;
    auto stage = [&](int it, float* buf) {
        const bool seg = it >= n0;
        const int k0 = seg ? lo + (it - n0) * WT_KEYS : it * WT_KEYS, kend = seg ? hi + 1 : nf;
        for (int i = tid; i < WT_KEYS * d4n; i += WT_THREADS) {
            const int c = i / d4n, d4 = i - c * d4n, key = k0 + c;
            const bool ok = key < kend;             // rows beyond the end are filled with zeros (a copy of no source bytes)
            const float* src = ok ? a.cache + ((size_t)pt[key >> 6] * 64 + (key & 63)) * rowsz + (size_t)g * a.dim + 4 * d4 : a.cache;
            cp_async16_zfill(buf + c * ldq + 4 * d4, src, ok ? 16 : 0);
        }
        for (int i = tid; i < WT_KEYS * v4n; i += WT_THREADS) {
            const int c = i / v4n, d4 = i - c * v4n, key = k0 + c;
            const bool ok = key < kend;
            const float* src = ok ? a.cache + ((size_t)pt[key >> 6] * 64 + (key & 63)) * rowsz + (size_t)a.G * a.dim + (size_t)g * a.vdim + 4 * d4
                                  : a.cache;
            cp_async16_zfill(buf + WT_KEYS * ldq + c * ldv + 4 * d4, src, ok ? 16 : 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(0, KV);
    for (int it = 0; it < nt; ++it) {
        const bool seg = it >= n0;
        const int k0 = seg ? lo + (it - n0) * WT_KEYS : it * WT_KEYS, kend = seg ? hi + 1 : nf;
        const float* Ks = KV + (it & 1) * kvf;
        const float* Vs = alias ? Ks + a.v_in_key : Ks + WT_KEYS * ldq;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();                               // tile `it` has landed; the last tile's sums are done with the other buffer and Ps
        if (it + 1 < nt) stage(it + 1, KV + ((it + 1) & 1) * kvf);
        // a score is summed in two halves, even and odd channels side by side in one packed register: the 16-byte reads of
        // queries and keys are already pairs of neighbouring channels, so every multiply-add is two-wide without a move
        float sc[2][4];
        f32x2 sc2[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) sc2[i][c] = 0ull;
        for (int d4 = 0; d4 < d4n; ++d4) {
            const ulonglong2 q0v = *reinterpret_cast<const ulonglong2*>(Qs + (2 * ry) * ldq + 4 * d4);
            const ulonglong2 q1v = *reinterpret_cast<const ulonglong2*>(Qs + (2 * ry + 1) * ldq + 4 * d4);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(Ks + (cx + 8 * c) * ldq + 4 * d4);
                sc2[0][c] = fma2(q0v.x, kv.x, sc2[0][c]); sc2[0][c] = fma2(q0v.y, kv.y, sc2[0][c]);
                sc2[1][c] = fma2(q1v.x, kv.x, sc2[1][c]); sc2[1][c] = fma2(q1v.y, kv.y, sc2[1][c]);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float ev, od;
                unpack2(sc2[i][c], ev, od);
                sc[i][c] = ev + od;
            }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float tmax = -INFINITY;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int key = k0 + cx + 8 * c;
                float v = sc[i][c] * a.scale;
                if (a.softcap > 0.f) v = a.softcap * tanhf(v / a.softcap);
                const bool vis = rv[i] && key < kend && key <= pr[i] &&
                                 (a.window <= 0 || (a.chunked ? key >= pr[i] - pr[i] % a.window : key > pr[i] - a.window) || key < a.keep_first);
                if (a.rel && vis) v += a.rel[(size_t)min(pr[i] - key, a.rel_n - 1) * a.H + g * grp + (2 * ry + i) % grp];
                sc[i][c] = vis ? v : -INFINITY;
                tmax = fmaxf(tmax, sc[i][c]);
            }
#pragma unroll
            for (int off = 1; off < 8; off <<= 1) tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, off));
            const float m_new = fmaxf(m[i], tmax);
            float corr = 1.f, psum = 0.f;
            if (m_new == -INFINITY) {
#pragma unroll
                for (int c = 0; c < 4; ++c) sc[i][c] = 0.f;
            } else {
                corr = expf(m[i] - m_new);
#pragma unroll
                for (int c = 0; c < 4; ++c) { sc[i][c] = expf(sc[i][c] - m_new); psum += sc[i][c]; }
            }
#pragma unroll
            for (int off = 1; off < 8; off <<= 1) psum += __shfl_xor_sync(0xffffffffu, psum, off);
            l[i] = l[i] * corr + psum;
            m[i] = m_new;
#pragma unroll
            for (int c = 0; c < 4; ++c) Ps[(2 * ry + i) * ldp + cx + 8 * c] = sc[i][c];
            if (cx == 0) cr[2 * ry + i] = corr;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float f = cr[8 * oy + r];
            const f32x2 f2 = pack2(f, f);
#pragma unroll
            for (int k = 0; k < VK; ++k)
#pragma unroll
                for (int c = 0; c < 2; ++c) acc[r][k][c] = mul2(acc[r][k][c], f2);
        }
        for (int c = 0; c < WT_KEYS; ++c) {
            ulonglong2 vv[VK];
#pragma unroll
            for (int k = 0; k < VK; ++k) {
                const int col = 4 * ox + 128 * k;
                vv[k] = col < a.vdim ? *reinterpret_cast<const ulonglong2*>(Vs + c * ldv + col) : make_ulonglong2(0ull, 0ull);
            }
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float pv = Ps[(8 * oy + r) * ldp + c];
                const f32x2 p2 = pack2(pv, pv);
#pragma unroll
                for (int k = 0; k < VK; ++k) {
                    acc[r][k][0] = fma2(p2, vv[k].x, acc[r][k][0]);
                    acc[r][k][1] = fma2(p2, vv[k].y, acc[r][k][1]);
                }
            }
        }
    }
    __syncthreads();
    if (cx == 0) {                                     // per row: what its sums are multiplied by at the end
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float f = 1.f / l[i];
            if (a.sink && rv[i]) {
                const float sk = a.sink[g * grp + (2 * ry + i) % grp], mf = fmaxf(m[i], sk), e = expf(m[i] - mf);
                f = e / (l[i] * e + expf(sk - mf));
            }
            cr[2 * ry + i] = f;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int row = 8 * oy + r;
        if (row >= rows_used) continue;
        const float inv = cr[row];
        float* orow = a.out + ((size_t)(row_base + row / grp) * a.H + g * grp + row % grp) * a.vdim;
        const float* gate = a.gate ? a.gate + (size_t)(row_base + row / grp) * a.ldg + (g * grp + row % grp) * a.vdim : nullptr;
#pragma unroll
        for (int k = 0; k < VK; ++k) {
            const int col = 4 * ox + 128 * k;
            if (col < a.vdim) {
                float o0, o1, o2, o3;
                unpack2(acc[r][k][0], o0, o1);
                unpack2(acc[r][k][1], o2, o3);
                if (gate) { o0 *= sigmoid_f(gate[col]); o1 *= sigmoid_f(gate[col + 1]); o2 *= sigmoid_f(gate[col + 2]); o3 *= sigmoid_f(gate[col + 3]); }
                *reinterpret_cast<float4*>(orow + col) = make_float4(o0 * inv, o1 * inv, o2 * inv, o3 * inv);
            }
        }
    }
}

// n_single: the step's first rows that are single tokens of running sequences (one CTA per (token, head) each); the prompt
// portions that follow them run on the tiled kernel when the head sizes allow it (multiples of 4, at most 64 query heads
// per key head), otherwise like the single tokens.
int launch_window_attention(const WindowArgs& a, int T, int n_single, const WindowTiles& tm, cudaStream_t stream) {
    FT_REQUIRE(a.H >= 1 && a.G >= 1 && a.H % a.G == 0 && a.dim >= 1 && a.vdim >= 1 && a.vdim <= 512,
               "window attention: bad head sizes (heads %d, kv heads %d, dim %d, vdim %d)", a.H, a.G, a.dim, a.vdim);
    FT_REQUIRE(a.rot_dims >= 0 && a.rot_dims <= a.dim && (a.rot_dims & 1) == 0,
               "window attention: rotary pairs need even sizes (dim %d, rotated %d)", a.dim, a.rot_dims);
    FT_REQUIRE(a.o_v >= 0 || a.v_in_key >= 0 || a.vdim == a.dim || a.no_kv, "window attention: keys used as values need vdim == dim");
    FT_REQUIRE(a.qk_norm >= 0 && a.qk_norm <= 2 && (!a.chunked || a.window > 0), "window attention: bad norm or chunk options");
    FT_REQUIRE(a.keep_first >= 0 && (!a.rel || a.rel_n >= 1) && (a.v_role == 0 || (a.v_first && a.o_v >= 0)) &&
                   (a.v_role != 2 || a.v_mix),
               "window attention: incomplete options");
    const int lanes = a.dim / 4;
    const uintptr_t all = (uintptr_t)a.proj | (uintptr_t)a.q_bias | (uintptr_t)a.k_bias | (uintptr_t)a.v_bias | (uintptr_t)a.q_gain | (uintptr_t)a.k_gain |
                          (uintptr_t)a.q_out | (uintptr_t)a.cache | (uintptr_t)a.v_first;
    const bool rows16 = a.qk_norm != 2 && a.dim % 16 == 0 && lanes <= 32 && (lanes & (lanes - 1)) == 0 && a.vdim % 4 == 0 && a.ldp % 4 == 0 &&
                        ((a.o_q | a.o_k) & 3) == 0 && (a.o_v < 0 || a.o_v % 4 == 0) && a.rot_dims % (a.rot_half ? 8 : 4) == 0 && (all & 15) == 0;
    // parts per token: as many as give about two CTAs per SM
    int parts = 1;
    while (a.qk_norm != 2 && parts < a.H && T * parts < 256 && parts < 16) parts *= 2;
    if (rows16) launch_after(window_write_rows_kernel, dim3(T, parts), 128, (size_t)a.rot_dims * 4, stream, a, lanes);
    else launch_after(window_write_kernel, dim3(T, parts), 128, (size_t)((a.qk_norm ? a.H + a.G : 0) + a.rot_dims) * 4, stream, a);
    FT_CHECK_CUDA(cudaGetLastError());
    const int grp = a.H / a.G;
    FT_REQUIRE(a.v_in_key < 0 || (a.v_in_key + a.vdim <= a.dim && a.v_role == 0), "window attention: values inside the keys exceed them");
    const size_t tsm = (size_t)((WT_ROWS + 2 * WT_KEYS) * (a.dim + 4) + (a.v_in_key >= 0 ? 0 : 2 * WT_KEYS * a.vdim) + WT_ROWS * (WT_KEYS + 1) + WT_ROWS) * 4;
    const bool tiled = tm.n_tiles > 0 && (a.dim & 3) == 0 && (a.vdim & 3) == 0 && grp <= WT_ROWS && a.vdim <= 256 && tsm <= 220 * 1024 &&
                       (a.v_in_key < 0 || (a.v_in_key & 3) == 0);
    int rows_each = T;                                 // rows of the one-CTA-per-(token, head) kernel
    if (tm.n_tiles > 0 && window_tc_ok(a)) {
        rows_each = n_single;
        if (int r = launch_window_tc(a, tm, stream)) return r;
    } else if (tiled) {
        rows_each = n_single;
        const int QT = WT_ROWS / grp, subs = (64 + QT - 1) / QT;
        dim3 grid(tm.n_tiles * subs, a.G);
        if (a.vdim <= 128) {
            FT_CHECK_CUDA(cudaFuncSetAttribute(window_tile_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsm));
            launch_after(window_tile_kernel<1>, grid, WT_THREADS, tsm, stream, a, tm, QT, subs);
        } else {
            FT_CHECK_CUDA(cudaFuncSetAttribute(window_tile_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsm));
            launch_after(window_tile_kernel<2>, grid, WT_THREADS, tsm, stream, a, tm, QT, subs);
        }
        FT_CHECK_CUDA(cudaGetLastError());
    }
    if (rows_each <= 0) return 0;
    T = rows_each;
    const size_t smem = (size_t)(((a.dim + 3) & ~3) + 2 * kWinWarps + kWinWarps * a.vdim) * 4;
    const bool vec = (a.dim & 3) == 0 && (a.vdim & 3) == 0;      // every key row then starts on 16 bytes
    const uintptr_t alias16 = (uintptr_t)a.cache | (uintptr_t)a.q_out | (a.v_in_key > 0 ? (uintptr_t)a.v_in_key * 4 : 0);
    // One query head per key head, or long heads and some tokens (us, before -> window_step_kernel, behind 10 / 150 / 600 keys in a window of 512: 8 key heads
    // of 64, one query head each, 4 tokens 4.5 / 9.2 / 16.9 -> 4.1 / 6.5 / 11.2; 4 key heads of 128 of four query heads, 16 tokens 6.5 / 15.2 / 31.9 -> 6.3 / 9.9 /
    // 18.3, one token 5.3 / 11.4 / 22.5 -> 5.9 / 9.5 / 17.6; one key head of 64 of four 5.0 / 9.5 / 17.1 -> 5.6 / 8.7 / 16.4, of 32 of three 4.3 / 8.4 / 14.9 -> 5.5 / 8.8 / 16.4).
    // Where more CTAs come than run at once, the small ones, but for heads shorter than 64 (before, eight warps, four, behind 10 / 40 / 150 / 600 keys: 16 key heads of 128, one
    // query head each, 32 tokens 6.8 / 8.9 / 28 / 68, 14 / 14 / 25 / 53, 4.4 / 6.7 / 13 / 46; of 64 64 tokens 5.9 / 8.6 / 23 / 63, 12 / 13 / 22 / 49, 5.0 / 8.2 / 19 / 51; 8 of 128 of
    // four query heads, 64 tokens 13 / 24 / 69 / 179, 23 / 23 / 39 / 77, 11 / 16 / 32 / 82; 32 of 32 of one, 32 tokens 5.1 / 7.0 / 14 / 44, 11 / 12 / 21 / 45, 4.9 / 8.1 / 18 / 50).
    if (vec && a.dim <= 128 && a.vdim <= 128 && (grp == 1 || (grp <= 4 && a.dim + a.vdim >= 192 && T >= 4)) && a.G <= 65535 && (alias16 & 15) == 0) {
        const int g = grp <= 2 ? grp : 4, row = (a.dim + a.vdim) * 4;
        const size_t rows = (size_t)8 * 16 * row;
        const int fit = (int)std::min<size_t>(step_ctas(g, 8), 227 * 1024 / (rows + 8 * 16 * g * 4 + 8 * g * 8 + 1024));      // the copies, the block's own, the system's
        const bool once = (long long)T * a.G <= (long long)device_sms() * fit;
        auto step = [&](auto kernel, int warps, size_t bytes) -> int {
            if (bytes > 40 * 1024) FT_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
            launch_after(kernel, dim3(T, a.G), warps * 32, bytes, stream, a);
            FT_CHECK_CUDA(cudaGetLastError());
            return 0;
        };
        if (once) return g == 1 ? step(window_step_kernel<1, 8, 16>, 8, rows) : g == 2 ? step(window_step_kernel<2, 8, 16>, 8, rows) : step(window_step_kernel<4, 8, 16>, 8, rows);
        const size_t few = (size_t)4 * 8 * row;
        if (row >= 512) return g == 1 ? step(window_step_kernel<1, 4, 8>, 4, few) : g == 2 ? step(window_step_kernel<2, 4, 8>, 4, few) : step(window_step_kernel<4, 4, 8>, 4, few);
    }
    dim3 grid(T, a.H);
    const int vpl = (a.vdim + 31) / 32;
#define FT_WIN(V)                                                                                   \
    do {                                                                                            \
        if (vec) launch_after(window_attn_kernel<V, true>, grid, kWinWarps * 32, smem, stream, a);            \
        else launch_after(window_attn_kernel<V, false>, grid, kWinWarps * 32, smem, stream, a);               \
    } while (0)
    if (vpl <= 1) FT_WIN(1);
    else if (vpl <= 2) FT_WIN(2);
    else if (vpl <= 4) FT_WIN(4);
    else if (vpl <= 8) FT_WIN(8);
    else FT_WIN(16);
#undef FT_WIN
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

// ------------------------------------------------------------------ scalar-decay rule
// Lanes s = 0..LPC-1 of a column hold channels s * DPT .. s * DPT + DPT - 1 of that column of S.  Chunks of RCH tokens are
// staged in two shared-memory buffers one chunk ahead with asynchronous copies (keys and queries padded with zeros
// to LPC * DPT channels, each lane's run 4 floats apart from the next so that the 16-byte reads of the LPC runs fall into
// different banks), then the tokens of a chunk are taken in order.  A full chunk runs without a branch, so that the
// compiler can start the shared-memory reads of later tokens under the arithmetic of earlier ones, and the arithmetic
// itself is packed: two neighbouring channels of a column share every multiply-add (fma.rn.f32x2, the two-wide fp32
// form of sm_100; each half rounds as the scalar instruction does).  The state is the only dependence from token to token; the
// read-out o_t = S^T q_t (partial sums over a lane's run, then a shuffle tree over the LPC lanes) overlaps the next update.
constexpr int RCH = 16, RTHREADS = 128;
// stages of the ring for a padded row of DP floats: as deep as ~100-160 KB of shared memory allow
__host__ __device__ constexpr int rule_stages(int dp) { return 2; }
template <int N> __device__ __forceinline__ void cp_async_wait_pending() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_f32(float* dst_smem, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst_smem)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_f32x4(float* dst_smem, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst_smem)), "l"(src) : "memory");
}
// VEC: keys and queries are copied 16 bytes at a time (dim a multiple of 4, rows and bases on 16-byte boundaries).
// CPT: state columns per thread.  A thread reads its run of key and query channels once per token and uses it for all of
// its CPT columns — the shared-memory reads, not the arithmetic, bound the kernel with one column per thread (every one of
// a column's 128 / LPC sibling columns in the CTA reads the same runs again).  The CPT partial read-outs are summed over the
// LPC lanes by halving: in each of the first log2(CPT) steps a lane hands half of its columns to its partner and keeps the
// other half, afterwards every lane holds one column and the tree goes on as usual.
template <int LPC, int DPT, int CPT, bool VEC>
__global__ void __launch_bounds__(RTHREADS) decay_rule_kernel(RecurArgs a) {
    pdl_wait();
    constexpr int VB = RTHREADS / LPC * CPT, RUN = DPT + 4, DP = LPC * RUN;
    constexpr int BUF = 2 * RCH * DP + RCH * VB + RCH * 2;      // floats of one staged chunk: keys | queries | values | (a, b)
    constexpr int NST = rule_stages(DP);
    extern __shared__ __align__(16) float rs[];
    const int r = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * VB;
    const int s = threadIdx.x % LPC, jl = threadIdx.x / LPC, j = j0 + jl * CPT;      // the thread's first column
    const int t0 = a.req_start[r], t1 = a.req_start[r + 1];
    if (t1 <= t0) return;
    const int gh = h / (a.heads / a.qk_heads);
    float* S = a.state + (size_t)a.req_slot[r] * a.slot_stride + a.s_off + (size_t)h * a.dim * a.vd;
    if (LPC * DPT != a.dim || j0 + VB > a.vd)                                  // the padding stays zero from here on
        for (int i = threadIdx.x; i < NST * BUF; i += RTHREADS) rs[i] = 0.f;
    f32x2 st[CPT][DPT / 2];                  // per column: channels (2 i, 2 i + 1) of the lane's run
    const bool old = a.req_pos0[r] > 0;
    // four columns of a row are 16 bytes of the state when vd is a multiple of 4 (slots and heads then start on 16 bytes)
    const bool wide = CPT == 4 && (a.vd & 3) == 0 && (((uintptr_t)S) & 15) == 0;
    if (wide) {
#pragma unroll
        for (int i = 0; i < DPT; i += 2) {
            const int d = s * DPT + i;
            float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
            if (old && j < a.vd && d < a.dim) lo = *reinterpret_cast<const float4*>(S + (size_t)d * a.vd + j);
            if (old && j < a.vd && d + 1 < a.dim) hi = *reinterpret_cast<const float4*>(S + (size_t)(d + 1) * a.vd + j);
            const float l4[4] = {lo.x, lo.y, lo.z, lo.w}, h4[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
            for (int c = 0; c < CPT; ++c) st[c][i / 2] = pack2(l4[c], h4[c]);
        }
    } else {
#pragma unroll
        for (int c = 0; c < CPT; ++c)
#pragma unroll
            for (int i = 0; i < DPT; i += 2) {
                const int d = s * DPT + i;
                const bool in = old && j + c < a.vd;
                st[c][i / 2] = pack2(in && d < a.dim ? S[(size_t)d * a.vd + j + c] : 0.f, in && d + 1 < a.dim ? S[(size_t)(d + 1) * a.vd + j + c] : 0.f);
            }
    }
    __syncthreads();
    auto stage = [&](int buf, int c0) {          // always commits a group, an empty one past the end: the count stays uniform
        if (c0 >= t1) { asm volatile("cp.async.commit_group;" ::: "memory"); return; }
        float* sk = rs + buf * BUF;
        float* sq = sk + RCH * DP;
        float* sv = sq + RCH * DP;
        float* sab = sv + RCH * VB;
        const int nt = min(RCH, t1 - c0);
        if (VEC) {                                   // a warp per token row, a lane per four channels
            for (int tt = threadIdx.x >> 5; tt < nt; tt += RTHREADS / 32) {
                const float* kr = a.k + (size_t)(c0 + tt) * a.ldk + (size_t)gh * a.dim;
                const float* qr = a.q + (size_t)(c0 + tt) * a.ldq + (size_t)gh * a.dim;
                for (int d = (threadIdx.x & 31) * 4; d < a.dim; d += 128) {
                    const int at = tt * DP + (d / DPT) * RUN + (d % DPT);
                    cp_async_f32x4(sk + at, kr + d);
                    cp_async_f32x4(sq + at, qr + d);
                }
            }
        } else {
            for (int i = threadIdx.x; i < nt * a.dim; i += RTHREADS) {
                const int tt = i / a.dim, d = i - tt * a.dim;
                const int at = tt * DP + (d / DPT) * RUN + (d % DPT);
                cp_async_f32(sk + at, a.k + (size_t)(c0 + tt) * a.ldk + (size_t)gh * a.dim + d);
                cp_async_f32(sq + at, a.q + (size_t)(c0 + tt) * a.ldq + (size_t)gh * a.dim + d);
            }
        }
        for (int i = threadIdx.x; i < nt * VB; i += RTHREADS) {
            const int tt = i / VB, c = i % VB;
            if (j0 + c < a.vd) cp_async_f32(sv + i, a.v + (size_t)(c0 + tt) * a.ldv + (size_t)h * a.vd + j0 + c);
        }
        for (int i = threadIdx.x; i < nt * 2; i += RTHREADS)
            cp_async_f32(sab + i, a.ab + ((size_t)(c0 + i / 2) * a.heads + h) * 2 + (i & 1));
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < NST - 1; ++i) stage(i, t0 + i * RCH);
    int buf = 0;
    for (int c0 = t0; c0 < t1; c0 += RCH, buf = buf + 1 == NST ? 0 : buf + 1) {
        const int nt = min(RCH, t1 - c0);
        stage(buf == 0 ? NST - 1 : buf - 1, c0 + (NST - 1) * RCH);      // into the buffer the last iteration has finished with
        cp_async_wait_pending<NST - 1>();
        __syncthreads();
        const float* sk = rs + buf * BUF;
        const float* sq = sk + RCH * DP;
        const float* sv = sq + RCH * DP;
        const float* sab = sv + RCH * VB;
        // update: the token's state update and each column's partial read-out over the lane's run
        auto update = [&](int tt, float* o) {
            const float da = sab[2 * tt], db = sab[2 * tt + 1];
            const f32x2 da2 = pack2(da, da);
            f32x2 kk[DPT / 2], qq[DPT / 2];
            const ulonglong2* kp = reinterpret_cast<const ulonglong2*>(sk + tt * DP + s * RUN);
            const ulonglong2* qp = reinterpret_cast<const ulonglong2*>(sq + tt * DP + s * RUN);
#pragma unroll
            for (int i = 0; i < DPT / 4; ++i) {
                const ulonglong2 kv = kp[i], qv = qp[i];
                kk[2 * i] = kv.x; kk[2 * i + 1] = kv.y;
                qq[2 * i] = qv.x; qq[2 * i + 1] = qv.y;
            }
#pragma unroll
            for (int c = 0; c < CPT; ++c) {
                const float bv = db * sv[tt * VB + jl * CPT + c];
                const f32x2 bv2 = pack2(bv, bv);
                f32x2 o0 = 0ull, o1 = 0ull;
#pragma unroll
                for (int i = 0; i < DPT / 2; i += 2) {
                    st[c][i] = fma2(da2, st[c][i], mul2(bv2, kk[i]));
                    st[c][i + 1] = fma2(da2, st[c][i + 1], mul2(bv2, kk[i + 1]));
                    o0 = fma2(st[c][i], qq[i], o0);
                    o1 = fma2(st[c][i + 1], qq[i + 1], o1);
                }
                float p0, p1, p2, p3;
                unpack2(o0, p0, p1);
                unpack2(o1, p2, p3);
                o[c] = (p0 + p2) + (p1 + p3);
            }
        };
        // finish: sum over the LPC lanes; the column a lane ends up with is made of the lane bits used in the halving steps.
        // Taken for four tokens at a time, so that the shuffle chains of the four overlap instead of stalling the warp.
        auto finish = [&](int tt, const float* o) {
            int col = 0;
            float v = o[0];
            if (CPT == 4) {
                const bool up = (s & (LPC / 2)) != 0, up2 = (s & (LPC / 4)) != 0;
                const float g0 = __shfl_xor_sync(0xffffffffu, up ? o[0] : o[2], LPC / 2);
                const float g1 = __shfl_xor_sync(0xffffffffu, up ? o[1] : o[3], LPC / 2);
                const float k0 = (up ? o[2] : o[0]) + g0, k1 = (up ? o[3] : o[1]) + g1;
                const float g2 = __shfl_xor_sync(0xffffffffu, up2 ? k0 : k1, LPC / 4);
                v = (up2 ? k1 : k0) + g2;
                col = (up ? 2 : 0) + (up2 ? 1 : 0);
#pragma unroll
                for (int off = LPC / 8; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            } else if (CPT == 2) {
                const bool up = (s & (LPC / 2)) != 0;
                const float g0 = __shfl_xor_sync(0xffffffffu, up ? o[0] : o[1], LPC / 2);
                v = (up ? o[1] : o[0]) + g0;
                col = up ? 1 : 0;
#pragma unroll
                for (int off = LPC / 4; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            } else {
#pragma unroll
                for (int off = LPC / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            }
            if ((s & (LPC / CPT - 1)) == 0 && j + col < a.vd) a.o[(size_t)(c0 + tt) * a.ldo + (size_t)h * a.vd + j + col] = v;
        };
        if (nt == RCH) {
#pragma unroll 1
            for (int t4 = 0; t4 < RCH; t4 += 4) {
                float o[4][CPT];
#pragma unroll
                for (int x = 0; x < 4; ++x) update(t4 + x, o[x]);
#pragma unroll
                for (int x = 0; x < 4; ++x) finish(t4 + x, o[x]);
            }
        } else {
            for (int tt = 0; tt < nt; ++tt) {
                float o[CPT];
                update(tt, o);
                finish(tt, o);
            }
        }
        __syncthreads();
    }
    if (wide) {
#pragma unroll
        for (int i = 0; i < DPT; i += 2) {
            const int d = s * DPT + i;
            float l4[4], h4[4];
#pragma unroll
            for (int c = 0; c < CPT; ++c) unpack2(st[c][i / 2], l4[c], h4[c]);
            if (j < a.vd && d < a.dim) *reinterpret_cast<float4*>(S + (size_t)d * a.vd + j) = make_float4(l4[0], l4[1], l4[2], l4[3]);
            if (j < a.vd && d + 1 < a.dim) *reinterpret_cast<float4*>(S + (size_t)(d + 1) * a.vd + j) = make_float4(h4[0], h4[1], h4[2], h4[3]);
        }
        return;
    }
#pragma unroll
    for (int c = 0; c < CPT; ++c)
#pragma unroll
        for (int i = 0; i < DPT; i += 2) {
            const int d = s * DPT + i;
            float lo, hi;
            unpack2(st[c][i / 2], lo, hi);
            if (j + c < a.vd && d < a.dim) S[(size_t)d * a.vd + j + c] = lo;
            if (j + c < a.vd && d + 1 < a.dim) S[(size_t)(d + 1) * a.vd + j + c] = hi;
        }
}

// A step of single tokens: one pass over the state, which bounds it.  CTA (request, head, TX units of V columns): the threads of a row
// group read neighbouring units, eight rows on their way per thread, and the row groups' shares of the read-out meet in shared
// memory.  (More tokens than one are taken one after the other, each with a pass of its own.)  The kernel above, which stages chunks of
// 16 tokens for lanes that hold the state, took 17 us for 16 tokens of 16 heads of 128 x 128 and 25 us for 64 heads of 128 x 64; with this
// one a decode step of three such layers takes 40 us less.
template <int V>
__global__ void __launch_bounds__(256) decay_step_kernel(RecurArgs a, int TX) {
    pdl_wait();
    extern __shared__ __align__(16) float sh[];
    float* part = sh;                                 // [256][V]
    float *sk = sh + 256 * V, *sq = sk + a.dim;
    const int r = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const int t0 = a.req_start[r], t1 = a.req_start[r + 1];
    const int tx = tid % TX, rg = tid / TX, RG = 256 / TX, c = (blockIdx.z * TX + tx) * V;
    const bool live = c < a.vd;
    const int gh = h / (a.heads / a.qk_heads);
    float* S = a.state + (size_t)a.req_slot[r] * a.slot_stride + a.s_off + (size_t)h * a.dim * a.vd + c;
    bool old = a.req_pos0[r] > 0;
    for (int t = t0; t < t1; ++t, old = true) {
        for (int d = tid; d < a.dim; d += 256) {
            sk[d] = a.k[(size_t)t * a.ldk + (size_t)gh * a.dim + d];
            sq[d] = a.q[(size_t)t * a.ldq + (size_t)gh * a.dim + d];
        }
        const float da = a.ab[((size_t)t * a.heads + h) * 2], db = a.ab[((size_t)t * a.heads + h) * 2 + 1];
        float v[V], o[V];
#pragma unroll
        for (int i = 0; i < V; ++i) {
            v[i] = live ? db * a.v[(size_t)t * a.ldv + (size_t)h * a.vd + c + i] : 0.f;
            o[i] = 0.f;
        }
        __syncthreads();
        if (live)
            for (int d0 = rg; d0 < a.dim; d0 += 8 * RG) {
                float x[8][V];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int d = d0 + i * RG;
                    if (V == 4) {
                        const float4 f = old && d < a.dim ? *reinterpret_cast<const float4*>(S + (size_t)d * a.vd) : make_float4(0.f, 0.f, 0.f, 0.f);
                        x[i][0] = f.x; x[i][1 % V] = f.y; x[i][2 % V] = f.z; x[i][3 % V] = f.w;
                    } else {
                        x[i][0] = old && d < a.dim ? S[(size_t)d * a.vd] : 0.f;
                    }
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int d = d0 + i * RG;
                    if (d >= a.dim) break;
                    const float kk = sk[d], qq = sq[d];
#pragma unroll
                    for (int e = 0; e < V; ++e) {
                        x[i][e] = fmaf(da, x[i][e], v[e] * kk);
                        o[e] = fmaf(x[i][e], qq, o[e]);
                    }
                    if (V == 4) *reinterpret_cast<float4*>(S + (size_t)d * a.vd) = make_float4(x[i][0], x[i][1 % V], x[i][2 % V], x[i][3 % V]);
                    else S[(size_t)d * a.vd] = x[i][0];
                }
            }
#pragma unroll
        for (int e = 0; e < V; ++e) part[tid * V + e] = o[e];
        __syncthreads();
        for (int i = tid; i < TX * V; i += 256) {
            const int col = blockIdx.z * TX * V + i;
            float sum = 0.f;
            for (int g = 0; g < RG; ++g) sum += part[g * TX * V + i];
            if (col < a.vd) a.o[(size_t)t * a.ldo + (size_t)h * a.vd + col] = sum;
        }
        __syncthreads();
    }
}
// Units per CTA: 32 of a row's where there are so many.  A thread then has dim / 8 rows: with few channels and a full grid more units, so
// that it has eight (64 requests of 16 heads of 32 x 1024: 64.9 us with 32 units, 50.3 with 64), and while fewer CTAs than half of the
// SMs would run fewer units, until it has no more than the eight rows that are on their way together (one request of two heads of 256 x 256:
// 5.8 us with 32 units, 3.6 with eight).
struct StepPlan { bool wide; int TX; long long ctas; };
static StepPlan decay_step_plan(const RecurArgs& a, int n_req) {
    StepPlan p;
    p.wide = a.vd % 4 == 0 && a.slot_stride % 4 == 0 && a.s_off % 4 == 0 && ((uintptr_t)a.state & 15) == 0;
    const int units = p.wide ? a.vd / 4 : a.vd, sms = device_sms();
    auto ctas = [&](int tx) { return (long long)n_req * a.heads * ((units + tx - 1) / tx); };
    p.TX = 4;
    while (p.TX < 32 && p.TX < units) p.TX *= 2;
    while (p.TX < 256 && p.TX < units && a.dim * p.TX < 8 * 256 && ctas(2 * p.TX) >= sms) p.TX *= 2;
    while (p.TX > 4 && a.dim * p.TX > 8 * 256 && ctas(p.TX) < sms / 2) p.TX /= 2;
    p.ctas = ctas(p.TX);
    return p;
}
static int launch_decay_step(const RecurArgs& a, int n_req, const StepPlan& p, cudaStream_t stream) {
    const bool wide = p.wide;
    const int TX = p.TX;
    const dim3 grid(n_req, a.heads, ((wide ? a.vd / 4 : a.vd) + TX - 1) / TX);
    const size_t smem = (size_t)(256 * (wide ? 4 : 1) + 2 * a.dim) * 4;
    if (wide) launch_after(decay_step_kernel<4>, grid, 256, smem, stream, a, TX);
    else launch_after(decay_step_kernel<1>, grid, 256, smem, stream, a, TX);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

template <int LPC, int DPT, int CPT>
static int launch_decay_rule_t(const RecurArgs& a, int n_req, cudaStream_t stream) {
    constexpr int VB = RTHREADS / LPC * CPT, DP = LPC * (DPT + 4);
    const size_t smem = (size_t)rule_stages(DP) * (2 * RCH * DP + RCH * VB + RCH * 2) * 4;
    const bool vec = (a.dim & 3) == 0 && (a.ldk & 3) == 0 && (a.ldq & 3) == 0 && ((uintptr_t)a.k & 15) == 0 && ((uintptr_t)a.q & 15) == 0;
    if (smem > 48 * 1024) {
        FT_CHECK_CUDA(cudaFuncSetAttribute(decay_rule_kernel<LPC, DPT, CPT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        FT_CHECK_CUDA(cudaFuncSetAttribute(decay_rule_kernel<LPC, DPT, CPT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    }
    dim3 grid((a.vd + VB - 1) / VB, a.heads, n_req);
    if (vec) launch_after(decay_rule_kernel<LPC, DPT, CPT, true>, grid, RTHREADS, smem, stream, a);
    else launch_after(decay_rule_kernel<LPC, DPT, CPT, false>, grid, RTHREADS, smem, stream, a);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

// Lanes per column (LPC), channels per lane (DPT <= 16, 32 only beyond 512 channels) and columns per thread (CPT): the
// fewest lanes whose runs cover dim and four columns per thread — the widest column blocks, the best-coalesced state
// traffic and the fewest shared-memory reads per multiply-add; then, while fewer than 96 CTAs would run (one long prompt
// with few heads): two columns per thread, more lanes with shorter runs, at last one column (measured order).  The split
// changes the order of a sum, nothing else.  a.lanes fixes LPC.  Steps of single tokens (no more rows than requests) take the
// step kernel, except where many small states make a full grid; portions of many tokens go to the tensor cores (decay_tc.cu).
int launch_decay_rule(const RecurArgs& a, int n_req, int T, cudaStream_t stream) {
    FT_REQUIRE(a.heads >= 1 && a.qk_heads >= 1 && a.heads % a.qk_heads == 0 && a.dim >= 1 && a.dim <= 1024 && a.vd >= 1,
               "decay rule: bad sizes (heads %d, key heads %d, dim %d, values %d)", a.heads, a.qk_heads, a.dim, a.vd);
    if (n_req <= 0) return 0;
    if (a.lanes == 0 && T > 0 && T <= n_req) {
        // Not where a thread would have a row or two and the CTAs queue up: states so small go faster through the kernel by lanes
        // (64 requests of 16 heads of 16 x 64: 7.0 us, by lanes 4.8; of 64 heads of 32 x 64: 21.5 and 19.8, but of 16 heads 8.5 and 10.4).
        const StepPlan p = decay_step_plan(a, n_req);
        const int rows = a.dim * p.TX / 256;
        if (rows >= 4 || p.ctas <= (rows < 2 ? 2 : 16) * device_sms()) return launch_decay_step(a, n_req, p, stream);
    }
    if (a.lanes == 0 && decay_tc_ahead(a, n_req, T)) return launch_decay_tc(a, n_req, stream);
    int lpc = 4, dpt = 4;
    while (dpt < 16 && lpc * dpt < a.dim) dpt *= 2;
    while (lpc < 32 && lpc * dpt < a.dim) lpc *= 2;
    if (lpc * dpt < a.dim) dpt = 32;
    int cpt = dpt == 32 ? 2 : 4;
    auto ctas = [&](int l, int c) { return (long long)n_req * a.heads * ((a.vd + RTHREADS / l * c - 1) / (RTHREADS / l * c)); };
    if (a.lanes > 0) {
        FT_REQUIRE((a.lanes == 4 || a.lanes == 8 || a.lanes == 16 || a.lanes == 32) && a.lanes >= lpc,
                   "decay rule: %d lanes per column do not hold %d channels", a.lanes, a.dim);
        while (lpc < a.lanes && dpt > 4) { lpc *= 2; dpt /= 2; }
        cpt = dpt == 32 ? 2 : 4;
        while (cpt > 1 && ctas(lpc, cpt) < 96) cpt /= 2;
    } else {
        while (ctas(lpc, cpt) < 96) {
            if (cpt > 2) cpt = 2;
            else if (lpc < 32 && dpt > 4) { lpc *= 2; dpt /= 2; }
            else if (cpt > 1) cpt = 1;
            else break;
        }
    }
#define FT_RULE(L, D, C) if (lpc == L && dpt == D && cpt == C) return launch_decay_rule_t<L, D, C>(a, n_req, stream)
#define FT_RULE_L(L) FT_RULE(L, 4, 1); FT_RULE(L, 4, 2); FT_RULE(L, 4, 4); FT_RULE(L, 8, 1); FT_RULE(L, 8, 2); FT_RULE(L, 8, 4); \
                     FT_RULE(L, 16, 1); FT_RULE(L, 16, 2); FT_RULE(L, 16, 4)
    FT_RULE_L(4); FT_RULE_L(8); FT_RULE_L(16); FT_RULE_L(32);
    FT_RULE(32, 32, 1); FT_RULE(32, 32, 2);
#undef FT_RULE_L
#undef FT_RULE
    FT_REQUIRE(false, "decay rule: no kernel for %d lanes x %d channels x %d columns", lpc, dpt, cpt);
    return -1;
}

extern "C" int ft_decay_rule(const float* q, const float* k, const float* v, const float* ab, float* o, float* state,
                             const int* req_start, const int* req_pos0, const int* req_slot, int n_req, int heads, int qk_heads,
                             int dim, int vd, long long slot_stride, int lanes, int T, void* stream) {
    FT_REQUIRE(q && k && v && ab && o && state && req_start && req_pos0 && req_slot, "ft_decay_rule: null argument");
    RecurArgs a;
    a.q = q; a.k = k; a.v = v; a.ab = ab; a.o = o; a.state = state;
    a.ldq = a.ldk = qk_heads * dim; a.ldv = a.ldo = heads * vd;
    a.slot_stride = slot_stride; a.s_off = 0;
    a.req_start = req_start; a.req_pos0 = req_pos0; a.req_slot = req_slot;
    a.heads = heads; a.qk_heads = qk_heads; a.dim = dim; a.vd = vd; a.lanes = lanes;
    return launch_decay_rule(a, n_req, T, (cudaStream_t)stream);
}

// ------------------------------------------------------------------ gated matrix memory: gates and the running maximum
// Per token: values with a column of ones appended (the normaliser rides along as one more state column), and the log
// gates i = cap tanh((z_i + b_i) / cap), f = logsigmoid(cap tanh((z_f + b_f) / cap)).
__global__ void __launch_bounds__(128) memory_prep_kernel(MemoryArgs a) {
    pdl_wait();
    const int t = blockIdx.x, h = blockIdx.y;
    const float* pr = a.proj + (size_t)t * a.ldp;
    const int ve = a.vdim + 1;
    float* dst = a.v_ext + ((size_t)t * a.heads + h) * ve;
    for (int j = threadIdx.x; j < ve; j += blockDim.x) dst[j] = j < a.vdim ? pr[a.o_v + h * a.vdim + j] : 1.f;
    if (threadIdx.x == 0) {
        const float zi = pr[a.o_i + h] + a.gate_bias[h], zf = pr[a.o_f + h] + a.gate_bias[a.heads + h];
        const float gi = a.cap * tanhf(zi / a.cap);
        const float gf = -softplus_f(-(a.cap * tanhf(zf / a.cap)));
        a.gates[((size_t)t * a.heads + h) * 2] = gi;
        a.gates[((size_t)t * a.heads + h) * 2 + 1] = gf;
    }
}
// One warp per (request, head): m_t = max(f_t + m_(t-1), i_t) is a scan under the associative rule
// (F1, G1) o (F2, G2) = (F1 + F2, max(G1 + F2, G2)), so 32 tokens are taken at a time with shuffles and m enters each block as
// m_t = max(F_t + m_in, G_t).  Then a = exp(f + m_(t-1) - m_t), b = exp(i - m_t), floor[t] = exp(-m_t), the lower bound of the
// read-out's denominator.  m lives in the state slot, 0 at a sequence's start.
__global__ void __launch_bounds__(128) memory_scan_kernel(MemoryArgs a, int n_units) {
    pdl_wait();
    const int unit = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (unit >= n_units) return;
    const int r = unit / a.heads, h = unit % a.heads;
    const int t0 = a.req_start[r], t1 = a.req_start[r + 1];
    if (t1 <= t0) return;
    float* ms = a.state + (size_t)a.req_slot[r] * a.slot_stride + a.m_off + h;
    float m = a.req_pos0[r] > 0 ? *ms : 0.f;
    for (int b0 = t0; b0 < t1; b0 += 32) {
        const int t = b0 + lane;
        const bool in = t < t1;
        const size_t at = (size_t)(in ? t : t1 - 1) * a.heads + h;
        const float gi = in ? a.gates[2 * at] : -INFINITY, gf = in ? a.gates[2 * at + 1] : 0.f;
        float F = gf, G = gi;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const float pF = __shfl_up_sync(0xffffffffu, F, off), pG = __shfl_up_sync(0xffffffffu, G, off);
            if (lane >= off) { G = fmaxf(pG + F, G); F = pF + F; }
        }
        const float mt = fmaxf(F + m, G);
        float mp = __shfl_up_sync(0xffffffffu, mt, 1);
        if (lane == 0) mp = m;
        if (in) {
            a.ab[2 * at] = expf(gf + mp - mt);
            a.ab[2 * at + 1] = expf(gi - mt);
            a.floor[at] = expf(-mt);
        }
        m = __shfl_sync(0xffffffffu, mt, min(31, t1 - 1 - b0));
    }
    if (lane == 0) *ms = m;
}
int launch_memory_prep(const MemoryArgs& a, int T, int n_req, cudaStream_t stream) {
    FT_REQUIRE(a.heads >= 1 && a.cap > 0.f, "matrix memory: bad head count or gate cap");
    launch_after(memory_prep_kernel, dim3(T, a.heads), 128, 0, stream, a);
    FT_CHECK_CUDA(cudaGetLastError());
    const int units = n_req * a.heads;
    launch_after(memory_scan_kernel, (units + 3) / 4, 128, 0, stream, a, units);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

// ------------------------------------------------------------------ state space: convolution, step sizes, tails
// u = raw x | B | C channels of a token (proj columns o_x ..).  out[t][c] = silu(bias[c] + sum_j w[c][K-1-j] u[t-j][c]); rows
// before the step's first come from the slot's tail (the last K-1 raw inputs of the sequence), zeros before position 0.
// A CTA takes TB tokens of 256 channels, a thread one channel; the last group of channels also forms the step sizes.  Up to four taps
// whose inputs are all rows of this step and of one request are read once for the block.
template <int TB>
__global__ void __launch_bounds__(256) space_conv_kernel(SpaceArgs a, int T) {
    pdl_wait();
    const int t0 = blockIdx.x * TB, nt = min(TB, T - t0), K = a.taps;
    const int c = blockIdx.y * 256 + threadIdx.x;
    if (blockIdx.y + 1 == gridDim.y)
        for (int i = threadIdx.x; i < nt * a.heads; i += blockDim.x) {
            const int t = t0 + i / a.heads, h = i % a.heads;
            const float dt = softplus_f(a.proj[(size_t)t * a.ldp + a.o_dt + h] + a.dt_bias[h]);
            a.ab[((size_t)t * a.heads + h) * 2] = expf(-expf(a.a_log[h]) * dt);
            a.ab[((size_t)t * a.heads + h) * 2 + 1] = dt;
        }
    if (c >= a.channels) return;
    const float bias = a.conv_b ? a.conv_b[c] : 0.f;
    auto put = [&](int t, float acc) { a.xbc[(size_t)t * a.channels + c] = a.act ? silu_f(acc) : acc; };
    bool inside = TB > 1 && nt == TB && K <= 4;
    if (inside) {
        const int r = a.seq_rows[t0];
        inside = a.seq_rows[t0 + TB - 1] == r && t0 - a.req_start[r] >= 3;
    }
    if (inside) {
        float w[4], v[TB + 3];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = i >= 4 - K ? a.conv_w[(size_t)c * K + i - (4 - K)] : 0.f;
        const float* row = a.proj + (size_t)(t0 - 3) * a.ldp + a.o_x + c;
#pragma unroll
        for (int i = 0; i < TB + 3; ++i) v[i] = row[(size_t)i * (unsigned)a.ldp];
#pragma unroll
        for (int i = 0; i < TB; ++i) {
            float acc = bias;
#pragma unroll
            for (int j = 3; j >= 0; --j)                 // the current token's tap first, as below; rows out of reach are left out:
                if (j >= 4 - K) acc = fmaf(w[j], v[i + j], acc);      // a zero tap would make a NaN of an infinite one
            put(t0 + i, acc);
        }
        return;
    }
    for (int t = t0; t < t0 + nt; ++t) {
        const int r = a.seq_rows[t];
        const int start = a.req_start[r], pos0 = a.req_pos0[r];
        const int k = t - start;
        const float* tail = a.state + (size_t)a.req_slot[r] * a.slot_stride + a.tail_off;
        float acc = bias;
        for (int j = 0; j < K; ++j) {
            float u = 0.f;
            if (k - j >= 0) u = a.proj[(size_t)(t - j) * a.ldp + a.o_x + c];
            else if (pos0 + k - j >= 0) u = tail[(size_t)c * (K - 1) + (k - j + K - 1)];
            acc = fmaf(a.conv_w[(size_t)c * K + (K - 1 - j)], u, acc);
        }
        put(t, acc);
    }
}
// The same for blocks of eight tokens, rows on 16 bytes and four taps: a thread takes four channels (one: 27 us for 2313 tokens of 4352 channels; now
// 25.2 us, the bytes take 12).
__global__ void __launch_bounds__(128) space_conv_rows_kernel(SpaceArgs a, int T) {
    pdl_wait();
    constexpr int TB = 8;
    const int t0 = blockIdx.x * TB, nt = min(TB, T - t0);
    const int c = (blockIdx.y * 128 + threadIdx.x) * 4;
    if (blockIdx.y + 1 == gridDim.y)
        for (int i = threadIdx.x; i < nt * a.heads; i += blockDim.x) {
            const int t = t0 + i / a.heads, h = i % a.heads;
            const float dt = softplus_f(a.proj[(size_t)t * a.ldp + a.o_dt + h] + a.dt_bias[h]);
            a.ab[((size_t)t * a.heads + h) * 2] = expf(-expf(a.a_log[h]) * dt);
            a.ab[((size_t)t * a.heads + h) * 2 + 1] = dt;
        }
    if (c >= a.channels) return;
    const float4 bias = a.conv_b ? load_f4(a.conv_b + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 w[4];
    load_taps4(a.conv_w + (size_t)c * 4, w);
    auto put = [&](int t, float4 s) {
        if (a.act) s = make_float4(silu_f(s.x), silu_f(s.y), silu_f(s.z), silu_f(s.w));
        store_f4(a.xbc + (size_t)t * a.channels + c, s);
    };
    const int first = a.seq_rows[t0];
    if (nt == TB && a.seq_rows[t0 + TB - 1] == first && t0 - a.req_start[first] >= 3) {
        float4 v[TB + 3];
        const float* row = a.proj + (size_t)(t0 - 3) * a.ldp + a.o_x + c;
#pragma unroll
        for (int i = 0; i < TB + 3; ++i) v[i] = load_f4(row + (size_t)i * (unsigned)a.ldp);
#pragma unroll
        for (int i = 0; i < TB; ++i) {
            float4 acc = bias;
#pragma unroll
            for (int j = 3; j >= 0; --j) acc = fma_f4(w[j], v[i + j], acc);          // the current token's tap first, as above
            put(t0 + i, acc);
        }
        return;
    }
    for (int t = t0; t < t0 + nt; ++t) {
        const int r = a.seq_rows[t], k = t - a.req_start[r], pos0 = a.req_pos0[r];
        const float* tail = a.state + (size_t)a.req_slot[r] * a.slot_stride + a.tail_off;
        float4 acc = bias;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k - j >= 0) u = load_f4(a.proj + (size_t)(t - j) * a.ldp + a.o_x + c);
            else if (pos0 + k - j >= 0) {
                const float* p = tail + (size_t)c * 3 + (k - j + 3);
                u = make_float4(p[0], p[3], p[6], p[9]);
            }
            acc = fma_f4(w[3 - j], u, acc);
        }
        put(t, acc);
    }
}
// The slot's tail after the step: the raw inputs of the last K-1 positions, from this step's rows or the old tail.
constexpr int kMaxTaps = 16;
__global__ void __launch_bounds__(256) space_tail_kernel(SpaceArgs a) {
    pdl_wait();
    const int r = blockIdx.y;
    const int start = a.req_start[r], n = a.req_start[r + 1] - start, pos0 = a.req_pos0[r], K = a.taps;
    if (n <= 0 || K <= 1) return;
    float* tail = a.state + (size_t)a.req_slot[r] * a.slot_stride + a.tail_off;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < a.channels; c += gridDim.x * blockDim.x) {
        float nv[kMaxTaps];
        for (int i = 0; i < K - 1; ++i) {
            const int k = n - (K - 1) + i;
            float u = 0.f;
            if (k >= 0) u = a.proj[(size_t)(start + k) * a.ldp + a.o_x + c];
            else if (pos0 + k >= 0) u = tail[(size_t)c * (K - 1) + (k + K - 1)];
            nv[i] = u;
        }
        for (int i = 0; i < K - 1; ++i) tail[(size_t)c * (K - 1) + i] = nv[i];
    }
}
int launch_space_prep(const SpaceArgs& a, int T, int n_req, cudaStream_t stream) {
    FT_REQUIRE(a.taps >= 1 && a.taps <= kMaxTaps, "state space: 1 to %d convolution taps (got %d)", kMaxTaps, a.taps);
    const int groups = (a.channels + 255) / 256;
    const uintptr_t all = (uintptr_t)a.proj | (uintptr_t)a.conv_w | (uintptr_t)a.conv_b | (uintptr_t)a.xbc;
    if (T > 64 && a.taps == 4 && a.channels % 4 == 0 && a.ldp % 4 == 0 && a.o_x % 4 == 0 && (all & 15) == 0)
        launch_after(space_conv_rows_kernel, dim3((T + 7) / 8, (a.channels / 4 + 127) / 128), 128, 0, stream, a, T);
    else if (T > 64) launch_after(space_conv_kernel<8>, dim3((T + 7) / 8, groups), 256, 0, stream, a, T);
    else launch_after(space_conv_kernel<1>, dim3(T, groups), 256, 0, stream, a, T);
    FT_CHECK_CUDA(cudaGetLastError());
    launch_after(space_tail_kernel, dim3((a.channels + 255) / 256, n_req), 256, 0, stream, a);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

// ------------------------------------------------------------------ read-out of the recurrent branches
// One CTA per (token, norm group).  Value of column c = (head h, j):
//   o[t][h * vd + j] * q_scale                              (vd = vdim, or vdim + 1 with the normaliser in the last column)
//   / (max(|o[t][h * vd + vdim] * q_scale|, floor[t][h]) + 1e-6)      with a normaliser
//   + skip[h] * x[t][c]                                      with a skip
//   * silu(gate[t][c])                                       gate_kind 1 (before the norm)
// then divided by the root mean square of its group, times gain[c], times sigmoid (gate_kind 2) or silu (3) of gate[t][c].
__device__ __forceinline__ float readout_value(const ReadoutArgs& a, int t, int c) {
    const int h = c / a.vdim, j = c % a.vdim;
    const float* orow = a.o + (size_t)t * a.ldo + (size_t)h * a.vd;
    float v = orow[j] * a.q_scale;
    if (a.floor) v = v / (fmaxf(fabsf(orow[a.vdim] * a.q_scale), a.floor[(size_t)t * a.heads + h]) + 1e-6f);
    if (a.skip) v = fmaf(a.skip[h], a.x[(size_t)t * a.ldx + c], v);
    if (a.gate_kind == 1) v *= silu_f(a.gate[(size_t)t * a.ldg + c]);
    return v;
}
constexpr int kReadoutKeep = 8;      // values a thread keeps in registers between the two passes
__global__ void __launch_bounds__(256) readout_kernel(ReadoutArgs a) {
    pdl_wait();
    __shared__ float red[33];
    const int t = blockIdx.x / a.norm_groups, g = blockIdx.x % a.norm_groups;
    const int n = a.heads * a.vdim / a.norm_groups, c0 = g * n;
    float keep[kReadoutKeep];
    float ss = 0.f;
    int i = 0;
    for (int c = threadIdx.x; c < n; c += blockDim.x, ++i) {
        const float v = readout_value(a, t, c0 + c);
        if (i < kReadoutKeep) keep[i] = v;
        ss = fmaf(v, v, ss);
    }
    ss = blockDim.x == 32 ? warp_sum(ss) : cta_sum(ss, red);
    const float rr = 1.f / sqrtf(ss / (float)n + a.eps);
    i = 0;
    for (int c = threadIdx.x; c < n; c += blockDim.x, ++i) {
        float v = (i < kReadoutKeep ? keep[i] : readout_value(a, t, c0 + c)) * rr;
        if (a.gain) v *= a.gain[c0 + c];
        if (a.gate_kind == 2) v *= sigmoid_f(a.gate[(size_t)t * a.ldg + c0 + c]);
        else if (a.gate_kind == 3) v *= silu_f(a.gate[(size_t)t * a.ldg + c0 + c]);
        const size_t at = (size_t)t * a.heads * a.vdim + c0 + c;
        if (a.out_hi) {
            const __nv_bfloat16 b = __float2bfloat16_rn(v);
            ((__nv_bfloat16*)a.out_hi)[at] = b;
            ((__nv_bfloat16*)a.out_lo)[at] = __float2bfloat16_rn(v - __bfloat162float(b));
        } else {
            a.out[at] = v;
        }
    }
}
// The same with a normaliser and a norm per head: a warp per (token, head), two columns per lane and step, all of a head's columns in registers, the
// normaliser read once (a CTA per (token, head): 39 us for 2313 tokens of eight heads of 256; now 15.6 us, the bytes take 9).
template <int NP>
__global__ void __launch_bounds__(256) readout_heads_kernel(ReadoutArgs a, int n_pairs) {
    pdl_wait();
    const int id = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (id >= n_pairs) return;
    const int t = id / a.heads, h = id % a.heads, n = a.vdim, c0 = h * n;
    const float* orow = a.o + (size_t)t * a.ldo + (size_t)h * a.vd;
    float2 v[NP], z[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const int c = 2 * lane + 64 * i;
        v[i] = c < n ? make_float2(orow[c], orow[c + 1]) : make_float2(0.f, 0.f);
        z[i] = a.gate_kind && c < n ? *reinterpret_cast<const float2*>(a.gate + (size_t)t * a.ldg + c0 + c) : make_float2(0.f, 0.f);
    }
    const float den = fmaxf(fabsf(orow[n] * a.q_scale), a.floor[(size_t)t * a.heads + h]) + 1e-6f;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const int c = 2 * lane + 64 * i;
        if (c >= n) continue;
        v[i].x = v[i].x * a.q_scale / den;
        v[i].y = v[i].y * a.q_scale / den;
        if (a.skip) {
            const float2 x = *reinterpret_cast<const float2*>(a.x + (size_t)t * a.ldx + c0 + c);
            v[i].x = fmaf(a.skip[h], x.x, v[i].x);
            v[i].y = fmaf(a.skip[h], x.y, v[i].y);
        }
        if (a.gate_kind == 1) { v[i].x *= silu_f(z[i].x); v[i].y *= silu_f(z[i].y); }
        ss = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, ss));
    }
    const float rr = 1.f / sqrtf(warp_sum(ss) / (float)n + a.eps);
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const int c = 2 * lane + 64 * i;
        if (c >= n) continue;
        float x = v[i].x * rr, y = v[i].y * rr;
        if (a.gain) { x *= a.gain[c0 + c]; y *= a.gain[c0 + c + 1]; }
        if (a.gate_kind == 2) { x *= sigmoid_f(z[i].x); y *= sigmoid_f(z[i].y); }
        else if (a.gate_kind == 3) { x *= silu_f(z[i].x); y *= silu_f(z[i].y); }
        const size_t at = (size_t)t * a.heads * n + c0 + c;
        if (a.out_hi) {
            const uint32_t hi = pack_bf16(x, y);
            *reinterpret_cast<uint32_t*>((__nv_bfloat16*)a.out_hi + at) = hi;
            *reinterpret_cast<uint32_t*>((__nv_bfloat16*)a.out_lo + at) = pack_bf16(x - bf16_lo(hi), y - bf16_hi(hi));
        } else {
            *reinterpret_cast<float2*>(a.out + at) = make_float2(x, y);
        }
    }
}
// The same where a head's columns are whole 16-byte groups without a normaliser: NV groups of four columns per thread, all of the
// group's columns in registers between the two passes (one column at a time: 91 us for 2313 tokens of 4096 gated columns; now 36 us).
template <int NV>
__global__ void __launch_bounds__(256) readout_rows_kernel(ReadoutArgs a) {
    pdl_wait();
    __shared__ float red[33];
    const int t = blockIdx.x / a.norm_groups, g = blockIdx.x % a.norm_groups;
    const int n = a.heads * a.vdim / a.norm_groups, c0 = g * n;
    // Everything that a long row needs is asked for before the first number is used (4096 columns, 16 rows 8.9 us, so 6.7; 2313 rows 38, so 33); short rows want
    // the registers for more CTAs instead (2313 rows of 2048: 12.5 us, 14.1 that way).
    constexpr bool FIRST = NV > 2;
    float4 v[NV], x[FIRST ? NV : 1], z[FIRST ? NV : 1];
    float k[FIRST ? NV : 1];
    float ss = 0.f;
    auto gate4 = [&](int c) { return load_f4(a.gate + (size_t)t * a.ldg + c); };
    if (FIRST)
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = 4 * ((int)threadIdx.x + (int)blockDim.x * i);
            if (c < n) {
                v[i] = load_f4(a.o + (size_t)t * a.ldo + c0 + c);
                if (a.gate_kind) z[FIRST ? i : 0] = gate4(c0 + c);
                if (a.skip) {
                    x[FIRST ? i : 0] = load_f4(a.x + (size_t)t * a.ldx + c0 + c);
                    k[FIRST ? i : 0] = a.skip[(c0 + c) / a.vdim];
                }
            }
        }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = 4 * ((int)threadIdx.x + (int)blockDim.x * i);
        if (c >= n) continue;
        float4 o = FIRST ? v[i] : load_f4(a.o + (size_t)t * a.ldo + c0 + c);
        o.x *= a.q_scale; o.y *= a.q_scale; o.z *= a.q_scale; o.w *= a.q_scale;
        if (a.skip) {
            const float f = FIRST ? k[FIRST ? i : 0] : a.skip[(c0 + c) / a.vdim];
            const float4 u = FIRST ? x[FIRST ? i : 0] : load_f4(a.x + (size_t)t * a.ldx + c0 + c);
            o.x = fmaf(f, u.x, o.x); o.y = fmaf(f, u.y, o.y); o.z = fmaf(f, u.z, o.z); o.w = fmaf(f, u.w, o.w);
        }
        if (a.gate_kind == 1) {
            const float4 g = FIRST ? z[FIRST ? i : 0] : gate4(c0 + c);
            o.x *= silu_f(g.x); o.y *= silu_f(g.y); o.z *= silu_f(g.z); o.w *= silu_f(g.w);
        }
        v[i] = o;
        ss += o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w;
    }
    ss = blockDim.x == 32 ? warp_sum(ss) : cta_sum(ss, red);
    const float rr = 1.f / sqrtf(ss / (float)n + a.eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = 4 * ((int)threadIdx.x + (int)blockDim.x * i);
        if (c >= n) continue;
        float4 o = make_float4(v[i].x * rr, v[i].y * rr, v[i].z * rr, v[i].w * rr);
        if (a.gain) {
            const float4 w = *reinterpret_cast<const float4*>(a.gain + c0 + c);
            o.x *= w.x; o.y *= w.y; o.z *= w.z; o.w *= w.w;
        }
        if (a.gate_kind >= 2) {
            const float4 g = FIRST ? z[FIRST ? i : 0] : gate4(c0 + c);
            if (a.gate_kind == 2) { o.x *= sigmoid_f(g.x); o.y *= sigmoid_f(g.y); o.z *= sigmoid_f(g.z); o.w *= sigmoid_f(g.w); }
            else { o.x *= silu_f(g.x); o.y *= silu_f(g.y); o.z *= silu_f(g.z); o.w *= silu_f(g.w); }
        }
        const size_t at = (size_t)t * a.heads * a.vdim + c0 + c;
        if (a.out_hi) {                               // as the bf16 planes that the output projection reads
            uint2 h, l;
            h.x = pack_bf16(o.x, o.y); h.y = pack_bf16(o.z, o.w);
            l.x = pack_bf16(o.x - bf16_lo(h.x), o.y - bf16_hi(h.x)); l.y = pack_bf16(o.z - bf16_lo(h.y), o.w - bf16_hi(h.y));
            *reinterpret_cast<uint2*>((__nv_bfloat16*)a.out_hi + at) = h;
            *reinterpret_cast<uint2*>((__nv_bfloat16*)a.out_lo + at) = l;
        } else {
            *reinterpret_cast<float4*>(a.out + at) = o;
        }
    }
}
int launch_readout(const ReadoutArgs& a, int T, cudaStream_t stream) {
    FT_REQUIRE(a.norm_groups >= 1 && (a.heads * a.vdim) % a.norm_groups == 0, "read-out: %d columns do not split into %d norm groups",
               a.heads * a.vdim, a.norm_groups);
    const int n = a.heads * a.vdim / a.norm_groups;
    FT_REQUIRE(a.out || (a.out_hi && a.out_lo), "read-out: no place for the results");
    const uintptr_t all = (uintptr_t)a.o | (uintptr_t)a.out | (uintptr_t)a.gate | (uintptr_t)a.x | (uintptr_t)a.gain | (uintptr_t)a.out_hi | (uintptr_t)a.out_lo;
    if (!a.floor && a.vd == a.vdim && a.vdim % 4 == 0 && n % 4 == 0 && n <= 8192 && a.ldo % 4 == 0 && (!a.gate || a.ldg % 4 == 0) && (!a.skip || a.ldx % 4 == 0) &&
        (all & 15) == 0) {
        const int th = n <= 128 ? 32 : n <= 256 ? 64 : n <= 512 ? 128 : 256;
        if (n <= 4 * th) launch_after(readout_rows_kernel<1>, T * a.norm_groups, th, 0, stream, a);
        else if (n <= 8 * th) launch_after(readout_rows_kernel<2>, T * a.norm_groups, th, 0, stream, a);
        else if (n <= 16 * th) launch_after(readout_rows_kernel<4>, T * a.norm_groups, th, 0, stream, a);
        else launch_after(readout_rows_kernel<8>, T * a.norm_groups, th, 0, stream, a);
        FT_CHECK_CUDA(cudaGetLastError());
        return 0;
    }
    if (a.floor && a.norm_groups == a.heads && a.vdim % 2 == 0 && n <= 512 && (!a.gate_kind || a.ldg % 2 == 0) && (!a.skip || a.ldx % 2 == 0) &&
        (((uintptr_t)a.out | (uintptr_t)a.gate | (uintptr_t)a.x) & 7) == 0 && (((uintptr_t)a.out_hi | (uintptr_t)a.out_lo) & 3) == 0) {
        const int pairs = T * a.heads, grid = (pairs + 7) / 8;
        if (n <= 128) launch_after(readout_heads_kernel<2>, grid, 256, 0, stream, a, pairs);
        else if (n <= 256) launch_after(readout_heads_kernel<4>, grid, 256, 0, stream, a, pairs);
        else launch_after(readout_heads_kernel<8>, grid, 256, 0, stream, a, pairs);
        FT_CHECK_CUDA(cudaGetLastError());
        return 0;
    }
    const int threads = n <= 64 ? 32 : n <= 256 ? 64 : n <= 1024 ? 128 : 256;
    launch_after(readout_kernel, T * a.norm_groups, threads, 0, stream, a);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace ft

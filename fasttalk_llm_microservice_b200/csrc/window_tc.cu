// Window attention of prompt portions on the tensor cores, in fp32 accuracy (slices.cuh): against 64 bits scores, softmax weights and their sums come out as near as
// those of the fp32 kernels of branches.cu, or nearer, and a row shows nothing of keys that it does not see.
//
// A CTA takes 128 rows: a run of up to 64 tokens times the query heads of one key head.  Keys come 64 at a time from the first one the run's
// first token sees; every key and value row becomes three bf16 slices in shared memory once per CTA and serves all rows.  Scores: eight
// products 128 x 64 x D.  Softmax on the CUDA cores, a row by four threads of the same lane of four warps.  Weights as slices in tensor
// memory, eight products 128 x V x 64, and the sums join the rows' fp32 registers (rescaled there).  The fp32 kernel (64 rows and 32 keys at
// a time, multiply-adds and shared-memory reads bound it, 20 TFLOP/s of products) took 5.6 us per tile of half the keys and half the rows.  2313 tokens of 16
// heads of 128, window 512: 389 -> 132 us with a cap, 436 -> 145 us with a bias by distance.
//
// Per tile: value slices and the last tile's sums beside the scores' products, the next tile's key slices beside the sums' products;
// softmax alone.  Two barriers for the CTA, one for the four warps of a row.
//
// Shared memory: the queries' third slice | key slices, value slices (before them the staged queries, after them the staged results).
// TMEM columns: queries' first two slices 0..127; scores 128..255 (first | second accumulator), over them the weights' slices;
// sums 256..511 (first | second accumulator).
//
// Where a query, key or value is infinite, NaN or beyond 2^36 the CTA's rows go one by one through plain fp32 code: a hidden key's weight of
// zero must not make a NaN of its value.  Every wait has a limit; a CTA whose wait runs out marks `err`, leaves NaN and ends.
#include "common.cuh"
#include "ft_internal.h"
#include "slices.cuh"

#include <algorithm>

namespace ft {
namespace {

constexpr int WR_ROWS = 128, WR_KEYS = 64, WR_THREADS = 512, WR_WARPS = 16;
constexpr int WR_QBLK = WR_ROWS * 128, WR_KBLK = WR_KEYS * 128;      // bytes of a [128 rows] / [64 keys][64 columns] block
constexpr int WR_LDQ = 132;                             // floats between staged rows
constexpr int WR_COL_Q = 0, WR_COL_S = 128, WR_COL_P = 128, WR_COL_O = 256;
constexpr int WR_ISSUE_S = 15, WR_ISSUE_O = 10;         // the warps that issue scores' and sums' products, which holds them up for most of the products' time
constexpr unsigned WR_BIG = (127u + 36) << 23;

// tanh of up to 0.6 in size: x + x^3 Q(x^2), Q fitted to the smallest relative error over the range (6.0e-9; 0.68 ulp in fp32).  tanhf takes
// forty instructions an element on either of its two ways, 6000 clocks a tile.
constexpr float kTanhSmall = 0.6f;
__device__ __forceinline__ float tanh_small(float x) {
    const float z = x * x;
    float q = -0.005905867554247379f;
    q = __fmaf_rn(q, z, 0.02080538310110569f);
    q = __fmaf_rn(q, z, -0.053786683827638626f);
    q = __fmaf_rn(q, z, 0.13331958651542664f);
    q = __fmaf_rn(q, z, -0.33333298563957214f);
    return __fmaf_rn(x * z, q, x);
}

template <int DB, int VB>
constexpr size_t window_smem() {
    const size_t kv = (size_t)3 * (DB + VB) * WR_KBLK, rows = (size_t)WR_ROWS * WR_LDQ * 4;
    return 1024 + (size_t)DB * WR_QBLK + (kv > rows ? kv : rows);
}

// One row by one warp in plain fp32, for runs that hold numbers the slices do not take
__device__ __noinline__ void window_row(const WindowArgs& a, const int* pt, int t, int h, int p, int lane) {
    const int g = h / (a.H / a.G);
    const int lo = a.window > 0 ? (a.chunked ? p - p % a.window : max(0, p - a.window + 1)) : 0;
    const int nf = min(a.keep_first, lo), n = nf + p - lo + 1;
    const size_t rowsz = (size_t)a.G * (a.dim + a.vdim);
    const float* q = a.q_out + ((size_t)t * a.H + h) * a.dim;
    float m = -INFINITY, l = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int b0 = 0; b0 < n; b0 += 32) {
        const int idx = b0 + lane, key = idx < nf ? idx : lo + idx - nf;
        const bool valid = idx < n;
        const float* kr = a.cache + ((size_t)pt[(valid ? key : p) >> 6] * 64 + ((valid ? key : p) & 63)) * rowsz;
        float s = 0.f;
        for (int c = 0; c < a.dim; ++c) s = fmaf(q[c], kr[(size_t)g * a.dim + c], s);
        s *= a.scale;
        if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
        if (a.rel && valid) s += a.rel[(size_t)min(p - key, a.rel_n - 1) * a.H + h];
        if (!valid) s = -INFINITY;
        const float m_new = fmaxf(m, warp_max(s));
        const float corr = m_new == -INFINITY ? 1.f : expf(m - m_new), w = valid && m_new != -INFINITY ? expf(s - m_new) : 0.f;
        l = l * corr + warp_sum(w);
        m = m_new;
        for (int i = 0; i < 4; ++i) acc[i] *= corr;
        for (int x = 0; x < 32 && b0 + x < n; ++x) {
            const float wx = __shfl_sync(0xffffffffu, w, x);
            const float* vr = (const float*)__shfl_sync(0xffffffffu, (unsigned long long)kr, x) + (size_t)a.G * a.dim + (size_t)g * a.vdim;
            for (int i = 0; i < 4; ++i)
                if (lane + 32 * i < a.vdim) acc[i] = fmaf(wx, vr[lane + 32 * i], acc[i]);
        }
    }
    float f = 1.f / l;
    if (a.sink) {
        const float mf = fmaxf(m, a.sink[h]), e = expf(m - mf);
        f = e / (l * e + expf(a.sink[h] - mf));
    }
    for (int i = 0; i < 4; ++i) {
        const int c = lane + 32 * i;
        if (c >= a.vdim) break;
        float o = acc[i] * f;
        if (a.gate) o *= 1.f / (1.f + expf(-a.gate[(size_t)t * a.ldg + h * a.vdim + c]));
        a.out[((size_t)t * a.H + h) * a.vdim + c] = o;
    }
}

template <int DB, int VB>
__global__ void __launch_bounds__(WR_THREADS, 1) window_runs_kernel(WindowArgs a, WindowTiles tm, int QT, int subs) {
    pdl_wait();
    extern __shared__ uint8_t wr_raw[];
    __shared__ float part_max[4][WR_ROWS], part_sum[4][WR_ROWS];
    __shared__ uint64_t done[2];                         // scores, sums
    __shared__ uint32_t tmem_slot;
    __shared__ int odd;
    __shared__ volatile int dead;
    const int tile = blockIdx.x / subs, sub = blockIdx.x % subs, g = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int j = tm.tile_req[tile];
    const int q0 = tm.tile_q0[tile] + sub * QT;
    const int n_j = tm.req_q_start[j + 1] - tm.req_q_start[j];
    if (sub * QT >= 64 || q0 >= n_j) return;
    const int ntok = min(QT, min(n_j - q0, 64 - sub * QT)), grp = a.H / a.G, used = ntok * grp;
    const int row_base = tm.req_q_start[j] + q0, p_first = tm.req_pos0[j] + q0;
    const int* pt = a.page_table + (size_t)tm.req_slot[j] * a.max_pages;
    const size_t rowsz = (size_t)a.G * (a.dim + a.vdim);
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(wr_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *ql_s = smem, *k_s = smem + DB * WR_QBLK, *v_s = k_s + 3 * DB * WR_KBLK;
    float* stage = reinterpret_cast<float*>(k_s);
    constexpr int K_PLANE = DB * WR_KBLK, V_PLANE = VB * WR_KBLK;
    const int part = warp >> 2, row = (warp & 3) * 32 + lane;            // TMEM lane; scores: keys part * 16 .., sums: columns part * 16 * VB ..
    if (tid == 0) {
        mbar_init(&done[0], 1);
        mbar_init(&done[1], 1);
        fence_mbar_init();
        dead = 0;
        odd = 0;
    }
    if (warp == 0) {
        tmem_alloc(&tmem_slot, 512);
        tmem_relinquish();
    }
    // ---- queries: whole rows to shared memory, then every thread its part of its row as slices
    for (int r = warp; r < WR_ROWS; r += WR_WARPS) {
        const int c = lane * 4;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < used && c < a.dim) x = *reinterpret_cast<const float4*>(a.q_out + ((size_t)(row_base + r / grp) * a.H + g * grp + r % grp) * a.dim + c);
        *reinterpret_cast<float4*>(stage + r * WR_LDQ + c) = x;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot, lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    {
        constexpr int N = 8 * DB;                        // pairs of a thread
        f32x2 qx[N];
        const float* src = stage + row * WR_LDQ + part * 2 * N;
#pragma unroll
        for (int i = 0; i < N / 2; ++i) *reinterpret_cast<ulonglong2*>(qx + 2 * i) = *reinterpret_cast<const ulonglong2*>(src + 4 * i);
        if (abs_bits(top_of<N>(qx)) >= WR_BIG) odd = 1;
#pragma unroll
        for (int x = 0; x < DB; ++x) {
            uint32_t w[8];
            const int c = part * 2 * N + 16 * x;         // first of 16 channels
            slice_first<8>(qx + 8 * x, w);
            tmem_st8(lanes + WR_COL_Q + c / 2, w);
            slice_next<8>(qx + 8 * x, w);
            tmem_st8(lanes + WR_COL_Q + 64 + c / 2, w);
            slice_last<8>(qx + 8 * x, w);
            uint8_t* at = ql_s + (c >> 6) * WR_QBLK + row * 128;
            *reinterpret_cast<uint4*>(at + ((((c >> 3) & 7) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
            *reinterpret_cast<uint4*>(at + ((((c >> 3) & 7) + 1 ^ (row & 7)) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
        }
        tmem_st_wait();
    }
    __syncthreads();                                     // the staged rows make room for keys and values
    // ---- the keys in order: the kept first positions before the window, then the window's up to the run's last position
    const int lo = a.window > 0 ? (a.chunked ? p_first - p_first % a.window : max(0, p_first - a.window + 1)) : 0, hi = p_first + ntok - 1;
    const int nf = min(a.keep_first, lo), n0 = (nf + WR_KEYS - 1) / WR_KEYS, nt = n0 + (hi - lo) / WR_KEYS + 1;
    auto first_key = [&](int it) { return it >= n0 ? lo + (it - n0) * WR_KEYS : it * WR_KEYS; };
    auto end_key = [&](int it) { return it >= n0 ? hi + 1 : nf; };
    // a tile's rows: eight neighbouring lanes take 128 bytes of a row at a time
    // (a warp's four rows: two apart by four, so that their slices' 8-byte stores spread over all banks)
    const int kq = tid & 7, kr = (lane >> 3 & 1) * 4 + (lane >> 4) + (warp & 1) * 2 + (warp >> 1) * 8;
    auto load = [&](auto* x, int n, int it, int width, size_t at) {
        const int key = first_key(it) + kr;
        const bool live = it < nt && key < end_key(it);
        const float* src = live ? a.cache + ((size_t)pt[key >> 6] * 64 + (key & 63)) * rowsz + at : nullptr;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i >= n) break;
            const int c = (kq + 8 * i) * 4;
            float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live && c < width) f = *reinterpret_cast<const float4*>(src + c);
            x[i][0] = pack2(f.x, f.y);
            x[i][1] = pack2(f.z, f.w);
        }
    };
    f32x2 kx[2 * DB][2], vx[2 * VB][2];
    auto load_k = [&](int it) { load(kx, 2 * DB, it, a.dim, (size_t)g * a.dim); };
    auto load_v = [&](int it) { load(vx, 2 * VB, it, a.vdim, (size_t)a.G * a.dim + (size_t)g * a.vdim); };
    auto place = [&](uint8_t* base, int u) { return base + (u >> 4) * WR_KBLK + kr * 128 + ((((u >> 1) & 7) ^ (kr & 7)) << 4) + (u & 1) * 8; };
    auto keys_out = [&]() {
        if (abs_bits(top_of<4 * VB>(vx[0], top_of<4 * DB>(kx[0]))) >= WR_BIG) odd = 1;
#pragma unroll
        for (int i = 0; i < 2 * DB; ++i) slice4(kx[i], place(k_s, kq + 8 * i), K_PLANE);
    };
    constexpr uint32_t id_s = slice_idesc(WR_ROWS, WR_KEYS), id_o = slice_idesc(WR_ROWS, 64 * VB, true);
    const uint64_t kd = umma_desc_k128(smem_u32(k_s)), vd = umma_desc_mn128(smem_u32(v_s), WR_KBLK), qd = umma_desc_k128(smem_u32(ql_s));
    // all operands but the addresses are known to the compiler: see decay_tc.cu
    auto issue_scores = [&]() {
        if (elect_one()) {
#pragma unroll
            for (int p = 0; p <= kSlicePairs; ++p) {
                const bool last = p == kSlicePairs;
                const int sa = last ? 0 : slice_a(p), sb = last ? 0 : slice_b(p);
                const uint32_t d = tmem + WR_COL_S + (last ? 0 : 64);
#pragma unroll
                for (int k = 0; k < 4 * DB; ++k) {
                    const uint64_t b = kd + sb * (K_PLANE >> 4) + (k >> 2) * (WR_KBLK >> 4) + (k & 3) * 2;
                    const bool more = k > 0 || (p > 0 && !last);
                    if (sa == 2) umma_bf16(d, qd + (k >> 2) * (WR_QBLK >> 4) + (k & 3) * 2, b, id_s, more);      // third slice of the queries, from shared memory
                    else umma_f16_ts(d, tmem + WR_COL_Q + 64 * sa + 8 * k, b, id_s, more);
                }
            }
            umma_commit(&done[0]);
        }
        __syncwarp();
    };
    auto issue_sums = [&]() {
        if (elect_one()) {
#pragma unroll
            for (int p = 0; p <= kSlicePairs; ++p) {
                const bool last = p == kSlicePairs;
                const int sa = last ? 0 : slice_a(p), sb = last ? 0 : slice_b(p);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    umma_f16_ts(tmem + WR_COL_O + (last ? 0 : 128), tmem + WR_COL_P + 32 * sa + 8 * k, vd + sb * (V_PLANE >> 4) + k * (2048 >> 4), id_o,
                                k > 0 || (p > 0 && !last));
            }
            umma_commit(&done[1]);
        }
        __syncwarp();
    };
    const bool real = row < used;
    const int pr = p_first + row / grp, h = g * grp + row % grp;
    // visible: from `seen` on to pr, and the kept ones
    const int seen = a.window <= 0 ? 0 : a.chunked ? pr - pr % a.window : pr - a.window + 1;
    float m = -INFINITY, l = 0.f, corr = 1.f;
    f32x2 acc[8 * VB];
#pragma unroll
    for (int i = 0; i < 8 * VB; ++i) acc[i] = 0ull;
    load_k(0);
    load_v(0);
    keys_out();
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    bool ok = true, plain = odd != 0;
    if (!plain && warp == WR_ISSUE_S) issue_scores();
    for (int it = 0; it < nt && !plain; ++it) {
        // ---- values as slices while the scores are made
#pragma unroll
        for (int i = 0; i < 2 * VB; ++i) slice4(vx[i], place(v_s, kq + 8 * i), V_PLANE);
        load_k(it + 1);
        ok = mbar_sleep_limited(&done[0], it & 1, &dead);
        tc_fence_after();
        __syncwarp();
        // ---- softmax of 16 keys of the row
        float s[16];
        float top = -INFINITY;
        if (ok) {
            float u[16];
            tmem_ld16_nowait(lanes + WR_COL_S + part * 16, reinterpret_cast<uint32_t*>(s));
            tmem_ld16_nowait(lanes + WR_COL_S + 64 + part * 16, reinterpret_cast<uint32_t*>(u));
            tmem_ld_wait();
            const int k0 = first_key(it) + part * 16, kend = end_key(it);
#pragma unroll
            for (int e = 0; e < 16; ++e) s[e] = __fmaf_rn(s[e], a.scale, rest_of(s[e], u[e]) * a.scale);
            if (a.softcap > 0.f) {
                float big = 0.f;
#pragma unroll
                for (int e = 0; e < 16; e += 2) big = top3(big, s[e], s[e + 1]);
                if (__any_sync(0xffffffffu, big > kTanhSmall * a.softcap)) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) s[e] = a.softcap * tanhf(s[e] / a.softcap);
                } else {
                    const float r = 1.f / a.softcap;
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const float x = s[e] * r;        // and what the product has lost of the quotient
                        s[e] = a.softcap * tanh_small(__fmaf_rn(__fmaf_rn(-x, a.softcap, s[e]), r, x));
                    }
                }
            }
            if (a.rel) {
#pragma unroll
                for (int e = 0; e < 16; ++e) s[e] += a.rel[(size_t)min(max(pr - k0 - e, 0), a.rel_n - 1) * a.H + h];
            }
            // all sixteen visible in most tiles
            const int from = max(seen, 0), upto = min(pr, kend - 1);
            if (!__all_sync(0xffffffffu, real && k0 >= from && k0 + 15 <= upto)) {
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const int key = k0 + e;
                    if (!(real && key <= upto && (key >= from || key < a.keep_first))) s[e] = -INFINITY;
                }
            }
#pragma unroll
            for (int e = 0; e < 16; ++e) top = fmaxf(top, s[e]);
        }
        part_max[part][row] = top;
        asm volatile("bar.sync %0, 128;" ::"r"(1 + (warp & 3)) : "memory");      // the four warps of these rows
        const float m_new = fmaxf(fmaxf(m, fmaxf(part_max[0][row], part_max[1][row])), fmaxf(part_max[2][row], part_max[3][row]));
        corr = 1.f;
        if (m_new == -INFINITY) {
#pragma unroll
            for (int e = 0; e < 16; ++e) s[e] = 0.f;
        } else {
            corr = expf(m - m_new);
            float sum = 0.f;
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                s[e] = expf(s[e] - m_new);
                sum += s[e];
            }
            l = l * corr + sum;
        }
        m = m_new;
        {
            f32x2 w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = pack2(s[2 * e], s[2 * e + 1]);
            slices_to_tmem<32>(w, lanes + WR_COL_P + part * 8);
        }
        load_v(it + 1);
        tmem_st_wait();
        fence_proxy_async();
        tc_fence_before();
        ok = __syncthreads_and(ok);
        tc_fence_after();
        if (!ok) break;
        if (warp == WR_ISSUE_O) issue_sums();
        // ---- the next tile's keys as slices while the sums are made
        if (it + 1 < nt) keys_out();
        ok = mbar_sleep_limited(&done[1], it & 1, &dead);
        tc_fence_after();
        fence_proxy_async();
        tc_fence_before();
        ok = __syncthreads_and(ok);
        tc_fence_after();
        if (!ok) break;
        plain = odd != 0;
        if (it + 1 < nt && !plain && warp == WR_ISSUE_S) issue_scores();
        // ---- this tile's sums join the row's
        const f32x2 c2 = pack2(corr, corr);
#pragma unroll
        for (int x = 0; x < VB; ++x) {
            f32x2 o0[8], o1[8];
            tmem_ld16_nowait(lanes + WR_COL_O + (part * VB + x) * 16, reinterpret_cast<uint32_t*>(o0));
            tmem_ld16_nowait(lanes + WR_COL_O + 128 + (part * VB + x) * 16, reinterpret_cast<uint32_t*>(o1));
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[x * 8 + e] = add2(o0[e], fma2(acc[x * 8 + e], c2, rest_of(o0[e], o1[e])));
        }
    }
    if (!ok) {
        if (tid == 0 && a.err) *a.err = 1;
        for (int i = tid; i < used * a.vdim; i += WR_THREADS) {
            const int r = i / a.vdim;
            a.out[((size_t)(row_base + r / grp) * a.H + g * grp + r % grp) * a.vdim + i % a.vdim] = __int_as_float(0x7fc00000);
        }
    } else if (plain) {
        for (int r = warp; r < used; r += WR_WARPS) window_row(a, pt, row_base + r / grp, g * grp + r % grp, p_first + r / grp, lane);
    } else {
        part_sum[part][row] = l;
        __syncthreads();
        l = (part_sum[0][row] + part_sum[1][row]) + (part_sum[2][row] + part_sum[3][row]);
        float f = 1.f / l;
        if (a.sink && real) {
            const float mf = fmaxf(m, a.sink[h]), e = expf(m - mf);
            f = e / (l * e + expf(a.sink[h] - mf));
        }
#pragma unroll
        for (int i = 0; i < 4 * VB; ++i) {
            float x, y, z, w;
            unpack2(acc[2 * i], x, y);
            unpack2(acc[2 * i + 1], z, w);
            *reinterpret_cast<float4*>(stage + row * WR_LDQ + part * 16 * VB + 4 * i) = make_float4(x * f, y * f, z * f, w * f);
        }
        __syncthreads();
        const int c = lane * 4;
        if (c < a.vdim)
            for (int r = warp; r < used; r += WR_WARPS) {
                const size_t t = row_base + r / grp;
                const int hh = g * grp + r % grp;
                float4 x = *reinterpret_cast<const float4*>(stage + r * WR_LDQ + c);
                if (a.gate) {
                    const float* gt = a.gate + t * a.ldg + hh * a.vdim + c;
                    x.x *= 1.f / (1.f + expf(-gt[0])); x.y *= 1.f / (1.f + expf(-gt[1]));
                    x.z *= 1.f / (1.f + expf(-gt[2])); x.w *= 1.f / (1.f + expf(-gt[3]));
                }
                *reinterpret_cast<float4*>(a.out + (t * a.H + hh) * a.vdim + c) = x;
            }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <int DB, int VB>
int launch_runs(const WindowArgs& a, const WindowTiles& tm, cudaStream_t stream) {
    static PerDeviceFlag attr;
    if (!attr.done()) {
        FT_CHECK_CUDA(cudaFuncSetAttribute(window_runs_kernel<DB, VB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)window_smem<DB, VB>()));
        attr.mark();
    }
    const int QT = std::min(64, WR_ROWS / (a.H / a.G)), subs = (64 + QT - 1) / QT;
    launch_after(window_runs_kernel<DB, VB>, dim3(tm.n_tiles * subs, a.G), WR_THREADS, window_smem<DB, VB>(), stream, a, tm, QT, subs);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace

// Heads of at most 128 channels and columns in whole 16-byte units, values beside the keys; no size is too small.  The fp32 tile kernel / this one, us, four heads of 128: 33 new
// tokens 25.5 / 16.1, 2 behind 600 cached ones 159 / 58, 500 new 153 / 54.  With all keys in its first half tile (32) the fp32 kernel is level: 16 heads of 128 in groups of
// four 2 tokens 14.9 / 15.0, 9: 16.3 / 15.7, 17: 15.6 / 16.9; how many keys there are stands in device memory.
bool window_tc_ok(const WindowArgs& a) {
    return a.dim <= 128 && a.vdim <= 128 && ((a.dim | a.vdim) & 3) == 0 && a.v_in_key < 0 && a.H / a.G <= WR_ROWS;
}
int launch_window_tc(const WindowArgs& a, const WindowTiles& tm, cudaStream_t stream) {
    FT_REQUIRE(window_tc_ok(a) && tm.n_tiles > 0, "window attention (tcgen05): head sizes %d / %d do not fit", a.dim, a.vdim);
    if (a.dim <= 64) return a.vdim <= 64 ? launch_runs<1, 1>(a, tm, stream) : launch_runs<1, 2>(a, tm, stream);
    return a.vdim <= 64 ? launch_runs<2, 1>(a, tm, stream) : launch_runs<2, 2>(a, tm, stream);
}

}  // namespace ft

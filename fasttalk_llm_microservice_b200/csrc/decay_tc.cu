// The scalar-decay rule S <- a_t S + b_t k_t v_t^T, o_t = S^T q_t over prompt portions as matrix products, in fp32 accuracy (slices.cuh).
//
// The token-by-token kernel (branches.cu) is a serial chain: one warp per scheduler, 0.28 us a token whatever runs beside it.  Here a CTA
// (request, head, 64 value columns) takes 128 tokens at a time.  With W_ij = a_(j+1) .. a_i and S the state before the run:
//     o_i = sum_{j<=i} W_ij (q_i . k_j) b_j v_j  +  (a_0 .. a_i) S^T q_i          S <- (a_0 .. a_(n-1)) S + sum_j W_(n-1)j k_j (b_j v_j)^T
// Four products per run, 128 x 128 x D, 128 x 64 x D and twice 128 x 64 x 128, each as six fp16 products: 8400 clocks of the tensor pipe.  A
// run takes 26000: forming the slices (some 10000 instruction slots per scheduler) and the barriers between the steps bound the kernel, then
// the 200 KB per run that an SM reads and writes.  The state stays on the chip (16 numbers per thread, fp32) from the first run to the last;
// decays are products of at most 128 numbers to 40 bits (never quotients or logarithms: a decay of zero is nothing special), rounded once.
// Three requests of 683 tokens: 16 heads of 128 x 128 188 -> 97 us, 64 heads of 128 x 64 280 -> 213 us, 8 heads of 128 x 257 189 -> 125 us.
// Error against 64 bits over 2048 tokens: results 1.1e-7 -> 6e-8, states 8e-8 -> 5e-8.
//
// Shared memory: slices of the keys | of the run's values (first weighted for the state, then for the results) | of the state.
// TMEM columns: the state 320..383 until the scores' slices need the place; queries' slices 0..191, after their last product what the run adds to the state 0..127; scores' second
// accumulator 192..319, their slices as an operand 192..383; scores' first accumulator 384..511, then the results (first | second accumulator).
//
// A run that holds infinities, NaN, numbers beyond 2^36 or decays beyond 1 by more than rounding, and runs of few tokens, go token by token: a product
// with a masked zero must not make a NaN of another token's infinity.  Every wait has a limit; a CTA whose wait runs out marks `err`, leaves NaN and ends.
#include "common.cuh"
#include "ft_internal.h"
#include "slices.cuh"

namespace ft {
namespace {

constexpr int DR_RUN = 128, DR_WARPS = 16, DR_THREADS = DR_WARPS * 32, DR_COLS = 64, DR_PARTS = DR_WARPS / 4;
constexpr int DR_FEW = 16;                               // tokens below which a run goes token by token (0.8 us each)
constexpr int DR_ISSUER = 12;                            // the warp that issues the products: its part of the scores lies above the diagonal
constexpr int DR_BLK = DR_RUN * 128;                     // bytes of one [128 rows][64 columns] block
constexpr int DR_K = 2 * DR_BLK;                         // a slice of the keys: 128 channels whatever dim is
constexpr size_t DR_SMEM = 1024 + 3 * (size_t)DR_K + 6 * (size_t)DR_BLK;
constexpr int DR_LDQ = 132, DR_LDO = 68;                 // floats between rows of the staged queries (in the keys' place) and results (in the values')
constexpr int DR_COL_Q = 0, DR_COL_U = 0, DR_COL_S = 192, DR_COL_P = 192, DR_COL_ST = 320, DR_COL_O = 384;
constexpr unsigned DR_BIG_IN = (127u + 36) << 23, DR_BIG_STATE = (127u + 80) << 23, DR_DECAY = 0x3f820000u;      // 2^36, 2^80, 1 + 2^-6

__device__ __forceinline__ void cp16_zfill(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

// A product kept as the unrounded sum of two fp32 numbers: 128 factors stay good to 2^-40.  (In 64 bits the same tables took 9000 clocks a run.)
struct Two { float h, l; };
__device__ __forceinline__ Two mul(Two a, Two b) {
    const float h = a.h * b.h;
    return {h, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.h, b.h, -h)))};
}
__device__ __forceinline__ Two shfl_up16(Two v, int o) { return {__shfl_up_sync(0xffffffffu, v.h, o, 16), __shfl_up_sync(0xffffffffu, v.l, o, 16)}; }
__device__ __forceinline__ Two shfl_down16(Two v, int o) { return {__shfl_down_sync(0xffffffffu, v.h, o, 16), __shfl_down_sync(0xffffffffu, v.l, o, 16)}; }

// D[tmem] (+)= A[tmem] B[smem] over N steps of 16 along the contraction; KMAJOR: B's blocks of 64 lie DR_BLK apart.  Everything but the
// addresses is known to the compiler: operands that are put together at run time cost the issuing thread 150 clocks a product, four
// times what the tensor cores take for it.
template <bool KMAJOR, int N>
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool first) {
#pragma unroll
    for (int k = 0; k < N; ++k)
        umma_f16_ts(d, a + k * 8, b + (KMAJOR ? (k >> 2) * (DR_BLK >> 4) + (k & 3) * 2 : k * (2048 >> 4)), idesc, !first || k > 0);
}
// the five products beside first x first: D (+)= A B, slices of A 64 columns apart, slices of B `plane` bytes
template <bool KMAJOR, int N>
__device__ __forceinline__ void mma_rest(uint32_t d, uint32_t a, uint64_t b, int plane, uint32_t idesc) {
#pragma unroll
    for (int p = 0; p < kSlicePairs; ++p) mma_ts<KMAJOR, N>(d, a + 64 * slice_a(p), b + slice_b(p) * (plane >> 4), idesc, p == 0);
}

// Nothing is computed from x before this point: work moved up across barriers would need more registers than there are.
template <int N>
__device__ __forceinline__ void hold(f32x2* x) {
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+l"(x[i]));
}
template <bool VEC, int DB>
__global__ void __launch_bounds__(DR_THREADS, 1) decay_runs_kernel(RecurArgs a, int* err) {
    extern __shared__ uint8_t dr_raw[];
    __shared__ Two pref[DR_RUN], suff[DR_RUN], full[8];      // products of decays inside a block of 16 tokens: up to and with i, behind j, all
    __shared__ Two mid[8][8], tail[8], head[9];          // of whole blocks: between two, behind one, before one (head[8]: of the run)
    __shared__ __align__(16) float ywk[DR_RUN];          // a block's decays behind j, times the unit of key j
    __shared__ __align__(16) float near[DR_RUN][20];     // decays inside a row's own block of 16
    __shared__ float sa[DR_RUN], sb[DR_RUN], kunit[DR_RUN];
    __shared__ unsigned qtop[DR_PARTS][DR_RUN], ptop[DR_PARTS][DR_RUN], wtop[3][DR_WARPS];
    __shared__ float red[4][DR_COLS];
    __shared__ uint64_t done[4];
    __shared__ uint32_t tmem_slot;
    __shared__ int odd;                                  // 1: the run goes token by token
    __shared__ volatile int dead;
    const int r = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * DR_COLS, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int t0 = a.req_start[r], t1 = a.req_start[r + 1];
    if (t1 <= t0) return;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dr_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *k_s = smem, *v_s = smem + 3 * DR_K, *s_s = v_s + 3 * DR_BLK;
    float *q_stage = reinterpret_cast<float*>(k_s), *o_stage = reinterpret_cast<float*>(v_s);
    const int gh = h / (a.heads / a.qk_heads), cols = min(DR_COLS, a.vd - j0);
    const int part = warp >> 2, row = (warp & 3) * 32 + lane, c0 = part * 16;      // TMEM lane: token of the run or key channel; columns of it
    if (tid == 0) {
        for (int i = 0; i < 4; ++i) mbar_init(&done[i], 1);
        fence_mbar_init();
        dead = 0;
    }
    if (warp == 0) {
        tmem_alloc(&tmem_slot, 512);
        tmem_relinquish();
    }
    // the state: channel `row`, 16 columns
    float* S = a.state + (size_t)a.req_slot[r] * a.slot_stride + a.s_off + ((size_t)h * a.dim + row) * a.vd + j0 + c0;
    const bool s4 = (a.vd & 3) == 0 && ((uintptr_t)S & 15) == 0, o4 = VEC && (a.ldo & 3) == 0 && (a.vd & 3) == 0 && ((uintptr_t)a.o & 15) == 0;
    const bool mine = row < a.dim;            // this thread holds a channel of the state
    float st[16];
    bool carried = a.req_pos0[r] > 0;
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
        const bool live = carried && mine;
        if (s4) {
            const float4 x = live && c0 + i < cols ? *reinterpret_cast<const float4*>(S + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            st[i] = x.x; st[i + 1] = x.y; st[i + 2] = x.z; st[i + 3] = x.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) st[i + e] = live && c0 + i + e < cols ? S[i + e] : 0.f;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot, lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    unsigned s_top = 0;                                  // the largest of the state, known to all threads
    auto all_top = [&](const unsigned* w) { return warp_umax(w[lane & (DR_WARPS - 1)]); };
    auto state_top = [&]() {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 16; i += 2) t = top3(t, st[i], st[i + 1]);
        const unsigned m = warp_umax(abs_bits(t));
        if (lane == 0) wtop[2][warp] = m;
        __syncthreads();
        s_top = all_top(wtop[2]);
    };
    // the state's slices to shared memory, [channel][64 columns]
    auto state_out = [&]() {
        const float inv = slice_inv(s_top);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            f32x2 v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = pack2(st[x * 8 + 2 * e], st[x * 8 + 2 * e + 1]);
            slice8(v, inv, s_s + row * 128 + (((part * 2 + x) ^ (row & 7)) << 4), DR_BLK);
        }
    };
    // four numbers of a row: columns c .. of n, zeros beyond
    auto load4 = [&](f32x2* x, const float* src, int c, int n, bool live) {
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (VEC) {
            if (live && c < n) f = *reinterpret_cast<const float4*>(src + c);
        } else {
            if (live && c < n) f.x = src[c];
            if (live && c + 1 < n) f.y = src[c + 1];
            if (live && c + 2 < n) f.z = src[c + 2];
            if (live && c + 3 < n) f.w = src[c + 3];
        }
        x[0] = pack2(f.x, f.y);
        x[1] = pack2(f.z, f.w);
    };
    // a run's queries to shared memory, a warp per row, so that every thread can then take a part of its own row
    auto stage_q = [&](int base) {
        if (base < t1) {
            const int c = lane * 4;
            for (int i = warp; i < DR_RUN; i += DR_WARPS) {
                const bool live = base + i < t1;
                const float* src = a.q + (size_t)(live ? base + i : base) * a.ldq + (size_t)gh * a.dim;
                float* dst = q_stage + i * DR_LDQ + c;
                if (VEC) {
                    cp16_zfill(dst, c < a.dim ? src + c : src, live && c < a.dim ? 16 : 0);
                } else {
                    float x[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[e] = live && c + e < a.dim ? src[c + e] : 0.f;
                    *reinterpret_cast<float4*>(dst) = make_float4(x[0], x[1], x[2], x[3]);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // neighbouring lanes take neighbouring 16 bytes.  Keys: four numbers from each eighth of row kr's 128; values: four of rows vr + 32 i
    const int kq = tid & 3, kr = tid >> 2, vc = tid & 15, vr = tid >> 4;
    auto load_k = [&](f32x2 (*k)[2], int base) {
        const float* kg = a.k + (size_t)(base + kr) * a.ldk + (size_t)gh * a.dim;
#pragma unroll
        for (int i = 0; i < 4 * DB; ++i) load4(k[i], kg, (kq + 4 * i) * 4, a.dim, base + kr < t1);
    };
    auto load_v = [&](f32x2 (*v)[2], int base) {
        const float* vg = a.v + (size_t)(base + vr) * a.ldv + (size_t)h * a.vd + j0;
#pragma unroll
        for (int i = 0; i < 4; ++i) load4(v[i], vg + (size_t)(32 * i) * a.ldv, vc * 4, cols, base + vr + 32 * i < t1);
    };
    auto scale_v = [&](f32x2* v, float f) {
        const f32x2 f2 = pack2(f, f);
        v[0] = mul2(v[0], f2);
        v[1] = mul2(v[1], f2);
    };
    auto values_out = [&](f32x2 (*x)[2], float inv) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = vr + 32 * i;
            slice4(x[i], inv, v_s + j * 128 + (((vc >> 1) ^ (j & 7)) << 4) + (vc & 1) * 8, DR_BLK);
        }
    };
    constexpr uint32_t id128 = umma_idesc_f16(128, DR_RUN), id64 = umma_idesc_f16(128, DR_COLS, true);
    const uint64_t kd = umma_desc_k128(smem_u32(k_s)), vd = umma_desc_mn128(smem_u32(v_s), DR_BLK), sd = umma_desc_mn128(smem_u32(s_s), DR_BLK);
    unsigned ph = 0;
    bool ok = true;
    // the next run's operands are on their way while this one's last products run: queries to shared memory, keys and values in registers
    auto load_ab = [&](int base) {
        const float* ab = a.ab + ((size_t)(base + tid) * a.heads + h) * 2;
        return tid < DR_RUN && base + tid < t1 ? make_float2(ab[0], ab[1]) : make_float2(1.f, 0.f);
    };
    f32x2 kx[4 * DB][2], v0[4][2];
    float2 ab_x = load_ab(t0);
    stage_q(t0);
    load_k(kx, t0);
    load_v(v0, t0);
    if (carried) {
        state_top();
        state_out();
    }
    for (int base = t0; base < t1; base += DR_RUN) {
        const int n = min(DR_RUN, t1 - base);
        if (tid == 0) odd = n < DR_FEW || s_top >= DR_BIG_STATE;
        if (tid < DR_RUN) {
            const float d = ab_x.x;
            sa[tid] = d;
            sb[tid] = ab_x.y;
            // products of decays inside a block of 16, by halves of a warp
            Two p = {d, 0.f}, q = p;
#pragma unroll
            for (int o = 1; o < 16; o *= 2) {
                const Two up = shfl_up16(p, o), dn = shfl_down16(q, o);
                if ((lane & 15) >= o) p = mul(p, up);
                if ((lane & 15) + o < 16) q = mul(q, dn);
            }
            q = shfl_down16(q, 1);
            if ((tid & 15) == 15) {
                full[tid >> 4] = p;
                q = {1.f, 0.f};
            }
            pref[tid] = p;
            suff[tid] = q;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // ---- the largest numbers of rows and tiles
        unsigned bad = 0, k_top;
        const float* qr = q_stage + row * DR_LDQ + part * 32;
        {
            float t = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 f = *reinterpret_cast<const float4*>(qr + 4 * i);
                t = top3(top3(t, f.x, f.y), f.z, f.w);
            }
            unsigned m = abs_bits(t);
            qtop[part][row] = m;
            bad |= m >= DR_BIG_IN;
            m = abs_bits(top_of<8 * DB>(kx[0]));
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
            k_top = m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
            bad |= m >= DR_BIG_IN;
            if (kq == 0) kunit[kr] = slice_unit(min(m, DR_BIG_IN));
            bad |= abs_bits(top_of<8>(v0[0])) >= DR_BIG_IN;
#pragma unroll
            for (int i = 0; i < 4; ++i) scale_v(v0[i], sb[vr + 32 * i]);
            m = warp_umax(abs_bits(top_of<8>(v0[0])));
            bad |= m >= DR_BIG_IN;
            if (lane == 0) wtop[0][warp] = m;
            if (tid < DR_RUN) bad |= abs_bits(sa[tid]) > DR_DECAY;
            if (tid >= DR_THREADS - 64) {
                const int b = tid & 7, c = (tid >> 3) & 7;
                Two f[8], p = {1.f, 0.f};
#pragma unroll
                for (int i = 0; i < 8; ++i) f[i] = full[i];
#pragma unroll
                for (int i = 1; i < 7; ++i) p = mul(p, i > b && i < c ? f[i] : Two{1.f, 0.f});
                mid[b][c] = p;                           // between blocks b and c
                if (c == 7) tail[b] = b < 7 ? mul(p, f[7]) : p;
                if (b == 0) head[c] = c > 0 ? mul(f[0], p) : p;
                if (b == 0 && c == 7) head[8] = mul(mul(f[0], p), f[7]);
            }
        }
        if (bad) odd = 1;
        __syncthreads();
        if (odd) {
            // token by token: a thread's 16 columns of its channel, the read-out summed over the channels of a warp and then over the warps
            const float* kg = a.k + (size_t)base * a.ldk + (size_t)gh * a.dim;
            const float *qg = a.q + (size_t)base * a.ldq + (size_t)gh * a.dim, *vg = a.v + (size_t)base * a.ldv + (size_t)h * a.vd + j0;
            stage_q(base + DR_RUN);
            for (int t = 0; t < n; ++t) {
                {
                    const float kk = mine ? kg[(size_t)t * a.ldk + row] : 0.f, qq = mine ? qg[(size_t)t * a.ldq + row] : 0.f, da = sa[t], dbv = sb[t];
                    float o[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        if (mine && c0 + i < cols) st[i] = __fmaf_rn(da, st[i], dbv * vg[(size_t)t * a.ldv + c0 + i] * kk);
                        o[i] = mine ? st[i] * qq : 0.f;
                    }
                    // halving over the lanes: 16 columns in four steps, then one more; lane bits 4..1 name the column
#pragma unroll
                    for (int half = 8; half >= 1; half >>= 1) {
                        const bool up = (lane & (2 * half)) != 0;
#pragma unroll
                        for (int i = 0; i < half; ++i) {
                            const float give = up ? o[i] : o[i + half], keep = up ? o[i + half] : o[i];
                            o[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * half);
                        }
                    }
                    o[0] += __shfl_xor_sync(0xffffffffu, o[0], 1);
                    if ((lane & 1) == 0) red[warp & 3][c0 + (lane >> 1)] = o[0];
                }
                __syncthreads();
                if (tid < cols) a.o[(size_t)(base + t) * a.ldo + (size_t)h * a.vd + j0 + tid] = (red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid]);
                __syncthreads();
            }
            carried = true;
            state_top();
            state_out();
            ab_x = load_ab(base + DR_RUN);
            load_k(kx, base + DR_RUN);
            load_v(v0, base + DR_RUN);
            continue;
        }
        // ---- queries and keys as slices; the state waits in tensor memory meanwhile; what a token's value weighs in the state after the run, with its key's unit
        unsigned q_top = 0;
        {
            tmem_st16(lanes + DR_COL_ST + c0, reinterpret_cast<const uint32_t*>(st));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int j = vr + 32 * i;
                const Two p = mul(suff[j], tail[j >> 4]);
                scale_v(v0[i], p.h + p.l);
                scale_v(v0[i], kunit[j]);
            }
            const unsigned m = warp_umax(abs_bits(top_of<8>(v0[0])));
            if (lane == 0) wtop[1][warp] = m;
            if (tid < DR_RUN) ywk[tid] = (suff[tid].h + suff[tid].l) * kunit[tid];
            q_top = max(max(qtop[0][row], qtop[1][row]), max(qtop[2][row], qtop[3][row]));
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                f32x2 qx[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) *reinterpret_cast<ulonglong2*>(qx + 2 * i) = *reinterpret_cast<const ulonglong2*>(qr + 16 * x + 4 * i);
                slices_to_tmem<64>(qx, slice_inv(q_top), lanes + DR_COL_Q + part * 16 + 8 * x);
            }
            __syncthreads();                             // the queries have been read: the keys take their place
            hold<8 * DB>(kx[0]);
            const float k_inv = slice_inv(k_top);
#pragma unroll
            for (int i = 0; i < 4 * DB; ++i) {
                const int u = kq + 4 * i;                // units of four channels, two to 16 bytes of a slice
                slice4(kx[i], k_inv, k_s + (u >> 4) * DR_BLK + kr * 128 + (((u >> 1 & 7) ^ (kr & 7)) << 4) + (u & 1) * 8, DR_K);
            }
            tmem_st_wait();
        }
        fence_proxy_async();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        // ---- scores
        if (warp == DR_ISSUER) {
            if (elect_one()) {
                mma_rest<true, 4 * DB>(tmem + DR_COL_S, tmem + DR_COL_Q, kd, DR_K, id128);
                mma_ts<true, 4 * DB>(tmem + DR_COL_O, tmem + DR_COL_Q, kd, id128, true);
                umma_commit(&done[0]);
            }
            __syncwarp();
        }
        const unsigned v_top = all_top(wtop[0]), g_top = all_top(wtop[1]);
        f32x2 sc[16];
        {
            hold<8>(v0[0]);
            values_out(v0, slice_inv(g_top));
            // decays from token j to the row's, times the unit of key j: inside the row's own block
            if (part == (warp & 3)) {
                const int b0 = row & ~15;
                Two p = {1.f, 0.f};
#pragma unroll
                for (int e = 15; e >= 0; --e) {
                    const bool seen = e <= (row & 15);
                    near[row][e] = seen ? (p.h + p.l) * kunit[b0 + e] : 0.f;
                    const Two q = mul(p, {sa[b0 + e], 0.f});
                    p.h = seen ? q.h : p.h;
                    p.l = seen ? q.l : p.l;
                }
            }
            ok = mbar_sleep_limited(&done[0], ph, &dead);
            tc_fence_after();
            __syncwarp();
        }
        if (ok) {
            // times the decays, zero above the diagonal
            unsigned m = 0;
            const int bi = row >> 4;
            if (part <= (warp & 3)) {
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int b = part * 2 + x;
                    f32x2 s[8], u[8];
                    tmem_ld16_nowait(lanes + DR_COL_S + b * 16, reinterpret_cast<uint32_t*>(s));
                    tmem_ld16_nowait(lanes + DR_COL_O + b * 16, reinterpret_cast<uint32_t*>(u));
                    float f = b == bi ? 1.f : 0.f;
                    if (b < bi) {
                        const Two p = mul(pref[row], mid[b][bi]);
                        f = p.h + p.l;
                    }
                    const f32x2 f2 = pack2(f, f);
                    const float* y = b == bi ? near[row] : ywk + b * 16;
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(y + 2 * e);
                        sc[x * 8 + e] = mul2(add2(s[e], u[e]), mul2(w.x, f2));
                        sc[x * 8 + e + 1] = mul2(add2(s[e + 1], u[e + 1]), mul2(w.y, f2));
                    }
                }
                m = abs_bits(top_of<16>(sc));
            }
            ptop[part][row] = m;
        }
        fence_proxy_async();                             // the weighted values
        tc_fence_before();
        ok = __syncthreads_and(ok);                      // every score has been read
        tc_fence_after();
        if (!ok) break;
        // ---- what the state gives, in the scores' place; then what the run adds to it, in the queries' place
        if (warp == DR_ISSUER) {
            if (elect_one()) {
                if (carried) {
                    mma_rest<false, 4 * DB>(tmem + DR_COL_O + 64, tmem + DR_COL_Q, sd, DR_BLK, id64);
                    mma_ts<false, 4 * DB>(tmem + DR_COL_O, tmem + DR_COL_Q, sd, id64, true);
                }
                umma_commit(&done[1]);
            }
            __syncwarp();
            ok = mbar_sleep_limited(&done[1], ph, &dead);
            tc_fence_after();
            if (ok && elect_one()) {
                constexpr uint32_t idg = id64 | (1u << 15);  // the keys MN-major too
                const uint64_t kt = umma_desc_mn128(smem_u32(k_s), DR_BLK);
#pragma unroll
                for (int p = 0; p <= kSlicePairs; ++p) {
                    const bool last = p == kSlicePairs;
                    const uint64_t A = kt + (last ? 0 : slice_a(p)) * (DR_K >> 4), B = vd + (last ? 0 : slice_b(p)) * (DR_BLK >> 4);
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        umma_bf16(tmem + DR_COL_U + (last ? 0 : 64), A + k * (2048 >> 4), B + k * (2048 >> 4), idg, k > 0 || (p > 0 && !last));
                }
                umma_commit(&done[2]);
            }
            __syncwarp();
        }
        // ---- weights of the values as slices
        unsigned p_top = 0;
        float o[16];
        const float q_unit = slice_unit(q_top);
        {
            p_top = max(max(ptop[0][row], ptop[1][row]), max(ptop[2][row], ptop[3][row]));
            load_v(v0, base);
            tmem_ld16(lanes + DR_COL_ST + c0, st);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const uint32_t at = lanes + DR_COL_P + part * 16 + 8 * x;
                if (part <= (warp & 3)) {
                    slices_to_tmem<64>(sc + 8 * x, slice_inv(p_top), at);
                } else {
                    const uint32_t zero[8] = {};
#pragma unroll
                    for (int i = 0; i < 3; ++i) tmem_st8(at + 64 * i, zero);
                }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = 0.f;
            ok = mbar_sleep_limited(&done[1], ph, &dead) && ok;
            tc_fence_after();
            __syncwarp();
            if (carried && ok) {
                const Two p = mul(pref[row], head[row >> 4]);
                const float f = (p.h + p.l) * (q_unit * slice_unit(s_top));
                float y[16];
                tmem_ld16(lanes + DR_COL_O + c0, o);
                tmem_ld16(lanes + DR_COL_O + 64 + c0, y);
#pragma unroll
                for (int i = 0; i < 16; ++i) o[i] = (o[i] + y[i]) * f;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) scale_v(v0[i], sb[vr + 32 * i]);
            tmem_st_wait();
            ok = ok && mbar_sleep_limited(&done[2], ph, &dead);     // the weighted values and the keys have been read
            tc_fence_after();
            __syncwarp();
            if (ok) values_out(v0, slice_inv(v_top));
        }
        fence_proxy_async();
        tc_fence_before();
        ok = __syncthreads_and(ok);
        tc_fence_after();
        if (!ok) break;
        if (warp == DR_ISSUER) {
            if (elect_one()) {
                mma_rest<false, 8>(tmem + DR_COL_O + 64, tmem + DR_COL_P, vd, DR_BLK, id64);
                mma_ts<false, 8>(tmem + DR_COL_O, tmem + DR_COL_P, vd, id64, true);
                umma_commit(&done[3]);
            }
            __syncwarp();
        }
        stage_q(base + DR_RUN);
        // ---- the state meanwhile
        {
            const float f = head[8].h + head[8].l, g = slice_unit(g_top);
            float u[16], x[16];
            tmem_ld16(lanes + DR_COL_U + c0, u);
            tmem_ld16(lanes + DR_COL_U + 64 + c0, x);
#pragma unroll
            for (int i = 0; i < 16; ++i) st[i] = mine ? __fmaf_rn(f, st[i], (u[i] + x[i]) * g) : 0.f;
        }
        state_top();
        const float f_o = slice_unit(p_top) * (q_unit * slice_unit(v_top));
        if (base + DR_RUN < t1) state_out();
        carried = true;
        ok = mbar_sleep_limited(&done[3], ph, &dead);
        tc_fence_after();
        __syncwarp();
        if (ok) {
            float x[16], y[16];
            tmem_ld16(lanes + DR_COL_O + c0, x);
            tmem_ld16(lanes + DR_COL_O + 64 + c0, y);
#pragma unroll
            for (int i = 0; i < 16; i += 4)
                *reinterpret_cast<float4*>(o_stage + row * DR_LDO + c0 + i) =
                    make_float4(__fmaf_rn(x[i] + y[i], f_o, o[i]), __fmaf_rn(x[i + 1] + y[i + 1], f_o, o[i + 1]),
                                __fmaf_rn(x[i + 2] + y[i + 2], f_o, o[i + 2]), __fmaf_rn(x[i + 3] + y[i + 3], f_o, o[i + 3]));
        }
        tc_fence_before();
        ok = __syncthreads_and(ok);
        tc_fence_after();
        if (!ok) break;
        {                                                // whole rows, 16 lanes each
            const int c = (tid & 15) * 4;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = (tid >> 4) + 32 * i;
                float* dst = a.o + (size_t)(base + t) * a.ldo + (size_t)h * a.vd + j0 + c;
                const float4 x = *reinterpret_cast<const float4*>(o_stage + t * DR_LDO + c);
                if (t < n) {
                    if (o4) {
                        if (c < cols) *reinterpret_cast<float4*>(dst) = x;
                    } else {
                        if (c < cols) dst[0] = x.x;
                        if (c + 1 < cols) dst[1] = x.y;
                        if (c + 2 < cols) dst[2] = x.z;
                        if (c + 3 < cols) dst[3] = x.w;
                    }
                }
            }
        }
        ab_x = load_ab(base + DR_RUN);
        load_k(kx, base + DR_RUN);
        load_v(v0, base + DR_RUN);
        ph ^= 1;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!ok) {
        if (tid == 0 && err) *err = 1;
        for (int i = tid; i < (t1 - t0) * cols; i += DR_THREADS)
            a.o[(size_t)(t0 + i / cols) * a.ldo + (size_t)h * a.vd + j0 + i % cols] = __int_as_float(0x7fc00000);
    } else if (mine) {
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
            if (s4) {
                if (c0 + i < cols) *reinterpret_cast<float4*>(S + i) = make_float4(st[i], st[i + 1], st[i + 2], st[i + 3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) if (c0 + i + e < cols) S[i + e] = st[i + e];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <bool VEC, int DB>
int launch_runs(const RecurArgs& a, dim3 grid, cudaStream_t stream) {
    static PerDeviceFlag attr;
    if (!attr.done()) {
        FT_CHECK_CUDA(cudaFuncSetAttribute(decay_runs_kernel<VEC, DB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DR_SMEM));
        attr.mark();
    }
    decay_runs_kernel<VEC, DB><<<grid, DR_THREADS, DR_SMEM, stream>>>(a, a.err);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace

// A run of 128 tokens takes about 14 us whatever the sizes (one CTA per SM), after 5 us for the launch and the first operands; the kernel that
// goes token by token 0.275 us a token, and in proportion longer when more than about 175 of its CTAs of 64 columns run.  Mean portions of L
// tokens, us by tokens / here: 3 requests x 16 heads of 128 x 128, L = 32: 13 / 21, 67: 23 / 22, 683: 188 / 97; 16 requests, L = 64: 56 / 76,
// 128: 102 / 84; 3 x 64 heads of 128 x 64 (two waves of CTAs), 683: 280 / 213; 3 x 8 heads of 128 x 257, 683: 189 / 125.
bool decay_tc_ahead(const RecurArgs& a, int n_req, int T) {
    if (a.dim > 128 || n_req < 1 || n_req > 65535) return false;
    const double L = (double)T / n_req, ctas = (double)n_req * a.heads * ((a.vd + DR_COLS - 1) / DR_COLS), sms = device_sms();
    const double whole = (double)(int)(L / DR_RUN), runs = whole + (L - whole * DR_RUN >= DR_FEW ? 1.0 : 0.0);
    const double waves = (double)(long long)((ctas + sms - 1) / sms);
    return L >= 64 && waves * (5.0 + 14.0 * runs) < 0.275 * L * (ctas > 1.2 * sms ? ctas / (1.2 * sms) : 1.0);
}

int launch_decay_tc(const RecurArgs& a, int n_req, cudaStream_t stream) {
    FT_REQUIRE(a.dim <= 128 && n_req >= 1 && n_req <= 65535, "decay rule (tcgen05): %d channels, %d requests do not fit", a.dim, n_req);
    const dim3 grid((a.vd + DR_COLS - 1) / DR_COLS, a.heads, n_req);
    const bool vec = ((a.dim | a.vd | a.ldk | a.ldq | a.ldv) & 3) == 0 && (((uintptr_t)a.k | (uintptr_t)a.q | (uintptr_t)a.v) & 15) == 0;
    if (a.dim <= 64) return vec ? launch_runs<true, 1>(a, grid, stream) : launch_runs<false, 1>(a, grid, stream);
    return vec ? launch_runs<true, 2>(a, grid, stream) : launch_runs<false, 2>(a, grid, stream);
}

}  // namespace ft

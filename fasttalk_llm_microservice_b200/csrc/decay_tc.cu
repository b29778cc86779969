// The scalar-decay rule S <- a_t S + b_t k_t v_t^T, o_t = S^T q_t over prompt portions as matrix products, in fp32 accuracy (slices.cuh).
//
// The token-by-token kernel (branches.cu) is a serial chain: one warp per scheduler, 0.28 us a token whatever runs beside it.  Here a CTA
// (request, head, 64 value columns) takes 128 tokens at a time.  With W_ij = a_(j+1) .. a_i and S the state before the run:
//     o_i = sum_{j<=i} W_ij (q_i . k_j) b_j v_j  +  (a_0 .. a_i) S^T q_i          S <- (a_0 .. a_(n-1)) S + sum_j W_(n-1)j k_j (b_j v_j)^T
// Four products per run, 128 x 128 x D, 128 x 64 x D and twice 128 x 64 x 128, each as eight bf16 products: 11200 clocks of the tensor pipe.  A
// run takes 27000: forming the slices (some 10000 instruction slots per scheduler) and the barriers between the steps bound the kernel, then
// the 200 KB per run that an SM reads and writes.  The state stays on the chip (16 numbers per thread, fp32) from the first run to the last;
// decays are products of at most 128 numbers to 40 bits (never quotients or logarithms: a decay of zero is nothing special), and what a score or a state is
// multiplied by keeps those bits, so that each of them is rounded once.
// Three requests of 683 tokens: 16 heads of 128 x 128 188 -> 106 us.
// Error against 64 bits over 2048 tokens: results 1.1e-7 -> 6.0e-8, states 8.4e-8 -> 5.1e-8; by single elements beside numbers 2^30 as large it is that of fp32.
//
// Shared memory: slices of the keys | of the run's values (first weighted for the state, then for the results) | of the state.
// TMEM columns: the state 320..383 until the scores' slices need the place; queries' slices 0..191, after their last product what the run adds to the state 0..127; scores' second
// accumulator 192..319, their slices as an operand 192..383; scores' first accumulator 384..511, then the results (first | second accumulator).
//
// What a token's row does not depend on (later tokens, other columns) leaves no trace in it: masked products are zeros in every slice, and no number is formed in
// units of another.  Only whether its run goes token by token follows from the whole run.
//
// A run that holds infinities, NaN, numbers beyond 2^36 or decays beyond 1 by more than rounding, and runs of few tokens, go token by token: a product
// with a masked zero must not make a NaN of another token's infinity.  Every wait has a limit; a CTA whose wait runs out marks `err`, leaves NaN and ends.
#include "common.cuh"
#include "ft_internal.h"
#include "slices.cuh"

#include <algorithm>
#include <cmath>

namespace ft {
namespace {

constexpr int DR_RUN = 128, DR_WARPS = 16, DR_THREADS = DR_WARPS * 32, DR_COLS = 64;
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

// D = A[tmem] B[smem] over N steps of 16 along the contraction, the seven small products `rest` columns from first x first.  Slices of A are 64 columns apart, slices
// of B `plane` bytes; KMAJOR: B's blocks of 64 lie DR_BLK apart.  Everything but the addresses is known to the compiler: operands that are put together at
// run time cost the issuing thread 150 clocks a product, four times what the tensor cores take for it.
template <bool KMAJOR, int N>
__device__ __forceinline__ void mma_slices(uint32_t d, int rest, uint32_t a, uint64_t b, int plane, uint32_t idesc) {
#pragma unroll
    for (int p = 0; p <= kSlicePairs; ++p) {
        const bool last = p == kSlicePairs;
        const int sa = last ? 0 : slice_a(p), sb = last ? 0 : slice_b(p);
#pragma unroll
        for (int k = 0; k < N; ++k)
            umma_f16_ts(last ? d : d + rest, a + 64 * sa + k * 8,
                        b + sb * (plane >> 4) + (KMAJOR ? (k >> 2) * (DR_BLK >> 4) + (k & 3) * 2 : k * (2048 >> 4)), idesc, k > 0 || (p > 0 && !last));
    }
}

// Nothing is computed from x before this point: work moved up across barriers would need more registers than there are.
template <int N>
__device__ __forceinline__ void hold(f32x2* x) {
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+l"(x[i]));
}
template <bool VEC, int DB>
__global__ void __launch_bounds__(DR_THREADS, 1) decay_runs_kernel(RecurArgs a, int* err) {
    pdl_wait();
    extern __shared__ uint8_t dr_raw[];
    __shared__ Two pref[DR_RUN], suff[DR_RUN], full[8];      // products of decays inside a block of 16 tokens: up to and with i, behind j, all
    __shared__ Two mid[8][8], tail[8], head[9];          // of whole blocks: between two, behind one, before one (head[8]: of the run)
    __shared__ __align__(16) float behind[2][DR_RUN];    // a block's decays behind j, times b_j: h and l of a Two
    __shared__ __align__(16) float near[2][DR_RUN][20];  // decays inside a row's own block of 16, times b_j
    __shared__ float sa[DR_RUN], sb[DR_RUN];
    __shared__ float red[4][DR_COLS];
    __shared__ uint64_t done[4];
    __shared__ uint32_t tmem_slot;
    __shared__ int odd, state_big;                       // 1: the run, or the one behind this state, goes token by token
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
        state_big = 0;
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
    // the state's slices to shared memory, [channel][64 columns]
    auto state_out = [&]() {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 16; i += 2) t = top3(t, st[i], st[i + 1]);
        if (abs_bits(t) >= DR_BIG_STATE) state_big = 1;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            f32x2 v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = pack2(st[x * 8 + 2 * e], st[x * 8 + 2 * e + 1]);
            slice8(v, s_s + row * 128 + (((part * 2 + x) ^ (row & 7)) << 4), DR_BLK);
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
    auto values_out = [&](f32x2 (*x)[2]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int j = vr + 32 * i;
            slice4(x[i], v_s + j * 128 + (((vc >> 1) ^ (j & 7)) << 4) + (vc & 1) * 8, DR_BLK);
        }
    };
    constexpr uint32_t id128 = slice_idesc(128, DR_RUN), id64 = slice_idesc(128, DR_COLS, true);
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
    if (carried) state_out();
    __syncthreads();
    for (int base = t0; base < t1; base += DR_RUN) {
        const int n = min(DR_RUN, t1 - base);
        if (tid == 0) odd = n < DR_FEW || state_big;
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
        // ---- numbers that do not go as slices
        bool bad = false;
        const float* qr = q_stage + row * DR_LDQ + part * 32;
        {
            if (tid == 0) state_big = 0;
            float t = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 f = *reinterpret_cast<const float4*>(qr + 4 * i);
                t = top3(top3(t, f.x, f.y), f.z, f.w);
            }
            bad = abs_bits(top_of<8>(v0[0], top_of<8 * DB>(kx[0], t))) >= DR_BIG_IN;
            if (tid < DR_RUN) bad |= abs_bits(sa[tid]) > DR_DECAY || abs_bits(sb[tid]) >= DR_BIG_IN;
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
            state_out();
            __syncthreads();
            ab_x = load_ab(base + DR_RUN);
            load_k(kx, base + DR_RUN);
            load_v(v0, base + DR_RUN);
            continue;
        }
        // ---- queries and keys as slices; the state waits in tensor memory meanwhile; what a token's value weighs in the state after the run
        {
            tmem_st16(lanes + DR_COL_ST + c0, reinterpret_cast<const uint32_t*>(st));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int j = vr + 32 * i;
                const Two p = mul(mul(suff[j], tail[j >> 4]), {sb[j], 0.f});
                scale_v(v0[i], p.h + p.l);
            }
            if (tid < DR_RUN) {
                const Two p = mul(suff[tid], {sb[tid], 0.f});
                behind[0][tid] = p.h;
                behind[1][tid] = p.l;
            }
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                f32x2 qx[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) *reinterpret_cast<ulonglong2*>(qx + 2 * i) = *reinterpret_cast<const ulonglong2*>(qr + 16 * x + 4 * i);
                slices_to_tmem<64>(qx, lanes + DR_COL_Q + part * 16 + 8 * x);
            }
            __syncthreads();                             // the queries have been read: the keys take their place
            hold<8 * DB>(kx[0]);
#pragma unroll
            for (int i = 0; i < 4 * DB; ++i) {
                const int u = kq + 4 * i;                // units of four channels, two to 16 bytes of a slice
                slice4(kx[i], k_s + (u >> 4) * DR_BLK + kr * 128 + (((u >> 1 & 7) ^ (kr & 7)) << 4) + (u & 1) * 8, DR_K);
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
                mma_slices<true, 4 * DB>(tmem + DR_COL_O, DR_COL_S - DR_COL_O, tmem + DR_COL_Q, kd, DR_K, id128);
                umma_commit(&done[0]);
            }
            __syncwarp();
        }
        f32x2 sc[16];
        {
            hold<8>(v0[0]);
            values_out(v0);
            // what token j's values weigh in the row's result but for the score, inside the row's own block
            if (part == (warp & 3)) {
                const int b0 = row & ~15;
                Two p = {1.f, 0.f};
#pragma unroll
                for (int e = 15; e >= 0; --e) {
                    const bool seen = e <= (row & 15);
                    const Two w = mul(p, {sb[b0 + e], 0.f});
                    near[0][row][e] = seen ? w.h : 0.f;
                    near[1][row][e] = seen ? w.l : 0.f;
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
            // times the decays and b, zero above the diagonal
            const int bi = row >> 4;
            if (part <= (warp & 3)) {
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int b = part * 2 + x;
                    f32x2 s[8], u[8];
                    tmem_ld16_nowait(lanes + DR_COL_S + b * 16, reinterpret_cast<uint32_t*>(s));
                    tmem_ld16_nowait(lanes + DR_COL_O + b * 16, reinterpret_cast<uint32_t*>(u));
                    Two f = {b == bi ? 1.f : 0.f, 0.f};
                    if (b < bi) f = mul(pref[row], mid[b][bi]);
                    const f32x2 fh = pack2(f.h, f.h), fl = pack2(f.l, f.l), minus = pack2(-1.f, -1.f);
                    const float *yh = b == bi ? near[0][row] : behind[0] + b * 16, *yl = b == bi ? near[1][row] : behind[1] + b * 16;
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        const ulonglong2 h = *reinterpret_cast<const ulonglong2*>(yh + 2 * e), l = *reinterpret_cast<const ulonglong2*>(yl + 2 * e);
                        // (u + rest) (wh + wl), rounded once
                        auto weighted = [&](f32x2 u, f32x2 s, f32x2 h, f32x2 l) {
                            const f32x2 wh = mul2(h, fh), wl = fma2(l, fh, fma2(h, fl, fma2(h, fh, mul2(wh, minus))));
                            return fma2(u, wh, fma2(u, wl, mul2(rest_of(u, s), wh)));
                        };
                        sc[x * 8 + e] = weighted(u[e], s[e], h.x, l.x);
                        sc[x * 8 + e + 1] = weighted(u[e + 1], s[e + 1], h.y, l.y);
                    }
                }
            }
        }
        fence_proxy_async();                             // the weighted values
        tc_fence_before();
        ok = __syncthreads_and(ok);                      // every score has been read
        tc_fence_after();
        if (!ok) break;
        // ---- what the state gives, in the scores' place; then what the run adds to it, in the queries' place
        if (warp == DR_ISSUER) {
            if (elect_one()) {
                if (carried) mma_slices<false, 4 * DB>(tmem + DR_COL_O, 64, tmem + DR_COL_Q, sd, DR_BLK, id64);
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
        float o[16];
        {
            load_v(v0, base);
            tmem_ld16(lanes + DR_COL_ST + c0, st);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const uint32_t at = lanes + DR_COL_P + part * 16 + 8 * x;
                if (part <= (warp & 3)) {
                    slices_to_tmem<64>(sc + 8 * x, at);
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
                float y[16];
                tmem_ld16(lanes + DR_COL_O + c0, o);
                tmem_ld16(lanes + DR_COL_O + 64 + c0, y);
#pragma unroll
                for (int i = 0; i < 16; ++i) o[i] = __fmaf_rn(o[i], p.h, __fmaf_rn(o[i], p.l, rest_of(o[i], y[i]) * p.h));
            }
            tmem_st_wait();
            ok = ok && mbar_sleep_limited(&done[2], ph, &dead);     // the weighted values and the keys have been read
            tc_fence_after();
            __syncwarp();
            if (ok) values_out(v0);
        }
        fence_proxy_async();
        tc_fence_before();
        ok = __syncthreads_and(ok);
        tc_fence_after();
        if (!ok) break;
        if (warp == DR_ISSUER) {
            if (elect_one()) {
                mma_slices<false, 8>(tmem + DR_COL_O, 64, tmem + DR_COL_P, vd, DR_BLK, id64);
                umma_commit(&done[3]);
            }
            __syncwarp();
        }
        stage_q(base + DR_RUN);
        // ---- the state meanwhile
        {
            const Two f = head[8];
            float u[16], x[16];
            tmem_ld16(lanes + DR_COL_U + c0, u);
            tmem_ld16(lanes + DR_COL_U + 64 + c0, x);
#pragma unroll
            for (int i = 0; i < 16; ++i) st[i] = mine ? __fmaf_rn(f.h, st[i], __fmaf_rn(f.l, st[i], rest_of(u[i], x[i]))) + u[i] : 0.f;
        }
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
                    make_float4(x[i] + (rest_of(x[i], y[i]) + o[i]), x[i + 1] + (rest_of(x[i + 1], y[i + 1]) + o[i + 1]),
                                x[i + 2] + (rest_of(x[i + 2], y[i + 2]) + o[i + 2]), x[i + 3] + (rest_of(x[i + 3], y[i + 3]) + o[i + 3]));
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
    launch_after(decay_runs_kernel<VEC, DB>, grid, DR_THREADS, DR_SMEM, stream, a, a.err);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace

static bool vectors(const RecurArgs& a) {
    return ((a.dim | a.vd | a.ldk | a.ldq | a.ldv) & 3) == 0 && (((uintptr_t)a.k | (uintptr_t)a.q | (uintptr_t)a.v) & 15) == 0;
}
// Both kernels' times in us from 1500 pairs of measurements (1 to 64 heads, 20 x 70 to 128 x 257, 1 to 40 portions of 17 to 1500 tokens; a mean of 7 % off).
// This one: rounds of CTAs, one per SM, of 4.5 us and 16.2 a run of 128 tokens (12.6 up to 64 channels), up to an eighth more when all SMs read, a fifth more off 16
// bytes; the last tokens of a portion take as long as a run from a dozen on.  Token by token: 4 us and per token 0.17 us with up to 30 CTAs, 0.0012 us more with each further
// one (of 64 columns, or 128 up to 64 channels).  By tokens / here, portions of L tokens: one of 16 heads of 128 x 128, L = 64: 15 / 20, 128: 26 / 20, 150: 30 / 35, 256: 48 /
// 36, 1500: 262 / 192; three, 683: 189 / 103; 40 of them (nine rounds), 100: 175 / 204, 128: 216 / 209, 150: 252 / 345; 16 of 64 heads of 128 x 64, 128: 173 / 175, 200: 263 /
// 289; eight heads of 128 x 257, 128: 26 / 27, 200: 38 / 44, 1024: 179 / 166.  Shorter portions than 64 never gained.
bool decay_tc_ahead(const RecurArgs& a, int n_req, int T) {
    if (a.dim > 128 || n_req < 1 || n_req > 65535) return false;
    const double L = (double)T / n_req, sms = device_sms();
    if (L < 64) return false;
    const double heads = (double)n_req * a.heads, ctas = heads * ((a.vd + DR_COLS - 1) / DR_COLS), token_ctas = heads * (a.dim <= 64 ? (a.vd + 127) / 128 : (a.vd + 63) / 64);
    const double whole = (double)(int)(L / DR_RUN), runs = whole + std::min(1.0, (L - whole * DR_RUN) / 12);
    const double run = (a.dim <= 64 ? 12.6 : 16.2) * (vectors(a) ? 1.0 : 1.2) * (1.0 + 0.13 * std::min(1.0, ctas / sms));
    const double here = std::ceil(ctas / sms) * (4.5 + run * runs), by_tokens = 4.0 + L * std::max(0.17, 0.13 + 0.0012 * token_ctas);
    return here < 0.9 * by_tokens;
}

int launch_decay_tc(const RecurArgs& a, int n_req, cudaStream_t stream) {
    FT_REQUIRE(a.dim <= 128 && n_req >= 1 && n_req <= 65535, "decay rule (tcgen05): %d channels, %d requests do not fit", a.dim, n_req);
    const dim3 grid((a.vd + DR_COLS - 1) / DR_COLS, a.heads, n_req);
    const bool vec = vectors(a);
    if (a.dim <= 64) return vec ? launch_runs<true, 1>(a, grid, stream) : launch_runs<false, 1>(a, grid, stream);
    return vec ? launch_runs<true, 2>(a, grid, stream) : launch_runs<false, 2>(a, grid, stream);
}

}  // namespace ft

// K6 on tcgen05 / TMEM — causal chunked-prefill attention over the paged KV cache (head_dim 64 or 128, GQA group of 3 or 4).
//
// One CTA = one (request, 64-query tile, KV head): the tile's 64 tokens x the G q heads of the group are 64 G query rows, handled as two
// halves of 32 tokens (row = token * G + head; 128 rows, of which a group of 3 leaves 32 unused), so that every K/V tile that reaches shared
// memory feeds both (the mma.sync kernel re-fetched each tile per q head).  Up to 32 tokens that see four key tiles or more are one half only: both
// halves then take the same queries and every other key tile each, and their results are put together at the end.  Per KV tile of 64 keys and per half:
//
//   S  = Q K^T   tcgen05.mma  M128 N64 K=D   A = Q half (TMA 3-D box -> 128-byte-swizzled rows in smem),
//                                           B = the K slab exactly as it lies in the cache: [64 keys][64 d] fp16
//                                           with chunk ^ (row & 7) IS the K-major SWIZZLE_128B operand layout
//   softmax      4 warps, one thread per row: tcgen05.ld of the row's 64 scores, running max / sum in fp32,
//                exp2, P -> fp16 -> TENSOR MEMORY (tcgen05.st, row = lane: the A operand of the next product)
//   O += P V     tcgen05.mma  M128 N=D K64   B = the V slab as it lies in the cache: [64 keys][64 d] is the
//                                           MN-major SWIZZLE_128B layout (d contiguous, 8-key groups 1 KB apart)
//
// S (two buffers per half, so the scores of tile j + 1 are ready before the softmax of tile j ends) and O live in TMEM, P over the first half of
// the scores that it came from (S 4 x 64 columns, O 2 x D).  O is rescaled lazily: the row maximum used for scaling only moves when
// the running maximum exceeds it by more than 2^8 (P stays far inside fp16 range, the accumulation is fp32, the
// final normalisation uses the same reference — exact arithmetic, not an approximation), so the TMEM round trip
// of a rescale happens on the first tiles only.  The two halves ping-pong: while the softmax warps of one half
// work on their scores, the tensor core runs the other half's products.
//
// Warp roles (320 threads): warp 0 = TMA producer (Q once, then a ring of K|V tiles of 16 KB (D = 64) or 32 KB, one bulk copy each),
// warp 1 = TMEM owner + MMA issuer (one elected thread), warps 2..5 = softmax / epilogue of half 0, warps 6..9 of
// half 1 (warp w may touch TMEM lanes 32 * (w % 4) .. +31), one thread per query row.
//
// What bounds it (in-kernel clock64 timelines, and this kernel with single parts left out): the hand-overs of a tile, load scores - maximum -
// exponentials - store P - products - next scores, each a few hundred clocks of latency; 2100 clk per 64-key tile where the
// exponentials alone take 1024 (the SFU's 16 / clk / SM) and the products 640 (d = 64) or 1280 (d = 128).  Without its
// exponentials, or with a quarter of its products, it is no more than 15 % faster.  Tried and not kept (four prompts of 2k / 211
// tokens over 5000, 1B / 8B shapes, us; 147 / 174 at that point): two threads per row 155 / 172 before the order below, one
// persistent CTA per SM with 128-key tiles at d = 64 and an issuing warp per half 163 / 175, the same with the halves'
// exponentials in turns 153 / 183 and with two threads per row 172 / 176, pages prefetched into L2 165 / 190.
// What helped: the longest tiles first over all KV heads (163 -> 149; the last round of CTAs was 15 % of the time), and keys shared by the halves where
// the queries fill one only (17 tokens over 5000 keys 74 -> 36 at d = 64, 79 -> 51 at d = 128; six requests of 211 174 -> 145).
#include "common.cuh"
#include "ft_internal.h"

#include <algorithm>
#include <mutex>
#include <vector>

namespace ft {

constexpr int TC_THREADS = 320;
constexpr int TC_ROWS = 128;                 // rows per half (UMMA M); 32 tokens x G heads of them are real
constexpr int TC_TOK = 64;                   // query tokens per CTA
constexpr int TC_SUB_BYTES = kKvTile * 128;  // one [64 tokens][64 dims] fp16 sub-slab = 8 KB; also 64 rows of a Q block
constexpr int TC_QBLK_BYTES = TC_ROWS * 128; // one 128-row x 64-dim block of Q = 16 KB
constexpr int TC_GRID_Y = 65535;             // query tiles of one launch
constexpr int TC_SPLIT_TILES = 4;            // key tiles from which a tile of few queries shares them between the halves
constexpr float TC_RESCALE_THRESHOLD = 8.f;  // log2 units

template <int D>
struct TcCfg {
    static constexpr int KH = D / 64;                                   // 64-dim blocks of the head
    static constexpr int TILE_BYTES = 2 * KH * TC_SUB_BYTES;             // K slab + V slab: 16 KB (d 64) / 32 KB (d 128)
    static constexpr int STAGES = D == 64 ? 6 : 4;
    static constexpr int Q_BYTES = 2 * KH * TC_QBLK_BYTES;               // both halves
    static constexpr size_t SMEM = 1024 + Q_BYTES + (size_t)STAGES * TILE_BYTES + 512;      // (d = 128: the largest that leaves 60 KB of L1; beyond it every launch takes 1 us longer)
    // TMEM columns: S, two buffers per half, 64 fp32 columns each; P (fp16, 32 columns) is written over the first half
    // of the S buffer it was computed from; O of the two halves behind them
    static constexpr int COL_S = 0, COL_O = 256, COLS = 512;
    static_assert(256 + 2 * D <= 512, "tensor memory");
};

// 3-D tiled tensor-map copy (d, head, token) -> shared memory
__device__ __forceinline__ void tma_tile_3d(void* dst_smem, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
            smem_u32(dst_smem)),
        "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
__device__ __forceinline__ void mbar_wait_sleep(uint64_t* bar, uint32_t parity) {
    while (!mbar_try_wait(bar, parity)) __nanosleep(20);
}

// FEW: the list has tiles whose keys the halves share.  A kernel of its own for the lists without one: the second way in the same kernel costs every CTA 0.1 to
// 0.25 us, also those that don't take it (64 requests of 30 tokens behind 100, 32 heads of 64 / 128: 27.2 / 36.3 us, without it 26.6 / 35.1; 16 of
// 64 behind 100 9.1 / 13.1, 8.9 / 12.6), and in there one copy of the rescale loop, which is rare, leaves its instructions for the rest (six of 211 behind 5000, in the
// caller's order 151 / 172 -> 138 / 168).
template <int D, int G, bool FEW>
__global__ void __launch_bounds__(TC_THREADS, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const uint8_t* __restrict__ kv_layer,
                       const int* __restrict__ page_table, int max_pages, const int* __restrict__ req_q_start,
                       const int* __restrict__ req_slot, const int* __restrict__ req_pos0,
                       const int* __restrict__ tile_req, const int* __restrict__ tile_q0,
                       __nv_bfloat16* __restrict__ out, __nv_bfloat16* __restrict__ out_lo, int nq, int nkv,
                       float scale_log2, int stagger_on) {
    using C = TcCfg<D>;
    constexpr int KH = C::KH;
    constexpr int R = 32 * G;                                 // real rows of a half (row = token * G + head)
    // the LAST tiles of the list see the most keys where it is in that order: back to front, all KV heads of a tile side by side, or the
    // longest CTAs would start last and the grid end in a long tail
    const int tile_idx = (int)gridDim.y - 1 - (int)blockIdx.y;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* q_s = smem;                                     // [2 halves][KH dim blocks][128 rows][128 B]
    uint8_t* kv_s = smem + C::Q_BYTES;                       // [STAGES][K: KH sub-slabs | V: KH sub-slabs]
    uint64_t* bars = reinterpret_cast<uint64_t*>(kv_s + (size_t)C::STAGES * C::TILE_BYTES);
    uint64_t* kv_full = bars;                                // [STAGES]
    uint64_t* kv_empty = kv_full + C::STAGES;                // [STAGES]
    uint64_t* q_full = kv_empty + C::STAGES;                 // [1]
    uint64_t* s_full = q_full + 1;                           // [2][2] scores of half h, buffer j & 1, are in TMEM
    uint64_t* p_full = s_full + 4;                           // [2][2] probabilities of half h, tile parity j & 1, are in TMEM
    uint64_t* pv_done = p_full + 4;                          // [2][2] O += P V of half h, tile parity j & 1, retired
    uint64_t* stagger = pv_done + 4;                         // [1] half 0 knows its first row maxima: half 1 may start
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(stagger + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&map_q);
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(&kv_full[s], 1);
            mbar_init(&kv_empty[s], 1);
        }
        mbar_init(q_full, 1);
        mbar_init(stagger, TC_ROWS / 32);
        for (int h = 0; h < 2; ++h) {
            mbar_init(&s_full[2 * h], 1);
            mbar_init(&s_full[2 * h + 1], 1);
            mbar_init(&p_full[2 * h], TC_ROWS / 32);         // one arrival per softmax warp
            mbar_init(&p_full[2 * h + 1], TC_ROWS / 32);
            mbar_init(&pv_done[2 * h], 1);
            mbar_init(&pv_done[2 * h + 1], 1);
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, C::COLS);
        tmem_relinquish();
    }
    if (R < TC_ROWS && warp >= 2) {
        // a GQA group of 3 fills 96 of a half's 128 rows: the other 32 rows of every Q block are zeroed so that their
        // (never stored) scores are finite.  Generic-proxy stores, made visible to the tensor core before the barrier.
        for (int i = threadIdx.x - 64; i < 2 * KH * (TC_ROWS - R) * 8; i += TC_THREADS - 64) {
            const int blk = i / ((TC_ROWS - R) * 8), rem = i % ((TC_ROWS - R) * 8);
            *reinterpret_cast<uint4*>(q_s + (size_t)blk * TC_QBLK_BYTES + (R + rem / 8) * 128 + (rem % 8) * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_proxy_async();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    pdl_launch_dependents();

    const int req = tile_req[tile_idx];
    const int q0 = tile_q0[tile_idx];
    const int q_row0 = req_q_start[req];
    const int q_len = req_q_start[req + 1] - q_row0;
    const int pos0 = req_pos0[req];
    const int kvh = blockIdx.x;
    const int rows_here = q_len - q0 < TC_TOK ? q_len - q0 : TC_TOK;
    const int last_pos = pos0 + q0 + rows_here - 1;
    const int n_tiles = last_pos / kKvTile + 1;
    // Up to 32 tokens would leave the second half idle: both take the same queries then, every other tile of keys each (tile j: half j & 1), and their
    // results are put together at the end (about a microsecond).
    const bool split = FEW && rows_here <= TC_TOK / 2 && n_tiles >= TC_SPLIT_TILES;
    const int* pt = page_table + (size_t)req_slot[req] * max_pages;

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) {
            mbar_expect_tx(q_full, (split ? 1 : 2) * KH * R * 128);
            for (int h = 0; h < (split ? 1 : 2); ++h)
                for (int kh = 0; kh < KH; ++kh)
                    tma_tile_3d(q_s + (size_t)(h * KH + kh) * TC_QBLK_BYTES, &map_q, kh * 64, kvh * G, q_row0 + q0 + 32 * h, q_full);
        }
        const uint64_t pol = policy_evict_last();            // re-read by the other KV heads' CTAs / later q tiles
        int stage = 0;
        uint32_t phase = 0;
        for (int t0 = 0; t0 < n_tiles; t0 += 32) {
            const int mine = t0 + lane;
            const int my_page = mine < n_tiles ? pt[mine] : 0;
            const int n = n_tiles - t0 < 32 ? n_tiles - t0 : 32;
            for (int i = 0; i < n; ++i) {
                const int page = __shfl_sync(0xffffffffu, my_page, i);
                if (lane == 0) {
                    mbar_wait_sleep(&kv_empty[stage], phase ^ 1);
                    mbar_expect_tx(&kv_full[stage], C::TILE_BYTES);
                    tma_bulk_g2s(kv_s + (size_t)stage * C::TILE_BYTES,
                                 kv_layer + ((size_t)page * nkv + kvh) * C::TILE_BYTES, C::TILE_BYTES, &kv_full[stage], pol);
                }
                if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc_qk = umma_idesc_f16(TC_ROWS, kKvTile, false);
            constexpr uint32_t idesc_pv = umma_idesc_f16(TC_ROWS, D, true);
            const uint32_t q_addr = smem_u32(q_s);
            auto issue_qk = [&](int h, int buf, uint32_t k_addr, int qh) {
#pragma unroll
                for (int kh = 0; kh < KH; ++kh) {
                    const uint64_t a = umma_desc_k128(q_addr + (qh * KH + kh) * TC_QBLK_BYTES);
                    const uint64_t b = umma_desc_k128(k_addr + kh * TC_SUB_BYTES);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16(tmem_base + C::COL_S + (2 * h + buf) * 64, a + 2 * k, b + 2 * k, idesc_qk, (kh | k) != 0);
                }
                umma_commit(&s_full[2 * h + buf]);
            };
            auto issue_pv = [&](int h, int buf, uint32_t v_addr, bool first) {
                const uint32_t p_tmem = tmem_base + C::COL_S + (2 * h + buf) * 64;    // 64 fp16 = 32 columns, over S
#pragma unroll
                for (int k = 0; k < kKvTile / 16; ++k)
                    umma_f16_ts(tmem_base + C::COL_O + h * D, p_tmem + 8 * k, umma_desc_mn128(v_addr + k * 2048), idesc_pv, k != 0 || !first);
                umma_commit(&pv_done[2 * h + buf]);
            };
            auto stage_of = [&](int j) { return j % C::STAGES; };
            auto k_addr_of = [&](int j) { return smem_u32(kv_s + (size_t)stage_of(j) * C::TILE_BYTES); };
            auto keys_here = [&](int j) {
                mbar_wait(&kv_full[stage_of(j)], (j / C::STAGES) & 1);
                tc_fence_after();
            };
            mbar_wait(q_full, 0);
            if (split) {
                // Scores run AHEAD tiles of the list ahead: three where the ring is deep enough that their keys set out three tiles ago, else two (the half's next
                // tile).  The product that read P out of their buffer was issued one or two tiles ago.  (Tile j is its half's (j / 2)-th and the
                // (j / 4)-th in its buffer.)
                constexpr int AHEAD = C::STAGES >= 6 ? 3 : 2;
#pragma unroll 1
                for (int j = -AHEAD; j < n_tiles; ++j) {
                    if (j >= 0) {
                        mbar_wait(&p_full[2 * (j & 1) + (j >> 1 & 1)], (j >> 2) & 1);
                        tc_fence_after();
                        issue_pv(j & 1, j >> 1 & 1, k_addr_of(j) + KH * TC_SUB_BYTES, j < 2);
                        umma_commit(&kv_empty[stage_of(j)]);
                    }
                    const int a = j + AHEAD;
                    if (a < n_tiles) {
                        keys_here(a);
                        issue_qk(a & 1, a >> 1 & 1, k_addr_of(a), 0);
                    }
                }
            } else {
                // scores run two tiles ahead of the softmax (two S buffers per half): tile j + 2 is issued as soon as the
                // product of tile j — which reads its P out of the same buffer — has been issued in front of it
                for (int j = 0; j < 2 && j < n_tiles; ++j) {
                    keys_here(j);
                    issue_qk(0, j & 1, k_addr_of(j), 0);
                    if (!stagger_on) issue_qk(1, j & 1, k_addr_of(j), 1);
                }
                if (stagger_on) {        // half 1 starts when half 0 is about to enter its SFU-bound phase, so that the two halves'
                                         // exponentials do not fall on the SFU at the same time (profiles/r02_attn_prefill_tc.md)
                    mbar_wait(stagger, 0);
                    for (int j = 0; j < 2 && j < n_tiles; ++j) issue_qk(1, j & 1, k_addr_of(j), 1);
                }
                for (int j = 0; j < n_tiles; ++j) {
                    for (int h = 0; h < 2; ++h) {
                        // Every hand-over has one barrier PER BUFFER (tile parity): the softmax of one half may run up to two
                        // tiles ahead of what this thread has observed (it is busy with the other half), and a single barrier
                        // completing two phases unobserved would look "not yet complete" again — a deadlock.
                        mbar_wait(&p_full[2 * h + (j & 1)], (j >> 1) & 1);   // P_h(j) written, S_h(j) consumed, O_h rescaled if needed
                        tc_fence_after();
                        issue_pv(h, j & 1, k_addr_of(j) + KH * TC_SUB_BYTES, j == 0);
                        if (h == 1) umma_commit(&kv_empty[stage_of(j)]);   // every product that reads this stage has been issued
                        if (j + 2 < n_tiles) {
                            if (h == 0) keys_here(j + 2);
                            issue_qk(h, j & 1, k_addr_of(j + 2), h);      // in order behind the product that read P out of this buffer
                        }
                    }
                }
            }
        }
    } else {
        // ---------------------------------------------------------------- softmax + epilogue (one thread per row)
        const int h = (warp - 2) >> 2;
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;                     // TMEM lane == row of the half
        const int tok = (split ? 0 : h * 32) + row / G;          // query token within the CTA's 64
        const int head = kvh * G + row % G;
        const int pos = pos0 + q0 + tok;                         // absolute position of this row's query
        const bool valid = row < R && q0 + tok < q_len;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const uint32_t s_taddr0 = lane_base + C::COL_S + 2 * h * 64, o_taddr = lane_base + C::COL_O + h * D;
        float m_ref = -INFINITY, l_run = 0.f;                    // m_ref in scaled (log2) units
        const int mine = split ? (n_tiles - h + 1) / 2 : n_tiles;
        for (int i = 0; i < mine; ++i) {
            const int j = split ? h + 2 * i : i;                 // tile of the list, the half's i-th
            mbar_wait(&s_full[2 * h + (i & 1)], (i >> 1) & 1);
            tc_fence_after();
            const uint32_t s_taddr = s_taddr0 + (i & 1) * 64;
            uint32_t sr[64];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld16_nowait(s_taddr + 16 * c, sr + 16 * c);
            tmem_ld_wait();
            float t4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};      // four chains instead of one of 64
            if (j * kKvTile + kKvTile - 1 > pos) {               // diagonal tile: causal mask
#pragma unroll
                for (int c = 0; c < 64; ++c) {
                    float v = __uint_as_float(sr[c]);
                    v = j * kKvTile + c <= pos ? v : -INFINITY;
                    sr[c] = __float_as_uint(v);
                    t4[c & 3] = fmaxf(t4[c & 3], v);
                }
            } else {
#pragma unroll
                for (int c = 0; c < 64; ++c) t4[c & 3] = fmaxf(t4[c & 3], __uint_as_float(sr[c]));
            }
            const float tmax = fmaxf(fmaxf(t4[0], t4[1]), fmaxf(t4[2], t4[3]));
            if (stagger_on && i == 0 && h == 0) {
                __syncwarp();
                if (lane == 0) mbar_arrive(stagger);
            }
            const float m_new = fmaxf(m_ref, tmax * scale_log2);
            // rows without a query of this request say nothing: a row's rounding depends on its own request alone
            const bool grow = valid && m_new > m_ref + TC_RESCALE_THRESHOLD;
            if (i == 0) {
                m_ref = m_new;
            } else if (__any_sync(0xffffffffu, grow)) {          // tcgen05.ld / st are warp-wide: rescale all 32 rows
                mbar_wait(&pv_done[2 * h + ((i - 1) & 1)], ((i - 1) >> 1) & 1);     // O_h complete up to the half's tile i - 1
                tc_fence_after();
                const float alpha = m_new == -INFINITY ? 1.f : exp2f(m_ref - m_new);        // rows that did not grow: m_new >= m_ref, alpha <= 1
                l_run *= alpha;
                m_ref = m_new;
#pragma unroll(FEW ? 1 : D / 16)
                for (int c = 0; c < D / 16; ++c) {
                    uint32_t orr[16];
                    tmem_ld16_nowait(o_taddr + 16 * c, orr);
                    tmem_ld_wait();
#pragma unroll
                    for (int k = 0; k < 16; ++k) orr[k] = __float_as_uint(__uint_as_float(orr[k]) * alpha);
                    tmem_st16(o_taddr + 16 * c, orr);
                }
                tmem_st_wait();
            }
            const float mu = m_ref == -INFINITY ? 0.f : m_ref;
            float ps[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c16 = 0; c16 < 2; ++c16) {                  // 32 keys -> 16 packed columns per store
                uint32_t pk[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float p0 = ex2_fast(fmaf(__uint_as_float(sr[c16 * 32 + 2 * e]), scale_log2, -mu));
                    const float p1 = ex2_fast(fmaf(__uint_as_float(sr[c16 * 32 + 2 * e + 1]), scale_log2, -mu));
                    ps[(2 * e) & 3] += p0;
                    ps[(2 * e + 1) & 3] += p1;
                    __half2 t = __floats2half2_rn(p0, p1);
                    pk[e] = *reinterpret_cast<uint32_t*>(&t);
                }
                tmem_st16(s_taddr + 16 * c16, pk);               // P over the scores it came from (this row has read them)
            }
            tmem_st_wait();
            l_run += (ps[0] + ps[1]) + (ps[2] + ps[3]);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[2 * h + (i & 1)]);
        }
        // ---- epilogue: O / l -> bf16 hi + lo planes
        mbar_wait(&pv_done[2 * h + ((mine - 1) & 1)], ((mine - 1) >> 1) & 1);
        tc_fence_after();
        float inv = 1.f / l_run, inv_other = 0.f;
        if (split) {                                             // each half forms half of the channels' results
            // maximum and sum by way of the scores' columns, which have all been read
            uint32_t ml[16] = {__float_as_uint(m_ref), __float_as_uint(l_run)};
            tmem_st16(s_taddr0, ml);
            tmem_st_wait();
            tc_fence_before();
            asm volatile("bar.sync 1, 256;" ::: "memory");
            tc_fence_after();
            tmem_ld16_nowait(lane_base + C::COL_S + 2 * (1 - h) * 64, ml);
            tmem_ld_wait();
            const float2 o = make_float2(__uint_as_float(ml[0]), __uint_as_float(ml[1]));
            const float m = fmaxf(m_ref, o.x), w = m_ref == -INFINITY ? 0.f : exp2f(m_ref - m), wo = o.x == -INFINITY ? 0.f : exp2f(o.x - m);
            const float r = 1.f / (h == 0 ? l_run * w + o.y * wo : o.y * wo + l_run * w);
            inv = w * r;
            inv_other = wo * r;
        }
        const size_t off = ((size_t)(q_row0 + q0 + tok) * nq + head) * D;
        auto put = [&](int c, const uint32_t* v) {               // 16 channels of the row
            uint32_t hi[8], lo[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float x = __uint_as_float(v[2 * k]), y = __uint_as_float(v[2 * k + 1]);
                hi[k] = pack_bf16(x, y);
                lo[k] = pack_bf16(x - bf16_lo(hi[k]), y - bf16_hi(hi[k]));
            }
            uint4* dst = reinterpret_cast<uint4*>(out + off + 16 * c);
            dst[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            dst[1] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
            if (out_lo) {
                uint4* dl = reinterpret_cast<uint4*>(out_lo + off + 16 * c);
                dl[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                dl[1] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
            }
        };
        if (!split) {
#pragma unroll
            for (int c = 0; c < D / 16; ++c) {
                uint32_t orr[16];
                tmem_ld16_nowait(o_taddr + 16 * c, orr);
                tmem_ld_wait();
                if (valid) {
#pragma unroll
                    for (int k = 0; k < 16; ++k) orr[k] = __float_as_uint(__uint_as_float(orr[k]) * inv);
                    put(c, orr);
                }
            }
        } else {
#pragma unroll 1
            for (int i = 0; i < D / 32; ++i) {
                const int c = D / 32 * h + i;
                uint32_t orr[16], x[16];
                tmem_ld16_nowait(o_taddr + 16 * c, orr);
                tmem_ld16_nowait(lane_base + C::COL_O + (1 - h) * D + 16 * c, x);
                tmem_ld_wait();
                if (valid) {
#pragma unroll
                    for (int k = 0; k < 16; ++k) orr[k] = __float_as_uint(fmaf(__uint_as_float(x[k]), inv_other, __uint_as_float(orr[k]) * inv));
                    put(c, orr);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::COLS);
    }
}

// ------------------------------------------------------------------ host side
bool attn_prefill_tc_supported(int nq, int nkv, int d) {
    static const bool off = getenv("FT_ATTN_PREFILL_MMA_SYNC") != nullptr;        // A/B switch (scripts/, tests)
    return !off && (d == 64 || d == 128) && nkv >= 1 && (nq == 4 * nkv || nq == 3 * nkv);
}

// The kernel takes its list back to front over all KV heads at once, so tiles that take longest belong at its end, or they start last and the grid ends in a
// long tail.  Tiles of a request side by side share its pages, though, so only differences that count are sorted by: an eighth of what
// an SM does in all, and four key tiles at least (us, 24 / 32 query heads of 128: in the caller's order, sorted by every key tile, this way; twelve requests of
// 500 tokens 70 / 75, 74 / 82, 71 / 77; four of 2048 174 / 186, 170 / 181, 170 / 179; six of 211 behind 5000 170 / 172, 142 / 144, 142 / 145; 128 of 100 behind 100
// 153 / 164, 159 / 170, 153 / 164).  The mma.sync kernel takes any list front to back, head by head; it stays as it is (sorted: six requests
// of 17 to 2048 tokens, 8 heads of 64, 85 -> 91 us).
bool order_query_tiles(const int* q_start, const int* pos0, int* tile_req, int* tile_q0, int n_tiles, int nq, int nkv, int d, int q_rows) {
    if (q_rows <= 0 || !attn_prefill_tc_supported(nq, nkv, d)) return false;
    struct Tile { long long work; int req, q0; };
    std::vector<Tile> t(n_tiles);
    long long all = 0;
    bool few = false;
    for (int i = 0; i < n_tiles; ++i) {
        const int r = tile_req[i], q0 = tile_q0[i], left = q_start[r + 1] - q_start[r] - q0, rows = std::min(left, TC_TOK);
        const int keys = (pos0[r] + q0 + rows - 1) / kKvTile + 1;
        const bool shared = rows <= TC_TOK / 2 && keys >= TC_SPLIT_TILES;                  // by the halves: half as many
        t[i] = {(shared ? (keys + 1) / 2 + 1 : keys) + 5, r, q0};                          // start and end of a CTA: five key tiles' time
        all += t[i].work;
        few |= shared;
    }
    const long long width = std::max(4LL, all * nkv / device_sms() / 8);
    std::stable_sort(t.begin(), t.end(), [&](const Tile& a, const Tile& b) { return a.work / width < b.work / width; });
    for (int i = 0; i < n_tiles; ++i) {
        tile_req[i] = t[i].req;
        tile_q0[i] = t[i].q0;
    }
    return few;
}

// q tensor maps are cached per (device, pointer, rows, heads, head_dim, group): the engine's q buffer never moves
struct QMapEntry { int dev; const void* q; int rows, nq, d, g; CUtensorMap map; };
static std::mutex g_qmap_mu;
static QMapEntry g_qmaps[16];
static int g_qmap_n = 0, g_qmap_next = 0;

template <int D, int G, bool FEW>
static int launch_tc(const CUtensorMap& map, const void* kv_layer, const int* page_table, int max_pages,
                     const int* req_q_start, const int* req_slot, const int* req_pos0, const int* tile_req,
                     const int* tile_q0, int n_tiles, void* out, void* out_lo, int nq, int nkv, bool pdl, cudaStream_t stream) {
    using C = TcCfg<D>;
    static PerDeviceFlag attr_set;
    if (!attr_set.done()) {
        FT_CHECK_CUDA(cudaFuncSetAttribute(attn_prefill_tc_kernel<D, G, FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
        attr_set.mark();
    }
    const float scale_log2 = 1.4426950408889634f / sqrtf((float)D);
    static const int stagger_on = getenv("FT_TC_STAGGER") ? atoi(getenv("FT_TC_STAGGER")) : 1;       // A/B switch; measured: 4–6 % at d = 64
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    for (int left = n_tiles; left > 0;) {                        // the end of the list first
        const int n = std::min(left, TC_GRID_Y);
        left -= n;
        cfg.gridDim = dim3(nkv, n);
        FT_CHECK_CUDA(cudaLaunchKernelEx(&cfg, attn_prefill_tc_kernel<D, G, FEW>, map, (const uint8_t*)kv_layer, page_table, max_pages,
                                         req_q_start, req_slot, req_pos0, tile_req + left, tile_q0 + left, (__nv_bfloat16*)out,
                                         (__nv_bfloat16*)out_lo, nq, nkv, scale_log2, stagger_on));
    }
    return 0;
}

int launch_attn_prefill_tc(const void* q, int q_rows, const void* kv_layer, const int* page_table, int max_pages,
                           const int* req_q_start, const int* req_slot, const int* req_pos0, const int* tile_req,
                           const int* tile_q0, int n_tiles, void* out, void* out_lo, int nq, int nkv, int d, bool few, bool pdl,
                           cudaStream_t stream) {
    FT_REQUIRE(q_rows >= 1, "attn_prefill (tcgen05): the q buffer's row count is needed for its tensor map");
    const int g = nq / nkv;
    CUtensorMap map;
    {
        std::lock_guard<std::mutex> lk(g_qmap_mu);
        const int dev = current_device_slot();
        const QMapEntry* hit = nullptr;
        for (int i = 0; i < g_qmap_n; ++i)
            if (g_qmaps[i].dev == dev && g_qmaps[i].q == q && g_qmaps[i].rows == q_rows && g_qmaps[i].nq == nq &&
                g_qmaps[i].d == d && g_qmaps[i].g == g)
                hit = &g_qmaps[i];
        if (!hit) {
            QMapEntry e{dev, q, q_rows, nq, d, g, {}};
            if (int r = make_tmap_f16_3d(&e.map, q, d, nq, q_rows, 64, g, 32)) return r;
            g_qmaps[g_qmap_next] = e;
            hit = &g_qmaps[g_qmap_next];
            g_qmap_next = (g_qmap_next + 1) % 16;
            if (g_qmap_n < 16) ++g_qmap_n;
        }
        map = hit->map;
    }
#define FT_TC_CASE(D_, G_)                                                                                               \
    if (d == D_ && g == G_)                                                                                              \
        return (few ? launch_tc<D_, G_, true> : launch_tc<D_, G_, false>)(map, kv_layer, page_table, max_pages,          \
                                                                          req_q_start, req_slot, req_pos0, tile_req,     \
                                                                          tile_q0, n_tiles, out, out_lo, nq, nkv, pdl, stream);
    FT_TC_CASE(64, 4)
    FT_TC_CASE(64, 3)
    FT_TC_CASE(128, 4)
    FT_TC_CASE(128, 3)
#undef FT_TC_CASE
    FT_REQUIRE(false, "attn_prefill (tcgen05): head_dim %d with a GQA group of %d is not built", d, g);
}

}  // namespace ft

// Plain projections on tcgen05: out[t][n] = sum_k (hi + lo)[t][k] W[n][k] in fp32, no fused layer step — every projection of the
// layered models, and ft_gemm_bf16 / ft_gemm_fused with unsplit fp32 results.  Operands as in gemm.cu (W rows are the UMMA A operand,
// the activation's two bf16 planes the B operand, fp32 accumulators in TMEM); two kernels:
//
//   many tokens   CTA pairs (cta_group::2) that walk units of 256 weight rows x `bn` tokens, two accumulators, as gemm_pair_kernel
//                 does, with a token tile whose width is a run-time value.  A projection of 2313 tokens and 2048 rows is 152 units of
//                 128 tokens for 74 pairs: three rounds, the last one nearly empty; 160 tokens wide it is 120 units in two.  The
//                 width that the launcher takes is the one with the least time over all rounds (plain_token_tile).
//                 Measured (2313 tokens, hi + lo, one CTA per tile before): 2048 -> 2048 45 -> 40 us, 2048 -> 10752 182 -> 143 us.
//   few tokens    up to 128, where few_tokens() says so: one token tile; K is shared by the up to eight CTAs of a cluster, which
//                 add their partial tiles through distributed shared memory in rank order: no slabs, no arrival words, no second launch.  Bound by latency (launch, first load,
//                 one pass over a few chunks), and per chunk by the tensor core's reads of the weight tile, which both planes share
//                 (16 tokens, 2048 x 2048: one CTA per 128 rows 13.1 us, K shared by eight 6.6, one product for both planes 5.9).
#include "common.cuh"
#include "ft_internal.h"

namespace ft {
namespace {

constexpr int PL_BM = 128, PL_BK = 64, PL_A = PL_BM * PL_BK * 2;      // weight rows per CTA, K chunk, bytes of a weight tile
constexpr int PL_THREADS = 320;                                       // many tokens: TMA warp, MMA warp, eight epilogue warps
constexpr int PL_MAX_STAGES = 8;

// ------------------------------------------------------------------ many tokens
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PL_THREADS, 1)
gemm_plain_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_hi,
                       const __grid_constant__ CUtensorMap map_lo, float* __restrict__ out, int n_out, int T, int k_chunks, int stages, int bn) {
    extern __shared__ uint8_t pl_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pl_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t full[PL_MAX_STAGES], empty[PL_MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    const int plane = bn / 2 * PL_BK * 2;                 // bytes of this CTA's half of one plane's tile
    const int stage_bytes = PL_A + 2 * plane;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank();
    const int row_pairs = (n_out / PL_BM + 1) / 2;        // the last pair's second tile may lie beyond the matrix: zero rows, not stored
    const int units = row_pairs * ((T + bn - 1) / bn);
    const int cl = (int)cluster_id_x(), n_cl = (int)gridDim.x / 2;
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&map_w);
        tma_prefetch_desc(&map_hi);
        tma_prefetch_desc(&map_lo);
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 2);                  // both CTAs' epilogues, on the leader's copy
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(&tmem_slot, 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_wait();
    if (warp == 0) {
        if (elect_one()) {
            // weights are read again by every token tile; a launch of one token tile streams them
            const bool multi = T > bn;
            const uint64_t pol_w = multi ? policy_evict_last() : policy_evict_first(), pol_x = multi ? policy_evict_first() : policy_evict_last();
            int it = 0;
            for (int u = cl; u < units; u += n_cl) {
                const int row0 = (2 * (u % row_pairs) + rank) * PL_BM, tok0 = u / row_pairs * bn + rank * (bn / 2);
                for (int i = 0; i < k_chunks; ++i, ++it) {
                    const int s = it % stages;
                    if (it >= stages) mbar_wait(&empty[s], ((it / stages) - 1) & 1);
                    if (rank == 0) mbar_expect_tx(&full[s], 2 * stage_bytes);
                    uint8_t* st = smem + (size_t)s * stage_bytes;
                    tma_tile_2d_pair(st, &map_w, i * PL_BK, row0, &full[s], pol_w);
                    tma_tile_2d_pair(st + PL_A, &map_hi, i * PL_BK, tok0, &full[s], pol_x);
                    tma_tile_2d_pair(st + PL_A + plane, &map_lo, i * PL_BK, tok0, &full[s], pol_x);
                }
            }
        }
    } else if (warp == 1 && rank == 0) {
        if (elect_one()) {
            const uint32_t idesc = umma_idesc_bf16(2 * PL_BM, bn);
            int it = 0;
            uint32_t use = 0;
            for (int u = cl; u < units; u += n_cl, ++use) {
                const uint32_t acc = use & 1;
                if (use >= 2) {
                    mbar_wait(&acc_empty[acc], ((use >> 1) - 1) & 1);
                    tc_fence_after();
                }
                const uint32_t d = tmem + acc * 256;
                for (int i = 0; i < k_chunks; ++i, ++it) {
                    const int s = it % stages;
                    mbar_wait(&full[s], (it / stages) & 1);
                    tc_fence_after();
                    const uint32_t base = smem_u32(smem + (size_t)s * stage_bytes);
                    const uint64_t wd = umma_desc_k128(base), hd = umma_desc_k128(base + PL_A), ld = umma_desc_k128(base + PL_A + plane);
#pragma unroll
                    for (int k = 0; k < PL_BK / 16; ++k) umma_bf16_pair(d, wd + 2 * k, hd + 2 * k, idesc, (i | k) != 0);
#pragma unroll
                    for (int k = 0; k < PL_BK / 16; ++k) umma_bf16_pair(d, wd + 2 * k, ld + 2 * k, idesc, 1u);
                    umma_commit_pair(&empty[s]);
                }
                umma_commit_pair(&acc_full[acc]);
            }
        }
    } else if (warp >= 2) {
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        uint32_t use = 0;
        for (int u = cl; u < units; u += n_cl, ++use) {
            const uint32_t acc = use & 1;
            const int row0 = (2 * (u % row_pairs) + rank) * PL_BM, tok0 = u / row_pairs * bn;
            const int n_tok = min(bn, T - tok0);
            mbar_wait(&acc_full[acc], (use >> 1) & 1);
            tc_fence_after();
            if (row0 < n_out) {
                float* p = out + (size_t)tok0 * n_out + row0 + quarter * 32 + lane;
                for (int c = 16 * half; c < n_tok; c += 32) {      // a row per lane: 128 consecutive bytes per warp and token
                    float v[16];
                    tmem_ld16(tmem + acc * 256 + ((uint32_t)(quarter * 32) << 16) + c, v);
                    float* q = p + (size_t)c * n_out;
                    if (c + 16 <= n_tok) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) q[(size_t)j * n_out] = v[j];
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (c + j < n_tok) q[(size_t)j * n_out] = v[j];
                    }
                }
            }
            tc_fence_before();
            asm volatile("bar.sync 2, 256;" ::: "memory");      // all eight warps have read the accumulator
            if (threadIdx.x == 64) mbar_arrive_leader(&acc_empty[acc]);
        }
    }
    tc_fence_before();
    cluster_sync_all();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem, 512);
    }
}

// ------------------------------------------------------------------ few tokens
constexpr int PF_THREADS = 192;                           // TMA warp, MMA warp, four epilogue warps

// grid (row tiles, S), clusters of (1, S): CTA (x, s) takes the s-th share of K of weight rows 128 x .. 128 x + 127.
template <int BN>
__global__ void __launch_bounds__(PF_THREADS)
gemm_plain_few_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_hi,
                      const __grid_constant__ CUtensorMap map_lo, float* __restrict__ out, int n_out, int T, int k_chunks, int stages) {
    constexpr int PLANE = BN * PL_BK * 2, STAGE = PL_A + 2 * PLANE;
    constexpr uint32_t COLS = 2 * BN;                     // the hi plane's products, then the lo plane's
    extern __shared__ uint8_t pf_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pf_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t full[PL_MAX_STAGES], empty[PL_MAX_STAGES], acc_full;
    __shared__ uint32_t tmem_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = (int)gridDim.y, rank = blockIdx.y, row0 = blockIdx.x * PL_BM;
    const int kc0 = k_chunks * rank / S, n_iter = k_chunks * (rank + 1) / S - kc0;      // at least one chunk each
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&map_w);
        tma_prefetch_desc(&map_hi);
        tma_prefetch_desc(&map_lo);
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&acc_full, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(&tmem_slot, COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_wait();
    if (warp == 0) {
        if (elect_one()) {
            const uint64_t pol_w = policy_evict_first(), pol_x = policy_evict_last();
            const int pre = min(n_iter, stages);
            for (int i = 0; i < pre; ++i) {               // the weights first: they come from memory, the activations out of L2
                mbar_expect_tx(&full[i], STAGE);
                tma_tile_2d(smem + (size_t)i * STAGE, &map_w, (kc0 + i) * PL_BK, row0, &full[i], pol_w);
            }
            for (int i = 0; i < n_iter; ++i) {
                const int s = i % stages;
                uint8_t* st = smem + (size_t)s * STAGE;
                if (i >= pre) {
                    mbar_wait(&empty[s], ((i / stages) - 1) & 1);
                    mbar_expect_tx(&full[s], STAGE);
                    tma_tile_2d(st, &map_w, (kc0 + i) * PL_BK, row0, &full[s], pol_w);
                }
                tma_tile_2d(st + PL_A, &map_hi, (kc0 + i) * PL_BK, 0, &full[s], pol_x);
                tma_tile_2d(st + PL_A + PLANE, &map_lo, (kc0 + i) * PL_BK, 0, &full[s], pol_x);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            // the two planes' tiles lie one after the other: ONE operand of 2 BN rows, so the weight tile is read once for both
            constexpr uint32_t idesc = umma_idesc_bf16(PL_BM, 2 * BN);
            for (int i = 0; i < n_iter; ++i) {
                const int s = i % stages;
                mbar_wait(&full[s], (i / stages) & 1);
                tc_fence_after();
                const uint32_t base = smem_u32(smem + (size_t)s * STAGE);
                const uint64_t wd = umma_desc_k128(base), xd = umma_desc_k128(base + PL_A);
#pragma unroll
                for (int k = 0; k < PL_BK / 16; ++k) umma_bf16(tmem, wd + 2 * k, xd + 2 * k, idesc, (i | k) != 0);
                umma_commit(&empty[s]);
            }
            umma_commit(&acc_full);
        }
    } else {
        mbar_wait(&acc_full, 0);
        tc_fence_after();
        const int quarter = warp & 3, f = quarter * 32 + lane;
        float* tile = reinterpret_cast<float*>(smem);     // [BN][128]: the stages are idle once the products have retired
#pragma unroll 1
        for (int c = 0; c < BN && c < T; c += 16) {
            float v[16], low[16];
            tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + c, v);
            tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + BN + c, low);
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] += low[j];
            if (S == 1) {
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (c + j < T) out[(size_t)(c + j) * n_out + row0 + f] = v[j];
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) tile[(c + j) * PL_BM + f] = v[j];
            }
        }
    }
    tc_fence_before();
    __syncthreads();                                      // the columns have been read; this CTA's share lies in its shared memory
    if (S > 1) cluster_arrive();
    if (warp == 1) {
        // Before the wait: a CTA that waits for the others holds no columns.  With them it could keep one of another stream's kernel
        // from its columns, and that one a CTA of this cluster on another SM.
        tc_fence_after();
        tmem_dealloc(tmem, COLS);
    }
    if (S > 1) {
        cluster_wait();                                   // every share of the row tile is there
        if (warp >= 2) {
            // This CTA adds every S-th token's shares, in rank order: a warp a token, four weight rows a lane, all of a token's reads of the cluster's
            // memory on their way at once (one row a thread, eight reads: 64 tokens of 1024 x 1024 with S = 8 7.1 us, so
            // 6.3; of 8192 x 2048 with S = 2 12.4 and 11.8; 16 tokens of 2048 x 2048 level).
            const float* mine = reinterpret_cast<const float*>(smem) + 4 * lane;      // (the same place in every CTA)
            float* dst = out + row0 + 4 * lane;
            const bool out16 = ((uintptr_t)out & 15) == 0;       // (n_out is a multiple of 128)
            uint32_t from[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) from[q] = peer_addr(mine, q & (S - 1));
            auto add = [&](auto SHARES, auto TOKENS) {
                constexpr int n = SHARES.value, m = TOKENS.value;      // m tokens' reads at a time
                for (int t0 = rank + n * (warp - 2); t0 < T; t0 += 4 * n * m) {
                    float4 v[m][n];
#pragma unroll
                    for (int i = 0; i < m; ++i)
#pragma unroll
                        for (int q = 0; q < n; ++q)
                            if (t0 + 4 * n * i < T) v[i][q] = peer_ld4_at(from[q] + (uint32_t)(t0 + 4 * n * i) * (PL_BM * 4));
#pragma unroll
                    for (int i = 0; i < m; ++i) {
                        if (t0 + 4 * n * i >= T) break;
                        float4 sum = v[i][0];
#pragma unroll
                        for (int q = 1; q < n; ++q) {
                            sum.x += v[i][q].x;
                            sum.y += v[i][q].y;
                            sum.z += v[i][q].z;
                            sum.w += v[i][q].w;
                        }
                        float* to = dst + (size_t)(t0 + 4 * n * i) * n_out;
                        if (out16) {
                            store_f4(to, sum);
                        } else {
                            to[0] = sum.x; to[1] = sum.y; to[2] = sum.z; to[3] = sum.w;
                        }
                    }
                }
            };
            if (S == 8) add(Int<8>{}, Int<1>{});
            else if (S == 4) add(Int<4>{}, Int<2>{});
            else add(Int<2>{}, Int<4>{});
        }
        cluster_sync_all();                               // nobody leaves while its tile is being read
    }
}

constexpr int PL_RING = 222 * 1024;                       // shared memory for the stages (+ 1 KB to align them)

// CTAs that share a row tile's K: as many as leave each three chunks and the grid one CTA per SM, from four CTAs per tile on nearly two
// (10752 x 2048 and 64 tokens: 14.7 us with S = 1, 17.2 with 2; 296 CTAs in clusters of four do not all find a place within their GPCs at
// once: 9472 x 3072, 64 tokens, 24.4 us, 15.3 in 148).  Where K is short the sharing costs what it saves: up to 512 columns none (64 tokens
// of 4096 x 512: 6.4 us, 10.2 with S = 2 and one token at a time), and up to 1984 fewer CTAs for more than 32 tokens, whose shares take
// longer to add (24 tokens of 8192 x 1024: 8.0 us with S = 4, 8.3 with 1; 64 tokens: 10.3 and 9.7; 3072 x 1024: 8.3 and 8.9).
int few_shares(int tiles, int kc, int T) {
    if (kc <= 8) return 1;
    const int sms = device_sms();
    auto most = [&](int S) { return kc < 32 && T > 32 ? (S == 8 ? 192 : S == 4 ? 136 : 80) : S >= 4 ? (T > 32 ? 14 : 15) * sms / 8 : sms; };
    int S = 8;
    while (S > 1 && (kc / S < 3 || tiles * S > most(S))) S /= 2;
    return S;
}
// Up to 128 tokens on the few-token kernel, or (more than 48) on CTA pairs.  The few-token kernel wins where K can be shared: 64 tokens
// and 4096 x 2048 10.3 against 12.5 us, 128 tokens and 2048 x 8192 21.1 against 37.  From 65 tokens on its token tile is as wide as the
// pairs' and adding the shares takes longer than they save, unless K is long or the row tiles are few (128 tokens: 8192 x 1024 15.3 against
// 9.7 us, 12288 x 4096 30.7 against 25.1, but 3072 x 3072 14.7 against 18.7).  Unshared, with a short K or on more than half of the SMs,
// pairs are ahead from 49 tokens on (64 tokens: 4096 x 512 7.1 against 6.4, 16384 x 2048 15.8 against 14.7).
bool few_tokens(int tiles, int kc, int T, int S) {
    if (T <= 48) return true;
    if (T <= 64) return S > 1 || (kc > 8 && 2 * tiles <= device_sms());
    return T <= 128 && S >= 4 && (kc >= 48 || (kc >= 32 && tiles <= (T <= 80 ? 32 : 16)));
}

template <int BN>
int launch_few(const CUtensorMap& mw, const CUtensorMap& mh, const CUtensorMap& ml, float* out, int n_out, int T, int K, int S, cudaStream_t stream) {
    constexpr int STAGE = PL_A + 2 * BN * PL_BK * 2;
    const int kc = K / PL_BK, tiles = n_out / PL_BM;
    // A deep ring where a CTA has an SM for itself, half of one otherwise.  Clusters of four or eight always leave room for a second CTA:
    // they must lie within one GPC, and with one CTA per SM sixteen clusters of eight do not all find one (2048 x 4096, 16 tokens:
    // 12.9 us with 160 KB per CTA, more than with half the CTAs).
    const int budget = tiles * S <= device_sms() && S <= 2 ? 200 * 1024 : 104 * 1024;
    int stages = budget / STAGE;
    if (stages > PL_MAX_STAGES) stages = PL_MAX_STAGES;
    if (stages > (kc + S - 1) / S) stages = (kc + S - 1) / S;
    if (stages < 1) stages = 1;
    size_t smem = (size_t)stages * STAGE;
    if (smem < (size_t)BN * PL_BM * 4) smem = (size_t)BN * PL_BM * 4;      // the partial tile
    smem += 1024;
    static PerDeviceFlag attr_set;
    if (!attr_set.done()) {
        FT_CHECK_CUDA(cudaFuncSetAttribute(gemm_plain_few_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, 201 * 1024));
        FT_CHECK_CUDA(cudaFuncSetAttribute(gemm_plain_few_kernel<BN>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        attr_set.mark();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles, S);
    cfg.blockDim = dim3(PF_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = S; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    FT_CHECK_CUDA(cudaLaunchKernelEx(&cfg, gemm_plain_few_kernel<BN>, mw, mh, ml, out, n_out, T, kc, stages));
    return 0;
}

// Pairs that can be resident at once.
int plain_clusters() {
    static int n_dev[kMaxDevices] = {};
    int& n = n_dev[current_device_slot()];
    if (!n) {
        FT_CHECK_CUDA(cudaFuncSetAttribute(gemm_plain_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PL_RING + 1024));
        cudaLaunchConfig_t q = {};
        q.gridDim = dim3(device_sms() & ~1);
        q.blockDim = dim3(PL_THREADS);
        q.dynamicSmemBytes = PL_RING + 1024;
        cudaLaunchAttribute qa[1];
        qa[0].id = cudaLaunchAttributeClusterDimension;
        qa[0].val.clusterDim.x = 2; qa[0].val.clusterDim.y = 1; qa[0].val.clusterDim.z = 1;
        q.attrs = qa;
        q.numAttrs = 1;
        int v = 0;
        if (cudaOccupancyMaxActiveClusters(&v, gemm_plain_pair_kernel, &q) != cudaSuccess || v <= 0) v = device_sms() / 2;
        n = v;
    }
    return n;
}

// Tokens per tile.  A round of units takes as long as its tile is wide, but not less than the weight tiles need to come out of L2
// (92 + bn / 3 tokens' time), and the last round's results leave after its products.  The constants are fitted to 2313 tokens of
// 2048 columns (us per round of K = 2048): 10.0 / 11.5 / 12.5 / 12.9 / 16.2 / 19.9 / 24.8 for 32 / 64 / 96 / 128 / 160 / 192 / 256 tokens.
// Multiples of 32: the widths a 256-row product has, and half of one, a CTA's share, is then whole 8-row swizzle groups.
int plain_token_tile(int row_pairs, int T, int clusters) {
    int best = 128;
    double least = 1e30;
    for (int bn = 32; bn <= 256; bn += 32) {
        const long long units = (long long)row_pairs * ((T + bn - 1) / bn), rounds = (units + clusters - 1) / clusters;
        const double round = bn > 92 + bn / 3.0 ? bn : 92 + bn / 3.0, t = rounds * round + 0.25 * bn;
        if (t < least) { least = t; best = bn; }
    }
    return best;
}

}  // namespace

int launch_gemm_plain(const void* w, const void* hi, const void* lo, float* out, int n_out, int T, int K, cudaStream_t stream) {
    FT_REQUIRE(w && hi && lo && out && n_out >= PL_BM && n_out % PL_BM == 0 && K >= PL_BK && K % PL_BK == 0 && T >= 1,
               "gemm (plain): bad sizes or operands (n_out %d, T %d, K %d)", n_out, T, K);
    CUtensorMap mw, mh, ml;
    if (int r = make_tmap_bf16_k64(&mw, w, n_out, K, PL_BM)) return r;
    const int S = few_shares(n_out / PL_BM, K / PL_BK, T);
    if (few_tokens(n_out / PL_BM, K / PL_BK, T, S)) {
        const int bn = gemm_pick_bn(T, true);
        if (int r = make_tmap_bf16_k64(&mh, hi, T, K, bn)) return r;
        if (int r = make_tmap_bf16_k64(&ml, lo, T, K, bn)) return r;
        switch (bn) {
            case 16: return launch_few<16>(mw, mh, ml, out, n_out, T, K, S, stream);
            case 32: return launch_few<32>(mw, mh, ml, out, n_out, T, K, S, stream);
            case 64: return launch_few<64>(mw, mh, ml, out, n_out, T, K, S, stream);
            default: return launch_few<128>(mw, mh, ml, out, n_out, T, K, S, stream);
        }
    }
    const int clusters = plain_clusters();
    if (clusters <= 0) return clusters;
    const int row_pairs = (n_out / PL_BM + 1) / 2, bn = plain_token_tile(row_pairs, T, clusters);
    if (int r = make_tmap_bf16_k64(&mh, hi, T, K, bn / 2)) return r;
    if (int r = make_tmap_bf16_k64(&ml, lo, T, K, bn / 2)) return r;
    const int units = row_pairs * ((T + bn - 1) / bn), stage = PL_A + bn * PL_BK * 2;
    int stages = PL_RING / stage;
    if (stages > PL_MAX_STAGES) stages = PL_MAX_STAGES;
    // the whole ring's memory, also where the stages take less: a pair's CTA holds all columns while it waits for its partner, so no
    // other kernel with columns of its own may have room beside it
    launch_after(gemm_plain_pair_kernel, 2 * (units < clusters ? units : clusters), PL_THREADS, PL_RING + 1024, stream, mw, mh, ml, out, n_out, T, K / PL_BK, stages, bn);
    FT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace ft

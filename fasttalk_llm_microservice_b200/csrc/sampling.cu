// K7 — fused temperature / top-k / top-p / argmax sampling over fp32 logits [B, V].
//
// One cluster of up to eight CTAs per sequence, each with one contiguous share of the row.  Greedy (temperature <= 0) is an
// argmax with lowest-index tie-break (torch.argmax semantics).  Otherwise every CTA keeps the weights e_i = exp((x_i - max)/T) of
// its share in shared memory, so the row is read from memory once, and the kept set is found WITHOUT sorting: a radix select over
// the (monotone) bit pattern of e_i finds first the k-th largest value (counts), then the nucleus threshold (masses), in at most
// three passes of 11 / 11 / 9 bits each — a pass ends the search as soon as its bin holds one element.  Histograms are whole
// numbers: a bin's mass is count * (smallest value of the bin) + (sum of the elements' offsets in it) * (their unit), which the
// native integer atomics of shared memory add up exactly and in any order, where adding the floats themselves would loop on
// compare-and-swap and depend on the order.  CTA r of the cluster sums bins [r, r + 1) * 2048 / C over the cluster's histograms.
// The draw walks the kept set in index order.
//
// What bounds it: a chain of short passes over data in shared memory and of cluster barriers (3 per radix pass).  One CTA per row
// with every pass reading the row again took 153 us for one row of 128256 and 203 us for 64 (greedy and sampled rows mixed); the
// cluster took 28 and 69 us on the device with a pass of its own for every step, and takes 19 and 50 with the first histogram filled
// where the weights are formed, two additions an element, a bin's reads from the other CTAs spread over all warps, and walks whose
// sums are one addition a step.
#include "common.cuh"
#include "ft_internal.h"

namespace ft {

constexpr int SAMPLE_THREADS = 512;
constexpr int SAMPLE_WARPS = SAMPLE_THREADS / 32;
constexpr int SAMPLE_BINS = 2048, SAMPLE_GROUPS = SAMPLE_BINS / 64;
constexpr int SAMPLE_MAX_CTAS = 8;          // portable cluster size
constexpr int SAMPLE_PARTS = 32;            // runs of a row whose sums the draw adds up
constexpr int SAMPLE_CACHE = 40960;         // weights a CTA keeps (160 KB); a longer share's rest is formed again in every pass

struct SampleSmem {
    unsigned cnt[SAMPLE_BINS], hi[SAMPLE_BINS], lo[SAMPLE_BINS];      // a bin's elements, and their offsets in two parts
    double total[SAMPLE_GROUPS];                                      // from here to `single`: written by every CTA of the cluster
    float group[SAMPLE_GROUPS], mass[SAMPLE_PARTS];
    float val[SAMPLE_MAX_CTAS], above, target;
    int idx[SAMPLE_MAX_CTAS];
    int bin, single;
    unsigned bins_c[SAMPLE_THREADS];                                  // this CTA's bins over the cluster, by parts of it: elements, offsets
    unsigned long long bins_o[SAMPLE_THREADS];
    float rnd;                                                        // the row's own number in [0, 1) and settings, read while its logits are
    int top_k;
    float top_p;
    float warp_f[SAMPLE_WARPS];
    int warp_i[SAMPLE_WARPS];
};

__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

__device__ __forceinline__ void peer_st(int* p, int rank, int v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_addr(p, rank)), "r"(v) : "memory");
}
__device__ __forceinline__ void peer_st(float* p, int rank, float v) { peer_st(reinterpret_cast<int*>(p), rank, __float_as_int(v)); }
__device__ __forceinline__ void peer_st(double* p, int rank, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(peer_addr(p, rank)), "d"(v) : "memory");
}

// The same for one CTA of C; alone it needs neither.
template <int C, typename T>
__device__ __forceinline__ void peer_put(T* p, int rank, T v) {
    if (C == 1) *p = v;
    else peer_st(p, rank, v);
}
template <int C>
__device__ __forceinline__ unsigned peer_get(const unsigned* p, int rank) {
    return C == 1 ? *p : peer_ld(p, rank);
}
// A barrier of all CTAs of a row; one CTA needs no more than its own.
template <int C>
__device__ __forceinline__ void row_sync() {
    if (C == 1) __syncthreads();
    else cluster_sync_all();
}

// e = exp((x - max) / T) as its bit pattern; 0 where the difference has no value (NaN logits, infinity minus infinity)
__device__ __forceinline__ uint32_t weight_key(float x, float maxv, float inv_t) {
    const float e = __expf((x - maxv) * inv_t);
    return e > 0.f ? __float_as_uint(e) : 0u;
}

// A CTA's share of the row: the cached weights, and the logits of what did not fit.
struct SampleShare {
    const uint32_t* key;
    const float* x;
    int n, cached;
    float maxv, inv_t;
    __device__ __forceinline__ uint32_t at(int i) const { return i < cached ? key[i] : weight_key(x[i], maxv, inv_t); }
    // the elements for which `in` holds, four cached ones at a time: mostly none of the four
    template <class P, class F>
    __device__ __forceinline__ void each(P&& in, F&& f) const {
        const int n4 = cached >> 2;
#pragma unroll 2
        for (int i = threadIdx.x; i < n4; i += SAMPLE_THREADS) {
            const uint4 v = reinterpret_cast<const uint4*>(key)[i];
            if (in(v.x) | in(v.y) | in(v.z) | in(v.w)) {
                if (in(v.x)) f(v.x);
                if (in(v.y)) f(v.y);
                if (in(v.z)) f(v.z);
                if (in(v.w)) f(v.w);
            }
        }
        for (int i = 4 * n4 + threadIdx.x; i < n; i += SAMPLE_THREADS) {
            const uint32_t k = at(i);
            if (in(k)) f(k);
        }
    }
};

// One element in the histograms: its bin's count and, for masses, its offset in the bin.  Shares of up to 16384 elements take two
// additions: `cnt` holds the count above the sum of the offsets' bits 17 .. 19 (at most 7 * 16384), `lo` that of the other 17.  Longer
// ones take three, the offset's upper and lower ten bits apart.
constexpr int SAMPLE_PACKED = 16384;
constexpr int SAMPLE_SHIFT0 = 20, SAMPLE_BITS0 = 11;      // the first pass's bins
template <bool MASS>
__device__ __forceinline__ void count_key(SampleSmem& sm, uint32_t key, int shift, int nb, bool packed) {
    const uint32_t b = (key >> shift) & (nb - 1), off = key & ((1u << shift) - 1);
    if (MASS && packed) {
        atomicAdd(&sm.cnt[b], (1u << 17) | (off >> 17));
        if (off & 0x1ffffu) atomicAdd(&sm.lo[b], off & 0x1ffffu);
        return;
    }
    atomicAdd(&sm.cnt[b], 1u);
    if (MASS && (off >> 10)) atomicAdd(&sm.hi[b], off >> 10);
    if (MASS && (off & 1023u)) atomicAdd(&sm.lo[b], off & 1023u);
}
// What a CTA's histograms hold for bin b
template <bool MASS, int C>
__device__ __forceinline__ void read_bin(const SampleSmem& sm, int b, int rank, bool packed, unsigned& c, unsigned& hi, unsigned& lo) {
    c = peer_get<C>(&sm.cnt[b], rank);
    hi = MASS && !packed ? peer_get<C>(&sm.hi[b], rank) : 0u;
    lo = MASS ? peer_get<C>(&sm.lo[b], rank) : 0u;
}
template <bool MASS>
__device__ __forceinline__ void add_bin(unsigned pc, unsigned ph, unsigned pl, bool packed, unsigned& c, unsigned long long& off) {
    if (MASS && packed) {
        c += pc >> 17;
        off += ((unsigned long long)(pc & 0x1ffffu) << 17) + pl;
    } else {
        c += pc;
        off += ((unsigned long long)ph << 10) + pl;
    }
}

// Adds the n lanes' values to acc one by one from the last lane down and stops at the first that would reach the target; -1: none does.
__device__ __forceinline__ int walk_down(float v, int n, float& acc, float target) {
    for (int top = n - 8; top >= 0; top -= 8) {
        float x[9];                                  // the sums in order first: one addition a step, the comparisons beside them
        x[0] = acc;
        unsigned hit = 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u + 1] = __shfl_sync(0xffffffffu, v, top + 7 - u);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            x[u + 1] += x[u];
            if (x[u + 1] >= target) hit |= 1u << u;
        }
        if (hit) {
            const int first = __ffs(hit) - 1;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (u == first) acc = x[u];
            return top + 7 - first;
        }
        acc = x[8];
    }
    return -1;
}

// Largest key K such that weight{key >= K, key >= min_key} >= target, or a smaller one that keeps the same elements.  MASS: the
// weight is the sum of the elements, and the target `part` of the sum of all elements with key >= min_key; otherwise the weight is
// their number and the target `part` itself.  The bins are walked from the top in 32-bit sums, 64 at a time and then one by one,
// whatever C is.  Every thread of the cluster calls; the result is the same for all.
// counted: the first pass's histograms of this CTA are there (min_key 0).
template <bool MASS, int C>
__device__ uint32_t radix_threshold(const SampleShare& s, uint32_t min_key, float part, int rank, SampleSmem& sm, bool counted, bool packed) {
    const int shifts[3] = {SAMPLE_SHIFT0, 9, 0}, bits[3] = {SAMPLE_BITS0, 11, 9};
    constexpr int groups = SAMPLE_GROUPS / C;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;      // this CTA's groups of 64 bins
    uint32_t prefix = 0, mask = 0;
    float above = 0.f, target = part;
    for (int lvl = 0; lvl < 3; ++lvl) {
        const int shift = shifts[lvl], nb = 1 << bits[lvl];
        if (!counted || lvl > 0) {
            for (int i = threadIdx.x; i < SAMPLE_BINS; i += SAMPLE_THREADS) {
                sm.cnt[i] = 0;
                if (MASS) sm.hi[i] = sm.lo[i] = 0;
            }
            __syncthreads();
            s.each([&](uint32_t key) { return key >= min_key && (key & mask) == prefix; },
                   [&](uint32_t key) { count_key<MASS>(sm, key, shift, nb, packed); });
        }
        row_sync<C>();                          // every histogram of the cluster is complete
        // The CTA's bins over the cluster: from four CTAs on a thread adds up one bin of four of them (whole numbers: in any order), so that
        // all warps have their reads on the way together; then warp w sums groups w and w + 16, two bins of each per lane.
        constexpr bool SPREAD = C >= 4;
        constexpr int mine = SAMPLE_BINS / C;
        if (SPREAD) {
            const int b = rank * mine + threadIdx.x % mine, p0 = threadIdx.x / mine * 4;
            unsigned pc[4], ph[4], pl[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) read_bin<MASS, C>(sm, b, p0 + p, packed, pc[p], ph[p], pl[p]);
            unsigned c = 0;
            unsigned long long off = 0;
#pragma unroll
            for (int p = 0; p < 4; ++p) add_bin<MASS>(pc[p], ph[p], pl[p], packed, c, off);
            sm.bins_c[threadIdx.x] = c;
            sm.bins_o[threadIdx.x] = off;
            __syncthreads();
        }
        float wt[2][2];
        unsigned ct[2][2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int g = w + SAMPLE_WARPS * x;
            if (g >= groups) break;
            double all = 0.0;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int at = g * 64 + 32 * j + l, b = rank * mine + at;
                unsigned c = 0;
                unsigned long long off = 0;
                if (SPREAD) {
#pragma unroll
                    for (int p = 0; p < C / 4; ++p) {
                        c += sm.bins_c[p * mine + at];
                        off += sm.bins_o[p * mine + at];
                    }
                } else {
                    unsigned pc[C], ph[C], pl[C];        // all reads in flight before the first sum
#pragma unroll
                    for (int p = 0; p < C; ++p) read_bin<MASS, C>(sm, b, p, packed, pc[p], ph[p], pl[p]);
#pragma unroll
                    for (int p = 0; p < C; ++p) add_bin<MASS>(pc[p], ph[p], pl[p], packed, c, off);
                }
                double m = (double)c;
                if (MASS && c) {
                    const uint32_t k0 = prefix | ((uint32_t)b << shift);
                    const double base = (double)__uint_as_float(k0);
                    m = m * base + (double)off * ((double)__uint_as_float(k0 + 1) - base);
                }
                wt[x][j] = (float)m;
                ct[x][j] = c;
                all += m;
            }
            const float sum = warp_sum(wt[x][0] + wt[x][1]);
            if (MASS && lvl == 0)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
            if (l < C) {
                peer_put<C>(&sm.group[rank * groups + g], l, sum);
                if (MASS && lvl == 0) peer_put<C>(&sm.total[rank * groups + g], l, all);
            }
        }
        row_sync<C>();                          // the groups' sums are everywhere; the histograms have been read
        if (w < groups) {
            if (MASS && lvl == 0) {
                double z = sm.total[l];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
                target = part * (float)z;
            }
            // every lane walks the same way: the group, and in the warp that summed it the bin
            const float gs = sm.group[l];
            float acc = above;
            const int in = walk_down(gs, SAMPLE_GROUPS, acc, target);
            const int at = max(in, 0) - rank * groups;
#pragma unroll
            for (int x = 0; x < 2; ++x)
                if (at == w + SAMPLE_WARPS * x && at < groups) {
                    int bin = 0;
                    float over = acc;
                    if (in >= 0) {
                        bin = walk_down(wt[x][1], 32, over, target);
                        bin = bin >= 0 ? bin + 32 : walk_down(wt[x][0], 32, over, target);
                        // rounding: the group's sum said yes, the walk said no
                        if (bin < 0) bin = 0, over -= __shfl_sync(0xffffffffu, wt[x][0], 0);
                    } else {                          // more than there is: keep everything
                        over -= __shfl_sync(0xffffffffu, wt[x][0], 0);
                    }
                    const unsigned c = bin < 32 ? __shfl_sync(0xffffffffu, ct[x][0], bin) : __shfl_sync(0xffffffffu, ct[x][1], bin - 32);
                    if (l < C) {
                        peer_put<C>(&sm.bin, l, max(in, 0) * 64 + bin);
                        peer_put<C>(&sm.single, l, (int)(c == 1u));
                        peer_put<C>(&sm.above, l, over);
                        peer_put<C>(&sm.target, l, target);
                    }
                }
        }
        row_sync<C>();
        prefix |= (uint32_t)sm.bin << shift;
        mask |= (uint32_t)(nb - 1) << shift;
        above = sm.above;
        target = sm.target;
        if (sm.single) break;                        // the bin's only element is the one: its lower edge keeps the same set
    }
    return prefix < min_key ? min_key : prefix;
}

// C CTAs per row (a cluster; consecutive blocks)
template <int C>
__global__ void __launch_bounds__(SAMPLE_THREADS, 2)
sample_kernel(const float* __restrict__ logits, int V, int span, int cache, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p,
              const unsigned long long* __restrict__ seeds, int* __restrict__ out_tokens) {
    __shared__ SampleSmem sm;
    extern __shared__ __align__(16) uint32_t keys[];
    const int b = blockIdx.x / C, rank = blockIdx.x % C;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (C > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    pdl_wait();
    pdl_launch_dependents();
    const int lo = min(rank * span, V), hi = min(lo + span, V);
    const float* x = logits + (size_t)b * V + lo;
    SampleShare s;
    s.key = keys; s.x = x; s.n = hi - lo;
    const float temp = temperature ? temperature[b] : 0.f;
    const bool greedy = temp <= 1e-6f;
    s.cached = greedy ? 0 : min(s.n, cache);
    if (!greedy && threadIdx.x == SAMPLE_THREADS - 1) {
        sm.rnd = (float)(splitmix64(seeds ? seeds[b] : 0x1234ull + b) >> 40) * (1.0f / 16777216.0f);
        sm.top_k = top_k ? top_k[b] : 0;
        sm.top_p = top_p ? top_p[b] : 1.f;
    }

    if (!greedy)
        for (int i = threadIdx.x; i < SAMPLE_BINS; i += SAMPLE_THREADS) sm.cnt[i] = sm.hi[i] = sm.lo[i] = 0;

    // ---- max (+ argmax, lowest index on ties); the logits of a sampled row stay in shared memory
    float best = -INFINITY;
    int best_i = 0x7fffffff;
    auto take = [&](float v, int i) {                // ascending index order inside the thread
        if (v > best) { best = v; best_i = lo + i; }
    };
    if ((s.n & 3) == 0 && (s.cached & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        // 16-byte loads, four in flight per thread
        const float4* x4 = reinterpret_cast<const float4*>(x);
        const int n4 = s.n >> 2;
        for (int i = threadIdx.x; i < n4; i += 4 * SAMPLE_THREADS) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i + u * SAMPLE_THREADS < n4) v[u] = __ldcg(x4 + i + u * SAMPLE_THREADS);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = 4 * (i + u * SAMPLE_THREADS);
                if (c >= s.n) break;
                take(v[u].x, c); take(v[u].y, c + 1); take(v[u].z, c + 2); take(v[u].w, c + 3);
                if (c < s.cached) *reinterpret_cast<float4*>(keys + c) = v[u];
            }
        }
    } else {
        for (int i = threadIdx.x; i < s.n; i += 8 * SAMPLE_THREADS) {      // eight in flight
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (i + u * SAMPLE_THREADS < s.n) v[u] = __ldcg(x + i + u * SAMPLE_THREADS);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int c = i + u * SAMPLE_THREADS;
                if (c >= s.n) break;
                take(v[u], c);
                if (c < s.cached) keys[c] = __float_as_uint(v[u]);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    if (l == 0) { sm.warp_f[w] = best; sm.warp_i[w] = best_i; }
    __syncthreads();
    if (C > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // every CTA of the cluster has started
    if (w == 0) {                                    // lane p tells CTA p
        best = sm.warp_f[l & (SAMPLE_WARPS - 1)];
        best_i = sm.warp_i[l & (SAMPLE_WARPS - 1)];
#pragma unroll
        for (int o = SAMPLE_WARPS / 2; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
            if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
        }
        if (l < C) {
            peer_put<C>(&sm.val[rank], l, best);
            peer_put<C>(&sm.idx[rank], l, best_i);
        }
    }
    row_sync<C>();
    float maxv = sm.val[0];
    for (int p = 1; p < C; ++p) maxv = fmaxf(maxv, sm.val[p]);
    auto most_likely = [&]() {                       // shares are in index order: the first maximum wins
        int at = sm.idx[0];
        float v = sm.val[0];
        for (int p = 1; p < C; ++p)
            if (sm.val[p] > v) { v = sm.val[p]; at = sm.idx[p]; }
        return at == 0x7fffffff ? 0 : at;            // no logit above minus infinity (all of them minus infinity or NaN): an index of the row all the same
    };
    if (greedy) {
        if (rank == 0 && threadIdx.x == 0) out_tokens[b] = most_likely();
        return;
    }
    s.maxv = maxv;
    s.inv_t = 1.f / temp;
    const int k = sm.top_k;
    const float p = sm.top_p;
    // The draw sees the row as SAMPLE_PARTS runs of `part` elements, 1 / C of them in this CTA's share.  A run is summed by one warp
    // and the runs' sums are added in order whatever C is, so that a token does not depend on how the row was shared out.
    constexpr int runs = SAMPLE_PARTS / C;
    const int part = span / runs;
    auto sum_runs = [&](auto&& weight) {
        for (int q = w; q < runs; q += SAMPLE_WARPS) {
            const int qhi = min((q + 1) * part, s.n);
            float mine = 0.f;
            int i = q * part + l;
            for (; i + 15 * 32 < qhi; i += 16 * 32) {     // sixteen reads in flight, added one by one
                float e[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) e[u] = weight(i + u * 32);
#pragma unroll
                for (int u = 0; u < 16; ++u) mine += e[u];
            }
            for (; i < qhi; i += 32) mine += weight(i);
            mine = warp_sum(mine);
            if (l == 0)
                for (int peer = 0; peer < C; ++peer) peer_put<C>(&sm.mass[rank * runs + q], peer, mine);
        }
    };
    uint32_t thr = 0;           // keep keys >= thr
    auto kept = [&](int i) {
        const uint32_t key = s.at(i);
        return key >= thr ? __uint_as_float(key) : 0.f;
    };
    auto kept_here = [&](int i) {                    // of a share that is cached whole
        const uint32_t key = keys[i];
        return key >= thr ? __uint_as_float(key) : 0.f;
    };
    if (C <= 2 && !(k > 0 && k < V) && !(p < 1.f)) {
        // a row without filters whose runs occupy all warps is summed while its weights are formed
        sum_runs([&](int i) {
            const uint32_t key = weight_key(i < s.cached ? __uint_as_float(keys[i]) : x[i], maxv, s.inv_t);
            if (i < s.cached) keys[i] = key;
            return __uint_as_float(key);
        });
    } else {
        // the weights, and with them the histograms of the first pass of the first filter
        const bool by_count = k > 0 && k < V, by_mass = p < 1.f && p > 0.f, packed = span <= SAMPLE_PACKED;
        auto form = [&](auto&& add) {
            const int n4 = s.cached >> 2;
            auto key_of = [&](uint32_t bits) {
                const uint32_t key = weight_key(__uint_as_float(bits), maxv, s.inv_t);
                add(key);
                return key;
            };
#pragma unroll 2
            for (int i = threadIdx.x; i < n4; i += SAMPLE_THREADS) {
                const uint4 v = reinterpret_cast<const uint4*>(keys)[i];
                reinterpret_cast<uint4*>(keys)[i] = make_uint4(key_of(v.x), key_of(v.y), key_of(v.z), key_of(v.w));
            }
            for (int i = 4 * n4 + threadIdx.x; i < s.cached; i += SAMPLE_THREADS) keys[i] = key_of(keys[i]);
            for (int i = s.cached + threadIdx.x; i < s.n; i += SAMPLE_THREADS) add(weight_key(x[i], maxv, s.inv_t));
        };
        if (by_count) form([&](uint32_t key) { count_key<false>(sm, key, SAMPLE_SHIFT0, 1 << SAMPLE_BITS0, packed); });
        else if (by_mass) form([&](uint32_t key) { count_key<true>(sm, key, SAMPLE_SHIFT0, 1 << SAMPLE_BITS0, packed); });
        else form([](uint32_t) {});
        __syncthreads();
        if (by_count) thr = radix_threshold<false, C>(s, 0u, (float)k, rank, sm, true, packed);
        if (p < 1.f) {
            if (p > 0.f) thr = radix_threshold<true, C>(s, thr, p, rank, sm, !by_count, packed);
            else thr = 0xffffffffu;                  // an empty nucleus: the most likely token
        }
        if (s.cached == s.n) sum_runs(kept_here);
        else sum_runs(kept);
    }
    row_sync<C>();                              // nothing is read from or written to another CTA after this
    // a run's sum per lane; the sum of all runs in order, of which a lane keeps the part before its own
    const float run_sum = sm.mass[l];
    float tot = 0.f, ahead = 0.f;
    for (int q0 = 0; q0 < SAMPLE_PARTS; q0 += 8) {
        float x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = __shfl_sync(0xffffffffu, run_sum, q0 + u);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (l == q0 + u) ahead = tot;
            tot += x[u];
        }
    }
    if (!(tot > 0.f)) {
        if (rank == 0 && threadIdx.x == 0) out_tokens[b] = most_likely();
        return;
    }
    const float u = sm.rnd * tot;               // [0, tot)
    const unsigned past = __ballot_sync(0xffffffffu, ahead + run_sum > u);
    int in = past ? __ffs(past) - 1 : SAMPLE_PARTS - 1;
    const float before = past ? __shfl_sync(0xffffffffu, ahead, in) : tot;
    while (in > 0 && sm.mass[in] == 0.f) --in;        // rounding pushed u past the total: the last run that holds mass
    if (in / runs != rank) return;
    // Inside the run: blocks of 32 elements, an inclusive scan in each.  All warps scan blocks and leave every block's sum and the
    // largest kept prefix in it; the running sum over the blocks then stops at the first one with a prefix beyond the point.
    const float need = u - before;
    const int wlo = in % runs * part, whi = min(wlo + part, s.n);
    float* bsum = reinterpret_cast<float*>(sm.cnt);
    float* bmax = reinterpret_cast<float*>(sm.hi);
    auto scan = [&](float e) {
        float inc = e;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float n = __shfl_up_sync(0xffffffffu, inc, o);
            if (l >= o) inc += n;
        }
        return inc;
    };
    auto element = [&](int i) { return i < whi ? kept(i) : 0.f; };
    int last_kept = -1;
    float run = 0.f;
    for (int c0 = wlo; c0 < whi; c0 += 32 * SAMPLE_BINS) {      // (one round, except for rows of more than two million)
        const int blocks = (min(c0 + 32 * SAMPLE_BINS, whi) - c0 + 31) / 32;
        __syncthreads();
        for (int q0 = w; q0 < (blocks + 7 & ~7); q0 += 4 * SAMPLE_WARPS) {      // four blocks at a time; those behind the last hold nothing
            float e[4], inc[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) e[x] = element(c0 + 32 * (q0 + x * SAMPLE_WARPS) + l);
#pragma unroll
            for (int x = 0; x < 4; ++x) inc[x] = scan(e[x]);
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int q = q0 + x * SAMPLE_WARPS;
                const unsigned most = __reduce_max_sync(0xffffffffu, e[x] > 0.f ? __float_as_uint(inc[x]) : 0u);      // (sums of kept ones are above zero)
                if (l == 31 && q < SAMPLE_BINS) { bsum[q] = inc[x]; bmax[q] = most ? __uint_as_float(most) : -1.f; }
            }
        }
        __syncthreads();
        int q = blocks;
        for (int q8 = 0; q8 < blocks && q == blocks; q8 += 8) {      // every thread walks the same way, eight blocks read at a time
            float before[9], bm[8];
            unsigned hit = 0, any = 0;
            before[0] = run;
#pragma unroll
            for (int x = 0; x < 8; ++x) { before[x + 1] = bsum[q8 + x]; bm[x] = bmax[q8 + x]; }
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                before[x + 1] += before[x];
                if (bm[x] >= 0.f && before[x] + bm[x] > need) hit |= 1u << x;
                if (bm[x] >= 0.f) any |= 1u << x;
            }
            if (hit) {
                const int first = __ffs(hit) - 1;
                q = q8 + first;
#pragma unroll
                for (int x = 0; x < 8; ++x)
                    if (x == first) run = before[x];
            } else {
                if (any) last_kept = q8 + 31 - __clz(any);
                run = before[8];
            }
        }
        if (q < blocks || last_kept >= 0) {
            if (w != 0) {
                if (q < blocks) return;
            } else {
                const int at = c0 + 32 * (q < blocks ? q : last_kept);
                const float e = element(at + l), inc = scan(e);
                const unsigned hit = __ballot_sync(0xffffffffu, e > 0.f && run + inc > need), any = __ballot_sync(0xffffffffu, e > 0.f);
                if (q < blocks) {
                    if (l == 0) out_tokens[b] = lo + at + __ffs(hit) - 1;
                    return;
                }
                if (l == 0) out_tokens[b] = lo + at + 31 - __clz(any);      // rounding: the last kept one, unless a later round holds it
                last_kept = -1;
            }
        }
    }
}

template <int C>
static int launch_rows(const float* logits, int B, int V, int span, int cache, const float* temperature, const int* top_k, const float* top_p,
                       const unsigned long long* seeds, int* out_tokens, bool pdl, cudaStream_t stream) {
    static PerDeviceFlag attr_set;
    if (!attr_set.done()) {
        FT_CHECK_CUDA(cudaFuncSetAttribute(sample_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, SAMPLE_CACHE * 4));
        attr_set.mark();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(B * C);
    cfg.blockDim = dim3(SAMPLE_THREADS);
    cfg.dynamicSmemBytes = temperature ? (size_t)cache * 4 : 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (C > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = C; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    FT_CHECK_CUDA(cudaLaunchKernelEx(&cfg, sample_kernel<C>, logits, V, span, cache, temperature, top_k, top_p, seeds, out_tokens));
    return 0;
}

int launch_sample(const float* logits, int B, int V, const float* temperature, const int* top_k,
                  const float* top_p, const unsigned long long* seeds, int* out_tokens, bool pdl,
                  cudaStream_t stream) {
    FT_REQUIRE(B >= 1 && V >= 1, "sample: B=%d V=%d", B, V);
    // CTAs per row: a share of 4096 logits keeps 512 threads busy for longer than a cluster barrier takes.  Rows of up to 65536
    // logits, and greedy ones, take no more CTAs than are resident at once, two per SM, and beyond half of the SMs in rows not those
    // that only shorten a share below 16384.  Nucleus / plain / greedy rows, with eight CTAs each whatever the batch and (last)
    // with one CTA that reads the row again in every pass, as it once was:
    //   256 rows of 32768   49 / 16 / 5.3 us   139 / 60 / 23    99 / 25 / 6.7
    //   128 rows of 50257   49 / 18 / 6.6       88 / 41 / 14    72 / 20 / 4.9
    // A longer row that is sampled wants its weights in shared memory whatever the batch (128 rows of 128256: 124 us in eight CTAs,
    // 145 in two; 96 rows: 96 and 139); its greedy neighbours pay for that (14 us, alone 7.9).
    const int sms = device_sms();
    const bool bounded = V <= 65536 || !temperature;
    const int per = bounded && 2LL * B > sms ? 16384 : 4096;
    int C = 1;
    while (C < SAMPLE_MAX_CTAS && V > per * C && (!bounded || 2LL * C * B <= 2LL * sms)) C *= 2;
    while (C > 1 && (long long)B * C > 0x7fffffffll) C /= 2;
    const int span = (V + SAMPLE_PARTS - 1) / SAMPLE_PARTS * (SAMPLE_PARTS / C);      // a multiple of 4: shares start on 16 bytes where the rows do
    // half of the weights where that lets a second CTA onto the SM and there is one (256 rows of 50257: 87 us, 126 with all)
    const int room = bounded && C <= 2 && (long long)B * C > sms ? SAMPLE_CACHE / 2 : SAMPLE_CACHE;
    const int cache = span < room ? span : room;
    switch (C) {
        case 1: return launch_rows<1>(logits, B, V, span, cache, temperature, top_k, top_p, seeds, out_tokens, pdl, stream);
        case 2: return launch_rows<2>(logits, B, V, span, cache, temperature, top_k, top_p, seeds, out_tokens, pdl, stream);
        case 4: return launch_rows<4>(logits, B, V, span, cache, temperature, top_k, top_p, seeds, out_tokens, pdl, stream);
        default: return launch_rows<8>(logits, B, V, span, cache, temperature, top_k, top_p, seeds, out_tokens, pdl, stream);
    }
}

}  // namespace ft

extern "C" int ft_sample(const float* logits, int B, int V, const float* temperature, const int* top_k,
                         const float* top_p, const unsigned long long* seeds, int* out_tokens,
                         void* stream) {
    return ft::launch_sample(logits, B, V, temperature, top_k, top_p, seeds, out_tokens, false,
                             static_cast<cudaStream_t>(stream));
}

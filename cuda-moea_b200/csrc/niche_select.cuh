// Niche selection of the last front by direction buckets, and the ordered
// survivor list, in one kernel: device code shared by the staged path
// (niching_cluster.cu: one CTA or a cluster of sixteen) and the batches (nsga3.cu:
// a cluster of two per instance).
//
// The reference selects with three stable sorts of the last front's members
// (niching.cu:96-178); the random words of the second and third hash the
// position in the order before.  None of the three orders has to be built to
// know a member's place in it, because each of the first two keeps the
// directions in ascending order:
//   order 1, by (direction, distance): position = members of smaller
//     directions (a prefix sum of the direction counts) + rank by (distance,
//     member) among the members of the same direction;
//   order 2, by (direction, word): the same prefix + rank by (word, order-1
//     position) inside the direction;
//   order 3, by (niche count + rank, word): only its first nrem members are
//     wanted and in no particular order, so a histogram of the first key
//     finds the level where nrem is reached, a histogram of the word's top
//     bits the bin of that level, and only the members of that bin are ranked.
// Ranks inside a direction are counted against its other members, which costs
// the sum of the squared bucket sizes: populations spread over the directions
// have buckets of a few members.  Where a few directions hold most of the
// front (the bounds below), the caller's sorts take over.
//
// Bound by the latency of its ten phases (each a global or distributed-memory
// round trip and a barrier, 3,000-4,000 clocks): DTLZ1 M=3 N=32768 (31,000
// prior and 2,000 last members, 32,640 directions) 21 us where the prior
// counts, the three sorts and the survivor list took 95; DTLZ2 M=8 N=6436
// (9,700 last members) 19 us against 125; 275 directions with buckets of up to
// 458 of 7,900 members 30 us against 120.
#pragma once

#include <cooperative_groups.h>

#include "internal.cuh"

namespace moea {

constexpr int kNsLevels = 1024;            // niche levels told apart; the last one also holds all above it
constexpr int kNsBins = 1024;              // bins of the boundary level's random words
constexpr int kNsWordStep = 512;           // survivor words written out per step (at most a block's threads)
constexpr int kNsMaxBucket = 2048;         // largest direction bucket ranked by counting
constexpr unsigned long long kNsMaxWork = 8ull << 20;  // largest sum of squared bucket sizes

// Scratch in device memory, shared by the CTAs that select together.
struct NicheScratch {
    int* rho;            // (H) members of the prior fronts per direction
    int* last;           // (H + 1) members of the last front per direction; [H]: none
    int* start;          // (H + 1) first position of each direction in its segment
    uint64_t* key_a;     // (nl)
    uint64_t* key_b;     // (nl)
    int* dir_of;         // (nl)
    uint32_t* mask;      // (ceil(n_mix / 32)) survivor bits
    int* hist;           // (kNsLevels) members per niche level, then (kNsBins) members per bin, then
                         // the length of the list of the boundary bin
};
constexpr int kNsHistWords = kNsLevels + kNsBins + 1;

NicheScratch niche_scratch(const Workspace& ws);

// Niche selection and ascending survivors on one cluster (niching_cluster.cu):
// merged populations up to niching_cluster_capacity().
int launch_niche_select(const int* idx, const float* dist, const int* sizes, const NicheScratch& S, int H,
                        uint64_t seed, unsigned long long* offset, const int* nds_gidx, int* selected, int n_mix, int N,
                        int* survivors, int* status, cudaStream_t stream);

// ITEMS: last-front members per thread, at most.
template <int THREADS, int ITEMS>
struct NicheShared {
    uint64_t stage[ITEMS * THREADS + 2 * kNsMaxBucket];  // the buckets that this CTA's members belong to
    int hist[kNsLevels];
    int wsum[THREADS / 32];
    unsigned long long wsum64[THREADS / 32];
    int wmax[THREADS / 32];
    int seg_total;                  // members in this CTA's segment of directions
    int seg_max;                    // largest bucket of the segment
    unsigned long long seg_work;    // sum of squared bucket sizes of the segment
    int seg_off[16];                // first position of each CTA's segment
    int max_bucket;
    int level, level_take, level_all, bin, bin_take;
    int word_off[kNsWordStep];
    int fallback;
};

// The CTAs that select together: a cluster, or one CTA.
struct NicheCluster {
    static constexpr bool kMany = true;
    cooperative_groups::cluster_group g = cooperative_groups::this_cluster();
    __device__ __forceinline__ int rank() const { return (int)g.block_rank(); }
    __device__ __forceinline__ int count() const { return (int)g.num_blocks(); }
    __device__ __forceinline__ void sync() { g.sync(); }
    template <class T>
    __device__ __forceinline__ T* map(T* p, int r) { return g.map_shared_rank(p, r); }
};
struct NicheSolo {
    static constexpr bool kMany = false;
    __device__ __forceinline__ int rank() const { return 0; }
    __device__ __forceinline__ int count() const { return 1; }
    __device__ __forceinline__ void sync() { __syncthreads(); }
    template <class T>
    __device__ __forceinline__ T* map(T* p, int) { return p; }
};

// Exclusive sum over the block; *total receives the block's sum.
template <int THREADS>
__device__ __forceinline__ int niche_scan(int v, int* wsum, int* total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    __syncthreads();  // wsum free
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int x = (lane < THREADS / 32) ? wsum[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    *total = __shfl_sync(0xFFFFFFFFu, x, THREADS / 32 - 1);
    const int before = __shfl_sync(0xFFFFFFFFu, x, warp > 0 ? warp - 1 : 0);
    return incl - v + (warp > 0 ? before : 0);
}

// The bin of a histogram in device memory where the running count reaches
// `want`: the bin, the members to take from it and its size.
template <int THREADS>
__device__ __forceinline__ void niche_threshold(const int* hist, int want, int* wsum, int* out_bin, int* out_take,
                                                int* out_size)
{
    static_assert(kNsLevels == kNsBins && kNsLevels % THREADS == 0, "bins per thread");
    constexpr int kPer = kNsLevels / THREADS;
    int v[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        v[k] = __ldcg(hist + threadIdx.x * kPer + k);
        sum += v[k];
    }
    int total;
    int before = niche_scan<THREADS>(sum, wsum, &total);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        if (before < want && before + v[k] >= want) {
            *out_bin = threadIdx.x * kPer + k;
            *out_take = want - before;
            *out_size = v[k];
        }
        before += v[k];
    }
    __syncthreads();
}

// Keys of w[0, n) below k, eight loads in flight.
__device__ __forceinline__ int niche_rank(const uint64_t* w, int n, uint64_t k)
{
    int rank = 0, u = 0;
    for (; u + 8 <= n; u += 8) {
        uint64_t a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = w[u + i];
#pragma unroll
        for (int i = 0; i < 8; ++i) rank += a[i] < k ? 1 : 0;
    }
    for (; u < n; ++u) rank += w[u] < k ? 1 : 0;
    return rank;
}

__device__ __forceinline__ void niche_mark(uint32_t* mask, int g) { atomicOr(mask + (g >> 5), 1u << (g & 31)); }

// Marks the survivors of one selection in S.mask: every member of the prior
// fronts and, unless it returns false, the nrem members of the last front
// that the three orders above put first.  It returns false (in every thread
// of the group, with S.rho and the prior members' bits complete) when the
// buckets are too large to be ranked by counting.  nl <= ITEMS * THREADS * CTAs.  Ends with the group in step.
template <int THREADS, int ITEMS, class G>
__device__ bool niche_buckets(G& grp, NicheShared<THREADS, ITEMS>& sm, const NicheScratch& S, const int* __restrict__ idx,
                              const float* __restrict__ dist, const int* __restrict__ gidx, int np, int nl, int nrem,
                              int H, uint64_t seed, unsigned long long off, int n_mix)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = grp.rank(), C = grp.count(), T = C * THREADS, gt = c * THREADS + tid;
    for (int i = gt; i < H; i += T) S.rho[i] = 0;
    for (int i = gt; i <= H; i += T) S.last[i] = 0;
    for (int i = gt; i < (n_mix + 31) >> 5; i += T) S.mask[i] = 0;
    for (int i = gt; i < kNsHistWords; i += T) S.hist[i] = 0;
    for (int i = tid; i < kNsLevels; i += THREADS) sm.hist[i] = 0;
    if (tid == 0) {
        sm.level = nrem > 0 ? 1 << 30 : -1;  // stays when all members of the last front are taken, or none
        sm.level_take = sm.level_all = 0;
        sm.bin = -1;
        sm.bin_take = 0;
    }
    // this CTA's members, as well as its positions in the orders below: [lo, hi)
    const int slice = (nl + C - 1) / C;
    const int lo = min(nl, c * slice), hi = min(nl, lo + slice);
    int dir[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int p = lo + tid + j * THREADS;
        dir[j] = -1;
        if (p < hi) {
            const int r = idx[np + p];
            dir[j] = (r >= 0 && r < H) ? r : H;
        }
    }
    grp.sync();
    // direction counts; a member's slot in its direction comes from the count
    int slot[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        if (lo + warp * 32 + j * THREADS >= hi) break;  // warp-uniform
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, dir[j]);
        const int leader = __ffs(peers) - 1;
        int base = 0;
        if (dir[j] >= 0 && lane == leader) base = atomicAdd(S.last + dir[j], __popc(peers));
        slot[j] = __shfl_sync(0xFFFFFFFFu, base, leader) + __popc(peers & ((1u << lane) - 1u));
    }
    for (int i = gt; i - lane < np; i += 4 * T) {  // warp-uniform
        int r[4], g[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            r[k] = (i + k * T < np) ? idx[i + k * T] : -1;
            g[k] = (i + k * T < np) ? gidx[i + k * T] : -1;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (g[k] >= 0) niche_mark(S.mask, g[k]);
            const unsigned peers = __match_any_sync(0xFFFFFFFFu, r[k]);
            if (r[k] >= 0 && r[k] < H && lane == __ffs(peers) - 1) atomicAdd(S.rho + r[k], __popc(peers));
        }
    }
    grp.sync();
    // first position of each direction: every CTA scans a segment of directions
    const int per = (((H + 1 + C - 1) / C) + 3) & ~3;
    {
        const int b_lo = c * per, b_hi = min(H + 1, b_lo + per);
        int carry = 0, big = 0;
        unsigned long long work = 0;
        for (int b0 = b_lo; b0 < b_hi; b0 += 4 * THREADS) {
            const int b = b0 + 4 * tid;
            int v[4] = {0, 0, 0, 0};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (b + k < b_hi) v[k] = __ldcg(S.last + b + k);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                big = max(big, v[k]);
                work += (unsigned long long)v[k] * (unsigned long long)v[k];
            }
            int total;
            int at = carry + niche_scan<THREADS>(v[0] + v[1] + v[2] + v[3], sm.wsum, &total);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (b + k < b_hi) __stcg(S.start + b + k, at);
                at += v[k];
            }
            carry += total;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            big = max(big, __shfl_xor_sync(0xFFFFFFFFu, big, o));
            work += __shfl_xor_sync(0xFFFFFFFFu, work, o);
        }
        if (lane == 0) {
            sm.wmax[warp] = big;
            sm.wsum64[warp] = work;
        }
        __syncthreads();
        if (warp == 0) {
            big = lane < THREADS / 32 ? sm.wmax[lane] : 0;
            work = lane < THREADS / 32 ? sm.wsum64[lane] : 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                big = max(big, __shfl_xor_sync(0xFFFFFFFFu, big, o));
                work += __shfl_xor_sync(0xFFFFFFFFu, work, o);
            }
            if (lane == 0) {
                sm.seg_total = carry;
                sm.seg_max = big;
                sm.seg_work = work;
            }
        }
    }
    grp.sync();
    if (warp == 0) {
        int at = 0, big = 0;
        unsigned long long work = 0;
        if (lane < C) {
            at = *grp.map(&sm.seg_total, lane);
            big = *grp.map(&sm.seg_max, lane);
            work = *grp.map(&sm.seg_work, lane);
        }
        int incl = at;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += y;
            big = max(big, __shfl_xor_sync(0xFFFFFFFFu, big, o));
            work += __shfl_xor_sync(0xFFFFFFFFu, work, o);
        }
        if (lane < C) sm.seg_off[lane] = incl - at;
        if (lane == 0) {
            sm.max_bucket = big;
            sm.fallback = (big > kNsMaxBucket || work > kNsMaxWork) ? 1 : 0;
        }
    }
    __syncthreads();
    if (sm.fallback) {  // the same in every CTA
        grp.sync();     // the segment words were read everywhere
        return false;
    }
    // members into their direction's bucket, keyed by (distance, member)
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int p = lo + tid + j * THREADS;
        if (p >= hi) break;
        const int b = dir[j];
        const int pos = sm.seg_off[b / per] + __ldcg(S.start + b) + slot[j];
        __stcg(S.key_a + pos, ((uint64_t)__float_as_uint(dist[np + p]) << 32) | (uint32_t)p);
        __stcg(S.dir_of + pos, b);
    }
    grp.sync();
    // The buckets of this CTA's positions reach at most the largest bucket
    // beyond them: they are ranked in shared memory.  Order 1 inside the
    // buckets, and the words of order 2.
    const int w_lo = max(0, lo - sm.max_bucket), w_hi = lo < hi ? min(nl, hi + sm.max_bucket) : w_lo;
    int first[ITEMS], size[ITEMS], prior[ITEMS], member[ITEMS];
    for (int u = w_lo + tid; u < w_hi; u += THREADS) sm.stage[u - w_lo] = __ldcg(S.key_a + u);
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int q = lo + tid + j * THREADS;
        first[j] = size[j] = prior[j] = member[j] = 0;
        if (q >= hi) continue;
        const int b = __ldcg(S.dir_of + q);
        first[j] = sm.seg_off[b / per] + __ldcg(S.start + b);
        size[j] = __ldcg(S.last + b);
        prior[j] = b < H ? __ldcg(S.rho + b) : 0;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int q = lo + tid + j * THREADS;
        if (q >= hi) break;
        const uint64_t k = sm.stage[q - w_lo];
        const int rank = niche_rank(sm.stage + (first[j] - w_lo), size[j], k);
        const int at = first[j] + rank;
        const uint32_t rnd = splitmix_u32(off + (uint64_t)at, seed);
        const uint32_t low = (prior[j] == 0 && rank == 0) ? 0u : (rnd | 1u);
        __stcg(S.key_b + q, ((uint64_t)low << 32) | (uint32_t)at);
        member[j] = (int)(uint32_t)k;
    }
    grp.sync();
    // order 2 inside the buckets; the levels and words of order 3
    uint32_t word[ITEMS];
    int pos2[ITEMS];
    for (int u = w_lo + tid; u < w_hi; u += THREADS) sm.stage[u - w_lo] = __ldcg(S.key_b + u);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int q = lo + tid + j * THREADS;
        if (q >= hi) break;
        const uint64_t k = sm.stage[q - w_lo];
        const int rank = niche_rank(sm.stage + (first[j] - w_lo), size[j], k);
        pos2[j] = first[j] + rank;
        word[j] = splitmix_u32(off + (uint64_t)nl + (uint64_t)pos2[j], seed);
        prior[j] += rank;  // the level
        atomicAdd(sm.hist + min(prior[j], kNsLevels - 1), 1);
    }
    const bool part = nrem > 0 && nrem < nl;
    bool split = false;
    if (part) {
        __syncthreads();
        for (int i = tid; i < kNsLevels; i += THREADS)
            if (sm.hist[i]) atomicAdd(S.hist + i, sm.hist[i]);
        grp.sync();
        niche_threshold<THREADS>(S.hist, nrem, sm.wsum, &sm.level, &sm.level_take, &sm.level_all);
        if (sm.level == kNsLevels - 1 && sm.level_take < sm.level_all) {  // levels above are not told apart
            grp.sync();
            return false;
        }
        split = sm.level_take < sm.level_all;
    }
    const int level = sm.level;
    if (split) {
        int* bins = S.hist + kNsLevels;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            if (lo + tid + j * THREADS >= hi) break;
            if (prior[j] == level) atomicAdd(bins + (word[j] >> 22), 1);
        }
        grp.sync();
        niche_threshold<THREADS>(bins, sm.level_take, sm.wsum, &sm.bin, &sm.bin_take, &sm.level_all);
    }
    const int bin = sm.bin, bin_take = sm.bin_take;
    int* list_count = S.hist + kNsLevels + kNsBins;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        if (lo + tid + j * THREADS >= hi) break;
        bool take = prior[j] < level || (prior[j] == level && !split);
        if (split && prior[j] == level) {
            const int wb = (int)(word[j] >> 22);
            take = wb < bin;
            if (wb == bin)  // ranked below
                __stcg(S.key_a + atomicAdd(list_count, 1), ((uint64_t)word[j] << 32) | (uint32_t)pos2[j]);
        }
        if (take) niche_mark(S.mask, gidx[np + member[j]]);
    }
    grp.sync();  // the list is complete
    if (split) {
        const int ln = __ldcg(list_count);
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            if (lo + tid + j * THREADS >= hi) break;
            if (prior[j] != level || (int)(word[j] >> 22) != bin) continue;
            const uint64_t k = ((uint64_t)word[j] << 32) | (uint32_t)pos2[j];
            int rank = 0;
            for (int u = 0; u < ln; ++u) rank += __ldcg(S.key_a + u) < k ? 1 : 0;
            if (rank < bin_take) niche_mark(S.mask, gidx[np + member[j]]);
        }
        grp.sync();
    }
    return true;
}

// Survivors in ascending order from the bits of S.mask (complete, the group in
// step).  Every CTA counts the words before its own and writes its own out.
template <int THREADS, int ITEMS, class G>
__device__ void niche_survivors(G& grp, NicheShared<THREADS, ITEMS>& sm, const uint32_t* mask, int n_mix,
                                int* __restrict__ survivors, int cap)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int words = (n_mix + 31) >> 5;
    const int per = (words + grp.count() - 1) / grp.count();
    const int lo = min(words, grp.rank() * per), hi = min(words, lo + per);
    int before = 0;
    for (int w = tid; w < lo; w += THREADS) before += __popc(__ldcg(mask + w));
    int base;
    niche_scan<THREADS>(before, sm.wsum, &base);
    for (int w0 = lo; w0 < hi; w0 += kNsWordStep) {
        const int w = w0 + tid;
        int total;
        const int at = niche_scan<THREADS>(tid < kNsWordStep && w < hi ? __popc(__ldcg(mask + w)) : 0, sm.wsum, &total);
        if (tid < kNsWordStep) sm.word_off[tid] = base + at;
        __syncthreads();
        const int n = min(kNsWordStep, hi - w0);
        for (int k = warp; k < n; k += THREADS / 32) {
            const uint32_t bits = __ldcg(mask + w0 + k);
            const int to = sm.word_off[k] + __popc(bits & ((1u << lane) - 1u));
            if (((bits >> lane) & 1u) && to < cap) survivors[to] = (w0 + k) * 32 + lane;
        }
        base += total;
        __syncthreads();
    }
}

}  // namespace moea

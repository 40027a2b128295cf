// Niche selection of the last front by direction buckets, and the ordered
// survivor list, in one kernel: device code shared by the cluster kernel of
// the staged path (niching_cluster.cu) and the one-CTA kernel of the fused
// path (nsga3.cu).
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
#pragma once

#include <cooperative_groups.h>

#include "internal.cuh"

namespace moea {

constexpr int kNsLevels = 1024;            // niche levels told apart; the last one also holds all above it
constexpr int kNsBins = 1024;              // bins of the boundary level's random words
constexpr int kNsWordStep = 512;           // survivor words written out per step (at most a block's threads)
constexpr int kNsItems = 8;                // last-front members per thread, at most
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
    int* list_count;     // (1)
};

NicheScratch niche_scratch(const Workspace& ws);

// Niche selection and ascending survivors on one cluster (niching_cluster.cu):
// merged populations up to niching_cluster_capacity().
int launch_niche_select(const int* idx, const float* dist, const int* sizes, const NicheScratch& S, int H,
                        uint64_t seed, unsigned long long* offset, const int* nds_gidx, int* selected, int n_mix, int N,
                        int* survivors, int* status, cudaStream_t stream);

template <int THREADS>
struct NicheShared {
    int hist[kNsLevels];
    int bins[kNsBins];
    int wsum[THREADS / 32];
    unsigned long long wsum64[THREADS / 32];
    int wmax[THREADS / 32];
    int seg_total;                  // members in this CTA's segment of directions
    int seg_max;                    // largest bucket of the segment
    unsigned long long seg_work;    // sum of squared bucket sizes of the segment
    int seg_off[16];                // first position of each CTA's segment
    int level, level_take, level_all, bin, bin_take;
    int word_off[kNsWordStep];
    int fallback;
};

// The CTAs that select together: a cluster, or one CTA.
struct NicheCluster {
    cooperative_groups::cluster_group g;
    __device__ __forceinline__ int rank() const { return (int)g.block_rank(); }
    __device__ __forceinline__ int count() const { return (int)g.num_blocks(); }
    __device__ __forceinline__ void sync() { g.sync(); }
    template <class T>
    __device__ __forceinline__ T* map(T* p, int r) { return g.map_shared_rank(p, r); }
};
struct NicheSolo {
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

// The bin of a histogram held by every CTA of the group (summed over them)
// where the running count reaches `want`: the bin, the members to take from it
// and its size.  Every thread of every CTA calls; the result is in sm.
template <int THREADS, class G>
__device__ __forceinline__ void niche_threshold(G& grp, int* hist, int nbins, int want, int* wsum, int* out_bin,
                                                int* out_take, int* out_size)
{
    static_assert(kNsLevels % THREADS == 0 || THREADS % kNsLevels == 0, "bins per thread");
    constexpr int kPer = kNsLevels > THREADS ? kNsLevels / THREADS : 1;
    const int C = grp.count();
    int v[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int b = threadIdx.x * kPer + k;
        v[k] = 0;
        if (b < nbins)
            for (int r = 0; r < C; ++r) v[k] += grp.map(hist, r)[b];
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

__device__ __forceinline__ void niche_mark(uint32_t* mask, int g) { atomicOr(mask + (g >> 5), 1u << (g & 31)); }

// Marks the survivors of one selection in S.mask: every member of the prior
// fronts and, unless it returns false, the nrem members of the last front
// that the three orders above put first.  It returns false (in every thread
// of the group, with S.rho and the prior members' bits complete) when the
// buckets are too large to be ranked by counting.  nl <= kNsItems * THREADS *
// CTAs.  Ends with the group in step.
template <int THREADS, class G>
__device__ bool niche_buckets(G& grp, NicheShared<THREADS>& sm, const NicheScratch& S, const int* __restrict__ idx,
                              const float* __restrict__ dist, const int* __restrict__ gidx, int np, int nl, int nrem,
                              int H, uint64_t seed, unsigned long long off, int n_mix)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = grp.rank(), C = grp.count(), T = C * THREADS, gt = c * THREADS + tid;
    for (int i = gt; i < H; i += T) S.rho[i] = 0;
    for (int i = gt; i <= H; i += T) S.last[i] = 0;
    for (int i = gt; i < (n_mix + 31) >> 5; i += T) S.mask[i] = 0;
    for (int i = tid; i < kNsLevels; i += THREADS) sm.hist[i] = 0;
    for (int i = tid; i < kNsBins; i += THREADS) sm.bins[i] = 0;
    if (gt == 0) *S.list_count = 0;
    if (tid == 0) {
        sm.level = nrem > 0 ? 1 << 30 : -1;  // stays when all members of the last front are taken, or none
        sm.level_take = sm.level_all = 0;
        sm.bin = -1;
        sm.bin_take = 0;
    }
    grp.sync();
    // direction counts; a member's slot in its direction comes from the count
    for (int i = gt; i < np; i += T) {
        const int r = idx[i];
        niche_mark(S.mask, gidx[i]);
        if (r >= 0 && r < H) atomicAdd(S.rho + r, 1);
    }
    int bucket[kNsItems], slot[kNsItems];
#pragma unroll
    for (int j = 0; j < kNsItems; ++j) {
        const int p = gt + j * T;
        if (p - lane >= nl) break;  // warp-uniform
        const bool valid = p < nl;
        int b = -1;
        if (valid) {
            const int r = idx[np + p];
            b = (r >= 0 && r < H) ? r : H;
        }
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, b);
        const int leader = __ffs(peers) - 1;
        int base = 0;
        if (valid && lane == leader) base = atomicAdd(S.last + b, __popc(peers));
        base = __shfl_sync(0xFFFFFFFFu, base, leader);
        bucket[j] = b;
        slot[j] = base + __popc(peers & ((1u << lane) - 1u));
    }
    grp.sync();
    // first position of each direction: every CTA scans a segment of directions
    const int per = (((H + 1 + C - 1) / C) + 3) & ~3;
    {
        const int lo = c * per, hi = min(H + 1, lo + per);
        int carry = 0, big = 0;
        unsigned long long work = 0;
        for (int b0 = lo; b0 < hi; b0 += 4 * THREADS) {
            const int b = b0 + 4 * tid;
            int v[4] = {0, 0, 0, 0};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (b + k < hi) v[k] = __ldcg(S.last + b + k);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                big = max(big, v[k]);
                work += (unsigned long long)v[k] * (unsigned long long)v[k];
            }
            int total;
            int at = carry + niche_scan<THREADS>(v[0] + v[1] + v[2] + v[3], sm.wsum, &total);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (b + k < hi) __stcg(S.start + b + k, at);
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
        if (tid == 0) {
            for (int w = 1; w < THREADS / 32; ++w) {
                big = max(big, sm.wmax[w]);
                work += sm.wsum64[w];
            }
            sm.seg_total = carry;
            sm.seg_max = big;
            sm.seg_work = work;
        }
    }
    grp.sync();
    if (tid == 0) {
        int at = 0, big = 0;
        unsigned long long work = 0;
        for (int r = 0; r < C; ++r) {
            sm.seg_off[r] = at;
            at += *grp.map(&sm.seg_total, r);
            big = max(big, *grp.map(&sm.seg_max, r));
            work += *grp.map(&sm.seg_work, r);
        }
        sm.fallback = (big > kNsMaxBucket || work > kNsMaxWork) ? 1 : 0;
    }
    __syncthreads();
    if (sm.fallback) {  // the same in every CTA
        grp.sync();     // the segment words were read everywhere
        return false;
    }
    // members into their direction's bucket, keyed by (distance, member)
#pragma unroll
    for (int j = 0; j < kNsItems; ++j) {
        const int p = gt + j * T;
        if (p >= nl) break;
        const int b = bucket[j];
        const int pos = sm.seg_off[b / per] + __ldcg(S.start + b) + slot[j];
        __stcg(S.key_a + pos, ((uint64_t)__float_as_uint(dist[np + p]) << 32) | (uint32_t)p);
        __stcg(S.dir_of + pos, b);
    }
    grp.sync();
    // order 1 inside the buckets, and the words of order 2
    int first[kNsItems], size[kNsItems], prior[kNsItems], member[kNsItems];
#pragma unroll
    for (int j = 0; j < kNsItems; ++j) {
        const int q = gt + j * T;
        if (q >= nl) break;
        const int b = S.dir_of[q];
        const int s = sm.seg_off[b / per] + S.start[b], n = S.last[b];
        const uint64_t k = S.key_a[q];
        const int pr = b < H ? S.rho[b] : 0;
        int rank = 0;
#pragma unroll 8
        for (int u = 0; u < n; ++u) rank += S.key_a[s + u] < k ? 1 : 0;
        const uint32_t rnd = splitmix_u32(off + (uint64_t)(s + rank), seed);
        const uint32_t low = (pr == 0 && rank == 0) ? 0u : (rnd | 1u);
        S.key_b[q] = ((uint64_t)low << 32) | (uint32_t)(s + rank);
        first[j] = s;
        size[j] = n;
        prior[j] = pr;
        member[j] = (int)(uint32_t)k;
    }
    grp.sync();
    // order 2 inside the buckets; the levels and words of order 3
    uint32_t word[kNsItems];
    int at[kNsItems];
#pragma unroll
    for (int j = 0; j < kNsItems; ++j) {
        const int q = gt + j * T;
        if (q >= nl) break;
        const int s = first[j], n = size[j];
        const uint64_t k = S.key_b[q];
        int rank = 0;
#pragma unroll 8
        for (int u = 0; u < n; ++u) rank += S.key_b[s + u] < k ? 1 : 0;
        at[j] = s + rank;
        word[j] = splitmix_u32(off + (uint64_t)nl + (uint64_t)(s + rank), seed);
        prior[j] += rank;  // the level
        atomicAdd(sm.hist + min(prior[j], kNsLevels - 1), 1);
    }
    grp.sync();
    const bool part = nrem > 0 && nrem < nl;
    if (part) {
        niche_threshold<THREADS>(grp, sm.hist, kNsLevels, nrem, sm.wsum, &sm.level, &sm.level_take, &sm.level_all);
        if (sm.level == kNsLevels - 1 && sm.level_take < sm.level_all) {  // levels above are not told apart
            grp.sync();
            return false;
        }
        if (sm.level_take < sm.level_all) {
#pragma unroll
            for (int j = 0; j < kNsItems; ++j) {
                if (gt + j * T >= nl) break;
                if (prior[j] == sm.level) atomicAdd(sm.bins + (word[j] >> 22), 1);
            }
        }
    }
    const int level = sm.level;
    const bool split = part && sm.level_take < sm.level_all;
    grp.sync();  // bins complete; the level histograms were read
    if (split) niche_threshold<THREADS>(grp, sm.bins, kNsBins, sm.level_take, sm.wsum, &sm.bin, &sm.bin_take, &sm.level_all);
    const int bin = sm.bin, bin_take = sm.bin_take;
#pragma unroll
    for (int j = 0; j < kNsItems; ++j) {
        if (gt + j * T >= nl) break;
        bool take = prior[j] < level || (prior[j] == level && !split);
        if (split && prior[j] == level) {
            const int wb = (int)(word[j] >> 22);
            take = wb < bin;
            if (wb == bin)  // ranked below
                S.key_a[atomicAdd(S.list_count, 1)] = ((uint64_t)word[j] << 32) | (uint32_t)at[j];
        }
        if (take) niche_mark(S.mask, gidx[np + member[j]]);
    }
    grp.sync();  // the list is complete; the bins were read
    if (split) {
        const int ln = __ldcg(S.list_count);
#pragma unroll
        for (int j = 0; j < kNsItems; ++j) {
            if (gt + j * T >= nl) break;
            if (prior[j] != level || (int)(word[j] >> 22) != bin) continue;
            const uint64_t k = ((uint64_t)word[j] << 32) | (uint32_t)at[j];
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
template <int THREADS, class G>
__device__ void niche_survivors(G& grp, NicheShared<THREADS>& sm, const uint32_t* mask, int n_mix,
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

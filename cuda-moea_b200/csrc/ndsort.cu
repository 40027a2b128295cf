// Constraint-dominance non-dominated sorting for sm_100a.
//
// Replaces run_ndsort / run_ndsort_init and the COO / CSR / bitmask paths of
// CUDA-MOEA (nat/src/selection/nsga3/kernels/non_dominated_sort.cu:158-1574).
// Same result (front index per point, -1 past the stop rule, index of the last
// front), different mechanism:
//
//  1. Sort of the points by (class, f0 | cv, S), a 56-bit key, in sorted tiles
//     and rank merges (nds_sort_tiles, nds_sort_merge), S the top 22 bits of the
//     order key of the FP32 sum f1 + ... + f_{M-1}.
//     Class 0 = feasible, 1 = feasible with a NaN objective, 2 = infeasible,
//     3 = infeasible with NaN violation.  FP32 addition rounds monotonically,
//     so a feasible dominator p of q has f0(p) <= f0(q) and S(p) <= S(q); runs
//     of equal keys in class 0 are then ordered lexicographically by
//     (f1, ..., f_{M-1}, index) (nds_tie_rank, nds_tie_fix_long).  In this
//     order every dominator of a point lies strictly before it, identical
//     vectors are adjacent, and a feasible dominator already satisfies
//     f0 <= q0.
//  2. For every sorted position q, dup[q] is the first position that cannot
//     dominate q: the start of q's run of identical objective vectors (class 0),
//     0 (class 1: nothing dominates it), the start of q's run of equal violation
//     (class 2) or the number of feasible points (class 3).  Then
//       infeasible q:  p dominates q  <=>  p < dup[q]
//       feasible q:    p dominates q  <=>  p < dup[q] and f_m(p) <= f_m(q), m >= 1
//     which is the reference relation (non_dominated_sort.cu:190-239) with one
//     integer and M-1 float comparisons per pair on the lower triangle only.
//  3. For every block of sorted positions (256 or 128; words of 32 in the
//     alternative) and every objective m >= 1 the positions are sorted by f_m
//     once, with the prefix sets of that order.  A row kernel then evaluates
//     the test for one dominatee per lane: the dominators of a block with
//     f_m(p) <= f_m(q) are one prefix set, found by a tree descent, and the
//     row words are the AND of those sets with the dup mask.  It stores for
//     every q the bit row of its dominators.
//  4. One cooperative persistent kernel peels the fronts: q joins front k when
//     no still-unassigned point is left in its row.  Each point remembers one
//     unassigned dominator ("blocker"); while that blocker is unassigned the
//     point is skipped without touching memory, so every row is scanned at most
//     once over the whole sort.  Fronts are separated by a bounded grid barrier
//     and the loop stops once `target` points are assigned, like the
//     reference's front propagation loops (:792-843, :1070-1279).
//
// Populations whose pair tests one CTA does in a few microseconds skip the
// order (nds_small): each thread keeps its point's dominators in registers.
#include <algorithm>

#include <cooperative_groups.h>
#include <cub/cub.cuh>

#include "internal.cuh"

namespace cg = cooperative_groups;

namespace moea {
namespace {

constexpr int kQB = 128;      // sorted positions (dominatees) per tile CTA
constexpr int kTileThreads = 256;
constexpr int kPeelThreads = 1024;
constexpr int kScanQueue = 1024;   // rows per CTA and front for the chunked scan
constexpr int kProbeWords = 16;    // row words probed below an assigned blocker
constexpr int kScanChunk = 512;    // words per chunk (16 per lane)
constexpr uint32_t kInfeasibleBit = 0x80000000u;
// Sort key: class (2 bits), the order key of f0 or of the violation (32
// bits), the top kSortSBits bits of the order key of S.  22 bits of S keep
// runs of equal keys as rare as 30 did and leave the eight bits that carry the
// lane in a tile's first sort (seven radix passes in the fused sort); with 14
// the runs grew and the tie fix-up cost more than the pass it saved.
constexpr int kSortSBits = 22;
constexpr int kSortKeyBits = 2 + 32 + kSortSBits;
constexpr int kSortClassShift = 32 + kSortSBits;

// ---------------------------------------------------------------------------
// 1. classification and lexicographic sort
// ---------------------------------------------------------------------------

// Sort key of point i of class cls with key0 low word val: class << 54 |
// val << 22 | S (class 0), kSortKeyBits bits, S the top 22 bits of the order key of the FP32 sum f1 + ... + f_{M-1}
// (monotone in every f_m; +inf + -inf (NaN) sorts with +inf sums).
__device__ __forceinline__ uint64_t sort_key(const SplitPop& pop, int M, int i, uint32_t cls, uint32_t val)
{
    uint32_t s30 = 0;
    if (cls == 0u) {
        float sum = 0.0f;
        for (int m = 1; m < M; ++m) sum = __fadd_rn(sum, pop.obj(m, i));
        s30 = float_order_key(isnan(sum) ? INFINITY : sum) >> 2;
    }
    return ((uint64_t)cls << kSortClassShift) | ((uint64_t)val << kSortSBits) | (s30 >> (30 - kSortSBits));
}

// Class of point i, and its key0 low word: the order key of f0 (class 0) or of
// the violation (class 2).
__device__ __forceinline__ uint32_t classify_point(const SplitPop& pop, int M, int i, uint32_t* val)
{
    const float cv = pop.cvv(i);
    *val = 0;
    if (cv == 0.0f) {
        bool nan = false;
        for (int m = 0; m < M; ++m) nan |= isnan(pop.obj(m, i));
        if (!nan) *val = float_order_key(pop.obj(0, i));
        return nan ? 1u : 0u;
    }
    if (isnan(cv)) return 3u;
    *val = float_order_key(cv);
    return 2u;
}

// Count of the len ascending values a[] that are <= x, len <= L, L a power of two.
__device__ __forceinline__ int count_le_step(const uint64_t* a, int len, int c, int s, uint64_t x)
{
    return (c + s <= len && a[c + s - 1] <= x) ? c + s : c;
}

// The sort of the keys, by rank instead of by digit.  A radix sort of the 56
// key bits needs seven passes over all keys, each a launch bound by its
// latency (9-10 us a pass at 4,000 to 65,536 points: 75 us with its histogram
// and its classification).  Here tiles of 1024 keys are sorted in one CTA each
// (a bitonic network per warp, then ranks by binary search in the CTA's other
// runs: 8 x 32 -> 256, 4 x 256 -> 1024), and each merge pass places every key
// by its rank in the seven other runs of its group: one pass up to 8192
// points, two up to 65536, with the seven searches of a key side by side.
// Equal keys keep their index order, as in the stable radix sort.
constexpr int kSortTile = 1024;
constexpr int kSortWays = 8;   // runs merged per pass

// key0[i] = class << 32 | order key of f0 (class 0) or cv (class 2); sorted
// tiles of (sort_key, index) into skey and perm.  Clears the sort's counters.
__device__ __forceinline__ void sort_tile(int tile, const SplitPop& pop, int M, uint64_t* __restrict__ key0,
                                          uint64_t* __restrict__ skey, int* __restrict__ perm,
                                          int* __restrict__ counters)
{
    __shared__ uint64_t s_a[kSortTile], s_b[kSortTile];
    __shared__ unsigned short s_i[kSortTile];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int base = tile * kSortTile, i = base + t;
    if (tile == 0 && t < 20 && (t < 5 || (t >= 10 && t <= 13) || t >= 16)) counters[t] = 0;
    uint64_t key = (1ull << kSortKeyBits) - 1ull;  // padding: above every real key
    if (i < pop.n) {
        uint32_t val;
        const uint32_t cls = classify_point(pop, M, i, &val);
        key0[i] = ((uint64_t)cls << 32) | val;
        key = sort_key(pop, M, i, cls, val);
    }
    uint64_t v = (key << 8) | (unsigned)lane;  // 56 + 8 bits; every real key is positive
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const uint64_t o = __shfl_xor_sync(0xFFFFFFFFu, v, j);
            const bool take_min = ((lane & j) == 0) == ((lane & k) == 0);
            v = take_min ? (o < v ? o : v) : (o > v ? o : v);
        }
    }
    s_a[t] = v;
    __syncthreads();
    {
        const uint64_t hi = v | 0xFFull, lo = (v & ~0xFFull) - 1ull;  // counts of <= key and < key
        const int w0 = warp & ~7;
        int c[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) c[r] = 0;
#pragma unroll
        for (int s = 16; s >= 1; s >>= 1)
#pragma unroll
            for (int r = 0; r < 8; ++r)
                c[r] = count_le_step(s_a + (w0 + r) * 32, 32, c[r], s, w0 + r < warp ? hi : lo);
        int rank = lane;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            c[r] = count_le_step(s_a + (w0 + r) * 32, 32, c[r], 1, w0 + r < warp ? hi : lo);
            if (w0 + r != warp) rank += c[r];
        }
        s_b[w0 * 32 + rank] = v & ~0xFFull;
        s_i[w0 * 32 + rank] = (unsigned short)(warp * 32 + (int)(v & 31ull));
    }
    __syncthreads();
    v = s_b[t];
    const int g = t >> 8;
    int c[4] = {0, 0, 0, 0};
#pragma unroll
    for (int s = 128; s >= 1; s >>= 1)
#pragma unroll
        for (int r = 0; r < 4; ++r) c[r] = count_le_step(s_b + r * 256, 256, c[r], s, r < g ? v : v - 1ull);
    int rank = t & 255;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        c[r] = count_le_step(s_b + r * 256, 256, c[r], 1, r < g ? v : v - 1ull);
        if (r != g) rank += c[r];
    }
    if (base + rank < pop.n) {
        skey[base + rank] = v >> 8;
        perm[base + rank] = base + (int)s_i[t];
    }
}

__global__ void __launch_bounds__(kSortTile)
nds_sort_tiles(SplitPop pop, int M, uint64_t* __restrict__ key0, uint64_t* __restrict__ skey, int* __restrict__ perm,
               int* __restrict__ counters)
{
    sort_tile(blockIdx.x, pop, M, key0, skey, perm, counters);
}

// Key i of sorted runs of L keys (L a power of two) to its place among the
// kSortWays runs of its group.
__device__ __forceinline__ void sort_merge_key(int i, const uint64_t* __restrict__ key_in,
                                               const int* __restrict__ perm_in, uint64_t* __restrict__ key_out,
                                               int* __restrict__ perm_out, int n, int L)
{
    const uint64_t key = key_in[i];
    const int run = i / L, r0 = run & ~(kSortWays - 1);
    const long long first = (long long)r0 * L;
    int c[kSortWays], len[kSortWays];
#pragma unroll
    for (int r = 0; r < kSortWays; ++r) {
        const long long left = (long long)n - (first + (long long)r * L);
        c[r] = 0;
        len[r] = (r0 + r == run || left <= 0) ? 0 : (int)(left < L ? left : L);
    }
    for (int s = L >> 1; s >= 1; s >>= 1)
#pragma unroll
        for (int r = 0; r < kSortWays; ++r)
            c[r] = count_le_step(key_in + first + (long long)r * L, len[r], c[r], s, r0 + r < run ? key : key - 1ull);
    long long at = first + (i - (long long)run * L);
#pragma unroll
    for (int r = 0; r < kSortWays; ++r)
        at += count_le_step(key_in + first + (long long)r * L, len[r], c[r], 1, r0 + r < run ? key : key - 1ull);
    key_out[at] = key;
    perm_out[at] = perm_in[i];
}

__global__ void __launch_bounds__(256)
nds_sort_merge(const uint64_t* __restrict__ key_in, const int* __restrict__ perm_in, uint64_t* __restrict__ key_out,
               int* __restrict__ perm_out, int n, int L)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) sort_merge_key(i, key_in, perm_in, key_out, perm_out, n, L);
}

// Total order inside a run of equal sort keys of class 0: lexicographic on
// the order keys of f1 .. f_{M-1}, then the point index.
__device__ __forceinline__ bool tie_less(const SplitPop& pop, int M, int a, int b)
{
    for (int m = 1; m < M; ++m) {
        const uint32_t ka = float_order_key(pop.obj(m, a)), kb = float_order_key(pop.obj(m, b));
        if (ka != kb) return ka < kb;
    }
    return a < b;
}

constexpr int kTieShort = 32;         // runs up to this length: one thread, insertion sort
constexpr int kTieLongThreads = 1024;
constexpr int kTieLongCtas = 64;        // CTAs of nds_tie_fix_long, each taking runs in turn
constexpr int kTieSmemSort = 4096;    // longer runs: bitonic in shared memory up to this size

// Runs of equal keys in class 0 into lexicographic order: every member of a run
// of at most kTieShort counts the members before it; longer runs are copied
// and listed for nds_tie_fix_long.  Every lane of the warp calls, with active
// false past the last point.  The lanes of the warp step through their runs
// together, and no lane leaves a comparison early: lanes that each followed their
// own loops ran one after another (5000 points of 243 vectors of five objectives:
// 258 us, 16 now; points without ties 3-4 us either way).
__device__ __forceinline__ void tie_rank(int pos, bool active, const SplitPop& pop, int M,
                                         const uint64_t* __restrict__ skey, const int* __restrict__ perm_in,
                                         int* __restrict__ perm_out, int* __restrict__ long_runs,
                                         int* __restrict__ n_long)
{
    const int n = pop.n;
    const uint64_t k = active ? skey[pos] : 0ull;
    const int pt = active ? perm_in[pos] : 0;
    const bool ranked = active && (k >> kSortClassShift) == 0u;
    int a = pos, b = pos + 1;  // the run, as far as kTieShort reaches
    bool more = ranked;
    while (__any_sync(0xFFFFFFFFu, more)) {
        more = more && a > 0 && pos - a <= kTieShort && skey[a - 1] == k;
        if (more) --a;
    }
    more = ranked;
    while (__any_sync(0xFFFFFFFFu, more)) {
        more = more && b < n && b - a <= kTieShort && skey[b] == k;
        if (more) ++b;
    }
    int to = pos, members = 0;
    if (ranked && b - a > kTieShort) {
        if (a == pos) long_runs[atomicAdd(n_long, 1)] = pos;
    } else if (ranked && b - a > 1) {
        to = a;
        members = b - a;
    }
    const int steps = __reduce_max_sync(0xFFFFFFFFu, members);
    for (int i = 0; i < steps; ++i) {
        if (i < members) {
            const int other = perm_in[a + i];
            bool less = false, equal = true;
#pragma unroll 4
            for (int m = 1; m < M; ++m) {
                const uint32_t ka = float_order_key(pop.obj(m, other)), kb = float_order_key(pop.obj(m, pt));
                less |= equal && ka < kb;
                equal &= ka == kb;
            }
            to += (less || (equal && other < pt)) ? 1 : 0;
        }
        __syncwarp();
    }
    if (active) perm_out[to] = pt;
}

__global__ void nds_tie_rank(SplitPop pop, int M, const uint64_t* __restrict__ skey, const int* __restrict__ perm_in,
                             int* __restrict__ perm_out, int* __restrict__ long_runs, int* __restrict__ n_long)
{
    const int pos = blockIdx.x * blockDim.x + threadIdx.x;
    tie_rank(pos, pos < pop.n, pop, M, skey, perm_in, perm_out, long_runs, n_long);
}

// Ascending bitonic network over a[0, L) with virtual +inf padding to the
// power of two P >= L (pairs reaching past L are skipped: +inf already sits
// last).  Every merge opens with the mirrored comparison, so all blocks sort
// ascending.  Called by every thread of the CTA.
__device__ void tie_bitonic(const SplitPop& pop, int M, int* a, int L)
{
    int P = 1;
    while (P < L) P <<= 1;
    for (int k = 2; k <= P; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int q = threadIdx.x; q < P / 2; q += blockDim.x) {
                int i, p;
                if (j == k >> 1) {  // mirror inside the block of k
                    const int half = k >> 1;
                    i = (q / half) * k + (q % half);
                    p = (q / half) * k + (k - 1 - (q % half));
                } else {
                    i = (q / j) * 2 * j + (q % j);
                    p = i + j;
                }
                if (p < L) {
                    const int x = a[i], y = a[p];
                    if (tie_less(pop, M, y, x)) {
                        a[i] = y;
                        a[p] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// One CTA per listed run longer than kTieShort (first, first + step, ... of the
// list): its length, then a bitonic sort unless the run is already in order
// (runs of identical vectors are).
__device__ __forceinline__ void tie_fix_long(int first, int step, const SplitPop& pop, int M,
                                             const uint64_t* __restrict__ skey, int* __restrict__ perm,
                                             const int* __restrict__ long_runs, const int* __restrict__ n_long)
{
    __shared__ int s_arr[kTieSmemSort];
    __shared__ int s_len, s_unsorted;
    const int n = pop.n;
    const int count = *n_long;
    for (int r = first; r < count; r += step) {
        const int start = long_runs[r];
        const uint64_t k = skey[start];
        if (threadIdx.x == 0) {
            s_len = n - start;
            s_unsorted = 0;
        }
        __syncthreads();
        for (int base = start; base < n; base += blockDim.x) {
            const int pos = base + threadIdx.x;
            if (pos < n && skey[pos] != k) atomicMin(&s_len, pos - start);
            __syncthreads();
            const bool found = s_len < n - start;
            __syncthreads();  // every thread has read s_len before the next atomicMin
            if (found) break;
        }
        const int L = s_len;
        int* a = perm + start;
        for (int x = threadIdx.x; x + 1 < L; x += blockDim.x)
            if (tie_less(pop, M, a[x + 1], a[x])) s_unsorted = 1;
        __syncthreads();
        if (s_unsorted) {
            if (L <= kTieSmemSort) {
                for (int x = threadIdx.x; x < L; x += blockDim.x) s_arr[x] = a[x];
                __syncthreads();
                tie_bitonic(pop, M, s_arr, L);
                for (int x = threadIdx.x; x < L; x += blockDim.x) a[x] = s_arr[x];
            } else {
                tie_bitonic(pop, M, a, L);
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kTieLongThreads)
nds_tie_fix_long(SplitPop pop, int M, const uint64_t* __restrict__ skey, int* __restrict__ perm,
                 const int* __restrict__ long_runs, const int* __restrict__ n_long)
{
    tie_fix_long(blockIdx.x, gridDim.x, pop, M, skey, perm, long_runs, n_long);
}

// Sorted copy of objectives 1..M-1, the dup positions, the peel's initial state
// and the class counts.  The start of a run of identical vectors (class 0) or
// violations (class 2) is found by doubling steps back and a binary search:
// positions between two identical ones are identical, and nearly every run has
// one member, so no scan over the positions is needed.
__device__ __forceinline__ void finalize_row(int pos, const SplitPop& pop, int M, const uint64_t* __restrict__ key0,
                                             const uint64_t* __restrict__ skey, const int* __restrict__ perm,
                                             float* __restrict__ sf, int sf_stride, int* __restrict__ counters,
                                             int* __restrict__ qinfo, int* __restrict__ blocker,
                                             int* __restrict__ front_sorted)
{
    const int n = pop.n;
    const int pt = perm[pos];
    const uint64_t k0 = key0[pt];
    const uint32_t cls = (uint32_t)(k0 >> 32);
    for (int m = 1; m < M; ++m) sf[(size_t)(m - 1) * sf_stride + pos] = pop.obj(m, pt);
    auto same = [&](int p) {
        const int pp = perm[p];
        if (key0[pp] != k0) return false;
        bool eq = true;
        if (cls == 0u)
            for (int m = 1; m < M; ++m) eq &= float_order_key(pop.obj(m, pt)) == float_order_key(pop.obj(m, pp));
        return eq;
    };
    uint32_t d = 0u;
    if (cls == 0u || cls == 2u) {
        int start = pos;
        if (pos > 0 && same(pos - 1)) {
            start = pos - 1;
            int step = 2;
            while (pos - step >= 0 && same(pos - step)) {
                start = pos - step;
                step *= 2;
            }
            int lo = max(-1, pos - step);  // differs (or before the first)
            while (start - lo > 1) {
                const int mid = (start + lo) >> 1;
                if (same(mid)) start = mid;
                else lo = mid;
            }
        }
        d = (uint32_t)start | (cls == 2u ? kInfeasibleBit : 0u);
    } else if (cls == 3u) {
        int lo = 0, hi = pos;  // first position of an infeasible class
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if ((skey[mid] >> kSortClassShift) >= 2u) hi = mid;
            else lo = mid + 1;
        }
        d = (uint32_t)lo | kInfeasibleBit;
    }
    qinfo[pos] = (int)d;
    blocker[pos] = -1;
    front_sorted[pos] = -1;
    // [0] feasible points, [10] class 2, [11] class 3, from the class boundaries
    const uint32_t before = pos > 0 ? (uint32_t)(skey[pos - 1] >> kSortClassShift) : 0u;
    if (cls >= 2u && before < 2u) {
        counters[0] = pos;
        atomicAdd(counters + 10, -pos);
    }
    if (cls == 3u && before < 3u) {
        counters[11] = n - pos;
        atomicAdd(counters + 10, pos);
    }
    if (pos == n - 1) {
        if (cls < 2u) counters[0] = n;
        if (cls == 2u) atomicAdd(counters + 10, n);
    }
}

// Also empties the peel's front masks.
__global__ void nds_finalize_rows(SplitPop pop, int M, const uint64_t* __restrict__ key0,
                                  const uint64_t* __restrict__ skey, const int* __restrict__ perm,
                                  float* __restrict__ sf, int sf_stride, int* __restrict__ counters,
                                  int* __restrict__ qinfo, int* __restrict__ blocker, int* __restrict__ front_sorted,
                                  uint32_t* __restrict__ fmask, int fmask_words)
{
    const int pos = blockIdx.x * blockDim.x + threadIdx.x;
    for (int w = pos; w < fmask_words; w += gridDim.x * blockDim.x) fmask[w] = 0u;
    if (pos < pop.n)
        finalize_row(pos, pop, M, key0, skey, perm, sf, sf_stride, counters, qinfo, blocker, front_sorted);
}

// ---------------------------------------------------------------------------
// 2. dominance rows
// ---------------------------------------------------------------------------

// Order key of an objective value for the dominance test; NaN maps above
// every other key so that a NaN dominator never satisfies key(p) <= key(q).
__device__ __forceinline__ uint32_t dom_key(float f)
{
    return isnan(f) ? 0xFFFFFFFFu : float_order_key(f);
}

// Per word of 32 sorted positions and per objective m >= 1: the 32 order
// keys in ascending order (keys[m][32 w + k]) and the prefix sets
// bits[m][33 w + k] = positions (bit j = position 32 w + j) of the k smallest
// keys, k = 0..32.  For a value v, the positions of the word whose objective
// is <= v are bits[m][33 w + c] with c = #{keys <= key(v)}: ties at the
// boundary all lie inside the prefix, whatever their order.  Positions >= n
// get the NaN key.  One warp per (word, objective): bitonic sort of
// (key, lane) pairs, then an inclusive OR-scan of the lane bits.
__device__ __forceinline__ void chunk_warp(int gw, int lane, const float* __restrict__ sf, int sf_stride,
                                           int n, int W, uint32_t* __restrict__ ckeys,
                                           uint32_t* __restrict__ cbits)
{
    const int m = gw / W, w = gw - m * W;
    const int p = w * 32 + lane;
    const uint32_t key = (p < n) ? dom_key(sf[(size_t)m * sf_stride + p]) : 0xFFFFFFFFu;
    unsigned long long kv = ((unsigned long long)key << 32) | (unsigned)lane;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const unsigned long long o = __shfl_xor_sync(0xFFFFFFFFu, kv, j);
            const bool take_min = ((lane & j) == 0) == ((lane & k) == 0);
            kv = take_min ? (o < kv ? o : kv) : (o > kv ? o : kv);
        }
    }
    uint32_t pre = 1u << (unsigned)(kv & 31ull);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, pre, o);
        if (lane >= o) pre |= t;
    }
    ckeys[(size_t)m * W * 32 + (size_t)w * 32 + lane] = (uint32_t)(kv >> 32);
    uint32_t* b = cbits + (size_t)m * W * 33 + (size_t)w * 33;
    b[lane + 1] = pre;
    if (lane == 0) b[0] = 0u;
}

__global__ void nds_chunks(const float* __restrict__ sf, int sf_stride, int n, int W, int MF,
                           uint32_t* __restrict__ ckeys, uint32_t* __restrict__ cbits)
{
    const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (gw >= W * MF) return;
    chunk_warp(gw, threadIdx.x & 31, sf, sf_stride, n, W, ckeys, cbits);
}

// Dominator words per tile CTA (32 positions each), sized so that the staged
// word tables and the transposed output fit in 48 KB of shared memory.
template <int M>
struct TileCfg {
    static constexpr int kPW = (M <= 4) ? 32 : ((M <= 8) ? 16 : 8);
    static constexpr int kMF = (M > 1) ? M - 1 : 1;   // objectives 1..M-1
};

// Count of the 32 ascending keys at shared address a that are <= v, as the
// byte offset 4 * count: binary search with steps of 16, 8, 4, 2, 1 keys and
// a last probe that reaches 32 only from 31.  Each probe is one shared load
// with an immediate offset, one compare and one predicated add.
__device__ __forceinline__ uint32_t word_count_bytes(uint32_t a, uint32_t v)
{
    const uint32_t a0 = a;
    asm("{\n\t.reg .pred p;\n\t.reg .u32 t;\n\t"
        "ld.shared.u32 t, [%0+60];\n\tsetp.le.u32 p, t, %1;\n\t@p add.u32 %0, %0, 64;\n\t"
        "ld.shared.u32 t, [%0+28];\n\tsetp.le.u32 p, t, %1;\n\t@p add.u32 %0, %0, 32;\n\t"
        "ld.shared.u32 t, [%0+12];\n\tsetp.le.u32 p, t, %1;\n\t@p add.u32 %0, %0, 16;\n\t"
        "ld.shared.u32 t, [%0+4];\n\tsetp.le.u32 p, t, %1;\n\t@p add.u32 %0, %0, 8;\n\t"
        "ld.shared.u32 t, [%0];\n\tsetp.le.u32 p, t, %1;\n\t@p add.u32 %0, %0, 4;\n\t"
        "ld.shared.u32 t, [%0];\n\tsetp.le.u32 p, t, %1;\n\t@p add.u32 %0, %0, 4;\n\t}"
        : "+r"(a)
        : "r"(v)
        : "memory");
    return a - a0;
}

__device__ __forceinline__ uint32_t ld_shared_u32(uint32_t a)
{
    uint32_t x;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(a) : "memory");
    return x;
}

// One CTA covers kQB dominatees q (one per lane of warps 0-3, again of warps
// 4-7) against kPW words of dominator positions p (the first half of the
// words for warps 0-3, the second half for warps 4-7).  The word tables of
// nds_chunks are staged in shared memory; for each word and objective a lane
// finds the count of dominator keys <= its own key with a six-probe search
// and ANDs the prefix set of that count into its row word, so a word of 32
// pairs costs about 13 integer operations per objective instead of 32
// comparisons.  Words are transposed through shared memory and written as
// coalesced row segments.  The epilogue raises blocker[q] to the highest
// dominator position seen, so that after the kernel blocker[q] == -1 exactly
// for the points that nothing dominates (front 0).
template <int M, int PW = TileCfg<M>::kPW>
__device__ __forceinline__ void tile_block(int bx, int by, const float* __restrict__ sf, int sf_stride,
                                           const int* __restrict__ qinfo,
                                           const uint32_t* __restrict__ ckeys,
                                           const uint32_t* __restrict__ cbits, int n, int W, int Wc,
                                           uint32_t* __restrict__ rows, int* __restrict__ blocker)
{
    constexpr int MF = TileCfg<M>::kMF;
    const int q0 = by * kQB;
    if (q0 >= n) return;
    const int qend = min(q0 + kQB, n);
    // dominators of the block lie at positions < qend - 1
    const int nwords = (qend - 1 + 31) >> 5;
    const int w0 = bx * PW;
    if (w0 >= nwords) return;
    const int wcount = min(PW, nwords - w0);

    __shared__ uint32_t s_key[MF][PW * 32];
    __shared__ uint32_t s_bits[MF][PW * 33];
    __shared__ uint32_t so[kQB][PW + 1];
    if (M > 1) {
        for (int t = threadIdx.x; t < wcount * 32; t += kTileThreads) {
#pragma unroll
            for (int m = 0; m < MF; ++m) s_key[m][t] = ckeys[(size_t)m * Wc * 32 + (size_t)w0 * 32 + t];
        }
        for (int t = threadIdx.x; t < wcount * 33; t += kTileThreads) {
#pragma unroll
            for (int m = 0; m < MF; ++m) s_bits[m][t] = cbits[(size_t)m * Wc * 33 + (size_t)w0 * 33 + t];
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ql = (warp & 3) * 32 + lane;
    const int q = q0 + ql;
    uint32_t qk[MF];
    int dup = 0;
    bool inf = false;
#pragma unroll
    for (int m = 0; m < MF; ++m) qk[m] = 0u;
    if (q < n) {
        if (M > 1) {
#pragma unroll
            for (int m = 0; m < MF; ++m) qk[m] = dom_key(sf[(size_t)m * sf_stride + q]);
        }
        const uint32_t info = (uint32_t)qinfo[q];
        inf = (info & kInfeasibleBit) != 0u;
        dup = (int)(info & ~kInfeasibleBit);
    }
    __syncthreads();

    constexpr int kHalf = PW / 2;
    const int wb = (warp >> 2) * kHalf;
    const int wend = min(wb + kHalf, wcount);
    // words whose 32 positions lie below dup[q] for every lane of the warp
    // need no dup mask (most of them)
    uint32_t key_addr[MF], bits_addr[MF];
#pragma unroll
    for (int m = 0; m < MF; ++m) {
        key_addr[m] = (uint32_t)__cvta_generic_to_shared(&s_key[m][0]);
        bits_addr[m] = (uint32_t)__cvta_generic_to_shared(&s_bits[m][0]);
    }
    const int lane_full = (q < n) ? (dup >> 5) - w0 : 0x7FFFFFFF;
    const int wfull = min(wend, max(wb, __reduce_min_sync(0xFFFFFFFFu, lane_full)));
    // Every lane searches (the masks decide).  The prefix set of count c
    // sits at byte 4 c of the word's bit table.  Running shared addresses
    // step by one word table per iteration.
#pragma unroll
    for (int m = 0; m < MF; ++m) {
        key_addr[m] += (uint32_t)wb * 128u;
        bits_addr[m] += (uint32_t)wb * 132u;
    }
    uint32_t* so_row = &so[ql][0];
    const uint32_t infm = inf ? 0xFFFFFFFFu : 0u;
    auto word_bits = [&]() -> uint32_t {
        uint32_t cmp = 0xFFFFFFFFu;
        if (M > 1) {
#pragma unroll
            for (int m = 0; m < MF; ++m) {
                const uint32_t off = word_count_bytes(key_addr[m], qk[m]);
                cmp &= ld_shared_u32(bits_addr[m] + off);
                key_addr[m] += 128u;
                bits_addr[m] += 132u;
            }
        }
        return cmp | infm;
    };
    // The peel never reaches an infeasible point (each is dominated by every
    // feasible one, and the peel ends with the feasible fronts), so its row is
    // never read: a warp of infeasible q (they sort last, so whole warps are)
    // computes nothing, and a CTA of them stores nothing.  Rows of infeasible
    // q in a mixed CTA hold unspecified words.
    const bool all_inf = __all_sync(0xFFFFFFFFu, inf || q >= n);
    if (!all_inf) {
        int wl = wb;
        for (; wl < wfull; ++wl) so_row[wl] = word_bits();   // all positions below dup[q]
        for (; wl < wend; ++wl) {
            // positions p < dup[q] of this word
            const int rem = dup - (w0 + wl) * 32;
            const uint32_t mask = rem >= 32 ? 0xFFFFFFFFu : (rem <= 0 ? 0u : ((1u << rem) - 1u));
            so_row[wl] = mask & word_bits();
        }
    }
    if (__syncthreads_and(all_inf)) return;
    for (int r = warp; r < kQB; r += kTileThreads / 32) {
        const int pos = q0 + r;
        if (pos >= n) break;
        const uint32_t word = (lane < wcount) ? so[r][lane] : 0u;
        if (lane < wcount) rows[(size_t)pos * W + w0 + lane] = word;
        const unsigned nz = __ballot_sync(0xFFFFFFFFu, word != 0u);
        if (nz && lane == 31 - __clz(nz))
            atomicMax(blocker + pos, (w0 + lane) * 32 + (31 - __clz(word)));
    }
}

template <int M>
__global__ void __launch_bounds__(kTileThreads)
nds_tiles(const float* __restrict__ sf, int sf_stride, const int* __restrict__ qinfo,
          const uint32_t* __restrict__ ckeys, const uint32_t* __restrict__ cbits, int n, int W,
          int Wc, uint32_t* __restrict__ rows, int* __restrict__ blocker)
{
    tile_block<M>(blockIdx.x, blockIdx.y, sf, sf_stride, qinfo, ckeys, cbits, n, W, Wc, rows, blocker);
}

// ---------------------------------------------------------------------------
// 3. front peeling
// ---------------------------------------------------------------------------

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ int ld_acquire_gpu(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid barrier over co-resident CTAs.  The arrivals count up during one
// launch (counters[4] is zeroed before it): barrier number `epoch` is passed
// when the count reaches epoch * nblocks, so no CTA resets or releases
// anything and the wait ends one acquire load after the last arrival.
// Waits at most limit_ns (2 s in the peel), then records kDevBarrierTimeout
// in the status word and returns false.  Every thread of the CTA passes the
// same epoch.
__device__ bool grid_barrier(int* counters, unsigned nblocks, int epoch,
                             unsigned long long limit_ns = 2000000000ull)
{
    __shared__ int s_ok;
    __syncthreads();
    if (nblocks == 1) {  // single-CTA peel: a block barrier suffices
        __syncthreads();
        return true;
    }
    if (threadIdx.x == 0) {
        const int target = epoch * (int)nblocks;
        // release at GPU scope: with the CTA barrier above it orders every
        // thread's earlier writes before the arrival
        asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(counters + 4) : "memory");
        int ok = 1;
        const unsigned long long t0 = global_ns();
        while (ld_acquire_gpu(counters + 4) < target) {
            if (*((volatile int*)counters + 6) != 0) { ok = 0; break; }
            if (global_ns() - t0 > limit_ns) {
                atomicExch(counters + 6, kDevBarrierTimeout);
                ok = 0;
                break;
            }
            __nanosleep(32);
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Marks the free lanes of a warp, all in the 32-position group of word gw,
// as members of front k: one atomicOr into the front's mask per warp.
__device__ __forceinline__ void peel_mark_group(bool is_free, int q, int gw, int k, int lane, uint32_t* G,
                                                int* front_sorted)
{
    const unsigned fm = __ballot_sync(0xFFFFFFFFu, is_free);
    if (!fm) return;
    if (lane == 0) atomicOr(G + gw, fm);
    if (is_free) front_sorted[q] = k;
}

// Body of the peel, run by CTA `block` of `nblocks` co-resident CTAs; U is the
// CTA's bitmask of unassigned positions (W words of shared memory), the same
// in every CTA.  Per front k:
//   1. groups: every alive point whose blocker (an unassigned dominator) was
//      assigned probes the blocker's row word and the one below; a hit is the
//      new blocker, no dominator at all makes the point free, and the other
//      rows are queued;
//   2. the CTA scans its queued rows in chunks of kScanChunk words, level by
//      level (the top chunk of every row first);
//   3. free points set their bit in the front's mask (fmask, three in
//      rotation, so no CTA appends to a shared list); after one grid barrier
//      every CTA removes the front from U and counts it.
template <int kInflight>
__device__ __forceinline__ void peel_body(int block, int nblocks, uint32_t* U,
                                          const uint32_t* __restrict__ rows, int W, int n, int target,
                                          const int* __restrict__ qinfo, int* __restrict__ blocker,
                                          int* __restrict__ front_sorted, uint32_t* __restrict__ fmask,
                                          int* counters)
{
    __shared__ int s_nscan, s_ntask;
    __shared__ int s_sq[kScanQueue], s_sw[kScanQueue], s_found[kScanQueue];
    __shared__ int s_wsum[32];
    if (threadIdx.x == 0) s_nscan = 0;
    // Feasible positions come first in the sorted order.  Infeasible ones are
    // never assigned here (each is dominated by every feasible point, and the
    // peel ends with the feasible fronts or the target), so they start out of
    // the unassigned set: they are never examined and their rows never read.
    const int nf = min(n, counters[0]);
    for (int w = threadIdx.x; w < W; w += blockDim.x) {
        const int lo = w * 32;
        U[w] = (lo + 32 <= nf) ? 0xFFFFFFFFu : (lo >= nf ? 0u : ((1u << (nf - lo)) - 1u));
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    // groups of 32 positions interleaved over the CTAs: every CTA holds low
    // (short rows) and high (long rows) positions alike
    const int gwarp = warp * nblocks + block;
    const int twarps = nblocks * wpb;
    const int ngroups = (n + 31) >> 5;
    int total = 0, k = 0, epoch = 0;
    // With fewer feasible points than the target, the peel covers the
    // feasible fronts only; the infeasible fronts follow in closed form
    // (nds_infeasible_fronts).  Without feasible points there is nothing to peel.
    const int feasible = counters[0];
    const bool feasible_only = feasible < target;
    __syncthreads();
    if (feasible_only && feasible == 0) {
        if (block == 0 && threadIdx.x == 0) {
            counters[2] = -1;
            counters[12] = -1;
        }
        return;
    }

    for (;;) {
        uint32_t* G = fmask + (size_t)(k % 3) * W;  // members of front k
        // the mask front k + 1 will write: last read (as front k - 2's) before
        // the barrier of front k - 1, written again only after this front's
        const uint32_t nextw = (uint32_t)((k + 1) % 3);
        for (int w = block * blockDim.x + threadIdx.x; w < W; w += nblocks * blockDim.x)
            fmask[(size_t)nextw * W + w] = 0u;
        for (int g0 = gwarp; g0 < ngroups; g0 += twarps * kInflight) {
            int qv[kInflight], bv[kInflight];
            uint32_t pw[kInflight][kProbeWords];
            bool alive[kInflight], probe[kInflight];
#pragma unroll
            for (int u = 0; u < kInflight; ++u) {
                const int g = g0 + u * twarps;
                const int q = g * 32 + lane;
                qv[u] = q;
                alive[u] = g < ngroups && q < n && ((U[q >> 5] >> (q & 31)) & 1u);
                // blocker[q] is an unassigned dominator of q, or -1 when nothing
                // dominates q; whichever CTA resolved q's row wrote it: read through L2
                bv[u] = alive[u] ? __ldcg(blocker + q) : -1;
            }
#pragma unroll
            for (int u = 0; u < kInflight; ++u) {
                const int b = bv[u];
                // blocker assigned: probe its word and the kProbeWords - 1
                // below it; bits above it were already free of unassigned
                // dominators
                probe[u] = alive[u] && b >= 0 && !((U[b >> 5] >> (b & 31)) & 1u);
#pragma unroll
                for (int i = 0; i < kProbeWords; ++i) pw[u][i] = 0u;
                if (probe[u]) {
                    const uint32_t* row = rows + (size_t)qv[u] * W;
                    const int w = b >> 5;
#pragma unroll
                    for (int i = 0; i < kProbeWords; ++i)
                        if (w - i >= 0) pw[u][i] = __ldg(row + w - i);
                }
            }
#pragma unroll
            for (int u = 0; u < kInflight; ++u) {
                const int g = g0 + u * twarps;
                if (g >= ngroups) break;  // warp-uniform
                const int q = qv[u];
                bool is_free = false, need = false;
                int start_w = -1;
                if (alive[u]) {
                    const int b = bv[u];
                    if (b < 0) {
                        is_free = true;
                    } else if (probe[u]) {
                        const int w = b >> 5;
                        int hit = -1;
#pragma unroll
                        for (int i = 0; i < kProbeWords; ++i) {
                            const uint32_t bits = (w - i >= 0) ? (pw[u][i] & U[w - i]) : 0u;
                            if (hit < 0 && bits) hit = (w - i) * 32 + (31 - __clz(bits));
                        }
                        if (hit >= 0) {
                            blocker[q] = hit;
                        } else if (w - kProbeWords < 0) {
                            is_free = true;
                        } else {
                            need = true;
                            start_w = w - kProbeWords;
                        }
                    }
                }
                // rows not resolved by the probe go to the CTA's list; when it
                // is full the whole warp scans each of them downwards
                if (need) {
                    const int slot = atomicAdd(&s_nscan, 1);
                    if (slot < kScanQueue) {
                        s_sq[slot] = qv[u];
                        s_sw[slot] = start_w;
                        need = false;
                    }
                }
                unsigned needm = __ballot_sync(0xFFFFFFFFu, need);
                while (needm) {
                    const int L = __ffs(needm) - 1;
                    needm &= needm - 1;
                    const int qL = g * 32 + L;
                    const uint32_t* row = rows + (size_t)qL * W;
                    const int sw = __shfl_sync(0xFFFFFFFFu, start_w, L);
                    int found = -1;
                    for (int w0 = sw; w0 >= 0 && found < 0; w0 -= 256) {
                        uint32_t acc[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int w = w0 - lane - 32 * i;
                            acc[i] = (w >= 0) ? (__ldg(row + w) & U[w]) : 0u;
                        }
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const unsigned nz = __ballot_sync(0xFFFFFFFFu, acc[i] != 0u);
                            if (nz) {
                                const int src = __ffs(nz) - 1;
                                const uint32_t bb = __shfl_sync(0xFFFFFFFFu, acc[i], src);
                                found = (w0 - src - 32 * i) * 32 + (31 - __clz(bb));
                                break;
                            }
                        }
                    }
                    if (lane == L) {
                        if (found >= 0) blocker[q] = found;
                        else is_free = true;
                    }
                }
                peel_mark_group(is_free, q, g, k, lane, G, front_sorted);
            }
        }
        __syncthreads();
        const int nscan = min(s_nscan, kScanQueue);
        if (nscan > 0) {
            // chunks of the queued rows: row s covers words sw[s]..0 in
            // chunks of kScanChunk from the top.  Tasks go level by level (the
            // top chunk of every row first), and a chunk is skipped once an
            // unassigned dominator above it has been found: the highest one
            // found is the same, and most rows end in their top chunk.  A hit
            // found lower down (a later chunk can finish first) skips nothing.
            if (warp == 0) {
                int levels = 0;
                for (int s0 = 0; s0 < nscan; s0 += 32) {
                    const int sidx = s0 + lane;
                    if (sidx < nscan) {
                        levels = max(levels, s_sw[sidx] / kScanChunk + 1);
                        s_found[sidx] = -1;
                    }
                }
#pragma unroll
                for (int o = 16; o; o >>= 1) levels = max(levels, __shfl_xor_sync(0xFFFFFFFFu, levels, o));
                if (lane == 0) s_ntask = levels * nscan;
            }
            __syncthreads();
            const int ntask = s_ntask;
            for (int task = warp; task < ntask; task += wpb) {
                const int level = task / nscan, lo = task - level * nscan;
                if (level > s_sw[lo] / kScanChunk) continue;
                const int top = s_sw[lo] - level * kScanChunk;
                // warp-uniform: the chunk scan below is warp-collective
                const int found_hi = __shfl_sync(0xFFFFFFFFu, *((volatile int*)s_found + lo), 0);
                if (found_hi > top * 32 + 31) continue;
                const uint32_t* row = rows + (size_t)s_sq[lo] * W;
                uint32_t acc[kScanChunk / 32];
#pragma unroll
                for (int i = 0; i < kScanChunk / 32; ++i) {
                    const int w = top - lane - 32 * i;
                    acc[i] = (w >= 0 && w > top - kScanChunk) ? (__ldg(row + w) & U[w]) : 0u;
                }
#pragma unroll
                for (int i = 0; i < kScanChunk / 32; ++i) {
                    const unsigned nz = __ballot_sync(0xFFFFFFFFu, acc[i] != 0u);
                    if (nz) {
                        const int src = __ffs(nz) - 1;
                        const uint32_t bb = __shfl_sync(0xFFFFFFFFu, acc[i], src);
                        if (lane == 0) atomicMax(s_found + lo, (top - src - 32 * i) * 32 + (31 - __clz(bb)));
                        break;
                    }
                }
            }
            __syncthreads();
            // highest unassigned dominator found: new blocker; none: free
            for (int s0 = 0; s0 < nscan; s0 += blockDim.x) {
                const int sidx = s0 + threadIdx.x;
                bool is_free = false;
                int q = 0;
                if (sidx < nscan) {
                    q = s_sq[sidx];
                    const int f = s_found[sidx];
                    if (f >= 0) blocker[q] = f;
                    else is_free = true;
                }
                if (is_free) {
                    atomicOr(G + (q >> 5), 1u << (q & 31));
                    front_sorted[q] = k;
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) s_nscan = 0;  // read again only after the barrier below
        if (!grid_barrier(counters, (unsigned)nblocks, ++epoch)) return;
        // front k is complete: remove it from U and count it
        int c = 0;
        for (int w0 = threadIdx.x; w0 < W; w0 += 4 * blockDim.x) {
            uint32_t g[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int w = w0 + i * blockDim.x;
                g[i] = (w < W) ? __ldcg(G + w) : 0u;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (g[i]) {
                    U[w0 + i * blockDim.x] &= ~g[i];
                    c += __popc(g[i]);
                }
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
        if (lane == 0) s_wsum[warp] = c;
        __syncthreads();
        int ck = 0;
        for (int w = 0; w < wpb; ++w) ck += s_wsum[w];
        __syncthreads();  // s_wsum is reused by the next front
        total += ck;
        if (total >= target || ck == 0 || (feasible_only && total >= feasible)) {
            if (block == 0 && threadIdx.x == 0) {
                counters[2] = k;
                counters[3] = total;
                counters[12] = k;
                if (ck == 0 && total < (feasible_only ? feasible : target))
                    atomicExch(counters + 6, kDevPeelInconsistent);
            }
            return;
        }
        ++k;
    }
}

__global__ void __launch_bounds__(kPeelThreads, 1)
nds_peel(const uint32_t* __restrict__ rows, int W, int n, int target, const int* __restrict__ qinfo,
         int* __restrict__ blocker, int* __restrict__ front_sorted, uint32_t* __restrict__ fmask,
         int* counters)
{
    extern __shared__ uint32_t U[];  // unassigned positions, one bit each
    peel_body<1>(blockIdx.x, gridDim.x, U, rows, W, n, target, qinfo, blocker, front_sorted, fmask, counters);
}

// ---- peel with lane-owned points ------------------------------------------
//
// When every warp of the grid owns at most one group of 32 positions
// (n <= 32 * 32 * CTAs), a lane keeps its point's state across the fronts:
// the blocker in a register and a window of at least kWin row words (the
// blocker's word and those below it) in shared memory, as three aligned
// 16-byte chunks.  The window is refilled with cp.async whenever fewer than
// kWin of its words lie at or below the blocker, so the copy lands while the
// grid waits at the barrier and the next front's probe reads only shared
// memory.  Row strides are multiples of four words (the workspace rounds
// them), which keeps every chunk 16-byte aligned.  Rows the window cannot settle go through the CTA's
// level-ordered scan as in peel_body.  The barrier carries the front sizes:
// a CTA adds (1 << 32) + (its free points) to one of two 64-bit words (front
// parity), so the front's size arrives with the barrier and no block-wide
// count is needed.  A CTA can run at most one front ahead of the slowest, so
// the word of front k holds only fronts k, k-2, ... when it is read.

constexpr int kWin = 8;        // row words cached per lane at and below its blocker
constexpr int kWinChunks = 3;  // 16-byte chunks of a window: 12 words from a multiple of 4
constexpr unsigned long long kPeelWaitNs = 2000000000ull;  // limit of one barrier wait

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void cp_async16(uint4* dst, const uint32_t* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Row words wlo .. wt of `row` into a lane's window (chunk stride
// kPeelThreads), wlo = wt - kWin + 1 rounded down to a multiple of 4; chunks
// below word 0 read as empty, chunks above wt are not copied.  Returns wlo.
__device__ __forceinline__ int window_fill(uint4* win, const uint32_t* row, int wt)
{
    const int wlo = (wt - (kWin - 1)) & ~3;
#pragma unroll
    for (int c = 0; c < kWinChunks; ++c) {
        const int w0 = wlo + 4 * c;
        if (w0 > wt) break;
        if (w0 >= 0) cp_async16(win + c * kPeelThreads, row + w0);
        else win[c * kPeelThreads] = make_uint4(0u, 0u, 0u, 0u);
    }
    return wlo;
}

// Arrival at a front barrier that also sums the fronts' sizes: adds
// (1 << 32) + count to *word and waits until the high half reaches `need`.
// Returns the word's value, or ~0 after `limit_ns` (status kDevBarrierTimeout)
// or when another CTA has failed.  Thread 0 only.
__device__ unsigned long long counted_arrive(unsigned long long* word, unsigned count, unsigned long long need,
                                             int* status, unsigned long long limit_ns)
{
    const unsigned long long add = (1ull << 32) | count;
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(add) : "memory");
    const unsigned long long t0 = global_ns();
    for (;;) {
        unsigned long long v;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(word) : "memory");
        if ((v >> 32) >= need) return v;
        if (*((volatile int*)status) != 0) return ~0ull;
        if (global_ns() - t0 > limit_ns) {
            atomicExch(status, kDevBarrierTimeout);
            return ~0ull;
        }
        __nanosleep(32);
    }
}

// Highest unassigned dominator of a row in its words 0 .. sw (-1: none), found
// by G lanes of a warp (l their rank, the same result in each): 256 words a
// step, in chunks of four from the top, those without unassigned points not
// read at all.  Every lane of the warp calls it, a group without a row with
// sw = -1.
template <int G>
__device__ __forceinline__ int scan_row_group(const uint32_t* __restrict__ row, const uint32_t* U, int sw, int l)
{
    constexpr int kLoads = 64 / G;  // 16-byte chunks a lane has in flight
    const uint4* row4 = reinterpret_cast<const uint4*>(row);
    const uint4* U4 = reinterpret_cast<const uint4*>(U);
    int found = -1;
    int top = sw >= 0 ? sw >> 2 : -1;  // highest chunk not yet read
    while (__any_sync(0xFFFFFFFFu, top >= 0)) {
        uint4 v[kLoads];
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
            const int c = top - l - G * i;
            v[i] = make_uint4(0u, 0u, 0u, 0u);
            if (c < 0) continue;
            uint4 u = U4[c];
            if (4 * c + 3 > sw) {  // words above the start are probed, or not of this row
                u.w = 0u;
                if (4 * c + 2 > sw) u.z = 0u;
                if (4 * c + 1 > sw) u.y = 0u;
            }
            if (u.x | u.y | u.z | u.w) {
                const uint4 r = __ldg(row4 + c);
                v[i] = make_uint4(r.x & u.x, r.y & u.y, r.z & u.z, r.w & u.w);
            }
        }
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
            if (found >= 0 || !(v[i].x | v[i].y | v[i].z | v[i].w)) continue;
            const int w = v[i].w ? 3 : v[i].z ? 2 : v[i].y ? 1 : 0;
            const uint32_t bb = v[i].w ? v[i].w : v[i].z ? v[i].z : v[i].y ? v[i].y : v[i].x;
            found = (4 * (top - l - G * i) + w) * 32 + (31 - __clz(bb));
        }
#pragma unroll
        for (int o = G / 2; o; o >>= 1) found = max(found, __shfl_xor_sync(0xFFFFFFFFu, found, o));
        top = found >= 0 ? -1 : top - 64;
    }
    return found;
}

// Thin fronts by one CTA.  A front of a few points costs the grid a barrier
// (about 3 us with its round trips through L2), one CTA three block barriers and
// a row read.  When the first kThinAfter fronts hold at most thin_total points,
// CTA 0 goes on alone with every point's blocker in its shared memory (five
// generations of DTLZ4, M=2: N=1024 6.7 -> 3.7 ms, N=4096 24.9 -> 20.3; sorts of
// 2000 and 8000 points along a chain 2.5 -> 1.3 and 7.4 -> 4.3 ms).  Larger
// populations have thicker fronts at the same total, whose rows one CTA reads
// more slowly: M=2 with 34 points a front, N=2048, 18.7 ms by the grid and 21.3.
// A call, so that the grid's loop keeps its registers.
constexpr int kSoloPoints = 8192;
constexpr int kThinAfter = 8;
__device__ __forceinline__ int thin_total(int nf) { return nf <= 2048 ? 160 : nf <= 4096 ? 96 : 64; }
static_assert(kSoloPoints * (sizeof(int) + sizeof(unsigned short)) <= kWinChunks * kPeelThreads * sizeof(uint4),
              "blockers and queue fit the windows' shared memory");

// Fronts k, k + 1, ... of nf points: U without the fronts before, which hold
// `total` points.  mem: the windows' shared memory.  Ends with the counters as
// nds_peel_owned.
__device__ __noinline__ void peel_solo(const uint32_t* __restrict__ rows, int W, int nf, int target, bool feasible_only,
                                          int feasible, const int* __restrict__ blocker0, int* __restrict__ front_sorted,
                                          uint32_t* U, void* mem, int k, int total, int* counters)
{
    __shared__ int s_queued[2], s_free[2];
    int* blk = reinterpret_cast<int*>(mem);  // unassigned dominator a point waits for, -1: assigned
    unsigned short* queue = reinterpret_cast<unsigned short*>(blk + kSoloPoints);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    constexpr int kWarps = kPeelThreads / 32;
    for (int q = t; q < nf; q += kPeelThreads) blk[q] = ((U[q >> 5] >> (q & 31)) & 1u) ? blocker0[q] : -1;
    if (t < 2) s_queued[t] = s_free[t] = 0;
    __syncthreads();
    for (;; ++k) {
        const int par = k & 1;
        for (int q = t; q < nf; q += kPeelThreads) {
            const int b = blk[q];
            if (b >= 0 && !((U[b >> 5] >> (b & 31)) & 1u)) queue[atomicAdd(&s_queued[par], 1)] = (unsigned short)q;
        }
        __syncthreads();
        const int qn = s_queued[par];
        if (t == 0) s_queued[par ^ 1] = s_free[par ^ 1] = 0;  // last read before this barrier
        // up to one row per warp by all its lanes, else four by eight lanes each
        const int width = qn <= kWarps ? 32 : 8;
        for (int e0 = 0; e0 < qn; e0 += kWarps * (32 / width)) {
            const int e = e0 + warp + kWarps * (lane / width);
            const bool act = e < qn;
            const int q = act ? queue[e] : 0;
            const int sw = act ? blk[q] >> 5 : -1;
            const uint32_t* row = rows + (size_t)q * W;
            const int found = width == 32 ? scan_row_group<32>(row, U, sw, lane) : scan_row_group<8>(row, U, sw, lane & 7);
            if (act && (lane & (width - 1)) == 0) {
                blk[q] = found;
                if (found < 0) {
                    front_sorted[q] = k;
                    atomicAdd(&s_free[par], 1);
                }
            }
        }
        __syncthreads();
        const int ck = s_free[par];
        for (int e = t; e < qn; e += kPeelThreads) {
            const int q = queue[e];
            if (blk[q] < 0) atomicAnd(U + (q >> 5), ~(1u << (q & 31)));
        }
        __syncthreads();
        total += ck;
        if (total >= target || ck == 0 || (feasible_only && total >= feasible)) {
            if (t == 0) {
                counters[2] = k;
                counters[3] = total;
                counters[12] = k;
                if (ck == 0 && total < (feasible_only ? feasible : target)) atomicExch(counters + 6, kDevPeelInconsistent);
            }
            return;
        }
    }
}

__global__ void __launch_bounds__(kPeelThreads, 1)
nds_peel_owned(const uint32_t* __restrict__ rows, int W, int n, int target, const int* __restrict__ blocker0,
               int* __restrict__ front_sorted, uint32_t* __restrict__ fmask, int* counters)
{
    extern __shared__ uint32_t smem[];
    uint32_t* U = smem;                              // unassigned positions, one bit each
    uint4* s_win = reinterpret_cast<uint4*>(smem + ((W + 3) & ~3));  // [kWinChunks][kPeelThreads]
    __shared__ int s_nscan, s_ntask, s_cnt, s_ok, s_ck, s_total;
    __shared__ int s_sq[kScanQueue], s_sw[kScanQueue], s_found[kScanQueue];
    static_assert(kScanQueue >= kPeelThreads, "every owned point must fit the scan queue");
    const int nblocks = gridDim.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const int nf = min(n, counters[0]);
    const int feasible = counters[0];
    const bool feasible_only = feasible < target;
    // feasible positions come first; infeasible ones never enter U (peel_body)
    for (int w = threadIdx.x; w < W; w += blockDim.x) {
        const int lo = w * 32;
        U[w] = (lo + 32 <= nf) ? 0xFFFFFFFFu : (lo >= nf ? 0u : ((1u << (nf - lo)) - 1u));
    }
    if (threadIdx.x == 0) {
        s_nscan = 0;
        s_cnt = 0;
    }
    // this lane's point: group g = warp * nblocks + blockIdx.x (interleaved,
    // like peel_body), at most one per warp
    const int g = warp * nblocks + blockIdx.x;
    const int q = g * 32 + lane;
    bool alive = q < nf;
    int b = -1, wlo = 0;
    uint4* win = s_win + threadIdx.x;
    const uint32_t* row = rows + (size_t)(alive ? q : 0) * W;
    if (alive) {
        b = blocker0[q];
        if (b >= 0) wlo = window_fill(win, row, b >> 5);
    }
    cp_async_commit();
    __syncthreads();
    if (feasible_only && feasible == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            counters[2] = -1;
            counters[12] = -1;
        }
        cp_async_wait_all();
        return;
    }
    unsigned long long* sizes = reinterpret_cast<unsigned long long*>(counters + 16);
    unsigned cum_even = 0u, cum_odd = 0u;  // thread 0: summed sizes of the even and odd fronts
    int k = 0;
    for (;;) {
        uint32_t* G = fmask + (size_t)(k % 3) * W;  // members of front k
        const uint32_t nextw = (uint32_t)((k + 1) % 3);
        for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < W; w += nblocks * blockDim.x)
            fmask[(size_t)nextw * W + w] = 0u;
        cp_async_wait_all();
        // 1. probe: the window of a point whose blocker was assigned
        bool is_free = false;
        int slot = -1;
        if (alive) {
            if (b < 0) {
                is_free = true;
            } else if (!((U[b >> 5] >> (b & 31)) & 1u)) {
                // the window's chunks from the top, each ANDed with the same
                // four words of U (16-byte shared loads, no data-dependent
                // branch); row words above the blocker's word are masked:
                // beyond q's own word they are not part of the row
                const int w = b >> 5;
                const int lo = max(wlo, 0);
                const uint4* U4 = reinterpret_cast<const uint4*>(U);
                int hit = -1;
#pragma unroll
                for (int c = kWinChunks - 1; c >= 0; --c) {
                    const int w0 = wlo + 4 * c;
                    if (w0 >= 0 && w0 <= w) {
                        const uint4 v = win[c * kPeelThreads];
                        const uint4 u = U4[w0 >> 2];
                        const uint32_t m[4] = {v.x & u.x, w0 + 1 <= w ? v.y & u.y : 0u,
                                               w0 + 2 <= w ? v.z & u.z : 0u, w0 + 3 <= w ? v.w & u.w : 0u};
#pragma unroll
                        for (int j = 3; j >= 0; --j)
                            if (hit < 0 && m[j]) hit = (w0 + j) * 32 + (31 - __clz(m[j]));
                    }
                }
                if (hit >= 0) {
                    b = hit;
                } else if (lo == 0) {
                    is_free = true;
                } else {
                    slot = atomicAdd(&s_nscan, 1);
                    s_sq[slot] = q;
                    s_sw[slot] = lo - 1;
                }
            }
        }
        __syncthreads();
        // 2. the CTA's level-ordered scans of the queued rows (peel_body)
        const int nscan = s_nscan;
        if (nscan > 0) {
            if (warp == 0) {
                int levels = 0;
                for (int s0 = 0; s0 < nscan; s0 += 32) {
                    const int sidx = s0 + lane;
                    if (sidx < nscan) {
                        levels = max(levels, s_sw[sidx] / kScanChunk + 1);
                        s_found[sidx] = -1;
                    }
                }
#pragma unroll
                for (int o = 16; o; o >>= 1) levels = max(levels, __shfl_xor_sync(0xFFFFFFFFu, levels, o));
                if (lane == 0) s_ntask = levels * nscan;
            }
            __syncthreads();
            const int ntask = s_ntask;
            for (int task = warp; task < ntask; task += wpb) {
                const int level = task / nscan, lo = task - level * nscan;
                if (level > s_sw[lo] / kScanChunk) continue;
                const int top = s_sw[lo] - level * kScanChunk;
                const int found_hi = __shfl_sync(0xFFFFFFFFu, *((volatile int*)s_found + lo), 0);
                if (found_hi > top * 32 + 31) continue;
                const uint32_t* srow = rows + (size_t)s_sq[lo] * W;
                uint32_t acc[kScanChunk / 32];
#pragma unroll
                for (int i = 0; i < kScanChunk / 32; ++i) {
                    const int w = top - lane - 32 * i;
                    acc[i] = (w >= 0 && w > top - kScanChunk) ? (__ldg(srow + w) & U[w]) : 0u;
                }
                // every loaded word is consumed (no load left in flight)
                int si = -1;
                unsigned snz = 0u;
                uint32_t sel = 0u;
#pragma unroll
                for (int i = 0; i < kScanChunk / 32; ++i) {
                    const unsigned nz = __ballot_sync(0xFFFFFFFFu, acc[i] != 0u);
                    if (si < 0 && nz) {
                        si = i;
                        snz = nz;
                        sel = acc[i];
                    }
                }
                if (si >= 0) {
                    const int src = __ffs(snz) - 1;
                    const uint32_t bb = __shfl_sync(0xFFFFFFFFu, sel, src);
                    if (lane == 0) atomicMax(s_found + lo, (top - src - 32 * si) * 32 + (31 - __clz(bb)));
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) s_nscan = 0;  // next written after two more CTA barriers
        }
        if (slot >= 0) {
            const int f = s_found[slot];
            if (f >= 0) b = f;
            else is_free = true;
        }
        // fewer than kWin window words at or below the blocker: refill the
        // window for the next front
        if (alive && !is_free && b >= 0 && (b >> 5) - wlo < kWin - 1) wlo = window_fill(win, row, b >> 5);
        cp_async_commit();
        // 3. members of front k: the front's mask and the CTA's count
        const unsigned fm = __ballot_sync(0xFFFFFFFFu, is_free);
        if (fm) {
            if (lane == 0) {
                atomicOr(G + g, fm);
                atomicAdd(&s_cnt, __popc(fm));
            }
            if (is_free) {
                front_sorted[q] = k;
                alive = false;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const unsigned long long v = counted_arrive(sizes + (k & 1), (unsigned)s_cnt,
                                                        (unsigned long long)(k / 2 + 1) * (unsigned)nblocks,
                                                        counters + 6, kPeelWaitNs);
            s_cnt = 0;
            s_ok = v != ~0ull;
            if (s_ok) {
                const unsigned c = (unsigned)v;
                if (k & 1) {
                    s_ck = (int)(c - cum_odd);
                    cum_odd = c;
                } else {
                    s_ck = (int)(c - cum_even);
                    cum_even = c;
                }
                s_total = (int)(cum_even + cum_odd);
            }
        }
        __syncthreads();
        if (!s_ok) {
            cp_async_wait_all();
            return;
        }
        // front k is complete: remove it from U
        for (int w = threadIdx.x; w < W; w += blockDim.x) {
            const uint32_t gv = __ldcg(G + w);
            if (gv) U[w] &= ~gv;
        }
        __syncthreads();
        const int ck = s_ck, total = s_total;
        if (total >= target || ck == 0 || (feasible_only && total >= feasible)) {
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                counters[2] = k;
                counters[3] = total;
                counters[12] = k;
                if (ck == 0 && total < (feasible_only ? feasible : target))
                    atomicExch(counters + 6, kDevPeelInconsistent);
            }
            cp_async_wait_all();
            return;
        }
        if (__builtin_expect(k == kThinAfter - 1, 0) && total <= thin_total(nf) && nf <= kSoloPoints) {  // the same in every CTA
            cp_async_wait_all();
            __syncthreads();  // no window is in use any more
            if (blockIdx.x == 0)
                peel_solo(rows, W, nf, target, feasible_only, feasible, blocker0, front_sorted, U, s_win, k + 1, total,
                          counters);
            return;
        }
        ++k;
    }
}

// Shared memory of nds_peel_owned beyond its static arrays.
size_t peel_owned_smem(int W)
{
    return (size_t)((W + 3) & ~3) * sizeof(uint32_t) + (size_t)kWinChunks * kPeelThreads * sizeof(uint4);
}

// Fronts in point order, and the closed-form fronts of the infeasible points
// when the feasible ones number fewer than the target.  Every infeasible point
// is dominated by all feasible points, a class-2 point also by every class-2
// point of smaller violation, a class-3 point (NaN violation) by the feasible
// points only.  With F the last feasible front (-1 without feasible points):
// class 3 forms front F + 1 together with the first class-2 run of equal
// violations, class-2 run j is front F + 1 + j.  The stop rule of the peel
// keeps the fronts up to the first whose cumulative count reaches the target:
// run j (j > 0) is kept when n3 + start_j < target.  One 8-CTA cluster: each
// CTA numbers the runs of a segment, the segments' counts pass through the
// cluster's shared memory (a launch instead of the head, scan and scatter
// launches that it takes without).
constexpr int kFrontCtas = 8, kFrontThreads = 1024;
__global__ void __cluster_dims__(kFrontCtas, 1, 1) __launch_bounds__(kFrontThreads)
nds_fronts(int n, const int* __restrict__ perm, const int* __restrict__ qinfo, const int* __restrict__ front_sorted,
           int* counters, int target, int* __restrict__ fronts)
{
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ int s_runs, s_w[kFrontThreads / 32];
    const int c = (int)cluster.block_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int fc = counters[0], n2 = counters[10], n3 = counters[11], F1 = counters[12] + 1;
    const bool closed = fc < target;  // uniform over the cluster
    const int plain = closed ? fc : n;
    for (int pos = c * kFrontThreads + tid; pos < n; pos += kFrontCtas * kFrontThreads)
        if (pos < plain) fronts[perm[pos]] = front_sorted[pos];
        else if (pos >= fc + n2) fronts[perm[pos]] = F1;
    if (!closed) return;
    if (n2 == 0) {
        if (c == 0 && tid == 0) counters[2] = F1;
        return;
    }
    auto start_of = [&](int pos) { return (int)((uint32_t)qinfo[pos] & ~kInfeasibleBit); };
    const int per = (n2 + kFrontCtas - 1) / kFrontCtas;
    const int lo = fc + min(n2, c * per), hi = min(fc + n2, lo + per);
    int runs = 0;
    for (int pos = lo + tid; pos < hi; pos += kFrontThreads) runs += start_of(pos) == pos ? 1 : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) runs += __shfl_xor_sync(0xFFFFFFFFu, runs, o);
    if (lane == 0) s_w[warp] = runs;
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kFrontThreads / 32; ++w) runs += s_w[w];
        s_runs = runs;
    }
    cluster.sync();
    int base = 0;
    for (int r = 0; r < c; ++r) base += *cluster.map_shared_rank(&s_runs, r);
    cluster.sync();  // the counts were read everywhere
    // the position whose front is the last one kept
    int p_last = target - n3 - 1;
    p_last = p_last < fc ? fc : (p_last > fc + n2 - 1 ? fc + n2 - 1 : p_last);
    for (int p0 = lo; p0 < hi; p0 += kFrontThreads) {
        const int pos = p0 + tid;
        const int start = pos < hi ? start_of(pos) : -1;
        const unsigned heads = __ballot_sync(0xFFFFFFFFu, pos < hi && start == pos);
        __syncthreads();  // s_w free
        if (lane == 0) s_w[warp] = __popc(heads);
        __syncthreads();
        int before = base, total = base;
        for (int w = 0; w < kFrontThreads / 32; ++w) {
            before += w < warp ? s_w[w] : 0;
            total += s_w[w];
        }
        if (pos < hi) {
            const int j = before + __popc(heads & (0xFFFFFFFFu >> (31 - lane))) - 1;
            fronts[perm[pos]] = (j == 0 || n3 + start < target) ? F1 + j : -1;
            if (pos == p_last) counters[2] = F1 + j;
        }
        base = total;
    }
}

__global__ void nds_reset_counters(int* counters)
{
    if (threadIdx.x < 4) counters[threadIdx.x] = 0;
    if (threadIdx.x == 4) counters[4] = 0;
    if (threadIdx.x >= 10 && threadIdx.x <= 13) counters[threadIdx.x] = 0;
    if (threadIdx.x >= 16 && threadIdx.x <= 19) counters[threadIdx.x] = 0;  // front sizes (nds_peel_owned)
}

// ---------------------------------------------------------------------------
// 2b. dominance rows from block prefix sets (one workspace, any n)
// ---------------------------------------------------------------------------
//
// For every block of B sorted positions and every objective m >= 1 one table
// of BlockTable<B>::kSize words:
//   E[0]          the largest of the block's B order keys;
//   E[1 .. B-1]   the other B-1 keys as an implicit search tree (node k has
//                 children 2k and 2k+1; the in-order walk is ascending);
//   S[c], c = 0..B, from word B on: the positions of the c smallest keys
//                 (bit j of word i = position 32 i + j of the block), B/32
//                 words each.  For B = 256 the two 16-byte halves of S[c] are
//                 swapped when bit 2 of c is set, so that the 16-byte loads
//                 of eight lanes with different c spread over all eight bank
//                 groups.
// The count c of the block's keys <= v is the leaf that a log2(B)-level
// descent of the tree reaches (go right when E[k] <= v) plus (E[0] <= v); the
// block's positions whose objective is <= f_m(q) are then S[c], ties included
// whatever their order.  A lane holding q thus gets B row bits of objective m
// from log2(B) + 1 shared loads and B/128 16-byte loads, where the per-word
// tables of nds_tiles take B/32 six-probe searches.  Positions >= n carry the
// NaN key, above every key of a feasible q.
template <int B>
struct BlockTable {
    static constexpr int kWords = B / 32;                // row words per block
    static constexpr int kLevels = B == 256 ? 8 : 7;     // B = 2^kLevels
    static constexpr int kSize = B + (B + 1) * kWords;   // words per (block, objective)
};
static_assert(BlockTable<256>::kSize % 4 == 0 && BlockTable<128>::kSize % 4 == 0,
              "tables are copied in 16-byte chunks");

// Block size by objective count: up to M = 4 the double-buffered tables of
// 256 positions (9 KB per objective) leave room for several CTAs per SM;
// beyond, blocks of 128 positions (2.5 KB per objective) keep the SMs full.
template <int M>
struct BlockCfg {
    static constexpr int kB = M <= 4 ? 256 : 128;
};

// Dominatees q per row CTA, one per thread.  Every CTA stages each of its
// blocks' tables once, so more q per CTA mean fewer shared-memory writes per
// row word.
constexpr int kBlkThreads = 512;
constexpr int kBlkPerCtaMax = 8;  // blocks of dominators per row CTA, at most
constexpr int kBlkCtasPerSm = 8;  // row CTAs per SM the launch aims at (with fewer blocks per CTA)

// Count of the 32 ascending keys a[] that are <= x (six probes).
__device__ __forceinline__ int count_le32(const uint32_t* a, uint32_t x)
{
    int c = 0;
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1)
        if (a[c + s - 1] <= x) c += s;
    if (a[c] <= x) ++c;
    return c;
}

// One CTA of B threads per (block, objective): each warp sorts its 32
// (key, lane) pairs with a bitonic network; the rank of a key in the block is
// its place in its warp plus, for every other warp, the count of that warp's
// keys <= it (lower warps) or < it (higher warps), which orders equal keys
// by position.  Then the tree placement of the sorted keys, and warp w builds
// word w of every prefix set with one ballot per set.
template <int B>
__device__ __forceinline__ void block_table(int cta, const float* __restrict__ sf, int sf_stride, int n, int MF,
                                            uint32_t* __restrict__ tables)
{
    using T = BlockTable<B>;
    constexpr int NW = B / 32;
    __shared__ uint32_t s_sorted[NW][32];
    __shared__ int s_rank[B];
    const int blk = cta / MF, m = cta - blk * MF;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = blk * B + threadIdx.x;
    const uint32_t key = p < n ? dom_key(sf[(size_t)m * sf_stride + p]) : 0xFFFFFFFFu;
    unsigned long long kv = ((unsigned long long)key << 32) | (unsigned)lane;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const unsigned long long o = __shfl_xor_sync(0xFFFFFFFFu, kv, j);
            const bool take_min = ((lane & j) == 0) == ((lane & k) == 0);
            kv = take_min ? (o < kv ? o : kv) : (o > kv ? o : kv);
        }
    }
    const uint32_t skey = (uint32_t)(kv >> 32);
    const int src = (int)(kv & 31ull);  // this lane holds the key of lane src
    s_sorted[warp][lane] = skey;
    __syncthreads();
    int r = lane;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        if (w < warp) r += count_le32(s_sorted[w], skey);
        else if (w > warp && skey > 0u) r += count_le32(s_sorted[w], skey - 1u);
    }
    s_rank[warp * 32 + src] = r;
    uint32_t* tab = tables + ((size_t)blk * MF + m) * T::kSize;
    if (r == B - 1) {
        tab[0] = skey;
    } else {
        const int i = r + 1, h = __ffs(i) - 1;  // in-order index, height above the leaves
        tab[(1 << (T::kLevels - 1 - h)) + (i >> (h + 1))] = skey;
    }
    __syncthreads();
    const int rk = s_rank[threadIdx.x];  // rank of position 32 warp + lane
    uint32_t* S = tab + B;
    for (int c0 = 0; c0 <= B; c0 += 32) {
        uint32_t mine = 0u;
#pragma unroll 8
        for (int cc = 0; cc < 32; ++cc) {
            const uint32_t bits = __ballot_sync(0xFFFFFFFFu, rk < c0 + cc);
            if (cc == lane) mine = bits;
        }
        const int c = c0 + lane;
        if (c <= B) {
            const int wj = NW == 8 ? (warp ^ (((c >> 2) & 1) << 2)) : warp;  // the half swap
            S[c * NW + wj] = mine;
        }
    }
}

template <int B>
__global__ void __launch_bounds__(B)
nds_block_tables(const float* __restrict__ sf, int sf_stride, int n, int MF, uint32_t* __restrict__ tables)
{
    block_table<B>(blockIdx.x, sf, sf_stride, n, MF, tables);
}

__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

constexpr int kRowSegWords = 16;   // row words per lane collected before the stores
constexpr int kOutStride = 20;     // shared words per lane of the collected rows (16-byte rows, no conflicts)

// Rows are collected in shared memory for blocks of 256 positions (M <= 4).
// With blocks of 128 positions the search of the M-1 >= 4 objectives
// outweighs the stores, and the 40 KB for the collected rows would cost a
// resident CTA per SM: each lane stores its own words.
template <int B>
constexpr bool collect_rows() { return B == 256; }

// Rows of kBlkThreads dominatees (one per thread) against bpc blocks of B
// dominator positions.  The blocks' tables (all objectives) are staged in
// shared memory with cp.async, the next block's while the current one is
// searched.  Per block a lane descends the M-1 trees side by side and ANDs the
// M-1 prefix sets and the dup mask into its B/32 row words.  With
// collect_rows<B>() the lane puts them into shared memory and every
// kRowSegWords words the CTA writes the collected row segments (64 bytes per
// row), eight rows per warp instruction, where stores by the lanes themselves
// touch 32 rows per instruction; otherwise the lane stores them itself.  The lane remembers
// the highest dominator seen and raises blocker[q] to it once.  Infeasible q
// are skipped: the peel never reaches them, so their rows are never read.
template <int M, int B>
__device__ __forceinline__ void block_rows(int bx, int by, const float* __restrict__ sf, int sf_stride,
                                           const int* __restrict__ qinfo, const uint32_t* __restrict__ tables, int n,
                                           int W, int bpc, uint32_t* __restrict__ rows, int* __restrict__ blocker)
{
    using T = BlockTable<B>;
    constexpr int MF = M - 1;
    constexpr int KW = T::kWords;
    constexpr int TS = T::kSize;
    constexpr int CH = MF * TS / 4;  // 16-byte chunks of one block's tables
    constexpr int G = kRowSegWords / KW;  // blocks per collected segment
    extern __shared__ uint4 s_tab[];  // [2][CH] tables, then (collect_rows) [kBlkThreads][kOutStride] row words
    __shared__ unsigned char s_live[kBlkThreads];
    uint32_t* s_out = reinterpret_cast<uint32_t*>(s_tab + 2 * CH);
    const int q0 = by * kBlkThreads;
    if (q0 >= n) return;
    const int qend = min(q0 + kBlkThreads, n);
    const int nb = (qend - 1 + B - 1) / B;  // blocks holding the dominators (positions < qend - 1)
    const int b_lo = bx * bpc;
    if (b_lo >= nb) return;
    const int b_hi = min(nb, b_lo + bpc);
    const int q = q0 + threadIdx.x;
    uint32_t qk[MF];
    int dup = 0;
    bool live = false;
    if (q < n) {
        const uint32_t info = (uint32_t)qinfo[q];
        live = (info & kInfeasibleBit) == 0u;
        dup = (int)(info & ~kInfeasibleBit);
    }
#pragma unroll
    for (int m = 0; m < MF; ++m) qk[m] = live ? dom_key(sf[(size_t)m * sf_stride + q]) : 0u;
    s_live[threadIdx.x] = live ? 1 : 0;
    if (!__syncthreads_or(live)) return;

    const uint4* src = reinterpret_cast<const uint4*>(tables);
    auto stage = [&](int b, int buf) {
        const uint4* g = src + (size_t)b * CH;
        uint4* d = s_tab + buf * CH;
        for (int i = threadIdx.x; i < CH; i += kBlkThreads)
            cp_async16(d + i, reinterpret_cast<const uint32_t*>(g + i));
        cp_async_commit();
    };
    stage(b_lo, 0);
    int best = -1;
    uint32_t* my_out = s_out + threadIdx.x * kOutStride;
    int seg = b_lo;  // first block of the segment being collected
    for (int b = b_lo; b < b_hi; ++b) {
        const int buf = (b - b_lo) & 1;
        if (b + 1 < b_hi) {
            stage(b + 1, buf ^ 1);
            cp_async_wait_one();
        } else {
            cp_async_wait_all();
        }
        __syncthreads();
        if (live) {
            const int lo = b * B;
            const int rem = dup - lo;  // positions of the block below dup[q]
            uint32_t acc[KW];
#pragma unroll
            for (int j = 0; j < KW; ++j) acc[j] = rem > 0 ? 0xFFFFFFFFu : 0u;
            if (rem > 0) {
                const uint32_t* tab = reinterpret_cast<const uint32_t*>(s_tab + buf * CH);
                int k[MF];
#pragma unroll
                for (int m = 0; m < MF; ++m) k[m] = 1;
#pragma unroll
                for (int l = 0; l < T::kLevels; ++l) {
#pragma unroll
                    for (int m = 0; m < MF; ++m) k[m] = 2 * k[m] + (tab[m * TS + k[m]] <= qk[m] ? 1 : 0);
                }
#pragma unroll
                for (int m = 0; m < MF; ++m) {
                    const uint32_t* E = tab + m * TS;
                    const int c = k[m] - B + (E[0] <= qk[m] ? 1 : 0);
                    const uint4* S = reinterpret_cast<const uint4*>(E + B) + c * (KW / 4);
                    if constexpr (KW == 8) {
                        const int sw = (c >> 2) & 1;
                        const uint4 x = S[sw], y = S[sw ^ 1];
                        acc[0] &= x.x; acc[1] &= x.y; acc[2] &= x.z; acc[3] &= x.w;
                        acc[4] &= y.x; acc[5] &= y.y; acc[6] &= y.z; acc[7] &= y.w;
                    } else {
                        const uint4 x = S[0];
                        acc[0] &= x.x; acc[1] &= x.y; acc[2] &= x.z; acc[3] &= x.w;
                    }
                }
                if (rem < B) {
#pragma unroll
                    for (int j = 0; j < KW; ++j) {
                        const int r = rem - 32 * j;
                        acc[j] &= r >= 32 ? 0xFFFFFFFFu : (r <= 0 ? 0u : ((1u << r) - 1u));
                    }
                }
            }
            if constexpr (collect_rows<B>()) {
                uint4* o = reinterpret_cast<uint4*>(my_out + (b - seg) * KW);
                o[0] = make_uint4(acc[0], acc[1], acc[2], acc[3]);
                if constexpr (KW == 8) o[1] = make_uint4(acc[4], acc[5], acc[6], acc[7]);
            } else {
                uint4* dst = reinterpret_cast<uint4*>(rows + (size_t)q * W + b * KW);
                dst[0] = make_uint4(acc[0], acc[1], acc[2], acc[3]);
                if constexpr (KW == 8) {
                    if (b * KW + 8 <= W) dst[1] = make_uint4(acc[4], acc[5], acc[6], acc[7]);
                }
            }
#pragma unroll
            for (int j = 0; j < KW; ++j)
                if (acc[j]) best = lo + 32 * j + 31 - __clz(acc[j]);
        }
        if (collect_rows<B>() && (b - seg + 1 == G || b + 1 == b_hi)) {
            // the segment's words seg*KW .. seg*KW + nw - 1 of every live row:
            // a warp writes 8 rows x 4 chunks of 16 bytes, lanes 8i .. 8i+7
            // reading rows R+i and R+i+4 (distinct bank groups)
            __syncthreads();
            const int nw = (b - seg + 1) * KW;
            for (int c = threadIdx.x; c < kBlkThreads * (kRowSegWords / 4); c += kBlkThreads) {
                const int l = c & 31, rsel = l >> 2, part = l & 3;
                const int r = (c >> 5) * 8 + ((rsel & 1) << 2) + (rsel >> 1);
                const int gw = seg * KW + part * 4;
                if (part * 4 < nw && gw + 4 <= W && s_live[r])
                    *reinterpret_cast<uint4*>(rows + (size_t)(q0 + r) * W + gw) =
                        *reinterpret_cast<const uint4*>(s_out + r * kOutStride + part * 4);
            }
            seg = b + 1;
        }
        __syncthreads();  // the table buffer is staged again two blocks on, the row words rewritten
    }
    if (best >= 0) atomicMax(blocker + q, best);
}

template <int M, int B>
__global__ void __launch_bounds__(kBlkThreads)
nds_block_rows(const float* __restrict__ sf, int sf_stride, const int* __restrict__ qinfo,
               const uint32_t* __restrict__ tables, int n, int W, int bpc, uint32_t* __restrict__ rows,
               int* __restrict__ blocker)
{
    block_rows<M, B>(blockIdx.x, blockIdx.y, sf, sf_stride, qinfo, tables, n, W, bpc, rows, blocker);
}

template <int M>
constexpr int block_rows_smem()
{
    constexpr int B = BlockCfg<M>::kB;
    return 2 * (M - 1) * BlockTable<B>::kSize * 4 + (collect_rows<B>() ? kBlkThreads * kOutStride * 4 : 0);
}

template <int M>
void launch_block_rows(const Workspace& ws, int n, cudaStream_t stream)
{
    constexpr int B = BlockCfg<M>::kB;
    if (n < 2) return;  // no pairs: every blocker stays -1
    nds_block_tables<B><<<ceil_div(n, B) * (M - 1), B, 0, stream>>>(ws.sorted_f, ws.n_max, n, M - 1,
                                                                     ws.block_tables);
    // blocks per CTA: the most (up to kBlkPerCtaMax) that still give
    // kBlkCtasPerSm working CTAs per SM; fewer blocks per CTA overlap less
    // staging with searching, but small sorts need the CTAs
    const int ntiles = ceil_div(n, kBlkThreads);
    const int nb = ceil_div(n - 1, B);
    int bpc = kBlkPerCtaMax;
    for (; bpc > 1; bpc >>= 1) {
        long long ctas = 0;
        for (int t = 0; t < ntiles; ++t) ctas += ceil_div(ceil_div(std::min((t + 1) * kBlkThreads, n) - 1, B), bpc);
        if (ctas >= (long long)kBlkCtasPerSm * ws.sm_count) break;
    }
    dim3 grid(ceil_div(nb, bpc), ntiles);
    nds_block_rows<M, B><<<grid, kBlkThreads, block_rows_smem<M>(), stream>>>(
        ws.sorted_f, ws.n_max, ws.qinfo, ws.block_tables, n, ws.words, bpc, ws.rows, ws.blocker);
}

template <int M>
void launch_tiles(const Workspace& ws, int n, cudaStream_t stream)
{
    if constexpr (M > 1) {
        if (!ws.word_tiles) {
            launch_block_rows<M>(ws, n, stream);
            return;
        }
    }
    const int nqb = ceil_div(n, kQB);
    const int maxw = ceil_div(n, 32);
    if (M > 1) {
        const int warps = maxw * (M - 1);
        nds_chunks<<<ceil_div(warps, 8), 256, 0, stream>>>(ws.sorted_f, ws.n_max, n, maxw, M - 1,
                                                         ws.chunk_keys, ws.chunk_bits);
    }
    dim3 grid(ceil_div(maxw, TileCfg<M>::kPW), nqb);
    nds_tiles<M><<<grid, kTileThreads, 0, stream>>>(ws.sorted_f, ws.n_max, ws.qinfo, ws.chunk_keys,
                                                     ws.chunk_bits, n, ws.words, maxw, ws.rows,
                                                     ws.blocker);
}

// ---------------------------------------------------------------------------
// fused batch: one launch per stage for every instance (n = 2N <= 8192)
// ---------------------------------------------------------------------------

// The sort and the dominance rows of every instance (blockIdx.y) by the CTAs
// and threads of the staged path: tiles, one rank merge above kSortTile points,
// runs of equal keys, sorted objectives and dup positions.  The passes of one
// CTA per instance that these replace (a block radix sort, and the rows from
// per-word tables) took 269 + 71 + 913 us over 256 instances.
static_assert(kFusedSortTile == kSortTile && kFusedMaxPoints == kSortTile * kSortWays, "one merge pass");
__device__ __forceinline__ SplitPop batch_pop(const BatchInst& I)
{
    return SplitPop{I.objsP, I.objsO, I.cvP, I.cvO, I.N, I.N, I.N, I.n};
}

__global__ void __launch_bounds__(kSortTile)
fused_sort_tiles(const BatchInst* __restrict__ insts, const int* __restrict__ ids)
{
    const BatchInst& I = insts[ids[blockIdx.y]];
    if ((int)blockIdx.x * kSortTile < I.n) sort_tile(blockIdx.x, batch_pop(I), I.M, I.key0, I.key64, I.perm_a, I.counters);
}

__global__ void __launch_bounds__(256)
fused_sort_merge(const BatchInst* __restrict__ insts, const int* __restrict__ ids)
{
    const BatchInst& I = insts[ids[blockIdx.y]];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (I.n > kSortTile && i < I.n) sort_merge_key(i, I.key64, I.perm_a, I.key64b, I.perm_b, I.n, kSortTile);
}

__global__ void __launch_bounds__(256)
fused_tie_rank(const BatchInst* __restrict__ insts, const int* __restrict__ ids)
{
    const BatchInst& I = insts[ids[blockIdx.y]];
    const int pos = blockIdx.x * blockDim.x + threadIdx.x;
    tie_rank(pos, pos < I.n, batch_pop(I), I.M, I.n > kSortTile ? I.key64b : I.key64,
             I.n > kSortTile ? I.perm_b : I.perm_a, I.perm, I.long_runs, I.counters + 13);
}

__global__ void __launch_bounds__(kTieLongThreads)
fused_tie_long(const BatchInst* __restrict__ insts, const int* __restrict__ ids)
{
    const BatchInst& I = insts[ids[blockIdx.x]];
    tie_fix_long(0, 1, batch_pop(I), I.M, I.n > kSortTile ? I.key64b : I.key64, I.perm, I.long_runs, I.counters + 13);
}

__global__ void __launch_bounds__(256)
fused_finalize_rows(const BatchInst* __restrict__ insts, const int* __restrict__ ids)
{
    const BatchInst& I = insts[ids[blockIdx.y]];
    const int pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos < I.n)
        finalize_row(pos, batch_pop(I), I.M, I.key0, I.n > kSortTile ? I.key64b : I.key64, I.perm, I.sorted_f, I.n_max,
                     I.counters, I.qinfo, I.blocker, I.front_sorted);
}

template <int M>
__global__ void __launch_bounds__(BlockCfg<M>::kB)
fused_block_tables(const BatchInst* __restrict__ insts, const int* __restrict__ ids)
{
    const BatchInst& I = insts[ids[blockIdx.y]];
    if ((int)(blockIdx.x / (M - 1)) * BlockCfg<M>::kB < I.n)
        block_table<BlockCfg<M>::kB>(blockIdx.x, I.sorted_f, I.n_max, I.n, M - 1, I.block_tables);
}

// Row CTAs of one instance of n points with bpc blocks each; the CTA `cta`
// of them as (block range, tile).
template <int B>
__host__ __device__ inline int row_ctas(int n, int bpc, int cta, int* bx, int* by)
{
    int first = 0;
    for (int t = 0; t * kBlkThreads < n; ++t) {
        const int end = (t + 1) * kBlkThreads < n ? (t + 1) * kBlkThreads : n;
        const int nb = (end - 1 + B - 1) / B, here = (nb + bpc - 1) / bpc;
        if (cta >= first && cta < first + here) {
            *bx = cta - first;
            *by = t;
        }
        first += here;
    }
    return first;
}

// Dominator positions per row CTA of a batch (tile shapes 0 and 1): batches
// fill the device, so a CTA keeps many blocks and stages them in turn.
constexpr int kBatchRowPositions[kTileShapes] = {1024, 512};

// Row CTAs of all instances with M objectives, flattened: CTA b belongs to
// the instance whose range [prefix[k], prefix[k+1]) contains b.
template <int M>
__global__ void __launch_bounds__(kBlkThreads)
fused_block_rows(const BatchInst* __restrict__ insts, const int* __restrict__ ids, const int* __restrict__ prefix,
                 int count, int bpc)
{
    constexpr int B = BlockCfg<M>::kB;
    const int b = blockIdx.x;
    int lo = 0, hi = count;  // largest k with prefix[k] <= b
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(prefix + mid) <= b) lo = mid; else hi = mid;
    }
    const BatchInst& I = insts[__ldg(ids + lo)];
    int bx = 0, by = 0;
    row_ctas<B>(I.n, bpc, b - __ldg(prefix + lo), &bx, &by);
    block_rows<M, B>(bx, by, I.sorted_f, I.n_max, I.qinfo, I.block_tables, I.n, I.W, bpc, I.rows, I.blocker);
}

// One objective: rows from the dup positions alone.
__global__ void __launch_bounds__(kTileThreads)
fused_tiles_one(const BatchInst* __restrict__ insts, const int* __restrict__ ids, const int* __restrict__ prefix,
                int count)
{
    const int b = blockIdx.x;
    int lo = 0, hi = count;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(prefix + mid) <= b) lo = mid; else hi = mid;
    }
    const BatchInst& I = insts[__ldg(ids + lo)];
    const int maxw = (I.n + 31) >> 5;
    constexpr int PW = TileCfg<1>::kPW;
    const int gx = (maxw + PW - 1) / PW;
    const int lb = b - __ldg(prefix + lo);
    tile_block<1, PW>(lb % gx, lb / gx, I.sorted_f, I.n_max, I.qinfo, nullptr, nullptr, I.n, I.W, maxw, I.rows,
                      I.blocker);
}

constexpr int kFusedPeelThreads = 1024;
constexpr int kWalkHops = 64;  // waiting points followed from one member before the pass over all points

// Peel of one instance per CTA in shared memory.  Every unassigned point waits
// for one unassigned dominator, its blocker, and the points that wait for the
// same one form a list (head, next).  A member of front k leaves the
// unassigned set U and queues its list; each queued point is searched from the
// former blocker's word downwards (bits above it stay free of unassigned
// dominators) and either waits for the next unassigned dominator found or,
// having none, joins front k + 1.  Thin fronts bound the peel (DTLZ4, M=3: 460
// fronts of ten points), each a chain of two block barriers, the lists and one
// row read: 1.33 ms with a pass over all blockers per front, a probe of two
// words and then a scan by a warp, 1.08 ms now.  Shared memory: U (W words), blocker, head,
// next, list and queue (n ints each).
__global__ void __launch_bounds__(kFusedPeelThreads, 1)
fused_peel(const BatchInst* __restrict__ insts, const int* __restrict__ ids)
{
    extern __shared__ __align__(16) uint32_t fp_smem[];
    __shared__ int s_cnt, s_qn[2], s_long[2];
    const BatchInst& I = insts[ids[blockIdx.x]];
    const int n = I.n, W = I.W, target = I.N;
    uint32_t* U = fp_smem;
    int* blk = reinterpret_cast<int*>(fp_smem + W);
    int* list = blk + n;
    int* queue = list + n;
    int* head = queue + n;
    int* next = head + n;
    const uint32_t* rows = I.rows;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarps = blockDim.x >> 5;

    for (int w = t; w < W; w += blockDim.x) {
        const int lo = w * 32;
        U[w] = (lo + 32 <= n) ? 0xFFFFFFFFu : (lo >= n ? 0u : ((1u << (n - lo)) - 1u));
    }
    for (int q = t; q < n; q += blockDim.x) head[q] = -1;
    if (t < 2) {
        s_qn[t] = 0;
        s_long[t] = 0;
    }
    if (t == 0) s_cnt = 0;
    __syncthreads();
    for (int q = t; q < n; q += blockDim.x) {
        const int b = I.blocker[q];
        blk[q] = b;
        if (b < 0) {
            list[atomicAdd(&s_cnt, 1)] = q;
            I.front_sorted[q] = 0;
        } else {
            next[q] = atomicExch(head + b, q);
        }
    }
    __syncthreads();
    int len_prev = 0, len = s_cnt, total = 0, k = 0;
    for (;;) {
        const int ck = len - len_prev;
        total += ck;
        if (total >= target || ck == 0) {
            if (t == 0) {
                I.counters[1] = len;
                I.counters[2] = k;
                I.counters[3] = total;
                if (ck == 0 && total < target) atomicExch(I.counters + 6, kDevPeelInconsistent);
            }
            for (int q = t; q < n; q += blockDim.x) I.fronts[I.perm[q]] = I.front_sorted[q];
            return;
        }
        const int par = k & 1;
        for (int i = t; i < ck; i += blockDim.x) {
            const int p = list[len_prev + i];
            atomicAnd(U + (p >> 5), ~(1u << (p & 31)));
            int hops = 0;
            for (int q = head[p]; q >= 0; q = next[q]) {
                if (++hops > kWalkHops) {
                    s_long[par] = 1;
                    break;
                }
                queue[atomicAdd(&s_qn[par], 1)] = q;
            }
        }
        __syncthreads();
        if (s_long[par]) {
            // a list longer than one thread should follow: a pass over all
            // blockers instead (a member of a front has none)
            __syncthreads();
            if (t == 0) s_qn[par] = 0;
            __syncthreads();
            for (int q = t; q < n; q += blockDim.x) {
                const int b = blk[q];
                if (b >= 0 && !((U[b >> 5] >> (b & 31)) & 1u)) queue[atomicAdd(&s_qn[par], 1)] = q;
            }
            __syncthreads();
        }
        const int qn = s_qn[par];
        if (t == 0) {  // of the next front: last read before two barriers
            s_qn[par ^ 1] = 0;
            s_long[par ^ 1] = 0;
        }
        // Entries interleaved over the warps.  Up to one row per warp it is
        // read by all lanes, up to four by eight lanes each; a longer queue
        // probes two words per lane first, which resolves most rows.
        const int width = qn <= nwarps ? 32 : qn <= 4 * nwarps ? 8 : 1;
        const int sub = lane / width;
        for (int r = 0; r * 32 * nwarps < qn; ++r) {
            const int e = warp + nwarps * (width > 1 ? sub : r * 32 + lane);
            const bool act = e < qn;
            const int q = act ? queue[e] : 0;
            bool is_free = false, need = false;
            int start_w = -1;
            if (width > 1) {
                const int sw = act ? blk[q] >> 5 : -1;
                const uint32_t* row = rows + (size_t)q * W;
                const int found = width == 32 ? scan_row_group<32>(row, U, sw, lane)
                                              : scan_row_group<8>(row, U, sw, lane & 7);
                if (act && (lane & (width - 1)) == 0) {
                    if (found >= 0) {
                        blk[q] = found;
                        next[q] = atomicExch(head + found, q);
                    } else {
                        is_free = true;
                    }
                }
            } else if (act) {
                const uint32_t* row = rows + (size_t)q * W;
                int w = blk[q] >> 5;
                const uint32_t hiw = __ldg(row + w);
                const uint32_t low = (w > 0) ? __ldg(row + w - 1) : 0u;
                uint32_t bits = hiw & U[w];
                if (!bits && w > 0) {
                    --w;
                    bits = low & U[w];
                }
                if (bits) {
                    const int f = w * 32 + (31 - __clz(bits));
                    blk[q] = f;
                    next[q] = atomicExch(head + f, q);
                } else if (w == 0) {
                    is_free = true;
                } else {
                    need = true;
                    start_w = w - 1;
                }
            }
            // rows not resolved by the probe: eight lanes scan each of them
            // downwards over the words that still hold unassigned points,
            // four rows of the warp side by side
            const int grp = lane >> 3;
            unsigned needm = __ballot_sync(0xFFFFFFFFu, need);
            while (needm) {
                unsigned m = needm;  // its sub-th set bit is this group's row
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    if (j < grp) m &= m - 1;
                const int L = m ? __ffs(m) - 1 : -1;
#pragma unroll
                for (int j = 0; j < 4; ++j) needm &= needm - 1;
                const int qL = __shfl_sync(0xFFFFFFFFu, q, max(L, 0));
                const int sw = __shfl_sync(0xFFFFFFFFu, start_w, max(L, 0));
                const int found = scan_row_group<8>(rows + (size_t)qL * W, U, L >= 0 ? sw : -1, lane & 7);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int Lj = __shfl_sync(0xFFFFFFFFu, L, 8 * j);
                    const int fj = __shfl_sync(0xFFFFFFFFu, found, 8 * j);
                    if (lane == Lj) {
                        if (fj >= 0) {
                            blk[q] = fj;
                            next[q] = atomicExch(head + fj, q);
                        } else {
                            is_free = true;
                        }
                    }
                }
            }
            const unsigned fm = __ballot_sync(0xFFFFFFFFu, is_free);
            if (fm) {
                int slot = 0;
                if (lane == 0) slot = atomicAdd(&s_cnt, __popc(fm));
                slot = __shfl_sync(0xFFFFFFFFu, slot, 0);
                if (is_free) {
                    list[slot + __popc(fm & ((1u << lane) - 1u))] = q;
                    blk[q] = -1;
                    I.front_sorted[q] = k + 1;
                }
            }
        }
        __syncthreads();
        len_prev = len;
        len = s_cnt;
        ++k;
    }
}

template <int M>
int tile_blocks_of(int n, int shape)
{
    if constexpr (M == 1) return ceil_div(ceil_div(n, 32), TileCfg<1>::kPW) * ceil_div(n, kQB);
    int bx, by;
    return row_ctas<BlockCfg<M>::kB>(n, kBatchRowPositions[shape] / BlockCfg<M>::kB, -1, &bx, &by);
}

template <int M>
int launch_fused_rows(const BatchInst* d_inst, const FusedBucket& b, cudaStream_t s)
{
    if constexpr (M == 1) {
        fused_tiles_one<<<b.tile_blocks, kTileThreads, 0, s>>>(d_inst, b.d_ids, b.d_tile_prefix, b.count);
    } else {
        constexpr int B = BlockCfg<M>::kB;
        fused_block_tables<M><<<dim3(ceil_div(b.max_n, B) * (M - 1), b.count), B, 0, s>>>(d_inst, b.d_ids);
        fused_block_rows<M><<<b.tile_blocks, kBlkThreads, block_rows_smem<M>(), s>>>(
            d_inst, b.d_ids, b.d_tile_prefix, b.count, kBatchRowPositions[b.shape] / B);
    }
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

// ---------------------------------------------------------------------------
// small populations: the whole sort in one CTA
// ---------------------------------------------------------------------------
//
// Up to kSmallPoints points nothing has to be ordered: a thread per point tests
// every other point against its own and keeps its dominators as bits in
// registers, and a front costs one look at the unassigned words in shared
// memory and two barriers.  Infeasible points take part in the same relation
// (every feasible point, and those of smaller violation, dominate one).  The
// eight launches of the general sort are bound by their latency at this size
// (n = 184, M = 3: 39 us and the gaps between them, against 8: 72 -> 51 us a
// generation).  The pair tests grow with n^2 (M + 1): at 2^20 of them (512 points
// of three objectives, 341 of eight) the general sort draws level.
constexpr int kSmallPoints = 512;
constexpr long long kSmallWork = 1ll << 20;
constexpr int kSmallWords = kSmallPoints / 32;

template <int M>
__global__ void __launch_bounds__(kSmallPoints)
nds_small(SplitPop pop, int target, int* __restrict__ fronts, int* __restrict__ counters)
{
    constexpr int kM4 = (M + 3) & ~3;
    __shared__ __align__(16) float s_f[kSmallPoints][kM4];
    __shared__ float s_cv[kSmallPoints];
    __shared__ unsigned s_feas[kSmallWords], s_inf[kSmallWords];  // class 0; class 2
    __shared__ unsigned s_any[kSmallWords];                       // class 0 or 1
    __shared__ unsigned s_u[kSmallWords];                         // unassigned
    __shared__ int s_cnt[2];
    const int n = pop.n, q = threadIdx.x, lane = q & 31, warp = q >> 5;
    const int words = (n + 31) >> 5;
    float f[kM4];
#pragma unroll
    for (int m = 0; m < kM4; ++m) f[m] = 0.0f;
    float cv = 0.0f;
    int cls = 4;
    if (q < n) {
        cv = pop.cvv(q);
        bool nan = false;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            f[m] = pop.obj(m, q);
            nan |= isnan(f[m]);
        }
        cls = cv == 0.0f ? (nan ? 1 : 0) : (isnan(cv) ? 3 : 2);
    }
#pragma unroll
    for (int m = 0; m < kM4; ++m) s_f[q][m] = f[m];
    s_cv[q] = cv;
    const unsigned c0 = __ballot_sync(0xFFFFFFFFu, cls == 0), c2 = __ballot_sync(0xFFFFFFFFu, cls == 2);
    const unsigned c01 = __ballot_sync(0xFFFFFFFFu, cls <= 1), all = __ballot_sync(0xFFFFFFFFu, cls <= 3);
    if (lane == 0) {
        s_feas[warp] = c0;
        s_inf[warp] = c2;
        s_any[warp] = c01;
        s_u[warp] = all;
    }
    if (q < 2) s_cnt[q] = 0;
    __syncthreads();
    // dominators of q among the words of points
    uint32_t row[kSmallWords];
#pragma unroll
    for (int w = 0; w < kSmallWords; ++w) {
        row[w] = 0u;
        if (w >= words) continue;
        uint32_t bits = 0u;
        if (cls == 0) {
#pragma unroll 4
            for (int k = 0; k < 32; ++k) {
                bool le = true, lt = false;
#pragma unroll
                for (int v = 0; v < kM4; v += 4) {
                    const float4 g = *reinterpret_cast<const float4*>(&s_f[32 * w + k][v]);
                    const float p[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
                    for (int m = v; m < v + 4 && m < M; ++m) {
                        le &= p[m - v] <= f[m];
                        lt |= p[m - v] < f[m];
                    }
                }
                bits |= (le && lt ? 1u : 0u) << k;
            }
            bits &= s_feas[w];
        } else if (cls == 2) {
            for (int k = 0; k < 32; ++k) bits |= (s_cv[32 * w + k] < cv ? 1u : 0u) << k;
            bits = (bits & s_inf[w]) | s_any[w];
        } else if (cls == 3) {
            bits = s_any[w];
        }
        row[w] = bits;
    }
    int mine = -1, total = 0, k = 0;
    bool alive = q < n;
    for (;; ++k) {
        uint32_t left = 0u;
#pragma unroll
        for (int w = 0; w < kSmallWords; ++w)
            if (w < words) left |= row[w] & s_u[w];
        const bool is_free = alive && left == 0u;
        const unsigned fm = __ballot_sync(0xFFFFFFFFu, is_free);
        if (lane == 0 && fm) atomicAdd(&s_cnt[k & 1], __popc(fm));
        if (is_free) {
            mine = k;
            alive = false;
        }
        __syncthreads();  // everyone has read U; the front's size is complete
        const int ck = s_cnt[k & 1];
        if (lane == 0) s_u[warp] &= ~fm;
        total += ck;
        if (total >= target || ck == 0) {
            if (q == 0) {
                counters[2] = k;
                counters[3] = total;
                if (ck == 0 && total < target) atomicExch(counters + 6, kDevPeelInconsistent);
            }
            break;
        }
        if (q == 0) s_cnt[(k + 1) & 1] = 0;
        __syncthreads();  // U without front k; the next counter is clear
    }
    if (q < n) fronts[q] = mine;
}

template <int M>
void launch_small(const SplitPop& pop, int target, int* fronts, int* counters, cudaStream_t stream)
{
    nds_small<M><<<1, ((pop.n + 31) >> 5) * 32, 0, stream>>>(pop, target, fronts, counters);
}

// Self-test of the peel's two barrier waits with a short limit: every CTA
// arrives, but the barrier asks for one arrival more than the grid has, so
// the wait runs out and records kDevBarrierTimeout.  which 0: the counted
// barrier of nds_peel_owned; 1: grid_barrier of nds_peel.
__global__ void selftest_barrier_wait(int* counters, int which, unsigned long long limit_ns)
{
    if (which == 0) {
        if (threadIdx.x == 0)
            counted_arrive(reinterpret_cast<unsigned long long*>(counters + 16), 0u,
                           (unsigned long long)gridDim.x + 1ull, counters + 6, limit_ns);
    } else {
        grid_barrier(counters, gridDim.x + 1u, 1, limit_ns);
    }
}

}  // namespace

int selftest_barrier_timeout(Workspace& ws, int which, unsigned long long limit_ns, cudaStream_t stream)
{
    nds_reset_counters<<<1, 32, 0, stream>>>(ws.counters);
    selftest_barrier_wait<<<2, 32, 0, stream>>>(ws.counters, which, limit_ns);
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

size_t cub_temp_bytes_needed(int n_max)
{
    size_t a = 0, b = 0, c = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, a, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (int*)nullptr, (int*)nullptr, n_max);
    cub::DeviceRadixSort::SortPairs(nullptr, b, (uint64_t*)nullptr, (uint64_t*)nullptr,
                                    (int*)nullptr, (int*)nullptr, n_max);
    cub::DeviceScan::InclusiveScan(nullptr, c, (int*)nullptr, (int*)nullptr, cub::Max(), n_max);
    size_t m = a > b ? a : b;
    return m > c ? m : c;
}

int run_ndsort(Workspace& ws, const SplitPop& pop, int M, int target, int* out_fronts,
               cudaStream_t stream)
{
    const int n = pop.n;
    if (n <= 0) return MOEA_OK;
    if (n > ws.n_max || M < 1 || M > ws.m_max)
        return set_error(MOEA_ERR_INVALID_ARGUMENT, "ndsort: n=%d M=%d exceed the workspace (%d, %d)",
                         n, M, ws.n_max, ws.m_max);
    if (target > n) target = n;
    if (target < 1) target = 1;
    int* fronts = out_fronts ? out_fronts : ws.fronts;
    const int T = 256, G = ceil_div(n, T);

    if (n <= kSmallPoints && (long long)n * n * (M + 1) <= kSmallWork && !ws.peel_general && !ws.word_tiles) {
        switch (M) {
#define MOEA_SM_CASE(K) case K: launch_small<K>(pop, target, fronts, ws.counters, stream); break;
        MOEA_SM_CASE(1) MOEA_SM_CASE(2) MOEA_SM_CASE(3) MOEA_SM_CASE(4)
        MOEA_SM_CASE(5) MOEA_SM_CASE(6) MOEA_SM_CASE(7) MOEA_SM_CASE(8)
        MOEA_SM_CASE(9) MOEA_SM_CASE(10) MOEA_SM_CASE(11) MOEA_SM_CASE(12)
        MOEA_SM_CASE(13) MOEA_SM_CASE(14) MOEA_SM_CASE(15) MOEA_SM_CASE(16)
#undef MOEA_SM_CASE
        default: return set_error(MOEA_ERR_UNSUPPORTED, "ndsort: M=%d", M);
        }
        MOEA_CUDA_TRY(cudaGetLastError());
        stage_mark("ndsort.peel", stream);
        return MOEA_OK;
    }
    nds_sort_tiles<<<ceil_div(n, kSortTile), kSortTile, 0, stream>>>(pop, M, ws.key0, ws.key64[0], ws.perm[0],
                                                                     ws.counters);
    int cur = 0;
    for (long long L = kSortTile; L < n; L *= kSortWays, cur ^= 1)
        nds_sort_merge<<<G, T, 0, stream>>>(ws.key64[cur], ws.perm[cur], ws.key64[cur ^ 1], ws.perm[cur ^ 1], n, (int)L);
    const uint64_t* skey = ws.key64[cur];
    int* perm = ws.perm[cur ^ 1];
    // runs of equal keys in class 0 into lexicographic order; ws.run_start
    // holds the list of long runs
    nds_tie_rank<<<G, T, 0, stream>>>(pop, M, skey, ws.perm[cur], perm, ws.run_start, ws.counters + 13);
    nds_tie_fix_long<<<kTieLongCtas, kTieLongThreads, 0, stream>>>(pop, M, skey, perm, ws.run_start, ws.counters + 13);
    int* qinfo = ws.qinfo;
    nds_finalize_rows<<<G, T, 0, stream>>>(pop, M, ws.key0, skey, perm, ws.sorted_f, ws.n_max, ws.counters, qinfo,
                                           ws.blocker, ws.front_sorted, ws.peel_fmask, 3 * ws.words);
    MOEA_CUDA_TRY(cudaGetLastError());
    stage_mark("ndsort.lexsort", stream);

    switch (M) {
    case 1: launch_tiles<1>(ws, n, stream); break;
    case 2: launch_tiles<2>(ws, n, stream); break;
    case 3: launch_tiles<3>(ws, n, stream); break;
    case 4: launch_tiles<4>(ws, n, stream); break;
    case 5: launch_tiles<5>(ws, n, stream); break;
    case 6: launch_tiles<6>(ws, n, stream); break;
    case 7: launch_tiles<7>(ws, n, stream); break;
    case 8: launch_tiles<8>(ws, n, stream); break;
    case 9: launch_tiles<9>(ws, n, stream); break;
    case 10: launch_tiles<10>(ws, n, stream); break;
    case 11: launch_tiles<11>(ws, n, stream); break;
    case 12: launch_tiles<12>(ws, n, stream); break;
    case 13: launch_tiles<13>(ws, n, stream); break;
    case 14: launch_tiles<14>(ws, n, stream); break;
    case 15: launch_tiles<15>(ws, n, stream); break;
    case 16: launch_tiles<16>(ws, n, stream); break;
    default: return set_error(MOEA_ERR_UNSUPPORTED, "ndsort: M=%d", M);
    }
    MOEA_CUDA_TRY(cudaGetLastError());
    stage_mark("ndsort.dominance_tiles", stream);

    // cooperative peel; nds_finalize_rows left its three front masks empty
    // every co-resident CTA with at least one group of 32 positions: each
    // CTA scans the rows of its own groups, so more CTAs mean fewer rows per
    // CTA and front (one CTA per group of 32 warps left half the SMs idle)
    int grid = ceil_div(n, 32);
    if (grid > ws.peel_grid) grid = ws.peel_grid;
    if (grid < 1 || ws.peel_single_cta) grid = 1;
    const uint32_t* rows = ws.rows;
    int Wp = ws.words;
    int nn = n, tt = target;
    const int* qi = qinfo;
    int* blk = ws.blocker;
    int* fs = ws.front_sorted;
    uint32_t* fmask = ws.peel_fmask;
    int* ctr = ws.counters;
    void* args[] = {(void*)&rows, (void*)&Wp, (void*)&nn, (void*)&tt, (void*)&qi,
                    (void*)&blk, (void*)&fs, (void*)&fmask, (void*)&ctr};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kPeelThreads);
    cfg.dynamicSmemBytes = (size_t)ws.words * sizeof(uint32_t);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // lane-owned points when every warp of the grid holds at most one group
    // of 32 positions and the rows are 16-byte aligned
    const bool owned = !ws.peel_general && ws.peel_owned_grid > 0 && ceil_div(n, 32) <= 32 * min(grid, ws.peel_owned_grid) &&
                       Wp >= kWin && (Wp & 3) == 0;
    if (owned) {
        if (grid > ws.peel_owned_grid) grid = ws.peel_owned_grid;
        const int* b0 = ws.blocker;
        void* oargs[] = {(void*)&rows, (void*)&Wp, (void*)&nn, (void*)&tt, (void*)&b0,
                         (void*)&fs, (void*)&fmask, (void*)&ctr};
        cfg.gridDim = dim3(grid);
        cfg.dynamicSmemBytes = peel_owned_smem(Wp);
        if (grid == 1) {
            nds_peel_owned<<<1, kPeelThreads, cfg.dynamicSmemBytes, stream>>>(rows, Wp, nn, tt, b0, fs, fmask,
                                                                              ctr);
        } else {
            MOEA_CUDA_TRY(cudaLaunchKernelExC(&cfg, (const void*)nds_peel_owned, oargs));
        }
    } else if (grid == 1) {
        // one CTA needs no co-residency guarantee: an ordinary launch, which
        // may run beside other work (batched instances)
        nds_peel<<<1, kPeelThreads, cfg.dynamicSmemBytes, stream>>>(rows, Wp, nn, tt, qi, blk, fs, fmask,
                                                                    ctr);
    } else {
        MOEA_CUDA_TRY(cudaLaunchKernelExC(&cfg, (const void*)nds_peel, args));
    }

    nds_fronts<<<kFrontCtas, kFrontThreads, 0, stream>>>(n, perm, qinfo, ws.front_sorted, ws.counters, target, fronts);
    MOEA_CUDA_TRY(cudaGetLastError());
    stage_mark("ndsort.peel", stream);
    return MOEA_OK;
}

// Raises a kernel's dynamic shared-memory limit to at least `bytes`.  The
// limit belongs to the function, not to a workspace, so it is never lowered:
// a smaller workspace created later must not shrink the launch of a larger one.
static int raise_dynamic_smem(const void* func, size_t bytes)
{
    cudaFuncAttributes fa = {};
    MOEA_CUDA_TRY(cudaFuncGetAttributes(&fa, func));
    if ((size_t)fa.maxDynamicSharedSizeBytes < bytes)
        MOEA_CUDA_TRY(cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return MOEA_OK;
}

// Words of block tables a workspace of n_max points and m_max objectives
// needs for every objective count up to m_max.
size_t block_table_words(int n_max, int m_max)
{
    if (m_max < 2) return 0;
    const size_t lo = (size_t)ceil_div(n_max, 256) * (size_t)(m_max < 4 ? m_max - 1 : 3) * BlockTable<256>::kSize;
    const size_t hi = m_max >= 5 ? (size_t)ceil_div(n_max, 128) * (size_t)(m_max - 1) * BlockTable<128>::kSize : 0;
    return lo > hi ? lo : hi;
}

// Shared-memory limits of the block-row kernels beyond 48 KB.
int configure_block_rows()
{
#define MOEA_BR_CASE(K) \
    if (block_rows_smem<K>() > 48 * 1024) \
        MOEA_TRY(raise_dynamic_smem((const void*)nds_block_rows<K, BlockCfg<K>::kB>, block_rows_smem<K>()));
    MOEA_BR_CASE(2) MOEA_BR_CASE(3) MOEA_BR_CASE(4) MOEA_BR_CASE(5) MOEA_BR_CASE(6) MOEA_BR_CASE(7)
    MOEA_BR_CASE(8) MOEA_BR_CASE(9) MOEA_BR_CASE(10) MOEA_BR_CASE(11) MOEA_BR_CASE(12) MOEA_BR_CASE(13)
    MOEA_BR_CASE(14) MOEA_BR_CASE(15) MOEA_BR_CASE(16)
#undef MOEA_BR_CASE
    return MOEA_OK;
}

// Configure the co-resident grid of the peel kernel for this device.
int configure_peel(Workspace& ws)
{
    const size_t smem = (size_t)ws.words * sizeof(uint32_t);
    if (smem > 48 * 1024) MOEA_TRY(raise_dynamic_smem((const void*)nds_peel, smem));
    int per_sm = 0;
    MOEA_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, nds_peel, kPeelThreads,
                                                                smem));
    int sms = 0;
    MOEA_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ws.device));
    ws.sm_count = sms;
    if (per_sm < 1)
        return set_error(MOEA_ERR_UNSUPPORTED, "peel kernel does not fit on an SM (smem %zu)", smem);
    ws.peel_grid = sms * (per_sm > 2 ? 2 : per_sm);
    ws.peel_smem = (int)smem;
    // the lane-owned peel: one CTA per SM
    ws.peel_owned_grid = 0;
    const size_t osmem = peel_owned_smem(ws.words);
    int optin = 0;
    MOEA_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ws.device));
    cudaFuncAttributes ofa = {};
    MOEA_CUDA_TRY(cudaFuncGetAttributes(&ofa, (const void*)nds_peel_owned));
    if (ws.words >= kWin && osmem + ofa.sharedSizeBytes <= (size_t)optin) {
        MOEA_TRY(raise_dynamic_smem((const void*)nds_peel_owned, osmem));
        int oper = 0;
        MOEA_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&oper, nds_peel_owned, kPeelThreads, osmem));
        if (oper >= 1) ws.peel_owned_grid = sms;
    }
    return MOEA_OK;
}

int fused_tile_blocks(int M, int n, int shape)
{
    switch (M) {
#define MOEA_TB_CASE(K) case K: return tile_blocks_of<K>(n, shape);
    MOEA_TB_CASE(1) MOEA_TB_CASE(2) MOEA_TB_CASE(3) MOEA_TB_CASE(4)
    MOEA_TB_CASE(5) MOEA_TB_CASE(6) MOEA_TB_CASE(7) MOEA_TB_CASE(8)
    MOEA_TB_CASE(9) MOEA_TB_CASE(10) MOEA_TB_CASE(11) MOEA_TB_CASE(12)
    MOEA_TB_CASE(13) MOEA_TB_CASE(14) MOEA_TB_CASE(15) MOEA_TB_CASE(16)
#undef MOEA_TB_CASE
    default: return 0;
    }
}

// U takes the workspace's row words W (4 * ceil(n / 128) for a workspace of n
// merged points), then blockers, front list, queue, heads and
// links of n entries each.
size_t fused_peel_smem(int W, int n) { return (size_t)W * sizeof(uint32_t) + 5 * (size_t)n * sizeof(int); }

int fused_ndsort_configure()
{
#define MOEA_BR_CASE(K) \
    if (block_rows_smem<K>() > 48 * 1024) \
        MOEA_TRY(raise_dynamic_smem((const void*)fused_block_rows<K>, block_rows_smem<K>()));
    MOEA_BR_CASE(2) MOEA_BR_CASE(3) MOEA_BR_CASE(4) MOEA_BR_CASE(5) MOEA_BR_CASE(6) MOEA_BR_CASE(7)
    MOEA_BR_CASE(8) MOEA_BR_CASE(9) MOEA_BR_CASE(10) MOEA_BR_CASE(11) MOEA_BR_CASE(12) MOEA_BR_CASE(13)
    MOEA_BR_CASE(14) MOEA_BR_CASE(15) MOEA_BR_CASE(16)
#undef MOEA_BR_CASE
    MOEA_CUDA_TRY(cudaFuncSetAttribute(fused_peel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)fused_peel_smem(4 * ceil_div(kFusedMaxPoints, 128), kFusedMaxPoints)));
    return MOEA_OK;
}

int fused_ndsort(const BatchInst* d_inst, const FusedGroup& g, cudaStream_t s)
{
    const dim3 points(ceil_div(g.max_n, 256), g.count);
    fused_sort_tiles<<<dim3(ceil_div(g.max_n, kSortTile), g.count), kSortTile, 0, s>>>(d_inst, g.d_ids);
    if (g.max_n > kSortTile) fused_sort_merge<<<points, 256, 0, s>>>(d_inst, g.d_ids);
    fused_tie_rank<<<points, 256, 0, s>>>(d_inst, g.d_ids);
    fused_tie_long<<<g.count, kTieLongThreads, 0, s>>>(d_inst, g.d_ids);
    fused_finalize_rows<<<points, 256, 0, s>>>(d_inst, g.d_ids);
    MOEA_CUDA_TRY(cudaGetLastError());
    for (const FusedBucket& b : g.buckets) {
        switch (b.M) {
#define MOEA_FT_CASE(K) case K: MOEA_TRY(launch_fused_rows<K>(d_inst, b, s)); break;
        MOEA_FT_CASE(1) MOEA_FT_CASE(2) MOEA_FT_CASE(3) MOEA_FT_CASE(4)
        MOEA_FT_CASE(5) MOEA_FT_CASE(6) MOEA_FT_CASE(7) MOEA_FT_CASE(8)
        MOEA_FT_CASE(9) MOEA_FT_CASE(10) MOEA_FT_CASE(11) MOEA_FT_CASE(12)
        MOEA_FT_CASE(13) MOEA_FT_CASE(14) MOEA_FT_CASE(15) MOEA_FT_CASE(16)
#undef MOEA_FT_CASE
        default: return set_error(MOEA_ERR_UNSUPPORTED, "fused ndsort: M=%d", b.M);
        }
    }
    fused_peel<<<g.count, kFusedPeelThreads, fused_peel_smem(g.max_W, g.max_n), s>>>(d_inst, g.d_ids);
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

}  // namespace moea

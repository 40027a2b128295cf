// Association by a dense search in FP32: every direction visited by every
// point (association.cu:86-188, 397-447, 586-608 of the reference's NSGA-III
// kernels).
//
// For unit directions r_j the perpendicular distance satisfies
// d2_j = |x|^2 - (x.r_j)^2 up to rounding, so the reference argmin is found
// among the directions whose dot^2 lies within a rounding margin
// (assoc_margin) of the largest.  Two passes: the first forms only the largest
// |dot| of each point and tile of directions (M FMAs and one maximum per pair,
// no branch); the second re-scores, with the reference's FP32 formula
// (association.cu:139-170: fmaf dot, contracted residual, fmaf sum of squares),
// the directions of the tiles whose largest dot^2 reaches the point's threshold
// -- one or two tiles of 32 for most points, a warp per point, a lane per
// direction.  The minimum of (d2, index) over them is the reference's argmin
// with its tie rule.  Points whose squared length overflows re-score every tile,
// points with a coordinate that is not finite none; directions far from unit
// length take one pass over every distance (dense_block_free).
//
// A CTA holds 32 or 64 points; its eight warps take the tiles in turn, each
// through its own 32-direction buffer in shared memory, so the first pass has
// no block barrier.  With 64 points (two per lane, every lane on the same
// direction) it is bound by issue: M + 1 instructions per pair, and 130 per point
// for the re-score.  Four directions side by side with eight points per lane
// need fewer reads but four LSU cycles for each: 428 against 341 us over the 85
// eight-objective instances of a batch.  With 32 points, for populations that
// do not fill the SMs, the same split (four points per lane) shortens a warp's
// chain: M=3 N=2048 H=1953 14 against 18 us with event overhead, M=5 N=3002
// H=2380 20 against 24.
#include "assoc_dense.cuh"

namespace moea {
namespace {

constexpr int kDenseWarps = 8;
constexpr int kDenseThreads = 32 * kDenseWarps;
constexpr int kDenseMaxTiles = 128;   // tiles per point told apart; a tile holds a multiple of 32 directions

template <int M, int PTS>
struct DenseShared {
    static constexpr int kM4 = (M + 3) & ~3;
    static constexpr int kLanes = PTS == 32 ? 8 : 32;  // lanes that hold all points
    static constexpr int kPer = PTS / kLanes;          // points per lane
    static constexpr int kGroups = 32 / kLanes;        // directions side by side
    float dir[kDenseWarps][32][kM4];
    float tile[kDenseMaxTiles][PTS];
    float x[PTS][M];
    float part[kDenseThreads / PTS][PTS];
    uint32_t todo[kDenseThreads / PTS][PTS];  // candidate tiles: bit i of part k is tile i * parts + k
    float margin[PTS], thr[PTS];
};

// dense_block for directions that are not of unit length (the margin is infinite
// for every point): the pass over the tiles forms every distance itself, where
// the re-score of all tiles would read the directions of each point again from
// device memory.
template <int M, int PTS>
__device__ __noinline__ void dense_block_free(DenseShared<M, PTS>& sm, int p0, const float* __restrict__ x,
                                                 int x_stride, const float* __restrict__ scale,
                                                 const float* __restrict__ refs, int H, int n,
                                                 int* __restrict__ idx_out, float* __restrict__ dist_out)
{
    using S = DenseShared<M, PTS>;
    constexpr int P = S::kPer;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = lane % S::kLanes, grp = lane / S::kLanes;
    const int chunks = (H + 31) >> 5;
    float next[M];
    auto fetch = [&](int chunk) {
        const int j = chunk * 32 + lane;
#pragma unroll
        for (int m = 0; m < M; ++m) next[m] = j < H ? __ldg(refs + (size_t)m * H + j) : 0.0f;
    };
    if (warp < chunks) fetch(warp);
    float xr[P][M], best[P];
    int bj[P];
#pragma unroll
    for (int c = 0; c < P; ++c) {
        const int i = p0 + sub + S::kLanes * c;
        best[c] = INFINITY;
        bj[c] = -1;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const float v = i < n ? x[(size_t)m * x_stride + i] : 0.0f;
            xr[c][m] = scale ? v * scale[m] : v;
        }
    }
    for (int ch = warp; ch < chunks; ch += kDenseWarps) {
        __syncwarp();
#pragma unroll
        for (int m = 0; m < M; ++m) sm.dir[warp][lane][m] = next[m];
        __syncwarp();
        if (ch + kDenseWarps < chunks) fetch(ch + kDenseWarps);
        const int cnt = min(32, H - ch * 32);
#pragma unroll 2
        for (int k = grp; k < cnt; k += S::kGroups) {
            float r[S::kM4];
#pragma unroll
            for (int v = 0; v < S::kM4; v += 4) {
                const float4 d = *reinterpret_cast<const float4*>(&sm.dir[warp][k][v]);
                r[v] = d.x;
                r[v + 1] = d.y;
                r[v + 2] = d.z;
                r[v + 3] = d.w;
            }
#pragma unroll
            for (int c = 0; c < P; ++c) {
                float dot = 0.0f, d2 = 0.0f;
#pragma unroll
                for (int m = 0; m < M; ++m) dot = fmaf(xr[c][m], r[m], dot);
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const float res = fmaf(-dot, r[m], xr[c][m]);
                    d2 = fmaf(res, res, d2);
                }
                if (d2 < best[c]) {  // ascending directions: the first of equal ones stays
                    best[c] = d2;
                    bj[c] = ch * 32 + k;
                }
            }
        }
    }
    // (distance, index) minima over the groups and the warps; none found is +inf and -1
    unsigned long long (*found)[PTS] = reinterpret_cast<unsigned long long (*)[PTS]>(&sm.tile[0][0]);
    static_assert(sizeof(sm.tile) >= sizeof(unsigned long long) * kDenseWarps * PTS, "minima fit the tiles' maxima");
#pragma unroll
    for (int c = 0; c < P; ++c) {
        unsigned long long key = ((unsigned long long)__float_as_uint(best[c]) << 32) | (unsigned)bj[c];
#pragma unroll
        for (int o = S::kLanes; o < 32; o <<= 1) {
            const unsigned long long other = __shfl_xor_sync(0xFFFFFFFFu, key, o);
            key = other < key ? other : key;
        }
        if (grp == 0) found[warp][sub + S::kLanes * c] = key;
    }
    __syncthreads();
    if (tid < PTS && p0 + tid < n) {
        unsigned long long key = found[0][tid];
#pragma unroll
        for (int w = 1; w < kDenseWarps; ++w) key = found[w][tid] < key ? found[w][tid] : key;
        idx_out[p0 + tid] = (int)(unsigned)(key & 0xFFFFFFFFull);
        dist_out[p0 + tid] = sqrtf(__uint_as_float((unsigned)(key >> 32)));
    }
}

// kUnit: the host knows that the directions are of unit length (runs and batches;
// a single search finds the deviation on the device).
template <int M, int PTS, bool kUnit>
__device__ __forceinline__ void dense_block(DenseShared<M, PTS>& sm, int p0, const float* __restrict__ x, int x_stride,
                                            const float* __restrict__ scale, const float* __restrict__ refs, int H,
                                            int n, float delta, int* __restrict__ idx_out, float* __restrict__ dist_out)
{
    if (!kUnit && !(delta <= kAssocMaxDelta)) {  // the same for the whole launch, or instance
        dense_block_free<M, PTS>(sm, p0, x, x_stride, scale, refs, H, n, idx_out, dist_out);
        return;
    }
    using S = DenseShared<M, PTS>;
    constexpr int P = S::kPer;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = lane % S::kLanes, grp = lane / S::kLanes;
    // tiles of a multiple of 32 directions
    const int chunks = (H + 31) >> 5;
    const int per = (chunks + kDenseMaxTiles - 1) / kDenseMaxTiles;
    const int tiles = (chunks + per - 1) / per;
    float next[M];
    auto fetch = [&](int chunk) {
        const int j = chunk * 32 + lane;
#pragma unroll
        for (int m = 0; m < M; ++m) next[m] = j < H ? __ldg(refs + (size_t)m * H + j) : 0.0f;
    };
    if (warp < tiles) fetch(warp * per);
    if (tid < PTS) {
        const int i = p0 + tid;
        float xx = 0.0f;
        bool finite = true;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            float v = i < n ? x[(size_t)m * x_stride + i] : 0.0f;
            if (scale) v = v * scale[m];
            sm.x[tid][m] = v;
            finite &= isfinite(v) != 0;
            xx = fmaf(v, v, xx);
        }
        // a coordinate that is not finite leaves NaN distances only: no candidates
        sm.margin[tid] = finite ? assoc_margin(M, xx, delta) : -1.0f;
    }
    __syncthreads();
    float xr[P][M];
#pragma unroll
    for (int c = 0; c < P; ++c)
#pragma unroll
        for (int m = 0; m < M; ++m) xr[c][m] = sm.x[sub + S::kLanes * c][m];
    for (int t = warp; t < tiles; t += kDenseWarps) {
        float mx[P];
#pragma unroll
        for (int c = 0; c < P; ++c) mx[c] = 0.0f;  // |dot| >= 0; a point without a finite dot re-scores everything
        const int c1 = min(chunks, (t + 1) * per);
        for (int ch = t * per; ch < c1; ++ch) {
            __syncwarp();
#pragma unroll
            for (int m = 0; m < M; ++m) sm.dir[warp][lane][m] = next[m];
            __syncwarp();
            if (ch + 1 < c1) fetch(ch + 1);
            else if (t + kDenseWarps < tiles) fetch((t + kDenseWarps) * per);
#pragma unroll (S::kGroups == 1 ? 8 : 2)
            for (int k = grp; k < 32; k += S::kGroups) {
                float r[S::kM4];
#pragma unroll
                for (int v = 0; v < S::kM4; v += 4) {
                    const float4 d = *reinterpret_cast<const float4*>(&sm.dir[warp][k][v]);
                    r[v] = d.x;
                    r[v + 1] = d.y;
                    r[v + 2] = d.z;
                    r[v + 3] = d.w;
                }
#pragma unroll
                for (int c = 0; c < P; ++c) {
                    float dot = 0.0f;
#pragma unroll
                    for (int m = 0; m < M; ++m) dot = fmaf(xr[c][m], r[m], dot);
                    mx[c] = fmaxf(mx[c], fabsf(dot));
                }
            }
        }
#pragma unroll
        for (int c = 0; c < P; ++c) {
#pragma unroll
            for (int o = S::kLanes; o < 32; o <<= 1) mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xFFFFFFFFu, mx[c], o));
            if (grp == 0) sm.tile[t][sub + S::kLanes * c] = mx[c];
        }
    }
    __syncthreads();
    // the points' thresholds
    {
        constexpr int kParts = kDenseThreads / PTS;
        const int q = tid % PTS, part = tid / PTS;
        float m = 0.0f;
        for (int t = part; t < tiles; t += kParts) m = fmaxf(m, sm.tile[t][q]);
        sm.part[part][q] = m;
        __syncthreads();
        if (tid < PTS) {
#pragma unroll
            for (int k = 1; k < kParts; ++k) m = fmaxf(m, sm.part[k][q]);
            const float thr = m * m - sm.margin[q];
            sm.thr[q] = (thr == thr) ? thr : -INFINITY;
        }
        __syncthreads();
        const float thr = sm.thr[q];
        const bool some = !(sm.margin[q] < 0.0f);
        uint32_t todo = 0u;
        for (int t = part, i = 0; t < tiles; t += kParts, ++i) {
            const float tm = sm.tile[t][q];
            todo |= (some && tm * tm >= thr ? 1u : 0u) << i;
        }
        sm.todo[part][q] = todo;
        __syncthreads();
    }
    // re-score: a warp per point, a lane per direction
    constexpr int kParts = kDenseThreads / PTS;
    static_assert(kDenseMaxTiles / kParts <= 32, "a part's candidate tiles fit a word");
    for (int q = warp; q < PTS; q += kDenseWarps) {
        if (p0 + q >= n) break;
        const float thr = sm.thr[q];
        float xq[M];
#pragma unroll
        for (int m = 0; m < M; ++m) xq[m] = sm.x[q][m];
        float best = INFINITY;
        int bj = -1;
        for (int part = 0; part < kParts; ++part) {
            uint32_t todo = sm.todo[part][q];
            while (todo) {
                const int t = (__ffs(todo) - 1) * kParts + part;
                todo &= todo - 1;
                const int c1 = min(chunks, (t + 1) * per);
                for (int ch = t * per; ch < c1; ++ch) {
                    const int j = ch * 32 + lane;
                    if (j >= H) continue;
                    float r[M], dot = 0.0f;
#pragma unroll
                    for (int m = 0; m < M; ++m) r[m] = __ldg(refs + (size_t)m * H + j);
#pragma unroll
                    for (int m = 0; m < M; ++m) dot = fmaf(xq[m], r[m], dot);
                    const float dd = dot * dot;
                    if (!(dd >= thr)) continue;
                    float d2 = 0.0f;
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        const float res = fmaf(-dot, r[m], xq[m]);
                        d2 = fmaf(res, res, d2);
                    }
                    if (d2 < best || (d2 == best && j < bj)) {  // an infinite distance is never taken
                        best = d2;
                        bj = j;
                    }
                }
            }
        }
        // non-negative floats order as their bits; none found is +inf and index -1
        const unsigned bits = __reduce_min_sync(0xFFFFFFFFu, __float_as_uint(best));
        const unsigned j = __reduce_min_sync(0xFFFFFFFFu, __float_as_uint(best) == bits ? (unsigned)bj : 0xFFFFFFFFu);
        if (lane == 0) {
            idx_out[p0 + q] = (int)j;
            dist_out[p0 + q] = sqrtf(__uint_as_float(bits));
        }
    }
}

template <int M, int PTS, bool kUnit>
__global__ void __launch_bounds__(kDenseThreads)
assoc_dense(const float* __restrict__ x, int x_stride, const float* __restrict__ scale, const float* __restrict__ refs,
            int H, const int* __restrict__ d_n, float delta, const float* __restrict__ d_delta, int* __restrict__ idx_out,
            float* __restrict__ dist_out)
{
    extern __shared__ __align__(16) unsigned char dense_raw[];
    const int n = *d_n, p0 = blockIdx.x * PTS;
    if (p0 >= n) return;
    dense_block<M, PTS, kUnit>(*reinterpret_cast<DenseShared<M, PTS>*>(dense_raw), p0, x, x_stride, scale, refs, H, n,
                      d_delta ? *d_delta : delta, idx_out, dist_out);
}

// Every instance of a bucket of M objectives (blockIdx.y).
template <int M, int PTS, bool kUnit>
__global__ void __launch_bounds__(kDenseThreads)
fused_assoc_dense(const BatchInst* __restrict__ insts, const int* __restrict__ ids)
{
    extern __shared__ __align__(16) unsigned char dense_raw[];
    const BatchInst& I = insts[ids[blockIdx.y]];
    const int n = I.sizes[3], p0 = blockIdx.x * PTS;
    if (p0 >= n) return;
    dense_block<M, PTS, kUnit>(*reinterpret_cast<DenseShared<M, PTS>*>(dense_raw), p0, I.nds_objs, I.n_max, I.rcp_b, I.t_dirs_orig,
                      I.H, n, I.t_delta, I.assoc_idx, I.assoc_dist);
}

// Raises the kernel's shared-memory limit when its block needs more than 48 KB.
template <class K>
cudaError_t dense_smem(K kernel, size_t bytes)
{
    return bytes > 48 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)
                             : cudaSuccess;
}

template <int M, int PTS, bool kUnit>
int launch_dense(const float* x, int x_stride, const float* scale, const float* refs, int H, const int* d_n, int n_cap,
                 float delta, const float* d_delta, int* idx, float* dist, cudaStream_t stream)
{
    constexpr size_t smem = sizeof(DenseShared<M, PTS>);
    MOEA_CUDA_TRY((dense_smem(assoc_dense<M, PTS, kUnit>, smem)));
    assoc_dense<M, PTS, kUnit><<<ceil_div(n_cap, PTS), kDenseThreads, smem, stream>>>(x, x_stride, scale, refs, H, d_n,
                                                                                      delta, d_delta, idx, dist);
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

// Points from which CTAs of 64 are used: half of the SMs have a second one then
// (M=3 / 8 with 30,000 directions, CTAs of 32 and of 64: 12,500 points 126 / 171
// and 227 / 281 us, 16,000 points 155 / 175 and 298 / 282).
constexpr int kDenseWideFrom = 148 * 96;

// Where the dense search is the faster one (both with random directions,
// microseconds, dense / scan).  One objective: every direction is a candidate
// (64 points, 10,000 directions 153 / 48).  Up to two chunks of directions, or few
// beside the points, most warps have no tile (60,000 points, M=16: 33 directions
// 44 / 16, 300 60 / 46, 1,000 93 / 115).  Two objectives: neighbouring directions
// fall within the margin (500 points: 4,000 29 / 44, 8,000 58 / 47; 16,000
// points: 2,000 33 / 44, 4,000 63 / 51).  Many directions and few points leave SMs
// without a block of points (M=5, 64 points: 10,000 38 / 50, 16,000 55 / 54,
// 100,000 290 / 100; 4,000 points: 20,000 68 / 87, 100,000 302 / 279), from twelve
// objectives on and with directions of any length a little earlier (M=16, 64
// points: 8,000 110 / 105, 10,000 136 / 107).
inline bool dense_search_wins(int M, int n, int H)
{
    if (M == 1 || H <= 64 || (M >= 12 ? 64ll : 128ll) * H <= n) return false;
    if (M == 2) return H <= (n < 148 * 64 ? 4096 : 2048);
    return H <= (M >= 12 ? 8192 : 12288) || (long long)H <= 6ll * n;
}

}  // namespace

template <bool kUnit>
static int run_assoc_dense(const float* x, int x_stride, const float* scale, const float* refs, int M, const int* d_n,
                           int n_cap, int H, float delta, const float* d_delta, int* idx, float* dist,
                           cudaStream_t stream)
{
    const bool wide = n_cap >= kDenseWideFrom;
    switch (M) {
#define MOEA_DENSE_CASE(K)                                                                                         \
    case K:                                                                                                        \
        return wide ? launch_dense<K, 64, kUnit>(x, x_stride, scale, refs, H, d_n, n_cap, delta, d_delta, idx, dist, \
                                                 stream)                                                           \
                    : launch_dense<K, 32, kUnit>(x, x_stride, scale, refs, H, d_n, n_cap, delta, d_delta, idx, dist, \
                                                 stream);
    MOEA_DENSE_CASE(2) MOEA_DENSE_CASE(3) MOEA_DENSE_CASE(4) MOEA_DENSE_CASE(5) MOEA_DENSE_CASE(6)
    MOEA_DENSE_CASE(7) MOEA_DENSE_CASE(8) MOEA_DENSE_CASE(9) MOEA_DENSE_CASE(10) MOEA_DENSE_CASE(11)
    MOEA_DENSE_CASE(12) MOEA_DENSE_CASE(13) MOEA_DENSE_CASE(14) MOEA_DENSE_CASE(15) MOEA_DENSE_CASE(16)
#undef MOEA_DENSE_CASE
    default: return set_error(MOEA_ERR_UNSUPPORTED, "associate: M=%d", M);
    }
}

int run_assoc_search(const float* x, int x_stride, const float* scale, const float* refs, int M, const int* d_n, int n_cap,
                     int H, float delta, const float* d_delta, unsigned long long* best, int sms, int* idx, float* dist,
                     cudaStream_t stream)
{
    if (n_cap <= 0) return MOEA_OK;
    if (dense_search_wins(M, n_cap, H))
        return !d_delta && delta <= kAssocMaxDelta
                   ? run_assoc_dense<true>(x, x_stride, scale, refs, M, d_n, n_cap, H, delta, nullptr, idx, dist, stream)
                   : run_assoc_dense<false>(x, x_stride, scale, refs, M, d_n, n_cap, H, delta, d_delta, idx, dist, stream);
    return run_assoc_scan(x, x_stride, scale, refs, M, d_n, n_cap, H, delta, d_delta, best, sms, idx, dist, stream);
}

template <int M, bool kUnit>
static int launch_fused_dense(const BatchInst* d_inst, const FusedBucket& b, cudaStream_t s)
{
    constexpr size_t smem = sizeof(DenseShared<M, 64>);
    MOEA_CUDA_TRY((dense_smem(fused_assoc_dense<M, 64, kUnit>, smem)));
    fused_assoc_dense<M, 64, kUnit><<<dim3(ceil_div(b.max_n, 64), b.count), kDenseThreads, smem, s>>>(d_inst, b.d_ids);
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

int fused_associate_dense(const BatchInst* d_inst, const FusedBucket& b, cudaStream_t s)
{
    switch (b.M) {
#define MOEA_DENSE_CASE(K) \
    case K: return b.unit ? launch_fused_dense<K, true>(d_inst, b, s) : launch_fused_dense<K, false>(d_inst, b, s);
    MOEA_DENSE_CASE(1) MOEA_DENSE_CASE(2) MOEA_DENSE_CASE(3) MOEA_DENSE_CASE(4)
    MOEA_DENSE_CASE(5) MOEA_DENSE_CASE(6) MOEA_DENSE_CASE(7) MOEA_DENSE_CASE(8)
    MOEA_DENSE_CASE(9) MOEA_DENSE_CASE(10) MOEA_DENSE_CASE(11) MOEA_DENSE_CASE(12)
    MOEA_DENSE_CASE(13) MOEA_DENSE_CASE(14) MOEA_DENSE_CASE(15) MOEA_DENSE_CASE(16)
#undef MOEA_DENSE_CASE
    default: return set_error(MOEA_ERR_UNSUPPORTED, "fused associate: M=%d", b.M);
    }
}

}  // namespace moea

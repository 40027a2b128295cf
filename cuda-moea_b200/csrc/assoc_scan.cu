// Association by a thread per point over ranges of directions (association.cu:86-188,
// 397-447, 586-608 of the reference's NSGA-III kernels), where the dense search
// (assoc_dense.cu) has too little to do or too many candidates.
//
// Each thread keeps a running maximum of dot^2 and evaluates the reference's FP32
// formula (association.cu:139-170) for the directions within the rounding margin
// of it only.  Ties keep the smaller index within a thread (ascending j, strict <)
// and across ranges through a packed (d2 bits, j) atomicMin, so the result is the
// reference's argmin, as the dense search's.
#include "assoc_dense.cuh"

namespace moea {
namespace {

constexpr int kAssocThreads = 256;
constexpr int kAssocTile = 1024;

template <int M>
struct DirTile {
    static constexpr int kLen = (M <= 4) ? kAssocTile : 512;  // directions per shared-memory tile
};

// One block of points (bx) against one range of directions (by).  With
// best_out the packed (d2, index) minimum is merged atomically across ranges;
// without it the block covers every direction and writes idx/dist directly.
template <int M>
__device__ __forceinline__ void assoc_scan_block(int bx, int by, const float* __restrict__ x, int x_stride,
                                                 const float* __restrict__ scale,
                                                 const float* __restrict__ refs, int H, int n, int split_len,
                                                 float delta, unsigned long long* __restrict__ best_out,
                                                 int* __restrict__ idx_out, float* __restrict__ dist_out)
{
    constexpr int TL = DirTile<M>::kLen;
    __shared__ __align__(16) float s_dir[TL * ((M <= 4) ? 4 : M)];
    const int i = bx * kAssocThreads + threadIdx.x;
    const int j_begin = by * split_len;
    const int j_end = min(H, j_begin + split_len);
    if (bx * kAssocThreads >= n || j_begin >= j_end) return;
    const bool valid = i < n;
    float xr[M];
    float xx = 0.0f;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        float v = valid ? x[(size_t)m * x_stride + i] : 0.0f;
        if (scale) v = v * scale[m];
        xr[m] = v;
        xx = fmaf(v, v, xx);
    }
    const float margin = assoc_margin(M, xx, delta);
    // coarse pre-pass over a strided subset to start with a tight threshold
    float maxd = -INFINITY;
    for (int j = j_begin; j < j_end; j += 61) {
        float dot = 0.0f;
#pragma unroll
        for (int m = 0; m < M; ++m) dot = fmaf(xr[m], __ldg(refs + (size_t)m * H + j), dot);
        maxd = fmaxf(maxd, dot * dot);
    }
    float thr = maxd - margin;
    if (!(thr == thr)) thr = -INFINITY;
    float best = INFINITY;
    int bj = -1;
    for (int t0 = j_begin; t0 < j_end; t0 += TL) {
        const int cnt = min(TL, j_end - t0);
        __syncthreads();
        for (int t = threadIdx.x; t < cnt; t += kAssocThreads) {
            if (M <= 4) {
                float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
                d.x = refs[t0 + t];
                if (M > 1) d.y = refs[(size_t)H + t0 + t];
                if (M > 2) d.z = refs[(size_t)2 * H + t0 + t];
                if (M > 3) d.w = refs[(size_t)3 * H + t0 + t];
                reinterpret_cast<float4*>(s_dir)[t] = d;
            } else {
#pragma unroll
                for (int m = 0; m < M; ++m) s_dir[(size_t)m * TL + t] = refs[(size_t)m * H + t0 + t];
            }
        }
        __syncthreads();
        if (!valid) continue;
#pragma unroll 4
        for (int t = 0; t < cnt; ++t) {
            float r[M];
            if (M <= 4) {
                const float4 d = reinterpret_cast<const float4*>(s_dir)[t];
                r[0] = d.x;
                if (M > 1) r[1 % M] = d.y;
                if (M > 2) r[2 % M] = d.z;
                if (M > 3) r[3 % M] = d.w;
            } else {
#pragma unroll
                for (int m = 0; m < M; ++m) r[m] = s_dir[(size_t)m * TL + t];
            }
            float dot = 0.0f;
#pragma unroll
            for (int m = 0; m < M; ++m) dot = fmaf(xr[m], r[m], dot);
            const float dd = dot * dot;
            if (dd >= thr) {
                float d2 = 0.0f;
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const float res = fmaf(-dot, r[m], xr[m]);
                    d2 = fmaf(res, res, d2);
                }
                if (d2 < best) { best = d2; bj = t0 + t; }
                if (dd > maxd) {
                    maxd = dd;
                    const float nt = maxd - margin;
                    thr = (nt == nt) ? nt : -INFINITY;
                }
            }
        }
    }
    if (best_out) {
        if (valid && best < INFINITY) {
            const unsigned long long packed =
                ((unsigned long long)__float_as_uint(best) << 32) | (unsigned)bj;
            atomicMin(best_out + i, packed);
        }
    } else if (valid) {
        const bool found = best < INFINITY;
        idx_out[i] = found ? bj : -1;
        dist_out[i] = found ? sqrtf(best) : INFINITY;
    }
}

template <int M>
__global__ void __launch_bounds__(kAssocThreads)
assoc_scan(const float* __restrict__ x, int x_stride, const float* __restrict__ scale, const float* __restrict__ refs,
           int H, const int* __restrict__ d_n, int split_len, float delta, const float* __restrict__ d_delta,
           unsigned long long* __restrict__ best_out, int* __restrict__ idx_out, float* __restrict__ dist_out)
{
    assoc_scan_block<M>(blockIdx.x, blockIdx.y, x, x_stride, scale, refs, H, *d_n, split_len,
                        d_delta ? *d_delta : delta, best_out, idx_out, dist_out);
}

}  // namespace

int run_assoc_scan(const float* x, int x_stride, const float* scale, const float* refs, int M, const int* d_n, int n_cap,
                   int H, float delta, const float* d_delta, unsigned long long* best, int sms, int* idx, float* dist,
                   cudaStream_t stream)
{
    if (n_cap <= 0) return MOEA_OK;
    const int pb = ceil_div(n_cap, kAssocThreads);
    int splits = ceil_div(8LL * sms, pb);
    const int max_splits = ceil_div(H, kAssocTile);
    if (splits > max_splits) splits = max_splits;
    if (splits < 1) splits = 1;
    const int split_len = ceil_div(H, splits);
    // one range: the blocks write the result; several merge in best
    unsigned long long* merge = splits > 1 ? best : nullptr;
    if (merge) MOEA_TRY(run_assoc_reset(merge, n_cap, stream));
    switch (M) {
#define MOEA_ASSOC_CASE(K)                                                                                           \
    case K:                                                                                                          \
        assoc_scan<K><<<dim3(pb, splits), kAssocThreads, 0, stream>>>(x, x_stride, scale, refs, H, d_n, split_len,   \
                                                                      delta, d_delta, merge, idx, dist);             \
        break;
    MOEA_ASSOC_CASE(1) MOEA_ASSOC_CASE(2) MOEA_ASSOC_CASE(3) MOEA_ASSOC_CASE(4)
    MOEA_ASSOC_CASE(5) MOEA_ASSOC_CASE(6) MOEA_ASSOC_CASE(7) MOEA_ASSOC_CASE(8)
    MOEA_ASSOC_CASE(9) MOEA_ASSOC_CASE(10) MOEA_ASSOC_CASE(11) MOEA_ASSOC_CASE(12)
    MOEA_ASSOC_CASE(13) MOEA_ASSOC_CASE(14) MOEA_ASSOC_CASE(15) MOEA_ASSOC_CASE(16)
#undef MOEA_ASSOC_CASE
    default: return set_error(MOEA_ERR_UNSUPPORTED, "associate: M=%d", M);
    }
    MOEA_CUDA_TRY(cudaGetLastError());
    return merge ? run_assoc_finish(merge, d_n, n_cap, idx, dist, stream) : MOEA_OK;
}

}  // namespace moea

// Inverted generational distance in FP64 on the GPU.
//
// Reference: tests/evaluation/metrics/igd.py:23-47 (igd) and :8-20
// (nondominated_mask).  The approximation keeps its rows whose objectives are
// all finite and, optionally, of those the non-dominated ones; the IGD is the
// mean over the reference points of the Euclidean distance to the nearest
// kept row.  Distances are direct FP64 differences (the reference's
// torch.cdist may expand |a-b|^2 into a matrix product for large inputs), and
// the mean is a fixed-order FP64 block sum.
//
// Non-dominated filter: up to kIgdPairPoints rows every pair is compared
// directly (n^2 tests over the whole device); above, front 0 of the
// non-dominated sort, where rows with a non-finite objective get a violation
// of 1, so they never dominate a finite row and never enter front 0.  Either
// way the rows kept are exactly the reference's (identical rows do not
// dominate each other).
#include <cmath>

#include "internal.cuh"

namespace moea {

int run_ndsort(Workspace& ws, const SplitPop& pop, int M, int target, int* out_fronts, cudaStream_t stream);

namespace {

constexpr int kIgdThreads = 128;
constexpr int kIgdTile = 128;          // rows staged at a time
constexpr int kIgdPairPoints = 8192;   // direct filter up to here: 3-12 us where the sort's launches take
                                       // 45 us; at 8192 rows of 8 objectives both take about 30 us

// One word of results for the host: the mean and the number of finite rows.
struct IgdResult {
    double mean;
    long long finite;
};

// Finite rows, and the reference points' distances set to "none".
__global__ void igd_mark(const float* __restrict__ objs, int n, int M, float* __restrict__ cv, int* __restrict__ keep,
                         IgdResult* __restrict__ result, unsigned long long* __restrict__ d2, int r)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool ok = false;
    if (i < n) {
        ok = true;
        for (int m = 0; m < M; ++m) ok &= isfinite(objs[(size_t)m * n + i]);
        cv[i] = ok ? 0.0f : 1.0f;
        keep[i] = ok ? 1 : 0;
    }
    for (int k = i; k < r; k += gridDim.x * blockDim.x) d2[k] = 0x7FF0000000000000ull;  // +inf
    const unsigned b = __ballot_sync(0xFFFFFFFFu, ok);
    if ((threadIdx.x & 31) == 0 && b)
        atomicAdd(reinterpret_cast<unsigned long long*>(&result->finite), (unsigned long long)__popc(b));
}

// keep[i] after the sort: finite rows of front 0
__global__ void igd_keep(const float* __restrict__ cv, const int* __restrict__ fronts, int n, int* __restrict__ keep)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) keep[i] = (cv[i] == 0.0f) && fronts[i] == 0;
}

// Clears keep[q] of the rows q that a finite row of the tile blockIdx.y
// dominates.  A finite row that dominates stays one whether it is kept or not,
// so the test uses cv, not keep.
template <int M>
__global__ void __launch_bounds__(kIgdThreads)
igd_dominated(const float* __restrict__ objs, const float* __restrict__ cv, int n, int* __restrict__ keep)
{
    __shared__ float s_p[kIgdTile][M];
    __shared__ int s_n;
    const int t = threadIdx.x, q = blockIdx.x * kIgdThreads + t, p = blockIdx.y * kIgdTile + t;
    if (t == 0) s_n = 0;
    __syncthreads();
    if (p < n && cv[p] == 0.0f) {
        const int at = atomicAdd(&s_n, 1);
#pragma unroll
        for (int m = 0; m < M; ++m) s_p[at][m] = objs[(size_t)m * n + p];
    }
    __syncthreads();
    if (q >= n || cv[q] != 0.0f) return;
    float f[M];
#pragma unroll
    for (int m = 0; m < M; ++m) f[m] = objs[(size_t)m * n + q];
    bool dominated = false;
    for (int k = 0; k < s_n; ++k) {
        bool no_worse = true, better = false;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            no_worse &= s_p[k][m] <= f[m];
            better |= s_p[k][m] < f[m];
        }
        dominated |= no_worse && better;
    }
    if (dominated) keep[q] = 0;
}

// Squared distance of every reference point to its nearest kept row of the
// range blockIdx.y: kPer reference points per thread, the kept rows of a tile
// gathered in shared memory in FP64 and read as broadcasts; the ranges merge
// through an atomic minimum (the order of non-negative doubles is that of
// their bits).  FP64-issue bound: 20000 x 1024 x 3 took 174 us with one thread
// per reference point over all rows (79 CTAs on 148 SMs) and its coordinates
// in local memory.
template <int M>
struct IgdCfg {
    static constexpr int kPer = M <= 4 ? 4 : (M <= 8 ? 2 : 1);
};
template <int M>
__global__ void __launch_bounds__(kIgdThreads)
igd_min_dist(const double* __restrict__ ref, int r, const float* __restrict__ objs, const int* __restrict__ keep,
             int n, int rows_per, unsigned long long* __restrict__ out)
{
    constexpr int kPer = IgdCfg<M>::kPer;
    __shared__ double s_p[kIgdTile][M];
    __shared__ int s_n;
    const int t = threadIdx.x;
    const int k0 = blockIdx.x * kIgdThreads * kPer + t;
    double q[kPer][M], best[kPer];
#pragma unroll
    for (int c = 0; c < kPer; ++c) {
        const int k = k0 + c * kIgdThreads;
        best[c] = INFINITY;
#pragma unroll
        for (int m = 0; m < M; ++m) q[c][m] = (k < r) ? ref[(size_t)k * M + m] : 0.0;
    }
    const int lo = blockIdx.y * rows_per, hi = min(n, lo + rows_per);
    for (int t0 = lo; t0 < hi; t0 += kIgdTile) {
        __syncthreads();
        if (t == 0) s_n = 0;
        __syncthreads();
        const int i = t0 + t;
        if (i < hi && keep[i]) {
            const int at = atomicAdd(&s_n, 1);
#pragma unroll
            for (int m = 0; m < M; ++m) s_p[at][m] = (double)objs[(size_t)m * n + i];
        }
        __syncthreads();
        const int cnt = s_n;
        for (int u = 0; u < cnt; ++u) {
            double p[M];
#pragma unroll
            for (int m = 0; m < M; ++m) p[m] = s_p[u][m];
#pragma unroll
            for (int c = 0; c < kPer; ++c) {
                double d2 = 0.0;
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const double d = q[c][m] - p[m];
                    d2 = fma(d, d, d2);
                }
                best[c] = fmin(best[c], d2);
            }
        }
    }
#pragma unroll
    for (int c = 0; c < kPer; ++c) {
        const int k = k0 + c * kIgdThreads;
        if (k < r && best[c] < INFINITY)
            atomicMin(out + k, (unsigned long long)__double_as_longlong(best[c]));
    }
}

// Distances in place of the squares, and their mean in FP64: strided partial
// sums, then a fixed tree.
__global__ void __launch_bounds__(1024) igd_mean(double* __restrict__ v, int r, IgdResult* __restrict__ result)
{
    __shared__ double s[1024];
    double a = 0.0;
    for (int i = threadIdx.x; i < r; i += 8 * 1024) {
        double x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = i + k * 1024 < r ? v[i + k * 1024] : 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = sqrt(x[k]);
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (i + k * 1024 < r) {
                v[i + k * 1024] = x[k];
                a += x[k];
            }
    }
    s[threadIdx.x] = a;
    __syncthreads();
    for (int o = blockDim.x >> 1; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) result->mean = s[0] / (double)r;
}

template <int M>
void launch_igd(Workspace& ws, const float* objs, const float* cv, int n, const double* ref, int r, bool pairs,
                unsigned long long* d2, cudaStream_t stream)
{
    if (pairs)
        igd_dominated<M><<<dim3(ceil_div(n, kIgdThreads), ceil_div(n, kIgdTile)), kIgdThreads, 0, stream>>>(objs, cv, n,
                                                                                                     ws.flags);
    // enough row ranges for eight CTAs per SM, of a tile or more each
    const int gx = ceil_div(r, kIgdThreads * IgdCfg<M>::kPer);
    int ranges = ceil_div(8 * ws.sm_count, gx);
    ranges = ranges < ceil_div(n, kIgdTile) ? ranges : ceil_div(n, kIgdTile);
    const int per = ceil_div(ceil_div(n, ranges), kIgdTile) * kIgdTile;
    igd_min_dist<M><<<dim3(gx, ceil_div(n, per)), kIgdThreads, 0, stream>>>(ref, r, objs, ws.flags, n, per, d2);
}

}  // namespace

int run_igd(Workspace& ws, const float* objs, int n, int M, const double* ref, int r, int filter,
            double* d_min_dist, double* h_igd, cudaStream_t stream)
{
    if (n < 1 || n > ws.n_max || M < 1 || M > ws.m_max || M > 16 || r < 1 || !ref || !d_min_dist || !h_igd)
        return set_error(MOEA_ERR_INVALID_ARGUMENT, "igd: bad arguments (n=%d M=%d r=%d)", n, M, r);
    float* cv = ws.nds_objs;   // scratch: violations of the rows
    IgdResult* result = reinterpret_cast<IgdResult*>(ws.scalar_d);
    unsigned long long* d2 = reinterpret_cast<unsigned long long*>(d_min_dist);
    MOEA_CUDA_TRY(cudaMemsetAsync(result, 0, sizeof(IgdResult), stream));
    const int G = ceil_div(n, 256);
    igd_mark<<<G, 256, 0, stream>>>(objs, n, M, cv, ws.flags, result, d2, r);
    const bool pairs = filter && n <= kIgdPairPoints;
    if (filter && !pairs) {
        MOEA_TRY(run_ndsort(ws, merged_view(objs, cv, n), M, 1, ws.fronts, stream));
        igd_keep<<<G, 256, 0, stream>>>(cv, ws.fronts, n, ws.flags);
    }
    switch (M) {
#define MOEA_IGD_CASE(K) case K: launch_igd<K>(ws, objs, cv, n, ref, r, pairs, d2, stream); break;
    MOEA_IGD_CASE(1) MOEA_IGD_CASE(2) MOEA_IGD_CASE(3) MOEA_IGD_CASE(4)
    MOEA_IGD_CASE(5) MOEA_IGD_CASE(6) MOEA_IGD_CASE(7) MOEA_IGD_CASE(8)
    MOEA_IGD_CASE(9) MOEA_IGD_CASE(10) MOEA_IGD_CASE(11) MOEA_IGD_CASE(12)
    MOEA_IGD_CASE(13) MOEA_IGD_CASE(14) MOEA_IGD_CASE(15) MOEA_IGD_CASE(16)
#undef MOEA_IGD_CASE
    }
    igd_mean<<<1, 1024, 0, stream>>>(d_min_dist, r, result);
    MOEA_CUDA_TRY(cudaGetLastError());
    IgdResult host{};
    MOEA_CUDA_TRY(cudaMemcpyAsync(&host, result, sizeof(host), cudaMemcpyDeviceToHost, stream));
    MOEA_CUDA_TRY(cudaStreamSynchronize(stream));
    if (host.finite == 0) return set_error(MOEA_ERR_INVALID_ARGUMENT, "approximation contains no finite objective rows");
    *h_igd = host.mean;
    return MOEA_OK;
}

}  // namespace moea

using namespace moea;

extern "C" moea_status moea_igd(moea_workspace* w, const float* d_objs, int n, int M, const double* d_ref, int r,
                                int filter_nondominated, double* d_min_dist, double* h_igd, void* stream)
{
    if (!w || !d_objs) return set_error(MOEA_ERR_INVALID_ARGUMENT, "igd: NULL argument");
    return run_igd(w->ws, d_objs, n, M, d_ref, r, filter_nondominated, d_min_dist, h_igd,
                   static_cast<cudaStream_t>(stream));
}

// Built-in test problems (DTLZ family, constrained variants, CSDP) for sm_100a.
//
// Reference: python/csrc/native/src/problem/dtlz/dtlz_kernels.cu:28-1176.
// Objectives are written straight into the objective-major (M,N) layout (the
// reference writes (N,M) and transposes, :748-819).  The g-term reduction
// keeps the reference's summation order -- virtual thread t of a 256-thread
// row accumulates terms t, t+256, ..., each group of 32 folds with a
// shuffle-down tree, and the eight partials are added in order (DTLZ5 folds
// them with a second tree) -- and every formula keeps the reference's
// expression shape (double-precision pi products, the same fused
// multiply-adds), so the FP32 objectives are the reference's bit for bit on
// the GPU.  Rows with at most 256 g-terms use one warp per row; longer rows
// (large D) use one 256-thread block per row reading the row coalesced.
#include <math_constants.h>

#include "internal.cuh"
#include "dtlz.cuh"

namespace moea {
namespace {

template <int B>
__global__ void __launch_bounds__(256)
dtlz_warp_rows(const float* __restrict__ vars, int N, int D, int M, float* __restrict__ objs)
{
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= N) return;
    dtlz_group_row<B, 32>(row, true, threadIdx.x & 31, vars + (size_t)row * D, N, D, M, objs);
}

// One 256-thread block per row, the reference's strided accumulation.
template <int B>
__global__ void __launch_bounds__(256)
dtlz_block_rows(const float* __restrict__ vars, int N, int D, int M, float* __restrict__ objs)
{
    const int row = blockIdx.x;
    if (row >= N) return;
    const float* x = vars + (size_t)row * D;
    const int start = (B == kDTLZ7) ? D - (D - M + 1) : M - 1;
    const int k = D - start;
    float a = 0.0f;
    for (int i = threadIdx.x; i < k; i += 256) a = g_accumulate<B>(a, __ldg(x + start + i));
    a = warp_tree(a);
    __shared__ float ws[8];
    __shared__ float s_total;
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        float w8[8];
        for (int w = 0; w < 8; ++w) w8[w] = ws[w];
        s_total = fold_partials<B>(w8);
    }
    __syncthreads();
    if ((int)threadIdx.x < M) objs[(size_t)threadIdx.x * N + row] = row_objective<B>(threadIdx.x, s_total, x, D, M);
}

__global__ void cv_kernel(int kind, const float* __restrict__ objs, int N, int M, float R, float* __restrict__ cvout)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) cvout[i] = constraint_violation(kind, objs + i, N, M, R);
}

// CSDP car-side-impact problem (dtlz_kernels.cu:719-747, 1046-1092).
__global__ void csdp_kernel(const float* __restrict__ vars, int N, float* __restrict__ objs,
                            float* __restrict__ cvout)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const float* x = vars + (size_t)i * 7;
    const float x1 = x[0], x2 = x[1], x3 = x[2], x4 = x[3], x5 = x[4], x6 = x[5], x7 = x[6];
    {
        const float F = 4.72 - 0.5 * x4 - 0.19 * x2 * x3;
        const float V_MBP = 10.58 - 0.674 * x1 * x2 - 0.67275 * x2;
        const float V_FD = 16.45 - 0.489 * x3 * x7 - 0.843 * x5 * x6;
        objs[i] = 1.98 + 4.9 * x1 + 6.67 * x2 + 6.98 * x3 + 4.01 * x4 + 1.78 * x5 + 0.00001 * x6 + 2.73 * x7;
        objs[(size_t)N + i] = F;
        objs[(size_t)2 * N + i] = 0.5f * (V_MBP + V_FD);
    }
    const float F = 4.72f - 0.5f * x4 - 0.19f * x2 * x3;
    const float V_MBP = 10.58f - 0.674f * x1 * x2 - 0.67275f * x2;
    const float V_FD = 16.45f - 0.489f * x3 * x7 - 0.843f * x5 * x6;
    float g[10];
    g[0] = 1.16f - 0.3717f * x2 * x4 - 0.0092928f * x3 - 1.0f;
    g[1] = 0.261f - 0.0159f * x1 * x2 - 0.06486f * x1 - 0.019f * x2 * x7 + 0.0144f * x3 * x5 + 0.0154464f * x6 - 0.32f;
    g[2] = 0.214f + 0.00817f * x5 - 0.045195f * x1 - 0.0135168f * x1 + 0.03099f * x2 * x6 - 0.018f * x2 * x7
         + 0.007176f * x3 + 0.023232f * x3 - 0.00364f * x5 * x6 - 0.018f * x2 * x2 - 0.32f;
    g[3] = 0.74f - 0.61f * x2 - 0.031296f * x3 - 0.031872f * x7 + 0.227f * x2 * x2 - 0.32f;
    g[4] = 28.98f + 3.818f * x3 - 4.2f * x1 * x2 + 1.27296f * x6 - 2.68065f * x7 - 32.0f;
    g[5] = 33.86f + 2.95f * x3 - 5.057f * x1 * x2 - 3.795f * x2 - 3.4431f * x7 + 1.45728f - 32.0f;
    g[6] = 46.36f - 9.9f * x2 - 4.4505f * x1 - 32.0f;
    g[7] = F - 4.0f;
    g[8] = V_MBP - 9.9f;
    g[9] = V_FD - 15.7f;
    float s = 0.0f;
    for (int j = 0; j < 10; ++j) s += fmaxf(g[j], 0.0f);
    cvout[i] = s;
}

__global__ void zero_kernel(float* p, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = 0.0f;
}

template <int B>
void launch_rows(const float* x, int N, int D, int M, float* objs, cudaStream_t s)
{
    const int k = (B == kDTLZ7) ? D - M + 1 : D - (M - 1);
    if (k <= 256)
        dtlz_warp_rows<B><<<ceil_div(N, 8), 256, 0, s>>>(x, N, D, M, objs);
    else
        dtlz_block_rows<B><<<N, 256, 0, s>>>(x, N, D, M, objs);
}

}  // namespace

// Validates a built-in problem configuration (problem_factory / dtlz_problem.cu).
int validate_problem(int kind, int D, int M)
{
    if (kind < 1 || kind > 15) return set_error(MOEA_ERR_INVALID_ARGUMENT, "unknown problem kind %d", kind);
    if (M < 1 || M > kMaxObjectives)
        return set_error(MOEA_ERR_UNSUPPORTED, "problem: objectives=%d (1..%d)", M, kMaxObjectives);
    if (kind == 15) {
        if (D != 7 || M != 3) return set_error(MOEA_ERR_INVALID_ARGUMENT, "CSDP requires D=7, M=3");
        return MOEA_OK;
    }
    if (D < M) return set_error(MOEA_ERR_INVALID_ARGUMENT, "problem: dimension %d < objectives %d", D, M);
    if (kind == 10 && !(M == 2 || M == 3 || M == 5 || M == 8 || M == 10 || M == 15))
        return set_error(MOEA_ERR_INVALID_ARGUMENT, "C1-DTLZ3 supports M in {2,3,5,8,10,15}");
    if (kind == 11 && !(M == 2 || M == 3 || M == 5 || M == 8 || M == 10 || M == 15))
        return set_error(MOEA_ERR_INVALID_ARGUMENT, "C2-DTLZ2 supports M in {2,3,5,8,10,15}");
    if (kind == 12 && !(M == 3 || M == 5 || M == 8 || M == 10 || M == 15))
        return set_error(MOEA_ERR_INVALID_ARGUMENT, "C2-ConvexDTLZ2 supports M in {3,5,8,10,15}");
    return MOEA_OK;
}

int run_problem(int kind, const float* x, int N, int D, int M, float* objs, float* cv,
                cudaStream_t s)
{
    MOEA_TRY(validate_problem(kind, D, M));
    if (N <= 0) return MOEA_OK;
    if (kind == 15) {
        csdp_kernel<<<ceil_div(N, 256), 256, 0, s>>>(x, N, objs, cv);
        MOEA_CUDA_TRY(cudaGetLastError());
        return MOEA_OK;
    }
    switch (base_kind(kind)) {
    case kDTLZ1: launch_rows<kDTLZ1>(x, N, D, M, objs, s); break;
    case kDTLZ2: launch_rows<kDTLZ2>(x, N, D, M, objs, s); break;
    case kDTLZ3: launch_rows<kDTLZ3>(x, N, D, M, objs, s); break;
    case kDTLZ4: launch_rows<kDTLZ4>(x, N, D, M, objs, s); break;
    case kDTLZ5: launch_rows<kDTLZ5>(x, N, D, M, objs, s); break;
    case kDTLZ6: launch_rows<kDTLZ6>(x, N, D, M, objs, s); break;
    case kDTLZ7: launch_rows<kDTLZ7>(x, N, D, M, objs, s); break;
    case kConvexDTLZ2: launch_rows<kConvexDTLZ2>(x, N, D, M, objs, s); break;
    default: return set_error(MOEA_ERR_INVALID_ARGUMENT, "unknown problem kind %d", kind);
    }
    if (kind >= 9)
        cv_kernel<<<ceil_div(N, 256), 256, 0, s>>>(kind, objs, N, M, cv_radius(kind, M), cv);
    else
        zero_kernel<<<ceil_div(N, 256), 256, 0, s>>>(cv, N);
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

}  // namespace moea

extern "C" moea_status moea_problem_evaluate(int kind, const float* d_x, int N, int D, int M,
                                             float* d_objs, float* d_cv, void* stream)
{
    if (!d_x || !d_objs || !d_cv || N < 0)
        return moea::set_error(MOEA_ERR_INVALID_ARGUMENT, "problem_evaluate: bad arguments");
    return moea::run_problem(kind, d_x, N, D, M, d_objs, d_cv, (cudaStream_t)stream);
}

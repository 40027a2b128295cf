// The offspring of one generation in one launch: mating, SBX, polynomial
// mutation and evaluation of each pair of children by one group of lanes.
//
// Reference: reproduction/mating_selection.cu:11-108, sbx_crossover.cu:12-190,
// polynomial_mutation.cu:12-124 and problem/dtlz/dtlz_kernels.cu:28-1176, one
// kernel (or several) each.  Here a group of lanes takes a pair.  A pair of children depends on its two parents
// only, so the stages need no barrier between pairs: the pair's variables stay
// in shared memory from the crossover to the evaluation and are written once.
// The draws, the expressions and their order are those of the separate
// kernels (variation.cuh, dtlz.cuh), which remain for the rows that do not fit
// (more than 256 g-terms), for mating callbacks and for the operator calls.
//
// Bound by latency: up to a few thousand children one warp per scheduler runs
// the chain of a pair, and four to six launches of 2.5-7.5 us become one.
#include "dtlz.cuh"
#include "offspring.cuh"
#include "variation.cuh"

namespace moea {
namespace {

constexpr int kOffThreads = 256;

// Shared floats of one pair: two rows, on a 16-byte boundary.
__host__ __device__ inline int offspring_stride(int D) { return 2 * ((D + 3) & ~3); }

// Children 2p and 2p + 1 by a group of G lanes (8 or 32); rows: the pair's
// shared floats.  Every lane of the warp calls.  B: base kind of the problem,
// 0 to leave the evaluation to the caller.
template <int B, int G>
__device__ __forceinline__ void offspring_pair(int p, float* rows, const OffspringArgs& A, uint32_t gen, int active)
{
    const int gl = threadIdx.x & (G - 1);
    const int pairs = A.n_off / 2, ca = 2 * p, D = A.D, D4 = (D + 3) >> 2;
    const int children = p < pairs ? 2 : (ca < A.n_off ? 1 : 0);
    if (gl < children) mating_child(ca + gl, A.cv, A.rank, active, A.seed, gen, A.pidx);
    __syncwarp();
    float* base = rows - (size_t)ca * D;  // row r of the population at base + r * D
    const float eta_c = annealed_eta(A.sbx_eta0, A.sbx_eta1, (int)gen, A.total);
    if (children)
        for (int j = gl; j < D4; j += G)
            crossover_group<true>(p * D4 + j, p, j, A.parents, A.pidx, A.bounds, base, pairs, D, A.vec != 0, eta_c, A.sbx_prob,
                            A.copy_prob, A.seed, gen);
    __syncwarp();
    if (A.mutate) {
        const bool mine = (gl >> 2) < children;  // four lanes per child
        mutate_child4<true>(mine ? ca + (gl >> 2) : ca, mine, gl & 3, base, A.bounds, A.n_off, D,
                      annealed_eta(A.pm_eta0, A.pm_eta1, (int)gen, A.total), A.pm_prob, A.seed, gen);
        __syncwarp();
    }
    for (int i = gl; i < children * D; i += G) A.off[(size_t)ca * D + i] = rows[i];
    if constexpr (B != 0) {
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
            const int r = ca + h;
            dtlz_group_row<B, G, true>(r, h < children, gl, rows + (size_t)h * D, A.n_off, D, A.M, A.objs);
            if (A.kind >= 9) __syncwarp();  // the row's objectives, written by the group's other lanes
            if (gl == 0 && h < children)
                A.cv_out[r] = A.kind >= 9 && (!A.cv_table || A.cv_table[gen])
                                  ? constraint_violation(A.kind, A.objs + r, A.n_off, A.M, A.radius)
                                  : 0.0f;
        }
    }
}

template <int B, int G>
__global__ void __launch_bounds__(kOffThreads) offspring_kernel(OffspringArgs A)
{
    extern __shared__ __align__(16) float off_rows[];
    const int g = threadIdx.x / G;
    offspring_pair<B, G>(blockIdx.x * (kOffThreads / G) + g, off_rows + g * offspring_stride(A.D), A,
                         A.d_gen ? (uint32_t)*A.d_gen : A.gen, A.d_active ? *A.d_active : A.active);
}

// Every instance of a batch (blockIdx.y): problem kinds 1..8, whose violation
// is zero.  Batches fill the device, so a pair takes eight lanes.
constexpr int kFusedGroup = 8;
__global__ void __launch_bounds__(kOffThreads, 3)
fused_offspring(const BatchInst* __restrict__ insts, const int* __restrict__ ids)
{
    extern __shared__ __align__(16) float off_rows[];
    const BatchInst& I = insts[ids[blockIdx.y]];
    const int g = threadIdx.x / kFusedGroup;
    const int p0 = blockIdx.x * (kOffThreads / kFusedGroup), p = p0 + g;
    if (2 * p0 >= I.N) return;
    const bool vec = (I.D & 3) == 0 && ((uintptr_t)I.varsP & 15) == 0 && ((uintptr_t)I.bounds & 15) == 0;
    const OffspringArgs A{I.varsP, I.cvP, I.tournament ? I.rankP : nullptr, nullptr, I.N, I.bounds, I.varsO, I.pidx,
                          I.objsO, I.cvO, nullptr, I.N, I.D, I.M, I.kind, I.mutate, vec, I.T, I.sbx_eta0, I.sbx_eta1,
                          I.sbx_prob, I.sbx_copy, I.pm_eta0, I.pm_eta1, I.pm_prob, 0.0f, I.seed, nullptr, 0u};
    float* rows = off_rows + g * offspring_stride(I.D);
    const uint32_t gen = (uint32_t)*I.d_gen;
    switch (I.kind) {
#define MOEA_OFF_CASE(K) case K: offspring_pair<K, kFusedGroup>(p, rows, A, gen, I.N); break;
    MOEA_OFF_CASE(1) MOEA_OFF_CASE(2) MOEA_OFF_CASE(3) MOEA_OFF_CASE(4)
    MOEA_OFF_CASE(5) MOEA_OFF_CASE(6) MOEA_OFF_CASE(7) MOEA_OFF_CASE(8)
#undef MOEA_OFF_CASE
    default: break;
    }
}

template <int B>
void launch_offspring(const OffspringArgs& A, cudaStream_t stream)
{
    const int pairs = (A.n_off + 1) / 2;
    // Eight lanes per pair, unless the rows are longer than eight lanes' first
    // groups of four and too few to fill the schedulers with eight lanes each.
    if (A.D <= kOffspringGroupD && (A.D <= 32 || pairs >= 8192))
        offspring_kernel<B, 8><<<ceil_div(pairs, kOffThreads / 8), kOffThreads,
                                 sizeof(float) * (kOffThreads / 8) * offspring_stride(A.D), stream>>>(A);
    else
        offspring_kernel<B, 32><<<ceil_div(pairs, kOffThreads / 32), kOffThreads,
                                  sizeof(float) * (kOffThreads / 32) * offspring_stride(A.D), stream>>>(A);
}

}  // namespace

// Rows that two warps' worth of shared memory and one warp's g-terms hold.
bool offspring_eligible(int kind, int D, int M)
{
    if (kind == 0) return D <= kOffspringMaxD;
    if (kind < 1 || kind > 14) return false;
    const int k = base_kind(kind) == kDTLZ7 ? D - M + 1 : D - (M - 1);
    return k >= 1 && k <= 256 && D <= kOffspringMaxD;
}

int run_offspring(OffspringArgs A, cudaStream_t stream)
{
    if (A.n_off < 1) return MOEA_OK;
    A.vec = (A.D & 3) == 0 && ((uintptr_t)A.parents & 15) == 0 && ((uintptr_t)A.bounds & 15) == 0;
    A.radius = cv_radius(A.kind, A.M);
    switch (A.kind == 0 ? 0 : base_kind(A.kind)) {
#define MOEA_OFF_CASE(K) case K: launch_offspring<K>(A, stream); break;
    MOEA_OFF_CASE(0) MOEA_OFF_CASE(1) MOEA_OFF_CASE(2) MOEA_OFF_CASE(3) MOEA_OFF_CASE(4)
    MOEA_OFF_CASE(5) MOEA_OFF_CASE(6) MOEA_OFF_CASE(7) MOEA_OFF_CASE(8)
#undef MOEA_OFF_CASE
    default: return set_error(MOEA_ERR_INVALID_ARGUMENT, "offspring: problem kind %d", A.kind);
    }
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

// The shared-memory limit of fused_offspring for the longest rows that a fused
// batch holds (256 g-terms behind kMaxObjectives - 1 position variables).  The
// limit belongs to the function: set by each launch for its own rows, a smaller
// launch on another thread could lower it under a larger one.
int fused_offspring_configure()
{
    constexpr int kPairs = kOffThreads / kFusedGroup;
    MOEA_CUDA_TRY(cudaFuncSetAttribute(fused_offspring, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(float) * kPairs * offspring_stride(256 + kMaxObjectives - 1)));
    return MOEA_OK;
}

int fused_reproduce(const BatchInst* d_inst, const FusedGroup& g, cudaStream_t s)
{
    constexpr int kPairs = kOffThreads / kFusedGroup;
    const size_t smem = sizeof(float) * kPairs * offspring_stride(g.max_D);
    fused_offspring<<<dim3(ceil_div((g.max_N + 1) / 2, kPairs), g.count), kOffThreads, smem, s>>>(d_inst, g.d_ids);
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

}  // namespace moea

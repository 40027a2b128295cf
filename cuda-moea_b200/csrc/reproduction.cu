// Mating selection, SBX and polynomial mutation for sm_100a.
//
// Reference operators (paths relative to python/csrc/native/src/reproduction/):
//   tournament / random mating   mating_selection.cu:11-108
//   SBX                          sbx_crossover.cu:12-190
//   polynomial mutation          polynomial_mutation.cu:12-124
// The reference fills global buffers with cuRAND draws (three launches for SBX,
// one for PM, one for mating) whose element-to-thread mapping depends on the
// GPU model.  Here every draw is a Philox4x32-10 block computed in registers
// from (seed, element, generation, tag): no random buffers, the same numbers on
// every GPU, and the streams can be regenerated on the host for checking.  The
// `*_explicit` kernels take the draws as arrays instead, which is how the
// stage parity tests feed identical numbers to the oracle.
#include <algorithm>

#include "internal.cuh"
#include "variation.cuh"

namespace moea {
namespace {

__global__ void tournament_explicit(const int2* __restrict__ cand, const int* __restrict__ rank,
                                    const float* __restrict__ cv, int n, int* __restrict__ winners)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int2 c = cand[i];
    winners[i] = tournament_pick(c.x, c.y, cv, rank);
}

__global__ void sbx_explicit(const float* __restrict__ parents, const int* __restrict__ pidx,
                             const float* __restrict__ bounds, const float2* __restrict__ u,
                             const int* __restrict__ sign, const float* __restrict__ copy,
                             float* __restrict__ off, float eta, float prob, float copy_prob,
                             int pairs, int D)
{
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)pairs * D) return;
    const int p = (int)(e / D), d = (int)(e % D);
    const int ca = 2 * p, cb = ca + 1;
    const float x1 = parents[(size_t)pidx[ca] * D + d];
    const float x2 = parents[(size_t)pidx[cb] * D + d];
    const float2 r = u[e];
    float c1, c2;
    sbx_pair(x1, x2, r.x, r.y, sign[e], copy[e], eta, prob, copy_prob, bounds[2 * d],
             bounds[2 * d + 1], c1, c2);
    off[(size_t)ca * D + d] = c1;
    off[(size_t)cb * D + d] = c2;
}

__global__ void copy_last_child(const float* __restrict__ parents, const int* __restrict__ pidx,
                                float* __restrict__ off, int child, int D)
{
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d < D) off[(size_t)child * D + d] = parents[(size_t)pidx[child] * D + d];
}

__global__ void pm_explicit(float* __restrict__ off, const float* __restrict__ bounds,
                            const float2* __restrict__ u, float eta, float prob, long long count,
                            int D)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const int d = (int)(i % D);
    const float2 r = u[i];
    off[i] = pm_value(off[i], r.x, r.y, eta, prob, D, bounds[2 * d], bounds[2 * d + 1]);
}

__global__ void mating_philox(const float* __restrict__ cv, const int* __restrict__ rank,
                              const int* __restrict__ d_active, int active_host, int n_off,
                              uint64_t seed, const int* __restrict__ d_gen, uint32_t gen_host,
                              int* __restrict__ pidx)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_off) return;
    const int active = d_active ? *d_active : active_host;
    const uint32_t gen = d_gen ? (uint32_t)*d_gen : gen_host;
    mating_child(i, cv, rank, active, seed, gen, pidx);
}

__global__ void crossover_philox(const float* __restrict__ parents, const int* __restrict__ pidx,
                                 const float* __restrict__ bounds, float* __restrict__ off, int n_off, int D,
                                 bool vec, float sbx_eta0, float sbx_eta1, float sbx_prob, float copy_prob,
                                 int total, uint64_t seed, const int* __restrict__ d_gen, uint32_t gen_host)
{
    const int pairs = n_off / 2;
    const int D4 = (D + 3) >> 2;
    const long long count = (long long)(pairs + (n_off & 1)) * D4;
    const uint32_t gen = d_gen ? (uint32_t)*d_gen : gen_host;
    const float eta_c = annealed_eta(sbx_eta0, sbx_eta1, (int)gen, total);
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < count;
         t += (long long)gridDim.x * blockDim.x) {
        const int p = (int)(t / D4);
        crossover_group((int)t, p, (int)(t - (long long)p * D4), parents, pidx, bounds, off, pairs, D, vec, eta_c,
                        sbx_prob, copy_prob, seed, gen);
    }
}

// Crossover of long rows (D a multiple of 4, 16-byte aligned): blockIdx.y walks
// the pairs and blockIdx.x the groups of four variables, so a thread divides
// nothing and its block reads the parent indices once; kPlain: every variable
// is crossed (no test or copy draw can change it).  Bound by instruction issue
// (the powf): at D = 131072, 512 pairs, the flat kernel above spent a fifth of
// its instructions on the 64-bit division of its group index and the tests
// (378 -> 317 us a launch).
template <bool kPlain>
__global__ void __launch_bounds__(256)
crossover_rows(const float* __restrict__ parents, const int* __restrict__ pidx, const float* __restrict__ bounds,
               float* __restrict__ off, int pairs, int D, float sbx_eta0, float sbx_eta1, float sbx_prob,
               float copy_prob, int total, uint64_t seed, const int* __restrict__ d_gen, uint32_t gen_host)
{
    const int D4 = D >> 2;
    const uint32_t gen = d_gen ? (uint32_t)*d_gen : gen_host;
    const float eta = annealed_eta(sbx_eta0, sbx_eta1, (int)gen, total);
    for (int p = blockIdx.y; p < pairs; p += gridDim.y) {
        const float4* xa = reinterpret_cast<const float4*>(parents + (size_t)pidx[2 * p] * D);
        const float4* xb = reinterpret_cast<const float4*>(parents + (size_t)pidx[2 * p + 1] * D);
        float4* oa = reinterpret_cast<float4*>(off + (size_t)(2 * p) * D);
        float4* ob = oa + D4;
        for (int j = blockIdx.x * 256 + threadIdx.x; j < D4; j += gridDim.x * 256) {
            const float4 a4 = __ldg(xa + j), b4 = __ldg(xb + j);
            const float4 l01 = __ldg(reinterpret_cast<const float4*>(bounds) + 2 * j);
            const float4 l23 = __ldg(reinterpret_cast<const float4*>(bounds) + 2 * j + 1);
            const uint64_t block = (uint64_t)((uint32_t)p * (uint32_t)D4 + (uint32_t)j);
            uint32_t r[4], rt[4] = {0u, 0u, 0u, 0u}, rc[4] = {0u, 0u, 0u, 0u};
            rng_block(seed, block, gen, kTagCrossover, r);
            if (!kPlain) {
                if (sbx_prob < 1.0f) rng_block(seed, block, gen, kTagCrossTest, rt);
                if (copy_prob > 0.0f) rng_block(seed, block, gen, kTagCopy, rc);
            }
            const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
            const float lo[4] = {l01.x, l01.z, l23.x, l23.z}, hi[4] = {l01.y, l01.w, l23.y, l23.w};
            float c1[4], c2[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                sbx_pair(a[i], b[i], u32_to_unit(r[i]), kPlain ? 0.0f : u32_to_unit(rt[i]), (int)(r[i] & 1u),
                         kPlain ? 0.0f : u32_to_unit(rc[i]), eta, kPlain ? 1.0f : sbx_prob, kPlain ? 0.0f : copy_prob,
                         lo[i], hi[i], c1[i], c2[i]);
            oa[j] = make_float4(c1[0], c1[1], c1[2], c1[3]);
            ob[j] = make_float4(c2[0], c2[1], c2[2], c2[3]);
        }
    }
}

__global__ void mutation_philox(float* __restrict__ off, const float* __restrict__ bounds, int n_off, int D,
                                float pm_eta0, float pm_eta1, float pm_prob, int total, uint64_t seed,
                                const int* __restrict__ d_gen, uint32_t gen_host)
{
    const int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 2);
    const uint32_t gen = d_gen ? (uint32_t)*d_gen : gen_host;
    const float eta_m = annealed_eta(pm_eta0, pm_eta1, (int)gen, total);
    mutate_child4(c < n_off ? c : 0, c < n_off, (int)(threadIdx.x & 3u), off, bounds, n_off, D, eta_m, pm_prob,
                  seed, gen);
}

__global__ void rng_blocks_kernel(uint64_t seed, uint32_t gen, uint32_t tag, long long count,
                                  uint4* out)
{
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= count) return;
    uint32_t r[4];
    rng_block(seed, (uint64_t)e, gen, tag, r);
    out[e] = make_uint4(r[0], r[1], r[2], r[3]);
}

// x = lb + u (ub - lb) (population.cu:12-24, 97-115) with Philox draws: a
// thread takes the four elements of one block of draws (one element per thread,
// each with the whole block and a 64-bit remainder, took 773 us for 134 M
// elements; 164 us now).
__global__ void init_uniform(float* __restrict__ vars, const float* __restrict__ bounds, long long count, int D,
                             uint64_t seed)
{
    const long long blocks = (count + 3) >> 2;
    const long long step = (long long)gridDim.x * blockDim.x;
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int d = (int)((4 * e) % D);
    const int advance = (int)((4 * step) % D);
    const bool vec = (D & 3) == 0 && ((uintptr_t)vars & 15) == 0 && ((uintptr_t)bounds & 15) == 0;
    for (; e < blocks; e += step) {
        uint32_t r[4];
        rng_block(seed, (uint64_t)e, 0u, kTagInit, r);
        if (vec) {  // D a multiple of 4: the four elements are one aligned group of a row
            const float4 l01 = __ldg(reinterpret_cast<const float4*>(bounds + 2 * d));
            const float4 l23 = __ldg(reinterpret_cast<const float4*>(bounds + 2 * d) + 1);
            reinterpret_cast<float4*>(vars)[e] =
                make_float4(l01.x + u32_to_unit(r[0]) * (l01.y - l01.x), l01.z + u32_to_unit(r[1]) * (l01.w - l01.z),
                            l23.x + u32_to_unit(r[2]) * (l23.y - l23.x), l23.z + u32_to_unit(r[3]) * (l23.w - l23.z));
            d += advance;
            if (d >= D) d -= D;
            continue;
        }
        int dk = d;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (4 * e + k < count) {
                const float lower = bounds[2 * dk], upper = bounds[2 * dk + 1];
                vars[4 * e + k] = lower + u32_to_unit(r[k]) * (upper - lower);
            }
            dk = dk + 1 < D ? dk + 1 : 0;
        }
        d += advance;
        if (d >= D) d -= D;
    }
}

constexpr int kRowCrossoverD = 1024;  // rows from which a block of 256 groups is one row's

inline int grid_for(long long count, int threads, int cap = 148 * 32)
{
    long long g = (count + threads - 1) / threads;
    if (g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

}  // namespace

int run_mating(const float* cv, const int* rank, const int* d_active, int active, int n_off,
               uint64_t seed, const int* d_gen, uint32_t gen, int* pidx, cudaStream_t stream)
{
    mating_philox<<<ceil_div(n_off, 256), 256, 0, stream>>>(cv, rank, d_active, active, n_off, seed,
                                                            d_gen, gen, pidx);
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

int run_variation_pass(int passes, const float* parents, const int* pidx, const float* bounds, float* off,
                       int n_off, int D, float sbx_eta0, float sbx_eta1, float sbx_prob, float copy_prob,
                       int mutate, float pm_eta0, float pm_eta1, float pm_prob, int total,
                       uint64_t seed, const int* d_gen, uint32_t gen, cudaStream_t stream)
{
    if (passes & kPassCrossover) {
        const long long count = (long long)(n_off / 2 + (n_off & 1)) * ((D + 3) / 4);
        // 16-byte loads and stores when every row and the bounds are aligned
        const bool vec = (D & 3) == 0 && ((uintptr_t)parents & 15) == 0 && ((uintptr_t)off & 15) == 0 &&
                         ((uintptr_t)bounds & 15) == 0;
        if (vec && D >= kRowCrossoverD && (n_off & 1) == 0 && count < (1ll << 31)) {
            // 32 blocks per SM in flight, rows split into blocks of 256 groups: up
            // to 64 a row, or as many as fill the device with few pairs (one pair
            // of 2^20 variables with its mating and mutation 29 us with 64, 21 now)
            const int gx = std::min(ceil_div(D / 4, 256), std::max(64, 148 * 32 / (n_off / 2 > 0 ? n_off / 2 : 1)));
            const dim3 grid(gx, std::max(1, std::min(n_off / 2, 148 * 32 / gx)));
            if (sbx_prob >= 1.0f && copy_prob <= 0.0f)
                crossover_rows<true><<<grid, 256, 0, stream>>>(parents, pidx, bounds, off, n_off / 2, D, sbx_eta0, sbx_eta1,
                                                               sbx_prob, copy_prob, total, seed, d_gen, gen);
            else
                crossover_rows<false><<<grid, 256, 0, stream>>>(parents, pidx, bounds, off, n_off / 2, D, sbx_eta0,
                                                                sbx_eta1, sbx_prob, copy_prob, total, seed, d_gen, gen);
        } else {
            crossover_philox<<<grid_for(count, 256), 256, 0, stream>>>(parents, pidx, bounds, off, n_off, D, vec,
                                                                       sbx_eta0, sbx_eta1, sbx_prob, copy_prob, total,
                                                                       seed, d_gen, gen);
        }
        MOEA_CUDA_TRY(cudaGetLastError());
    }
    if ((passes & kPassMutation) && mutate && n_off > 0) {
        mutation_philox<<<ceil_div(4 * n_off, 128), 128, 0, stream>>>(off, bounds, n_off, D, pm_eta0, pm_eta1,
                                                                      pm_prob, total, seed, d_gen, gen);
        MOEA_CUDA_TRY(cudaGetLastError());
    }
    return MOEA_OK;
}

int run_variation(const float* parents, const int* pidx, const float* bounds, float* off,
                  int n_off, int D, float sbx_eta0, float sbx_eta1, float sbx_prob, float copy_prob,
                  int mutate, float pm_eta0, float pm_eta1, float pm_prob, int total,
                  uint64_t seed, const int* d_gen, uint32_t gen, cudaStream_t stream)
{
    return run_variation_pass(kPassBoth, parents, pidx, bounds, off, n_off, D, sbx_eta0, sbx_eta1, sbx_prob,
                              copy_prob, mutate, pm_eta0, pm_eta1, pm_prob, total, seed, d_gen, gen, stream);
}

int run_init_uniform(float* vars, const float* bounds, int N, int D, uint64_t seed,
                     cudaStream_t stream)
{
    const long long count = (long long)N * D;
    init_uniform<<<grid_for((count + 3) / 4, 256), 256, 0, stream>>>(vars, bounds, count, D, seed);
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

}  // namespace moea

using namespace moea;

extern "C" {

moea_status moea_tournament(const int* d_cand, const int* d_rank, const float* d_cv, int n,
                            int* d_winners, void* stream)
{
    if (!d_cand || !d_rank || !d_cv || !d_winners || n < 0)
        return set_error(MOEA_ERR_INVALID_ARGUMENT, "tournament: bad arguments");
    if (n == 0) return MOEA_OK;
    tournament_explicit<<<ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const int2*>(d_cand), d_rank, d_cv, n, d_winners);
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

moea_status moea_sbx(const float* d_parents, const int* d_pidx, const float* d_bounds,
                     const float* d_u, const int* d_sign, const float* d_copy, float* d_off,
                     float eta, float prob, float copy_prob, int n_off, int D, void* stream)
{
    if (!d_parents || !d_pidx || !d_bounds || !d_u || !d_sign || !d_copy || !d_off || n_off < 0 ||
        D < 1 || !(eta > 0.0f) || prob < 0.0f || prob > 1.0f || copy_prob < 0.0f || copy_prob > 1.0f)
        return set_error(MOEA_ERR_INVALID_ARGUMENT, "sbx: bad arguments");
    const cudaStream_t s = (cudaStream_t)stream;
    const int pairs = n_off / 2;
    const long long count = (long long)pairs * D;
    if (count > 0)
        sbx_explicit<<<(int)((count + 255) / 256), 256, 0, s>>>(
            d_parents, d_pidx, d_bounds, reinterpret_cast<const float2*>(d_u), d_sign, d_copy,
            d_off, eta, prob, copy_prob, pairs, D);
    if (n_off & 1)
        copy_last_child<<<ceil_div(D, 256), 256, 0, s>>>(d_parents, d_pidx, d_off, n_off - 1, D);
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

moea_status moea_pm(float* d_off, const float* d_bounds, const float* d_u, float eta, float prob,
                    int n, int D, void* stream)
{
    if (!d_off || !d_bounds || !d_u || n < 0 || D < 1 || !(eta > 0.0f) || prob < 0.0f || prob > 1.0f)
        return set_error(MOEA_ERR_INVALID_ARGUMENT, "pm: bad arguments");
    const long long count = (long long)n * D;
    if (count > 0)
        pm_explicit<<<(int)((count + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
            d_off, d_bounds, reinterpret_cast<const float2*>(d_u), eta, prob, count, D);
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

moea_status moea_reproduce(const float* d_parents, const float* d_parent_cv, const int* d_rank,
                           int active, const float* d_bounds, float* d_off, int* d_parent_idx,
                           int n_parents, int n_off, int D, int mating, float sbx_eta,
                           float sbx_prob, float sbx_copy_prob, int mutate, float pm_eta,
                           float pm_prob, uint64_t seed, uint32_t generation, void* stream)
{
    if (!d_parents || !d_bounds || !d_off || !d_parent_idx || n_off < 1 || D < 1 ||
        active < 1 || active > n_parents || (mating == MOEA_MATING_TOURNAMENT && (!d_rank || !d_parent_cv)))
        return set_error(MOEA_ERR_INVALID_ARGUMENT, "reproduce: bad arguments");
    const cudaStream_t s = (cudaStream_t)stream;
    MOEA_TRY(run_mating(d_parent_cv, mating == MOEA_MATING_TOURNAMENT ? d_rank : nullptr, nullptr,
                        active, n_off, seed, nullptr, generation, d_parent_idx, s));
    return run_variation(d_parents, d_parent_idx, d_bounds, d_off, n_off, D, sbx_eta, sbx_eta,
                         sbx_prob, sbx_copy_prob, mutate, pm_eta, pm_eta, pm_prob, 0, seed, nullptr,
                         generation, s);
}

moea_status moea_initialize_population(uint64_t seed, uint32_t epoch, const float* d_bounds, int N, int D,
                                      float* d_vars, void* stream)
{
    if (!d_bounds || !d_vars || N < 1 || D < 1)
        return set_error(MOEA_ERR_INVALID_ARGUMENT, "initialize_population: bad arguments");
    return run_init_uniform(d_vars, d_bounds, N, D, derive_seed(seed) ^ ((uint64_t)epoch << 48),
                            (cudaStream_t)stream);
}

moea_status moea_rng_blocks(uint64_t seed, uint32_t generation, uint32_t tag, int64_t count,
                            uint32_t* d_out, void* stream)
{
    if (!d_out || count < 0) return set_error(MOEA_ERR_INVALID_ARGUMENT, "rng_blocks: bad arguments");
    if (count == 0) return MOEA_OK;
    rng_blocks_kernel<<<(int)((count + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        seed, generation, tag, count, reinterpret_cast<uint4*>(d_out));
    MOEA_CUDA_TRY(cudaGetLastError());
    return MOEA_OK;
}

}  // extern "C"

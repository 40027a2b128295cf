// Mating, SBX and polynomial mutation of one child or pair (device code of
// reproduction.cu and offspring.cu).
#pragma once

#include "internal.cuh"

namespace moea {
namespace {

// Winner of a binary tournament (mating_selection.cu:11-35): feasible first,
// then smaller violation (ties to a), then rank (ties to a).
__device__ __forceinline__ int tournament_pick(int a, int b, const float* __restrict__ cv,
                                               const int* __restrict__ rank)
{
    const float ca = cv[a], cb = cv[b];
    if (ca == 0.0f && cb != 0.0f) return a;
    if (ca != 0.0f && cb == 0.0f) return b;
    if (ca != 0.0f && cb != 0.0f) return ca <= cb ? a : b;
    return rank[a] <= rank[b] ? a : b;
}

// Annealed distribution index; the product and sum are kept separate so the
// value is the one the reference computes on the host (sbx_crossover.cu:12-18).
__device__ __forceinline__ float annealed_eta(float begin, float end, int gen, int total)
{
    float p = 1.0f;
    if (total > 0) {
        p = __fdiv_rn((float)gen, (float)total);
        p = fminf(fmaxf(p, 0.0f), 1.0f);
    }
    return __fadd_rn(begin, __fmul_rn(__fsub_rn(end, begin), p));
}

// powf as a call (the same function, one copy of its code in a kernel).  The
// kernels that do everything for a pair of children hold up to a dozen powf,
// sinf and cosf; inlined, their code outgrew the instruction cache (a batch of
// mixed problems: 4.8 of 11 stall cycles per instruction were fetches).
__device__ __noinline__ float powf_call(float a, float b) { return powf(a, b); }
template <bool kCall>
__device__ __forceinline__ float power(float a, float b)
{
    if constexpr (kCall) return powf_call(a, b);
    else return powf(a, b);
}

// SBX on one variable pair (sbx_crossover.cu:44-70).  Returns false when the
// pair is copied unchanged.
template <bool kCall = false>
__device__ __forceinline__ void sbx_pair(float x1, float x2, float u1, float u2, int sign,
                                         float copy, float eta, float prob, float copy_prob,
                                         float lo, float hi, float& c1, float& c2)
{
    if (u2 >= prob || copy < copy_prob) {
        c1 = x1;
        c2 = x2;
        return;
    }
    const float exponent = 1.0f / (1.0f + eta);
    // one powf on the selected base (the same value as calling it in either
    // branch, without a warp running both when its lanes disagree)
    const float base = u1 < 0.5f ? 2.0f * u1 : 1.0f / (2.0f - 2.0f * u1);
    float beta = power<kCall>(base, exponent);
    beta *= 2 * sign - 1;
    const float midpoint = 0.5f * (x1 + x2);
    const float delta = 0.5f * beta * (x1 - x2);
    c1 = fminf(fmaxf(midpoint + delta, lo), hi);
    c2 = fminf(fmaxf(midpoint - delta, lo), hi);
}

// Deb's bounded polynomial mutation of one value (polynomial_mutation.cu:30-59).
// The outer powf stay inline: their last product is contracted with the
// subtraction, so as a call they would round differently.
template <bool kCall = false>
__device__ __forceinline__ float pm_value(float value, float u1, float u2, float eta, float prob,
                                          int D, float lo, float hi)
{
    if (u1 >= prob / static_cast<float>(D)) return value;
    const float range = hi - lo;
    const float normalized = (value - lo) / range;
    const float exponent = eta + 1.0f;
    float delta;
    if (u2 <= 0.5f) {
        const float xy = 1.0f - normalized;
        const float value_mut = 2.0f * u2 + (1.0f - 2.0f * u2) * power<kCall>(xy, exponent);
        delta = powf(value_mut, 1.0f / exponent) - 1.0f;
    } else {
        const float xy = normalized;
        const float value_mut = 2.0f * (1.0f - u2) + 2.0f * (u2 - 0.5f) * power<kCall>(xy, exponent);
        delta = 1.0f - powf(value_mut, 1.0f / exponent);
    }
    return fminf(fmaxf(value + delta * range, lo), hi);
}

// Mating with Philox draws: child i draws block (i, generation, kTagMating).
__device__ __forceinline__ void mating_child(int i, const float* __restrict__ cv,
                                             const int* __restrict__ rank, int active, uint64_t seed,
                                             uint32_t gen, int* __restrict__ pidx)
{
    uint32_t r[4];
    rng_block(seed, (uint64_t)i, gen, kTagMating, r);
    const int a = (int)(r[0] % (uint32_t)active);
    if (rank == nullptr) {
        pidx[i] = a;
        return;
    }
    const int b = (int)(r[1] % (uint32_t)active);
    pidx[i] = tournament_pick(a, b, cv, rank);
}

// ---- variation with Philox draws ------------------------------------------
//
// Draw layout (this project's own stream; the same in the fused pass, the
// crossover-only pass followed by the mutation-only pass, and the batched
// form):
//
//  crossover of pair p, variables 4j .. 4j+3: block b = p * ceil(D/4) + j of
//    tag kTagCrossover; word i gives variable 4j+i its spread draw
//    u1 = unit(w) and its sign (w & 1).  Only when sbx_prob < 1 the block b
//    of tag kTagCrossTest gives the crossover test u2 (word i), and only when
//    copy_prob > 0 the block b of tag kTagCopy gives the copy draw.  Skipping
//    those draws changes nothing: u2 < 1 <= sbx_prob always passes and
//    copy < copy_prob <= 0 never holds.
//  mutation of child c: its mutated variables are drawn as geometric gaps,
//    which gives every variable an independent chance limit = pm_prob / D (in
//    FP32, the reference's test, polynomial_mutation.cu:34).  Draw k of child
//    c is block k * n_off + c of tag kTagMutation: gap = floor(ln u / ln(1 -
//    limit)) in FP64 with u = ((w0 >> 8) + 1) 2^-24, the site is the last
//    site + 1 + gap, and unit(w1) is the site's amplitude draw.
//
// One block per four variables (instead of one per variable) and no per
// variable mutation test: at large D the variation is then bound by its
// powf and its HBM stream, not by Philox rounds.

template <bool kCall = false>
__device__ __forceinline__ void crossover_group(int t, int p, int j, const float* __restrict__ parents,
                                                const int* __restrict__ pidx, const float* __restrict__ bounds,
                                                float* __restrict__ off, int pairs, int D, bool vec, float eta_c,
                                                float sbx_prob, float copy_prob, uint64_t seed, uint32_t gen)
{
    const int ca = 2 * p, cb = ca + 1;
    const int d0 = 4 * j;
    const int cnt = min(4, D - d0);
    const float* xa = parents + (size_t)pidx[ca] * D + d0;
    if (p >= pairs) {  // odd population: the last child copies its parent
        for (int i = 0; i < cnt; ++i) off[(size_t)ca * D + d0 + i] = xa[i];
        return;
    }
    const float* xb = parents + (size_t)pidx[cb] * D + d0;
    float a[4], bv[4], lo[4], hi[4];
    if (vec) {
        const float4 a4 = __ldg(reinterpret_cast<const float4*>(xa));
        const float4 b4 = __ldg(reinterpret_cast<const float4*>(xb));
        const float4 l01 = __ldg(reinterpret_cast<const float4*>(bounds + 2 * d0));
        const float4 l23 = __ldg(reinterpret_cast<const float4*>(bounds + 2 * d0 + 4));
        a[0] = a4.x; a[1] = a4.y; a[2] = a4.z; a[3] = a4.w;
        bv[0] = b4.x; bv[1] = b4.y; bv[2] = b4.z; bv[3] = b4.w;
        lo[0] = l01.x; hi[0] = l01.y; lo[1] = l01.z; hi[1] = l01.w;
        lo[2] = l23.x; hi[2] = l23.y; lo[3] = l23.z; hi[3] = l23.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool in = i < cnt;
            a[i] = in ? xa[i] : 0.0f;
            bv[i] = in ? xb[i] : 0.0f;
            lo[i] = in ? bounds[2 * (d0 + i)] : 0.0f;
            hi[i] = in ? bounds[2 * (d0 + i) + 1] : 0.0f;
        }
    }
    uint32_t r[4], rt[4] = {0u, 0u, 0u, 0u}, rc[4] = {0u, 0u, 0u, 0u};
    rng_block(seed, (uint64_t)t, gen, kTagCrossover, r);
    if (sbx_prob < 1.0f) rng_block(seed, (uint64_t)t, gen, kTagCrossTest, rt);
    if (copy_prob > 0.0f) rng_block(seed, (uint64_t)t, gen, kTagCopy, rc);
    float c1[4], c2[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        sbx_pair<kCall>(a[i], bv[i], u32_to_unit(r[i]), u32_to_unit(rt[i]), (int)(r[i] & 1u), u32_to_unit(rc[i]), eta_c,
                 sbx_prob, copy_prob, lo[i], hi[i], c1[i], c2[i]);
    float* oa = off + (size_t)ca * D + d0;
    float* ob = off + (size_t)cb * D + d0;
    if (vec) {
        *reinterpret_cast<float4*>(oa) = make_float4(c1[0], c1[1], c1[2], c1[3]);
        *reinterpret_cast<float4*>(ob) = make_float4(c2[0], c2[1], c2[2], c2[3]);
    } else {
        for (int i = 0; i < cnt; ++i) {
            oa[i] = c1[i];
            ob[i] = c2[i];
        }
    }
}

// Polynomial mutation of child c in place at its geometric sites (layout
// above), by the four lanes sub = 0..3 of a lane group: draws k = 4i + sub
// are evaluated side by side, their gaps summed with shuffles, and every lane
// mutates its own site (sites are distinct).  Each draw moves the site by at
// least one, so a child takes at most D/4 + 1 rounds.  All four lanes of the
// group call this together (c and `active` uniform within the group).
template <bool kCall = false>
__device__ __forceinline__ void mutate_child4(int c, bool active, int sub, float* __restrict__ off,
                                              const float* __restrict__ bounds, int n_off, int D, float eta_m,
                                              float pm_prob, uint64_t seed, uint32_t gen)
{
    const float limit = pm_prob / static_cast<float>(D);
    const double log_keep = limit >= 1.0f ? 0.0 : log1p(-(double)limit);
    const unsigned group = 0xFu << (threadIdx.x & 28u);
    float* row = off + (size_t)c * D;
    long long site = -1;  // the group's last site
    bool live = active && limit > 0.0f;
    for (long long k0 = 0; __any_sync(group, live); k0 += 4) {
        uint32_t w[4] = {0u, 0u, 0u, 0u};
        long long step = 1;
        if (live) {
            rng_block(seed, (uint64_t)(k0 + sub) * (uint64_t)n_off + (uint64_t)c, gen, kTagMutation, w);
            if (log_keep < 0.0) {
                const double u = (double)((w[0] >> 8) + 1u) * (1.0 / 16777216.0);
                const double g = floor(log(u) / log_keep);
                step += g < (double)D ? (long long)g : (long long)D;
            }
        }
        // inclusive sum of the steps over the group's lanes 0..sub
        long long acc = step;
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            const long long v = __shfl_up_sync(group, acc, o, 4);
            if (sub >= o) acc += v;
        }
        const long long my_site = site + acc;
        if (live && my_site < D) {
            const int d = (int)my_site;
            // test draw 0 < limit: the site mutates (pm_value's own test passes)
            row[d] = pm_value<kCall>(row[d], 0.0f, u32_to_unit(w[1]), eta_m, pm_prob, D, bounds[2 * d], bounds[2 * d + 1]);
        }
        site = __shfl_sync(group, my_site, 3, 4);
        live = live && site < D;
    }
}

}  // namespace
}  // namespace moea

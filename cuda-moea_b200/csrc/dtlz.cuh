// Objectives and violation of one row of the DTLZ family (device code of
// problems.cu and offspring.cu; the summation order is described there).
#pragma once

#include <math_constants.h>

#include "internal.cuh"
#include "variation.cuh"

namespace moea {
namespace {

enum Base { kDTLZ1 = 1, kDTLZ2, kDTLZ3, kDTLZ4, kDTLZ5, kDTLZ6, kDTLZ7, kConvexDTLZ2 };

__host__ __device__ inline int base_kind(int kind)
{
    switch (kind) {
    case 9: return kDTLZ1;    // C1-DTLZ1
    case 10: return kDTLZ3;   // C1-DTLZ3
    case 11: return kDTLZ2;   // C2-DTLZ2
    case 12: return kConvexDTLZ2;
    case 13: return kDTLZ1;   // C3-DTLZ1
    case 14: return kDTLZ4;   // C3-DTLZ4
    default: return kind;
    }
}

// The math functions as calls for the kernels that hold many of them (see
// powf_call).
__device__ __noinline__ float cosf_call(float a) { return cosf(a); }
__device__ __noinline__ float sinf_call(float a) { return sinf(a); }
template <bool kCall>
__device__ __forceinline__ float cosine(float a)
{
    if constexpr (kCall) return cosf_call(a);
    else return cosf(a);
}
template <bool kCall>
__device__ __forceinline__ float sine(float a)
{
    if constexpr (kCall) return sinf_call(a);
    else return sinf(a);
}

// One g-term added to a running partial.
template <int B, bool kCall = false>
__device__ __forceinline__ float g_accumulate(float thread_sum, float xv)
{
    if (B == kDTLZ1 || B == kDTLZ3) {
        const float val = xv - 0.5f;
        thread_sum += val * val - cosf(20.0f * M_PI * val);  // contracted with the cosine's last product: inline
    } else if (B == kDTLZ6) {
        thread_sum += power<kCall>(xv, 0.1f);
    } else if (B == kDTLZ7) {
        thread_sum += xv;
    } else {
        const float val = xv - 0.5f;
        thread_sum += val * val;
    }
    return thread_sum;
}

__device__ __forceinline__ float warp_tree(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
    return v;
}

// Final fold of the eight warp partials (lane 0 holds them in ws).
template <int B>
__device__ __forceinline__ float fold_partials(const float* ws)
{
    if (B == kDTLZ5) {
        // warp-0 shuffle tree over the partials, lanes 8..31 zero
        const float a = ws[0] + ws[4], b = ws[1] + ws[5], c = ws[2] + ws[6], d = ws[3] + ws[7];
        return (a + c) + (b + d);
    }
    float total = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) total += ws[w];
    return total;
}

__device__ __forceinline__ float safe_cos_hp(float v) { return fmaxf(0.0f, cosf(v * M_PI / 2.0f)); }

// Objective m of one row from its g sum; x points at the row.  Each
// objective is the reference's expression for it (dtlz_kernels.cu:28-716),
// evaluated independently, so different threads may compute different m.
template <int B>
__device__ float row_objective(int m, float total_sum, const float* x, int D, int M)
{
    const int k = D - (M - 1);
    if (B == kDTLZ1) {
        const float g = 100.0f * (static_cast<float>(k) + total_sum);
        const float scalar = 0.5f * (1.0f + g);
        float f = scalar;
        for (int j = 0; j < M - 1 - m; ++j) f *= fmaxf(0.0f, fminf(1.0f, x[j]));
        if (m > 0) f *= fmaxf(0.0f, 1.0f - x[M - 1 - m]);
        return f;
    } else if (B == kDTLZ2 || B == kDTLZ3 || B == kConvexDTLZ2 || B == kDTLZ4) {
        const float g = (B == kDTLZ3) ? 100.0f * (static_cast<float>(k) + total_sum) : total_sum;
        float f = 1.0f + g;
        for (int j = 0; j < M - 1 - m; ++j)
            f *= (B == kDTLZ4) ? fmaxf(0.0f, cosf(powf(x[j], 100.0f) * M_PI / 2.0f))
                               : safe_cos_hp(x[j]);
        if (m > 0)
            f *= (B == kDTLZ4) ? sinf(powf(x[M - 1 - m], 100.0f) * M_PI / 2.0f)
                               : sinf(x[M - 1 - m] * M_PI / 2.0f);
        if (B == kConvexDTLZ2) {
            if (m < M - 1) { f = f * f; f = f * f; } else { f = f * f; }
        }
        return f;
    } else if (B == kDTLZ5 || B == kDTLZ6) {
        const float g = total_sum;
        const float denom = 2.0f * (1.0f + g);
        auto theta = [&](int i) -> float {
            if (i == 0) return x[0];
            float t = (1.0f + 2.0f * g * x[i]) / denom;
            if (B == kDTLZ5) t = fmaxf(0.0f, fminf(1.0f, t));
            return t;
        };
        float f = 1.0f + g;
        for (int j = 0; j < M - 1 - m; ++j)
            f *= (B == kDTLZ5) ? fmaxf(0.0f, __cosf(theta(j) * M_PI * 0.5f))
                               : fmaxf(0.0f, cosf(theta(j) * M_PI * 0.5f));
        if (m > 0)
            f *= (B == kDTLZ5) ? __sinf(theta(M - 1 - m) * M_PI * 0.5f)
                               : sinf(theta(M - 1 - m) * M_PI * 0.5f);
        return f;
    } else {  // kDTLZ7
        if (m < M - 1) return x[m];
        const float g = 1.0f + (9.0f / static_cast<float>(k)) * total_sum;
        float h_sum = 0.0f;
        for (int i = 0; i < M - 1; ++i) {
            const float fi = x[i];
            h_sum += (fi / (1.0f + g)) * (1.0f + sinf(3.0f * M_PI * fi));
        }
        const float h = static_cast<float>(M) - h_sum;
        return (1.0f + g) * h;
    }
}

// The two factors of position variable q that row_objective evaluates (with its
// multiply-adds spelled out): cosine
// and sine of its angle, or the factors of its term in DTLZ7's h.
template <int B, bool kCall>
__device__ __forceinline__ void row_factors(int q, float total_sum, const float* x, int D, int M, float* a, float* b)
{
    const int k = D - (M - 1);
    if (B == kDTLZ2 || B == kDTLZ3 || B == kConvexDTLZ2) {
        *a = fmaxf(0.0f, cosine<kCall>(x[q] * M_PI / 2.0f));
        *b = sine<kCall>(x[q] * M_PI / 2.0f);
    } else if (B == kDTLZ4) {
        const float p = power<kCall>(x[q], 100.0f);
        *a = fmaxf(0.0f, cosine<kCall>(p * M_PI / 2.0f));
        *b = sine<kCall>(p * M_PI / 2.0f);
    } else if (B == kDTLZ5 || B == kDTLZ6) {
        const float g = total_sum;
        float t = x[0];
        if (q > 0) {
            t = fmaf(2.0f * g, x[q], 1.0f) / (2.0f * (1.0f + g));
            if (B == kDTLZ5) t = fmaxf(0.0f, fminf(1.0f, t));
        }
        *a = (B == kDTLZ5) ? fmaxf(0.0f, __cosf(t * M_PI * 0.5f)) : fmaxf(0.0f, cosine<kCall>(t * M_PI * 0.5f));
        *b = (B == kDTLZ5) ? __sinf(t * M_PI * 0.5f) : sine<kCall>(t * M_PI * 0.5f);
    } else {  // kDTLZ7
        const float g = fmaf(9.0f / static_cast<float>(k), total_sum, 1.0f);
        const float fi = x[q];
        *a = fi / (1.0f + g);
        *b = 1.0f + sine<kCall>(3.0f * M_PI * fi);
    }
}

// row_objective from the factors (called by every lane of the group; m >= M and
// rows that are not valid give no result).
template <int B, class FA, class FB>
__device__ __forceinline__ float combine_factors(int m, float total_sum, const float* x, int D, int M, bool valid,
                                                 FA fa, FB fb)
{
    const int k = D - (M - 1);
    if (B == kDTLZ7) {
        const float g = fmaf(9.0f / static_cast<float>(k), total_sum, 1.0f);
        float h_sum = 0.0f;
        for (int i = 0; i < M - 1; ++i) {
            const float a = fa(i), b = fb(i);
            h_sum = fmaf(a, b, h_sum);
        }
        const float h = static_cast<float>(M) - h_sum;
        return m < M - 1 ? (valid ? x[m] : 0.0f) : (1.0f + g) * h;
    }
    const float g = (B == kDTLZ3) ? 100.0f * (static_cast<float>(k) + total_sum) : total_sum;
    float f = 1.0f + g;
    for (int j = 0; j < M - 1; ++j) {
        const float c = fa(j);
        if (j < M - 1 - m) f *= c;
    }
    const float s = fb(m > 0 && m < M ? M - 1 - m : 0);
    if (m > 0) f *= s;
    if (B == kConvexDTLZ2) {
        if (m < M - 1) {
            f = f * f;
            f = f * f;
        } else {
            f = f * f;
        }
    }
    return f;
}

// A group of G lanes (8 or 32) per row; valid when the row has at most 256
// g-terms.  Every lane of the warp calls; rows that are not `valid` write
// nothing.  The partials are those of a shuffle-down tree over 32 lanes: with
// G = 8 a lane holds four of its leaves and folds the first two levels itself.
template <int B, int G, bool kCall = false>
__device__ __forceinline__ void dtlz_group_row(int row, bool valid, int gl, const float* x, int N, int D, int M,
                                               float* objs)
{
    constexpr int kLeaves = 32 / G;
    const int start = (B == kDTLZ7) ? D - (D - M + 1) : M - 1;
    const int k = D - start;
    // partial w: the tree over the terms 32 w .. 32 w + 31 (zero without terms)
    auto partial = [&](int w) {
        float v[kLeaves];
#pragma unroll
        for (int i = 0; i < kLeaves; ++i) {
            const int t = gl + G * i + 32 * w;
            v[i] = 0.0f;
            if (valid && t < k) v[i] = g_accumulate<B, kCall>(v[i], x[start + t]);
        }
#pragma unroll
        for (int o = kLeaves / 2; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < o; ++i) v[i] += v[i + o];
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v[0] += __shfl_down_sync(0xFFFFFFFFu, v[0], o, G);
        return v[0];
    };
    float total = 0.0f;
    if constexpr (B == kDTLZ5) {
        float ws[8];
#pragma unroll
        for (int w = 0; w < 8; ++w) ws[w] = 32 * w < k ? partial(w) : 0.0f;
        total = fold_partials<B>(ws);
    } else {
        // in order, as fold_partials adds them
#pragma unroll 1
        for (int w = 0; 32 * w < k; ++w) total += partial(w);
    }
    total = __shfl_sync(0xFFFFFFFFu, total, 0, G);
    if constexpr (B == kDTLZ1) {
        if (valid)
            for (int m = gl; m < M; m += G) objs[(size_t)m * N + row] = row_objective<B>(m, total, x, D, M);
    } else {
        // The factors of position variable j (cosine and sine, or the two
        // factors of a DTLZ7 term) belong to every objective: lane j mod G
        // evaluates them once and the products pick them up with shuffles, in
        // row_objective's order (M - 1 evaluations per lane without: eight
        // objectives of DTLZ4 took 14 powf per child and lane).
        constexpr int kSlots = kMaxObjectives / G > 0 ? kMaxObjectives / G : 1;
        float fa[kSlots], fb[kSlots];
#pragma unroll
        for (int v = 0; v < kSlots; ++v) {
            const int q = gl + G * v;
            fa[v] = fb[v] = 0.0f;
            if (valid && q < M - 1) row_factors<B, kCall>(q, total, x, D, M, &fa[v], &fb[v]);
        }
        auto pick = [&](const float (&f)[kSlots], int q) {  // factor q of the row, by every lane
            float r = 0.0f;
#pragma unroll
            for (int v = 0; v < kSlots; ++v) {
                const float y = __shfl_sync(0xFFFFFFFFu, f[v], q & (G - 1), G);
                if (q / G == v) r = y;
            }
            return r;
        };
        for (int m0 = 0; m0 < M; m0 += G) {
            const int m = m0 + gl;
            const float f = combine_factors<B>(m, total, x, D, M, valid, [&](int q) { return pick(fa, q); },
                                               [&](int q) { return pick(fb, q); });
            if (valid && m < M) objs[(size_t)m * N + row] = f;
        }
    }
}

// Constraint violation of one row from its objectives f[m * N]
// (dtlz_kernels.cu:824-1090).
__device__ __forceinline__ float constraint_violation(int kind, const float* f, int N, int M, float R)
{
    float cv = 0.0f;
    switch (kind) {
    case 9: {
        float constraint = f[(size_t)(M - 1) * N] / 0.6f;
        for (int m = 0; m < M - 1; m++) {
            const float f_m = f[(size_t)m * N];
            constraint += f_m / 0.5f;
        }
        cv = fmaxf(constraint - 1.0f, 0.0f);
        break;
    }
    case 10: {
        const float R_sqr = R * R;
        float fv_sqr = 0.0f;
        for (int m = 0; m < M; m++) {
            const float f_m = f[(size_t)m * N];
            fv_sqr += f_m * f_m;
        }
        cv = fmaxf((fv_sqr - 16.0f) * (R_sqr - fv_sqr), 0.0f);
        break;
    }
    case 11: {
        const float inv_sqrt_M = 1.0f / sqrtf((float)M);
        const float r2 = R * R;
        const float inv_r2 = 1.0f / r2;
        float sum_f2 = 0.0f;
        for (int m = 0; m < M; ++m) {
            const float fm = f[(size_t)m * N];
            sum_f2 = fmaf(fm, fm, sum_f2);
        }
        float min_cv = CUDART_INF_F;
        for (int m = 0; m < M; ++m) {
            const float fm = f[(size_t)m * N];
            const float diff = fm - 1.0f;
            const float dist2 = fmaf(diff, diff, sum_f2 - fm * fm);
            min_cv = fminf(min_cv, dist2 * inv_r2 - 1.0f);
        }
        float center_sum2 = 0.0f;
        for (int m = 0; m < M; ++m) {
            const float df = f[(size_t)m * N] - inv_sqrt_M;
            center_sum2 = fmaf(df, df, center_sum2);
        }
        cv = fmaxf(fminf(min_cv, center_sum2 * inv_r2 - 1.0f), 0.0f);
        break;
    }
    case 12: {
        const float inv_M = 1.0f / static_cast<float>(M);
        const float inv_R_sqr = 1.0f / (R * R);
        float sum = 0.0f, sum_sq = 0.0f;
        for (int m = 0; m < M; m++) {
            const float f_m = f[(size_t)m * N];
            sum += f_m;
            sum_sq += f_m * f_m;
        }
        const float mean = sum * inv_M;
        const float variance = sum_sq - static_cast<float>(M) * mean * mean;
        cv = fmaxf(1.0f - variance * inv_R_sqr, 0.0f);
        break;
    }
    case 13: {
        float fv_sum = 0.0f;
        for (int m = 0; m < M; m++) fv_sum += f[(size_t)m * N];
        fv_sum *= 2.0f;
        for (int m = 0; m < M; m++) {
            float c = f[(size_t)m * N] + 1.0f - fv_sum;
            cv += fmaxf(c, 0.0f);
        }
        break;
    }
    case 14: {
        float fv_sqr = 0.0f;
        for (int m = 0; m < M; m++) {
            const float f_m = f[(size_t)m * N];
            fv_sqr += f_m * f_m;
        }
        for (int m = 0; m < M; m++) {
            const float f_m = f[(size_t)m * N];
            float c = 0.75f * (f_m * f_m) - fv_sqr;
            c += 1.0f;
            cv += fmaxf(c, 0.0f);
        }
        break;
    }
    default: break;
    }
    return cv;
}

inline float cv_radius(int kind, int M)
{
    switch (kind) {
    case 10: return M == 2 ? 6.0f : M == 3 ? 5.0f : M == 5 ? 12.5f : 15.0f;
    case 11: return M == 2 ? 0.15f : M == 3 ? 0.40f : 1.0f;
    case 12: return M == 3 ? 0.20f : M == 5 ? 0.225f : (M == 8 || M == 10) ? 0.26f : M == 15 ? 0.27f : 0.225f;
    default: return 0.0f;
    }
}

}  // namespace
}  // namespace moea

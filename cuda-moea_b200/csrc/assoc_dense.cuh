// FP32 association by a search over every direction: dense (assoc_dense.cu) or
// split over ranges of directions (assoc_scan.cu).
#pragma once

#include "internal.cuh"

namespace moea {

// Nearest of H directions (M, H) for the first *d_n <= n_cap points of x, each
// objective multiplied by scale (may be null).  delta: max | |r|^2 - 1 | of the
// directions, from d_delta when it is not null.  best: n_cap words of scratch;
// sms: multiprocessors of the device.
int run_assoc_search(const float* x, int x_stride, const float* scale, const float* refs, int M, const int* d_n, int n_cap,
                     int H, float delta, const float* d_delta, unsigned long long* best, int sms, int* idx, float* dist,
                     cudaStream_t stream);

int run_assoc_scan(const float* x, int x_stride, const float* scale, const float* refs, int M, const int* d_n, int n_cap,
                   int H, float delta, const float* d_delta, unsigned long long* best, int sms, int* idx, float* dist,
                   cudaStream_t stream);

int fused_associate_dense(const BatchInst* d_inst, const FusedBucket& b, cudaStream_t s);

}  // namespace moea

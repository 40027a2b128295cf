// Offspring of one generation in one launch (offspring.cu).
#pragma once

#include "internal.cuh"

namespace moea {

constexpr int kOffspringMaxD = 704;    // eight pairs' rows in 48 KB of shared memory
constexpr int kOffspringGroupD = 184;  // thirty-two pairs' rows

struct OffspringArgs {
    const float* parents;
    const float* cv;           // violations and
    const int* rank;           // ranks of the parents (tournament; null: random mating)
    const int* d_active;       // device count of usable parents, or null:
    int active;
    const float* bounds;
    float* off;
    int* pidx;
    float* objs;
    float* cv_out;
    const int* cv_table;       // per generation: violations count (null: always)
    int n_off, D, M;
    int kind;                  // problem kind, 0: evaluated by the caller
    int mutate, vec, total;
    float sbx_eta0, sbx_eta1, sbx_prob, copy_prob, pm_eta0, pm_eta1, pm_prob;
    float radius;
    uint64_t seed;
    const int* d_gen;          // device generation, or null:
    uint32_t gen;
};

bool offspring_eligible(int kind, int D, int M);
int run_offspring(OffspringArgs args, cudaStream_t stream);

}  // namespace moea

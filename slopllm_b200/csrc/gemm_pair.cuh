// GEMM on pairs of SMs (gemm_pair_tcgen05.cu), called by the entry points of gemm_tcgen05.cu.
#pragma once

#include "common.cuh"

struct GemmPairParams {
    void* C; int ldc, out_f32;
    int M, N, K;
    int a_group_cols, a_group_stride;      // batched product: output columns per group (0: plain), A columns between groups
    int* err;
    int tiles_m, tiles_n, total;           // set by the launcher
    int gated;                             // N output columns silu(gate) * up of 2 N weight rows gate | up (bf16 output)
};

// Whether the pair kernel is the faster one: as many 256 x 256 tiles as there are pairs (fewer leave SMs idle that 128-row tiles use), and no
// second round for a product that 128-row tiles do in one.
bool gemm_pair_ok(int M, int N);
int gemm_pair(const void* A, const void* B, GemmPairParams p, int lda, int ldb, int a_cols, cudaStream_t s);

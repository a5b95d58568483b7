// out[M, N] = x[M, K] · w[N, K]^T in true float32 (no reduced-precision unit): the 32-bit path's product, where K is a
// multiple of 4 of at least GF_MIN_K and both operands start on 16 bytes (gemm_generic.cu has the rest).
#pragma once
#include "common.cuh"

// Below, a tile is all set-up and store, which gemm_generic.cu's small CTAs overlap better: 4 096 x 16 at 2 048 rows 17 us there and 23
// with the best of these tiles, 1 024 x 16 5.9 and 7.2 (the choice is one of K alone: the two add up in different orders).
#define GF_MIN_K 48

// 0 on success, as every entry point.  `act` as in common.cuh.
int qe_gemm_f32(const float* x, const float* w, float* out, int M, int N, int K, int act, cudaStream_t stream);

// out[M, N] = x[M, K] · w[N, K]^T in true float32 (no reduced-precision unit): the 32-bit path's product, where K is a
// multiple of 4 and both operands start on 16 bytes (gemm_generic.cu has the rest).
#pragma once
#include "common.cuh"

// 0 on success, as every entry point.  `act` as in common.cuh.
int qe_gemm_f32(const float* x, const float* w, float* out, int M, int N, int K, int act, cudaStream_t stream);

// The 32-bit products that the launchers of gemm_simt.cu and gemm_skinny.cu hand on: fp32 rows,
// fp32 weights.  Both return false where they do not apply (nothing is launched then).
#pragma once

#include "common.cuh"

// out[M,N] = act(X W^T + bias) (+ residual) in 64 x 64 tiles, any number of rows (gemm_f32.cu).
template <typename TOut>
bool nb_gemm_f32_tiles(const float* X, const float* W, const float* bias, const float* residual,
                       TOut* out, int M, int N, int K, int act, cudaStream_t stream,
                       cudaError_t* err);

// The same for the few rows of a decode step: weights through registers (gemm_rows_f32.cu).
template <typename TOut>
bool nb_gemm_f32_rows(const float* X, const float* W, const float* bias, const float* residual,
                      TOut* out, int M, int N, int K, int act, cudaStream_t stream,
                      cudaError_t* err);

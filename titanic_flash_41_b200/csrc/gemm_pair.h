// The bf16 form of the pair GEMM (gemm_mx.cu), called by tf_gemm_tc.
#pragma once
#include <cuda_runtime.h>

// C[M, N] (ldc elements a row; out_kind 0 f32, 2 bf16) = A[M, K] B[N, K]^T, bf16, lda / ldb elements; K a multiple of 64
int tf_gemm_pair_bf16(const void* A, long lda, const void* B, long ldb, void* C, int ldc, int out_kind, int M, int N, int K,
                      void* status, cudaStream_t st);

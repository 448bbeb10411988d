// Launcher of the fp32 CUDA-core GEMM.
#pragma once
#include "common.cuh"

namespace blstm {

// C[M,N] = A*B (+bias0+bias1), dense.  a_kc: A(m,k) = A[m*lda + k], else A[k*lda + m]; b_kc: B(k,n) = B[n*ldb + k], else
// B[k*ldb + n].  (A along M with B along K is not provided.)  splits > 1 needs `partials` [splits][M][N].
int f32_gemm(int M, int N, int K, const float* A, long long lda, bool a_kc, const float* B, long long ldb, bool b_kc, float* C,
             const float* bias0, const float* bias1, int splits, float* partials, cudaStream_t st);
int f32_gemm_splits(int M, int N, int K, int sm_count);

}  // namespace blstm

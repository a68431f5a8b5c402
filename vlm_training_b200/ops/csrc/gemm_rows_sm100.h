// GEMM of at most 128 rows, both operands K-major, bf16 D of any alignment (gemm_rows_sm100.cu).  splits (1 to 8): blocks of a cluster that
// share a tile's K; every one needs a part of it.
#pragma once
#include <cuda_runtime.h>
#ifdef __cplusplus
extern "C" {
#endif
// the split for these sizes, 0: not the kernel for them
int vlmt_gemm_rows_splits(int M, int N, int K, int num_sms);
int vlmt_gemm_rows(const void* X, const void* W, void* D, const void* bias, int M, int N, int K, int lda, int ldb, int ldd, int epilogue,
                   const float* alpha, int splits, int* status, int num_sms, cudaStream_t stream);
// act[M, I] = silu(gate) * up with [gate; up] = X(M,K) W(2 I,K)^T; gu (or null) [M, 2 I]; I a multiple of 64, act and gu on 8 bytes
int vlmt_gemm_rows_glu(const void* X, const void* W, void* gu, void* act, int M, int I, int K, int lda, int ldb, int splits, int* status, int num_sms,
                       cudaStream_t stream);
#ifdef __cplusplus
}
#endif

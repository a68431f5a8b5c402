// CTA-pair GEMM for large outputs (gemm_pair_sm100.cu); operand layouts as vlmt_gemm_bf16, bf16 D with 16-byte aligned rows.
// k_splits > 1 (accumulate only): K parts of kb_per_split 64-wide blocks are added to D one by one.  parts = 2 (k_splits 1, at most
// vlmt_gemm_pair_clusters() tiles): the pairs of a cluster compute a K part of one tile each and sum them, in fp32.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#ifdef __cplusplus
extern "C" {
#endif
int vlmt_gemm_pair_enabled();   // 0 with VLMT_GEMM_PAIR=0: every GEMM, bf16 and FP8, on one-block tiles (A/B comparison)
int vlmt_gemm_pair(const void* A, const void* B, void* D, const void* bias, int M, int N, int K, int lda, int ldb, int ldd, int a_mn_major,
                   int b_mn_major, int epilogue, int accumulate, const float* alpha, int k_splits, int kb_per_split, int parts, int* status,
                   cudaStream_t stream);
int vlmt_gemm_pair_clusters();
int vlmt_gemm_pair_grouped(const void* A, const void* B, void* D, const int* prefix, int groups, int M, int N, int rows, int lda, int ldb, int ldd,
                           int accumulate, int* status, cudaStream_t stream);
int vlmt_gemm_pair_gelu(const void* X, const void* W, const void* bias, void* x, void* y, int M, int N, int K, int ldx, int ldw, int epilogue,
                        int* status, cudaStream_t stream);
int vlmt_gemm_pair_gelu_bwd(const void* dY, const void* W, const void* x, void* dx, void* y, int M, int N, int K, int ldy, int ldw, int epilogue,
                            int* status, cudaStream_t stream);
int vlmt_gemm_pair_glu_bwd(const void* dY, const void* W, const void* gu, void* dgu, void* act, int M, int I, int K, int ldy, int ldw, int* status,
                           cudaStream_t stream);
int vlmt_gemm_pair_glu(const void* X, const void* W, void* gu, void* act, int M, int I, int K, int ldx, int ldw, int* status, cudaStream_t stream);
// D (+)= rec_a[1] * rec_b[1] * A(M,K) * B(N,K)^T, one byte per element, arguments checked by vlmt_gemm_fp8; idesc: instruction
// descriptor of kind::f8f6f4 for M = 256, N = 256.  k_splits as above in parts of kb_per_split 128-wide blocks.
int vlmt_gemm_pair_fp8(const void* A, const void* B, void* D, int M, int N, int K, long lda, long ldb, long ldd, uint32_t idesc, const float* rec_a,
                       const float* rec_b, int accumulate, int k_splits, int kb_per_split, int* status, cudaStream_t stream);
#ifdef __cplusplus
}
#endif

// C entry points of the cross-entropy and AdamW kernels (loss_optim.cu).
#pragma once
#include <cuda_runtime.h>
// destination of a column sum: fp32 or bf16 values, or a bf16 gradient it is added to
enum { VLMT_SUM_F32 = 0, VLMT_SUM_BF16 = 1, VLMT_SUM_ADD_BF16 = 2 };
// up to two sums over the rows of partial[i] (row stride ld) in one launch
struct VlmtRowSums { const float* partial[2]; long ld; void* out[2]; int mode[2]; };
#ifdef __cplusplus
extern "C" {
#endif
// In place: logits[rows, V] -> grad_scale * (softmax - onehot); loss[row] = lse - logit[target] (0 if ignored).
// want_grad == 0: the loss only, the logits stay.
void vlmt_ce_fwd_bwd(void* logits, long ld, const long* targets, float* loss, float grad_scale, int rows, int V, long ignore_index,
                     int want_grad, cudaStream_t st);
// m / v are fp32, or bf16 when state_bf16 != 0
// zero_grad != 0: the gradient range is cleared after it has been consumed
void vlmt_adamw(void* grad, int grad_fp32, float* master, void* m, void* v, int state_bf16, void* param, long n, float lr, float b1,
                float b2, float eps, float wd, float bc1, float bc2, float grad_scale, int zero_grad, cudaStream_t st);
// One launch for a parameter bucket of n elements (a multiple of 8, bf16 gradient and parameter, 16-byte aligned bases): segment s
// covers elements [8 seg_start[s], 8 seg_start[s + 1]) (seg_start has one entry more than there are segments) and belongs to
// group seg_group[s] (lr[g], wd[g], at most 16 groups); chunk_seg[c] is the segment of element c * vlmt_adamw_chunk(), with one
// entry behind the last chunk.  The gradient is cleared.
int vlmt_adamw_chunk();
int vlmt_adamw_bucket(void* grad, float* master, void* m, void* v, int state_bf16, void* param, long n, const int* seg_start, const int* seg_group,
                      const int* chunk_seg, const float* lr, const float* wd, int groups, float b1, float b2, float eps, float bc1, float bc2,
                      float grad_scale, cudaStream_t st);
void vlmt_sum_rows(const struct VlmtRowSums* a, int sums, int rows, int cols, cudaStream_t st);
int vlmt_colsum_slabs(int rows);   // 0: no partial sums in memory
int vlmt_colsum(const void* x, long ld, int rows, int cols, float* partial, void* out, int mode, cudaStream_t st);
int vlmt_embed_blocks(int T);
int vlmt_embed_bwd(const void* dy, const long* ids, const long* perm, int T, int D, void* grad, float* part, cudaStream_t st);
void vlmt_sumsq(const void* x, int fp32, long n, float* out, cudaStream_t st);
#ifdef __cplusplus
}
#endif

// C entry points of the kernels that make per-batch tables (rotary tables, the vision tower's plan) and apply the vision tower's
// interpolated position embedding (plan_kernels.cu).
#pragma once
#include <cuda_runtime.h>
#ifdef __cplusplus
extern "C" {
#endif
// cos / sin [T, 2 n] fp32 of pos * inv_freq [n], both halves alike.  pos int64 [axes, T], axes 1 or 3; with 3, frequency j takes
// axis 1 when j % 3 == 1 and j < 3 sec1, axis 2 when j % 3 == 2 and j < 3 sec2, else axis 0.
void vlmt_rope_tables(const long* pos, int axes, const float* inv_freq, int n, int sec1, int sec2, long T, float* cosv, float* sinv,
                      cudaStream_t st);
// images int32 [n_img, 4]: frames, height, width in patches, first patch.  Patches are in merge-block order (merge x merge blocks).
// cosv / sinv [N, 4 nf] fp32, gathered from trig [coords, nf, 2] (cosine and sine of every row or column times every frequency, 8-byte
// aligned; coords above the largest height and width); pe_index int64 [4, N], pe_weight fp32 [4, N]: corners and weights of the bilinear
// resampling of a side x side table onto each image's grid.
void vlmt_vision_plan(const int* images, int n_img, const float* trig, int coords, int nf, int side, int merge, long N, float* cosv,
                      float* sinv, long* pe_index, float* pe_weight, cudaStream_t st);
// out[n] = x[n] + bf16(sum_c pe_weight[c, n] * table[pe_index[c, n]]), rows of D bf16 (D a multiple of 8)
void vlmt_pos_embed_fwd(const void* x, const void* table, const long* pe_index, const float* pe_weight, void* out, long N, int D, cudaStream_t st);
// gradient of the table [side * side, D] from dy [N, D]: stored in, or (accumulate) added to, the bf16 `dtable`
void vlmt_pos_embed_bwd(const void* dy, const int* images, int n_img, int side, int merge, long N, void* dtable, int accumulate, int D,
                        cudaStream_t st);
#ifdef __cplusplus
}
#endif

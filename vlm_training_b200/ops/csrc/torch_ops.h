// Tensor-level entry points of the kernels (bindings*.cpp), shared by the Python bindings and the C++ autograd functions
// (bindings_autograd.cpp).
#pragma once
#include <torch/extension.h>

#include <vector>

namespace vlmt {
using torch::Tensor;
using OptTensor = c10::optional<Tensor>;

int num_sms();
void count_launches(int n);   // of this package's kernels, see op_launches
void gemm(const Tensor& a, const Tensor& b, Tensor& out, bool a_mn, bool b_mn, const OptTensor& bias, int64_t epilogue, bool accumulate,
          const OptTensor& alpha, bool one_sum = false);   // one_sum: see vlmt_gemm_bf16
bool gemm_gelu(const Tensor& x, const Tensor& w, const OptTensor& bias, bool tanh_approx, Tensor* pre, Tensor& act);
bool gemm_gelu_bwd(const Tensor& dy, const Tensor& w, const Tensor& x, bool tanh_approx, Tensor& dx, Tensor* y);   // gradient of x from dy w
bool gemm_glu_bwd(const Tensor& dy, const Tensor& w, const Tensor& gu, Tensor& dgu, Tensor* act);   // gradient of gate and up from dy w
bool gemm_glu(const Tensor& x, const Tensor& w, Tensor* gu, Tensor& act);   // silu(gate) * up of a gate / up projection; false: not for these sizes
std::vector<Tensor> rmsnorm_fwd(const Tensor& x, const OptTensor& res, const Tensor& w, double eps, bool offset);
// *_partial: the weight gradients as per-block partial rows, to be summed by vlmt_sum_rows
std::vector<Tensor> rmsnorm_bwd_partial(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& rstd, const OptTensor& dres, bool offset,
                                        Tensor* yn = nullptr);   // yn: rmsnorm_fwd(x) from the same pass, in the place of dy; left alone where the kernel has no such form
std::vector<Tensor> layernorm_fwd(const Tensor& x, const Tensor& w, const OptTensor& b, double eps);
std::vector<Tensor> layernorm_bwd_partial(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& mean, const Tensor& rstd,
                                          const OptTensor& b = c10::nullopt, Tensor* yn = nullptr);   // yn: layernorm_fwd(x) with bias b, as above
std::vector<Tensor> rmsnorm_gated_fwd(const Tensor& x, const Tensor& z, const Tensor& w, double eps);
std::vector<Tensor> rmsnorm_gated_bwd_partial(const Tensor& dy, const Tensor& x, const Tensor& z, const Tensor& w, const Tensor& rstd);
Tensor swiglu_fwd(const Tensor& gu);
Tensor swiglu_bwd(const Tensor& dout, const Tensor& gu, Tensor* out = nullptr);   // out: swiglu_fwd(gu) from the same pass, in the place of dout
Tensor sigmoid_mul_fwd(const Tensor& x, const Tensor& gate);
std::vector<Tensor> sigmoid_mul_bwd(const Tensor& dout, const Tensor& x, const Tensor& gate);
Tensor gelu_fwd(const Tensor& x, bool tanh_approx);
Tensor gelu_bwd(const Tensor& dy, const Tensor& x, bool tanh_approx, Tensor* y = nullptr);   // y: gelu_fwd(x) from the same pass, in the place of dy
std::vector<Tensor> qkv_norm_rope_fwd(const Tensor& qkv, int64_t n_q, int64_t n_kv, int64_t D, const OptTensor& qw, const OptTensor& kw,
                                      const Tensor& cosv, const Tensor& sinv, double eps, bool offset, bool gated);
std::vector<Tensor> qkv_norm_rope_bwd_partial(const Tensor& dq, const Tensor& dk, const Tensor& dv, const OptTensor& dgate, const Tensor& qkv,
                                              const OptTensor& qw, const OptTensor& kw, const Tensor& cosv, const Tensor& sinv, const Tensor& rstd,
                                              int64_t n_q, int64_t n_kv, int64_t D, bool offset, bool gated);
Tensor rope_generic(const Tensor& x, const Tensor& cosv, const Tensor& sinv, bool transpose, int64_t d_out);
void rows_update(Tensor& out, const Tensor& index, const Tensor& src, bool add);
Tensor rows_gather(const Tensor& src, const Tensor& index);
void colsum_into(const Tensor& x, void* out, int mode);
std::vector<Tensor> attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu, int64_t max_seqlen, bool causal, double scale);
std::vector<Tensor> attn_bwd(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse,
                             const Tensor& cu, int64_t max_seqlen, bool causal, double scale);
}  // namespace vlmt

// The ops of a dense decoder layer and of a ViT block as C++ autograd functions.
//
// The Python form of such a function costs 25 - 40 us of host time per call and direction (argument unwrapping, context
// object, interpreter, one binding call and one allocation call per kernel); a step of the smallest VLM preset makes about
// 150 of them and was bound by that, 8 ms for 2.8 ms of kernels.  Here a call is one binding crossing, and the backward
// pass runs without the interpreter.
//
// Gradients of parameters whose `.grad` belongs to the optimizer engine (Python attribute `_vlmt_grad_in_place`) are added
// there by the kernel that forms them: the weight-gradient GEMM's epilogue, or the kernel that sums a norm weight's or
// bias's partial rows (one rounding, and no conversion, no autograd accumulation launch).  Autograd then gets nothing and the
// engine's gradient-ready callback (`_vlmt_grad_ready`) is called here.  A parameter with tensor hooks (`register_hook`), and every parameter
// in a pass that was asked for particular gradients, takes the ordinary way through autograd.
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/extension.h>

#include <atomic>

#include "elementwise.h"
#include "loss_optim.h"
#include "plan_kernels.h"
#include "torch_ops.h"

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

namespace py = pybind11;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace vlmt {
namespace {
std::atomic<int64_t> g_launches{0};   // kernels of this package launched from here (added to the Python counter)
void tick(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
bool g_in_place = true;

inline cudaStream_t cur_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

// ------------------------------------------------------------------ gradient targets
// A parameter whose gradient goes straight into `.grad`, and the engine's callback for it.
struct GradTarget : torch::CustomClassHolder {
  Tensor param;
  PyObject* ready = nullptr;
  ~GradTarget() override {
    if (ready != nullptr && Py_IsInitialized()) {
      py::gil_scoped_acquire gil;
      Py_DECREF(ready);
    }
  }
  void report() const {
    if (ready == nullptr) return;
    py::gil_scoped_acquire gil;
    py::reinterpret_borrow<py::object>(ready)(py::cast(param));
  }
};
using Target = c10::intrusive_ptr<GradTarget>;

Target target_of(const py::object& w) {
  static PyObject* k_in_place = PyUnicode_InternFromString("_vlmt_grad_in_place");
  static PyObject* k_ready = PyUnicode_InternFromString("_vlmt_grad_ready");
  if (!g_in_place || w.is_none() || !c10::GradMode::is_enabled()) return Target();
  py::object dict = py::reinterpret_steal<py::object>(PyObject_GenericGetDict(w.ptr(), nullptr));
  if (!dict) { PyErr_Clear(); return Target(); }
  PyObject* flag = PyDict_GetItemWithError(dict.ptr(), k_in_place);
  if (flag == nullptr || PyObject_IsTrue(flag) != 1) { PyErr_Clear(); return Target(); }
  Target t = c10::make_intrusive<GradTarget>();
  t->param = w.cast<Tensor>();
  PyObject* ready = PyDict_GetItemWithError(dict.ptr(), k_ready);
  if (ready != nullptr) { Py_INCREF(ready); t->ready = ready; }
  return t;
}
// Whether a gradient may be added to `.grad` behind autograd's back.  Not when somebody waits for it on the way: a tensor hook, or
// `autograd.grad` / `backward(inputs=...)`, whose graph task knows which nodes it executes (`backward()` executes all and names
// none).  Post-accumulate hooks run either way: autograd accumulates an undefined gradient and calls them.  Called in the backward pass.
bool may_add(const Tensor& param) {
  const auto* named = torch::autograd::get_current_graph_task_exec_info();
  return (named == nullptr || named->empty()) && torch::autograd::impl::hooks(param).empty();
}
bool may_add(const Target& t) { return t && may_add(t->param); }

Tensor as_tensor(const py::object& o) { return o.is_none() ? Tensor() : o.cast<Tensor>(); }
OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }
Tensor get(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }

// 2-D, unit inner stride, 16-byte aligned row stride and base (TMA requirements)
Tensor operand(const Tensor& t) {
  if (t.stride(-1) != 1 || t.stride(0) % 8 != 0 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0) return t.contiguous();
  return t;
}
Tensor rows_of(const Tensor& t) { return t.dim() == 2 ? operand(t) : operand(t.reshape({-1, t.size(-1)})); }

void check_storage(const Tensor& t) {
  // a sharded parameter (or its gradient bucket) whose storage is released: an error here, never a kernel on freed memory
  TORCH_CHECK(t.storage().nbytes() != 0 || t.numel() == 0,
              "GEMM operand without storage: a sharded parameter was used outside the forward / backward of its unit");
}
Tensor mm(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const Tensor& bias = Tensor()) {
  check_storage(b);
  Tensor out = torch::empty({a.size(a_mn ? 1 : 0), b.size(b_mn ? 1 : 0)}, a.options());
  gemm(a, b, out, a_mn, b_mn, opt(bias), 0, false, c10::nullopt);
  tick(1);
  return out;
}
// dW[N, K] = dY^T[N, M] . X[M, K], called when every other kernel of the backward pass that reads the weight has been enqueued: a tagged parameter is
// reported here, and its bucket's update may run on another stream, or in a peer's kernel, from that moment on.
Tensor weight_grad(const Tensor& dy, const Tensor& x, const Target& t) {
  if (may_add(t)) {
    Tensor g = t->param.grad();
    if (g.defined() && g.scalar_type() == at::kBFloat16 && g.dim() == 2 && g.size(0) == dy.size(1) && g.size(1) == x.size(1) &&
        g.stride(1) == 1 && g.stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(g.data_ptr()) % 16 == 0) {
      check_storage(g);
      gemm(dy, x, g, true, true, c10::nullopt, 0, true, c10::nullopt);
      tick(1);
      t->report();
      return Tensor();
    }
  }
  return mm(dy, x, true, true);
}
// where the gradient of a 1-D parameter goes: added to a tagged .grad, or a new tensor of the parameter's type
struct VecGrad {
  Tensor out, ret;
  int mode;
  bool in_place = false, convert = false;
  VecGrad(const Tensor& w, const Target& t) {
    if (may_add(t)) {
      out = t->param.grad();
      if (out.defined() && out.scalar_type() == at::kBFloat16 && out.is_contiguous() && out.numel() == w.numel()) {
        check_storage(out);
        mode = VLMT_SUM_ADD_BF16;
        in_place = true;
        return;
      }
    }
    const bool bf = w.scalar_type() == at::kBFloat16;
    mode = bf ? VLMT_SUM_BF16 : VLMT_SUM_F32;
    out = ret = torch::empty({w.numel()}, w.options().dtype(bf ? at::kBFloat16 : at::kFloat));
    convert = !bf && w.scalar_type() != at::kFloat;
  }
  Tensor finish(const Tensor& w, const Target& t) {
    if (in_place) {
      t->report();
      return Tensor();
    }
    return convert ? ret.to(w.scalar_type()).view(w.sizes()) : ret.view(w.sizes());
  }
};
// sums the partial rows of one or two 1-D parameters ([blocks, cols] each with row stride ld) in one launch
void sum_rows(const float* p0, const float* p1, long ld, int rows, int cols, const VecGrad& g0, const VecGrad* g1) {
  c10::cuda::CUDAGuard guard(g0.out.device());
  VlmtRowSums a{};
  a.ld = ld;
  a.partial[0] = p0; a.out[0] = g0.out.data_ptr(); a.mode[0] = g0.mode;
  if (g1 != nullptr) { a.partial[1] = p1; a.out[1] = g1->out.data_ptr(); a.mode[1] = g1->mode; }
  vlmt_sum_rows(&a, g1 != nullptr ? 2 : 1, rows, cols, cur_stream());
  tick(1);
}
Tensor bias_grad(const Tensor& dy, const Tensor& b, const Target& t) {
  if (dy.size(1) % 8 != 0 || dy.stride(1) != 1 || dy.stride(0) % 8 != 0 || reinterpret_cast<uintptr_t>(dy.data_ptr()) % 16 != 0 ||
      dy.scalar_type() != at::kBFloat16)
    return dy.to(at::kFloat).sum(0).to(b.scalar_type());
  VecGrad g(b, t);
  colsum_into(dy, g.out.data_ptr(), g.mode);
  return g.finish(b, t);
}

// what a function keeps besides tensors
struct Cfg : torch::CustomClassHolder {
  double eps = 0, scale = 0;
  bool offset = false, tanh = false, causal = false, gated = false, add = false;
  bool need[6] = {false, false, false, false, false, false};   // inputs that require a gradient, in argument order
  int64_t n_q = 0, n_kv = 0, D = 0, max_seqlen = 0;
  std::vector<int64_t> shape;
  Target t[4];
  bool want_act = false;   // LnLinear: gelu of the output too, into `act`; GeluLinear takes it from there
  Tensor act;
};
using CfgPtr = c10::intrusive_ptr<Cfg>;
void keep(AutogradContext* ctx, const CfgPtr& c) { ctx->saved_data["cfg"] = c10::IValue::make_capsule(c); }
CfgPtr kept(AutogradContext* ctx) { return c10::static_intrusive_pointer_cast<Cfg>(ctx->saved_data["cfg"].toCapsule()); }
bool wants(const Tensor& t) { return t.defined() && t.requires_grad(); }
// No graph is to be built: gradients are off, and no operand carries a forward-mode tangent (which `Function::apply` refuses and a
// direct call of the kernels would drop).
template <typename... T>
bool no_graph(const T&... operands) {
  if (c10::GradMode::is_enabled()) return false;
  return !((operands.defined() && operands._fw_grad(0).defined()) || ...);
}

// Exceptions of Python hooks on saved tensors (activation checkpointing stops a recomputation with one) keep their type.
template <typename F>
auto guarded(F&& f) -> decltype(f()) {
  try {
    return f();
  } catch (python_error& e) {
    e.restore();
    throw py::error_already_set();
  }
}

// ------------------------------------------------------------------ linear
struct Linear : torch::autograd::Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& b_, CfgPtr c) {
    const Tensor b = get(b_);
    Tensor x2 = rows_of(x), wc = operand(w);
    c->need[0] = wants(x); c->need[1] = wants(w); c->need[2] = wants(b);
    Tensor y = mm(x2, wc, false, false, b);
    c->shape = x.sizes().vec();
    keep(ctx, c);
    ctx->save_for_backward(b.defined() ? variable_list{x2, wc, b} : variable_list{x2, wc});
    if (x.dim() == 2) return y;
    auto out = x.sizes().vec();
    out.back() = w.size(0);
    return y.view(out);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    auto c = kept(ctx);
    const Tensor &x2 = saved[0], &w = saved[1];
    Tensor dy = rows_of(grads[0]), dx, dw, db;
    if (c->need[0]) dx = mm(dy, w, false, true).view(c->shape);
    if (c->need[1]) dw = weight_grad(dy, x2, c->t[0]);
    if (c->need[2]) db = bias_grad(dy, saved[2], c->t[1]);
    return {dx, dw, db, Tensor()};
  }
};
Tensor op_linear(const Tensor& x, const py::object& w_, const py::object& b_) {
  return guarded([&] {
    Tensor w = w_.cast<Tensor>(), b = as_tensor(b_);
    if (no_graph(x, w, b)) {
      Tensor y = mm(rows_of(x), operand(w), false, false, b);
      if (x.dim() == 2) return y;
      auto out = x.sizes().vec();
      out.back() = w.size(0);
      return y.view(out);
    }
    auto c = c10::make_intrusive<Cfg>();
    c->t[0] = target_of(w_); c->t[1] = target_of(b_);
    return Linear::apply(x, w, opt(b), c);
  });
}

// ------------------------------------------------------------------ norm / activation + linear
// (x [+ residual]) -> RMSNorm -> linear, keeping the un-normalised stream and rstd; the normalised rows are made again by the
// norm's backward kernel.  Second output: x + residual.
struct NormLinear : torch::autograd::Function<NormLinear> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const OptTensor& res_, const Tensor& nw, const Tensor& w, CfgPtr c) {
    const Tensor res = get(res_);
    ctx->set_materialize_grads(false);
    Tensor xc = x.contiguous();
    auto r = rmsnorm_fwd(xc, res.defined() ? OptTensor(res.contiguous()) : OptTensor(), nw, c->eps, c->offset);
    Tensor wc = operand(w), y = mm(r[0], wc, false, false);
    tick(1);
    c->need[2] = wants(nw); c->need[3] = wants(w);
    keep(ctx, c);
    ctx->save_for_backward({res.defined() ? r[2] : xc, nw, r[1], wc});
    if (res.defined()) return {y, r[2]};
    return {y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    auto c = kept(ctx);
    const Tensor &r = saved[0], &nw = saved[1], &rstd = saved[2], &w = saved[3];
    Tensor dr = grads.size() > 1 ? grads[1] : Tensor(), dx, dnw, dw;
    if (!grads[0].defined()) {   // only the residual stream was used
      dx = dr;
    } else {
      Tensor dy = rows_of(grads[0]), yn;
      auto b = rmsnorm_bwd_partial(mm(dy, w, false, true), r, nw, rstd, dr.defined() ? OptTensor(dr.contiguous()) : OptTensor(), c->offset,
                                   c->need[3] ? &yn : nullptr);
      dx = b[0];
      tick(1);
      if (c->need[3]) {
        if (!yn.defined()) { yn = rmsnorm_fwd(r, c10::nullopt, nw, c->eps, c->offset)[0]; tick(1); }
        dw = weight_grad(dy, yn, c->t[1]);
        yn.reset();
      }
      if (c->need[2]) {
        VecGrad g(nw, c->t[0]);
        sum_rows(b[1].data_ptr<float>(), nullptr, b[1].size(1), b[1].size(0), b[1].size(1), g, nullptr);
        dnw = g.finish(nw, c->t[0]);
      }
    }
    return {dx, grads.size() > 1 ? dx : Tensor(), dnw, dw, Tensor()};
  }
};
py::object op_norm_linear(const Tensor& x, const py::object& res_, const py::object& nw_, const py::object& w_, double eps, bool offset) {
  return guarded([&]() -> py::object {
    Tensor res = as_tensor(res_), nw = nw_.cast<Tensor>(), w = w_.cast<Tensor>();
    if (no_graph(x, res, nw, w)) {
      auto r = rmsnorm_fwd(x.contiguous(), res.defined() ? OptTensor(res.contiguous()) : OptTensor(), nw, eps, offset);
      tick(1);
      Tensor y = mm(r[0], operand(w), false, false);
      return res.defined() ? py::object(py::make_tuple(y, r[2])) : py::cast(y);
    }
    auto c = c10::make_intrusive<Cfg>();
    c->eps = eps; c->offset = offset;
    c->t[0] = target_of(nw_); c->t[1] = target_of(w_);
    auto out = NormLinear::apply(x, opt(res), nw, w, c);
    return res.defined() ? py::object(py::make_tuple(out[0], out[1])) : py::cast(out[0]);
  });
}

// LayerNorm -> linear, the normalised rows made again by the norm's backward kernel
struct LnLinear : torch::autograd::Function<LnLinear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& lw, const OptTensor& lb_, const Tensor& w, const OptTensor& b_, CfgPtr c) {
    const Tensor lb = get(lb_), b = get(b_);
    Tensor xc = x.contiguous();
    auto r = layernorm_fwd(xc, lw, opt(lb), c->eps);
    Tensor wc = operand(w), y;
    check_storage(wc);
    if (c->want_act && gemm_gelu(r[0], wc, opt(b), c->tanh, &y, c->act)) tick(1);
    else y = mm(r[0], wc, false, false, b);
    tick(1);
    c->need[1] = wants(lw); c->need[2] = wants(lb); c->need[3] = wants(w); c->need[4] = wants(b);
    keep(ctx, c);
    variable_list s{xc, lw, r[1], r[2], wc};
    c->n_q = lb.defined(); c->n_kv = b.defined();
    if (lb.defined()) s.push_back(lb);
    if (b.defined()) s.push_back(b);
    ctx->save_for_backward(s);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    auto c = kept(ctx);
    const Tensor &x = saved[0], &lw = saved[1], &mean = saved[2], &rstd = saved[3], &w = saved[4];
    Tensor lb = c->n_q ? saved[5] : Tensor(), b = c->n_kv ? saved[5 + c->n_q] : Tensor();
    Tensor dy = rows_of(grads[0]), yn, dlw, dlb, dw, db;
    auto r = layernorm_bwd_partial(mm(dy, w, false, true), x, lw, mean, rstd, opt(lb), c->need[3] ? &yn : nullptr);
    tick(1);
    if (c->need[3]) {
      if (!yn.defined()) { yn = layernorm_fwd(x, lw, opt(lb), c->eps)[0]; tick(1); }
      dw = weight_grad(dy, yn, c->t[2]);
      yn.reset();
    }
    if (c->need[1] || c->need[2]) {
      VecGrad gw(lw, c->need[1] ? c->t[0] : Target());
      const int rows = r[1].size(0), cols = r[1].size(1);
      if (lb.defined() && c->need[2]) {
        VecGrad gb(lb, c->t[1]);
        sum_rows(r[1].data_ptr<float>(), r[2].data_ptr<float>(), cols, rows, cols, gw, &gb);
        dlb = gb.finish(lb, c->t[1]);
      } else {
        sum_rows(r[1].data_ptr<float>(), nullptr, cols, rows, cols, gw, nullptr);
      }
      if (c->need[1]) dlw = gw.finish(lw, c->t[0]);
    }
    if (c->need[4]) db = bias_grad(dy, b, c->t[3]);
    return {r[0], dlw, dlb, dw, db, Tensor()};
  }
};
// gelu_kind: 0 no activation, 1 gelu(output) in `act` too, 2 the tanh form of it; undefined where the sizes have no such kernel.  Without a graph the
// output itself is undefined where `act` is not.
Tensor ln_linear(const Tensor& x, const py::object& lw_, const py::object& lb_, const py::object& w_, const py::object& b_, double eps, int gelu_kind,
                 Tensor* act) {
  return guarded([&] {
    Tensor lw = lw_.cast<Tensor>(), lb = as_tensor(lb_), w = w_.cast<Tensor>(), b = as_tensor(b_);
    if (no_graph(x, lw, lb, w, b)) {
      tick(1);
      Tensor h = layernorm_fwd(x.contiguous(), lw, opt(lb), eps)[0], wc = operand(w);
      check_storage(wc);
      if (gelu_kind != 0 && gemm_gelu(h, wc, opt(b), gelu_kind == 2, nullptr, *act)) {
        tick(1);
        return Tensor();
      }
      return mm(h, wc, false, false, b);
    }
    auto c = c10::make_intrusive<Cfg>();
    c->eps = eps;
    c->want_act = gelu_kind != 0; c->tanh = gelu_kind == 2;
    c->t[0] = target_of(lw_); c->t[1] = target_of(lb_); c->t[2] = target_of(w_); c->t[3] = target_of(b_);
    Tensor y = LnLinear::apply(x, lw, opt(lb), w, opt(b), c);
    if (act != nullptr) *act = std::move(c->act);
    return y;
  });
}
Tensor op_ln_linear(const Tensor& x, const py::object& lw_, const py::object& lb_, const py::object& w_, const py::object& b_, double eps) {
  return ln_linear(x, lw_, lb_, w_, b_, eps, 0, nullptr);
}

// gelu(pre) -> linear, only `pre` is kept
struct GeluLinear : torch::autograd::Function<GeluLinear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& pre, const Tensor& w, const OptTensor& b_, CfgPtr c) {
    const Tensor b = get(b_);
    Tensor pc = pre.contiguous(), wc = operand(w);
    Tensor act = std::move(c->act);
    if (!act.defined()) { act = gelu_fwd(pc, c->tanh); tick(1); }
    Tensor y = mm(act, wc, false, false, b);
    c->need[1] = wants(w); c->need[2] = wants(b);
    keep(ctx, c);
    ctx->save_for_backward(b.defined() ? variable_list{pc, wc, b} : variable_list{pc, wc});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    auto c = kept(ctx);
    const Tensor &pre = saved[0], &w = saved[1];
    Tensor dy = rows_of(grads[0]), dw, db;
    Tensor act, dpre;
    check_storage(w);
    if (!gemm_gelu_bwd(dy, w, pre, c->tanh, dpre, c->need[1] ? &act : nullptr))
      dpre = gelu_bwd(mm(dy, w, false, true), pre, c->tanh, c->need[1] ? &act : nullptr);
    tick(1);
    if (c->need[1]) dw = weight_grad(dy, act, c->t[0]);
    if (c->need[2]) db = bias_grad(dy, saved[2], c->t[1]);
    return {dpre, dw, db, Tensor()};
  }
};
// `act`: gelu(pre) where its kernel has made it
Tensor gelu_linear(const Tensor& pre, const py::object& w_, const py::object& b_, bool tanh_approx, Tensor act) {
  return guarded([&] {
    Tensor w = w_.cast<Tensor>(), b = as_tensor(b_);
    if (no_graph(pre, w, b)) {
      if (!act.defined()) { act = gelu_fwd(pre.contiguous(), tanh_approx); tick(1); }
      return mm(act, operand(w), false, false, b);
    }
    auto c = c10::make_intrusive<Cfg>();
    c->tanh = tanh_approx;
    c->act = std::move(act);
    c->t[0] = target_of(w_); c->t[1] = target_of(b_);
    return GeluLinear::apply(pre, w, opt(b), c);
  });
}
Tensor op_gelu_linear(const Tensor& pre, const py::object& w_, const py::object& b_, bool tanh_approx) {
  return gelu_linear(pre, w_, b_, tanh_approx, Tensor());
}

// Gradient of [gate, up] behind y = (silu(gate) * up) w^T; h (or null) gets silu(gate) * up.
Tensor glu_grad(const Tensor& dy, const Tensor& w, const Tensor& gu, Tensor* h) {
  check_storage(w);
  Tensor dgu;
  if (!gemm_glu_bwd(dy, w, gu, dgu, h)) dgu = swiglu_bwd(mm(dy, w, false, true), gu, h);
  tick(1);
  return dgu;
}
// silu(gate) * up -> linear for a fused [T, 2 I] input, only the input is kept
struct SwigluLinear : torch::autograd::Function<SwigluLinear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& gu, const Tensor& w, CfgPtr c) {
    Tensor g = gu.contiguous(), wc = operand(w);
    Tensor y = mm(swiglu_fwd(g), wc, false, false);
    tick(1);
    c->need[1] = wants(w);
    keep(ctx, c);
    ctx->save_for_backward({g, wc});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    auto c = kept(ctx);
    Tensor dy = rows_of(grads[0]), dw;
    Tensor h, dgu = glu_grad(dy, saved[1], saved[0], c->need[1] ? &h : nullptr);
    if (c->need[1]) dw = weight_grad(dy, h, c->t[0]);
    return {dgu, dw, Tensor()};
  }
};
Tensor op_swiglu_linear(const Tensor& gu, const py::object& w_) {
  return guarded([&] {
    Tensor w = w_.cast<Tensor>();
    if (no_graph(gu, w)) {
      tick(1);
      return mm(swiglu_fwd(gu.contiguous()), operand(w), false, false);
    }
    auto c = c10::make_intrusive<Cfg>();
    c->t[0] = target_of(w_);
    return SwigluLinear::apply(gu, w, c);
  });
}

// x + residual -> RMSNorm -> gate / up -> silu(gate) * up -> down: the two functions above with the activation made by the gate / up product's kernel
// where the sizes have one.  Second output: x + residual.
struct NormMlp : torch::autograd::Function<NormMlp> {
  // out, x + residual, rstd, gate and up (undefined where they are not kept)
  static std::array<Tensor, 4> run(const Tensor& x, const Tensor& res, const Tensor& nw, const Tensor& wgu, const Tensor& wd, const Cfg& c, bool keep_gu) {
    auto r = rmsnorm_fwd(x.contiguous(), OptTensor(res.contiguous()), nw, c.eps, c.offset);
    check_storage(wgu);
    Tensor gu, act;
    if (gemm_glu(r[0], wgu, keep_gu ? &gu : nullptr, act)) {
      tick(1);
    } else {
      gu = mm(r[0], wgu, false, false);
      act = swiglu_fwd(gu);
      tick(1);
    }
    tick(1);
    r[0].reset();
    return {mm(act, wd, false, false), r[2], r[1], gu};
  }
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& res, const Tensor& nw, const Tensor& wgu_, const Tensor& wd_, CfgPtr c) {
    ctx->set_materialize_grads(false);
    Tensor wgu = operand(wgu_), wd = operand(wd_);
    auto r = run(x, res, nw, wgu, wd, *c, true);
    c->need[2] = wants(nw); c->need[3] = wants(wgu_); c->need[4] = wants(wd_);
    keep(ctx, c);
    ctx->save_for_backward({r[1], nw, r[2], wgu, r[3], wd});
    return {r[0], r[1]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto s = ctx->get_saved_variables();
    auto c = kept(ctx);
    const Tensor &r = s[0], &nw = s[1], &rstd = s[2], &wgu = s[3], &gu = s[4], &wd = s[5];
    Tensor dr = grads[1], dx, dnw, dwgu, dwd;
    if (!grads[0].defined()) {   // only the residual stream was used
      dx = dr;
    } else {
      Tensor dy = rows_of(grads[0]), h, yn;
      Tensor dgu = glu_grad(dy, wd, gu, c->need[4] ? &h : nullptr);
      if (c->need[4]) dwd = weight_grad(dy, h, c->t[2]);
      h.reset();
      auto b = rmsnorm_bwd_partial(mm(dgu, wgu, false, true), r, nw, rstd, dr.defined() ? OptTensor(dr.contiguous()) : OptTensor(), c->offset,
                                   c->need[3] ? &yn : nullptr);
      dx = b[0];
      tick(1);
      if (c->need[3]) {
        if (!yn.defined()) { yn = rmsnorm_fwd(r, c10::nullopt, nw, c->eps, c->offset)[0]; tick(1); }
        dwgu = weight_grad(dgu, yn, c->t[1]);
        yn.reset();
      }
      if (c->need[2]) {
        VecGrad g(nw, c->t[0]);
        sum_rows(b[1].data_ptr<float>(), nullptr, b[1].size(1), b[1].size(0), b[1].size(1), g, nullptr);
        dnw = g.finish(nw, c->t[0]);
      }
    }
    return {dx, dx, dnw, dwgu, dwd, Tensor()};
  }
};
std::array<Tensor, 2> norm_mlp(const Tensor& x, const Tensor& res, const py::object& nw_, const py::object& wgu_, const py::object& wd_, double eps, bool offset) {
  return guarded([&]() -> std::array<Tensor, 2> {
    Tensor nw = nw_.cast<Tensor>(), wgu = wgu_.cast<Tensor>(), wd = wd_.cast<Tensor>();
    auto c = c10::make_intrusive<Cfg>();
    c->eps = eps; c->offset = offset;
    if (no_graph(x, res, nw, wgu, wd)) {
      auto r = NormMlp::run(x, res, nw, operand(wgu), operand(wd), *c, false);
      return {r[0], r[1]};
    }
    c->t[0] = target_of(nw_); c->t[1] = target_of(wgu_); c->t[2] = target_of(wd_);
    auto out = NormMlp::apply(x, res, nw, wgu, wd, c);
    return {out[0], out[1]};
  });
}

// ------------------------------------------------------------------ norms
struct RmsNorm : torch::autograd::Function<RmsNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const OptTensor& res_, const Tensor& w, CfgPtr c) {
    const Tensor res = get(res_);
    ctx->set_materialize_grads(false);
    Tensor xc = x.contiguous();
    auto r = rmsnorm_fwd(xc, res.defined() ? OptTensor(res.contiguous()) : OptTensor(), w, c->eps, c->offset);
    tick(1);
    c->need[2] = wants(w);
    keep(ctx, c);
    ctx->save_for_backward({res.defined() ? r[2] : xc, w, r[1]});
    if (res.defined()) return {r[0], r[2]};
    return {r[0]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    auto c = kept(ctx);
    Tensor dr = grads.size() > 1 ? grads[1] : Tensor(), dx, dw;
    if (!grads[0].defined()) {
      dx = dr;
    } else {
      auto b = rmsnorm_bwd_partial(grads[0].contiguous(), saved[0], saved[1], saved[2], dr.defined() ? OptTensor(dr.contiguous()) : OptTensor(),
                                   c->offset);
      dx = b[0];
      tick(1);
      if (c->need[2]) {
        VecGrad g(saved[1], c->t[0]);
        sum_rows(b[1].data_ptr<float>(), nullptr, b[1].size(1), b[1].size(0), b[1].size(1), g, nullptr);
        dw = g.finish(saved[1], c->t[0]);
      }
    }
    return {dx, grads.size() > 1 ? dx : Tensor(), dw, Tensor()};
  }
};
py::object op_rms_norm(const Tensor& x, const py::object& res_, const py::object& w_, double eps, bool offset) {
  return guarded([&]() -> py::object {
    Tensor res = as_tensor(res_), w = w_.cast<Tensor>();
    variable_list out;
    if (no_graph(x, res, w)) {
      auto r = rmsnorm_fwd(x.contiguous(), res.defined() ? OptTensor(res.contiguous()) : OptTensor(), w, eps, offset);
      tick(1);
      out = res.defined() ? variable_list{r[0], r[2]} : variable_list{r[0]};
    } else {
      auto c = c10::make_intrusive<Cfg>();
      c->eps = eps; c->offset = offset;
      c->t[0] = target_of(w_);
      out = RmsNorm::apply(x, opt(res), w, c);
    }
    return res.defined() ? py::object(py::make_tuple(out[0], out[1])) : py::cast(out[0]);
  });
}

struct LayerNorm : torch::autograd::Function<LayerNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& b_, CfgPtr c) {
    const Tensor b = get(b_);
    Tensor xc = x.contiguous();
    auto r = layernorm_fwd(xc, w, opt(b), c->eps);
    tick(1);
    c->need[1] = wants(w); c->need[2] = wants(b);
    keep(ctx, c);
    ctx->save_for_backward(b.defined() ? variable_list{xc, w, r[1], r[2], b} : variable_list{xc, w, r[1], r[2]});
    return r[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    auto c = kept(ctx);
    auto r = layernorm_bwd_partial(grads[0].contiguous(), saved[0], saved[1], saved[2], saved[3]);
    tick(1);
    Tensor dw, db;
    if (c->need[1] || c->need[2]) {
      VecGrad gw(saved[1], c->need[1] ? c->t[0] : Target());
      const int rows = r[1].size(0), cols = r[1].size(1);
      if (c->need[2]) {
        VecGrad gb(saved[4], c->t[1]);
        sum_rows(r[1].data_ptr<float>(), r[2].data_ptr<float>(), cols, rows, cols, gw, &gb);
        db = gb.finish(saved[4], c->t[1]);
      } else {
        sum_rows(r[1].data_ptr<float>(), nullptr, cols, rows, cols, gw, nullptr);
      }
      if (c->need[1]) dw = gw.finish(saved[1], c->t[0]);
    }
    return {r[0], dw, db, Tensor()};
  }
};
Tensor op_layer_norm(const Tensor& x, const py::object& w_, const py::object& b_, double eps) {
  return guarded([&] {
    Tensor w = w_.cast<Tensor>(), b = as_tensor(b_);
    if (no_graph(x, w, b)) {
      tick(1);
      return layernorm_fwd(x.contiguous(), w, opt(b), eps)[0];
    }
    auto c = c10::make_intrusive<Cfg>();
    c->eps = eps;
    c->t[0] = target_of(w_); c->t[1] = target_of(b_);
    return LayerNorm::apply(x, w, opt(b), c);
  });
}

struct GatedRmsNorm : torch::autograd::Function<GatedRmsNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& z, const Tensor& w, CfgPtr c) {
    Tensor xc = x.contiguous(), zc = z.contiguous();
    auto r = rmsnorm_gated_fwd(xc, zc, w, c->eps);
    tick(1);
    c->need[2] = wants(w);
    keep(ctx, c);
    ctx->save_for_backward({xc, zc, w, r[1]});
    return r[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    auto c = kept(ctx);
    auto r = rmsnorm_gated_bwd_partial(grads[0].contiguous(), saved[0], saved[1], saved[2], saved[3]);
    tick(1);
    Tensor dw;
    if (c->need[2]) {
      VecGrad g(saved[2], c->t[0]);
      sum_rows(r[2].data_ptr<float>(), nullptr, r[2].size(1), r[2].size(0), r[2].size(1), g, nullptr);
      dw = g.finish(saved[2], c->t[0]);
    }
    return {r[0], r[1], dw, Tensor()};
  }
};
Tensor op_rms_norm_gated(const Tensor& x, const Tensor& z, const py::object& w_, double eps) {
  return guarded([&] {
    Tensor w = w_.cast<Tensor>();
    if (no_graph(x, z, w)) {
      tick(1);
      return rmsnorm_gated_fwd(x.contiguous(), z.contiguous(), w, eps)[0];
    }
    auto c = c10::make_intrusive<Cfg>();
    c->eps = eps;
    c->t[0] = target_of(w_);
    return GatedRmsNorm::apply(x, z, w, c);
  });
}

// ------------------------------------------------------------------ activations
struct Swiglu : torch::autograd::Function<Swiglu> {
  static Tensor forward(AutogradContext* ctx, const Tensor& gu) {
    Tensor g = gu.contiguous();
    ctx->save_for_backward({g});
    tick(1);
    return swiglu_fwd(g);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    tick(1);
    return {swiglu_bwd(grads[0].contiguous(), ctx->get_saved_variables()[0])};
  }
};
struct SigmoidMul : torch::autograd::Function<SigmoidMul> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& gate) {
    Tensor xc = x.contiguous(), gc = gate.contiguous();
    ctx->save_for_backward({xc, gc});
    tick(1);
    return sigmoid_mul_fwd(xc, gc);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    tick(1);
    auto r = sigmoid_mul_bwd(grads[0].contiguous(), saved[0], saved[1]);
    return {r[0], r[1]};
  }
};
struct Gelu : torch::autograd::Function<Gelu> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, bool tanh_approx) {
    Tensor xc = x.contiguous();
    ctx->save_for_backward({xc});
    ctx->saved_data["tanh"] = tanh_approx;
    tick(1);
    return gelu_fwd(xc, tanh_approx);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    tick(1);
    return {gelu_bwd(grads[0].contiguous(), ctx->get_saved_variables()[0], ctx->saved_data["tanh"].toBool()), Tensor()};
  }
};

// ------------------------------------------------------------------ attention inputs
struct QkvNormRope : torch::autograd::Function<QkvNormRope> {
  static variable_list forward(AutogradContext* ctx, const Tensor& qkv, const OptTensor& qw_, const OptTensor& kw_, const Tensor& cosv, const Tensor& sinv,
                               CfgPtr c) {
    const Tensor qw = get(qw_), kw = get(kw_);
    Tensor x = qkv.contiguous();
    auto r = qkv_norm_rope_fwd(x, c->n_q, c->n_kv, c->D, opt(qw), opt(kw), cosv, sinv, c->eps, c->offset, c->gated);
    tick(1);
    c->need[1] = wants(qw); c->need[2] = wants(kw);
    keep(ctx, c);
    ctx->save_for_backward(qw.defined() ? variable_list{x, cosv, sinv, r[3], qw, kw} : variable_list{x, cosv, sinv, r[3]});
    if (c->gated) return {r[0], r[1], r[2], r[4]};
    return {r[0], r[1], r[2]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    auto c = kept(ctx);
    Tensor qw = saved.size() > 4 ? saved[4] : Tensor(), kw = saved.size() > 4 ? saved[5] : Tensor(), dqw, dkw;
    auto r = qkv_norm_rope_bwd_partial(grads[0].contiguous(), grads[1].contiguous(), grads[2].contiguous(),
                                       c->gated ? OptTensor(grads[3].contiguous()) : OptTensor(), saved[0], opt(qw), opt(kw), saved[1], saved[2],
                                       saved[3], c->n_q, c->n_kv, c->D, c->offset, c->gated);
    tick(1);
    if (c->need[1] || c->need[2]) {
      VecGrad gq(qw, c->need[1] ? c->t[0] : Target()), gk(kw, c->need[2] ? c->t[1] : Target());
      const float* p = r[1].data_ptr<float>();   // [blocks, 2, D]
      sum_rows(p, p + c->D, 2 * c->D, r[1].size(0), c->D, gq, &gk);
      if (c->need[1]) dqw = gq.finish(qw, c->t[0]);
      if (c->need[2]) dkw = gk.finish(kw, c->t[1]);
    }
    return {r[0], dqw, dkw, Tensor(), Tensor(), Tensor()};
  }
};
py::tuple op_qkv_norm_rope(const Tensor& qkv, const py::object& qw_, const py::object& kw_, const Tensor& cosv, const Tensor& sinv, int64_t n_q,
                           int64_t n_kv, int64_t D, double eps, bool offset, bool gated) {
  return guarded([&]() -> py::tuple {
    Tensor qw = as_tensor(qw_), kw = as_tensor(kw_);
    if (no_graph(qkv, qw, kw, cosv, sinv)) {
      auto r = qkv_norm_rope_fwd(qkv.contiguous(), n_q, n_kv, D, opt(qw), opt(kw), cosv, sinv, eps, offset, gated);
      tick(1);
      return py::make_tuple(r[0], r[1], r[2], gated ? py::cast(r[4]) : py::object(py::none()));
    }
    auto c = c10::make_intrusive<Cfg>();
    c->n_q = n_q; c->n_kv = n_kv; c->D = D; c->eps = eps; c->offset = offset; c->gated = gated;
    c->t[0] = target_of(qw_); c->t[1] = target_of(kw_);
    auto out = QkvNormRope::apply(qkv, opt(qw), opt(kw), cosv, sinv, c);
    return py::make_tuple(out[0], out[1], out[2], gated ? py::cast(out[3]) : py::object(py::none()));
  });
}

struct Rope : torch::autograd::Function<Rope> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& cosv, const Tensor& sinv, int64_t d_out) {
    ctx->save_for_backward({cosv, sinv});
    ctx->saved_data["d"] = x.size(-1);
    tick(1);
    return rope_generic(x, cosv, sinv, false, d_out);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    const int64_t d = ctx->saved_data["d"].toInt();
    tick(1);
    return {rope_generic(grads[0].stride(-1) == 1 ? grads[0].narrow(-1, 0, d) : grads[0].narrow(-1, 0, d).contiguous(), saved[0], saved[1], true, d),
            Tensor(), Tensor(), Tensor()};
  }
};
Tensor op_rope(const Tensor& x, const Tensor& cosv, const Tensor& sinv, int64_t d_out) {
  return guarded([&] {
    if (no_graph(x, cosv, sinv)) {
      tick(1);
      return rope_generic(x, cosv, sinv, false, d_out);
    }
    return Rope::apply(x, cosv, sinv, d_out);
  });
}

// ------------------------------------------------------------------ attention
// [T, H, d] as the kernels' tensor maps can read it: unit channel stride, 16-byte aligned head and token strides and base (a
// slice of a fused projection qualifies); anything else is copied.
Tensor heads_in_place(const Tensor& t) {
  if (t.stride(2) == 1 && t.stride(1) % 8 == 0 && t.stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0) return t;
  return t.contiguous();
}
struct Attention : torch::autograd::Function<Attention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& cu, CfgPtr c) {
    Tensor q = heads_in_place(q_), k = heads_in_place(k_), v = heads_in_place(v_);
    auto r = attn_fwd(q, k, v, cu, c->max_seqlen, c->causal, c->scale);
    tick(1);
    keep(ctx, c);
    ctx->save_for_backward({q, k, v, r[0], r[1], cu});
    return r[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto s = ctx->get_saved_variables();
    auto c = kept(ctx);
    auto r = attn_bwd(grads[0].contiguous(), s[0], s[1], s[2], s[3], s[4], s[5], c->max_seqlen, c->causal, c->scale);
    tick(3);
    return {r[0], r[1], r[2], Tensor(), Tensor()};
  }
};
Tensor op_attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu, int64_t max_seqlen, bool causal, double scale) {
  return guarded([&] {
    if (no_graph(q, k, v)) {
      tick(1);
      return attn_fwd(heads_in_place(q), heads_in_place(k), heads_in_place(v), cu, max_seqlen, causal, scale)[0];
    }
    auto c = c10::make_intrusive<Cfg>();
    c->max_seqlen = max_seqlen; c->causal = causal; c->scale = scale;
    return Attention::apply(q, k, v, cu, c);
  });
}

// Bidirectional attention over a fused projection [S, 3 H D]: rotary on q and k, v read in place, and one gradient for the whole projection
// instead of three that autograd would put together.
struct RopeAttention : torch::autograd::Function<RopeAttention> {
  static std::vector<Tensor> run(const Tensor& x, const Tensor& cosv, const Tensor& sinv, const Tensor& cu, const CfgPtr& c) {
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t S = x.size(0), H = c->n_q, D = c->D;
    Tensor q = torch::empty({S, H, D}, x.options()), k = torch::empty_like(q);
    vlmt_rope_qkv_fwd(x.data_ptr(), x.stride(0), cosv.data_ptr<float>(), sinv.data_ptr<float>(), q.data_ptr(), k.data_ptr(), (int)S, (int)H, (int)D,
                      cur_stream());
    auto r = attn_fwd(q, k, x.view({S, 3, H, D}).select(1, 2), cu, c->max_seqlen, false, c->scale);
    tick(2);
    return {q, k, r[0], r[1]};
  }
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const Tensor& cosv, const Tensor& sinv, const Tensor& cu, CfgPtr c) {
    Tensor x = qkv.contiguous();
    auto r = run(x, cosv, sinv, cu, c);
    keep(ctx, c);
    ctx->save_for_backward({x, cosv, sinv, cu, r[0], r[1], r[2], r[3]});
    return r[2];
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto s = ctx->get_saved_variables();
    auto c = kept(ctx);
    const int64_t S = s[0].size(0), H = c->n_q, D = c->D;
    auto r = attn_bwd(grads[0].contiguous(), s[4], s[5], s[0].view({S, 3, H, D}).select(1, 2), s[6], s[7], s[3], c->max_seqlen, false, c->scale);
    c10::cuda::CUDAGuard guard(s[0].device());
    Tensor dqkv = torch::empty_like(s[0]);
    vlmt_rope_qkv_bwd(r[0].data_ptr(), r[1].data_ptr(), r[2].data_ptr(), s[1].data_ptr<float>(), s[2].data_ptr<float>(), dqkv.data_ptr(), (int)S, (int)H,
                      (int)D, cur_stream());
    tick(4);
    return {dqkv, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};
Tensor rope_attention(const Tensor& qkv, const Tensor& cosv, const Tensor& sinv, const Tensor& cu, int64_t max_seqlen, int64_t H, int64_t D, double scale) {
  return guarded([&] {
    auto c = c10::make_intrusive<Cfg>();
    c->max_seqlen = max_seqlen; c->scale = scale; c->n_q = H; c->D = D;
    if (no_graph(qkv, cosv, sinv)) return RopeAttention::run(qkv.contiguous(), cosv, sinv, cu, c)[2];
    return RopeAttention::apply(qkv, cosv, sinv, cu, c);
  });
}

// ------------------------------------------------------------------ rows of a packed sequence
struct RowsUpdate : torch::autograd::Function<RowsUpdate> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& index, const Tensor& src, bool add) {
    Tensor out = x.clone();
    rows_update(out, index, src.contiguous().to(x.scalar_type()), add);
    ctx->save_for_backward({index});
    ctx->saved_data["add"] = add;
    tick(1);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    Tensor index = ctx->get_saved_variables()[0], dout = grads[0].contiguous();
    Tensor dsrc = rows_gather(dout, index);
    tick(1);
    if (ctx->saved_data["add"].toBool()) return {dout, Tensor(), dsrc, Tensor()};
    Tensor dx = dout.clone();
    rows_update(dx, index, torch::zeros_like(dsrc), false);
    tick(1);
    return {dx, Tensor(), dsrc, Tensor()};
  }
};

// ------------------------------------------------------------------ vision tower: interpolated position embedding, tables
struct PosEmbed : torch::autograd::Function<PosEmbed> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& table, const Tensor& index, const Tensor& weight, const Tensor& images,
                        CfgPtr c) {
    c10::cuda::CUDAGuard guard(x.device());
    Tensor xc = x.contiguous(), out = torch::empty_like(xc);
    vlmt_pos_embed_fwd(xc.data_ptr(), table.data_ptr(), index.data_ptr<int64_t>(), weight.data_ptr<float>(), out.data_ptr(), x.size(0), x.size(1),
                       cur_stream());
    tick(1);
    c->need[1] = wants(table);
    keep(ctx, c);
    ctx->save_for_backward({table, images});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto saved = ctx->get_saved_variables();
    auto c = kept(ctx);
    c10::cuda::CUDAGuard guard(grads[0].device());
    Tensor dy = grads[0].contiguous(), dt;
    if (reinterpret_cast<uintptr_t>(dy.data_ptr()) % 16) dy = dy.clone();
    if (c->need[1]) {
      const Tensor& table = saved[0];
      Tensor g = may_add(c->t[0]) ? c->t[0]->param.grad() : Tensor();
      const bool in_place = g.defined() && g.scalar_type() == at::kBFloat16 && g.is_contiguous() && g.sizes() == table.sizes() &&
                            reinterpret_cast<uintptr_t>(g.data_ptr()) % 16 == 0;
      if (in_place) check_storage(g);
      Tensor out = in_place ? g : torch::empty_like(table);
      vlmt_pos_embed_bwd(dy.data_ptr(), saved[1].data_ptr<int>(), (int)saved[1].size(0), (int)c->n_q, (int)c->n_kv, dy.size(0), out.data_ptr(),
                         in_place, (int)table.size(1), cur_stream());
      tick(1);
      if (in_place) c->t[0]->report(); else dt = out;
    }
    return {dy, dt, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};
Tensor op_pos_embed(const Tensor& x, const py::object& table_, const Tensor& index, const Tensor& weight, const Tensor& images, int64_t side,
                    int64_t merge) {
  Tensor table = table_.cast<Tensor>();
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.size(1) % 8 == 0 && table.scalar_type() == at::kBFloat16 &&
              table.is_contiguous() && table.dim() == 2 && table.size(0) == side * side && table.size(1) == x.size(1), "op_pos_embed: bad operands");
  TORCH_CHECK(index.scalar_type() == at::kLong && index.is_contiguous() && index.dim() == 2 && index.size(0) == 4 && index.size(1) == x.size(0) &&
              weight.scalar_type() == at::kFloat && weight.is_contiguous() && weight.sizes() == index.sizes() && images.scalar_type() == at::kInt &&
              images.is_contiguous() && images.dim() == 2 && images.size(1) == 4, "op_pos_embed: bad plan");
  return guarded([&] {
    auto c = c10::make_intrusive<Cfg>();
    c->n_q = side; c->n_kv = merge;
    c->t[0] = target_of(table_);
    return PosEmbed::apply(x, table, index, weight, images, c);
  });
}

std::vector<Tensor> rope_tables(const Tensor& pos, const Tensor& inv_freq, int64_t sec1, int64_t sec2) {
  TORCH_CHECK(pos.is_cuda() && pos.scalar_type() == at::kLong && pos.is_contiguous() && pos.dim() == 2 && (pos.size(0) == 1 || pos.size(0) == 3) &&
              inv_freq.scalar_type() == at::kFloat && inv_freq.is_contiguous() && inv_freq.is_cuda(), "rope_tables: positions int64 [1 or 3, T]");
  c10::cuda::CUDAGuard guard(pos.device());
  const int64_t T = pos.size(1), n = inv_freq.numel();
  Tensor cs = torch::empty({2, T, 2 * n}, inv_freq.options());
  Tensor c = cs[0], s = cs[1];
  vlmt_rope_tables(pos.data_ptr<int64_t>(), (int)pos.size(0), inv_freq.data_ptr<float>(), (int)n, (int)sec1, (int)sec2, T, c.data_ptr<float>(),
                   s.data_ptr<float>(), cur_stream());
  tick(1);
  return {c, s};
}

// ------------------------------------------------------------------ embedding
// Rows of a table; the gradient of a tagged table is added to .grad row by row (loss_optim.cu) instead of as a dense tensor of the table's size.
struct Embedding : torch::autograd::Function<Embedding> {
  static Tensor forward(AutogradContext* ctx, const Tensor& ids, const Tensor& w, CfgPtr c) {
    c->n_q = w.size(0);
    keep(ctx, c);
    ctx->save_for_backward({ids});
    return at::embedding(w, ids);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto c = kept(ctx);
    Tensor ids = ctx->get_saved_variables()[0], dy = grads[0];
    if (may_add(c->t[0])) {
      Tensor g = c->t[0]->param.grad();
      if (g.defined() && g.scalar_type() == at::kBFloat16 && dy.scalar_type() == at::kBFloat16 && g.dim() == 2 && g.size(0) == c->n_q &&
          g.size(1) == dy.size(-1) && g.is_contiguous() && g.size(1) % 8 == 0 && reinterpret_cast<uintptr_t>(g.data_ptr()) % 16 == 0) {
        check_storage(g);
        c10::cuda::CUDAGuard guard(g.device());
        const int64_t T = ids.numel(), D = g.size(1);
        Tensor rows = dy.contiguous().view({T, D});
        if (reinterpret_cast<uintptr_t>(rows.data_ptr()) % 16 != 0) rows = rows.clone();
        auto sorted = ids.reshape({-1}).sort(/*stable=*/true, 0, false);
        Tensor part = torch::empty({vlmt_embed_blocks((int)T), 2, D}, g.options().dtype(at::kFloat));
        const int r = vlmt_embed_bwd(rows.data_ptr(), std::get<0>(sorted).data_ptr<int64_t>(), std::get<1>(sorted).data_ptr<int64_t>(), (int)T, (int)D,
                                     g.data_ptr(), part.data_ptr<float>(), cur_stream());
        TORCH_CHECK(r == 0, "vlmt_embed_bwd failed with code ", r);
        tick(2);
        c->t[0]->report();
        return {Tensor(), Tensor(), Tensor()};
      }
    }
    return {Tensor(), at::embedding_dense_backward(dy, ids, c->n_q, -1, false), Tensor()};
  }
};
Tensor op_embedding(const Tensor& ids, const py::object& w_) {
  return guarded([&] {
    Tensor w = w_.cast<Tensor>();
    if (no_graph(w)) return at::embedding(w, ids);
    auto c = c10::make_intrusive<Cfg>();
    c->t[0] = target_of(w_);
    if (!c->t[0] || !w.requires_grad()) return at::embedding(w, ids);   // autograd's own
    return Embedding::apply(ids, w, c);
  });
}

// ------------------------------------------------------------------ whole blocks
// A decoder layer and the blocks of the vision tower as one binding call each: the functions above in the order in which the modules call them one by
// one, so graph, gradients and results are the same; what is saved is the interpreter between them (a step of the smallest vision model, bound by the
// host: forward 1.95 -> 1.6 ms of it, the pass 4.3 -> 3.85; a 37-token chat through four layers 632 -> 504 us of host).  None where a weight does not take the plain bf16 path: the modules then go their own way.
bool plain_weight(const py::object& w, int64_t in) {
  static PyObject* k_fp8 = PyUnicode_InternFromString("_vlmt_fp8");
  static PyObject* k_sharded = PyUnicode_InternFromString("_vlmt_resharded");
  if (!THPVariable_Check(w.ptr())) return false;
  const Tensor& t = THPVariable_Unpack(w.ptr());
  if (!t.is_cuda() || t.scalar_type() != at::kBFloat16 || t.dim() != 2 || t.size(0) < 16 || t.size(0) % 8 != 0 || t.size(1) % 8 != 0 || t.size(1) != in) return false;
  py::object dict = py::reinterpret_steal<py::object>(PyObject_GenericGetDict(w.ptr(), nullptr));
  if (!dict) { PyErr_Clear(); return true; }
  for (PyObject* key : {k_fp8, k_sharded}) {
    PyObject* flag = PyDict_GetItemWithError(dict.ptr(), key);
    if (flag != nullptr && PyObject_IsTrue(flag) != 0) return false;
  }
  return true;
}
bool plain_vector(const py::object& w, int64_t n, bool optional = false) {
  if (w.is_none()) return optional;
  if (!THPVariable_Check(w.ptr())) return false;
  const Tensor& t = THPVariable_Unpack(w.ptr());
  return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 1 && t.size(0) == n;
}
bool plain_rows(const Tensor& x) { return x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.size(0) > 0 && x.size(1) % 8 == 0; }
bool plain_table(const Tensor& t) { return t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
bool plain_heads(int64_t D) { return D == 256 || (D <= 128 && D % 8 == 0); }

py::object op_decoder_layer(const Tensor& x, const py::tuple& w, const Tensor& cosv, const Tensor& sinv, const Tensor& cu, int64_t max_seqlen, int64_t n_q,
                            int64_t n_kv, int64_t D, double eps1, double eps2, double eps_qk, bool offset1, bool offset2, bool offset_qk, bool gated,
                            double scale) {
  const py::object norm1 = w[0], w_qkv = w[1], q_norm = w[2], k_norm = w[3], w_o = w[4], norm2 = w[5], w_gu = w[6], w_down = w[7];
  const int64_t H = plain_rows(x) ? x.size(1) : 0;
  if (H == 0 || !plain_heads(D) || !plain_table(cosv) || !plain_table(sinv) || cu.scalar_type() != at::kInt || !plain_vector(norm1, H) ||
      !plain_vector(norm2, H) || !plain_vector(q_norm, D) || !plain_vector(k_norm, D) || !plain_weight(w_qkv, H) || !plain_weight(w_o, n_q * D) ||
      !plain_weight(w_gu, H))
    return py::none();
  const int64_t inter = THPVariable_Unpack(w_gu.ptr()).size(0) / 2;
  if (inter % 8 != 0 || !plain_weight(w_down, inter)) return py::none();
  Tensor qkv = op_norm_linear(x, py::none(), norm1, w_qkv, eps1, offset1).cast<Tensor>();
  py::tuple heads = op_qkv_norm_rope(qkv, q_norm, k_norm, cosv, sinv, n_q, n_kv, D, eps_qk, offset_qk, gated);
  qkv.reset();
  Tensor o = op_attention(heads[0].cast<Tensor>(), heads[1].cast<Tensor>(), heads[2].cast<Tensor>(), cu, max_seqlen, true, scale);
  o = o.reshape({x.size(0), n_q * D});
  if (gated) o = guarded([&] { return SigmoidMul::apply(o, heads[3].cast<Tensor>()); });
  heads = py::tuple();
  Tensor h = op_linear(o, w_o, py::none());
  o.reset();
  auto mlp = norm_mlp(h, x, norm2, w_gu, w_down, eps2, offset2);
  h.reset();
  return py::cast(guarded([&] { return mlp[1] + mlp[0]; }));
}

// norm1 (weight, bias), qkv, proj, norm2, fc1, fc2 (each weight, bias)
py::object op_vision_block(const Tensor& x, const py::tuple& w, const Tensor& cosv, const Tensor& sinv, const Tensor& cu, int64_t max_seqlen, int64_t heads,
                           int64_t D, double eps1, double eps2, double scale, bool tanh_approx) {
  const int64_t H = plain_rows(x) ? x.size(1) : 0;
  if (H == 0 || H != heads * D || D > 128 || !vlmt_rope_qkv_usable((int)D) || cosv.sizes() != sinv.sizes() || cosv.dim() != 2 || cosv.size(0) != x.size(0) ||
      cosv.size(1) != D || cosv.requires_grad() || sinv.requires_grad() || !plain_table(cosv) || !plain_table(sinv) || cu.scalar_type() != at::kInt ||
      !plain_vector(w[0], H) || !plain_vector(w[1], H, true) || !plain_weight(w[2], H) || !plain_vector(w[3], 3 * H, true) || !plain_weight(w[4], H) ||
      !plain_vector(w[5], H, true) || !plain_vector(w[6], H) || !plain_vector(w[7], H, true) || !plain_weight(w[8], H))
    return py::none();
  const int64_t inter = THPVariable_Unpack(w[8].ptr()).size(0);
  if (!plain_vector(w[9], inter, true) || !plain_weight(w[10], inter) || !plain_vector(w[11], H, true)) return py::none();
  const int64_t S = x.size(0);
  Tensor qkv = op_ln_linear(x, w[0], w[1], w[2], w[3], eps1);
  Tensor o = rope_attention(qkv, cosv, sinv, cu, max_seqlen, heads, D, scale);
  qkv.reset();
  Tensor a = op_linear(o.reshape({S, H}), w[4], w[5]);
  o.reset();
  Tensor r = guarded([&] { return x + a; });
  a.reset();
  Tensor act, pre = ln_linear(r, w[6], w[7], w[8], w[9], eps2, tanh_approx ? 2 : 1, &act);
  Tensor out = gelu_linear(pre, w[10], w[11], tanh_approx, std::move(act));
  pre.reset();
  return py::cast(guarded([&] { return r + out; }));
}

// norm, fc1, fc2 (each weight, bias); `grouped`: the norm works on the merged vectors, else on the patches
py::object op_patch_merger(const Tensor& x, const py::tuple& w, int64_t merged, bool grouped, double eps) {
  const int64_t H = plain_rows(x) && x.is_contiguous() && x.numel() % merged == 0 ? x.size(1) : 0;
  if (H == 0 || merged % 8 != 0 || !plain_vector(w[0], grouped ? merged : H) || !plain_vector(w[1], grouped ? merged : H, true) || !plain_weight(w[2], merged))
    return py::none();
  const int64_t inner = THPVariable_Unpack(w[2].ptr()).size(0);
  if (!plain_vector(w[3], inner, true) || !plain_weight(w[4], inner) || !plain_vector(w[5], THPVariable_Unpack(w[4].ptr()).size(0), true)) return py::none();
  Tensor h = guarded([&] { return grouped ? x.view({-1, merged}) : x; });
  h = op_layer_norm(h, w[0], w[1], eps);
  if (!grouped) h = guarded([&] { return h.view({-1, merged}); });
  Tensor pre = op_linear(h, w[2], w[3]);
  return py::cast(op_gelu_linear(pre, w[4], w[5], false));
}

// images int32 [n_img, 4] on the device (frames, height, width, first patch), n patches -> cos, sin, index, weight
std::vector<Tensor> vision_plan(const Tensor& images, const Tensor& trig, int64_t nf, int64_t side, int64_t merge, int64_t n) {
  TORCH_CHECK(images.is_cuda() && images.scalar_type() == at::kInt && images.is_contiguous() && images.dim() == 2 && images.size(1) == 4 &&
              trig.scalar_type() == at::kFloat && trig.is_contiguous() && trig.is_cuda() && nf > 0 && trig.numel() > 0 && trig.numel() % (2 * nf) == 0 &&
              (uintptr_t)trig.data_ptr() % 8 == 0 && side > 0 && merge > 0 && images.size(0) > 0);
  c10::cuda::CUDAGuard guard(images.device());
  auto fo = trig.options();
  Tensor c = torch::empty({n, 4 * nf}, fo), s = torch::empty({n, 4 * nf}, fo), index = torch::empty({4, n}, fo.dtype(at::kLong)),
         weight = torch::empty({4, n}, fo);
  vlmt_vision_plan(images.data_ptr<int>(), (int)images.size(0), trig.data_ptr<float>(), (int)(trig.numel() / (2 * nf)), (int)nf, (int)side, (int)merge, n, c.data_ptr<float>(),
                   s.data_ptr<float>(), index.data_ptr<int64_t>(), weight.data_ptr<float>(), cur_stream());
  tick(1);
  return {c, s, index, weight};
}
}  // namespace
void count_launches(int n) { tick(n); }
}  // namespace vlmt

void bind_autograd(py::module_& m) {
  using namespace vlmt;
  m.def("op_linear", &op_linear);
  m.def("op_norm_linear", &op_norm_linear);
  m.def("op_ln_linear", &op_ln_linear);
  m.def("op_gelu_linear", &op_gelu_linear);
  m.def("op_swiglu_linear", &op_swiglu_linear);
  m.def("op_rms_norm", &op_rms_norm);
  m.def("op_layer_norm", &op_layer_norm);
  m.def("op_rms_norm_gated", &op_rms_norm_gated);
  m.def("op_swiglu", [](const Tensor& gu) { return guarded([&] { return Swiglu::apply(gu); }); });
  m.def("op_sigmoid_mul", [](const Tensor& x, const Tensor& gate) { return guarded([&] { return SigmoidMul::apply(x, gate); }); });
  m.def("op_gelu", [](const Tensor& x, bool tanh_approx) { return guarded([&] { return Gelu::apply(x, tanh_approx); }); });
  m.def("op_qkv_norm_rope", &op_qkv_norm_rope);
  m.def("op_rope", &op_rope);
  m.def("op_attention", &op_attention);
  m.def("op_rows_update", [](const Tensor& x, const Tensor& index, const Tensor& src, bool add) {
    return guarded([&] { return RowsUpdate::apply(x, index, src, add); });
  });
  m.def("op_pos_embed", &op_pos_embed);
  m.def("op_embedding", &op_embedding);
  m.def("op_decoder_layer", &op_decoder_layer);
  m.def("op_vision_block", &op_vision_block);
  m.def("op_patch_merger", &op_patch_merger);
  m.def("rope_tables", &rope_tables);
  m.def("vision_plan", &vision_plan);
  m.def("op_launches", [] { return g_launches.load(); });
  m.def("may_add_grad", [](const Tensor& param) { return may_add(param); });
  m.def("op_grad_in_place", [](bool on) { g_in_place = on; });
}

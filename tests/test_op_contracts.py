"""What the ops and tables promise beyond their values: inputs that are refused, layouts and types that are accepted, when a gradient
is reported as ready, what user hooks see, and what is held in memory between and during the passes."""
import numpy as np
import pytest
import torch

from vlm_training_b200 import ops

DEV = "cuda"
gpu = pytest.mark.gpu


def _rand(*shape, scale=1.0, seed=0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed + sum(shape))) * scale).to(DEV, dtype)


# sides off the merge size, smaller than it, negative: refused on the host before anything reaches the device
@pytest.mark.parametrize("device", ["cpu", "cuda"])
@pytest.mark.parametrize("grids", [[[1, 2, 3]], [[1, 3, 2]], [[1, 1, 1]], [[1, 28, 37]], [[1, 27, 36]], [[1, 4, 4], [1, 1, 4]], [[1, -2, -2]]])
def test_image_sizes_off_the_merge_size_are_refused(grids, device):
    from vlm_training_b200.models.config import VisionConfig
    from vlm_training_b200.models.vision import VisionPlan

    with pytest.raises(ValueError):
        VisionPlan.build(grids, VisionConfig(hidden_size=64, num_heads=2, num_position_embeddings=2304, spatial_merge_size=2), device)


@gpu
def test_position_indices_stay_in_the_table():
    """The plan kernel clamps its coordinates to the tables, whatever the image sizes say."""
    images = torch.tensor([[1, 3, 37, 0], [1, 2, 1, 111]], dtype=torch.int32, device=DEV)
    trig = torch.ones(37 * 4 * 2, device=DEV)
    index = ops.vision_plan(images, trig, 4, 48, 2, 113)[2]
    assert int(index.min()) >= 0 and int(index.max()) < 48 * 48


_T, _H, _N = 256, 128, 384
_ROWS = torch.arange(_T)
# name -> (op of (x, parameters), parameter shapes, width of x)
_PARAM_OPS = {
    "linear": (lambda x, p: ops.linear(x, p["w"], p["b"]), dict(w=(_N, _H), b=(_N,)), _H),
    "norm_linear": (lambda x, p: ops.rms_norm_linear(x, p["nw"], p["w"]), dict(nw=(_H,), w=(_N, _H)), _H),
    "norm_linear_residual": (lambda x, p: ops.rms_norm_linear(x, p["nw"], p["w"], residual=_rand(_T, _H, seed=5)), dict(nw=(_H,), w=(_N, _H)), _H),
    "ln_linear": (lambda x, p: ops.layer_norm_linear(x, p["nw"], p["nb"], p["w"], p["b"]), dict(nw=(_H,), nb=(_H,), w=(_N, _H), b=(_N,)), _H),
    "gelu_linear": (lambda x, p: ops.gelu_linear(x, p["w"], p["b"]), dict(w=(_N, _H), b=(_N,)), _H),
    "swiglu_linear": (lambda x, p: ops.swiglu_linear(x, p["w"]), dict(w=(_N, _H)), 2 * _H),
    "rms_norm": (lambda x, p: ops.rms_norm(x, p["nw"]), dict(nw=(_H,)), _H),
    "layer_norm": (lambda x, p: ops.layer_norm(x, p["nw"], p["nb"]), dict(nw=(_H,), nb=(_H,)), _H),
    "rms_norm_gated": (lambda x, p: ops.rms_norm_gated(x, _rand(_T, _H, seed=6), p["nw"]), dict(nw=(_H,)), _H),
    "qkv_norm_rope": (lambda x, p: ops.qkv_norm_rope(x, 2, 1, 128, p["qw"], p["kw"], _rand(_T, 128, seed=7).float(), _rand(_T, 128, seed=8).float())[:3],
                      dict(qw=(128,), kw=(128,)), 512),
    "loss": (lambda x, p: ops.linear_cross_entropy(x, p["w"], (_ROWS * 7 % _N).to(DEV), 64, grad_in_place=True)[0], dict(w=(_N, _H)), _H),
    "experts": (lambda x, p: ops.moe_experts(x, p["gu"], p["dn"], torch.full((_T, 2), 0.5, device=DEV, dtype=torch.bfloat16),
                                             torch.stack((_ROWS % 4, (_ROWS + 1) % 4), 1).to(DEV)), dict(gu=(4, 256, _H), dn=(4, _H, 128)), _H),
}


def _leaves(name, tag=None, grad=0.0, fp8=False, resharded=False):
    """``x`` and the op's parameters; ``tag``: gradients of the parameters land in views of an engine's buffer, which it is called on."""
    _, shapes, width = _PARAM_OPS[name]
    x = _rand(_T, width, seed=1).requires_grad_()
    params = {}
    for i, (k, shape) in enumerate(shapes.items()):
        p = params[k] = torch.nn.Parameter(_rand(*shape, scale=0.2, seed=10 + i) + (1.0 if k in ("nw", "qw", "kw") else 0.0))
        if tag is not None:
            p.grad = torch.full_like(p, grad)
            p._vlmt_grad_in_place, p._vlmt_grad_ready = True, tag
        if fp8:
            p._vlmt_fp8 = p.dim() == 2
        if resharded:
            p._vlmt_resharded = True
    return x, params


def _backward(name, x, params, seed=30, **kw):
    out = _PARAM_OPS[name][0](x, params)
    outs = [o for o in (out if isinstance(out, tuple) else (out,)) if o is not None]
    torch.autograd.backward(outs, [_rand(*o.shape, seed=seed + i, dtype=o.dtype) if o.dim() else torch.full_like(o, 1.7) for i, o in enumerate(outs)], **kw)


@gpu
@pytest.mark.parametrize("name,form", [(n, "") for n in _PARAM_OPS] + [("linear", "fp8"), ("linear", "resharded"), ("norm_linear", "resharded"),
                                                                       ("norm_linear_residual", "resharded"), ("ln_linear", "resharded")])
def test_a_parameter_is_reported_ready_after_its_last_read(name, form):
    """The engine may enqueue the update of a parameter (and store it into the peers' memory) as soon as its gradient is reported: the
    callback here overwrites the parameter on the current stream, and the gradient of ``x`` must not change."""
    kw = {form: True} if form else {}
    x0, plain = _leaves(name, **kw)
    _backward(name, x0, plain)
    seen = []

    def overwrite(p):
        seen.append(id(p))
        p.data.fill_(float("nan"))

    x1, tagged = _leaves(name, overwrite, **kw)
    _backward(name, x1, tagged)
    assert torch.equal(x0.grad, x1.grad)
    for k, p in tagged.items():
        assert torch.equal(p.grad, plain[k].grad), k
        assert seen.count(id(p)) == (1 if id(p) in seen else 0), k
    assert seen


# tiles with an odd number of 64-column slabs (N mod 256 up to 64, or 129 to 192) that are followed by more work of the same block or pair,
# and an epilogue that lags (one or two blocks of K): the next item's first slab reuses the staging buffer of this item's last one
@gpu
@pytest.mark.parametrize("M,N,K", [(40000, 576, 64), (40000, 448, 128), (40000, 64, 64), (20000, 192, 64)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_gemm_epilogue_with_odd_slabs(M, N, K, accumulate):
    from vlm_training_b200.ops import cuda as cu

    a, b, base = _rand(M, K, seed=1), _rand(N, K, seed=2), _rand(M, N, seed=3)
    out = base.clone()
    cu._gemm(a, b, out=out, accumulate=accumulate)
    want = a.float() @ b.float().t() + (base.float() if accumulate else 0.0)
    torch.testing.assert_close(out.float(), want, atol=0.1 if accumulate else 1e-2, rtol=1.6e-2 if accumulate else 8e-3)   # one or two bf16 roundings
    cu.check_status()


@gpu
@pytest.mark.parametrize("M,N,K", [(40000, 576, 128), (40000, 64, 128), (128 * 16, 192, 128)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_fp8_gemm_epilogue_with_odd_slabs(M, N, K, accumulate):
    from vlm_training_b200.ops import cuda as cu
    from vlm_training_b200.ops.float8 import E4M3

    a8, _, ra = cu._C.fp8_quantize(_rand(M, K, seed=1), E4M3, True, False)
    b8, _, rb = cu._C.fp8_quantize(_rand(N, K, seed=2), E4M3, True, False)
    base = _rand(M, N, seed=3)
    out = base.clone()
    cu._C.gemm_fp8(a8, b8, out, ra, rb, E4M3, E4M3, accumulate)
    f8 = torch.float8_e4m3fn
    want = (a8.view(f8).float() @ b8.view(f8).float().t()) * (ra[1] * rb[1]) + (base.float() if accumulate else 0.0)
    torch.testing.assert_close(out.float(), want, atol=0.1 if accumulate else 2e-2, rtol=1.6e-2 if accumulate else 8e-3)
    cu.check_status()


# weight gradients with few tiles and a long K, which may be cut over K: the head of the smallest presets with a full row, and two in between
@gpu
@pytest.mark.parametrize("V,H,T", [(8192, 512, 8192), (32000, 256, 4096), (1024, 256, 4100), (9, 64, 64)])
def test_loss_adds_its_weight_gradient_with_one_rounding(V, H, T):
    """In a tagged ``.grad`` (fp32 sums, rounded once, added once): bit for bit the gradient that autograd gets without a tag; an earlier
    micro-batch in the buffer stays; the callback fires once per pass and autograd adds nothing."""
    V = (V + 7) // 8 * 8
    tgt = (torch.arange(T) * 13 % V).to(DEV)
    tgt[::5] = -100

    def grads(w, seed, scale):
        h = _rand(T, H, scale=0.5, seed=seed).requires_grad_()
        loss, n = ops.linear_cross_entropy(h, w, tgt, 1000, grad_in_place=True)
        (loss * (scale / n)).backward()
        return h

    plain = torch.nn.Parameter(_rand(V, H, scale=0.05, seed=3))
    parts = []
    for seed, scale in ((1, 1.0), (2, 1.7)):
        plain.grad = None
        h = grads(plain, seed, scale)
        parts.append((plain.grad.clone(), h.grad))
    tagged = torch.nn.Parameter(plain.detach().clone())
    seen = []
    tagged.grad = torch.zeros_like(tagged)
    tagged._vlmt_grad_in_place, tagged._vlmt_grad_ready = True, lambda p: seen.append(id(p))
    assert torch.equal(grads(tagged, 1, 1.0).grad, parts[0][1])
    assert torch.equal(tagged.grad, parts[0][0])
    assert torch.equal(grads(tagged, 2, 1.7).grad, parts[1][1])
    # the second sum is rounded to bf16 and added, or (split over a cluster) added in fp32: the forms differ by the rounding of the second
    # part (2^-9 of it) and of the total in each form (2^-9 each)
    total = parts[0][0].float() + parts[1][0].float()
    assert bool(((tagged.grad.float() - total).abs() <= 2.0 ** -8 * (parts[1][0].float().abs() + total.abs())).all())
    assert seen == [id(tagged)] * 2
    # against 32 bits: bf16 logits and d(logits) (2^-8 each), one rounding of the sum
    hr, wr = _rand(T, H, scale=0.5, seed=1).float(), plain.detach().float().requires_grad_()
    torch.nn.functional.cross_entropy((hr @ wr.t()).to(torch.bfloat16).float(), tgt, ignore_index=-100).backward()
    assert float((parts[0][0].float() - wr.grad).norm() / wr.grad.norm()) < 1e-2


@gpu
def test_loss_with_a_frozen_head_keeps_nothing_of_vocabulary_size():
    T, H, V = 2048, 1024, 32768
    w, tgt = _rand(V, H, scale=0.05, seed=3), (torch.arange(T) * 13 % V).to(DEV)
    grads = []
    for frozen in (False, True):
        h = _rand(T, H, scale=0.5, seed=1).requires_grad_()
        w.requires_grad_(not frozen)
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        loss, _ = ops.linear_cross_entropy(h, w, tgt, 512)
        held = torch.cuda.memory_allocated() - before
        loss.backward()
        grads.append(h.grad)
    assert held <= 2 * T * H + (1 << 20)   # the hidden state's gradient
    torch.testing.assert_close(grads[0].float(), grads[1].float(), atol=1e-4, rtol=1.6e-2)   # chunks of rows may sum K in another order


@gpu
def test_rotary_tables_of_every_accepted_form_of_positions():
    """Four rows of positions (text and three axes), a single row, a batch dimension, and frequencies that are learned."""
    from vlm_training_b200.ops import reference as ref

    section, T = [24, 20, 20], 50
    inv = 1.0 / (1e6 ** (torch.arange(0, 128, 2, device=DEV).float() / 128))
    pos = torch.randint(0, 4000, (4, T), generator=torch.Generator().manual_seed(0)).to(DEV)
    for rows in (pos[:3], pos, pos.t().contiguous().t()[:3]):
        want = ref.mrope_cos_sin(rows, inv, section)
        assert all(torch.equal(a, b) for a, b in zip(ops.rope_tables(rows, inv, section), want))
    f = pos[:1][0].float().unsqueeze(-1) * inv
    want = (torch.cat((f, f), -1).cos(), torch.cat((f, f), -1).sin())
    for rows in (pos[:1], pos[:3], pos):
        assert all(torch.equal(a, b) for a, b in zip(ops.rope_tables(rows, inv), want))
    batch = pos.view(1, 4, T)
    assert all(torch.equal(a[0], b) for a, b in zip(ops.rope_tables(batch, inv), want))
    learned = inv.clone().requires_grad_()
    cos, _ = ops.rope_tables(pos[:1], learned)
    cos.sum().backward()
    assert learned.grad is not None and bool(learned.grad.abs().sum() > 0)


# a table with rows behind the last square or of a larger square, a transposed one, an index table with a gap
@gpu
@pytest.mark.parametrize("form", ["longer", "larger", "strided", "index"])
def test_position_embedding_forms_outside_the_kernel(form):
    import dataclasses

    from vlm_training_b200.models.config import VisionConfig
    from vlm_training_b200.models.vision import VisionPlan

    cfg = VisionConfig(hidden_size=64, num_heads=2, num_position_embeddings=2310, spatial_merge_size=2)
    plan = VisionPlan.build([[1, 4, 6], [1, 8, 2]], cfg, DEV)
    x = _rand(40, 64, seed=1)
    table = _rand({"longer": 2310, "larger": 2500}.get(form, 2304), 64, seed=2)
    if form == "strided":
        table = table.t().contiguous().t()
    if form == "index":
        plan = dataclasses.replace(plan, pe_index=plan.pe_index.t().contiguous().t())
    got, want = [], []
    for out, p in ((got, plan), (want, dataclasses.replace(plan, images=None))):
        t = table.detach().clone(memory_format=torch.preserve_format).requires_grad_()
        y = ops.pos_embed_add(x, t, p, 2)
        y.backward(torch.ones_like(y))
        out += [y, t.grad]
    assert torch.equal(got[0], want[0])
    torch.testing.assert_close(got[1].float(), want[1].float(), atol=2e-2, rtol=1.6e-2)


def _sparse_inputs(lens, Hq=8, Hkv=1, D=256, seed=0):
    T = sum(lens)
    q, k, v = (_rand(T, h, D, seed=seed + i) for i, h in enumerate((Hq, Hkv, Hkv)))
    index = [_rand(T, 4, 64, seed=seed + 3), _rand(T, 64, seed=seed + 4), _rand(T, 4, seed=seed + 5)]
    return q, k, v, index, [0] + torch.tensor(lens).cumsum(0).tolist()


# documents up to 16 times the selected keys (masked) and beyond (gathered); boundaries on the host, as 64-bit values, with a gap between them, absent
@gpu
@pytest.mark.parametrize("lens", [[300, 40], [2200]])
@pytest.mark.parametrize("form", ["host", "int64", "gap", "absent"])
def test_sparse_attention_takes_boundaries_of_any_form(lens, form):
    topk = 64 if len(lens) > 1 else 128
    q, k, v, index, bounds = _sparse_inputs(lens)
    cu = torch.tensor(bounds, dtype=torch.int32, device=DEV)
    want = ops.dsa_attention(q, k, v, *index, cu, topk, None, bounds)
    other = {"host": cu.cpu(), "int64": cu.long(), "gap": torch.stack((cu, cu), 1)[:, 0], "absent": None}[form]
    assert torch.equal(ops.dsa_attention(q, k, v, *index, other, topk, None, bounds), want)


@gpu
@pytest.mark.parametrize("scale", [-0.05, 0.0])
def test_sparse_attention_with_a_scale_that_is_not_positive(scale):
    """Against the float32 softmax over the same keys; tolerances: bf16 rounding of P and of the results."""
    from vlm_training_b200.ops import cuda as cu

    L, topk = 500, 32
    q, k, v, index, bounds = _sparse_inputs([L], Hq=8, Hkv=1)
    sel = cu._C.dsa_select(index[0], index[1], index[2].float(), 0, 0, 0, L, topk).long()
    keep = torch.zeros(L, L + 1, dtype=torch.bool, device=DEV).scatter_(1, torch.where(sel < 0, L, sel), True)[:, :L]
    o = ops.dsa_attention(q, k, v, *index, torch.tensor(bounds, dtype=torch.int32, device=DEV), topk, scale, bounds)
    att = torch.einsum("qhd,kd->hqk", q.float(), k[:, 0].float()) * scale
    want = torch.einsum("hqk,kd->qhd", att.masked_fill(~keep, float("-inf")).softmax(-1), v[:, 0].float())
    torch.testing.assert_close(o.float(), want, atol=2e-2, rtol=2e-2)
    cu.check_status()


# masked (equal bit for bit), gathered (key and value gradients are summed by atomics: fp32 order, one bf16 rounding) and with every key kept
@gpu
@pytest.mark.parametrize("topk", [64, 16, 512])
def test_sparse_attention_never_reads_padding(topk):
    """Rows behind the last boundary may hold anything; their outputs and gradients are zero.  Inside a document every key and value
    row has to be finite, selected or not, as the op says."""
    q, k, v, index, bounds = _sparse_inputs([300, 70], Hq=8, Hkv=1)
    results = []
    for fill in (0.0, float("nan"), float("inf")):
        leaves = []
        for t in (q, k, v):
            t = torch.cat((t, torch.full_like(t[:50], fill)), 0).requires_grad_()
            leaves.append(t)
        idx = [torch.cat((t, torch.full_like(t[:50], fill)), 0) for t in index]
        o = ops.dsa_attention(*leaves, *idx, torch.tensor(bounds, dtype=torch.int32, device=DEV), topk, None, bounds)
        o.backward(_rand(*o.shape, seed=9))
        results.append([o] + [t.grad for t in leaves])
    for other in results[1:]:
        for a, b in zip(results[0], other):
            torch.testing.assert_close(a, b, atol=1e-2 if topk == 16 else 0.0, rtol=8e-3 if topk == 16 else 0.0)
    assert all(float(t[370:].abs().sum()) == 0.0 for t in results[0])


@gpu
@pytest.mark.parametrize("name,key,form", [(n, k, "") for n, (_, shapes, _) in _PARAM_OPS.items() for k in shapes] + [("linear", "w", "fp8"), ("norm_linear", "w", "resharded")])
def test_user_hooks_and_partial_backward_passes_see_tagged_gradients(name, key, form):
    """A parameter with a tensor hook gets its gradient through autograd; ``autograd.grad`` returns it and adds nothing;
    ``backward(inputs=...)`` touches only what was asked for."""
    kw = {form: True} if form else {}
    x0, plain = _leaves(name, **kw)
    _backward(name, x0, plain)
    want = plain[key].grad
    x1, tagged = _leaves(name, lambda p: None, **kw)
    p = tagged[key]
    handle = p.register_hook(lambda g: g * 2)
    after = []
    p.register_post_accumulate_grad_hook(lambda q: after.append(q.grad.clone()))
    _backward(name, x1, tagged)
    assert torch.equal(p.grad, want * 2)
    assert len(after) == 1 and torch.equal(after[0], p.grad)
    handle.remove()

    x2, tagged = _leaves(name, lambda p: None, **kw)
    out = _PARAM_OPS[name][0](x2, tagged)
    outs = [o for o in (out if isinstance(out, tuple) else (out,)) if o is not None]
    cot = [_rand(*o.shape, seed=30 + i, dtype=o.dtype) if o.dim() else torch.full_like(o, 1.7) for i, o in enumerate(outs)]
    (got,) = torch.autograd.grad(outs, [tagged[key]], cot)
    assert torch.equal(got, want) and float(tagged[key].grad.abs().sum()) == 0.0

    x3, tagged = _leaves(name, lambda p: None, **kw)
    _backward(name, x3, tagged, inputs=[x3])
    assert torch.equal(x3.grad, x0.grad) and float(tagged[key].grad.abs().sum()) == 0.0


@gpu
@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("name", list(_PARAM_OPS))
def test_forward_mode_tangents_are_refused(name, grad):
    """The ops have no forward-mode derivative: a tangent is refused, never dropped, with and without gradients."""
    import torch.autograd.forward_ad as fwad

    x, params = _leaves(name)
    with torch.set_grad_enabled(grad), fwad.dual_level():
        with pytest.raises(RuntimeError):
            _PARAM_OPS[name][0](fwad.make_dual(x.detach(), torch.ones_like(x)), params)


@pytest.mark.multigpu
def test_position_embedding_runs_on_the_device_of_its_operands():
    """The current device is another one, and the kernel goes to the operands' device and its stream."""
    import dataclasses

    from vlm_training_b200.models.config import VisionConfig
    from vlm_training_b200.models.vision import VisionPlan

    cfg = VisionConfig(hidden_size=64, num_heads=2, num_position_embeddings=2304, spatial_merge_size=2)
    with torch.cuda.device(0):
        plan = VisionPlan.build([[1, 4, 6], [1, 8, 2]], cfg, "cuda:1")
        x, table = _rand(40, 64, seed=1).to("cuda:1").requires_grad_(), _rand(2304, 64, seed=2).to("cuda:1").requires_grad_()
        y = ops.pos_embed_add(x, table, plan, 2)
        y.sum().backward()
        assert torch.equal(y, ops.pos_embed_add(x, table, dataclasses.replace(plan, images=None), 2)) and table.grad is not None


# bytes beyond what lives before the pass, in units of one [rows, I] bf16: d(activation), which the kernel overwrites with the
# activation, and d(pre-activation) (two for SwiGLU's pair); the weight gradients land in the tagged .grad
@gpu
@pytest.mark.parametrize("name,units", [("gelu", 2), ("swiglu", 3)])
def test_mlp_backward_peak_memory(name, units):
    T, I, H = 4096, 8192, 256
    pre = _rand(T, I * (2 if name == "swiglu" else 1), seed=1).requires_grad_()
    w = torch.nn.Parameter(_rand(H, I, scale=0.02, seed=2))
    w.grad, w._vlmt_grad_in_place = torch.zeros_like(w), True
    y = ops.gelu_linear(pre, w) if name == "gelu" else ops.swiglu_linear(pre, w)
    g = torch.ones_like(y)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    y.backward(g)
    assert torch.cuda.max_memory_allocated() - before <= units * T * I * 2 + (4 << 20)


@gpu
def test_expert_gradient_without_storage_is_refused():
    """A gradient bucket whose storage is released (a sharded unit outside its backward pass): an error, never a kernel on freed memory."""
    x, params = _leaves("experts", lambda p: None)
    out = _PARAM_OPS["experts"][0](x, params)
    params["dn"].grad.untyped_storage().resize_(0)
    with pytest.raises(RuntimeError):
        out.backward(torch.ones_like(out))


@gpu
@pytest.mark.parametrize("fp8", [False, True])
def test_cta_pairs_can_be_switched_off(fp8):
    """``VLMT_GEMM_PAIR=0`` (read once per process) keeps the pair kernel out of both GEMMs."""
    import os
    import subprocess
    import sys

    code = """
import torch
from torch.profiler import ProfilerActivity, profile
from vlm_training_b200.ops import cuda as cu
a, b, out = (torch.ones(4096, k, device="cuda", dtype=torch.bfloat16) for k in (256, 256, 4096))
with profile(activities=[ProfilerActivity.CUDA]) as prof:
    if %r:
        a8, _, ra = cu._C.fp8_quantize(a, 0, True, False)
        cu._C.gemm_fp8(a8, a8, out, ra, ra, 0, 0, False)
    else:
        cu._gemm(a, b, out=out)
    torch.cuda.synchronize()
assert float(out.float().mean()) == 256.0
print("pairs" if any("pair" in e.key for e in prof.key_averages()) else "blocks")
""" % fp8
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    said = [subprocess.run([sys.executable, "-c", code], cwd=root, env={**os.environ, "VLMT_GEMM_PAIR": on}, capture_output=True, text=True).stdout.split()[-1:]
            for on in ("1", "0")]
    assert said == [["pairs"], ["blocks"]]


@gpu
def test_loss_of_no_rows():
    """No tokens: a loss of zero, a zero weight gradient and an empty input gradient, with and without a graph."""
    h, w = _rand(0, 64).requires_grad_(), _rand(128, 64, seed=1).requires_grad_()
    tgt = torch.empty(0, dtype=torch.int64, device=DEV)
    loss, n = ops.linear_cross_entropy(h, w, tgt, 32)
    loss.backward()
    assert float(loss) == 0.0 and int(n) == 0 and h.grad.shape == (0, 64) and float(w.grad.abs().sum()) == 0.0
    with torch.no_grad():
        assert float(ops.linear_cross_entropy(h, w, tgt, 32)[0]) == 0.0

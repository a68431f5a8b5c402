"""Kernel variants and dispatch branches at the sizes where they can go wrong (edges of tiles, remainders, smallest and largest of
a range), against the plain-PyTorch fp32 statement of the same op.  All tests here need a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from vlm_training_b200 import ops

DEV = "cuda"


@pytest.fixture(autouse=True)
def _seed():
    torch.manual_seed(11)


def _rand(*shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device=DEV) * scale).to(dtype)


def _close(got, want, atol, rtol, what=""):
    got, want = got.float(), want.float()
    err = (got - want).abs()
    tol = atol + rtol * want.abs()
    assert bool((err <= tol).all()), f"{what}: max err {err.max().item():.4g}, max ref {want.abs().max().item():.4g}, " \
                                     f"frac bad {(err > tol).float().mean().item():.4g}"


# few output tiles: K split inside a cluster, whose blocks sum their fp32 parts through shared memory (odd rows and columns, a last part
# shorter than the others, one row)
@pytest.mark.parametrize("M,N,K", [(37, 4096, 4096), (1, 520, 2048), (200, 392, 1096), (130, 128, 4104)])
@pytest.mark.parametrize("layout", ["fwd", "dgrad", "wgrad"])
def test_gemm_split_over_k(M, N, K, layout):
    from vlm_training_b200.ops import cuda as cu

    a = _rand(K, (M + 7) // 8 * 8, scale=0.5)[:, :M] if layout == "wgrad" else _rand(M, K, scale=0.5)
    b = _rand(N, K, scale=0.5) if layout == "fwd" else _rand(K, N, scale=0.5)
    bias, alpha = _rand(N), torch.tensor(0.37, device=DEV)
    ar, br = (a.t() if layout == "wgrad" else a).float(), (b if layout == "fwd" else b.t()).float()
    want = 0.37 * (ar @ br.t())
    # fp32 accumulation of K products of size about 0.25, then one bf16 rounding (2^-8 of the value)
    tol = dict(atol=2e-2 * (K / 4096) ** 0.5, rtol=8e-3)
    got = [cu._gemm(a, b, a_mn=layout == "wgrad", b_mn=layout != "fwd", bias=bias, alpha=alpha) for _ in range(2)]
    torch.testing.assert_close(got[0].float(), want + bias.float(), **tol)
    assert torch.equal(got[0], got[1])   # the parts are summed in rank order
    base = _rand(M, N)
    acc = base.clone()
    cu._gemm(a, b, a_mn=layout == "wgrad", b_mn=layout != "fwd", out=acc, accumulate=True, alpha=alpha)
    torch.testing.assert_close(acc.float(), want + base.float(), atol=tol["atol"] * 2, rtol=1.6e-2)   # two roundings
    f32 = torch.zeros(M, N, device=DEV)
    cu._gemm(a, b, a_mn=layout == "wgrad", b_mn=layout != "fwd", out=f32, accumulate=True, alpha=alpha)
    torch.testing.assert_close(f32, want, atol=1e-2, rtol=1e-3)
    cu.check_status()


# gated RMS norm: rows of 128 and 256 in groups of four and two per warp (a last group that is not full), other widths and alignments in the general form
@pytest.mark.parametrize("rows", [1, 3, 4, 5, 33, 4097])
@pytest.mark.parametrize("D,shift", [(128, 0), (256, 0), (64, 0), (128, 1)])
def test_gated_norm_rows(rows, D, shift):
    def part():
        return _rand(rows * D + shift)[shift:].view(rows, D).requires_grad_()

    x, z, w, g = part(), part(), (_rand(D) + 1).requires_grad_(), _rand(rows, D)
    y = ops.rms_norm_gated(x, z, w, 1e-6)
    got = [y, *torch.autograd.grad(y, [x, z, w], g)]
    xf, zf, wf = (t.detach().float().requires_grad_() for t in (x, z, w))
    want = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-6) * wf * torch.nn.functional.silu(zf)
    want = [want, *torch.autograd.grad(want, [xf, zf, wf], g.float())]
    for name, a, b in zip(("y", "dx", "dz"), got, want):
        _close(a, b, 1e-2, 8e-3, name)   # fp32 inside, one bf16 rounding (2^-9 of the value)
    _close(got[3], want[3], 4e-3 * rows ** 0.5, 8e-3, "dw")


# gate / up projection with its activation in one kernel: the bits of the product and the activation kernel behind one another, for few rows (one and
# several parts of K, ragged K) and on CTA pairs (rows off the tile edges), gate and up kept or not; sizes without such a kernel are refused
@pytest.mark.parametrize("M,I,K,there", [(1, 12288, 4096, True), (37, 12288, 4096, True), (17, 256, 1096, True), (100, 1536, 520, True), (128, 128, 64, True),
                                         (451, 12288, 1032, True), (2049, 1280, 264, True), (1000, 9728, 512, True), (37, 192, 512, False), (300, 256, 512, False)])
def test_gate_up_with_its_activation(M, I, K, there):
    from vlm_training_b200.ops import cuda as cu

    x, w = _rand(M, K, scale=0.5), _rand(2 * I, K, scale=0.5)
    got = cu._C.gemm_glu(x, w, True)
    assert (got is not None) == there
    if there:
        gu = cu._gemm(x, w)
        assert torch.equal(got[1], gu) and torch.equal(got[0], cu._C.op_swiglu(gu))
        alone = cu._C.gemm_glu(x, w, False)
        assert torch.equal(alone[0], got[0]) and alone[1] is None
    cu.check_status()


# column sums: one cluster per 64 columns up to 2048 rows (a last block with fewer rows or none), slabs of 256 rows behind
@pytest.mark.parametrize("rows", [1, 256, 257, 513, 1793, 2048, 2049])
@pytest.mark.parametrize("cols", [8, 64, 72, 1160])
def test_column_sums(rows, cols):
    from vlm_training_b200.ops import cuda as cu

    x = _rand(rows, cols + 8)[:, :cols]
    # fp32 sums of up to 2049 values of size 1: a few roundings of 2^-24 of partial sums up to about 100
    torch.testing.assert_close(cu._C.colsum(x).double(), x.double().sum(0), atol=1e-4, rtol=1e-6)


# at most 128 rows: every width of the row tile at its edges, a feature tile that ends early, a short last block and part of K, activations, rows and
# columns behind the last ones, an output whose rows start anywhere
@pytest.mark.parametrize("M", [1, 16, 17, 48, 49, 64, 65, 96, 97, 128])
@pytest.mark.parametrize("N,K,splits", [(24584, 72, 1), (9224, 520, None), (136, 1160, None), (4304, 1152, 4), (8, 2056, None)])
def test_gemm_of_few_rows(M, N, K, splits):
    from vlm_training_b200.ops import cuda as cu

    assert cu._C.gemm_rows_splits(M, N, K) == splits or (splits is None and cu._C.gemm_rows_splits(M, N, K) > 0)
    a, w, bias, alpha = _rand(M, K, scale=0.5), _rand(N, K, scale=0.5), _rand(N), torch.tensor(0.37, device=DEV)
    want = 0.37 * (a.float() @ w.float().t()) + bias.float()
    # fp32 accumulation of K products of size about 0.25, then one bf16 rounding (2^-8 of the value)
    tol = dict(atol=2e-2 * (K / 4096) ** 0.5, rtol=8e-3)
    got = [cu._gemm(a, w, bias=bias, alpha=alpha) for _ in range(2)]
    torch.testing.assert_close(got[0].float(), want, **tol)
    assert torch.equal(got[0], got[1])   # the parts are summed in rank order
    for epilogue, approximate in ((1, "tanh"), (2, "none")):
        got = cu._gemm(a, w, bias=bias, alpha=alpha, epilogue=epilogue)
        torch.testing.assert_close(got.float(), torch.nn.functional.gelu(want, approximate=approximate), **tol)
    out = torch.full((M + 1, N + 3), 7.0, device=DEV, dtype=torch.bfloat16)
    cu._gemm(a, w, bias=bias, alpha=alpha, out=out[:M, 1:1 + N])
    torch.testing.assert_close(out[:M, 1:1 + N].float(), want, **tol)
    assert bool((out[M] == 7.0).all() and (out[:, 0] == 7.0).all() and (out[:, 1 + N:] == 7.0).all())
    cu.check_status()


# large outputs on CTA pairs (256 x 256 tiles): rows and columns off the tile edges, a pair whose second block has no rows, a K tail
@pytest.mark.parametrize("M,N,K", [(2500, 2600, 520), (2304 + 100, 2304, 1096), (10000, 512, 72)])
@pytest.mark.parametrize("layout", ["fwd", "dgrad", "wgrad"])
def test_gemm_cta_pairs(M, N, K, layout):
    from vlm_training_b200.ops import cuda as cu

    a = _rand(K, (M + 7) // 8 * 8, scale=0.5)[:, :M] if layout == "wgrad" else _rand(M, K, scale=0.5)
    b = _rand(N, K, scale=0.5) if layout == "fwd" else _rand(K, N, scale=0.5)
    bias, alpha = _rand(N), torch.tensor(0.37, device=DEV)
    want = 0.37 * ((a.t() if layout == "wgrad" else a).float() @ (b if layout == "fwd" else b.t()).float().t())
    # fp32 accumulation of K products of size about 0.25, then one bf16 rounding (2^-8 of the value); two when added to bf16
    tol = dict(atol=1e-2, rtol=8e-3)
    got = cu._gemm(a, b, a_mn=layout == "wgrad", b_mn=layout != "fwd", bias=bias, alpha=alpha)
    torch.testing.assert_close(got.float(), want + bias.float(), **tol)
    base = _rand(M, N)
    acc = base.clone()
    cu._gemm(a, b, a_mn=layout == "wgrad", b_mn=layout != "fwd", out=acc, accumulate=True, alpha=alpha)
    torch.testing.assert_close(acc.float(), want + base.float(), atol=4e-2, rtol=1.6e-2)
    cu.check_status()


# two CTA pairs of a cluster share a tile and its K: rows and columns off the tile edges, an odd number of K blocks, every layout, added to D,
# activations, and a last column off the groups of four
@pytest.mark.parametrize("M,N,K,layout", [(451, 3592, 4168, "fwd"), (520, 2056, 4104, "dgrad"), (392, 3200, 8200, "wgrad")])
def test_gemm_cta_pairs_split_over_k(M, N, K, layout):
    from vlm_training_b200.ops import cuda as cu

    assert cu._C.gemm_form(M, N, K, pair_clusters=cu._C.gemm_pair_clusters())[3:] == (True, 2)
    test_gemm_cta_pairs(M, N, K, layout)
    a, b = _rand(M, K, scale=0.5), _rand(N, K, scale=0.5)
    assert torch.equal(cu._gemm(a, b), cu._gemm(a, b))   # the parts are summed in rank order
    bias, n = _rand(N), N - 6
    pre = (a.float() @ b.float().t() + bias.float()) / 16
    for epilogue, approximate in ((1, "tanh"), (2, "none")):
        got = cu._gemm(a, b / 16, bias=bias / 16, epilogue=epilogue)
        torch.testing.assert_close(got.float(), torch.nn.functional.gelu(pre, approximate=approximate), atol=1e-2, rtol=8e-3)
    out = torch.full((M, N), 7.0, device=DEV, dtype=torch.bfloat16)
    cu._gemm(a, b[:n], bias=bias[:n], out=out[:, :n])
    torch.testing.assert_close(out[:, :n].float(), pre[:, :n] * 16, atol=1e-2, rtol=8e-3)
    assert bool((out[:, n:] == 7.0).all())   # columns behind the last one are not written
    cu.check_status()


# CTA pairs with up to one wave of tiles, where K would else be split; raster groups of 16 pairs, the last one short
@pytest.mark.parametrize("M,N,K,pairs", [(300, 6536, 520, True), (1000, 5000, 584, True), (1000, 2600, 72, False), (4360, 8200, 2056, True)])
def test_gemm_cta_pairs_raster_and_single_wave(M, N, K, pairs):
    from vlm_training_b200.ops import cuda as cu

    assert cu._C.gemm_form(M, N, K)[3] == pairs
    a, b, bias = _rand(M, K, scale=0.5), _rand(N, K, scale=0.5), _rand(N)
    want = a.float() @ b.float().t() + bias.float()
    torch.testing.assert_close(cu._gemm(a, b, bias=bias).float(), want, atol=1e-2, rtol=8e-3)   # one bf16 rounding (2^-8 of the value)
    cu.check_status()


# the first case keeps d(logits) for backward (T <= 2 H), the second forms the gradients chunk by chunk (T > 2 H, V large)
@pytest.mark.parametrize("T,H,V,chunk", [(700, 512, 5000, 256), (1030, 256, 151936, 512)])
def test_linear_cross_entropy_both_gradient_forms_and_evaluation(T, H, V, chunk):
    """Tolerances as for the training path of the op (bf16 logits and gradients); the evaluation path runs the same loss kernel
    without its gradient half, so the losses are equal."""
    h = _rand(T, H, scale=0.5).requires_grad_()
    w = _rand(V, H, scale=0.05).requires_grad_()
    tgt = torch.randint(0, V, (T,), device=DEV)
    tgt[::7] = -100
    loss_sum, n = ops.linear_cross_entropy(h, w, tgt, chunk)
    (loss_sum / n).backward()
    hr, wr = h.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    logits = (hr @ wr.t()).to(torch.bfloat16).float()  # the kernel sees bf16 logits
    torch.nn.functional.cross_entropy(logits, tgt, ignore_index=-100).backward()
    _close(h.grad, hr.grad, 2e-4, 5e-2, "dh")
    _close(w.grad, wr.grad, 2e-4, 5e-2, "dw")
    with torch.no_grad():
        loss_eval, n_eval = ops.linear_cross_entropy(h, w, tgt, chunk)
    assert int(n_eval) == int(n) and torch.equal(loss_eval, loss_sum.detach())


@pytest.mark.parametrize("lens,state", [([8], torch.float32), ([5, 4096, 3], torch.bfloat16), ([40, 4088, 4096 * 3 + 1, 17, 9000], torch.float32)])
def test_adamw_bucket_matches_segment_launches(lens, state):
    """One launch over a bucket of several optimizer groups (chunks of 4096 elements, edges inside and on chunk boundaries,
    padding between segments) gives bit for bit what one launch per segment gives."""
    from vlm_training_b200.ops import cuda as cu

    starts, n = [], 0
    for ln in lens:
        starts.append(n)
        n += (ln + 7) // 8 * 8
    groups = [i % 3 for i in range(len(lens))]
    lr, wd = [1e-2, 3e-3, 5e-2], [0.1, 0.0, 0.01]
    g = torch.zeros(n, device=DEV, dtype=torch.bfloat16)
    for s, ln in zip(starts, lens):
        g[s:s + ln] = torch.randn(ln, device=DEV)
    master = torch.where(g != 0, torch.randn(n, device=DEV), torch.zeros(n, device=DEV))
    m, v = torch.zeros(n, device=DEV, dtype=state), torch.zeros(n, device=DEV, dtype=state)
    one = [g.clone(), master.clone(), m.clone(), v.clone(), torch.zeros(n, device=DEV, dtype=torch.bfloat16)]
    per = [t.clone() for t in one]
    tables = cu.adamw_tables(list(zip(starts, groups)), n, DEV)
    for step in (1, 2):
        one[0].copy_(g)
        per[0].copy_(g)
        cu.adamw_bucket_(*one, tables, lr, wd, 0.9, 0.95, 1e-8, step, 0.5)
        for s, ln, gi in zip(starts, lens, groups):
            e = s + (ln + 7) // 8 * 8
            cu.adamw_step_(*(t[s:e] for t in per), lr[gi], 0.9, 0.95, 1e-8, wd[gi], step, 0.5, zero_grad=True)
    for a, b in zip(one, per):
        assert torch.equal(a, b)


# documents below, at and beyond the number of selected keys; ends on and off the 64- / 128-row tiles; one token; 1, 2 and 8 query heads per kv head
# the selection where it can go wrong: integer scores, so the oracle's are the same to the last bit; a bin of equal steps between smallest and largest
# score holds few keys ("spread"), a few hundred of them equal ("equal"), nearly all ("clustered": one far outlier), infinite scores, one value only
@pytest.mark.parametrize("kind", ["spread", "equal", "clustered", "infinite", "constant"])
@pytest.mark.parametrize("L,topk", [(1500, 64), (1301, 1000), (129, 128), (2500, 1)])
def test_dsa_selection_of_integer_scores(kind, L, topk):
    from vlm_training_b200.ops import cuda as cu

    iq, ik, w = torch.randint(-3, 4, (L, 4, 64), device=DEV), torch.randint(-3, 4, (L, 64), device=DEV), torch.randint(-2, 3, (L, 4), device=DEV)
    if kind == "equal":
        ik[:, 2:] = 0
    elif kind == "clustered":
        ik[3], iq[..., 0], w[:] = 128, iq[..., 0].abs() + 200, 1
    elif kind == "constant":
        ik[:] = 0
    iq, ik, w = iq.to(torch.bfloat16), ik.to(torch.bfloat16), w.float()
    if kind == "infinite":
        iq[..., 0], ik[7, 0], w[:] = 1.0, float("inf"), 1.0
    scores = (torch.einsum("thd,sd->ths", iq.float(), ik.float()).relu() * w[..., None]).sum(1)
    pos = torch.arange(L, device=DEV)
    causal = pos[None, :] <= pos[:, None]
    # the largest first, equal ones (-0 below 0, as the kernel orders them) in the order of their index
    order = torch.where(causal, scores, float("-inf")).sort(dim=1, descending=True, stable=True).indices[:, :topk]
    want = torch.zeros(L, L, dtype=torch.bool, device=DEV).scatter_(1, order, True) & causal
    bits = cu._C.dsa_select_bits(iq, ik, w, [0, L], topk)
    cu.check_status()
    got = ((bits[: (L + 63) // 64].t()[:, pos // 64] >> (pos % 64)) & 1).bool() & (pos[None, :] <= (pos[:, None] | 127))
    assert torch.equal(got.sum(1), want.sum(1)) and bool((got <= causal).all())
    assert torch.equal(got & (scores != 0), want & (scores != 0))   # zeros carry a sign, which a different order of the sum may change
    b0 = max(0, L - 1024)
    rows = cu._C.dsa_select(iq, ik, w, b0, b0, 0, L - b0, min(topk, L)).long()
    listed = torch.zeros(L - b0, L + 1, dtype=torch.bool, device=DEV).scatter_(1, torch.where(rows < 0, L, rows), True)[:, :L]
    assert torch.equal(listed, got[b0:])


# a threshold that several keys share, of which only some are kept: the rows whose warps go on counting behind the search, on every SM and many times over
@pytest.mark.parametrize("L,topk", [(2300, 700), (1100, 130)])
def test_dsa_selection_with_a_shared_threshold(L, topk):
    from vlm_training_b200.ops import cuda as cu

    # a key's score is its level for every query; half of the keys share one level
    level = torch.randint(0, 400, (L,), device=DEV)
    level[torch.rand(L, device=DEV) < 0.5] = 200
    iq, ik, w = torch.zeros(L, 4, 64, device=DEV), torch.zeros(L, 64, device=DEV), torch.zeros(L, 4, device=DEV)
    iq[..., 0], iq[..., 1], w[:, 0] = 1.0, 16.0, 1.0
    ik[:, 0], ik[:, 1] = level % 16, level // 16
    iq, ik = iq.to(torch.bfloat16), ik.to(torch.bfloat16)
    pos = torch.arange(L, device=DEV)
    causal = pos[None, :] <= pos[:, None]
    order = torch.where(causal, level[None, :].expand(L, L), -1).sort(dim=1, descending=True, stable=True).indices[:, :topk]
    want = torch.zeros(L, L, dtype=torch.bool, device=DEV).scatter_(1, order, True) & causal
    kept = torch.where(want, level[None, :], 1 << 20).amin(1)
    shared = ((level[None, :] == kept[:, None]) & causal & ~want).any(1)
    assert int(shared.sum()) > L // 4   # rows that go through the counting
    b0 = max(0, L - 1024)
    for _ in range(30):
        bits = cu._C.dsa_select_bits(iq, ik, w, [0, L], topk)
        got = ((bits[: (L + 63) // 64].t()[:, pos // 64] >> (pos % 64)) & 1).bool() & (pos[None, :] <= (pos[:, None] | 127))
        assert torch.equal(got, want)
        rows = cu._C.dsa_select(iq, ik, w, b0, b0, 0, L - b0, topk).long()
        assert bool(((rows >= -1) & (rows <= pos[b0:, None])).all())   # -1: a row with fewer keys
        assert torch.equal(torch.zeros(L - b0, L + 1, dtype=torch.bool, device=DEV).scatter_(1, torch.where(rows < 0, L, rows), True)[:, :L], want[b0:])
    cu.check_status()


# as many keys as a block's shared memory holds, and one more, which is refused
def test_dsa_selection_from_the_longest_document():
    from vlm_training_b200.ops import cuda as cu

    L, B, topk = 56044, 3, 2048
    level = torch.randint(0, 4000, (L + 1,), device=DEV)
    iq, ik, w = torch.zeros(L + 1, 4, 64, device=DEV), torch.zeros(L + 1, 64, device=DEV), torch.zeros(L + 1, 4, device=DEV)
    iq[..., 0], iq[..., 1], w[:, 0] = 1.0, 64.0, 1.0
    ik[:, 0], ik[:, 1] = level % 64, level // 64
    iq, ik = iq.to(torch.bfloat16), ik.to(torch.bfloat16)
    rows = cu._C.dsa_select(iq, ik, w, L - B, L - B, 0, B, topk).long()
    for b in range(B):
        n = L - B + b + 1
        want = level[:n].sort(descending=True, stable=True).indices[:topk].sort().values
        assert torch.equal(rows[b].sort().values, want)
    with pytest.raises(RuntimeError, match="code -3"):
        cu._C.dsa_select(iq, ik, w, L + 1 - B, L + 1 - B, 0, B, topk)
    cu.check_status()


@pytest.mark.parametrize("lens,topk,Hq,Hkv", [([700, 64, 1, 129, 300], 64, 16, 2), ([128, 1024, 257], 128, 8, 1), ([2100, 90], 512, 4, 4), ([1090], 1000, 4, 2)])
def test_dsa_masked_dense_attention(lens, topk, Hq, Hkv):
    """Bit masks hold exactly the keys of the list form, and attention under them (forward, all gradients) matches the float32
    softmax over the same keys.  Tolerances: bf16 rounding of P / dS and of the results, as for the dense kernels above."""
    from vlm_training_b200.ops import cuda as cu, dsa_cuda

    T, D = sum(lens), 256
    bounds = [0] + torch.tensor(lens).cumsum(0).tolist()
    cu_seq = torch.tensor(bounds, dtype=torch.int32, device=DEV)
    iq, ik, w = torch.randn(T, 4, 64, device=DEV).bfloat16(), torch.randn(T, 64, device=DEV).bfloat16(), torch.randn(T, 4, device=DEV)
    bits = cu._C.dsa_select_bits(iq, ik, w, bounds, topk)
    keep = torch.zeros(T, T, dtype=torch.bool, device=DEV)
    for s, e in zip(bounds[:-1], bounds[1:]):
        L = e - s
        pos = torch.arange(L, device=DEV)
        if L <= topk:
            keep[s:e, s:e] = pos[None, :] <= pos[:, None]
            continue
        words = bits[: (L + 63) // 64, s:e].t()                                     # [L, key tiles]
        m = ((words[:, pos // 64] >> (pos % 64)) & 1).bool()
        lists = torch.cat([cu._C.dsa_select(iq, ik, w, s + b, b, s, min(1024, L - b), min(topk, b + min(1024, L - b))).long()
                           if topk <= b + min(1024, L - b) else None for b in range(0, L, 1024)])
        want = torch.zeros(L, L + 1, dtype=torch.bool, device=DEV).scatter_(1, torch.where(lists < 0, L, lists), True)[:, :L]
        m = m & (pos[None, :] <= (pos[:, None] | 127))                              # words behind a query's 128-row tile are not written
        assert torch.equal(m, want)
        keep[s:e, s:e] = want
    q, k, v = (torch.randn(T, h, D, device=DEV).bfloat16().requires_grad_() for h in (Hq, Hkv, Hkv))
    o = dsa_cuda._MaskedAttention.apply(q, k, v, cu_seq, bits, topk, D ** -0.5)
    g = torch.randn(T, Hq, D, device=DEV).bfloat16()
    o.backward(g)
    cu.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    kx, vx = (t.repeat_interleave(Hq // Hkv, 1) for t in (kr, vr))
    att = torch.einsum("qhd,khd->hqk", qr, kx) * D ** -0.5
    o_r = torch.einsum("hqk,khd->qhd", att.masked_fill(~keep, float("-inf")).softmax(-1), vx)
    o_r.backward(g.float())
    _close(o, o_r, 0.02, 2e-2, "out")
    _close(q.grad, qr.grad, 0.05, 3e-2, "dq")
    _close(k.grad, kr.grad, 0.05, 3e-2, "dk")
    _close(v.grad, vr.grad, 0.05, 3e-2, "dv")


@pytest.mark.parametrize("grids,side,merge", [([[1, 2, 2]], 48, 2), ([[1, 64, 26], [2, 4, 8], [1, 14, 52]], 48, 2), ([[1, 6, 6]], 4, 2), ([[1, 8, 4]], 1, 2)])
def test_vision_plan_and_position_embedding_kernels(grids, side, merge):
    """Tables made on the device against the host's numpy form (all equal), and the position embedding with its gradient against the gathered statement of the op."""
    import dataclasses

    from vlm_training_b200.models.config import VisionConfig
    from vlm_training_b200.models.vision import VisionPlan

    cfg = VisionConfig(hidden_size=288, num_heads=4, num_position_embeddings=side * side, spatial_merge_size=merge)
    want, got = VisionPlan.build(grids, cfg, "cpu"), VisionPlan.build(grids, cfg, DEV)
    assert got.max_seqlen == want.max_seqlen and torch.equal(got.cu_seqlens.cpu(), want.cu_seqlens)
    assert torch.equal(got.pe_index.cpu(), want.pe_index) and torch.equal(got.pe_weight.cpu(), want.pe_weight)
    assert torch.equal(got.cos.cpu(), want.cos) and torch.equal(got.sin.cpu(), want.sin)
    n = got.cos.shape[0]
    x, table, g = _rand(n, 288).requires_grad_(), _rand(side * side, 288).requires_grad_(), _rand(n, 288)
    y = ops.pos_embed_add(x, table, got, merge)
    y.backward(g)
    y_ref = ops.pos_embed_add(x.detach(), table.detach(), dataclasses.replace(got, images=None), merge)
    assert torch.equal(y, y_ref)
    assert torch.equal(x.grad, g)
    dt = torch.zeros(side * side, 288, device=DEV)
    for c in range(4):
        dt.index_add_(0, got.pe_index[c], got.pe_weight[c].unsqueeze(1) * g.float())
    _close(table.grad, dt, 1e-4 * float(dt.abs().max()) + 1e-6, 4e-3, "dtable")   # fp32 sums, one bf16 rounding


@pytest.mark.parametrize("axes,section", [(3, [24, 20, 20]), (1, None), (1, [11, 11, 10])])
def test_rope_tables_kernel(axes, section):
    from vlm_training_b200.ops import reference as ref

    n, T = (sum(section) if section else 64), 1000
    pos = torch.randint(0, 40000, (axes, T), device=DEV)
    inv = 1.0 / (1e6 ** (torch.arange(0, 2 * n, 2, device=DEV).float() / (2 * n)))
    cos, sin = ops.rope_tables(pos, inv, section)
    f = pos[0].float().unsqueeze(-1) * inv
    want = ref.mrope_cos_sin(pos.expand(3, -1), inv, section) if section else (torch.cat((f, f), -1).cos(), torch.cat((f, f), -1).sin())
    assert torch.equal(cos, want[0]) and torch.equal(sin, want[1])   # FP8 operands behind the rotation magnify a last bit


# FP8 on CTA pairs: rows and columns off the tile edges, a pair whose second block has no rows, a K tail, both operand formats
@pytest.mark.parametrize("M,N,K,fa", [(2512, 2608, 528, torch.float8_e5m2), (2304 + 112, 2304, 1104, torch.float8_e4m3fn), (10000, 512, 80, torch.float8_e5m2)])
def test_gemm_fp8_cta_pairs(M, N, K, fa):
    from vlm_training_b200.ops import cuda as cu
    from vlm_training_b200.ops.float8 import E4M3, E5M2

    fmt_a = E5M2 if fa == torch.float8_e5m2 else E4M3
    a8, _, ra = cu._C.fp8_quantize(_rand(M, K), fmt_a, True, False)
    b8, _, rb = cu._C.fp8_quantize(_rand(N, K), E4M3, True, False)
    want = (a8.view(fa).float() @ b8.view(torch.float8_e4m3fn).float().t()) * (ra[1] * rb[1])
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    cu._C.gemm_fp8(a8, b8, out, ra, rb, fmt_a, E4M3, False)
    tol = dict(atol=1e-3 * K ** 0.5, rtol=8e-3)   # order of K products of size 1, one bf16 rounding
    torch.testing.assert_close(out.float(), want, **tol)
    base = _rand(M, N)
    acc = base.clone()
    cu._C.gemm_fp8(a8, b8, acc, ra, rb, fmt_a, E4M3, True)
    torch.testing.assert_close(acc.float(), want + base.float(), atol=2e-3 * K ** 0.5 + 0.02, rtol=1.6e-2)   # two roundings
    cu.check_status()


@pytest.mark.parametrize("tiles,M,N", [([1, 0, 3], 256, 136), ([0, 2], 128, 64), ([0, 0], 128, 520)])
def test_grouped_weight_gradient_added_in_place(tiles, M, N):
    """Equal to the product added by a pass of its own, bit for bit; groups without rows keep what was there."""
    from vlm_training_b200.ops import cuda as cu

    prefix = torch.tensor([sum(tiles[:i]) for i in range(len(tiles) + 1)], dtype=torch.int32, device=DEV)
    rows = (sum(tiles) + 1) * 128
    a, b, base = _rand(rows, M), _rand(rows, N), _rand(len(tiles) * M, N)
    out = torch.empty_like(base)
    cu._C.gemm_grouped(a, b, out, prefix, 2, True)
    acc = base.clone()
    cu._C.gemm_grouped(a, b, acc, prefix, 2, True, True)
    assert torch.equal(acc, base + out)
    for g, n in enumerate(tiles):
        assert n or torch.equal(acc[g * M:(g + 1) * M], base[g * M:(g + 1) * M])
    cu.check_status()


# on CTA pairs: columns off the tile edges, groups of one 128-row tile and of none, long enough groups added
@pytest.mark.parametrize("tiles,M,N", [([1, 0, 3, 2], 512, 264), ([0, 1], 256, 520), ([4, 6], 256, 256)])
def test_grouped_weight_gradient_on_cta_pairs(tiles, M, N):
    from vlm_training_b200.ops import cuda as cu

    first = [sum(tiles[:i]) for i in range(len(tiles) + 1)]
    prefix = torch.tensor(first, dtype=torch.int32, device=DEV)
    a, b = _rand(first[-1] * 128, M, scale=0.5), _rand(first[-1] * 128, N, scale=0.5)
    want = torch.cat([a[128 * s:128 * e].float().t() @ b[128 * s:128 * e].float() for s, e in zip(first[:-1], first[1:])])
    out = torch.full((len(tiles) * M, N), 7.0, dtype=torch.bfloat16, device=DEV)
    cu._C.gemm_grouped(a, b, out, prefix, 2, True, False)
    torch.testing.assert_close(out.float(), want, atol=1e-3, rtol=8e-3)   # one bf16 rounding; a group without rows is zero
    base = _rand(len(tiles) * M, N)
    acc = base.clone()
    cu._C.gemm_grouped(a, b, acc, prefix, 2, True, True)
    assert torch.equal(acc, base + out)
    cu.check_status()


def _reference(fn):
    import vlm_training_b200.ops as O

    O._FORCE_REF = True
    try:
        return fn()
    finally:
        O._FORCE_REF = False


# 128-wide heads with full rotary, two heads per warp step, groups of 12 heads: odd counts, a lone last head, one token, gates, offset
@pytest.mark.parametrize("T,n_q,n_kv,gated,offset", [(1, 1, 1, False, False), (77, 3, 1, True, True), (50, 8, 3, False, True), (33, 13, 5, True, False)])
def test_qkv_norm_rope_128(T, n_q, n_kv, gated, offset):
    D = 128
    qkv, qw, kw = _rand(T, (n_q * (2 if gated else 1) + 2 * n_kv) * D), _rand(D, scale=0.3), _rand(D, scale=0.3)
    ang = torch.rand(T, D, device=DEV) * 6.28     # the two halves of a head may have different angles
    leaves = [t.requires_grad_() for t in (qkv, qw, kw)]
    exact = [t.detach().float().requires_grad_() for t in leaves]
    outs = [o for o in ops.qkv_norm_rope(qkv, n_q, n_kv, D, qw, kw, ang.cos(), ang.sin(), 1e-6, offset, gated) if o is not None]
    want = _reference(lambda: [o for o in ops.qkv_norm_rope(exact[0], n_q, n_kv, D, *exact[1:], ang.cos(), ang.sin(), 1e-6, offset, gated)
                               if o is not None])
    g = [_rand(*o.shape) for o in outs]
    torch.autograd.backward(outs, g)
    torch.autograd.backward(want, [x.float() for x in g])
    for a, b in zip(outs, want):
        _close(a, b, 0.03, 2e-2, "out")           # bf16 between norm and rotation, and of the result (2^-8 each of values up to 4)
    _close(qkv.grad, exact[0].grad, 0.06, 3e-2, "dqkv")
    for a, b in zip(leaves[1:], exact[1:]):       # sums of T heads' products, one bf16 rounding
        _close(a.grad, b.grad, 0.8, 3e-2, "dw")


# slabs of 128 tokens (64 forward) in groups of four with three tokens of lookahead: lengths around both, documents shorter than the window
@pytest.mark.parametrize("lens", [[1], [2, 1, 1], [127], [128], [129, 2], [130], [131, 126, 3], [63, 1, 64, 260]])
def test_short_convolution(lens):
    from vlm_training_b200.ops import reference as ref

    T, C = sum(lens), 520
    cu_seq = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), device=DEV, dtype=torch.int32)
    seq_idx = ref.seq_idx_from_cu(cu_seq, T)
    x, w, g = _rand(T, C).requires_grad_(), _rand(C, 4, scale=0.5).requires_grad_(), _rand(T, C)
    xr, wr = (t.detach().float().requires_grad_() for t in (x, w))
    y, y_r = ops.causal_conv1d_silu(x, w, seq_idx), ref.causal_conv1d_silu(xr, wr, seq_idx)
    y.backward(g)
    y_r.backward(g.float())
    _close(y, y_r, 0.03, 1e-2, "y")
    _close(x.grad, xr.grad, 0.05, 2e-2, "dx")
    _close(w.grad, wr.grad, 0.05, 1e-2, "dw")     # fp32 sums over the tokens, one bf16 rounding


@pytest.mark.parametrize("rows,cols,pad", [(1, 16, 0), (3, 4096, 0), (700, 1040, 0), (700, 1040, 8), (5000, 272, 16)])
def test_fp8_amax(rows, cols, pad):
    """Rows with and without a gap; the largest value in any place, also in the remainder of the four-wide loop."""
    from vlm_training_b200.ops import cuda as cu

    x = torch.full((rows, cols + pad), 100.0, device=DEV, dtype=torch.bfloat16)[:, :cols]   # the gap must not be read
    for r, c in ((0, 0), (rows - 1, cols - 1), (rows // 2, cols // 3)):
        x.copy_(_rand(rows, cols, scale=0.1))
        x[r, c] = -7.0
        assert float(cu._C.fp8_quantize(x, 0, True, False)[2][0]) == 7.0


# heads of 256: key tiles shared by clusters of 1, 2 and 4 blocks or pairs, documents of one key, of one tile and a bit, no causal mask
@pytest.mark.parametrize("lens,Hq,Hkv,causal", [([130, 1, 700], 16, 2, True), ([65, 129], 8, 2, False), ([64, 300], 6, 3, True), ([200], 3, 1, True)])
def test_attention_256_shared_key_tiles(lens, Hq, Hkv, causal):
    from vlm_training_b200.ops import cuda as cu, reference as ref

    T = sum(lens)
    cu_seq = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    q, k, v = (_rand(T, h, 256).requires_grad_() for h in (Hq, Hkv, Hkv))
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    g = _rand(T, Hq, 256)
    o, o_r = ops.attention_varlen(q, k, v, cu_seq, max(lens), causal, None), ref.attention_varlen(qr, kr, vr, cu_seq, max(lens), causal, None)
    o.backward(g)
    o_r.backward(g.float())
    cu.check_status()
    _close(o, o_r, 0.02, 2e-2, "out")
    for a, b, n in ((q, qr, "dq"), (k, kr, "dk"), (v, vr, "dv")):   # sums over up to Hq / Hkv heads of bf16 products
        _close(a.grad, b.grad, 0.05 * max(1.0, (Hq / Hkv) ** 0.5 / 2), 3e-2, n)


# heads of 256 on single blocks (rows of short documents): a key to a tile and a bit, key tiles shared by 4 blocks and by none, an odd group, no
# causal mask, more documents than a warp has lanes and twice that
@pytest.mark.parametrize("lens,Hq,Hkv,causal", [([1, 63, 64, 65, 127, 128, 129], 16, 2, True), ([65, 129], 8, 2, False), ([40] * 40, 4, 4, True),
                                                ([3] * 70, 5, 1, False), ([128] * 33, 2, 1, True), ([100], 8, 1, True)])
def test_attention_256_short_documents(lens, Hq, Hkv, causal):
    from vlm_training_b200.ops import cuda as cu

    assert cu._C.attn256_plan(sum(lens), len(lens), max(lens), Hq, Hkv, causal, False)[:2] == (False, False)
    test_attention_256_shared_key_tiles(lens, Hq, Hkv, causal)


# a block looks for its document 32 at a time: on pairs too, with documents that have no rows
@pytest.mark.parametrize("lens,Hq,Hkv", [([200 + 40 * i for i in range(34)], 2, 1), ([50, 0, 90, 0, 0, 700], 4, 2), ([0, 0, 0, 1500], 2, 2)])
def test_attention_256_pairs_find_their_document(lens, Hq, Hkv):
    from vlm_training_b200.ops import cuda as cu

    assert all(cu._C.attn256_plan(sum(lens), len(lens), max(lens), Hq, Hkv, True, False)[:2])
    test_attention_256_shared_key_tiles(lens, Hq, Hkv, True)


# heads of 256 on CTA pairs: key tiles shared by 4 and 2 pairs and by none, groups of 2 and 4 heads; an odd number of heads per key head, whose pairs
# take neighbouring query tiles, with the second one missing, of one row, and full
@pytest.mark.parametrize("lens,Hq,Hkv,causal,parts", [([1300], 8, 2, True, 4), ([2600], 20, 10, True, 2), ([2816], 20, 10, True, 1), ([2816], 40, 10, True, 1),
                                                      ([1152, 1409, 1536], 5, 1, True, 1), ([1409, 1280], 3, 3, False, 1)])
def test_attention_256_pairs(lens, Hq, Hkv, causal, parts):
    from vlm_training_b200.ops import cuda as cu

    assert cu._C.attn256_plan(sum(lens), len(lens), max(lens), Hq, Hkv, causal, False) == (True, True, parts)
    test_attention_256_shared_key_tiles(lens, Hq, Hkv, causal)


# the running maximum jumps by 17 powers of two in the second 64 keys of a step: in the first step, after several, in the last; without and with a
# selection, whose bits are fetched once per group of heads, and with the group of heads split over pairs and whole
@pytest.mark.parametrize("L,Hq,Hkv,topk,parts", [(1500, 4, 2, 0, 2), (1500, 8, 1, 64, 4), (2816, 20, 10, 96, 1)])
def test_attention_256_maximum_jumps_within_a_step(L, Hq, Hkv, topk, parts):
    from vlm_training_b200.ops import cuda as cu
    from vlm_training_b200.ops.dsa_cuda import _MaskedAttention

    assert cu._C.attn256_plan(L, 1, L, Hq, Hkv, True, topk > 0) == (True, True, parts)
    q, k, v, g = _rand(L, Hq, 256), _rand(L, Hkv, 256), _rand(L, Hkv, 256), _rand(L, Hq, 256)
    at = torch.arange(L, device=DEV)
    q[..., 0] = 16.0   # channel 0 adds its key's value to every score (the scale is 1 / 16)
    k[..., 0] = (12.0 * ((at >= 64).float() + (at >= 4 * 128 + 64) + (at >= L - L % 128 - 64)))[:, None].to(k.dtype)
    keep = torch.ones(L, L, dtype=torch.bool, device=DEV).tril()
    leaves, ref = [t.clone().requires_grad_() for t in (q, k, v)], [t.float().requires_grad_() for t in (q, k, v)]
    if topk:
        index = _rand(L, 4, 64), _rand(L, 64), _rand(L, 4).float()
        bits = cu._C.dsa_select_bits(*index, [0, L], topk)
        sel = cu._C.dsa_select(*index, 0, 0, 0, L, topk).long()
        keep = torch.zeros(L, L + 1, dtype=torch.bool, device=DEV).scatter_(1, torch.where(sel < 0, L, sel), True)[:, :L]
        o = _MaskedAttention.apply(*leaves, torch.tensor([0, L], dtype=torch.int32, device=DEV), bits, topk, 1 / 16)
    else:
        o = ops.attention_varlen(*leaves, torch.tensor([0, L], dtype=torch.int32, device=DEV), L, True, None)
    o.backward(g)
    att = torch.einsum("qhd,khd->hqk", ref[0], ref[1].repeat_interleave(Hq // Hkv, 1)) / 16
    o_r = torch.einsum("hqk,khd->qhd", att.masked_fill(~keep, float("-inf")).softmax(-1), ref[2].repeat_interleave(Hq // Hkv, 1))
    o_r.backward(g.float())
    cu.check_status()
    _close(o, o_r, 0.03, 2e-2, "out")
    # few keys carry a row, so dS is of order 1: its bf16 rounding (2^-9) times keys and queries of order 4, for a key over hundreds of rows;
    # channel 0 multiplies it by up to 36 and is left out
    for a, b, n in zip(leaves, ref, ("dq", "dk", "dv")):
        err, size = (a.grad.float() - b.grad)[..., 1:], b.grad[..., 1:]
        assert float(err.norm() / size.norm()) < 6e-3, n   # bf16 P and dS, bf16 result: 2.3e-3 to 2.7e-3 on random rows


def test_rope_tables_and_position_embedding_outside_the_kernels_forms():
    """Positions that are not int64, and operands off a 16-byte boundary, take the general forms."""
    import dataclasses

    from vlm_training_b200.models.config import VisionConfig
    from vlm_training_b200.models.vision import VisionPlan

    inv = 1.0 / (1e6 ** (torch.arange(0, 128, 2, device=DEV).float() / 128))
    pos = torch.arange(300, device=DEV)[None]
    want = ops.rope_tables(pos, inv)
    for other in (pos.int(), pos.float()):
        assert all(torch.equal(a, b) for a, b in zip(ops.rope_tables(other, inv), want))
    plan = VisionPlan.build([[1, 4, 6]], VisionConfig(hidden_size=64, num_heads=2, num_position_embeddings=16, spatial_merge_size=2), DEV)
    x, table = _rand(24 * 64 + 1)[1:].view(24, 64), _rand(16 * 64 + 1)[1:].view(16, 64)
    assert torch.equal(ops.pos_embed_add(x, table, plan, 2), ops.pos_embed_add(x, table, dataclasses.replace(plan, images=None), 2))
    with pytest.raises(ValueError):   # no patches: refused as on the host
        VisionPlan.build([[1, 0, 0]], VisionConfig(hidden_size=64, num_heads=2, num_position_embeddings=16), DEV)


# whole blocks as one call of the extension against the same block run module by module (a hook on a module that the block calls forces it): the same
# bits in outputs and gradients, with and without a graph; weights that take another path, and hooks, keep their say
@pytest.mark.parametrize("preset,layer", [("tiny-qwen3-vl-gpu", 0), ("qwen3.5-dense", 3)])
@pytest.mark.parametrize("block", ["decoder", "vision", "merger"])
def test_blocks_in_one_call(preset, layer, block):
    from vlm_training_b200.models import BatchPlan, ModelConfig
    from vlm_training_b200.models.causal_lm import rotary_inv_freq, rotary_tables
    from vlm_training_b200.models.layers import DecoderLayer, RowContext
    from vlm_training_b200.models.vision import PatchMerger, VisionBlock, VisionPlan

    cfg = ModelConfig.preset(preset)
    if block != "decoder" and preset != "tiny-qwen3-vl-gpu":
        pytest.skip("the vision tower of one preset is enough")
    if block == "decoder":
        cfg.text.hidden_size, cfg.text.intermediate_size = 512, 768
        m, hooked = DecoderLayer(cfg.text, layer), "self_attn.o_proj"
        bounds = [0, 100, 333]
        plan = BatchPlan.build(cfg, torch.zeros(333, dtype=torch.int64).numpy(), torch.tensor(bounds, dtype=torch.int32), None, DEV)
        ctx = RowContext(plan.cu_seqlens, plan.max_seqlen, *rotary_tables(cfg.text, plan.position_ids, rotary_inv_freq(cfg.text, torch.device(DEV)), torch.float32),
                         plan.seq_idx, plan.extras)
        x, args = _rand(333, 512), (ctx,)
    else:
        plan = VisionPlan.build([[1, 6, 10], [1, 4, 4]], cfg.vision, torch.device(DEV))
        m, hooked, args = (VisionBlock(cfg.vision), "attn.proj", (plan,)) if block == "vision" else (PatchMerger(cfg.vision, layer == 0), "", ())
        x = _rand(76, cfg.vision.hidden_size)
    m = m.to(DEV, torch.bfloat16)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(_rand(*p.shape, scale=0.05) + (1.0 if p.dim() == 1 else 0.0))

    def run(grad):
        with torch.set_grad_enabled(grad):
            xi = x.clone().requires_grad_(grad)
            y = m(xi, *args)
            if not grad:
                return [y]
            g = torch.autograd.grad(y, [xi, *m.parameters()], torch.ones_like(y))
            return [y.detach(), *g]

    one = run(True), run(False)
    calls = []
    target = m.get_submodule(hooked)
    if block == "merger":
        handle = None
        m.linear_fc1.weight._vlmt_resharded = True   # a weight that is gathered by the module that reads it
    else:
        handle = target.register_forward_hook(lambda *_: calls.append(1))
    apart = run(True), run(False)
    assert block == "merger" or len(calls) == 2
    for a, b in zip(one, apart):
        for s, t in zip(a, b):
            assert torch.equal(s, t)
    if handle is not None:
        handle.remove()


def test_expert_gradients_are_stored_only_over_zeros():
    """The first gradient behind a clearing is stored, every other one is added: accumulation, a step, a clearing by hand, and gradients that
    the caller has written into meanwhile."""
    from vlm_training_b200.config import Config
    from vlm_training_b200.parallel.mesh import get_mesh
    from vlm_training_b200.train.optimizer import create_optimizer

    T, H, I, E, k = 300, 256, 128, 8, 2
    m = torch.nn.Module()
    m.gate_up_proj, m.down_proj = (torch.nn.Parameter(_rand(*s, scale=0.05)) for s in ((E, 2 * I, H), (E, H, I)))
    t = Config().training
    t.lr_llm = t.lr_mlp = t.lr_vit = 1e-3
    t.data_parallel = "fsdp"
    engine = create_optimizer(m, t, get_mesh(1, torch.device(DEV)))
    engine.set_requires_gradient_sync(False)   # no update under a backward pass that no step follows
    x, dy = _rand(T, H), _rand(T, H)
    w, chosen = ops.moe_router(_rand(T, E)[:, :E - 1].contiguous(), k)   # the last expert gets no token

    def backward():
        ops.moe_experts(x, m.gate_up_proj, m.down_proj, w.to(x.dtype), chosen).backward(dy)

    ps = m.gate_up_proj, m.down_proj
    alone = [torch.autograd.grad(ops.moe_experts(x, *ps, w.to(x.dtype), chosen), ps, dy)[i] for i in range(2)]
    for p in ps:
        assert not bool(p.grad.any())
    backward()                                                # over the zeros of a new engine
    for p, a in zip(ps, alone):
        assert torch.equal(p.grad, a) and not bool(p.grad[-1].any())
    backward()                                                # added
    for p, a in zip(ps, alone):
        assert torch.equal(p.grad, a + a)
    engine.zero_grad()
    for p in ps:
        assert not bool(p.grad.any())
        p.grad.add_(1.0)                                      # the caller's own part
    backward()
    for p, a in zip(ps, alone):
        torch.testing.assert_close(p.grad.float(), a.float() + 1, atol=0, rtol=8e-3)   # one bf16 rounding of the sum
    engine.zero_grad()
    engine.set_requires_gradient_sync(True)
    backward()
    engine.step()
    engine.set_requires_gradient_sync(False)
    for p in ps:
        assert not bool(p.grad.any())                         # cleared by the update
    engine.zero_grad()
    alone = torch.autograd.grad(ops.moe_experts(x, *ps, w.to(x.dtype), chosen), ps, dy)
    backward()
    for p, a in zip(ps, alone):
        assert torch.equal(p.grad, a)
    engine.zero_grad()
    ps[0].grad = torch.full_like(ps[0], 2.0)                  # not the engine's buffer
    backward()
    torch.testing.assert_close(ps[0].grad.float(), alone[0].float() + 2, atol=0, rtol=8e-3)


# rows of one id in a block of 32 neighbours, over its edge, over several blocks, and all of them; a last block with one row; a second chunk of columns
@pytest.mark.parametrize("counts", [(1,), (32, 1), (31, 2, 5), (33, 64, 96), (7, 500, 1, 1, 90), (1000,), ()])
@pytest.mark.parametrize("D", [8, 1032])
def test_embedding_gradient_in_place(counts, D):
    n = sum(counts)
    ids = torch.cat([torch.full((c,), 3 * i, device=DEV) for i, c in enumerate(counts)] + [torch.empty(0, dtype=torch.long, device=DEV)])
    ids = ids[torch.randperm(n, device=DEV)]
    w = torch.nn.Parameter(_rand(20, D))
    w._vlmt_grad_in_place = True
    start = _rand(20, D)
    w.grad = start.clone()
    seen = []
    w._vlmt_grad_ready = seen.append
    dy = _rand(n, D)
    y = ops.embedding(ids, w, grad_in_place=True)
    assert torch.equal(y, w.detach()[ids])
    y.backward(dy)
    want = start.double().index_add(0, ids, dy.double())
    # fp32 sums of up to 1000 values of size 1, then one bf16 rounding of the sum
    torch.testing.assert_close(w.grad.double(), want, atol=1e-4, rtol=4e-3)
    assert len(seen) == 1 and seen[0] is w
    first, w.grad = w.grad, start.clone()
    ops.embedding(ids, w, grad_in_place=True).backward(dy)
    assert torch.equal(w.grad, first)
    # whoever asks for the gradient, or waits for it, gets the dense one
    w.grad = start.clone()
    dense, = torch.autograd.grad(ops.embedding(ids, w, grad_in_place=True), w, dy)
    plain, = torch.autograd.grad(torch.nn.functional.embedding(ids, w), w, dy)
    assert torch.equal(dense, plain) and torch.equal(w.grad, start)


# tiles of 128 rows x 64 columns, patches of 4 rows x 8 columns: remainders of each, a gap between the rows, the transpose alone and not at all
@pytest.mark.parametrize("rows", [1, 3, 16, 127, 129, 255])
@pytest.mark.parametrize("cols,fmt", [(16, 0), (48, 1), (64, 0), (80, 1), (208, 0)])
def test_cast_tiles(rows, cols, fmt):
    from vlm_training_b200.ops import cuda as cu
    from vlm_training_b200.ops.float8 import quantize_ref

    x = _rand(rows, cols + 24)[:, :cols]
    want = quantize_ref(x, fmt)[0].view(torch.uint8)
    for rm, t in ((True, True), (False, True), (True, False)):
        q, qt, rec = cu._C.fp8_quantize(x, fmt, rm, t)
        assert float(rec[0]) == float(x.abs().max())
        assert q.numel() == 0 if not rm else torch.equal(q, want)
        assert qt.numel() == 0 if not t else torch.equal(qt, want.t())


# gradient of gate and up in the kernel of the down projection's input gradient: the bits of the product and the activation kernel behind one another;
# rows and columns off the tile edges, a short contraction, an empty half tile of rows, the activation wanted or not; sizes without such a kernel
@pytest.mark.parametrize("M,I,K,there", [(4000, 9728, 72, True), (8321, 4800, 520, True), (16130, 2496, 264, True), (8192, 12288, 1024, True),
                                         (8192, 4680, 520, False), (2049, 4864, 520, False), (37, 12288, 4096, False), (300, 256, 512, False)])
def test_gate_up_gradient_with_its_product(M, I, K, there):
    from vlm_training_b200.ops import cuda as cu

    dy, w, gu = _rand(M, K, scale=0.5), _rand(K, I, scale=0.05), _rand(M, 2 * I)
    got = cu._C.gemm_glu_bwd(dy, w, gu, True)
    assert (got is not None) == there
    if there:
        d = torch.empty(M, I, dtype=torch.bfloat16, device=DEV)
        cu._C.gemm(dy, w, d, False, True, None, 0, False)
        assert torch.equal(got[0], cu._C.swiglu_bwd(d, gu)) and torch.equal(got[1], cu._C.op_swiglu(gu))
        alone = cu._C.gemm_glu_bwd(dy, w, gu, False)
        assert torch.equal(alone[0], got[0]) and alone[1] is None
    cu.check_status()


# the same for a GELU, whose columns may end inside a slab
@pytest.mark.parametrize("M,N,K,tanh,there", [(10240, 4304, 1152, True, True), (8321, 4808, 520, False, True), (16130, 2504, 264, True, True), (37, 4304, 1152, True, False)])
def test_gelu_gradient_with_its_product(M, N, K, tanh, there):
    from vlm_training_b200.ops import cuda as cu

    dy, w, x = _rand(M, K, scale=0.5), _rand(K, N, scale=0.05), _rand(M, N, scale=2.0)
    got = cu._C.gemm_gelu_bwd(dy, w, x, tanh, True)
    assert (got is not None) == there
    if there:
        d = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        cu._C.gemm(dy, w, d, False, True, None, 0, False)
        assert torch.equal(got[0], cu._C.gelu_bwd(d, x, tanh)) and torch.equal(got[1], cu._C.op_gelu(x, tanh))
        alone = cu._C.gemm_gelu_bwd(dy, w, x, tanh, False)
        assert torch.equal(alone[0], got[0]) and alone[1] is None
    cu.check_status()


# first linear of a vision MLP with its activation: the bits of the product and the activation kernel behind one another
@pytest.mark.parametrize("M,N,K,tanh,bias,there", [(10240, 4304, 1152, True, True, True), (2049, 1288, 520, False, True, True), (4001, 2504, 72, True, False, True),
                                                   (37, 4304, 1152, True, True, False), (300, 256, 512, True, True, False)])
def test_linear_with_its_gelu(M, N, K, tanh, bias, there):
    from vlm_training_b200.ops import cuda as cu

    x, w, b = _rand(M, K, scale=0.5), _rand(N, K, scale=0.1), _rand(N) if bias else None
    got = cu._C.gemm_gelu(x, w, b, tanh, True)
    assert (got is not None) == there
    if there:
        pre = cu._gemm(x, w, bias=b)
        assert torch.equal(got[1], pre) and torch.equal(got[0], cu._C.op_gelu(pre, tanh))
        alone = cu._C.gemm_gelu(x, w, b, tanh, False)
        assert torch.equal(alone[0], got[0]) and alone[1] is None
    cu.check_status()


# a bias read as vectors (columns that end inside a slab, and between two) and one that is not (off 16 bytes, columns not in eights), on one block and on pairs:
# the bits do not depend on how it is read
@pytest.mark.parametrize("M,N,K", [(300, 264, 72), (450, 1160, 1152), (10240, 1160, 520), (2305, 3456, 264), (450, 1156, 136)])
def test_bias_of_the_common_epilogue(M, N, K):
    from vlm_training_b200.ops import cuda as cu

    x, w, b = _rand(M, K, scale=0.5), _rand(N, K, scale=0.5), _rand(N + 1)
    y = cu._gemm(x, w, bias=b[:N])
    # fp32 accumulation of K products of size about 0.25, then one bf16 rounding (2^-8 of the value)
    torch.testing.assert_close(y.float(), x.float() @ w.float().t() + b[:N].float(), atol=2e-2 * (K / 4096) ** 0.5, rtol=8e-3)
    off = torch.empty(N + 1, dtype=b.dtype, device=DEV)[1:]
    off.copy_(b[:N])
    assert torch.equal(cu._gemm(x, w, bias=off), y)
    cu.check_status()


def test_expert_gradients_are_added_to_what_the_caller_has_left_in_the_buffer():
    """Writes that a tensor's version does not show: through `.data`, and by the replay of a captured pass."""
    from vlm_training_b200.config import Config
    from vlm_training_b200.parallel.mesh import get_mesh
    from vlm_training_b200.train.optimizer import create_optimizer

    T, H, I, E, k = 300, 256, 128, 8, 2
    m = torch.nn.Module()
    m.gate_up_proj, m.down_proj = ps = [torch.nn.Parameter(_rand(*s, scale=0.05)) for s in ((E, 2 * I, H), (E, H, I))]
    t = Config().training
    t.lr_llm = t.lr_mlp = t.lr_vit = 1e-3
    t.data_parallel = "fsdp"
    engine = create_optimizer(m, t, get_mesh(1, torch.device(DEV)))
    engine.set_requires_gradient_sync(False)   # no update under a backward pass that no step follows
    x, dy = _rand(T, H), _rand(T, H)
    w, chosen = ops.moe_router(_rand(T, E), k)
    alone = torch.autograd.grad(ops.moe_experts(x, *ps, w.to(x.dtype), chosen), ps, dy)

    def backward():
        ops.moe_experts(x, *ps, w.to(x.dtype), chosen).backward(dy)

    engine.zero_grad()
    for p, a in zip(ps, alone):
        p.grad.data.copy_(a)                   # a gradient that was kept from before
    backward()
    for p, a in zip(ps, alone):
        assert torch.equal(p.grad, a + a)
    engine.zero_grad()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        backward()                             # workspaces of the first pass
        side.synchronize()
        engine.zero_grad()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            backward()
        graph.replay()
        graph.replay()
    side.synchronize()
    for p, a in zip(ps, alone):
        assert torch.equal(p.grad, a + a)


def test_launches_are_counted_where_they_are_made():
    from vlm_training_b200.ops import cuda as cu

    def launched(fn):
        before = cu.LAUNCHES["count"]
        fn()
        return cu.LAUNCHES["count"] - before

    assert launched(lambda: cu._colsum(_rand(2048, 64))) == 1   # one launch, then slabs and their sum
    assert launched(lambda: cu._colsum(_rand(2049, 64))) == 2
    iq, ik, w = _rand(40 * 129, 4, 64), _rand(40 * 129, 64), _rand(40 * 129, 4).float()
    for docs, times in ((1, 1), (32, 1), (33, 2), (40, 2)):     # 32 blocks of queries per pair of launches
        assert launched(lambda: cu._C.dsa_select_bits(iq, ik, w, [129 * i for i in range(docs + 1)], 128)) == 2 * times


# the same comparison, with both routes shown to be the ones that are meant, and enough rows for the activations in the products' epilogues
@pytest.mark.parametrize("block,preset,layer,rows", [("decoder", "tiny-qwen3-vl-gpu", 0, 333), ("decoder", "tiny-qwen3-vl-gpu", 0, 8192), ("decoder", "qwen3.5-dense", 3, 1500),
                                                     ("vision", "tiny-qwen3-vl-gpu", 0, 76), ("vision", "tiny-qwen3-vl-gpu", 0, 4096), ("merger", "tiny-qwen3-vl-gpu", 0, 76),
                                                     ("merger", "tiny-qwen3-vl-gpu", 1, 4096)])
def test_blocks_go_the_way_that_they_are_meant_to(block, preset, layer, rows):
    from vlm_training_b200.models import BatchPlan, ModelConfig
    from vlm_training_b200.models.causal_lm import rotary_inv_freq, rotary_tables
    from vlm_training_b200.models.layers import DecoderLayer, RowContext
    from vlm_training_b200.models.vision import PatchMerger, VisionBlock, VisionPlan
    from vlm_training_b200.ops import cuda as cu

    cfg = ModelConfig.preset(preset)
    if block == "decoder":
        cfg.text.hidden_size, cfg.text.intermediate_size = 512, 4864
        m, hooked = DecoderLayer(cfg.text, layer), "self_attn.o_proj"
        plan = BatchPlan.build(cfg, torch.zeros(rows, dtype=torch.int64).numpy(), torch.tensor([0, rows // 3, rows], dtype=torch.int32), None, DEV)
        args = (RowContext(plan.cu_seqlens, plan.max_seqlen, *rotary_tables(cfg.text, plan.position_ids, rotary_inv_freq(cfg.text, torch.device(DEV)), torch.float32),
                           plan.seq_idx, plan.extras),)
        x = _rand(rows, 512)
        if rows == 8192:   # SwiGLU and its gradient in the epilogues
            gu, act = cu._C.gemm_glu(x, _rand(2 * 4864, 512), True)[::-1]
            assert cu._C.gemm_glu_bwd(x, _rand(512, 4864), gu, True) is not None
    else:
        cfg.vision.hidden_size, cfg.vision.num_heads, cfg.vision.intermediate_size = 512, 8, 1280
        grid = [[1, 64, 64]] if rows == 4096 else [[1, 6, 10], [1, 4, 4]]
        plan = VisionPlan.build(grid, cfg.vision, torch.device(DEV))
        m, hooked, args = (VisionBlock(cfg.vision), "attn.proj", (plan,)) if block == "vision" else (PatchMerger(cfg.vision, layer == 0), "", ())
        x = _rand(rows, 512)
        if block == "vision" and rows == 4096:   # GELU and its gradient in the epilogues
            act, pre = cu._C.gemm_gelu(x, _rand(1280, 512), _rand(1280), True, True)
            assert cu._C.gemm_gelu_bwd(x, _rand(512, 1280), pre, True, True) is not None
    m = m.to(DEV, torch.bfloat16)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(_rand(*p.shape, scale=0.05) + (1.0 if p.dim() == 1 else 0.0))

    def in_one_call():
        if block != "merger":
            return m._in_one_call(x, *args) is not None
        w = tuple(t for n in ("norm", "linear_fc1", "linear_fc2") for t in (m.get_submodule(n).weight, m.get_submodule(n).bias))
        return ops.whole_blocks(x).op_patch_merger(x, w, m.merged, m.postshuffle, m.norm.eps) is not None

    dy = None

    def run(grad):
        nonlocal dy
        with torch.set_grad_enabled(grad):
            xi = x.clone().requires_grad_(grad)
            y = m(xi, *args)
            if not grad:
                return [y]
            dy = _rand(*y.shape) if dy is None else dy
            return [y.detach(), *torch.autograd.grad(y, [xi, *m.parameters()], dy)]

    assert in_one_call()
    one = run(True), run(False)
    if block == "merger":
        m.linear_fc1.weight._vlmt_resharded = True   # a weight that is gathered by the module that reads it
    else:
        m.get_submodule(hooked).register_forward_hook(lambda *_: None)
    assert not in_one_call()
    apart = run(True), run(False)
    for a, b in zip(one, apart):
        for s, t in zip(a, b):
            assert torch.equal(s, t)
    cu.check_status()


# the score buffer filled more than once: by 32 blocks of queries, and by its 64 MB, in the middle of a document
@pytest.mark.parametrize("lens,topk", [([129] * 40, 128), ([4100, 20, 3300], 512)])
def test_dsa_selection_fills_its_buffer_again(lens, topk):
    from vlm_training_b200.ops import cuda as cu

    T = sum(lens)
    level = torch.randint(0, 400, (T,), device=DEV)   # a key's score, for every query
    iq, ik, w = torch.zeros(T, 4, 64, device=DEV), torch.zeros(T, 64, device=DEV), torch.zeros(T, 4, device=DEV)
    iq[..., 0], iq[..., 1], w[:, 0] = 1.0, 16.0, 1.0
    ik[:, 0], ik[:, 1] = level % 16, level // 16
    bounds = [sum(lens[:i]) for i in range(len(lens) + 1)]
    bits = cu._C.dsa_select_bits(iq.to(torch.bfloat16), ik.to(torch.bfloat16), w, bounds, topk)
    for s, L in zip(bounds, lens):
        if L <= topk:
            continue
        pos = torch.arange(L, device=DEV)
        causal = pos[None, :] <= pos[:, None]
        order = torch.where(causal, level[None, s:s + L].expand(L, L), -1).sort(dim=1, descending=True, stable=True).indices[:, :topk]
        want = torch.zeros(L, L, dtype=torch.bool, device=DEV).scatter_(1, order, True) & causal
        got = ((bits[: (L + 63) // 64, s:s + L].t()[:, pos // 64] >> (pos % 64)) & 1).bool() & (pos[None, :] <= (pos[:, None] | 127))
        assert torch.equal(got, want)
    cu.check_status()


# no rows: the weight's gradient is a sum of nothing, whatever the memory held before
@pytest.mark.parametrize("form", ["linear", "layer_norm_linear", "rms_norm_linear", "gelu_linear", "swiglu_linear"])
def test_gradients_of_no_rows_are_zero(form):
    w = _rand(64, 128).requires_grad_()
    n = [_rand(128).requires_grad_() for _ in range(2)]
    x = torch.empty(0, 256 if form == "swiglu_linear" else 128, dtype=torch.bfloat16, device=DEV, requires_grad=True)
    y = {"linear": lambda: ops.linear(x, w), "layer_norm_linear": lambda: ops.layer_norm_linear(x, *n, w), "rms_norm_linear": lambda: ops.rms_norm_linear(x, n[0], w),
         "gelu_linear": lambda: ops.gelu_linear(x, w), "swiglu_linear": lambda: ops.swiglu_linear(x, w)}[form]()
    held = [torch.full((64, 128), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(64)]
    del held   # what the gradient's memory holds
    assert torch.equal(torch.autograd.grad(y, w, torch.empty_like(y))[0], torch.zeros_like(w))

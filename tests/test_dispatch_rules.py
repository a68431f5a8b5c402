"""Which form of a kernel a call takes: pure functions of its sizes, no GPU needed."""
import pytest


# 24 to 37 tiles of 256 x 256: CTA pairs share a tile's K only where it would be split in two anyway.  Whole, it is faster in narrow tiles
# (454 x 4096 x 2048 14.8 us against 18.4, added to D 14.6 against 28.9), and so are four parts of it (381 x 3072 x 3072).
@pytest.mark.parametrize("M,N,K,parts", [(454, 4096, 2048, 1), (507, 4088, 3072, 1), (251, 8184, 2560, 1), (381, 3072, 3072, 1), (1275, 1280, 2048, 1),
                                         (451, 4096, 4096, 2), (451, 4096, 12288, 2), (200, 6144, 4096, 2), (300, 4096, 12288, 2), (200, 4096, 12288, 1)])
@pytest.mark.parametrize("parts_of_d", [False, True])
def test_pairs_share_the_k_of_a_tile_only_where_it_would_be_split(M, N, K, parts, parts_of_d):
    from vlm_training_b200.ops import cuda as cu

    bn, cluster, k_splits, pairs, got = cu._C.gemm_form(M, N, K, parts_of_d)
    assert got == parts and pairs == (parts == 2)
    assert cu._C.gemm_form(M, N, K, parts_of_d, pair_clusters=0)[4] == 1   # a GPU that cannot hold such clusters


# Up to half as many 256 x 256 tiles as SMs: pairs where 128 x 128 tiles do not fit one wave and K is not tiny, and where those would be split in two
@pytest.mark.parametrize("M,N,K,pairs", [(1961, 1152, 3456, False), (1661, 1408, 1152, False), (893, 2432, 12288, False), (381, 6144, 8192, False),
                                         (1019, 4088, 256, False), (2043, 2040, 72, False), (451, 6144, 4096, True), (700, 4096, 12288, True),
                                         (2500, 1152, 4304, True), (1000, 4096, 512, True), (381, 6144, 4304, True)])
def test_a_wave_of_pairs_only_where_it_is_the_faster_one(M, N, K, pairs):
    from vlm_training_b200.ops import cuda as cu

    assert cu._C.gemm_form(M, N, K)[3] == pairs


# At most 128 rows: the blocks that share a tile's K all have a part of it and fit a cluster; where one-block tiles are faster they are taken
@pytest.mark.parametrize("M,N,K,splits", [(37, 6144, 4096, 3), (37, 4096, 4096, 4), (37, 24576, 4096, 1), (37, 10240, 4096, 3), (37, 18944, 4096, 2), (8, 1152, 4304, 8),
                                          (64, 2048, 2048, 4), (64, 512, 512, 1), (8, 8, 64, 1), (64, 151936, 4096, 1), (65, 151936, 4096, 0),
                                          (128, 18944, 4096, 0), (129, 4096, 4096, 0)])
def test_blocks_that_share_a_tile_of_few_rows(M, N, K, splits):
    from vlm_training_b200.ops import cuda as cu

    assert cu._C.gemm_rows_splits(M, N, K) == splits
    for n in range(8, 30000, 552):
        for k in range(8, 13000, 488):
            s, kb = cu._C.gemm_rows_splits(M, n, k), (k + 63) // 64
            assert 0 <= s <= 8 and (s <= 1 or (s - 1) * ((kb + s - 1) // s) < kb)


# Heads of 256: rows of short documents on single blocks, whose blocks all have keys; long ones, and all with a selection, on pairs
@pytest.mark.parametrize("lens,Hq,Hkv,forward,backward", [([64], 16, 4, False, False), ([128] * 64, 16, 4, False, False), ([64] * 32, 16, 2, False, False),
                                                          ([128] * 64, 4, 4, False, False), ([150] * 4, 16, 2, False, False), ([900], 16, 2, True, True),
                                                          ([8192], 16, 4, True, True), ([700] * 11, 16, 4, True, True), ([16384], 4, 4, True, True)])
def test_heads_of_256_take_pairs_where_documents_are_long(lens, Hq, Hkv, forward, backward):
    from vlm_training_b200.ops import cuda as cu

    row = sum(lens), len(lens), max(lens), Hq, Hkv, True
    assert cu._C.attn256_plan(*row, False)[:2] == (forward, backward)
    assert cu._C.attn256_plan(*row, True)[:2] == (True, True)


# The parts of a key tile's query heads: as many as fill the GPU and no more; they divide the group
@pytest.mark.parametrize("lens,Hq,Hkv,parts", [([900], 16, 2, 4), ([900], 6, 2, 1), ([300], 12, 2, 2), ([128] * 64, 16, 2, 1), ([64] * 32, 16, 4, 1),
                                               ([8192], 16, 4, 1), ([16384], 16, 2, 1), ([1500], 16, 4, 4)])
def test_parts_of_a_key_tile_of_256_wide_heads(lens, Hq, Hkv, parts):
    from vlm_training_b200.ops import cuda as cu

    assert cu._C.attn256_plan(sum(lens), len(lens), max(lens), Hq, Hkv, True, False)[2] == parts


def test_tensor_memory_is_allocated_before_the_next_kernel_may_start():
    """The GEMMs allocate tensor memory before they wait for their predecessor.  A predecessor that let them in before it had its own
    columns could wait for them for ever, on an SM that they share."""
    import pathlib
    import re

    import vlm_training_b200.ops as ops

    allocating = set()
    for path in sorted((pathlib.Path(ops.__file__).parent / "csrc").glob("*.cu")):
        src = re.sub(r"__launch_bounds__\([^)]*\)", "", re.sub(r"//[^\n]*", "", path.read_text()))
        for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\([^{;]*\)\s*\{", src):
            body = src[m.end():src.index("\n}", m.end())]
            at = max(body.find(s) for s in ("tmem_alloc", "cta_setup<", "setup_end("))   # the last two: functions that allocate
            if at >= 0:
                allocating.add(m.group(1))
                assert "pdl_begin" not in body and "pdl_trigger" not in body[:at], m.group(1)
    assert {"gemm_kernel", "gemm_pair_kernel", "gdn_scan_kernel", "gdn_prepare_fwd_kernel", "dsa_index_scores_kernel", "attn256_fwd_kernel"} <= allocating


def test_the_selections_result_is_not_read_from_words_that_are_counted_in():
    """Top-k selection: warps leave the search for the threshold without a barrier and begin to count in `warp_cnt`."""
    import pathlib
    import re

    import vlm_training_b200.ops as ops

    src = (pathlib.Path(ops.__file__).parent / "csrc" / "dsa_indexer_sm100.cu").read_text()
    reads = re.findall(r"out\[\d\] = \(uint32_t\)sh_i\[(\d+)\];", src)
    counted, = re.findall(r"warp_cnt = sh_res \+ (\d+);", src)
    assert len(reads) == 3 and max(map(int, reads)) < int(counted)


def test_a_refusal_with_a_number_in_its_message_is_an_exception():
    import os
    import subprocess
    import sys

    code = """
from vlm_training_b200.ops import cuda as cu
try:
    cu._C.gemm_set_flag_wait_ms(1000)
except RuntimeError as e:
    assert str(e).startswith("vlmt_gemm_set_flag_wait_ms failed with code "), e   # no device
    print("raised")
"""
    # a process of its own, which a second C++ library would end, and without a GPU
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env={**os.environ, "CUDA_VISIBLE_DEVICES": ""})
    assert r.returncode == 0 and r.stdout.strip() == "raised", (r.returncode, r.stdout, r.stderr)


class _Extension:
    """Stands for the binding calls that run a whole block: remembers the weights that it gets."""

    def __init__(self):
        self.w = None

    def __getattr__(self, name):
        def call(x, w, *_):
            self.w = w
            return x
        return call


def test_vision_blocks_in_one_call_get_pruned_and_parametrised_tensors(monkeypatch):
    import types

    import torch
    from torch.nn.utils import parametrize, prune

    from vlm_training_b200 import ops
    from vlm_training_b200.models import ModelConfig
    from vlm_training_b200.models.vision import PatchMerger, VisionBlock

    class Twice(torch.nn.Module):
        def forward(self, t):
            return 2 * t

    ext = _Extension()
    monkeypatch.setattr(ops, "whole_blocks", lambda x, *modules: ext)
    cfg = ModelConfig.preset("tiny-qwen3-vl").vision
    plan = types.SimpleNamespace(cos=None, sin=None, cu_seqlens=None, max_seqlen=1)
    block, merger = VisionBlock(cfg), PatchMerger(cfg, False)
    for p in (*block.parameters(), *merger.parameters()):
        torch.nn.init.normal_(p)
    prune.random_unstructured(block.norm1, "bias", 0.5)
    prune.random_unstructured(block.mlp.linear_fc1, "bias", 0.5)
    prune.random_unstructured(block.attn.proj, "weight", 0.5)
    parametrize.register_parametrization(block.norm2, "bias", Twice())
    prune.random_unstructured(merger.linear_fc2, "bias", 0.5)
    x = torch.zeros(4, cfg.hidden_size)
    for call, modules in ((lambda: block._in_one_call(x, plan), (block.norm1, block.attn.qkv, block.attn.proj, block.norm2, block.mlp.linear_fc1, block.mlp.linear_fc2)),
                          (lambda: merger(x), (merger.norm, merger.linear_fc1, merger.linear_fc2))):
        assert call() is x
        assert all(torch.equal(w, t) for w, t in zip(ext.w, (t for m in modules for t in (m.weight, m.bias)))) and len(ext.w) == 2 * len(modules)


def test_decoder_layers_in_one_call_get_pruned_and_parametrised_weights(monkeypatch):
    import types

    import torch
    from torch.nn.utils import parametrize, prune

    from vlm_training_b200 import ops
    from vlm_training_b200.models import ModelConfig
    from vlm_training_b200.models.layers import DecoderLayer

    class Twice(torch.nn.Module):
        def forward(self, t):
            return 2 * t

    ext = _Extension()
    monkeypatch.setattr(ops, "whole_blocks", lambda x, *modules: ext)
    cfg = ModelConfig.preset("tiny-qwen3-vl").text
    layer = DecoderLayer(cfg, 0)
    for p in layer.parameters():
        torch.nn.init.normal_(p)
    attn, mlp = layer.self_attn, layer.mlp
    prune.random_unstructured(attn.qkv, "weight", 0.5)
    parametrize.register_parametrization(mlp.gate_up, "weight", Twice())
    parametrize.register_parametrization(attn.k_norm, "weight", Twice())
    prune.random_unstructured(mlp.down_proj, "weight", 0.5)
    x, ctx = torch.zeros(4, cfg.hidden_size), types.SimpleNamespace(cos=None, sin=None, cu_seqlens=None, max_seqlen=1)
    assert layer._in_one_call(x, ctx) is x
    modules = (layer.input_layernorm, attn.qkv, attn.q_norm, attn.k_norm, attn.o_proj, layer.post_attention_layernorm, mlp.gate_up, mlp.down_proj)
    assert len(ext.w) == len(modules) and all(torch.equal(w, m.weight) for w, m in zip(ext.w, modules))


@pytest.mark.parametrize("replaced", ["self_attn.o_proj", "mlp.down_proj"])
def test_a_layer_with_a_replaced_projection_runs_module_by_module(monkeypatch, replaced):
    import types

    import torch

    from vlm_training_b200 import ops
    from vlm_training_b200.models import ModelConfig
    from vlm_training_b200.models.layers import DecoderLayer

    ext = _Extension()
    monkeypatch.setattr(ops, "whole_blocks", lambda x, *modules: ext)
    cfg = ModelConfig.preset("tiny-qwen3-vl").text
    layer = DecoderLayer(cfg, 0)
    x, ctx = torch.zeros(4, cfg.hidden_size), types.SimpleNamespace(cos=None, sin=None, cu_seqlens=None, max_seqlen=1)
    assert layer._in_one_call(x, ctx) is x
    old = layer.get_submodule(replaced)
    layer.set_submodule(replaced, torch.nn.Linear(old.weight.shape[1], old.weight.shape[0], bias=False))   # without `tp` and `parallel`
    assert layer._in_one_call(x, ctx) is None


@pytest.mark.parametrize("owner,method", [("", "mixer_half"), ("", "mlp_half"), ("mlp", "forward_prenorm")])
def test_a_layer_with_a_half_of_its_own_runs_it(monkeypatch, owner, method):
    import types

    import torch

    from vlm_training_b200 import ops
    from vlm_training_b200.models import ModelConfig
    from vlm_training_b200.models.layers import DecoderLayer

    monkeypatch.setattr(ops, "whole_blocks", lambda x, *modules: _Extension())
    cfg = ModelConfig.preset("tiny-qwen3-vl").text
    layer = DecoderLayer(cfg, 0)
    x, ctx = torch.zeros(4, cfg.hidden_size), types.SimpleNamespace(cos=None, sin=None, cu_seqlens=None, max_seqlen=1)
    module = layer.get_submodule(owner)
    setattr(module, method, getattr(module, method))   # what a wrapper around a method leaves on the instance
    assert layer._in_one_call(x, ctx) is None


def test_a_saved_parameter_does_not_take_the_optimizer_along():
    import io

    import torch

    from vlm_training_b200.config import Config
    from vlm_training_b200.parallel.mesh import get_mesh
    from vlm_training_b200.train.optimizer import create_optimizer

    m = torch.nn.Linear(256, 256, bias=False)
    t = Config().training
    t.data_parallel = "fsdp"
    engine = create_optimizer(m, t, get_mesh(1, torch.device("cpu")))
    file = io.BytesIO()
    torch.save(m.weight, file)
    state = sum(x.numel() * x.element_size() for d in engine.domains for x in (*d.master, *d.exp_avg, *d.exp_avg_sq))
    assert file.tell() < m.weight.numel() * m.weight.element_size() + state // 2


@pytest.mark.parametrize("owner,method", [("layers.SelfAttention", "forward"), ("layers.Linear", "forward"), ("layers.SwiGLUMLP", "forward_prenorm"),
                                          ("layers.DecoderLayer", "mixer_half"), ("layers.DecoderLayer", "mlp_half"),
                                          ("vision.VisionAttention", "forward"), ("vision.VisionMLP", "forward")])
def test_a_class_whose_method_is_replaced_runs_it(monkeypatch, owner, method):
    import importlib
    import types

    import torch

    from vlm_training_b200 import ops
    from vlm_training_b200.models import ModelConfig
    from vlm_training_b200.models.layers import DecoderLayer
    from vlm_training_b200.models.vision import VisionBlock

    monkeypatch.setattr(ops, "whole_blocks", lambda x, *modules: _Extension())
    cfg = ModelConfig.preset("tiny-qwen3-vl")
    ctx = types.SimpleNamespace(cos=None, sin=None, cu_seqlens=None, max_seqlen=1)
    layer, block = DecoderLayer(cfg.text, 0), VisionBlock(cfg.vision)
    x, patches = torch.zeros(4, cfg.text.hidden_size), torch.zeros(4, cfg.vision.hidden_size)
    assert layer._in_one_call(x, ctx) is x and block._in_one_call(patches, ctx) is patches
    module, cls = owner.split(".")
    cls = getattr(importlib.import_module(f"vlm_training_b200.models.{module}"), cls)
    old = getattr(cls, method)
    monkeypatch.setattr(cls, method, lambda *args, **kwargs: old(*args, **kwargs))
    one, passed_by = (layer, x) if module == "layers" else (block, patches)
    assert one._in_one_call(passed_by, ctx) is None


@pytest.mark.parametrize("name", ["attention_varlen", "linear", "gelu_linear", "qkv_norm_rope"])
def test_blocks_with_a_replaced_op_run_module_by_module(monkeypatch, name):
    import types

    import torch

    from vlm_training_b200 import ops

    cuda = types.SimpleNamespace(_GEMM_BACKEND="tcgen05", _C=object())
    monkeypatch.setattr(ops, "_use_cuda", lambda x: True)
    monkeypatch.setattr(ops, "_cu", lambda: cuda)
    monkeypatch.setattr(ops, "_CUDA_MODULE", cuda)
    x = torch.zeros(4, 64)
    assert ops.whole_blocks(x) is cuda._C
    old = getattr(ops, name)
    monkeypatch.setattr(ops, name, lambda *args, **kwargs: old(*args, **kwargs))
    assert ops.whole_blocks(x) is None


def test_products_of_few_rows_ask_for_their_shared_memory_on_every_device():
    """The attribute belongs to a device: a flag of the process would leave it out on the second one."""
    import pathlib

    import vlm_training_b200.ops as ops

    src = (pathlib.Path(ops.__file__).parent / "csrc" / "gemm_rows_sm100.cu").read_text()
    launch = src[src.index("int launch("):]
    assert "static bool" not in launch and launch.index("cudaGetDevice") < launch.index("cudaFuncSetAttribute") < launch.index("launch_pdl(")


def test_shared_arrays_that_are_accessed_as_vectors_are_aligned():
    import pathlib
    import re

    import vlm_training_b200.ops as ops

    src = (pathlib.Path(ops.__file__).parent / "csrc" / "elementwise.cu").read_text()
    found = 0
    for body in src.split("__global__")[1:]:
        for name in set(re.findall(r"reinterpret_cast<(?:const )?(?:float|uint)4\*>\(&(\w+)\[", body)):
            declared = re.search(rf"__shared__ ([^;]*?)\b{name}\[", body)
            if declared is not None:
                found += 1
                assert "__align__(16)" in declared.group(1), name
    assert found > 0

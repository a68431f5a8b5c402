"""Qwen3-VL / Qwen3.5 vision tower: patch embedding, ViT blocks with 2-D rotary
and per-frame bidirectional varlen attention, 2x2 spatial patch merger and
DeepStack mergers.  Module and parameter names follow the HF snapshot layout
(reference: models/qwen3_vl/model.py:336-600).
"""
from __future__ import annotations

from dataclasses import dataclass

import numpy as np
import torch
import torch.nn as nn

from .. import ops
from . import positions
from .config import VisionConfig
from .layers import Linear, tensors_of


def _inv_freq(half):
    return 1.0 / (10000.0 ** (np.arange(0, half, 2, dtype=np.float32) / half))


@dataclass
class VisionPlan:
    """Host-built metadata for one batch of images (see :mod:`.positions`)."""

    cu_seqlens: torch.Tensor  # int32 [n_frames + 1]
    max_seqlen: int
    cos: torch.Tensor  # [N, head_dim] fp32
    sin: torch.Tensor
    pe_index: torch.Tensor  # int64 [4, N]
    pe_weight: torch.Tensor  # fp32 [4, N]
    images: torch.Tensor | None = None  # GPU: int32 [n_img, 4], frames / height / width / first patch of every image
    side: int = 0  # GPU: rows (and columns) of the position table the plan was built for

    @staticmethod
    def build(grids, cfg: VisionConfig, device) -> "VisionPlan":
        g = np.asarray(grids, dtype=np.int64).reshape(-1, 3)
        merge = cfg.spatial_merge_size
        # the tables are in merge-block order: an image with patches has whole blocks only
        if (g < 0).any() or (g[g.prod(1) != 0, 1:] % merge).any():
            raise ValueError(f"image sizes (frames, height, width in patches) must be multiples of {merge} patches: {g.tolist()}")
        cu, mx = positions.vision_segments(g)
        if ops.tables_on_device(device) and g.prod(1).any():
            # the tables are functions of the grids alone: made on the device; the grids travel, and the sine and cosine of every row
            # or column times every frequency, as numpy rounds them
            first = np.concatenate(([0], np.cumsum(g.prod(1))))
            fr = np.arange(g[:, 1:].max(), dtype=np.float32)[:, None] * _inv_freq(cfg.head_dim // 2)
            trig = np.stack((np.cos(fr), np.sin(fr)), -1).astype(np.float32, copy=False)  # [coordinate, frequency, 2]
            small = np.concatenate((np.column_stack((g, first[:-1])).ravel(), cu)).astype(np.int32)
            both = torch.from_numpy(np.concatenate((trig.reshape(-1).view(np.int32), small))).to(device, non_blocking=True)
            small = both[trig.size:]
            images = small[:4 * len(g)].view(-1, 4)
            side = int(round(cfg.num_position_embeddings ** 0.5))
            cos, sin, idx, wt = ops.vision_plan(images, both[:trig.size].view(torch.float32), trig.shape[1], side, merge, int(first[-1]))
            return VisionPlan(small[4 * len(g):], mx, cos, sin, idx, wt, images, side)
        coords = positions.vision_rot_coords(grids, cfg.spatial_merge_size)
        half = cfg.head_dim // 2
        fr = coords[:, :, None].astype(np.float32) * _inv_freq(half)[None, None, :]  # [N, 2, half/2]
        rot = fr.reshape(coords.shape[0], -1)  # [N, half]
        emb = np.concatenate((rot, rot), -1)
        side = int(round(cfg.num_position_embeddings ** 0.5))
        idx, wt = positions.vision_pos_embed_plan(grids, side, cfg.spatial_merge_size)
        t = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a)).to(device=device, dtype=dt, non_blocking=True)
        return VisionPlan(t(cu, torch.int32), mx, t(np.cos(emb), torch.float32), t(np.sin(emb), torch.float32),
                          t(idx, torch.int64), t(wt, torch.float32))


class _PatchProj(nn.Module):
    """Conv3d with kernel == stride, i.e. a GEMM on flattened patches; the weight
    keeps the HF shape ``[hidden, C, Tp, P, P]``."""

    def __init__(self, cfg: VisionConfig):
        super().__init__()
        self.weight = nn.Parameter(torch.empty(cfg.hidden_size, cfg.in_channels, cfg.temporal_patch_size,
                                               cfg.patch_size, cfg.patch_size))
        self.bias = nn.Parameter(torch.zeros(cfg.hidden_size))


class PatchEmbed(nn.Module):
    def __init__(self, cfg: VisionConfig):
        super().__init__()
        self.proj = _PatchProj(cfg)

    def forward(self, pixels):
        w = self.proj.weight
        return ops.linear(pixels.to(w.dtype), w.view(w.shape[0], -1), self.proj.bias)


class VisionAttention(nn.Module):
    def __init__(self, cfg: VisionConfig):
        super().__init__()
        self.n_heads, self.head_dim = cfg.num_heads, cfg.head_dim
        self.qkv = Linear(cfg.hidden_size, 3 * cfg.hidden_size, bias=True)
        self.proj = Linear(cfg.hidden_size, cfg.hidden_size, bias=True)

    def forward(self, x, plan: VisionPlan, prenorm: "nn.LayerNorm | None" = None):
        S = x.shape[0]
        if prenorm is not None:
            qkv = ops.layer_norm_linear(x, prenorm.weight, prenorm.bias, self.qkv.weight, self.qkv.bias, prenorm.eps)
        else:
            qkv = self.qkv(x)
        qkv = qkv.view(S, 3, self.n_heads, self.head_dim)
        q, k, v = qkv.unbind(1)
        D = self.head_dim
        # q and k leave the rotary kernel as contiguous [S, H, D]; v is read in place from the fused projection (the
        # attention kernels take strided heads and any head size that is a multiple of 8, 72 here)
        q, k = ops.rope_vision(q, k, plan.cos, plan.sin)
        o = ops.attention_varlen(q, k, v, plan.cu_seqlens, plan.max_seqlen, False, D ** -0.5)
        return self.proj(o.reshape(S, -1))


class VisionMLP(nn.Module):
    def __init__(self, cfg: VisionConfig):
        super().__init__()
        self.linear_fc1 = Linear(cfg.hidden_size, cfg.intermediate_size, bias=True)
        self.linear_fc2 = Linear(cfg.intermediate_size, cfg.hidden_size, bias=True)
        self.approx = "tanh" if "tanh" in cfg.hidden_act else "none"

    def forward(self, x, prenorm: "nn.LayerNorm | None" = None):
        if prenorm is not None:
            pre = ops.layer_norm_linear(x, prenorm.weight, prenorm.bias, self.linear_fc1.weight, self.linear_fc1.bias, prenorm.eps)
        else:
            pre = ops.linear(x, self.linear_fc1.weight, self.linear_fc1.bias)
        return ops.gelu_linear(pre, self.linear_fc2.weight, self.linear_fc2.bias, self.approx)


class VisionBlock(nn.Module):
    def __init__(self, cfg: VisionConfig):
        super().__init__()
        self.norm1 = nn.LayerNorm(cfg.hidden_size, eps=1e-6)
        self.norm2 = nn.LayerNorm(cfg.hidden_size, eps=1e-6)
        self.attn = VisionAttention(cfg)
        self.mlp = VisionMLP(cfg)

    def forward(self, x, plan: VisionPlan):
        if type(self) is VisionBlock and x.is_cuda:
            out = self._in_one_call(x, plan)
            if out is not None:
                return out
        x = x + self.attn(x, plan, prenorm=self.norm1)
        return x + self.mlp(x, prenorm=self.norm2)

    def _in_one_call(self, x, plan: VisionPlan):
        """The whole block as one call of the extension, or ``None`` where its modules have to run one by one."""
        parts = self._modules
        attn, mlp, n1, n2 = parts["attn"], parts["mlp"], parts["norm1"], parts["norm2"]
        if type(attn) is not VisionAttention or type(mlp) is not VisionMLP or _block_methods() != _BLOCK_METHODS:
            return None
        qkv, proj, fc1, fc2 = attn._modules["qkv"], attn._modules["proj"], mlp._modules["linear_fc1"], mlp._modules["linear_fc2"]
        if any(type(m) is not Linear or m.parallel is not None for m in (qkv, proj, fc1, fc2)):
            return None
        ext = ops.whole_blocks(x, attn, proj, mlp)
        if ext is None:
            return None
        w = tensors_of((n1, qkv, proj, n2, fc1, fc2), ("weight", "bias"))
        return ext.op_vision_block(x, w, plan.cos, plan.sin, plan.cu_seqlens, int(plan.max_seqlen), attn.n_heads, attn.head_dim, n1.eps, n2.eps,
                                   attn.head_dim ** -0.5, mlp.approx == "tanh")


def _block_methods():
    return VisionAttention.forward, VisionMLP.forward, Linear.forward


_BLOCK_METHODS = _block_methods()   # what `VisionBlock._in_one_call` stands for; a class whose method is replaced later runs that


class PatchMerger(nn.Module):
    """2x2 spatial merge MLP.  The main merger normalises each patch (dim
    ``hidden``) before grouping four of them; DeepStack mergers normalise the
    grouped vector (dim ``4*hidden``) (reference: models/qwen3_vl/model.py:446-462)."""

    def __init__(self, cfg: VisionConfig, postshuffle_norm: bool):
        super().__init__()
        self.merged = cfg.hidden_size * cfg.spatial_merge_size ** 2
        self.postshuffle = postshuffle_norm
        self.norm = nn.LayerNorm(self.merged if postshuffle_norm else cfg.hidden_size, eps=1e-6)
        self.linear_fc1 = Linear(self.merged, self.merged, bias=True)
        self.linear_fc2 = Linear(self.merged, cfg.out_hidden_size, bias=True)

    def forward(self, x):
        ext = ops.whole_blocks(x) if type(self) is PatchMerger else None
        if ext is not None:
            parts = self._modules
            w = tensors_of((parts["norm"], parts["linear_fc1"], parts["linear_fc2"]), ("weight", "bias"))
            out = ext.op_patch_merger(x, w, self.merged, self.postshuffle, parts["norm"].eps)
            if out is not None:
                return out
        if self.postshuffle:
            x = ops.layer_norm(x.view(-1, self.merged), self.norm.weight, self.norm.bias, self.norm.eps)
        else:
            x = ops.layer_norm(x, self.norm.weight, self.norm.bias, self.norm.eps).view(-1, self.merged)
        pre = ops.linear(x, self.linear_fc1.weight, self.linear_fc1.bias)
        return ops.gelu_linear(pre, self.linear_fc2.weight, self.linear_fc2.bias, "none")


class VisionModel(nn.Module):
    def __init__(self, cfg: VisionConfig):
        super().__init__()
        self.cfg = cfg
        self.patch_embed = PatchEmbed(cfg)
        self.pos_embed = nn.Embedding(cfg.num_position_embeddings, cfg.hidden_size)
        self.blocks = nn.ModuleList([VisionBlock(cfg) for _ in range(cfg.depth)])
        self.merger = PatchMerger(cfg, postshuffle_norm=False)
        self.deepstack_visual_indexes = list(cfg.deepstack_visual_indexes)
        self.deepstack_merger_list = nn.ModuleList(
            [PatchMerger(cfg, postshuffle_norm=True) for _ in self.deepstack_visual_indexes])
        self.ac_mode = "off"

    def forward(self, pixels, grid_thw=None, plan: VisionPlan | None = None):
        """pixels ``[N, C*Tp*P*P]`` in merge-block order → ``(merged [N/4, out], [deepstack...])``."""
        if plan is None:
            plan = VisionPlan.build(grid_thw.tolist() if torch.is_tensor(grid_thw) else grid_thw, self.cfg, pixels.device)
        x = self.patch_embed(pixels)
        x = ops.pos_embed_add(x, self.pos_embed.weight, plan, self.cfg.spatial_merge_size)
        deep = []
        for i, blk in enumerate(self.blocks):
            if self.ac_mode != "off" and torch.is_grad_enabled():
                from ..parallel.ac import checkpoint_layer

                x = checkpoint_layer(blk, x, plan, "full")
            else:
                x = blk(x, plan)
            if i in self.deepstack_visual_indexes:
                deep.append(self.deepstack_merger_list[self.deepstack_visual_indexes.index(i)](x))
        return self.merger(x), deep

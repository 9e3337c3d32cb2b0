"""Rotary embedding + grouped-query expansion of the packed q / k / v projections: the step
right after the q/k/v GEMM.

Same surface as the reference's `qkv_rotate` (solution/attention.py:149-192): one kernel launch
forward, one backward, outputs fp16 with every k / v head repeated heads / kv_heads times, packed
(N, H, D) or padded (B, H, T, D).
"""

from __future__ import annotations

import torch

from . import _lib
from ._autograd import call


class _RotateOp:
    def __init__(self, batch, seq, heads, kv_heads, padded):
        self.batch, self.seq, self.heads, self.kv_heads = batch, seq, heads, kv_heads
        self.padded = bool(padded)

    def run(self, keep, q, k, v, cos, sin, b_idx, t_idx):
        if not q.is_cuda:
            raise ValueError("hackaton_b200: qkv_rotate needs CUDA tensors (there is no CPU path)")
        if q.dtype not in (torch.float16, torch.float32) or k.dtype != q.dtype or v.dtype != q.dtype:
            raise TypeError(f"hackaton_b200: qkv_rotate takes fp16 or fp32 projections, got {q.dtype}")
        if cos.dtype != torch.float32 or sin.dtype != torch.float32 or cos.dim() != 3:
            raise TypeError("hackaton_b200: qkv_rotate takes fp32 cos / sin of shape (1 or B, T, D)")
        *heads_out, cos, sin, b_idx, t_idx, geo = _lib.host().rotate_fwd(
            q, k, v, cos, sin, b_idx, t_idx, self.batch, self.seq, self.heads, self.kv_heads,
            q.shape[-1] // self.heads, self.padded)
        keep(cos, sin, b_idx, t_idx, geo=geo)
        return tuple(heads_out)

    def grad(self, kept, *head_grads):
        return _lib.host().rotate_bwd(*head_grads, *kept.tensors, kept.geo) + (None, None, None, None)


def qkv_rotate(q, k, v, cos, sin, b_idx, t_idx, batch, seq, heads, kv_heads, padded=False):
    """Packed (q, k, v) projections (N, heads * D) -> rotated, fp16, GQA-expanded heads
    (solution/attention.py:149-192)."""
    return call(_RotateOp(batch, seq, heads, kv_heads, padded), q, k, v, cos, sin, b_idx, t_idx)

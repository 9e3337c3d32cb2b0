"""Grouped launches for projections that sit side by side in the model.

In Qwen2 the q/k/v projections share the post-norm hidden state and gate/up share the MLP input
(the call sites the reference patches: solution/patches.py:32-41 and :98-99). Run one by one,
the small ones (k, v: 256 x 1536) leave most of a B200 idle. Here up to four NF4 weights with the
same number of input features go through ONE fused kernel launch:

    forward :  y_i = x . W_iᵀ (+ bias_i) (+ LoRA_i)        one x, one output per weight
    backward:  dx  = Σ_i dy_i . W_i (+ LoRA_i share)       one dx for the whole group

which is exactly what autograd computes for such a fan-out, only with fewer and fuller launches.
"""

from __future__ import annotations

from dataclasses import dataclass
from typing import Optional, Sequence

import torch

from . import _lib
from .lora import RANK, grad_buffer, lora_grad_batch, lora_side
from .nf4 import _require, _rows, scratch_bytes, streams, weight_ref

MAX_GROUP = 4


@dataclass
class Projection:
    """One member of a group: an NF4 weight and, optionally, its bias and LoRA pair."""
    packed: torch.Tensor
    state: object
    bias: Optional[torch.Tensor] = None
    lora_a: Optional[torch.Tensor] = None   # [16, K]
    lora_b: Optional[torch.Tensor] = None   # [N, 16]
    scaling: float = 1.0


def _workspace(device, rows, cols, m, backward):
    if m == 0:
        return 0
    return scratch_bytes(device, "nf4b200_workspace_bytes_group", len(rows), tuple(rows), cols, m, int(backward))


def _refs(items):
    refs = []
    for packed, state in items:
        packed = packed.reshape(-1)
        _require(packed, state)
        refs.append(weight_ref(packed, state).prepare())
    cols = refs[0].cols
    if any(r.cols != cols for r in refs):
        raise ValueError("grouped projections must have the same number of input features")
    if not 1 <= len(refs) <= MAX_GROUP:
        raise ValueError(f"a group holds 1..{MAX_GROUP} projections, got {len(refs)}")
    return refs


def linear_forward_group(x, weights: Sequence, biases=None, xas=None, lora_bs=None):
    """weights: [(packed, state), ...]. Returns the list of outputs y_i = x . W_iᵀ (+ ...)."""
    refs = _refs(weights)
    none = [None] * len(refs)
    if x.dtype != torch.float16:
        raise TypeError(f"hackaton_b200: the fused NF4 linear computes in fp16, got {x.dtype}")
    cols = refs[0].cols
    if x.shape[-1] != cols:
        raise ValueError(f"input has {x.shape[-1]} features, weights expect {cols}")
    m = _rows(x)
    ws_bytes = 0 if streams(m, *refs) else _workspace(x.device, [r.rows for r in refs], cols, m, False)
    return _lib.host().linear_fwd_group(
        [r.address for r in refs], x, none if biases is None else list(biases), none if xas is None else list(xas),
        none if lora_bs is None else list(lora_bs), ws_bytes)


def linear_backward_dx_group(grads: Sequence[torch.Tensor], weights: Sequence, us=None, lora_as=None):
    """dx = Σ_i grads[i] . W_i (+ u_i . lora_a_i). grads[i]: fp16 [..., N_i]."""
    refs = _refs(weights)
    none = [None] * len(refs)
    for g, r in zip(grads, refs):
        if g.dtype != torch.float16:
            raise TypeError(f"hackaton_b200: the fused NF4 linear computes in fp16, got {g.dtype}")
        if g.shape[-1] != r.rows:
            raise ValueError(f"gradient has {g.shape[-1]} features, weight gives {r.rows}")
    ws_bytes = _workspace(grads[0].device, [r.rows for r in refs], refs[0].cols, _rows(grads[0]), True)
    return _lib.host().linear_bwd_dx_group([r.address for r in refs], list(grads), none if us is None else list(us),
                                           none if lora_as is None else list(lora_as), ws_bytes)


class NF4LinearGroup(torch.autograd.Function):
    """Autograd wrapper: inputs (x, projections, bias_0, A_0, B_0, bias_1, ...), one output per
    projection. Weights are frozen; gradients flow to x, the biases and the LoRA pairs."""

    @staticmethod
    def forward(ctx, x, projs, *params):
        n = len(projs)
        biases, las, lbs = params[0::3], params[1::3], params[2::3]
        xas, b16 = [None] * n, [None] * n
        with_lora = [i for i, a in enumerate(las) if a is not None]
        kept = {}
        if with_lora:  # every adapter's scaling * x . Aᵀ and the fp16 factors in one launch
            train = any(ctx.needs_input_grad)
            downs, a16s, b16s, b16ts = lora_side(
                [x] * len(with_lora), [las[i] for i in with_lora], [projs[i].scaling for i in with_lora],
                [lbs[i] for i in with_lora], transpose=train)
            for i, xa, a, b, bt in zip(with_lora, downs, a16s, b16s, b16ts):
                xas[i], b16[i], kept[i] = xa, b, (a, bt)
        ys = linear_forward_group(x, [(pr.packed, pr.state) for pr in projs], biases, xas, b16)
        ctx.projs, ctx.n = projs, n
        ctx.bias_dtypes = [None if b is None else b.dtype for b in biases]
        ctx.has_lora = [a is not None for a in las]
        if any(ctx.needs_input_grad):
            saved = [x]
            for i in with_lora:
                saved += [las[i], lbs[i], xas[i], *kept[i]]
            ctx.save_for_backward(*saved)
        return tuple(ys)

    @staticmethod
    def backward(ctx, *grads):
        saved = list(ctx.saved_tensors)
        x = saved.pop(0)
        projs = ctx.projs
        lora = []
        for has in ctx.has_lora:
            lora.append(tuple(saved.pop(0) for _ in range(5)) if has else None)   # A, B, xa, A16, Bᵀ16
        grads = [g if g is not None else
                 torch.zeros(*x.shape[:-1], pr.state.shape[0], dtype=torch.float16, device=x.device)
                 for g, pr in zip(grads, projs)]
        us, a16 = [None] * len(projs), [None] * len(projs)
        with_lora = [i for i, lo in enumerate(lora) if lo is not None]
        # all LoRA weight gradients of the group in one launch, summed into a zeroed buffer
        jobs = []  # (z, s or None for u, rank-major output, projection, "a" | "b")
        for i in with_lora:
            if ctx.needs_input_grad[3 + 3 * i]:
                jobs.append((x, None, True, i, "a"))
            if ctx.needs_input_grad[4 + 3 * i]:
                jobs.append((grads[i], lora[i][2], False, i, "b"))
        flat = grad_buffer(jobs, x.device) if jobs else None
        if with_lora:  # every adapter's scaling * dy . B in one launch
            downs, *_ = lora_side([grads[i] for i in with_lora], [lora[i][4] for i in with_lora],
                                  [projs[i].scaling for i in with_lora], zero=flat)
            for i, u in zip(with_lora, downs):
                us[i] = u
                a16[i] = lora[i][3]
        grad_x = None
        if ctx.needs_input_grad[0]:
            grad_x = linear_backward_dx_group(grads, [(pr.packed, pr.state) for pr in projs], us, a16)
        wgrads = {}
        if jobs:
            res = lora_grad_batch([j[0] for j in jobs], [us[j[3]] if j[1] is None else j[1] for j in jobs],
                                  [j[2] for j in jobs], flat)
            for j, r in zip(jobs, res):
                wgrads[j[3:]] = r
        out = [grad_x, None]
        for i, (g, pr, lo) in enumerate(zip(grads, projs, lora)):
            gb = ga = gbb = None
            if ctx.needs_input_grad[2 + 3 * i] and ctx.bias_dtypes[i] is not None:
                gb = g.reshape(-1, g.shape[-1]).sum(0, dtype=ctx.bias_dtypes[i])
            if lo is not None:
                if (i, "a") in wgrads:
                    ga = wgrads[(i, "a")].to(lo[0].dtype)
                if (i, "b") in wgrads:
                    gbb = wgrads[(i, "b")].to(lo[1].dtype)
            out += [gb, ga, gbb]
        return tuple(out)


def nf4_linear_group(x, projections: Sequence[Projection]):
    """Outputs of all `projections` applied to the same x, computed by one grouped launch."""
    params = []
    for pr in projections:
        if (pr.lora_a is None) != (pr.lora_b is None):
            raise ValueError("a projection needs both LoRA factors or none")
        if pr.lora_a is not None and pr.lora_a.shape[0] != RANK:
            raise ValueError(f"LoRA rank must be {RANK}")
        params += [pr.bias, pr.lora_a, pr.lora_b]
    return NF4LinearGroup.apply(x, list(projections), *params)

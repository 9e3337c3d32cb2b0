"""Cross-entropy straight from the lm_head's logits, and lm_head + loss over row chunks.

Same surface as the reference's `ce_stats` / `ce_grad` / `fused_cross_entropy`
(solution/kernels.py:173-238) and `linear_cross_entropy` (solution/lm_loss.py:27-67). The
statistics pass and the gradient pass are this library's kernels (csrc/cross_entropy.cu), and so
are the two fp16 matrix products of a chunk (`dense.fp16_linear`: the tcgen05 kernel of the NF4
projections with the weight tiles brought by TMA).
"""

from __future__ import annotations

import torch

from . import _lib
from ._autograd import call
from .dense import fp16_linear
from .nf4 import _stream_ptr

# Rows of logits alive at a time: CHUNK_ROWS, halved while they would take more than LOGITS_BYTES or more
# than there is, down to MIN_ROWS (the reference's number, solution/lm_loss.py:27). Every chunk reads the
# whole head weight, so more rows pay: 2048 rows x 151,936 from 1536 features, both directions, 2247 us in
# chunks of 512, 2128 of 1024, 2064 in one that holds twice the memory.
CHUNK_ROWS = 1024
MIN_ROWS = 256
LOGITS_BYTES = 320 << 20
# Rows of the gradient's product: one tile of the GEMM. With more, its plan cuts the contraction over the
# vocabulary into fewer slices: longer chains of fp32 additions, and the error of d_hidden against 64 bits
# grows (2048 x 3584: 6.45e-4 with 256 and 512 rows, 6.50e-4 with 1024, 6.68e-4 with 2048).
CHUNK_TILE = 512
GRAD_SCALE = 1024.0   # the chunk gradients are kept in fp16 at this scale (solution/lm_loss.py:28)


def _dtype_code(logits):
    if not logits.is_cuda:
        raise ValueError("hackaton_b200: the cross-entropy kernels need CUDA tensors (there is no CPU path)")
    if logits.dtype == torch.float16:
        return _lib.F16
    if logits.dtype == torch.float32:
        return _lib.F32
    raise TypeError(f"hackaton_b200: logits must be fp16 or fp32, got {logits.dtype}")


def _opt_ptr(t):
    return None if t is None else t.data_ptr()


def ce_stats(logits, targets, want_entropy, out=None):
    """Per-row logsumexp, loss (0 for rows with target < 0) and, if asked, entropy of (rows,
    vocab) logits. `out` = (lse, loss, entropy, argmax) buffers to fill instead of new ones;
    the argmax is only written there (solution/kernels.py:182-204)."""
    rows, vocab = logits.shape
    if targets.dtype != torch.int64:
        raise TypeError("hackaton_b200: targets must be int64")
    if out is None:
        fresh = lambda: torch.empty(rows, dtype=torch.float32, device=logits.device)  # noqa: E731
        out = (fresh(), fresh(), fresh() if want_entropy else None, None)
    lse, loss, entropy, argmax = out
    with torch.cuda.device(logits.device):
        _lib.check(_lib.lib().nf4b200_ce_stats(
            logits.data_ptr(), _dtype_code(logits), targets.data_ptr(), lse.data_ptr(),
            loss.data_ptr(), _opt_ptr(entropy), _opt_ptr(argmax), rows, vocab,
            _stream_ptr(logits.device)))
    return lse, loss, entropy


def ce_grad(logits, targets, lse, scale, grad):
    """grad = scale * (softmax(logits) - onehot(targets)) per row, 0 for rows with target < 0;
    `scale` is one fp32 number on the device; `grad` may be `logits` itself
    (solution/kernels.py:173-179)."""
    rows, vocab = logits.shape
    with torch.cuda.device(logits.device):
        _lib.check(_lib.lib().nf4b200_ce_grad(
            logits.data_ptr(), _dtype_code(logits), targets.data_ptr(), lse.data_ptr(),
            scale.data_ptr(), grad.data_ptr(), rows, vocab, _stream_ptr(logits.device)))


class _LossFromLogits:
    """sum over rows of (logsumexp - logit[target]) / denom; the gradient may overwrite the
    logits."""

    def __init__(self, overwrite_logits):
        self.overwrite_logits = overwrite_logits

    def run(self, keep, logits, targets, denom):
        lse, per_row, _ = ce_stats(logits, targets, False)
        keep(logits, targets, lse, denom)
        return per_row.sum() / denom

    def grad(self, kept, upstream):
        logits, targets, lse, denom = kept.tensors
        d_logits = logits if self.overwrite_logits else torch.empty_like(logits)
        ce_grad(logits, targets, lse, (upstream / denom).float().reshape(1), d_logits)
        return d_logits, None, None


def fused_cross_entropy(logits, targets, denom, inplace_grad=False):
    """Mean-style loss of (rows, vocab) logits, rows with target < 0 ignored
    (solution/kernels.py:207-238)."""
    return call(_LossFromLogits(bool(inplace_grad)), logits.contiguous(), targets, denom)


def _head_products(hidden_rows, weight, logits):
    """The two matrix products of one chunk: logits = hidden_rows . weightᵀ, and, once the logits
    have been turned into their gradient, d_hidden = d_logits . weight. fp16 weights (the model's
    own lm_head) go through this library's tcgen05 kernel; other dtypes (a test in fp32) use
    torch's matmul. Returns the second one."""
    if hidden_rows.dtype == torch.float16 and weight.dtype == torch.float16:
        fp16_linear(hidden_rows, weight, out=logits)
        return lambda d_logits, out: fp16_linear(d_logits, weight, transposed=True, out=out)
    torch.mm(hidden_rows, weight.t(), out=logits)
    return lambda d_logits, out: torch.mm(d_logits, weight, out=out)


def _chunk_rows(vocab, itemsize):
    """Rows of (rows, vocab) logits that LOGITS_BYTES allows."""
    rows = CHUNK_ROWS
    while rows > MIN_ROWS and rows * vocab * itemsize > LOGITS_BYTES:
        rows //= 2
    return rows


def _logits_buffer(rows, vocab, like):
    """Room for the logits of a chunk of at most `rows` rows."""
    step = _chunk_rows(vocab, like.element_size())
    while True:
        try:
            return torch.empty(min(step, rows), vocab, dtype=like.dtype, device=like.device)
        except torch.OutOfMemoryError:
            if step <= MIN_ROWS:
                raise
            step //= 2


def _chunks(rows, step=None):
    """Row slices of `step` (CHUNK_ROWS) rows, the last one with what is left: few rows take the GEMM's
    smaller tiles, so a short chunk costs less than chunks of equal size in part-filled tiles."""
    step = step or CHUNK_ROWS
    return [slice(lo, min(lo + step, rows)) for lo in range(0, rows, step)]


class _HeadAndLoss:
    """lm_head + loss without ever holding the (tokens, vocab) logits: walks the rows in chunks;
    per chunk the logits are made, reduced to their statistics, turned in place into
    GRAD_SCALE * (softmax - onehot) and multiplied back through the (frozen) head weight, so the
    gradient with respect to `hidden` exists when the forward ends and the backward only rescales
    it (solution/lm_loss.py:31-62)."""

    def run(self, keep, hidden, weight, targets, denom):
        rows, device = hidden.shape[0], hidden.device
        stats = {name: torch.empty(rows, dtype=torch.float32, device=device)
                 for name in ("lse", "loss", "entropy")}
        argmax = torch.empty(rows, dtype=torch.int64, device=device)
        d_hidden = torch.empty_like(hidden)
        unit = torch.full((1,), GRAD_SCALE, dtype=torch.float32, device=device)
        with torch.autocast("cuda", enabled=False):
            buffer = _logits_buffer(rows, weight.shape[0], hidden)
            for rs in _chunks(rows, buffer.shape[0]):
                logits = buffer[:rs.stop - rs.start]
                back = _head_products(hidden[rs], weight, logits)
                ce_stats(logits, targets[rs], True,
                         out=(stats["lse"][rs], stats["loss"][rs], stats["entropy"][rs], argmax[rs]))
                ce_grad(logits, targets[rs], stats["lse"][rs], unit, logits)
                for part in _chunks(logits.shape[0], CHUNK_TILE):
                    back(logits[part], d_hidden[rs][part])
        keep(d_hidden, denom)
        keep.constant(stats["loss"], stats["entropy"], argmax)
        return stats["loss"].sum() / denom, stats["loss"], stats["entropy"], argmax

    def grad(self, kept, upstream, *_unused):
        d_hidden, denom = kept.tensors
        factor = (upstream.float() / (denom * GRAD_SCALE)).reshape(1, 1)
        return (d_hidden.float() * factor).to(d_hidden.dtype), None, None, None


def linear_cross_entropy(hidden, weight, targets, denom):
    """(loss, per-row losses, entropy, argmax) of hidden @ weightᵀ against `targets`
    (solution/lm_loss.py:65-67)."""
    return call(_HeadAndLoss(), hidden.contiguous(), weight, targets, denom)

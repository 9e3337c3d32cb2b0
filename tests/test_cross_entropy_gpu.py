"""GPU: cross-entropy statistics / gradient kernels and the chunked lm_head + loss through the
C ABI against the reference kernel's golden vectors, the oracle and plain PyTorch."""

from pathlib import Path

import numpy as np
import pytest
import torch

from oracle import nf4_oracle

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"


@pytest.mark.parametrize("name", ["ragged", "blocks"])    # 9,001 logits: scalar path; 4,096: vectors
@pytest.mark.parametrize("tag", ["f16", "f32"])
def test_matches_reference_kernel(cuda_lib, name, tag):
    from hackaton_b200.lm_loss import ce_grad, ce_stats

    z = np.load(GOLDEN / "ce_small.npz")
    t = lambda key: torch.from_numpy(z[f"{name}_{tag}_{key}"])
    logits, targets = t("logits").cuda(), torch.from_numpy(z[f"{name}_targets"]).cuda()
    rows = logits.shape[0]
    out = (torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda"),
           torch.empty(rows, dtype=torch.int64, device="cuda"))
    lse, loss, entropy = ce_stats(logits, targets, True, out=out)
    torch.testing.assert_close(lse.cpu(), t("lse"), rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(loss.cpu(), t("loss"), rtol=1e-5, atol=2e-5)
    torch.testing.assert_close(entropy.cpu(), t("entropy"), rtol=1e-4, atol=1e-4)
    assert torch.equal(out[3].cpu(), t("argmax"))
    assert float(lse[2]) == 0.0 and float(loss[2]) == 0.0
    scale = torch.tensor([0.37], device="cuda")
    grad = torch.empty_like(logits)
    ce_grad(logits, targets, lse, scale, grad)
    tol = dict(rtol=2e-3, atol=1e-6) if tag == "f16" else dict(rtol=1e-4, atol=1e-7)
    torch.testing.assert_close(grad.cpu().float(), t("grad").float(), **tol)
    assert not bool(grad[2].any())
    work = logits.clone()
    ce_grad(work, targets, lse, scale, work)                   # in place: the same bits
    assert torch.equal(work, grad)
    cuda_lib.device_status()


@pytest.mark.parametrize("rows,vocab,dtype", [(64, 151936, torch.float16), (33, 32000, torch.float32),
                                              (5, 1001, torch.float16)])
def test_fused_cross_entropy_matches_pytorch(cuda_lib, rows, vocab, dtype):
    from hackaton_b200.lm_loss import ce_stats, fused_cross_entropy

    g = torch.Generator(device="cuda").manual_seed(rows + vocab)
    logits = (torch.randn(rows, vocab, device="cuda", generator=g) * 4).to(dtype).requires_grad_()
    targets = torch.randint(0, vocab, (rows,), device="cuda", generator=g)
    targets[1] = -100
    denom = (targets >= 0).sum().float()
    ref = torch.nn.functional.cross_entropy(logits.float(), targets, ignore_index=-100, reduction="sum") / denom
    ref.backward()
    ref_grad = logits.grad.clone()
    logits.grad = None
    loss = fused_cross_entropy(logits, targets, denom)
    loss.backward()
    torch.testing.assert_close(loss, ref, rtol=1e-5, atol=1e-5)
    tol = dict(rtol=2e-3, atol=1e-6) if dtype == torch.float16 else dict(rtol=1e-4, atol=1e-8)
    torch.testing.assert_close(logits.grad.float(), ref_grad.float(), **tol)
    # statistics against the oracle on the same logits
    lse, losses, entropy = ce_stats(logits.detach(), targets, True)
    o_lse, o_loss, o_ent, o_arg = nf4_oracle.ce_stats(logits.detach().cpu(), targets.cpu())
    torch.testing.assert_close(lse.cpu(), o_lse, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(losses.cpu(), o_loss, rtol=1e-5, atol=2e-5)
    torch.testing.assert_close(entropy.cpu(), o_ent, rtol=1e-4, atol=1e-4)
    cuda_lib.device_status()


def test_linear_cross_entropy_matches_unchunked(cuda_lib):
    """solution/lm_loss.py: the chunked lm_head + loss gives the loss, metrics and d loss / d hidden
    of the plain computation (600 rows = three chunks, the last one ragged)."""
    from hackaton_b200.lm_loss import linear_cross_entropy

    g = torch.Generator(device="cuda").manual_seed(11)
    rows, hidden_size, vocab = 600, 256, 5000
    hidden = (torch.randn(rows, hidden_size, device="cuda", generator=g) * 0.5).half().requires_grad_()
    weight = (torch.randn(vocab, hidden_size, device="cuda", generator=g) * 0.1).half()
    targets = torch.randint(0, vocab, (rows,), device="cuda", generator=g)
    targets[::7] = -100
    denom = (targets >= 0).sum().float()
    logits = torch.nn.functional.linear(hidden, weight)
    ref = torch.nn.functional.cross_entropy(logits.float(), targets, ignore_index=-100, reduction="sum") / denom
    ref.backward()
    ref_grad = hidden.grad.clone()
    hidden.grad = None
    loss, losses, entropy, argmax = linear_cross_entropy(hidden, weight, targets, denom)
    loss.backward()
    torch.testing.assert_close(loss, ref, rtol=1e-4, atol=1e-4)
    assert torch.equal(argmax, torch.argmax(logits.float(), dim=-1))
    o = nf4_oracle.ce_stats(logits.detach().cpu(), targets.cpu())
    torch.testing.assert_close(losses.cpu(), o[1], rtol=1e-4, atol=1e-4)
    torch.testing.assert_close(entropy.cpu(), o[2], rtol=1e-3, atol=1e-3)
    torch.testing.assert_close(hidden.grad.float(), ref_grad.float(), rtol=2e-2, atol=2e-6)
    cuda_lib.device_status()


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("rows", [3, 593, 1185])                       # 512, 256 and 128 threads per row
@pytest.mark.parametrize("vocab", [1, 8, 1023, 8192, 8200, 16392])     # below, at and past a CTA's 8192 logits
def test_thread_counts_and_segments(cuda_lib, rows, vocab, dtype):
    """Every kernel the launcher picks, statistics and in-place gradient, against 64-bit arithmetic.
    Bounds: a sum of `vocab` fp32 terms of one sign (1e-5 covers it), the ex2 approximation (2^-22)
    and, for the fp16 gradient, one rounding of a value of at most 1024."""
    from hackaton_b200.lm_loss import ce_grad, ce_stats

    g = torch.Generator(device="cuda").manual_seed(rows + vocab)
    logits = (torch.randn(rows, vocab, generator=g, device="cuda") * 3).to(dtype)
    targets = torch.randint(0, vocab, (rows,), generator=g, device="cuda")
    targets[::5] = -100
    valid = targets >= 0
    out = tuple(torch.empty(rows, device="cuda") for _ in range(3)) + (
        torch.empty(rows, dtype=torch.int64, device="cuda"),)
    ce_stats(logits, targets, True, out=out)
    logp = torch.log_softmax(logits.double(), -1)
    want = torch.logsumexp(logits.double(), -1)
    picked = logp.gather(1, targets.clamp(min=0)[:, None])[:, 0]
    close = lambda a, b, t: torch.testing.assert_close(a.double(), b, rtol=t, atol=t)  # noqa: E731
    close(out[0][valid], want[valid], 1e-5)
    close(out[1], torch.where(valid, -picked, 0.0), 2e-5)
    close(out[2], -(logp.exp() * logp).sum(-1), 1e-4)
    at = torch.arange(vocab, device="cuda")          # the first of equal maxima (common in fp16)
    assert torch.equal(out[3], torch.where(logits == logits.amax(-1, keepdim=True), at, vocab).amin(-1))
    grad = logp.exp()
    grad.scatter_add_(1, targets.clamp(min=0)[:, None], torch.full_like(grad[:, :1], -1.0))
    grad = torch.where(valid[:, None], grad * 1024, 0.0)
    ce_grad(logits, targets, out[0], torch.full((1,), 1024.0, device="cuda"), logits)
    close(logits, grad, 1e-3)
    assert not logits[~valid].any()
    cuda_lib.device_status()


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("sms,extra", [(1, 0), (1, 1), (2, 0), (2, 1), (4, 0), (4, 1), (8, 0), (8, 1)])
@pytest.mark.parametrize("vocab", [65528, 65536, 65537, 8191])     # wide from 65,536 logits on; 16-byte rows or not
def test_thread_counts_follow_rows_and_vocabulary(cuda_lib, vocab, sms, extra, dtype):
    """Both sides of every line of the statistics' rule: rows against multiples of the SM count."""
    rows = sms * torch.cuda.get_device_properties(0).multi_processor_count + extra
    test_thread_counts_and_segments(cuda_lib, rows, vocab, dtype)


@pytest.mark.parametrize("rows", [2048, 2049, 2600])
def test_chunks_cover_the_rows(cuda_lib, rows):
    """Chunked against plain computation around the chunk limit (whole chunks, a last one of one row, a part-filled one)."""
    from hackaton_b200.lm_loss import CHUNK_ROWS, _chunks, linear_cross_entropy

    parts = _chunks(rows)
    assert [p.start for p in parts] == [0] + [p.stop for p in parts[:-1]] and parts[-1].stop == rows
    assert max(p.stop - p.start for p in parts) <= CHUNK_ROWS
    g = torch.Generator(device="cuda").manual_seed(rows)
    hidden = (torch.randn(rows, 64, device="cuda", generator=g) * 0.5).half().requires_grad_()
    weight = (torch.randn(1000, 64, device="cuda", generator=g) * 0.1).half()
    targets = torch.randint(0, 1000, (rows,), device="cuda", generator=g)
    denom = torch.tensor(float(rows), device="cuda")
    logits = (hidden.detach().double() @ weight.double().t()).requires_grad_()
    ref = torch.nn.functional.cross_entropy(logits, targets)
    want = torch.autograd.grad(ref, logits)[0] @ weight.double()
    loss, *_ = linear_cross_entropy(hidden, weight, targets, denom)
    grad, = torch.autograd.grad(loss, hidden)
    torch.testing.assert_close(loss.double(), ref, rtol=1e-4, atol=1e-4)
    assert (grad.double() - want).norm() <= 5e-3 * want.norm()   # fp16 logits, gradients and sums


@pytest.mark.parametrize("hidden_size", [1536, 3584])
def test_chunk_size_does_not_move_the_gradient(cuda_lib, monkeypatch, hidden_size):
    """The chunks in use give what the reference's 256 rows give, up to the order of the fp32 sums of
    the softmax statistics (their 1e-6 moves a few fp16 roundings of the logits' gradient): 1e-5. With
    more rows in the gradient's product its longer chains of fp32 additions make it 1e-4 to 2e-4."""
    from hackaton_b200 import lm_loss

    g = torch.Generator(device="cuda").manual_seed(hidden_size)
    hidden = torch.randn(2560, hidden_size, device="cuda", generator=g).half().requires_grad_()
    weight = (torch.randn(151_936, hidden_size, device="cuda", generator=g) * 0.04).half()
    targets = torch.randint(0, 151_936, (2560,), device="cuda", generator=g)
    denom = torch.tensor(2560.0, device="cuda")

    def run():
        loss, losses, entropy, argmax = lm_loss.linear_cross_entropy(hidden, weight, targets, denom)
        return losses, argmax, torch.autograd.grad(loss, hidden)[0]

    now = run()
    monkeypatch.setattr(lm_loss, "CHUNK_ROWS", 256)
    losses, argmax, grad = run()
    assert torch.equal(now[1], argmax)
    assert float((now[0] - losses).norm()) <= 1e-6 * float(losses.norm())
    assert float((now[2].double() - grad.double()).norm()) <= 1e-5 * float(grad.double().norm())
    cuda_lib.device_status()

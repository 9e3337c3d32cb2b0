"""GPU: LoRA r=16 fused into the NF4 linear (forward, dX, dA, dB) against the oracle formula.
Parity unpinned: the reference has no LoRA test (peft's code is third-party)."""

import pytest
import torch

from oracle import nf4_oracle
from tests.util import oracle_weight, synthetic_weight

pytestmark = pytest.mark.gpu
TOL = 1e-2


def make(m, n, k, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(m, k, generator=g).half()
    dy = torch.randn(m, n, generator=g).half()
    a = ((torch.rand(16, k, generator=g) * 2 - 1) / k ** 0.5).half()   # U(+-1/sqrt(K))
    b = (torch.randn(n, 16, generator=g) * 0.01).half()                # N(0, 0.01)
    return x, dy, a, b


@pytest.mark.parametrize("m,n,k", [(2048, 1536, 1536), (300, 256, 1536), (77, 264, 192),
                                   (1, 256, 64), (128, 512, 128)])
def test_lora_forward_backward_vs_oracle(cuda_lib, m, n, k):
    from hackaton_b200 import nf4_lora_linear

    packed, state = synthetic_weight(n, k, True, seed=m + n, device="cuda")
    w = oracle_weight(packed, state)
    x, dy, a, b = make(m, n, k, seed=m)
    # make the low-rank term visible next to the base product
    b = b * 20
    scaling = 2.0
    xg = x.cuda().requires_grad_()
    ag = a.cuda().requires_grad_()
    bg = b.cuda().requires_grad_()
    y = nf4_lora_linear(xg, packed, None, state, ag, bg, scaling)
    y.backward(dy.cuda())
    torch.cuda.synchronize()
    y_ref, _ = nf4_oracle.lora_fwd(x, w, a, b, scaling)
    dx_ref, da_ref, db_ref = nf4_oracle.lora_bwd(dy, x, w, a, b, scaling)
    assert nf4_oracle.max_rel_err(y.cpu(), y_ref) <= TOL
    assert nf4_oracle.max_rel_err(xg.grad.cpu(), dx_ref) <= TOL
    assert nf4_oracle.max_rel_err(ag.grad.cpu(), da_ref) <= TOL
    assert nf4_oracle.max_rel_err(bg.grad.cpu(), db_ref) <= TOL
    # the low-rank term really is in there
    base = nf4_oracle.linear_fwd(x, w)
    assert nf4_oracle.max_rel_err(base, y_ref) > 5 * TOL
    cuda_lib.device_status()


def test_lora_with_dropout_branch(cuda_lib):
    """x_lora != x (peft's lora_dropout in training): the two input gradients stay separate."""
    from hackaton_b200 import nf4_lora_linear

    m, n, k = 200, 256, 128
    packed, state = synthetic_weight(n, k, True, seed=1, device="cuda")
    w = oracle_weight(packed, state)
    x, dy, a, b = make(m, n, k, seed=3)
    b = b * 20
    g = torch.Generator().manual_seed(5)
    mask = (torch.rand(m, k, generator=g) > 0.05).half() / 0.95
    xl = (x * mask).half()
    xg, xlg = x.cuda().requires_grad_(), xl.cuda().requires_grad_()
    y = nf4_lora_linear(xg, packed, None, state, a.cuda(), b.cuda(), 2.0, x_lora=xlg)
    y.backward(dy.cuda())
    y_ref = (x.float() @ w.float().t() + 2.0 * (xl.float() @ a.float().t()) @ b.float().t())
    assert nf4_oracle.max_rel_err(y.cpu(), y_ref) <= TOL
    assert nf4_oracle.max_rel_err(xg.grad.cpu(), dy.float() @ w.float()) <= TOL
    dxl_ref = 2.0 * (dy.float() @ b.float()) @ a.float()
    assert nf4_oracle.max_rel_err(xlg.grad.cpu(), dxl_ref) <= TOL


def test_batched_lora_kernels_match_single(cuda_lib):
    """nf4b200_lora_down_batch / _grad_batch: same results as one call per problem."""
    from hackaton_b200.lora import lora_down, lora_down_batch, lora_grad, lora_grad_batch

    torch.manual_seed(11)
    m = 777
    x = torch.randn(m, 1536, device="cuda").half()
    a_q = (torch.randn(16, 1536, device="cuda") * 0.05).half()
    a_v = (torch.randn(16, 1536, device="cuda") * 0.05).half()
    got = lora_down_batch([x, x], [a_q, a_v], True, [2.0, 0.5])
    want = [lora_down(x, a_q, True, 2.0), lora_down(x, a_v, True, 0.5)]
    for g, w in zip(got, want):
        assert torch.equal(g, w)

    dy_q = torch.randn(m, 1536, device="cuda").half()
    dy_v = torch.randn(m, 256, device="cuda").half()
    b_q = (torch.randn(1536, 16, device="cuda") * 0.05).half()
    b_v = (torch.randn(256, 16, device="cuda") * 0.05).half()
    got = lora_down_batch([dy_q, dy_v], [b_q, b_v], False, [2.0, 2.0])
    want = [lora_down(dy_q, b_q, False, 2.0), lora_down(dy_v, b_v, False, 2.0)]
    for g, w in zip(got, want):
        assert torch.equal(g, w)

    u_q, u_v = want
    xa_q, xa_v = lora_down(x, a_q, True, 2.0), lora_down(x, a_v, True, 2.0)
    got = lora_grad_batch([x, dy_q, x, dy_v], [u_q, xa_q, u_v, xa_v], [True, False, True, False])
    want = [lora_grad(x, u_q, True), lora_grad(dy_q, xa_q, False), lora_grad(x, u_v, True),
            lora_grad(dy_v, xa_v, False)]
    for g, w in zip(got, want):
        assert g.shape == w.shape
        # fp32 atomics: the order of the block sums is not fixed
        assert (g - w).abs().max() <= 1e-4 * w.abs().max().clamp_min(1.0)


@pytest.mark.parametrize("m", [1, 15, 16, 17, 300])
@pytest.mark.parametrize("c,n", [(8, 8), (64, 264), (1544, 1536), (3584, 512)])   # ragged chunks of 32 columns
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_side_kernel(cuda_lib, m, c, n, dtype):
    """Products, fp16 copies, transpose and zeros of nf4b200_lora_side: copies exactly torch's rounding;
    products against 64-bit sums of the fp16 factors (fp32 accumulation and one fp16 rounding)."""
    from hackaton_b200.lora import lora_side

    g = torch.Generator(device="cuda").manual_seed(m + c)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    xs = [rand(m, c).half(), rand(m, c + 8).half()[:, :c]]
    ps, bs = [rand(16, c).to(dtype) for _ in range(2)], [rand(n, 16).to(dtype) for _ in range(2)]
    zero = rand(52)
    outs, p16s, b16s, b16ts = lora_side(xs, ps, [2.0, 0.5], bs, transpose=True, zero=zero)
    for x, p, b, s, o, p16, b16, bt in zip(xs, ps, bs, (2.0, 0.5), outs, p16s, b16s, b16ts):
        assert torch.equal(p16, p.half()) and torch.equal(b16, b.half()) and torch.equal(bt, b.half().t())
        want = s * x.double() @ p.half().double().t()
        scale = s * (x.double().abs() @ p.half().double().abs().t())
        assert ((o.double() - want).abs() <= 2.0 ** -11 * want.abs() + 1e-6 * scale + 1e-7).all()
    assert not zero.any()


def test_unmodified_when_only_b_needs_a_gradient(cuda_lib):
    """The gradient buffer is zeroed on every path (here: no product in the backward zeroes it)."""
    from hackaton_b200 import nf4_lora_linear

    packed, state = synthetic_weight(64, 128, True, seed=1, device="cuda")
    x = torch.randn(40, 128, device="cuda").half()
    a, b = torch.randn(16, 128, device="cuda"), torch.randn(64, 16, device="cuda", requires_grad=True)
    junk = torch.full((1 << 16,), 7.0, device="cuda")
    del junk                                   # a later allocation of this size is not zero
    y = nf4_lora_linear(x, packed, None, state, a, b, 2.0)
    gy = torch.randn_like(y)
    grad, = torch.autograd.grad(y, b, gy)
    want = gy.double().t() @ (2.0 * x.double() @ a.half().double().t()).half().double()
    assert float((grad.double() - want).abs().max()) <= 1e-3 * float(want.abs().max())


@pytest.mark.parametrize("c,offset", [(100, 0), (64, 3), (20, 1)])
def test_side_products_of_ragged_inputs(cuda_lib, c, offset):
    """Columns or addresses in no whole 16-byte pieces (the gradient of a weight with such a number of
    rows): the layout-agnostic product and copies by torch, same results."""
    from hackaton_b200.lora import lora_side

    x = torch.randn(12 * c + offset, device="cuda").half()[offset:].view(12, c)
    p, b, zero = torch.randn(16, c, device="cuda"), torch.randn(24, 16, device="cuda"), torch.ones(64, device="cuda")
    (o,), (p16,), (b16,), (bt,) = lora_side([x], [p], [0.5], [b], transpose=True, zero=zero)
    want = 0.5 * x.double() @ p.half().double().t()
    assert float((o.double() - want).abs().max()) <= 1e-3 * float(want.abs().max())
    assert torch.equal(p16, p.half()) and torch.equal(b16, b.half()) and torch.equal(bt, b.half().t())
    assert not zero.any()


def test_operands_that_do_not_fit_are_refused(cuda_lib):
    """A bias, a rank-16 operand or a gradient with too few rows is refused on the host, alone and in a
    group; the right sizes pass."""
    from hackaton_b200.group import linear_backward_dx_group, linear_forward_group
    from hackaton_b200.nf4 import linear_backward_dx, linear_forward

    n, k, m = 128, 192, 6
    w = synthetic_weight(n, k, True, seed=1, device="cuda")
    x, dy = (torch.randn(m, c, device="cuda").half() for c in (k, n))
    half = lambda *shape: torch.zeros(*shape, device="cuda", dtype=torch.float16)  # noqa: E731
    linear_forward(x, w[0], half(n), w[1], xa=half(m, 16), lora_b=half(n, 16))
    linear_backward_dx(dy, *w, u=half(m, 16), lora_a=half(16, k))
    for bias, xa, b in ((half(n - 8), None, None), (None, half(m - 1, 16), half(n, 16)),
                        (None, half(m, 16), half(n - 8, 16)), (None, half(m, 16), None)):
        with pytest.raises(RuntimeError):
            linear_forward(x, w[0], bias, w[1], xa=xa, lora_b=b)
        with pytest.raises(RuntimeError):
            linear_forward_group(x, [w], [bias], [xa], [b])
    for u, a in ((half(m - 1, 16), half(16, k)), (half(m, 16), half(15, k)), (None, half(16, k))):
        with pytest.raises(RuntimeError):
            linear_backward_dx(dy, *w, u=u, lora_a=a)
        with pytest.raises(RuntimeError):
            linear_backward_dx_group([dy], [w], [u], [a])
    with pytest.raises(RuntimeError):
        linear_backward_dx_group([dy, dy[:2]], [w, w])
    cuda_lib.device_status()

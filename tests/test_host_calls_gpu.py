"""GPU: the native call path (csrc/host.cpp) with several threads and streams."""

import threading
import time

import pytest
import torch

from tests.util import synthetic_weight

pytestmark = pytest.mark.gpu


def _busy(seconds):
    """Keeps the current stream's GPU work waiting for about that long (a bounded spin)."""
    torch.cuda._sleep(int(seconds * 1.9e9))


def _calls():
    """One call of every function of the module: name -> (inputs, function of the inputs)."""
    from hackaton_b200 import Projection, add_rms_norm, nf4_linear, nf4_linear_group, qkv_rotate, rms_norm

    g = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *shape, dtype=torch.float16: torch.randn(  # noqa: E731
        *shape, generator=g, device="cuda").to(dtype).requires_grad_()
    m, h = 70, 512
    q, k, v = (synthetic_weight(n, h, True, seed=n, device="cuda") for n in (512, 128, 128 + 16))
    lora = [rand(16, h, dtype=torch.float32), rand(512, 16, dtype=torch.float32)]
    weight = torch.ones(h, device="cuda")
    cos, sin = torch.rand(1, m, 128, device="cuda"), torch.rand(1, m, 128, device="cuda")
    at = torch.arange(m, device="cuda", dtype=torch.int32)
    return {
        "linear": ([rand(m, h)], lambda x: nf4_linear(x, k[0], None, k[1])),
        "group": ([rand(m, h), *lora], lambda x, a, b: nf4_linear_group(
            x, [Projection(*q, None, a, b, 2.0), Projection(*k), Projection(*v)])),
        "norm": ([rand(m, h, dtype=torch.float32)], lambda x: rms_norm(x, weight, 1e-6, to_half=True)),
        "add_norm": ([rand(m, h, dtype=torch.float32), rand(m, h)],
                     lambda x, d: add_rms_norm(x, d, weight, 1e-6, to_half=True)),
        "rotate": ([rand(m, 4 * 128), rand(m, 128), rand(m, 128)],
                   lambda a, b, c: qkv_rotate(a, b, c, cos, sin, at * 0, at, 1, m, 4, 1)),
    }


def _both_ways(inputs, fn):
    outs = fn(*inputs)
    outs = list(outs) if isinstance(outs, (tuple, list)) else [outs]
    grads = torch.autograd.grad(outs, inputs, [torch.ones_like(o) for o in outs])
    return [t.detach() for t in outs] + list(grads)


def _same(a, b):
    # (the LoRA gradients are summed atomically: the order of the fp32 sums)
    return all(x.shape == y.shape and float((x.double() - y.double()).norm()) <= 1e-5 * float(y.double().norm())
               for x, y in zip(a, b))


@pytest.mark.parametrize("name", ["linear", "group", "norm", "add_norm", "rotate"])
def test_calls_run_on_the_current_stream(cuda_lib, name):
    """On a side stream the calls come after the stream's own earlier work: their inputs are written there
    behind a wait, and a launch on another stream would read them before that."""
    inputs, fn = _calls()[name]
    want = _both_ways(inputs, fn)
    late = [torch.zeros_like(t).requires_grad_() for t in inputs]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        _busy(0.02)
        with torch.no_grad():
            for t, value in zip(late, inputs):
                t.copy_(value)
        got = _both_ways(late, fn)
    torch.cuda.synchronize()
    assert _same(got, want)
    cuda_lib.device_status()


@pytest.mark.parametrize("own_streams", [False, True])
def test_calls_of_two_threads(cuda_lib, own_streams):
    """Two threads, on the same stream or on two, each with its own inputs, some of them split along K
    with scratch and a second launch: both get what one alone gets."""
    from hackaton_b200.nf4 import linear_backward_dx, linear_forward, prepare_weights

    calls = _calls()
    down = synthetic_weight(256, 4096, True, seed=9, device="cuda")
    prepare_weights([down])
    g = torch.Generator(device="cuda").manual_seed(6)
    xs = [torch.randn(300, 4096, generator=g, device="cuda").half() for _ in range(2)]
    dys = [torch.randn(300, 256, generator=g, device="cuda").half() for _ in range(2)]

    def work(i):
        out = [linear_forward(xs[i], *down[:1], None, down[1]), linear_backward_dx(dys[i], *down)]
        for name in ("group", "add_norm", "rotate"):
            inputs, fn = calls[name]
            out += _both_ways([(t.detach() * (1 + i)).requires_grad_() for t in inputs], fn)
        return out

    want = [work(0), work(1)]
    torch.cuda.synchronize()
    wrong = []

    def run(i):
        try:
            stream = torch.cuda.Stream() if own_streams else torch.cuda.default_stream()
            with torch.cuda.stream(stream):
                for _ in range(20):
                    got = work(i)
                    stream.synchronize()
                    if not _same(got, want[i]):
                        wrong.append(i)
        except BaseException as e:  # noqa: BLE001
            wrong.append(repr(e))

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    cuda_lib.device_status()


def test_a_blocked_launch_leaves_the_interpreter_free(cuda_lib):
    """With the launch queue full a call waits for the GPU; other Python threads run meanwhile. The queue
    is filled behind a wait of 0.4 s, so that a call which held the interpreter's lock would stop the
    other thread for most of that."""
    from hackaton_b200.nf4 import linear_forward

    packed, state = synthetic_weight(64, 64, True, seed=1, device="cuda")
    x = torch.randn(4, 64, device="cuda").half()
    linear_forward(x, packed, None, state)
    torch.cuda.synchronize()
    done, gaps = threading.Event(), [0.0]

    def tick():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps[0] = max(gaps[0], now - last)
            last = now

    watcher = threading.Thread(target=tick)
    watcher.start()
    start = time.perf_counter()
    _busy(0.4)
    for _ in range(4000):     # more launches than a queue holds
        linear_forward(x, packed, None, state)
    blocked = time.perf_counter() - start
    torch.cuda.synchronize()
    done.set()
    watcher.join()
    assert blocked > 0.25, "the queue never filled: the test shows nothing"
    assert gaps[0] < 0.1, gaps[0]
    cuda_lib.device_status()

"""Cases that stand for what a QLoRA fine-tuning or serving program has this package compute.

Sizes are those of the two networks the package's tests and benchmark use (hidden 1536 / MLP 8960 /
12 + 2 heads and hidden 3584 / MLP 18944 / 28 + 4 heads, vocabulary 151,936) and ragged ones around
them. `listed` names the fixed cases, `draw` makes others from the same ranges, `prepare` builds
what a program holds before the call, `run` is one pass, `exact` the same result in 64 bits from
plain torch, `work` the bytes and operations a pass cannot do without.

Weights are NF4 codes drawn as often as Gaussian weights with a block maximum of 2.4 standard
deviations have them (zero mean, so that a deep stack of them stays well conditioned), with
double-quantised block scales of the size that initialised weights have: around 0.05 (a weight
with standard deviation 0.02) for 1536 input features, less by the square root for more of them.
"""

import math
import statistics

import torch

VOCAB = 151936
SMALL = {"hidden": 1536, "mlp": 8960, "heads": 12, "kv_heads": 2}
LARGE = {"hidden": 3584, "mlp": 18944, "heads": 28, "kv_heads": 4}
DIM = 128            # elements of an attention head
EPS = 1e-6
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}

# The NF4 data type (QLoRA, arXiv:2305.14314, appendix E).
LEVELS = (
    -1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453,
    -0.28444138169288635, -0.18477343022823334, -0.09105003625154495, 0.0,
    0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224,
    0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0,
)

# The code of each of 256 equally likely Gaussian values.
_NORMAL = statistics.NormalDist()
CODES = [min(range(16), key=lambda c: abs(LEVELS[c] - _NORMAL.inv_cdf((i + 0.5) / 256) / 2.4))
         for i in range(256)]


def listed():
    return [
        # one projection of one token: the smallest call, all latency
        {"name": "linear_1_token", "kind": "linear", "tokens": 1, "out": 1536, "in": 1536},
        # one new token through the whole stack and the head, the step captured once and replayed
        {"name": "decode_1_token", "kind": "decode", "tokens": 1, "layers": 28, **SMALL},
        # sixteen sequences served together on the larger network
        {"name": "decode_16_tokens_large", "kind": "decode", "tokens": 16, "layers": 28, **LARGE},
        # sixty-four sequences served together
        {"name": "decode_64_tokens", "kind": "decode", "tokens": 64, "layers": 28, **SMALL},
        # attention projections with LoRA in training, packed sequences of no round length
        {"name": "attn_train_packed", "kind": "attn", "tokens": 810, **SMALL},
        # the same on the larger network with a full batch
        {"name": "attn_train_large", "kind": "attn", "tokens": 4096, **LARGE},
        # the MLP of a training step
        {"name": "mlp_train", "kind": "mlp", "tokens": 2048, "train": True, **SMALL},
        # the MLP over a long prompt, no gradients: the largest call
        {"name": "mlp_prefill_large", "kind": "mlp", "tokens": 8192, "train": False, **LARGE},
        # residual add + norm, both directions, a full batch of packed tokens
        {"name": "norm_train", "kind": "norm", "tokens": 16384, "hidden": 1536},
        # rotary embedding and head expansion, both directions
        {"name": "rope_train", "kind": "rope", "tokens": 16384, "seq": 2048, "padded": False,
         "dtype": "fp16", "heads": 12, "kv_heads": 2},
        # lm_head and loss of a training step, both directions
        {"name": "lm_loss_train", "kind": "loss", "tokens": 2048, "hidden": 1536, "vocab": VOCAB},
        # a whole weight decoded, as for merging an adapter or exporting a checkpoint
        {"name": "dequant_large", "kind": "dequant", "rows": 18944, "cols": 3584, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "decode", "decode", "attn", "attn", "mlp", "mlp", "norm", "rope",
                       "loss", "dequant"])
    large = rng.random() < 0.35
    net = LARGE if large else SMALL
    if kind == "linear":
        return {"kind": kind, "tokens": _log(rng, 1, 64), "out": 8 * _log(rng, 8, 512),
                "in": 64 * _log(rng, 2, 64)}
    if kind == "decode":
        return {"kind": kind, "tokens": _log(rng, 1, 64), "layers": rng.randint(2, 16 if large else 28),
                **net}
    if kind == "attn":
        return {"kind": kind, "tokens": _log(rng, 64, 4096 if large else 8192), **net}
    if kind == "mlp":
        train = rng.random() < 0.6
        return {"kind": kind, "tokens": _log(rng, 64, 2048 if large and train else 8192), "train": train,
                **net}
    if kind == "norm":
        return {"kind": kind, "tokens": _log(rng, 64, 16384),
                "hidden": rng.choice([1536, 1536, 3584, 8 * rng.randint(32, 512)])}
    if kind == "rope":
        return {"kind": kind, "tokens": _log(rng, 64, 16384), "seq": rng.choice([512, 1000, 2048]),
                "padded": rng.random() < 0.3, "dtype": rng.choice(["fp16", "fp16", "fp32"]),
                "heads": net["heads"], "kv_heads": net["kv_heads"]}
    if kind == "loss":
        return {"kind": kind, "tokens": _log(rng, 64, 2048), "hidden": net["hidden"] if not large else 3584,
                "vocab": rng.choice([VOCAB, VOCAB, 8 * rng.randint(4000, VOCAB // 8)])}
    return {"kind": kind, "rows": 8 * _log(rng, 32, 2368), "cols": 64 * _log(rng, 4, 56),
            "dtype": rng.choice(["fp16", "bf16", "fp32"])}


# ---------------------------------------------------------------------------------------- inputs

class _Maker:
    """Seeded tensors on the GPU; the same calls give the same tensors."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def normal(self, *shape, scale=1.0, dtype=torch.float16):
        return (torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float32) * scale).to(dtype)

    def weight(self, rows, cols, dtype=torch.float16):
        """(packed codes, quant state) of a [rows, cols] NF4 weight."""
        from hackaton_b200.quantize import NestedState, QuantState

        def byte(n):
            return torch.randint(0, 256, (n,), generator=self.g, device="cuda", dtype=torch.uint8)

        n, blocks = rows * cols, rows * cols // 64
        codes = torch.tensor(CODES, dtype=torch.uint8, device="cuda")[byte(n).int()].view(-1, 2)
        packed = (codes[:, :1] << 4) | codes[:, 1:]
        absmax = byte(blocks)
        size = min(1.0, math.sqrt(1536 / cols))
        absmax2 = size * (0.015 + 0.01 * torch.rand((blocks + 255) // 256, generator=self.g, device="cuda"))
        code2 = torch.linspace(-1.0, 1.0, 256, device="cuda")
        state = QuantState(absmax=absmax, code=torch.tensor(LEVELS, device="cuda"), shape=(rows, cols),
                           dtype=dtype, nested=True,
                           state2=NestedState(absmax=absmax2, code=code2, blocksize=256),
                           offset=torch.tensor(0.05 * size, device="cuda"))
        return packed, state

    def ints(self, lo, hi, n):
        return torch.randint(lo, hi, (n,), generator=self.g, device="cuda")

    def uniform(self, n):
        return torch.rand(n, generator=self.g, device="cuda")


def _layer(make, case):
    h, f, kv = case["hidden"], case["mlp"], case["kv_heads"] * DIM
    return {"norm1": 1 + make.normal(h, scale=0.1, dtype=torch.float32),
            "norm2": 1 + make.normal(h, scale=0.1, dtype=torch.float32),
            "q": make.weight(h, h), "k": make.weight(kv, h), "v": make.weight(kv, h),
            "q_bias": make.normal(h, scale=0.1), "k_bias": make.normal(kv, scale=0.1),
            "v_bias": make.normal(kv, scale=0.1),
            "o": make.weight(h, h), "gate": make.weight(f, h), "up": make.weight(f, h),
            "down": make.weight(h, f)}


def _inputs(case, seed):
    make, kind = _Maker(seed), case["kind"]
    if kind == "linear":
        return {"w": make.weight(case["out"], case["in"]), "bias": make.normal(case["out"], scale=0.1),
                "x": make.normal(case["tokens"], case["in"])}
    if kind == "decode":
        h = case["hidden"]
        return {"layers": [_layer(make, case) for _ in range(case["layers"])],
                "norm": 1 + make.normal(h, scale=0.1, dtype=torch.float32),
                "head": make.normal(VOCAB, h, scale=0.04),
                "x": make.normal(case["tokens"], h, dtype=torch.float32)}
    if kind == "attn":
        h, kv, m = case["hidden"], case["kv_heads"] * DIM, case["tokens"]
        lora = lambda n: (make.normal(16, h, scale=0.02, dtype=torch.float32),  # noqa: E731
                          make.normal(n, 16, scale=0.02, dtype=torch.float32))
        return {"q": make.weight(h, h), "k": make.weight(kv, h), "v": make.weight(kv, h),
                "o": make.weight(h, h), "q_bias": make.normal(h, scale=0.1),
                "k_bias": make.normal(kv, scale=0.1), "v_bias": make.normal(kv, scale=0.1),
                "q_lora": lora(h), "v_lora": lora(kv),
                "x": make.normal(m, h), "attn": make.normal(m, h),
                "grads": [make.normal(m, h), make.normal(m, kv), make.normal(m, kv), make.normal(m, h)]}
    if kind == "mlp":
        h, f, m = case["hidden"], case["mlp"], case["tokens"]
        return {"gate": make.weight(f, h), "up": make.weight(f, h), "down": make.weight(h, f),
                "x": make.normal(m, h), "grad": make.normal(m, h) if case["train"] else None}
    if kind == "norm":
        m, h = case["tokens"], case["hidden"]
        return {"weight": 1 + make.normal(h, scale=0.1, dtype=torch.float32),
                "residual": make.normal(m, h, scale=2.0, dtype=torch.float32), "delta": make.normal(m, h),
                "grads": [make.normal(m, h, dtype=torch.float32), make.normal(m, h)]}
    if kind == "rope":
        m, seq, heads, kv = case["tokens"], case["seq"], case["heads"], case["kv_heads"]
        dtype = DTYPES[case["dtype"]]
        at = torch.arange(m, device="cuda", dtype=torch.int32)
        freq = 1.0 / (1e6 ** (torch.arange(0, DIM, 2, device="cuda").float() / DIM))
        angle = (torch.arange(seq, device="cuda").float()[:, None] * freq[None]).repeat(1, 2)[None]
        batch = (m + seq - 1) // seq
        out = (batch, heads, seq, DIM) if case["padded"] else (m, heads, DIM)
        return {"q": make.normal(m, heads * DIM, dtype=dtype), "k": make.normal(m, kv * DIM, dtype=dtype),
                "v": make.normal(m, kv * DIM, dtype=dtype), "cos": angle.cos(), "sin": angle.sin(),
                "b": at // seq, "t": at % seq, "batch": batch,
                "grads": [make.normal(*out) for _ in range(3)]}
    if kind == "loss":
        m, h, v = case["tokens"], case["hidden"], case["vocab"]
        targets = make.ints(0, v, m)
        targets[make.uniform(m) < 0.3] = -100       # prompt tokens carry no loss
        return {"hidden": make.normal(m, h), "head": make.normal(v, h, scale=0.04), "targets": targets,
                "count": (targets >= 0).sum().clamp(min=1).float()}
    return {"w": make.weight(case["rows"], case["cols"], DTYPES[case["dtype"]])}


def prepare(case, seed):
    state = _inputs(case, seed)
    state["case"] = case
    if case["kind"] == "decode":
        _capture(state)
    for name in ("x", "attn", "residual", "delta", "q", "k", "v", "hidden"):
        if case["kind"] in ("attn", "norm", "rope", "loss") or case.get("train"):
            if isinstance(state.get(name), torch.Tensor):
                state[name].requires_grad_()
    if case["kind"] == "attn":
        for name in ("q_lora", "v_lora"):
            for t in state[name]:
                t.requires_grad_()
    return state


def _decode(state, x):
    """One step of the stack without attention itself (not part of the package): o_proj reads the
    queries in its place. Returns the logits and every layer's new keys and values."""
    from hackaton_b200.dense import fp16_linear
    from hackaton_b200.group import Projection, nf4_linear_group
    from hackaton_b200.mlp import nf4_swiglu_mlp
    from hackaton_b200.nf4 import nf4_linear
    from hackaton_b200.rmsnorm import add_rms_norm, rms_norm

    cache, delta = [], None
    for lay in state["layers"]:
        if delta is None:
            h = rms_norm(x, lay["norm1"], EPS, to_half=True)
        else:
            x, h = add_rms_norm(x, delta, lay["norm1"], EPS, to_half=True)
        q, k, v = nf4_linear_group(h, [Projection(*lay[n], lay[n + "_bias"]) for n in "qkv"])
        cache += [k, v]
        x, h = add_rms_norm(x, nf4_linear(q, lay["o"][0], None, lay["o"][1]), lay["norm2"], EPS,
                            to_half=True)
        delta = nf4_swiglu_mlp(h, *(Projection(*lay[n]) for n in ("gate", "up", "down")))
    _, h = add_rms_norm(x, delta, state["norm"], EPS, to_half=True)
    return [fp16_linear(h, state["head"])] + cache


def _capture(state):
    """What a serving program does at start-up: scale tables, a warm-up pass, one captured step."""
    from hackaton_b200.nf4 import prepare_weights

    prepare_weights([w for lay in state["layers"] for w in lay.values() if isinstance(w, tuple)])
    state["input"] = state["x"].clone()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.no_grad(), torch.cuda.stream(stream):
        _decode(state, state["input"])
        stream.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"], stream=stream):
            state["output"] = _decode(state, state["input"])
    torch.cuda.synchronize()


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        from hackaton_b200.nf4 import nf4_linear
        with torch.no_grad():
            return nf4_linear(state["x"], state["w"][0], state["bias"], state["w"][1])
    if kind == "decode":
        state["input"].copy_(state["x"])
        state["graph"].replay()
        return state["output"]
    if kind == "attn":
        from hackaton_b200.group import Projection, nf4_linear_group
        from hackaton_b200.nf4 import nf4_linear
        ql, vl = state["q_lora"], state["v_lora"]
        outs = nf4_linear_group(state["x"], [Projection(*state["q"], state["q_bias"], *ql, 2.0),
                                             Projection(*state["k"], state["k_bias"]),
                                             Projection(*state["v"], state["v_bias"], *vl, 2.0)])
        outs = list(outs) + [nf4_linear(state["attn"], state["o"][0], None, state["o"][1])]
        grads = torch.autograd.grad(outs, [state["x"], state["attn"], *ql, *vl], state["grads"])
        return outs + list(grads)
    if kind == "mlp":
        from hackaton_b200.group import Projection
        from hackaton_b200.mlp import nf4_swiglu_mlp
        projs = [Projection(*state[n]) for n in ("gate", "up", "down")]
        if not case["train"]:
            with torch.no_grad():
                return nf4_swiglu_mlp(state["x"], *projs)
        y = nf4_swiglu_mlp(state["x"], *projs)
        return [y, torch.autograd.grad(y, state["x"], state["grad"])[0]]
    if kind == "norm":
        from hackaton_b200.rmsnorm import add_rms_norm
        outs = add_rms_norm(state["residual"], state["delta"], state["weight"], EPS, to_half=True)
        return list(outs) + list(torch.autograd.grad(outs, [state["residual"], state["delta"]],
                                                     state["grads"]))
    if kind == "rope":
        from hackaton_b200.rope import qkv_rotate
        ins = [state["q"], state["k"], state["v"]]
        outs = qkv_rotate(*ins, state["cos"], state["sin"], state["b"], state["t"], state["batch"],
                          case["seq"], case["heads"], case["kv_heads"], case["padded"])
        return list(outs) + list(torch.autograd.grad(outs, ins, state["grads"]))
    if kind == "loss":
        from hackaton_b200.lm_loss import linear_cross_entropy
        outs = linear_cross_entropy(state["hidden"], state["head"], state["targets"], state["count"])
        return list(outs) + [torch.autograd.grad(outs[0], state["hidden"])[0]]
    from hackaton_b200.nf4 import dequantize_nf4
    return dequantize_nf4(*state["w"])


# ----------------------------------------------------------------------------------- what it costs

def _nf4_bytes(rows, cols):
    blocks = rows * cols / 64
    return rows * cols / 2 + blocks + 4 * blocks / 256


def work(case):
    kind = case["kind"]
    if kind == "dequant":
        n = case["rows"] * case["cols"]
        return {"bytes": _nf4_bytes(case["rows"], case["cols"]) + n * DTYPES[case["dtype"]].itemsize,
                "flops": 0}
    m = case["tokens"]
    if kind == "linear":
        n, k = case["out"], case["in"]
        return {"bytes": _nf4_bytes(n, k) + 2 * (m * k + m * n + n), "flops": 2 * m * n * k}
    if kind == "norm":
        # forward: residual, delta in, sum, normalised out; backward: sum, two gradients in, two out
        return {"bytes": m * case["hidden"] * ((4 + 2 + 4 + 2) + (4 + 4 + 2 + 4 + 2)), "flops": 0}
    if kind == "rope":
        e, heads, kv = DTYPES[case["dtype"]].itemsize, case["heads"], case["kv_heads"]
        slots = (m + case["seq"] - 1) // case["seq"] * case["seq"] if case["padded"] else m
        one = m * (heads + 2 * kv) * DIM * e
        return {"bytes": 2 * one + 3 * heads * DIM * 2 * (slots + m), "flops": 0}
    h = case["hidden"]
    if kind == "loss":
        v = case["vocab"]
        return {"bytes": 2 * v * h + 2 * 2 * m * h + 8 * m + 20 * m, "flops": 4 * m * v * h}
    f, kv = case.get("mlp", 0), case["kv_heads"] * DIM
    attn_w = [(h, h), (kv, h), (kv, h), (h, h)]
    mlp_w = [(f, h), (f, h), (h, f)]
    if kind == "attn":
        params = sum(a * b for a, b in attn_w)
        acts = 2 * m * (2 * h + (2 * h + 2 * kv))          # inputs and outputs, once per direction
        lora = 2 * 16 * (2 * h + h + kv)
        return {"bytes": sum(_nf4_bytes(a, b) for a, b in attn_w) + 2 * acts + 4 * lora,
                "flops": 4 * m * params + 2 * m * 16 * (2 * h + h + kv) * 3}
    params = sum(a * b for a, b in mlp_w)
    if kind == "mlp":
        passes = 2 if case["train"] else 1
        return {"bytes": sum(_nf4_bytes(a, b) for a, b in mlp_w) + passes * 2 * m * 2 * h,
                "flops": passes * 2 * m * params}
    layer = sum(_nf4_bytes(a, b) for a, b in attn_w + mlp_w) + 2 * (h + 2 * kv) + 8 * h
    params += sum(a * b for a, b in attn_w)
    n = case["layers"]
    return {"bytes": n * (layer + 4 * m * kv) + 2 * VOCAB * h + 2 * m * VOCAB + 4 * m * h,
            "flops": 2 * m * (n * params + VOCAB * h)}


# ------------------------------------------------------------------------------------ correctness

def tolerance(case):
    return TOLERANCES[case["kind"]]


# About four times the largest error against 64 bits that was measured over the ranges of `draw`.
TOLERANCES = {
    "linear": {"rel": 1.6e-3},
    "decode": {"rel": 5e-3},
    "attn": {"rel": 1.6e-3},
    "mlp": {"rel": 3e-3},
    "norm": {"rel": 1e-3},
    "rope": {"rel": 1e-3},
    "loss": {"rel": 2.6e-3, "differ": 0.02},
    "dequant": "exact",
}


def _plain(w, dtype=torch.float64):
    """The weight of (packed, state) in 64 bits."""
    packed, state = w
    packed = packed.reshape(-1)
    codes = torch.stack((packed >> 4, packed & 15), 1).reshape(-1, 64)
    blocks = torch.arange(codes.shape[0], device=packed.device)
    scale = (state.state2.code[state.absmax.long()].to(dtype) * state.state2.absmax[blocks // 256].to(dtype)
             + state.offset.to(dtype))
    return (state.code.to(dtype)[codes.int()] * scale[:, None]).reshape(state.shape)


def _plain_norm(x, weight):
    return weight.double() * x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)


def exact(case, seed):
    s, kind = _inputs(case, seed), case["kind"]
    with torch.no_grad():
        if kind == "linear":
            return s["x"].double() @ _plain(s["w"]).T + s["bias"].double()
        if kind == "decode":
            x, cache = s["x"].double(), []
            for lay in s["layers"]:
                h = _plain_norm(x, lay["norm1"])
                q, k, v = (h @ _plain(lay[n]).T + lay[n + "_bias"].double() for n in "qkv")
                cache += [k, v]
                x = x + q @ _plain(lay["o"]).T
                h = _plain_norm(x, lay["norm2"])
                hidden = torch.nn.functional.silu(h @ _plain(lay["gate"]).T) * (h @ _plain(lay["up"]).T)
                x = x + hidden @ _plain(lay["down"]).T
            return [_plain_norm(x, s["norm"]) @ s["head"].double().T] + cache
        if kind == "mlp":
            gate, up, down = (_plain(s[n]) for n in ("gate", "up", "down"))
            x = s["x"].double()
            g, u = x @ gate.T, x @ up.T
            sig = torch.sigmoid(g)
            y = (g * sig * u) @ down.T
            if not case["train"]:
                return y
            dh = s["grad"].double() @ down
            return [y, (dh * u * sig * (1 + g * (1 - sig))) @ gate + (dh * g * sig) @ up]
        if kind == "attn":
            x, at = s["x"].double(), s["attn"].double()
            outs, dx, params = [], 0, []
            for n, dy in zip("qkv", s["grads"]):
                w, dy = _plain(s[n]), dy.double()
                y = x @ w.T + s[n + "_bias"].double()
                dx = dx + dy @ w
                if n + "_lora" in s:
                    a, b = (t.double() for t in s[n + "_lora"])
                    y = y + 2.0 * (x @ a.T) @ b.T
                    u = 2.0 * dy @ b
                    dx = dx + u @ a
                    params += [u.T @ x, dy.T @ (2.0 * x @ a.T)]
                outs.append(y)
            w = _plain(s["o"])
            return outs + [at @ w.T, dx, s["grads"][3].double() @ w] + params
        if kind == "norm":
            x = s["residual"].double() + s["delta"].double()
            w, dy = s["weight"].double(), s["grads"][1].double()
            rstd = torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)
            hat, g = x * rstd, dy * w
            dx = rstd * (g - hat * (g * hat).mean(-1, keepdim=True)) + s["grads"][0].double()
            return [x, w * hat, dx, dx]
        if kind == "rope":
            return _exact_rope(case, s)
        if kind == "loss":
            return _exact_loss(s)
        return _plain(s["w"], torch.float32).to(DTYPES[case["dtype"]])


def _exact_rope(case, s):
    heads, kv, m = case["heads"], case["kv_heads"], case["tokens"]
    cos, sin = (s[n].double()[0, s["t"].long()][:, None] for n in ("cos", "sin"))
    half = DIM // 2
    turn = lambda x: torch.cat((-x[..., half:], x[..., :half]), -1)  # noqa: E731
    q, k, v = (s[n].double().view(m, c, DIM) for n, c in zip("qkv", (heads, kv, kv)))
    rep = heads // kv
    outs = [q * cos + turn(q) * sin, (k * cos + turn(k) * sin).repeat_interleave(rep, 1),
            v.repeat_interleave(rep, 1)]
    grads = [g.double() for g in s["grads"]]
    if case["padded"]:
        b, t = s["b"].long(), s["t"].long()
        full = [torch.zeros(s["batch"], heads, case["seq"], DIM, dtype=torch.float64, device=q.device)
                for _ in outs]
        for f, o in zip(full, outs):
            f[b, :, t] = o
        outs, grads = full, [g[b, :, t] for g in grads]
    dq, dk, dv = grads
    dk, dv = (g.view(m, kv, rep, DIM).sum(2) for g in (dk, dv))
    back = lambda g: (g * cos - turn(g * sin)).reshape(m, -1)  # noqa: E731
    return outs + [back(dq), back(dk), dv.reshape(m, -1)]


def _exact_loss(s):
    head, targets = s["head"].double(), s["targets"]
    losses, entropy, top, grads = [], [], [], []
    for lo in range(0, len(targets), 256):
        h, t = s["hidden"][lo:lo + 256].double(), targets[lo:lo + 256]
        logits = h @ head.T
        logp = torch.log_softmax(logits, -1)
        p, valid, at = logp.exp(), t >= 0, t.clamp(min=0)[:, None]
        losses.append(torch.where(valid, -logp.gather(1, at)[:, 0], 0.0))
        entropy.append(-(p * logp).sum(-1))
        top.append(logits.argmax(-1))
        p.scatter_add_(1, at, torch.full_like(p[:, :1], -1.0))
        grads.append((p * valid[:, None] / s["count"].double()) @ head)
    losses = torch.cat(losses)
    return [losses.sum() / s["count"].double(), losses, torch.cat(entropy), torch.cat(top), torch.cat(grads)]

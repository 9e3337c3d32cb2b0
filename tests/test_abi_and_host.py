"""CPU: the C-ABI library builds, loads and exports every symbol include/nf4b200.h declares;
host-side guards and patches behave like the reference's (no compute calls here)."""

import ctypes
import re
import sys
import types
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def library():
    from hackaton_b200.build import build_library

    return ctypes.CDLL(str(build_library()))


def declared_functions():
    text = (ROOT / "include" / "nf4b200.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(nf4b200_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported(library):
    names = declared_functions()
    assert len(names) >= 8
    for name in names:
        assert hasattr(library, name), f"{name} declared in nf4b200.h but not exported"


def test_binding_covers_the_header():
    from hackaton_b200 import _lib

    assert sorted(_lib.EXPORTS) == declared_functions()


def test_struct_layout_matches_header():
    from hackaton_b200 import _lib

    assert ctypes.sizeof(_lib.Weight) == 6 * 8 + 2 * 8 + 4 * 4 + 8
    assert _lib.Weight.scales16.offset == 80
    assert ctypes.sizeof(_lib.Props) == 4 * 4 + 8


def test_no_gpu_means_error_not_fallback(library):
    """Without a CUDA device every compute entry point reports an error status."""
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    from hackaton_b200 import _lib

    w = _lib.Weight()
    rc = _lib.lib().nf4b200_dequant(ctypes.byref(w), None, 0, None)
    assert rc != 0
    assert _lib.lib().nf4b200_last_error()


def test_can_dequantize_guards():
    from hackaton_b200 import can_dequantize
    from tests.util import synthetic_weight

    packed, state = synthetic_weight(8, 64, True)
    assert not can_dequantize(packed, state)           # CPU tensors: never eligible
    assert not can_dequantize("not a tensor", state)


def test_product_does_not_import_the_oracle():
    for path in (ROOT / "hackaton_b200").rglob("*.py"):
        text = path.read_text()
        assert "oracle" not in re.sub(r'""".*?"""', "", text, flags=re.S), path


def test_matmul_patch_falls_through_to_original(monkeypatch):
    """solution/patches.py:266-275: whatever the kernels do not cover goes to the function that
    was installed before (here a fake bitsandbytes)."""
    calls = []
    fake = types.ModuleType("bitsandbytes")
    fake.matmul_4bit = lambda A, B, quant_state, out=None, bias=None: calls.append("orig") or "orig"
    fake.nn = types.SimpleNamespace(Linear4bit=type("Linear4bit", (), {}))
    monkeypatch.setitem(sys.modules, "bitsandbytes", fake)
    from hackaton_b200 import patches

    patches.patch_nf4_matmul()
    patched = fake.matmul_4bit
    assert patched._nf4b200
    patches.patch_nf4_matmul()                      # idempotent
    assert fake.matmul_4bit is patched
    x = torch.zeros(8, 64, dtype=torch.float16)     # CPU tensor -> not eligible
    assert fake.matmul_4bit(x, torch.zeros(1, 8, dtype=torch.uint8), None) == "orig"
    assert calls == ["orig"]
    assert patches._is_4bit_linear(fake.nn.Linear4bit())
    assert not patches._is_4bit_linear(object())


def test_lora_patch_falls_through_to_original():
    from hackaton_b200 import patches

    seen = []
    forward = patches.lora_forward_for(lambda self, x, *a, **k: seen.append(1) or "orig")
    module = types.SimpleNamespace(active_adapters=["default"], disable_adapters=True,
                                   merged=False, base_layer=None, lora_A={}, lora_B={})
    assert forward(module, torch.zeros(2, 64)) == "orig" and seen == [1]


def _fake_lora_module(k=128, n=64, rank=16, **extra):
    """A stand-in for peft's LoRA wrapper around a 4-bit linear, with the attributes the patch reads."""
    state = types.SimpleNamespace(shape=(n, k))
    base = types.SimpleNamespace(weight=types.SimpleNamespace(quant_state=state), bias=None)
    mod = types.SimpleNamespace(
        active_adapters=["default"], disable_adapters=False, merged=False, base_layer=base,
        lora_A={"default": types.SimpleNamespace(weight=torch.zeros(rank, k), bias=None)},
        lora_B={"default": types.SimpleNamespace(weight=torch.zeros(n, rank), bias=None)},
        lora_dropout={"default": torch.nn.Identity()}, scaling={"default": 2.0},
        forward=lambda x: "own")
    for key, value in extra.items():
        setattr(mod, key, value)
    return mod


@pytest.mark.parametrize("extra,fused", [
    ({}, True),
    ({"use_dora": {"default": True}}, False),                 # DoRA: another formula
    ({"use_dora": {"default": False}}, True),
    ({"lora_variant": {"default": object()}}, False),          # newer peft: any registered variant
    ({"lora_magnitude_vector": {"default": object()}}, False),
    ({"lora_variant": {}, "lora_magnitude_vector": {}}, True),
])
def test_lora_patch_leaves_adapter_variants_to_peft(monkeypatch, extra, fused):
    """Adapters whose forward is not the plain low-rank update (DoRA, entries of `lora_variant`)
    take peft's own forward, in the module patch and in the sibling groups alike."""
    from hackaton_b200 import patches

    monkeypatch.setattr(patches, "_eligible", lambda x, state, weight, bias: True)
    monkeypatch.setattr(patches, "nf4_lora_linear", lambda *a, **k: "fused")
    forward = patches.lora_forward_for(lambda self, x, *a, **k: "orig")
    module = _fake_lora_module(**extra)
    assert forward(module, torch.zeros(2, 128)) == ("fused" if fused else "orig")
    proj = patches.SiblingGroup([module])._projection(module, torch.zeros(2, 128))
    assert (proj is not None) == fused


def test_lora_patch_checks_rank_and_feature_counts(monkeypatch):
    from hackaton_b200 import patches

    monkeypatch.setattr(patches, "_eligible", lambda x, state, weight, bias: True)
    monkeypatch.setattr(patches, "nf4_lora_linear", lambda *a, **k: "fused")
    forward = patches.lora_forward_for(lambda self, x, *a, **k: "orig")
    assert forward(_fake_lora_module(rank=8), torch.zeros(2, 128)) == "orig"
    wrong_in = _fake_lora_module()
    wrong_in.lora_A["default"].weight = torch.zeros(16, 64)     # A does not read the base input
    assert forward(wrong_in, torch.zeros(2, 128)) == "orig"
    biased = _fake_lora_module()
    biased.lora_B["default"].bias = torch.zeros(64)
    assert forward(biased, torch.zeros(2, 128)) == "orig"


def test_sibling_group_routes_one_launch(monkeypatch):
    """q/k/v called one after the other with the same tensor: one grouped computation, every
    module gets its own share; another tensor, or an ineligible input, starts over or falls
    through to the module's own forward."""
    import types

    from hackaton_b200 import group, patches

    class Lin(torch.nn.Module):
        def __init__(self, tag):
            super().__init__()
            self.tag = tag
            self.weight = types.SimpleNamespace(quant_state=object())
            self.bias = None

        def forward(self, x):
            return ("own", self.tag)

    calls = []

    def fake_group(x, projections):
        calls.append(len(projections))
        return [("grouped", i, id(x)) for i in range(len(projections))]

    eligible = {"ok": True}
    monkeypatch.setattr(patches, "_eligible", lambda x, state, weight, bias: eligible["ok"])
    monkeypatch.setattr(group, "nf4_linear_group", fake_group)
    q, k, v = Lin("q"), Lin("k"), Lin("v")
    g = patches.SiblingGroup([q, k, v]).install()
    x = torch.zeros(2, 4)
    assert q(x) == ("grouped", 0, id(x))
    assert v(x) == ("grouped", 2, id(x))
    assert k(x) == ("grouped", 1, id(x))
    assert calls == [3]
    x2 = torch.zeros(2, 4)
    assert k(x2) == ("grouped", 1, id(x2)) and calls == [3, 3]
    assert k(x2) == ("grouped", 1, id(x2)) and calls == [3, 3, 3]   # its share was already taken
    eligible["ok"] = False
    assert q(torch.zeros(2, 4)) == ("own", "q")
    g.remove()
    eligible["ok"] = True
    assert q(x) == ("own", "q")


def test_patch_sibling_projections_finds_blocks(monkeypatch):
    import types

    from hackaton_b200 import patches

    class Lin(torch.nn.Module):
        def __init__(self, n_in):
            super().__init__()
            self.in_features = n_in

        def forward(self, x):
            return x

    monkeypatch.setattr(patches, "_is_4bit_linear", lambda m: isinstance(m, Lin))

    class Attn(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.q_proj, self.k_proj, self.v_proj, self.o_proj = Lin(8), Lin(8), Lin(8), Lin(8)

    class Mlp(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.gate_proj, self.up_proj, self.down_proj = Lin(8), Lin(8), Lin(16)

    model = torch.nn.Sequential(Attn(), Mlp(), Attn())
    groups = patches.patch_sibling_projections(model)
    assert [len(g.modules) for g in groups] == [3, 2, 3]
    assert patches.patch_sibling_projections(model) == []      # nothing left to group
    for g in groups:
        g.remove()


def test_mlp_patch_routes_and_falls_through(monkeypatch):
    """The Qwen2MLP replacement: eligible 4-bit gate/up go through the fused front half and
    down_proj sees its fp16 result; another activation, or an ineligible input, runs the
    original forward (solution/patches.py:32-41 has the same shape)."""
    import types

    from hackaton_b200 import mlp, patches

    class Lin(torch.nn.Module):
        def __init__(self, tag):
            super().__init__()
            self.tag = tag
            self.weight = types.SimpleNamespace(quant_state=types.SimpleNamespace(shape=(8, 4)))
            self.bias = None
            self.compute_dtype = torch.float16

        def forward(self, x):
            return ("down", x)

    class Mlp:
        def __init__(self, act="silu"):
            self.gate_proj, self.up_proj, self.down_proj = Lin("g"), Lin("u"), Lin("d")
            self.config = types.SimpleNamespace(hidden_act=act)

    class FakeCuda(torch.Tensor):
        is_cuda = True

    calls = []

    def fake_front(x16, gate, up):
        calls.append((x16.dtype, gate.packed, up.packed))
        return torch.ones(2, 8, dtype=torch.float16)

    class Out:
        def __init__(self, v):
            self.v = v

        def to(self, dtype):
            return ("cast", dtype, self.v)

    monkeypatch.setattr(patches, "_is_4bit_linear", lambda m: isinstance(m, Lin))
    monkeypatch.setattr(patches, "_eligible", lambda x, state, weight, bias: True)
    monkeypatch.setattr(mlp, "nf4_gate_up_swiglu", fake_front)
    monkeypatch.setattr(Lin, "forward", lambda self, x: Out(("down", tuple(x.shape), x.dtype)))
    forward = patches.mlp_forward_for(lambda self, x: "original")
    x = torch.zeros(2, 4, dtype=torch.float32).as_subclass(FakeCuda)
    block = Mlp()
    assert forward(block, x) == ("cast", torch.float32, ("down", (2, 8), torch.float16))
    assert calls == [(torch.float16, block.gate_proj.weight, block.up_proj.weight)]
    assert forward(Mlp("gelu"), x) == "original"
    assert forward(block, torch.zeros(2, 4)) == "original"            # not on a GPU
    monkeypatch.setattr(patches, "_eligible", lambda x, state, weight, bias: False)
    assert forward(block, x) == "original"
    assert len(calls) == 1


def test_loss_chunks_cover_every_row_once():
    """The row chunks of the lm_head loss: in order, without gaps, all full but the last."""
    from hackaton_b200.lm_loss import CHUNK_ROWS, CHUNK_TILE, _chunks

    assert _chunks(0) == [] and CHUNK_ROWS % CHUNK_TILE == 0
    for rows in [*range(1, 5200, 7), 2047, 2048, 2049, 4096, 4097, 6145, 8193, 100_000]:
        for step in (CHUNK_ROWS, CHUNK_TILE, 256):
            parts = _chunks(rows, step)
            sizes = [p.stop - p.start for p in parts]
            assert parts[0].start == 0 and parts[-1].stop == rows
            assert all(a.stop == b.start for a, b in zip(parts, parts[1:]))
            assert sizes[:-1] == [step] * (len(sizes) - 1) and 0 < sizes[-1] <= step
        assert _chunks(rows) == _chunks(rows, CHUNK_ROWS)


@pytest.mark.parametrize("vocab", [1000, 32_000, 151_936, 163_840, 163_848, 262_144, 1_000_000])
@pytest.mark.parametrize("itemsize", [2, 4])
def test_loss_chunks_bound_the_logits(vocab, itemsize):
    """The logits alive at a time take at most LOGITS_BYTES, or what the reference's 256 rows take."""
    from hackaton_b200.lm_loss import CHUNK_ROWS, LOGITS_BYTES, _chunk_rows

    rows = _chunk_rows(vocab, itemsize)
    assert 256 <= rows <= CHUNK_ROWS
    assert rows * vocab * itemsize <= max(LOGITS_BYTES, 256 * vocab * itemsize)


@pytest.mark.parametrize("most", [100, 255, 256, 700, 5000])
def test_loss_takes_fewer_rows_where_memory_is_short(monkeypatch, most):
    """An allocation that does not fit is tried with fewer rows, down to the reference's 256."""
    from hackaton_b200 import lm_loss

    real, asked = torch.empty, []

    def empty(rows, cols, **kw):
        asked.append(rows)
        if rows > most:
            raise torch.OutOfMemoryError("no room")
        return real(rows, cols, **kw)

    monkeypatch.setattr(lm_loss.torch, "empty", empty)
    like = torch.zeros(1, dtype=torch.float16)
    if most < 256:
        with pytest.raises(torch.OutOfMemoryError):
            lm_loss._logits_buffer(3000, 64, like)
    else:
        got = lm_loss._logits_buffer(3000, 64, like).shape[0]
        assert 256 <= got <= most and got * 2 > min(most, lm_loss.CHUNK_ROWS)
    assert asked[0] == lm_loss.CHUNK_ROWS and min(asked) >= 256


def test_sm_limit_drops_every_scratch_size(monkeypatch):
    """Scratch sizes follow the SM limit: what was asked under one limit is asked again under another,
    for every kind of call."""
    from hackaton_b200 import _lib, group, mlp, nf4

    asked = []

    class Library:
        def __getattr__(self, name):
            return lambda *args: asked.append(name) or (0 if name == "nf4b200_set_sm_limit" else 256)

    monkeypatch.setattr(_lib, "lib", Library)
    monkeypatch.setattr(nf4, "_ws_need", {})
    monkeypatch.setattr(nf4.torch.cuda, "device", lambda d: __import__("contextlib").nullcontext())
    device = torch.device("cuda", 0)
    calls = [lambda: nf4._workspace(device, 64, 64, 4, False), lambda: nf4._workspace(device, 64, 64, 4, True),
             lambda: (None, group._workspace(device, [64, 64], 64, 4, False)),
             lambda: (None, nf4.scratch_bytes(device, "nf4b200_gate_up_swiglu_workspace_bytes", 64, 64, 4, 1)),
             lambda: (None, nf4.scratch_bytes(device, "nf4b200_linear_bwd_dx_swiglu_workspace_bytes", 64, 64, 4))]
    for _ in range(2):
        assert all(call()[1] == 256 for call in calls)
    assert len(asked) == len(calls)
    _lib.set_sm_limit(8)
    assert all(call()[1] == 256 for call in calls)
    assert len(asked) == 2 * len(calls) + 1
    assert all(not hasattr(module, "_ws_need") for module in (group, mlp))


def test_weight_key_covers_what_the_descriptor_is_made_from():
    """Every tensor and size that a descriptor or its scale table depends on changes the key, replaced
    or written in place; a state nobody touched keeps it; inference tensors are taken."""
    from hackaton_b200.nf4 import _content_key
    from tests.util import synthetic_weight

    def changes(state):
        for owner in (state, state.state2):
            for field in ("absmax", "code"):
                t = getattr(owner, field)
                yield lambda t=t: t.mul_(1)
                yield lambda owner=owner, field=field, t=t: setattr(owner, field, t.clone())
            yield lambda owner=owner: setattr(owner, "blocksize", owner.blocksize * 2)
        yield lambda: state.offset.mul_(1)
        yield lambda: setattr(state, "offset", state.offset.clone())
        yield lambda: setattr(state, "offset", 0.25)
        yield lambda: setattr(state, "shape", tuple(reversed(state.shape)))

    packed, state = synthetic_weight(32, 128, True)
    seen = [_content_key(packed, state)]
    kept = []   # (a freed tensor's address could come back)
    for change in changes(state):
        kept.append((state.absmax, state.code, state.state2.absmax, state.state2.code, state.offset))
        change()
        seen.append(_content_key(packed, state))
        assert seen[-1] == _content_key(packed, state)
    packed.add_(0)
    seen.append(_content_key(packed, state))
    assert len(set(seen)) == len(seen)
    with torch.inference_mode():
        packed, state = synthetic_weight(32, 128, True)
    assert _content_key(packed, state) == _content_key(packed, state)


def test_rotation_without_heads_is_an_error(monkeypatch):
    """No query heads: Python's ZeroDivisionError, before any native code divides by it."""
    from hackaton_b200 import _lib
    from hackaton_b200.rope import _RotateOp

    calls = []
    host = types.SimpleNamespace(rotate_fwd=lambda *args: calls.append(args) or (None,) * 8)
    monkeypatch.setattr(_lib, "host", lambda: host)
    q = types.SimpleNamespace(is_cuda=True, dtype=torch.float16, shape=(4, 256))
    table = torch.zeros(1, 4, 128)
    with pytest.raises(ZeroDivisionError):
        _RotateOp(1, 4, 0, 1, False).run(lambda *a, **k: None, q, q, q, table, table, None, None)
    assert not calls
    _RotateOp(1, 4, 2, 1, False).run(lambda *a, **k: None, q, q, q, table, table, None, None)
    assert calls[0][7:] == (1, 4, 2, 1, 128, False)


def test_rows_view_gives_aligned_rows():
    """Rows the kernels accept from every layout: contiguous values, 16-byte aligned, eight elements
    apart; a copy only where the layout forces one. Columns that are no eights are left as they are."""
    from hackaton_b200.nf4 import _rows_view

    flat = torch.arange(4096, dtype=torch.float16)
    assert flat.data_ptr() % 16 == 0
    kept = [flat[:320].view(5, 64), flat[8:328].view(5, 64), flat.view(16, 256)[:, 8:72], flat[:64].view(1, 64)]
    copied = [flat[1:321].view(5, 64), flat[3:67].view(1, 64), flat[8:].as_strided((1, 64), (67, 1)),
              flat.as_strided((4, 64), (67, 1)), flat[:320].view(64, 5).t(), flat[:64].expand(3, 64),
              flat[1:65], flat[1:641].view(2, 5, 64), flat[:64].expand(1, 64)]
    for t in kept + copied:
        v = _rows_view(t, 64)
        assert torch.equal(v, t.reshape(-1, 64)) and v.stride(1) == 1 and v.stride(0) % 8 == 0
        assert v.data_ptr() % 16 == 0 and v.stride(0) >= 64
    assert all(_rows_view(t, 64).data_ptr() == t.data_ptr() for t in kept)
    odd = flat[1:1 + 5 * 63].view(5, 63)
    assert _rows_view(odd, 63).data_ptr() == odd.data_ptr()


def test_host_module_belongs_to_the_installed_torch(library, monkeypatch, tmp_path):
    """_host.so is built again for another torch or Python, however new the file is, and a module built
    for another one is refused by name."""
    import hackaton_b200
    from hackaton_b200 import _lib, build

    assert not build._host_stale() and _lib.host().built_for == build.host_target()
    copy = tmp_path / "_host.so"
    monkeypatch.setattr(build, "HOST", copy)
    assert build._host_stale()
    content = (build.PKG / "_host.so").read_bytes()
    copy.write_bytes(content)
    assert not build._host_stale()
    copy.write_bytes(content.replace(b"built for torch 2", b"built for torch 1"))
    assert build._host_stale()
    monkeypatch.setattr(_lib, "_host_module", None)
    other = types.ModuleType("hackaton_b200._host")
    other.built_for = "torch 1.0, python 3.1"
    monkeypatch.setitem(sys.modules, "hackaton_b200._host", other)
    monkeypatch.setattr(hackaton_b200, "_host", other, raising=False)
    with pytest.raises(RuntimeError, match="torch 1.0.*hackaton_b200.build"):
        _lib.host()


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int8, torch.float32, torch.bfloat16])
def test_lora_inputs_of_other_types_are_refused_before_the_launch(monkeypatch, dtype):
    """The side kernel reads two bytes per element of its inputs; a type of one byte would be read past
    its end. The refusal comes before anything is launched, alone and in a group."""
    from hackaton_b200 import _lib, lora
    from hackaton_b200.group import NF4LinearGroup, Projection

    calls = []
    host = types.SimpleNamespace(lora_side=lambda *args: calls.append(args))
    monkeypatch.setattr(_lib, "host", lambda: host)
    a, b = torch.zeros(16, 64), torch.zeros(32, 16)
    x = torch.zeros(4, 64).to(dtype)
    with pytest.raises(TypeError):
        lora.lora_side([x], [a], [1.0], [b])
    with pytest.raises(TypeError):
        NF4LinearGroup.apply(x, [Projection(None, None, None, a, b)], None, a, b)
    with pytest.raises(TypeError):
        lora.NF4LoRALinear.apply(x, x, None, None, None, a, b, 1.0)
    half = torch.zeros(4, 64, dtype=torch.float16)
    with pytest.raises(ValueError):
        lora.NF4LoRALinear.apply(half, half[:2], None, None, None, a, b, 1.0)
    assert not calls


def test_scale_table_found_ready_by_another_thread(monkeypatch):
    """Between a call's look at the pending build and its wait another thread may have seen it finish."""
    from hackaton_b200 import nf4

    ref = object.__new__(nf4.WeightRef)
    ref.scales16, ref._ready, ref.keep = torch.zeros(1), (object(), 0), [torch.zeros(1)]
    monkeypatch.setattr(nf4.torch.cuda, "is_current_stream_capturing", lambda: setattr(ref, "_ready", None))
    assert ref.prepare() is ref

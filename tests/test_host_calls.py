"""Native calls into the kernel library (csrc/host_calls.cpp): arguments, and what a layer's modules are asked, on the CPU."""
import ctypes as C
import sys

import pytest
import torch

from gpt_neox_b200 import build
from gpt_neox_b200.ops import _lib


@pytest.fixture(scope="module")
def calls():
    build.build_host_calls()
    return _lib._load_calls()


def test_the_module_is_this_interpreters(calls, monkeypatch, tmp_path):
    """The file names the interpreter that it was built under; another one does not load it, and is told what to do."""
    name = build.host_calls_path().name
    assert sys.implementation.cache_tag in name and calls.__spec__.origin.endswith(name)
    monkeypatch.setattr(build.sysconfig, "get_config_var", lambda key: ".cpython-399-x86_64-linux-gnu.so")
    with pytest.raises(_lib.KernelError, match="cpython-399.*this interpreter"):
        _lib._load_calls()
    monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    with pytest.raises(RuntimeError, match="headers"):
        build.build_host_calls()


class _OnGpu:
    """What the calls ask of a tensor."""

    def __init__(self, at, dtype=torch.bfloat16, is_cuda=True, contiguous=True):
        self.at, self.dtype, self.is_cuda, self._contiguous = at, dtype, is_cuda, contiguous

    def data_ptr(self):
        return self.at

    def is_contiguous(self):
        return self._contiguous


P, I, L, F = C.c_void_p, C.c_int, C.c_longlong, C.c_float


@pytest.mark.parametrize("name,types", [
    ("nx_norm_fwd", [I] + [P] * 9 + [L, I, F, P]), ("nx_norm_bwd_f16", [I] + [P] * 14 + [L, I, I, I, P]),
    ("nx_gemm_bf16", [P, P, P, I, I, I, L, L, L, I, I, P, P, P, P, L, I, F, P]), ("nx_gated_act_fwd", [P, P, L, I, I, P]),
    ("nx_layer_infer", [P, P])])
def test_bound_entry_gets_its_arguments(calls, name, types):
    got = []
    proto = C.CFUNCTYPE(I, *types)
    target = proto(lambda *a: (got.append(a), 7)[1])
    entry = calls.bind(name, C.cast(target, P).value)
    values = {P: (2 ** 40 + 16, 2 ** 40 + 16), I: (-2 ** 31, -2 ** 31), L: (2 ** 62 + 1, 2 ** 62 + 1), F: (0.5, 0.5)}
    for pointer, seen in ((_OnGpu(2 ** 47 + 32), 2 ** 47 + 32), (2 ** 47 + 64, 2 ** 47 + 64), (None, None), (0, None)):
        args = [pointer if t is P else values[t][0] for t in types]
        assert entry(*args) == 7
        assert got.pop() == tuple(seen if t is P else values[t][1] for t in types)
    args = [None if t is P else values[t][0] for t in types]
    with pytest.raises(TypeError):
        entry(*args[:-1])
    with pytest.raises(_lib.KernelError, match="host tensor"):
        entry(*[torch.zeros(2) if t is P else v for t, v in zip(types, args)])
    if I in types:
        with pytest.raises(OverflowError):
            entry(*[2 ** 31 if t is I else v for t, v in zip(types, args)])
        with pytest.raises(TypeError):
            entry(*["1" if t is I else v for t, v in zip(types, args)])
    assert got == [] and calls.bind("nx_gemm_bf16_grouped", 16) is None


def test_declarations_are_compared(calls):
    """A declaration that is not the native module's is refused; the library's own are taken when it is loaded."""
    assert calls.bind("nx_layer_infer", 16, "PP") is not None and calls.bind("nx_gated_act_fwd_f16", 16, "PPLIIP") is not None
    for name, types in (("nx_layer_infer", "PL"), ("nx_layer_infer", "PPP"), ("nx_gated_act_fwd", "PPIIIP"), ("nx_gated_act_fwd", "")):
        with pytest.raises(TypeError, match="declared"):
            calls.bind(name, 16, types)
    assert _lib._declare(C.CDLL(str(_lib._LIB_PATH)), calls) is not None
    moved = C.CDLL(str(_lib._LIB_PATH))

    class Other:
        bind = staticmethod(lambda name, at, types: calls.bind(name, at, types.replace("L", "I")))
    with pytest.raises(TypeError, match="declared"):
        _lib._declare(moved, Other)


def test_layer_arguments_say_their_size():
    """A block of another layout is refused before anything of it is used (without a GPU: no row to work on)."""
    from gpt_neox_b200.ops import layer_infer
    lib = _lib.lib(torch.bfloat16)
    block = lambda size: bytes(13 * 8) + layer_infer._TAIL.pack(size, *([0] * 19), 0.0, 0.0)
    assert len(block(0)) == layer_infer._BYTES
    assert lib.nx_layer_infer(block(layer_infer._BYTES), None) == 0
    for size in (0, layer_infer._BYTES - 8, layer_infer._BYTES + 8):
        assert lib.nx_layer_infer(block(size), None) > 0 and b"layer_infer" in lib.nx_last_error()


def test_bound_entry_takes_bytes(calls):
    seen = []
    target = C.CFUNCTYPE(I, P, P)(lambda a, b: (seen.append(C.string_at(a, 4)), 0)[1])
    assert calls.bind("nx_layer_infer", C.cast(target, P).value)(b"\x01\x02\x03\x00more", 0) == 0
    assert seen == [b"\x01\x02\x03\x00"]


class _Plain(torch.nn.Module):
    def __init__(self, bias=True):
        super().__init__()
        self.weight = torch.nn.Parameter(torch.zeros(4))
        self.register_parameter("bias", torch.nn.Parameter(torch.zeros(4)) if bias else None)
        self.child = torch.nn.Identity()
        self.register_buffer("table", torch.zeros(2))

    def forward(self, x):
        return x


def test_plain_modules(calls):
    forward = _Plain.forward
    ask = lambda m: calls.plain(_Plain(), _Plain, forward, m, _Plain, forward)
    assert ask(_Plain())
    m = _Plain()
    m.forward = lambda x: x
    assert not ask(m)
    for hook in ("register_forward_hook", "register_forward_pre_hook"):
        m = _Plain()
        handle = getattr(m, hook)(lambda *a: None)
        assert not ask(m)
        handle.remove()
        assert ask(m)
    assert not ask(type("Sub", (_Plain,), {})()) and not ask(torch.nn.Identity()) and not ask(None)
    try:
        _Plain.forward = lambda self, x: x
        assert not ask(_Plain())
    finally:
        _Plain.forward = forward


def test_submodules_and_buffers(calls):
    m = _Plain()
    assert calls.sub(m, "child") is m.child and calls.sub(m, "table") is m.table
    m.__dict__["child"] = 5                       # stands before the module's __getattr__
    assert calls.sub(m, "child") == 5 == m.child
    with pytest.raises(AttributeError):
        calls.sub(m, "nothing")


def test_pointers(calls):
    x = _OnGpu(64)
    a, b = _Plain(), _Plain(bias=False)
    hold = lambda m, w, bias=None: m.__dict__.update(weight=w, bias=bias)
    hold(a, _OnGpu(128), _OnGpu(256))
    hold(b, _OnGpu(512))
    got = calls.pointers(_lib.H16, x, a, b)
    assert [int.from_bytes(got[8 * i:8 * i + 8], "little") for i in range(5)] == [64, 128, 256, 512, 0] and len(got) == 40
    for bad in (_OnGpu(136), _OnGpu(128, dtype=torch.float16), _OnGpu(128, is_cuda=False), _OnGpu(128, contiguous=False)):
        hold(a, bad)
        assert calls.pointers(_lib.H16, x, a, b) is None
    assert calls.pointers(_lib.H16, _OnGpu(64, dtype=torch.float32), b) is None
    real = _Plain()                                # parameters where torch.nn.Module keeps them: on the host here
    assert calls.pointers(_lib.H16, x, real) is None
    del real._parameters["weight"]
    with pytest.raises(AttributeError):
        calls.pointers(_lib.H16, x, real)


class _Shaped(_OnGpu):
    def __init__(self, at, *shape):
        super().__init__(at)
        self.shape = torch.Size(shape)

    def numel(self):
        return self.shape.numel()


def test_weight_sizes(calls):
    """Addresses are given where every weight has the size beside its module, and its bias as many elements as it has rows."""
    x = _OnGpu(16)

    def held(weight, bias=None):
        m = _Plain()
        m.__dict__.update(weight=weight, bias=bias)
        return m

    def given(*modules_and_sizes):
        got, width = calls.weights(_lib.H16, x, *modules_and_sizes)
        return (None if got is None else [int.from_bytes(got[i:i + 8], "little") for i in range(0, len(got), 8)]), width

    a, b, norm = held(_Shaped(32, 6, 4), _Shaped(48, 6)), held(_Shaped(64, 4, 6)), held(_Shaped(80, 4), _Shaped(96, 4))
    where = [16, 80, 96, 32, 48, 64, 0]
    assert given(norm, 4, 0, a, 6, 4, b, 4, 6) == (where, -1)
    assert given(norm, 4, 0, a, -1, 4, b, 4, -1) == (where, 6)
    for m, n, k in ((a, 5, 4), (a, 6, 5), (a, 4, 6), (a, 6, 0), (norm, 4, 1), (norm, 3, 0)):
        assert given(b, 4, 6, m, n, k)[0] is None
    assert given(a, -1, 4, b, -1, 6)[0] is None and given(a, -1, 4, held(_Shaped(64, 4, 5)), 4, -1)[0] is None
    for bias in (_Shaped(48, 5), _Shaped(48, 0), _OnGpu(48, is_cuda=False), _Shaped(56, 6)):
        assert given(held(_Shaped(32, 6, 4), bias), 6, 4)[0] is None
    assert given(held(_Shaped(32, 6, 4, 1)), 6, 4)[0] is None and given(held(None), 6, 4)[0] is None
    for args in ((), (_lib.H16,), (_lib.H16, x, a, 6), (list(_lib.H16), x)):
        with pytest.raises(TypeError):
            calls.weights(*args)
    with pytest.raises(AttributeError):
        calls.weights(_lib.H16, x, torch.nn.Identity(), 1, 1)


def _resized_mlp(layer, up, down):
    """Parameters of other widths in a layer's MLP: a pruned or grown one."""
    m, h = layer.mlp, layer.mlp.linear2.weight.shape[0]
    like = m.linear1.weight
    new = lambda *s: torch.nn.Parameter(torch.randn(s, device=like.device, dtype=like.dtype) * 0.05)
    m.linear1.weight, m.linear1.bias, m.linear2.weight = new(up, h), new(up), new(h, down)


@pytest.mark.parametrize("up,down", [(None, None), (40, 40), (512, 512), (40, 64), (512, 40)])
def test_a_layer_in_one_call_goes_by_the_weights_it_is_given(calls, up, down, monkeypatch):
    """What the native layer call is told, with weights that stand in for ones on the GPU: the MLP's width is its weights', and
    weights that do not fit one another send the layer down the op-by-op path, which refuses them."""
    import types

    from common import tiny_config
    from test_generation import _model
    from gpt_neox_b200.models import transformer
    _, model = _model(hidden_size=256, num_attention_heads=4)
    model.eval()
    model.inference_mode(use_cache=True)
    layer = next(m for m in model.modules() if isinstance(m, transformer.ParallelTransformerLayer))
    if up is not None:
        _resized_mlp(layer, up, down)
    a, m = layer.attention, layer.mlp
    a.use_flash_attention = True
    width = m.linear1.weight.shape[0]
    for module in (layer.input_layernorm, layer.post_attention_layernorm, a.query_key_value, a.dense, m.linear1, m.linear2):
        for name in ("weight", "bias"):
            t = getattr(module, name)
            if t is not None:
                module.__dict__[name] = _Shaped(4096, *t.shape)
    h = a.hidden_size_per_attention_head * a.num_attention_heads_per_partition
    x = _OnGpu(4096)
    x.shape = torch.Size((2, 1, h))
    got = []
    monkeypatch.setattr(transformer.kernel_lib, "_CALLS", calls)
    monkeypatch.setattr(transformer, "layer_infer", lambda *args, **kw: got.append(kw["ffn"]) or "out")
    monkeypatch.setattr(transformer.kv_cache, "extend", lambda *args: types.SimpleNamespace())
    with torch.no_grad():
        out = layer._infer(x, None)
    assert (out, got) == (("out", [width]) if up == down else (None, []))
    # any other weight or bias that does not fit
    for module, name in ((layer.input_layernorm, "weight"), (a.query_key_value, "weight"), (a.dense, "weight"),
                         (m.linear1, "bias"), (m.linear2, "bias")):
        fake = module.__dict__[name]
        fit, fake.shape = fake.shape, torch.Size((fake.shape[0] + 8,) + tuple(fake.shape[1:]))
        with torch.no_grad():
            assert layer._infer(x, None) is None
        fake.shape = fit


@pytest.mark.gpu
@pytest.mark.parametrize("up,down", [(520, 520), (1536, 1536), (520, 1024)])
def test_a_generation_step_with_an_mlp_of_another_width(up, down, monkeypatch):
    """The same on the GPU: the bits of the op-by-op path, and its refusal of weights that do not fit one another."""
    from common import tiny_config
    from test_model_gpu import _build
    from gpt_neox_b200.models import transformer
    _, model = _build(tiny_config(num_layers=2, hidden_size=256, num_attention_heads=4, seq_length=512, pipe_parallel_size=0,
                                  max_position_embeddings=512, synthetic_vocab_size=1000, attention_config=[[["flash"], 2]],
                                  distributed_backend="nccl", precision="bfloat16"))
    model.eval()
    model.inference_mode(use_cache=True)
    layers = [m for m in model.modules() if isinstance(m, transformer.ParallelTransformerLayer)]
    _resized_mlp(layers[1], up, down)
    native, call = [], transformer.layer_infer
    monkeypatch.setattr(transformer, "layer_infer", lambda *a, **k: (native.append(k["ffn"]), call(*a, **k))[1])
    tokens, pos = torch.randint(0, 1000, (3, 300), device="cuda"), torch.arange(300, device="cuda")[None].expand(3, -1)

    def steps():
        model.clear_cache()
        out, at = [], 0
        with torch.no_grad():
            for n in (5, 1, 290, 1):
                out.append(model((tokens[:, at:at + n].contiguous(), pos[:, at:at + n].contiguous(), None)))
                at += n
        return out

    if up != down:
        with pytest.raises(AssertionError, match="inner dimensions differ"):
            steps()
        return
    one = steps()
    assert native == [1024, up] * 4
    handles = [l.mlp.register_forward_hook(lambda *a: None) for l in layers]
    ops = steps()
    for handle in handles:
        handle.remove()
    assert len(native) == 8 and all(torch.equal(a, b) for a, b in zip(one, ops))

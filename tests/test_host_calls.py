"""Native calls into the kernel library (csrc/host_calls.cpp): arguments, and what a layer's modules are asked, on the CPU."""
import ctypes as C

import pytest
import torch

from gpt_neox_b200 import build
from gpt_neox_b200.ops import _lib


@pytest.fixture(scope="module")
def calls():
    build.build_host_calls()
    return _lib._load_calls()


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

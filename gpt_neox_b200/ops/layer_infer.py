"""A parallel-residual transformer layer of a generation step in one native call (csrc/layer_infer.cu).

The kernels and their order are those of the op-by-op path; what goes is the host work between them (a step of a few
tokens is bound by it).  ``models/transformer.py`` decides when a layer may take this path.
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib
from .gemm import LAUNCHES, PAIR_GEMM

_P, _I, _F = C.c_void_p, C.c_int, C.c_float


class Args(C.Structure):
    """``nx_layer_infer_args`` of csrc/layer_infer.cu."""
    _fields_ = ([(n, _P) for n in ("x", "ln1_w", "ln1_b", "ln2_w", "ln2_b", "w_qkv", "b_qkv", "w_dense", "b_dense", "w1",
                                   "b1", "w2", "b2", "cos", "sin", "alibi", "cache", "work", "stats", "out")]
                + [("cache_kv_stride", C.c_longlong)]
                + [(n, _I) for n in ("s", "b", "h", "np", "kvp", "hn", "ffn", "past", "rot", "window", "gelu_tanh",
                                     "pair_gemm")]
                + [("eps", _F), ("scale", _F)])


def takes(*tensors) -> bool:
    """Whether the kernels read these tensors where they are: contiguous, 16-byte aligned, one 16-bit type."""
    dt = tensors[0].dtype
    return dt in _lib.H16 and all(t is None or (t.dtype == dt and t.is_cuda and t.is_contiguous() and t.data_ptr() % 16 == 0)
                                  for t in tensors)


def layer_infer(x, norms, qkv, dense, up, down, cos, sin, alibi, present, past, *, heads, kv_heads, head_dim, rot, window,
                scale, eps, gelu):
    """x [s, b, h] -> x + attention + MLP [s, b, h].  ``norms``: (w1, b1, w2, b2); ``qkv`` .. ``down``: (weight, bias or
    None); ``present`` [2, past + s, b, kv_heads, head_dim]: the cache, whose last s rows are written."""
    s, b, h = x.shape
    lib = _lib.lib(x)
    out = torch.empty_like(x)
    ptr = lambda t: None if t is None else t.data_ptr()
    args = Args(x.data_ptr(), *map(ptr, norms), *map(ptr, qkv), *map(ptr, dense), *map(ptr, up), *map(ptr, down), ptr(cos),
                ptr(sin), ptr(alibi), present.data_ptr(), None, None, out.data_ptr(), present.stride(0), s, b, h, heads,
                kv_heads, head_dim, up[0].shape[0], past, rot, window, int(gelu == "tanh"), int(PAIR_GEMM["on"]), eps, scale)
    work = torch.empty(lib.nx_layer_infer_work(C.byref(args)), device=x.device, dtype=x.dtype)
    stats = torch.empty(lib.nx_layer_infer_stats(C.byref(args)), device=x.device, dtype=torch.float32)
    args.work, args.stats = work.data_ptr(), stats.data_ptr()
    LAUNCHES["n"] += 7
    _lib.check(lib.nx_layer_infer(C.byref(args), _lib.stream()), "nx_layer_infer")
    return out

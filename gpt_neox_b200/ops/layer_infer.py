"""A parallel-residual transformer layer of a generation step in one native call (csrc/layer_infer.cu).

The kernels and their order are those of the op-by-op path; what goes is the host work between them (a step of a few
tokens is bound by it).  ``models/transformer.py`` decides when a layer may take this path.
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib
from .gemm import LAUNCHES, PAIR_GEMM, EPI_AUX_DERIV, EPI_GELU_ERF, EPI_GELU_TANH

_P, _I, _F = C.c_void_p, C.c_int, C.c_float


class Args(C.Structure):
    """``nx_layer_infer_args`` of csrc/layer_infer.cu."""
    _fields_ = ([(n, _P) for n in ("x", "ln1_w", "ln1_b", "ln2_w", "ln2_b", "w_qkv", "b_qkv", "w_dense", "b_dense", "w1",
                                   "b1", "w2", "b2", "cos", "sin", "cache", "work", "stats", "out")]
                + [("cache_kv_stride", C.c_longlong)]
                + [(n, _I) for n in ("s", "b", "h", "np", "kvp", "hn", "ffn", "past", "rot", "window", "act",
                                     "pair_gemm")]
                + [("eps", _F), ("scale", _F)])


def pointers(*tensors):
    """Device pointers (None for None) if the kernels read these tensors where they are: on the GPU, contiguous, 16-byte
    aligned, of one 16-bit type.  None otherwise."""
    dt = tensors[0].dtype
    if dt not in _lib.H16:
        return None
    out, bits = [], 0
    for t in tensors:
        if t is None:
            out.append(None)
            continue
        if not (t.is_cuda and t.dtype == dt and t.is_contiguous()):
            return None
        p = t.data_ptr()
        bits |= p
        out.append(p)
    return None if bits & 15 else out


def layer_infer(x, ptrs, cos, sin, present, past, *, heads, kv_heads, head_dim, ffn, rot, window, scale, eps, act):
    """x [s, b, h] -> x + attention + MLP [s, b, h].  ``ptrs``: ``pointers`` of x, the norms' weight, bias, weight, bias and
    weight, bias of qkv, dense, up and down; ``present`` [2, past + s, b, kv_heads, head_dim]: the cache, whose last s rows
    are written.  ``act``: ("tanh" or "erf", whether a recorded pass would store the GeLU's derivative).  One scratch
    allocation holds what csrc/layer_infer.cu names."""
    s, b, h = x.shape
    lib = _lib.lib(x)
    out = torch.empty_like(x)
    rows, width = s * b, heads * head_dim
    stats = (2 * rows + b * heads * ((s + 127) // 128 * 128) + 3) // 4 * 4      # fp32; what follows stays 16-byte aligned
    work = torch.empty(2 * stats + rows * (3 * h + 2 * width + 2 * kv_heads * head_dim + ffn), device=x.device, dtype=x.dtype)
    w = work.data_ptr()
    args = Args(*ptrs, cos.data_ptr(), sin.data_ptr(), present.data_ptr(), w + 4 * stats, w, out.data_ptr(), present.stride(0),
                s, b, h, heads, kv_heads, head_dim, ffn, past, rot, window, (EPI_GELU_TANH if act[0] == "tanh" else EPI_GELU_ERF) | (EPI_AUX_DERIV if act[1] else 0), int(PAIR_GEMM["on"]), eps, scale)
    LAUNCHES["n"] += 8
    _lib.check(lib.nx_layer_infer(C.byref(args), _lib.stream()), "nx_layer_infer")
    return out

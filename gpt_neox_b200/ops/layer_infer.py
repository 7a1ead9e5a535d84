"""A parallel-residual transformer layer of a generation step in one native call (csrc/layer_infer.cu).

The kernels and their order are those of the op-by-op path; what goes is the host work between them (a step of a few
tokens is bound by it).  ``models/transformer.py`` decides when a layer may take this path.
"""
from __future__ import annotations

import struct

import torch

from . import _lib
from .gemm import LAUNCHES, PAIR_GEMM, EPI_AUX_DERIV, EPI_GELU_ERF, EPI_GELU_TANH

#: ``nx_layer_infer_args`` of csrc/layer_infer.cu behind its first 13 pointers: the size of the whole; cos, sin, cache, work,
#: stats, out, cache_kv_stride; s, b, h, np, kvp, hn, ffn, past, rot, window, act, pair_gemm; eps, scale
_TAIL = struct.Struct("@q6Pq12i2f")
_BYTES = 13 * 8 + _TAIL.size


def layer_infer(x, ptrs, cos, sin, present, past, *, heads, kv_heads, head_dim, ffn, rot, window, scale, eps, act):
    """x [s, b, h] -> x + attention + MLP [s, b, h].  ``ptrs``: the addresses that ``weights`` of csrc/host_calls.cpp gives for x, the
    two norms, qkv, dense, up and down; ``present`` [2, past + s, b, kv_heads, head_dim]: the cache, whose last s rows are
    written.  ``act``: ("tanh" or "erf", whether a recorded pass would store the GeLU's derivative).  One scratch allocation
    holds what csrc/layer_infer.cu names."""
    s, b, h = x.shape
    lib = _lib.lib(x)
    out = torch.empty_like(x)
    rows, width = s * b, heads * head_dim
    stats = (2 * rows + b * heads * ((s + 127) // 128 * 128) + 3) // 4 * 4      # fp32; what follows stays 16-byte aligned
    work = torch.empty(2 * stats + rows * (3 * h + 2 * width + 2 * kv_heads * head_dim + ffn), device=x.device, dtype=x.dtype)
    w = work.data_ptr()
    args = ptrs + _TAIL.pack(
        _BYTES, cos.data_ptr(), sin.data_ptr(), present.data_ptr(), w + 4 * stats, w, out.data_ptr(), present.stride(0), s, b, h,
        heads, kv_heads, head_dim, ffn, past, rot, window,
        (EPI_GELU_TANH if act[0] == "tanh" else EPI_GELU_ERF) | (EPI_AUX_DERIV if act[1] else 0), int(PAIR_GEMM["on"]),
        eps, scale)
    status = lib.nx_layer_infer(args, _lib.stream())
    if status > 0:
        _lib.check(status, "nx_layer_infer")
    LAUNCHES["n"] -= status        # (minus the number of launches)
    return out

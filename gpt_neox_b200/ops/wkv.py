"""RWKV-6 WKV operator (csrc/wkv6.cu): chunk-parallel linear recurrence with data-dependent decay.

``r, k, v, w``: ``[batch, time, heads * N]`` views with contiguous channels (time-major memory is fine);
``u``: ``[heads, N]``.  ``w`` is the log-log decay: the per-step decay is ``exp(-exp(w))``.
Reference: ``WKV`` autograd function, megatron/model/rwkv/v6/rwkv.py:12-97.
"""
from __future__ import annotations

import torch

from . import _lib
from .gemm import LAUNCHES


def wkv6_reference(r, k, v, w, u):
    """Sequential fp32 statement. Returns y [b, t, c] in the dtype of ``r``."""
    B, T, C = r.shape
    H, N = u.shape
    dt = r.dtype
    r, k, v = (x.float().reshape(B, T, H, N) for x in (r, k, v))
    d = torch.exp(-torch.exp(w.float())).reshape(B, T, H, N)
    uf = u.float()
    S = r.new_zeros(B, H, N, N)
    ys = []
    for t in range(T):
        kv = k[:, t, :, :, None] * v[:, t, :, None, :]
        ys.append(torch.einsum("bhi,bhij->bhj", r[:, t], uf[None, :, :, None] * kv + S))
        S = d[:, t, :, :, None] * S + kv
    return torch.stack(ys, 1).reshape(B, T, C).to(dt)


def decay_grad_from_gr_gk(r, k, v, w, u, gy, gr, gk):
    """dL/dw from gr and gk: with Q_t[i] = sum_j dL/dS_t[i][j] * S_t[i][j] one has
    Q_{t-1} - Q_t = r_t gr_t - k_t gk_t and  dL/d(ew_t) = Q_t - k_t (gk_t - r_t u <gy_t, v_t>)."""
    B, T, C = r.shape
    H, N = u.shape
    f = lambda x: x.float().reshape(B, T, H, N)
    r_, k_, v_, gy_, gr_, gk_ = f(r), f(k), f(v), f(gy), f(gr), f(gk)
    s = (gy_ * v_).sum(-1, keepdim=True)
    delta = r_ * gr_ - k_ * gk_
    Q = delta.flip(1).cumsum(1).flip(1) - delta              # exclusive reverse cumulative sum
    g_ew = Q - k_ * (gk_ - r_ * u.float()[None, None] * s)
    ew = -torch.exp(w.float()).reshape(B, T, H, N)
    gw = (g_ew * ew).reshape(B, T, C)
    gu = (r_ * k_ * s).sum((0, 1))
    return gw, gu


def _same_layout(*ts):
    """Views sharing (batch, time) strides with contiguous channels; copies to time-major otherwise."""
    s0 = (ts[0].stride(0), ts[0].stride(1))
    if all(t.stride(2) == 1 and (t.stride(0), t.stride(1)) == s0 for t in ts):
        return ts
    B, T, C = ts[0].shape
    out = []
    for t in ts:
        buf = torch.empty((T, B, C), device=t.device, dtype=t.dtype).transpose(0, 1)
        buf.copy_(t)
        out.append(buf)
    return tuple(out)


class _WkvFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, r, k, v, w, u):
        B, T, C = r.shape
        H, N = u.shape
        r, k, v, w = _same_layout(r, k, v, w)
        u32 = u.float().contiguous()
        lib = _lib.lib(r)
        nc = lib.nx_wkv6_head_chunks(B, T, H, N)
        dev = r.device
        local = start = sumew = None
        if nc > 1:
            local = torch.empty((B, H, nc, N, N), device=dev, dtype=torch.float32)
            start = torch.empty_like(local)
            sumew = torch.empty((B, H, nc, N), device=dev, dtype=torch.float32)
        y = torch.empty((T, B, C), device=dev, dtype=r.dtype).transpose(0, 1)
        LAUNCHES["n"] += 1 if nc == 1 else 3
        _lib.check(lib.nx_wkv6_fwd(_lib.ptr(r), _lib.ptr(k), _lib.ptr(v), _lib.ptr(w), r.stride(0), r.stride(1),
                                   _lib.ptr(u32), _lib.ptr(y), y.stride(0), y.stride(1), _lib.ptr(local),
                                   _lib.ptr(start), _lib.ptr(sumew), B, T, H, N, _lib.stream()), "nx_wkv6_fwd")
        ctx.save_for_backward(r, k, v, w, u32, start)
        ctx.u_dtype = u.dtype
        return y

    @staticmethod
    def backward(ctx, gy):
        r, k, v, w, u32, start = ctx.saved_tensors
        B, T, C = r.shape
        H, N = u32.shape
        if gy.stride(2) != 1 or (gy.stride(0), gy.stride(1)) != (r.stride(0), r.stride(1)):
            gy = torch.empty((T, B, C), device=gy.device, dtype=gy.dtype).transpose(0, 1).copy_(gy)
            r, k, v, w, gy = _same_layout(r, k, v, w, gy)      # (time-major already, as a rule: nothing to copy)
        dev = r.device
        gr, gk, gv, gw = (torch.empty((T, B, C), device=dev, dtype=r.dtype).transpose(0, 1) for _ in range(4))
        gr32 = torch.empty((T, B, C), device=dev, dtype=torch.float32).transpose(0, 1)
        if B * T == 0:
            return gr, gk, gv, gw, torch.zeros((H, N), device=dev, dtype=ctx.u_dtype)
        gu = torch.empty((H, N), device=dev, dtype=torch.float32)
        gu_part = torch.empty((B, 1 if start is None else start.shape[2], H, N), device=dev, dtype=torch.float32)
        local = rstart = sumew = None
        if start is not None:
            local, rstart = torch.empty_like(start), torch.empty_like(start)
            sumew = torch.empty(start.shape[:4], device=dev, dtype=torch.float32)
        lib = _lib.lib(r)
        LAUNCHES["n"] += lib.nx_wkv6_bwd_launches(B, T, H, N) + (0 if start is None else 2)
        _lib.check(lib.nx_wkv6_bwd(
            _lib.ptr(r), _lib.ptr(k), _lib.ptr(v), _lib.ptr(w), _lib.ptr(gy), r.stride(0), r.stride(1), _lib.ptr(u32),
            _lib.ptr(gr), _lib.ptr(gk), _lib.ptr(gv), _lib.ptr(gw), _lib.ptr(gr32), _lib.ptr(gu), _lib.ptr(gu_part),
            gr.stride(0), gr.stride(1), _lib.ptr(local), _lib.ptr(start), _lib.ptr(rstart), _lib.ptr(sumew), B, T, H, N,
            _lib.stream()), "nx_wkv6_bwd")
        return gr, gk, gv, gw, gu.to(ctx.u_dtype)


def wkv6(r, k, v, w, u):
    """y [b, t, c] of the RWKV-6 recurrence; differentiable in all five arguments."""
    if r.is_cuda:
        if r.dtype not in _lib.H16 or u.shape[1] not in (32, 64):
            raise _lib.KernelError("wkv6: CUDA path needs bf16 and head size 32 or 64")
        return _WkvFn.apply(r, k, v, w, u)
    return wkv6_reference(r, k, v, w, u)

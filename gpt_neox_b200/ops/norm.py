"""LayerNorm / RMSNorm with fp32 statistics.

CUDA bf16 tensors run ``nx_norm_fwd`` / ``nx_norm_bwd`` (csrc/norm.cu); everything else runs the
PyTorch statement of the same math (megatron/model/norms.py:62-99 for RMSNorm,
``torch.nn.LayerNorm`` for LayerNorm), which is also the oracle in the tests.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from . import _lib
from .gemm import LAUNCHES

LN, RMS = 0, 1


def _cuda_ok(x: torch.Tensor) -> bool:
    return x.is_cuda and x.dtype in _lib.H16 and x.shape[-1] % 8 == 0


def _accum_param_grad(param: torch.Tensor, g_f32: torch.Tensor):
    """Route a fp32 parameter gradient: into ``main_grad`` if the engine installed one."""
    mg = getattr(param, "main_grad", None)
    if mg is not None:
        mg.add_(g_f32.view_as(mg))
        return None
    return g_f32.to(param.dtype)


def _forward(kind, x, gamma, beta, eps, gamma2, beta2):
    """-> (x as contiguous rows, y1, y2 or None, mean or None, rstd)."""
    H = x.shape[-1]
    x2 = x.reshape(-1, H)
    if not x2.is_contiguous():
        x2 = x2.contiguous()
    rows = x2.shape[0]
    y1 = torch.empty_like(x2)
    y2 = torch.empty_like(x2) if gamma2 is not None else None
    mean = torch.empty(rows, device=x.device, dtype=torch.float32) if kind == LN else None
    rstd = torch.empty(rows, device=x.device, dtype=torch.float32)
    LAUNCHES["n"] += 1
    _lib.check(_lib.lib(x2).nx_norm_fwd(
        kind, x2, gamma, beta, y1, gamma2,
        beta2, y2, mean, rstd, rows, H, float(eps),
        _lib.stream()), "nx_norm_fwd")
    return x2, y1, y2, mean, rstd


def _outputs(x, x2, y1, y2, carry):
    outs = (y1.view(x.shape),) + ((y2.view(x.shape),) if y2 is not None else ())
    if carry:
        return (x2.view(x.shape),) + outs
    return outs if y2 is not None else outs[0]


def _run(kind, x, gamma, beta, eps, gamma2=None, beta2=None, carry=False):
    if _lib.untracked():
        x2, y1, y2, _, _ = _forward(kind, x, gamma, beta, eps, gamma2, beta2)
        return _outputs(x, x2, y1, y2, carry)
    return _NormFn.apply(kind, x, gamma, beta, eps, gamma2, beta2, carry)


class _NormFn(torch.autograd.Function):
    """One or two norms of ``x``.  ``carry``: also return ``x`` itself as the first output, so that the
    gradient of the residual stream flows through this node and is added inside the backward kernel
    (no separate accumulation pass over the activations)."""

    @staticmethod
    def forward(ctx, kind, x, gamma, beta, eps, gamma2, beta2, carry):
        x2, y1, y2, mean, rstd = _forward(kind, x, gamma, beta, eps, gamma2, beta2)
        ctx.kind, ctx.dual, ctx.shape, ctx.carry = kind, gamma2 is not None, x.shape, carry
        ctx.params = (gamma, beta, gamma2, beta2)       # the parameters themselves: their main_grad takes the gradients
        ctx.save_for_backward(x2, gamma, gamma2, mean, rstd)
        return _outputs(x, x2, y1, y2, carry)

    @staticmethod
    def backward(ctx, *gys):
        x2, gamma, gamma2, mean, rstd = ctx.saved_tensors
        rows, H = x2.shape
        L = _lib.lib(x2)

        def flat(t):
            if t is None:
                return None
            t = t.reshape(rows, H)
            return t if t.is_contiguous() else t.contiguous()

        gres = flat(gys[0]) if ctx.carry else None
        gys = gys[1:] if ctx.carry else gys
        g1 = flat(gys[0])
        g2 = flat(gys[1]) if ctx.dual else None
        grads = [None] * 4                              # gamma, beta, gamma2, beta2
        dx = gres
        if g1 is not None or g2 is not None:
            # one gradient stream (ga with gamma ia) or, for a dual norm with both, two
            norms = [i for i, g in ((0, g1), (2, g2)) if g is not None]
            ia, both = norms[0], len(norms) == 2
            ga, gma, gmb = (g1, g2)[ia // 2], (gamma, gamma2)[ia // 2], (gamma2 if both else None)
            blocks = L.nx_norm_bwd_blocks(rows)
            ws = torch.empty(blocks * (4 if both else 2) * H, device=x2.device, dtype=torch.float32)
            dx = torch.empty_like(x2)
            # parameter gradients: straight into the fp32 main_grad buffers (added by the partial-sum reduction
            # kernel) when every parameter of this call has one of its own (the kernel's blocks add to them without
            # atomics: a parameter that both norms use must not be added to twice at once), else into fresh buffers: of
            # the parameters' own type when autograd takes them as they are, fp32 when some main_grad has to be added to
            need = ctx.needs_input_grad
            want = [i + j for i in norms for j in (0, 1) if ctx.params[i + j] is not None and need[(2, 3, 5, 6)[i + j]]]
            mgs = [getattr(ctx.params[i], "main_grad", None) for i in want]
            direct = all(m is not None and m.dtype == torch.float32 and m.is_contiguous() and m.numel() == H for m in mgs) \
                and len({m.data_ptr() for m in mgs}) == len(mgs)
            out16 = not direct and all(m is None and ctx.params[i].dtype == x2.dtype for i, m in zip(want, mgs))
            out = [None] * 4
            for i, m in zip(want, mgs):
                out[i] = m if direct else torch.empty(H, device=x2.device, dtype=x2.dtype if out16 else torch.float32)
            LAUNCHES["n"] += 2
            _lib.check(L.nx_norm_bwd(
                ctx.kind, ga, g2 if both else None, x2, mean, rstd,
                gma, gmb, gres, dx, out[ia], out[ia + 1],
                out[2] if both else None, out[3] if both else None, ws, rows, H,
                1 if direct else 0, 1 if out16 else 0, _lib.stream()), "nx_norm_bwd")
            if not direct:
                for i in want:
                    p = ctx.params[i]
                    grads[i] = out[i].view_as(p) if out16 else _accum_param_grad(p, out[i])
        return (None, dx.view(ctx.shape) if dx is not None else None, grads[0], grads[1], None, grads[2], grads[3], None)


def layer_norm(x, weight, bias=None, eps: float = 1e-5, carry: bool = False):
    """``carry``: return ``(x, y)``; the gradient of that ``x`` (the residual stream) is added to the
    norm's input gradient inside the backward kernel."""
    if _cuda_ok(x):
        return _run(LN, x, weight, bias, eps, carry=carry)
    if carry:
        return x, layer_norm(x, weight, bias, eps)
    if x.is_cuda:
        raise _lib.KernelError(f"layer_norm: CUDA path needs bf16 and H % 8 == 0, got {x.dtype} {tuple(x.shape)}")
    return F.layer_norm(x, (x.shape[-1],), weight, bias, eps)


def dual_layer_norm(x, w1, b1, w2, b2, eps: float = 1e-5, carry: bool = False):
    """Two LayerNorms of the same input from one pass (GPT-J parallel residual,
    megatron/model/transformer.py:1083).  ``carry``: return ``(x, y1, y2)`` where the first output
    stands for the residual stream; its gradient is added to the norms' input gradient inside the
    backward kernel."""
    if _cuda_ok(x):
        return _run(LN, x, w1, b1, eps, w2, b2, carry)
    y = layer_norm(x, w1, b1, eps), layer_norm(x, w2, b2, eps)
    return (x,) + y if carry else y


def rms_norm(x, weight, eps: float = 1e-8, carry: bool = False):
    if _cuda_ok(x):
        return _run(RMS, x, weight, None, eps, carry=carry)
    if carry:
        return x, rms_norm(x, weight, eps)
    if x.is_cuda:
        raise _lib.KernelError(f"rms_norm: CUDA path needs bf16 and H % 8 == 0, got {x.dtype}")
    dtype = x.dtype
    xf = x.float()
    var = xf.pow(2).mean(-1, keepdim=True)
    return (weight.float() * (xf * torch.rsqrt(var + eps))).to(dtype)


def dual_rms_norm(x, w1, w2, eps: float = 1e-8):
    if _cuda_ok(x):
        return _run(RMS, x, w1, None, eps, w2, None)
    return rms_norm(x, w1, eps), rms_norm(x, w2, eps)

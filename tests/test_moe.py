"""Dropless MoE on one rank against a per-token loop (reference tests: tests/model/test_model_train.py moe params)."""
import pytest
import torch

from gpt_neox_b200 import parallel as mpu
from gpt_neox_b200.config import NeoXArgs
from gpt_neox_b200.models.init_functions import get_init_methods
from gpt_neox_b200.models.moe import ParallelDroplessMoE

from common import tiny_config


def _args(**kw):
    cfg = tiny_config(**{**dict(use_cpu_initialization=True, moe_num_experts=4, moe_top_k=2,
                             moe_expert_interval=1), **kw})
    a = NeoXArgs.from_dict(cfg)
    mpu.destroy_model_parallel()
    mpu.initialize_model_parallel(1)
    return a


@pytest.mark.parametrize("act,router", [("gelu", "topk"), ("swiglu", "topk"), ("gelu", "sinkhorn")])
def test_dropless_moe_matches_token_loop(act, router):
    a = _args(activation=act, moe_router_type=router, precision="fp32")
    torch.manual_seed(0)
    im, om = get_init_methods(a)
    moe = ParallelDroplessMoE(a, im, om).eval()
    x = torch.randn(8, 2, a.hidden_size, requires_grad=True)
    y = moe(x)
    assert y.shape == x.shape
    w, idx = moe.router(x)
    mlp = moe.experts.mlp
    E = a.moe_num_experts
    x2 = x.reshape(-1, a.hidden_size)
    want = torch.zeros_like(x2)
    for t in range(x2.shape[0]):
        for j in range(idx.shape[1]):
            e = int(idx[t, j])
            w1 = mlp.w1.view(E, -1, a.hidden_size)[e]
            w2 = mlp.w2.view(E, -1, a.hidden_size)[e]
            if act == "swiglu":
                w3 = mlp.w3.view(E, -1, a.hidden_size)[e]
                h = torch.nn.functional.silu(x2[t] @ w1.T) * (x2[t] @ w3.T)
            else:
                h = torch.nn.functional.gelu(x2[t] @ w1.T)
            want[t] += w[t, j] * (h @ w2)
    torch.testing.assert_close(y.reshape(-1, a.hidden_size), want, rtol=1e-4, atol=1e-5)
    y.sum().backward()
    assert x.grad is not None and torch.isfinite(x.grad).all()
    assert mlp.w1.grad is not None and moe.router.layer.weight.grad is not None


def test_sinkhorn_training_balances_and_is_differentiable():
    a = _args(moe_router_type="sinkhorn", precision="fp32", moe_top_k=1)
    im, om = get_init_methods(a)
    moe = ParallelDroplessMoE(a, im, om).train()
    x = torch.randn(16, 2, a.hidden_size, requires_grad=True)
    moe(x).sum().backward()
    assert torch.isfinite(x.grad).all()


@pytest.mark.gpu
@pytest.mark.parametrize("T,k,E,h,ffn", [(512, 2, 4, 256, 512), (300, 1, 8, 128, 256), (1024, 2, 8, 768, 3072)])
def test_moe_kernel_path_matches_torch_path(T, k, E, h, ffn):
    """Plan / permute / grouped-GEMM kernels against the per-expert torch loop with the same weights."""
    from gpt_neox_b200.ops import _lib
    from gpt_neox_b200.ops import moe as M
    torch.manual_seed(0)
    dev = "cuda"
    x = torch.randn(T, h, device=dev).bfloat16().requires_grad_(True)
    w1 = (torch.randn(E * ffn, h, device=dev) * 0.05).bfloat16().requires_grad_(True)
    w2 = (torch.randn(E * ffn, h, device=dev) * 0.05).bfloat16().requires_grad_(True)
    logits = torch.randn(T, E, device=dev)
    wts, idx = torch.softmax(logits, -1).topk(k, dim=-1)
    wts = wts.bfloat16().requires_grad_(True)
    plan = M.Plan(idx, E)
    counts = torch.bincount(idx.reshape(-1), minlength=E)
    assert torch.equal(plan.counts.long(), counts)
    off = plan.offsets.long()
    assert bool((off % 128 == 0).all()) and bool(((off[1:] - off[:-1]) >= counts).all())
    # stable: copies of one expert keep their original order
    d = plan.dest_row.long()
    for e in range(E):
        rows = d[idx.reshape(-1) == e]
        assert bool((rows[1:] > rows[:-1]).all()) and (len(rows) == 0 or int(rows[0]) == int(off[e]))
    out = M.experts_gelu(x, wts, idx, w1, w2, E)
    g = torch.randn_like(out)
    out.backward(g)
    # fp32 statement
    xr, w1r, w2r, wr = (t.detach().float().requires_grad_(True) for t in (x, w1, w2, wts))
    ref = torch.zeros(T, h, device=dev)
    for e in range(E):
        sel = (idx == e)
        tok, slot = sel.nonzero(as_tuple=True)
        if len(tok) == 0:
            continue
        hh = torch.nn.functional.gelu(xr[tok] @ w1r[e * ffn:(e + 1) * ffn].t())
        ref = ref.index_add(0, tok, (hh @ w2r[e * ffn:(e + 1) * ffn]) * wr[tok, slot].unsqueeze(-1))
    ref.backward(g.float())
    rel = lambda a, b: ((a.float() - b).norm() / (b.norm() + 1e-9)).item()
    assert rel(out, ref) < 2e-2
    assert rel(x.grad, xr.grad) < 3e-2 and rel(w1.grad, w1r.grad) < 3e-2 and rel(w2.grad, w2r.grad) < 3e-2
    assert rel(wts.grad, wr.grad) < 3e-2
    assert _lib.read_device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("ws,T,k,E,h,ffn", [(2, 200, 2, 4, 256, 512), (4, 96, 1, 8, 128, 256), (8, 64, 2, 8, 768, 1024)])
def test_expert_parallel_peer_memory_path_matches_fp32_oracle(ws, T, k, E, h, ffn):
    """Expert parallelism over peer memory with the ranks emulated on one GPU: ``ws`` workspaces driven in
    lockstep phase by phase (stream order stands in for the rank barriers), against the fp32 per-expert loop
    over all ranks' tokens.  Covers the pull-gather, the pull-combine and the routing-weight gradient."""
    from gpt_neox_b200.ops import _lib
    from gpt_neox_b200.ops import moe_ep as EP
    torch.manual_seed(1)
    dev = "cuda"
    El = E // ws
    w1 = (torch.randn(E * ffn, h, device=dev) * 0.05).bfloat16()
    w2 = (torch.randn(E * ffn, h, device=dev) * 0.05).bfloat16()
    xs = [torch.randn(T, h, device=dev).bfloat16() for _ in range(ws)]
    routed = [torch.softmax(torch.randn(T, E, device=dev), -1).topk(k, dim=-1) for _ in range(ws)]
    wts = [r[0].bfloat16() for r in routed]
    idx = [r[1] for r in routed]
    gs = [torch.randn(T, h, device=dev).bfloat16() for _ in range(ws)]
    w1s = [w1[r * El * ffn:(r + 1) * El * ffn].contiguous() for r in range(ws)]
    w2s = [w2[r * El * ffn:(r + 1) * El * ffn].contiguous() for r in range(ws)]
    Ws = EP.EpWorkspace.emulated(ws, T, k, h, El)
    ids = [i.reshape(-1).to(torch.int32) for i in idx]
    wfs = [w.reshape(-1).contiguous() for w in wts]
    for r in range(ws):
        EP.fwd_publish(Ws[r], xs[r], ids[r])
    st = [EP.fwd_experts(Ws[r], w1s[r], w2s[r], "erf") for r in range(ws)]
    outs = [EP.fwd_combine(Ws[r], ids[r], wfs[r]) for r in range(ws)]
    for r in range(ws):
        EP.bwd_publish(Ws[r], gs[r], wfs[r])
    dws = [EP.bwd_experts(Ws[r], *st[r], w1s[r], w2s[r], "erf") for r in range(ws)]
    back = [EP.bwd_combine(Ws[r], ids[r]) for r in range(ws)]
    # fp32 statement over the concatenated tokens
    X = torch.cat(xs).float().requires_grad_(True)
    Wt = torch.cat(wts).float().requires_grad_(True)
    I = torch.cat(idx)
    w1r, w2r = w1.float().requires_grad_(True), w2.float().requires_grad_(True)
    ref = torch.zeros(ws * T, h, device=dev)
    for e in range(E):
        tok, slot = (I == e).nonzero(as_tuple=True)
        if len(tok) == 0:
            continue
        hh = torch.nn.functional.gelu(X[tok] @ w1r[e * ffn:(e + 1) * ffn].t())
        ref = ref.index_add(0, tok, (hh @ w2r[e * ffn:(e + 1) * ffn]) * Wt[tok, slot].unsqueeze(-1))
    ref.backward(torch.cat(gs).float())
    rel = lambda a, b: ((a.float() - b).norm() / (b.norm() + 1e-9)).item()
    assert rel(torch.cat(outs), ref) < 2e-2
    assert rel(torch.cat([b[0] for b in back]), X.grad) < 3e-2
    assert rel(torch.cat([b[1].view(T, k) for b in back]), Wt.grad) < 3e-2
    assert rel(torch.cat([d[0] for d in dws]), w1r.grad) < 3e-2
    assert rel(torch.cat([d[1] for d in dws]), w2r.grad) < 3e-2
    assert _lib.read_device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", ["erf", "tanh"])
@pytest.mark.parametrize("T,n,K", [(150, 136, 64), (150, 256, 200), (150, 264, 64), (150, 392, 136), (150, 776, 768),
                                   (12000, 1160, 64)])       # the last: several tiles per CTA, pieces prefetched across them
def test_grouped_rows_epilogues(T, n, K, kind, dtype):
    """GeLU with its derivative stored, and the product with a stored derivative, at ragged column counts (tiles of 256, a warp's
    half of 128, pieces of 32) against 64 bits: results are rounded once, the sums behind them are fp32."""
    from gpt_neox_b200.ops import moe as M
    torch.manual_seed(3)
    E = 3
    idx = torch.randint(0, E, (T, 2), device="cuda")
    plan = M.Plan(idx, E)
    src, rows = plan.src_copy, (plan.src_copy >= 0).nonzero().flatten()
    mk = lambda *s, scale=1.0: (torch.randn(*s, device="cuda") * scale).to(dtype)
    xp = M.gather_rows(mk(T, K), plan)
    w = mk(E * n, K, scale=K ** -0.5)
    deriv = torch.empty((plan.max_rows, n), device="cuda", dtype=dtype)
    act = M.grouped_gemm_rows(xp, w, plan, n, trans_b=False, gelu=kind, aux_out=deriv, aux_deriv=True)
    prod = M.grouped_gemm_rows(xp, w, plan, n, trans_b=False, dgelu_aux=deriv, dgelu="mul")
    expert = plan.tile_expert.long()[rows // 128]
    z = torch.einsum("rk,rnk->rn", xp[rows].double(), w.view(E, n, K).double()[expert]).requires_grad_()
    want = torch.nn.functional.gelu(z, approximate="tanh" if kind == "tanh" else "none")
    (wd,) = torch.autograd.grad(want.sum(), z)
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
    # (tanh.approx has an absolute error of 2^-11, the erf series 1e-7; |z| < 8)
    slack = 8 * 2 ** -11 if kind == "tanh" else 2 ** -18
    assert (act[rows] - want).abs().sub(eps * want.abs()).max() <= slack
    assert (deriv[rows] - wd).abs().sub(eps * wd.abs()).max() <= slack
    ref = z.detach() * deriv[rows].double()
    assert (prod[rows] - ref).abs().sub(eps * ref.abs()).max() <= 2 ** -18


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["mul", "erf", "tanh"])
@pytest.mark.parametrize("T,n,K", [(9000, 3072, 64), (20000, 520, 192)])
def test_grouped_rows_read_their_side_operand_before_the_next_piece(T, n, K, kind):
    """The side operand's pieces follow each other through one box of shared memory: short reductions, where the epilogue
    waits for nothing else, many pieces per CTA, run over and over.  Every run has the bits of the first, and those are the
    fp32 product rounded once (sums and erf are 2 ** -20 off, tanh.approx 2 ** -11, the derivative up to 16 times that)."""
    from gpt_neox_b200.ops import moe as M
    torch.manual_seed(5)
    E, dtype = 4, torch.bfloat16
    plan = M.Plan(torch.randint(0, E, (T, 2), device="cuda"), E)
    rows = (plan.src_copy >= 0).nonzero().flatten()
    xp = M.gather_rows(torch.randn(T, K, device="cuda").to(dtype), plan)
    w = (torch.randn(E * n, K, device="cuda") * K ** -0.5).to(dtype)
    side = torch.randn(plan.max_rows, n, device="cuda").to(dtype)
    run = lambda: M.grouped_gemm_rows(xp, w, plan, n, trans_b=False, dgelu_aux=side, dgelu=kind)
    first = run()
    for _ in range(20):
        assert torch.equal(run()[rows], first[rows])
    expert = plan.tile_expert.long()[rows // 128]
    for e in range(E):
        r = rows[expert == e]
        x = side[r].double().requires_grad_()
        d = x.detach() if kind == "mul" else torch.autograd.grad(
            torch.nn.functional.gelu(x, approximate="tanh" if kind == "tanh" else "none").sum(), x)[0]
        z = xp[r].double() @ w.view(E, n, K)[e].double().t()
        err = (first[r] - z * d).abs() - 2 ** -8 * (z * d).abs()
        assert err.max() <= (2 ** -7 if kind == "tanh" else 2 ** -16) * z.abs().max()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,E,M,N", [(40, 5, 8, 8), (300, 3, 264, 520), (700, 4, 40, 24), (1500, 2, 512, 256), (260, 9, 1000, 136)])
def test_grouped_gemms_at_tile_edges(T, E, M, N, dtype):
    """Row and reduction form against 64 bits at sizes that tiles of 256, pieces of 64 and 32 and 32-byte stores cut, with an
    expert that gets no token: the operand sums are fp32 and rounded once.  Weight gradients: zeros for that expert, and with
    an fp32 main_grad the sum with what was there."""
    from gpt_neox_b200.ops import moe as MO
    torch.manual_seed(7)
    idx = torch.randint(0, E - 1, (T, 2), device="cuda")                 # the last expert has no rows
    idx[idx == 0] = 0 if E < 4 else 1                                    # and with four or more the first one, too
    plan = MO.Plan(idx, E)
    rows = (plan.src_copy >= 0).nonzero().flatten()
    expert = plan.tile_expert.long()[rows // 128]
    mk = lambda *s: torch.randn(*s, device="cuda").to(dtype)
    a, b = MO.gather_rows(mk(T, M), plan), MO.gather_rows(mk(T, N), plan)
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11

    def slack(terms):
        # the tensor core adds 16 products at a time to an fp32 sum, which it cuts off: terms / 16 steps of at most 2^-22 of a
        # partial sum, which stays below 8 sqrt(terms) for products of order 1 (a bound of terms * 2^-22, as if partial sums
        # were of order 1, was too small for 3000 terms: 8e-4 at a sum of 122)
        return (terms / 16 + 1) * 8 * terms ** 0.5 * 2 ** -22

    def close(got, want, terms):
        assert ((got.double() - want).abs() <= eps * want.abs() + slack(terms)).all()       # one rounding to 16 bits

    w, wt = mk(E * N, M), mk(E * M, N)
    got = MO.grouped_gemm_rows(a, w, plan, N, trans_b=False)
    close(got[rows], torch.einsum("rk,rnk->rn", a[rows].double(), w.view(E, N, M).double()[expert]), M)
    got = MO.grouped_gemm_rows(a, wt, plan, N, trans_b=True)
    close(got[rows], torch.einsum("rk,rkn->rn", a[rows].double(), wt.view(E, M, N).double()[expert]), M)
    want = torch.stack([a[rows][expert == e].double().t() @ b[rows][expert == e].double() for e in range(E)])
    weight = torch.nn.Parameter(torch.empty(E * M, N, device="cuda", dtype=dtype))
    got = MO.grouped_wgrad(a, b, plan, weight).view(E, M, N)
    close(got, want, 2 * T)
    assert bool((got[E - 1] == 0).all())
    before = torch.randn(E, M, N, device="cuda")
    weight.main_grad = before.clone().view(E * M, N)
    assert MO.grouped_wgrad(a, b, plan, weight) is None
    got = weight.main_grad.view(E, M, N)
    assert ((got.double() - before.double() - want).abs() <= slack(2 * T) + 2 ** -23 * got.abs()).all()
    assert torch.equal(got[E - 1], before[E - 1])

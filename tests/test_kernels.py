"""Every memory-bound / fused CUDA kernel against a plain PyTorch fp32 reference of the same op."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"
DT = torch.bfloat16     # the 16-bit dtype under test; every test below runs once for bf16 and once for fp16


@pytest.fixture(autouse=True, params=[torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
def _dtype(request):
    global DT
    DT = request.param
    yield
    DT = torch.bfloat16


def rel(a, b):
    a, b = a.float(), b.float()
    return ((a - b).abs().max() / (b.abs().max() + 1e-6)).item()


def bf(*shape, scale=1.0, grad=False):
    t = (torch.randn(*shape, device=DEV) * scale).to(DT)
    return t.requires_grad_(grad)


@pytest.mark.parametrize("rows,H", [(7, 64), (300, 512), (1024, 2048), (33, 4096), (5, 6144), (700, 8192),
                                     (40, 16384), (20000, 1024), (5001, 6144)])   # the last two wrap the stage ring
def test_layernorm_fwd_bwd(rows, H):
    from gpt_neox_b200.ops.norm import layer_norm
    torch.manual_seed(0)
    x, w, b = bf(rows, H, grad=True), (1 + 0.1 * torch.randn(H, device=DEV)).to(DT).requires_grad_(True), \
        bf(H, scale=0.1, grad=True)
    y = layer_norm(x, w, b, 1e-5)
    g = bf(rows, H)
    y.backward(g)
    xr, wr, br = (t.detach().float().requires_grad_(True) for t in (x, w, b))
    yr = F.layer_norm(xr, (H,), wr, br, 1e-5)
    yr.backward(g.float())
    assert rel(y, yr) < 1e-2
    assert rel(x.grad, xr.grad) < 2e-2
    assert rel(w.grad, wr.grad) < 2e-2
    assert rel(b.grad, br.grad) < 2e-2


def test_dual_layernorm_matches_two_norms():
    from gpt_neox_b200.ops.norm import dual_layer_norm
    torch.manual_seed(1)
    rows, H = 257, 1024
    x = bf(rows, H, grad=True)
    ws = [(1 + 0.1 * torch.randn(H, device=DEV)).to(DT).requires_grad_(True) for _ in range(2)]
    bs = [bf(H, scale=0.1, grad=True) for _ in range(2)]
    y1, y2 = dual_layer_norm(x, ws[0], bs[0], ws[1], bs[1], 1e-5)
    g1, g2 = bf(rows, H), bf(rows, H)
    (y1 * g1).sum().backward(retain_graph=True)
    (y2 * g2).sum().backward()
    xr = x.detach().float().requires_grad_(True)
    wr = [w.detach().float().requires_grad_(True) for w in ws]
    br = [b.detach().float().requires_grad_(True) for b in bs]
    r1 = F.layer_norm(xr, (H,), wr[0], br[0], 1e-5)
    r2 = F.layer_norm(xr, (H,), wr[1], br[1], 1e-5)
    ((r1 * g1.float()).sum() + (r2 * g2.float()).sum()).backward()
    assert rel(y1, r1) < 1e-2 and rel(y2, r2) < 1e-2
    assert rel(x.grad, xr.grad) < 2e-2
    for i in range(2):
        assert rel(ws[i].grad, wr[i].grad) < 2e-2
        assert rel(bs[i].grad, br[i].grad) < 2e-2


@pytest.mark.parametrize("rows,H", [(1000, 4096), (77, 6144), (300, 8192), (9, 16384), (5, 32768), (9000, 4096)])
def test_dual_layernorm_with_residual_carry_one_backward_pass(rows, H):
    """(x, y1, y2) = dual norm with the residual stream carried through the node: dx = g_res + both
    norm gradients from ONE backward kernel launch."""
    from gpt_neox_b200.ops.norm import dual_layer_norm
    torch.manual_seed(4)
    x = bf(rows, H, grad=True)
    ws = [(1 + 0.1 * torch.randn(H, device=DEV)).to(DT).requires_grad_(True) for _ in range(2)]
    bs = [bf(H, scale=0.1, grad=True) for _ in range(2)]
    res, y1, y2 = dual_layer_norm(x, ws[0], bs[0], ws[1], bs[1], 1e-5, carry=True)
    g0, g1, g2 = bf(rows, H), bf(rows, H), bf(rows, H)
    ((res * g0).sum() + (y1 * g1).sum() + (y2 * g2).sum()).backward()
    xr = x.detach().float().requires_grad_(True)
    wr = [w.detach().float().requires_grad_(True) for w in ws]
    br = [b.detach().float().requires_grad_(True) for b in bs]
    r1 = F.layer_norm(xr, (H,), wr[0], br[0], 1e-5)
    r2 = F.layer_norm(xr, (H,), wr[1], br[1], 1e-5)
    ((xr * g0.float()).sum() + (r1 * g1.float()).sum() + (r2 * g2.float()).sum()).backward()
    assert torch.equal(res, x)
    assert rel(y1, r1) < 1e-2 and rel(y2, r2) < 1e-2
    assert rel(x.grad, xr.grad) < 2e-2
    for i in range(2):
        assert rel(ws[i].grad, wr[i].grad) < 2e-2
        assert rel(bs[i].grad, br[i].grad) < 2e-2


@pytest.mark.parametrize("rows,H", [(20000, 2048), (4096, 4096)])
def test_norm_gradients_with_residual_carry_repeat_bit_for_bit(rows, H):
    """Rows follow each other through one ring of shared memory; the residual stream's gradient is the value of a row that is
    only used after the next row may have been asked for."""
    from gpt_neox_b200.ops.norm import dual_layer_norm
    torch.manual_seed(31)
    x, ws = bf(rows, H, grad=True), [bf(H, grad=True) for _ in range(4)]
    gs = [bf(rows, H) for _ in range(3)]
    run = lambda: torch.autograd.grad(dual_layer_norm(x, *ws, carry=True), [x, *ws], gs)
    first = run()
    r = [t.detach().double().requires_grad_() for t in (x, *ws)]
    ys = [r[0]] + [F.layer_norm(r[0], (H,), r[i], r[i + 1], 1e-5) for i in (1, 3)]
    (want,) = torch.autograd.grad(ys, r[:1], [t.double() for t in gs])
    # a sum of three gradients in fp32, rounded once: half a unit in the last of 8 bits (11) is up to 2^-8 (2^-11) of the value
    eps = 2 ** -8 if DT == torch.bfloat16 else 2 ** -11
    err = (first[0] - want).abs()
    assert (err <= 1.01 * eps * want.abs() + 1e-5 * want.abs().max()).all()
    for _ in range(20):
        assert all(torch.equal(a, b) for a, b in zip(first, run()))



def test_rmsnorm_carry_adds_residual_gradient():
    from gpt_neox_b200.ops.norm import rms_norm
    torch.manual_seed(5)
    rows, H = 300, 4096
    x, w = bf(rows, H, grad=True), (1 + 0.1 * torch.randn(H, device=DEV)).to(DT).requires_grad_(True)
    res, y = rms_norm(x, w, 1e-6, carry=True)
    g0, g = bf(rows, H), bf(rows, H)
    ((res * g0).sum() + (y * g).sum()).backward()
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    yr = wr * (xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-6))
    ((xr * g0.float()).sum() + (yr * g.float()).sum()).backward()
    assert rel(x.grad, xr.grad) < 2e-2
    assert rel(w.grad, wr.grad) < 2e-2


@pytest.mark.parametrize("rows,H", [(64, 256), (513, 4096), (12000, 2048)])
def test_rmsnorm_fwd_bwd(rows, H):
    from gpt_neox_b200.ops.norm import rms_norm
    torch.manual_seed(2)
    x, w = bf(rows, H, grad=True), (1 + 0.1 * torch.randn(H, device=DEV)).to(DT).requires_grad_(True)
    y = rms_norm(x, w, 1e-8)
    g = bf(rows, H)
    y.backward(g)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    yr = wr * (xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-8))
    yr.backward(g.float())
    assert rel(y, yr) < 1e-2
    assert rel(x.grad, xr.grad) < 2e-2
    assert rel(w.grad, wr.grad) < 2e-2


@pytest.mark.parametrize("act", ["gelu", "gelu_tanh", "relu", "silu"])
def test_bias_act(act):
    from gpt_neox_b200.ops.elementwise import _torch_act, bias_act
    torch.manual_seed(3)
    x, b = bf(100, 768, grad=True), bf(768, grad=True)
    y = bias_act(x, b, act)
    g = bf(100, 768)
    y.backward(g)
    xr, br = x.detach().float().requires_grad_(True), b.detach().float().requires_grad_(True)
    yr = _torch_act(act, xr + br)
    yr.backward(g.float())
    assert rel(y, yr) < 1e-2
    assert rel(x.grad, xr.grad) < 2e-2
    assert rel(b.grad, br.grad) < 2e-2


@pytest.mark.parametrize("kind", ["swiglu", "geglu", "reglu", "bilinear", "glu"])
def test_gated_act(kind):
    from gpt_neox_b200.ops.elementwise import GATED, _torch_act, gated_act
    torch.manual_seed(4)
    x = bf(77, 512, grad=True)
    y = gated_act(x, kind)
    g = bf(77, 256)
    y.backward(g)
    xr = x.detach().float().requires_grad_(True)
    v, gate = xr.chunk(2, dim=-1)
    yr = v * _torch_act(GATED[kind], gate)
    yr.backward(g.float())
    assert rel(y, yr) < 1e-2
    assert rel(x.grad, xr.grad) < 2e-2


def test_bias_dropout_add_and_colsum():
    from gpt_neox_b200.ops.elementwise import bias_dropout_add, colsum
    torch.manual_seed(5)
    x, b, r = bf(64, 1024, grad=True), bf(1024, grad=True), bf(64, 1024, grad=True)
    y = bias_dropout_add(x, b, r, 0.0, True)
    assert rel(y, x.float() + b.float() + r.float()) < 1e-2
    y.sum().backward()
    assert rel(b.grad, torch.full((1024,), 64.0, device=DEV)) < 1e-2
    # dropout: kept fraction and scaling
    x2 = torch.ones(512, 1024, device=DEV, dtype=DT, requires_grad=True)
    y2 = bias_dropout_add(x2, None, None, 0.25, True)
    kept = (y2 != 0).float().mean().item()
    assert abs(kept - 0.75) < 0.02
    assert abs(y2.max().item() - 1 / 0.75) < 0.02
    y2.sum().backward()
    assert torch.equal((x2.grad != 0), (y2 != 0))
    big = bf(4097, 520)
    assert rel(colsum(big, torch.float32), big.float().sum(0)) < 1e-2


def test_softmax_causal_and_masked():
    from gpt_neox_b200.ops.softmax import scaled_causal_softmax, scaled_masked_softmax
    torch.manual_seed(6)
    x = bf(6, 200, 200, grad=True)
    y = scaled_causal_softmax(x, 0.37)
    g = bf(6, 200, 200)
    y.backward(g)
    xr = x.detach().float().requires_grad_(True)
    keep = torch.ones(200, 200, dtype=torch.bool, device=DEV).tril()
    yr = torch.softmax((xr * 0.37).masked_fill(~keep, float("-inf")), -1)
    yr.backward(g.float())
    assert rel(y, yr) < 1e-2
    assert rel(x.grad, xr.grad) < 3e-2
    x4 = bf(2, 3, 50, 3000, grad=True)          # longer than the reference kernels' 2048 cap
    mask = torch.rand(2, 1, 50, 3000, device=DEV) < 0.3
    y4 = scaled_masked_softmax(x4, mask, 0.5)
    g4 = bf(2, 3, 50, 3000)
    y4.backward(g4)
    x4r = x4.detach().float().requires_grad_(True)
    y4r = torch.softmax((x4r * 0.5).masked_fill(mask, -10000.0), -1)
    y4r.backward(g4.float())
    assert rel(y4, y4r) < 1e-2
    assert rel(x4.grad, x4r.grad) < 3e-2


@pytest.mark.parametrize("V,start,full", [(50304, 0, 50304), (1000, 1000, 3000), (257, 0, 257)])
def test_cross_entropy(V, start, full):
    from gpt_neox_b200.ops.cross_entropy import _combine_stats, vocab_parallel_cross_entropy
    torch.manual_seed(7)
    rows = 300
    logits = bf(rows, V, scale=2.0, grad=True)
    labels = torch.randint(0, full, (rows,), device=DEV)
    if full == V:
        loss = vocab_parallel_cross_entropy(logits, labels, start)
        lr = logits.detach().float().requires_grad_(True)
        ref = F.cross_entropy(lr, labels, reduction="none")
        assert rel(loss, ref) < 1e-3
        w = torch.rand(rows, device=DEV)
        (loss * w).sum().backward()
        (ref * w).sum().backward()
        assert rel(logits.grad, lr.grad) < 2e-2
    else:
        # a shard of a larger vocabulary: (max, sumexp, target) statistics must match
        from gpt_neox_b200.ops import _lib
        stats = torch.empty(rows, 3, device=DEV)
        _lib.check(_lib.lib(logits).nx_ce_fwd(_lib.ptr(logits), _lib.ptr(labels), _lib.ptr(stats), rows, V, V, start, 0,
                                        _lib.stream()))
        lf = logits.detach().float()
        m = lf.max(-1).values
        s = torch.exp(lf - m[:, None]).sum(-1)
        loc = labels - start
        inside = (loc >= 0) & (loc < V)
        t = torch.where(inside, lf.gather(-1, loc.clamp(0, V - 1)[:, None]).squeeze(-1), torch.zeros_like(m))
        assert rel(stats[:, 0], m) < 1e-5 and rel(stats[:, 1], s) < 1e-3 and rel(stats[:, 2], t) < 1e-5


def test_adamw_sumsq_clip():
    from gpt_neox_b200.ops.optim import adamw_step_, clip_coef_, sumsq_
    torch.manual_seed(8)
    n = 100003
    p = torch.randn(n, device=DEV)
    pr = p.clone().requires_grad_(True)
    m, v = torch.zeros(n, device=DEV), torch.zeros(n, device=DEV)
    lp = torch.empty(n, device=DEV, dtype=DT)
    opt = torch.optim.AdamW([pr], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    for step in range(1, 4):
        g = torch.randn(n, device=DEV).to(DT)
        acc = torch.zeros(2, device=DEV)
        sumsq_(g, acc)
        assert rel(acc[0], g.float().pow(2).sum()) < 1e-3
        out, skip = torch.ones(2, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        clip_coef_(acc, 1.0, 0.5, out, skip)
        norm = g.float().norm() * 0.5
        coef = min(1.0, 1.0 / (norm.item() + 1e-6)) * 0.5
        assert abs(out[0].item() - coef) / coef < 1e-3 and skip.item() == 0
        adamw_step_(p, m, v, g, lp, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=step,
                    grad_scale=out, skip=skip)
        pr.grad = g.float() * coef
        opt.step()
        assert rel(p, pr.detach()) < 1e-4
        assert rel(lp, pr.detach()) < 1e-2
    # non-finite gradients set the skip flag and the update is a no-op
    g = torch.full((n,), float("inf"), device=DEV).to(DT)
    acc = torch.zeros(2, device=DEV)
    sumsq_(g, acc)
    clip_coef_(acc, 1.0, 1.0, out, skip)
    assert skip.item() == 1
    before = p.clone()
    adamw_step_(p, m, v, g, lp, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=4,
                grad_scale=out, skip=skip)
    assert torch.equal(before, p)


@pytest.mark.parametrize("wide", [False, True], ids=["16bit", "fp32"])
@pytest.mark.parametrize("n", [1, 3, 1024, 1025, 1_212_421, 30_000_003])
def test_optimizer_step_repeats_bit_for_bit(n, wide):
    """Gradient norm, clip coefficient and AdamW from the same state give the same bits on every run, on two streams at
    once too, and the norm is that of 64 bits: a thread adds up to 100 squares in fp32, a block 256 threads in a tree."""
    from gpt_neox_b200.ops.optim import adamw_step_, clip_coef_, sumsq_
    torch.manual_seed(26)
    g, p0 = torch.randn(n, device=DEV) * 1e-2, torch.randn(n, device=DEV) * 0.02
    g = g if wide else g.to(DT)
    m0, v0 = torch.randn(n, device=DEV) * 1e-4, torch.rand(n, device=DEV) * 1e-8

    def step():
        p, m, v, lp = p0.clone(), m0.clone(), v0.clone(), torch.empty(n, device=DEV, dtype=DT)
        acc, out, skip = torch.full((2,), 0.0, device=DEV), torch.zeros(2, device=DEV), torch.ones(1, dtype=torch.int32, device=DEV)
        sumsq_(g, acc)
        one = acc.clone()
        sumsq_(g, acc)                     # a second buffer adds to the first
        clip_coef_(acc, 1e-3, 1.0, out, skip)
        adamw_step_(p, m, v, g, lp, lr=1e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=100, grad_scale=out,
                    skip=skip)
        return one, acc, out, skip, p, m, v, lp

    want = step()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for _ in range(4 if n > 10_000_000 else 20):
        with torch.cuda.stream(side):
            other = step()
        here = step()
        torch.cuda.current_stream().wait_stream(side)
        for a, b, c in zip(want, here, other):
            assert torch.equal(a, b) and torch.equal(a, c)
        side.wait_stream(torch.cuda.current_stream())
    total = g.double().square().sum()
    assert want[1][1] == 0 and want[3] == 0
    assert abs(want[0][0].double() - total) <= 2 ** -20 * total
    assert abs(want[1][0].double() - 2 * total) <= 2 ** -20 * 2 * total


@pytest.mark.parametrize("bad", [math.nan, math.inf, -math.inf])
@pytest.mark.parametrize("n,at", [(1, 0), (1025, 1024), (5_000_001, 3_333_333)])
def test_gradient_norm_marks_what_is_not_finite(n, at, bad):
    from gpt_neox_b200.ops.optim import sumsq_
    g, acc = torch.ones(n, device=DEV, dtype=DT), torch.zeros(2, device=DEV)
    sumsq_(g, acc)
    assert acc.tolist() == [n, 0.0]        # (below 2^24 ones add up exactly)
    g[at] = bad
    sumsq_(g, acc)
    assert acc[1] == 1 and not acc[0].isfinite()


def test_adamw_8bit_state_kernel_matches_the_pytorch_statement():
    """csrc/optim.cu adam8_kernel against ops/optim.py's PyTorch statement of the same update and the same 8-bit
    block-wise codes: the master weights agree to fp32 rounding, the codes agree except where a value sits on a
    rounding boundary of the logarithmic code (one step apart)."""
    from gpt_neox_b200.ops.optim import adamw8bit_step_, q8_blocks
    torch.manual_seed(9)
    n = 2048 * 5 + 1024
    p = torch.randn(n, device=DEV)
    pc = p.cpu().clone()
    st = [torch.zeros(n, dtype=torch.uint8), torch.zeros(n, dtype=torch.uint8), torch.zeros(q8_blocks(n)),
          torch.zeros(q8_blocks(n))]
    sg = [t.to(DEV) for t in st]
    lp = torch.empty(n, device=DEV, dtype=DT)
    scale = torch.tensor([0.5], device=DEV)
    skip = torch.zeros(1, dtype=torch.int32, device=DEV)
    kw = dict(lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1)
    for step in range(1, 5):
        g = (torch.randn(n, device=DEV) * torch.rand(n, device=DEV) ** 3).to(DT)
        adamw8bit_step_(p, *sg, g, lp, step=step, grad_scale=scale, skip=skip, **kw)
        adamw8bit_step_(pc, *st, g.cpu(), None, step=step, grad_scale=torch.tensor([0.5]), **kw)
        assert rel(p.cpu(), pc) < 1e-5
        assert rel(lp.cpu(), pc) < 1e-2
        for a, b in ((sg[0], st[0]), (sg[1], st[1])):
            d = (a.cpu().to(torch.int32) & 127) - (b.to(torch.int32) & 127) if a is sg[0] else \
                a.cpu().to(torch.int32) - b.to(torch.int32)
            assert d.abs().max().item() <= 1 and (d != 0).float().mean().item() < 0.02
            b.copy_(a.cpu())                     # continue from identical codes so that the steps stay comparable
        assert rel(sg[2].cpu(), st[2]) < 1e-5 and rel(sg[3].cpu(), st[3]) < 1e-5
    skip.fill_(1)
    before = p.clone()
    adamw8bit_step_(p, *sg, g, lp, step=5, grad_scale=scale, skip=skip, **kw)
    assert torch.equal(before, p)


@pytest.mark.parametrize("hn,rot", [(128, 32), (96, 24), (64, 64)])
def test_rope_strided(hn, rot):
    from gpt_neox_b200.ops.rope import apply_rotary, rotary_tables
    torch.manual_seed(9)
    s, b, h = 50, 3, 4
    qkv = bf(s, b, h, 3 * hn)
    q = qkv[..., :hn].detach().requires_grad_(True)     # strided view
    cos, sin = rotary_tables(rot, 64, device=DEV)
    y = apply_rotary(q, cos, sin, rot, 5)
    g = bf(s, b, h, hn)
    y.backward(g)
    qr = qkv[..., :hn].detach().float().cpu().requires_grad_(True)
    yr = apply_rotary(qr, cos.cpu(), sin.cpu(), rot, 5)
    yr.backward(g.float().cpu())
    assert rel(y.cpu(), yr) < 1e-2
    assert rel(q.grad.cpu(), qr.grad) < 1e-2


def test_embedding_fwd_bwd():
    from gpt_neox_b200.ops.embedding import embedding
    torch.manual_seed(10)
    V, H = 500, 256
    table = bf(V, H, grad=True)
    ids = torch.randint(0, 1000, (4, 33), device=DEV)
    out = embedding(ids, table, vocab_start=250)
    loc = ids - 250
    inside = (loc >= 0) & (loc < V)
    tr = table.detach().float().requires_grad_(True)
    ref = F.embedding(loc.clamp(0, V - 1), tr) * inside[..., None]
    assert rel(out, ref) < 1e-3
    g = bf(4, 33, H)
    out.backward(g)
    ref.backward(g.float())
    assert rel(table.grad, tr.grad) < 2e-2


def test_mlp_gelu_fused():
    from gpt_neox_b200.ops.fused import mlp_gelu
    torch.manual_seed(11)
    x = bf(3, 70, 256, grad=True)
    w1, b1 = bf(1024, 256, scale=0.05, grad=True), bf(1024, scale=0.1, grad=True)
    w2, b2 = bf(256, 1024, scale=0.05, grad=True), bf(256, scale=0.1, grad=True)
    res = bf(3, 70, 256, grad=True)
    for kind in ("erf", "tanh"):
        for t in (x, w1, b1, w2, b2, res):
            t.grad = None
        y = mlp_gelu(x, w1, b1, w2, b2, residual=res, kind=kind)
        g = bf(3, 70, 256)
        y.backward(g)
        r = [t.detach().float().requires_grad_(True) for t in (x, w1, b1, w2, b2, res)]
        yr = F.linear(F.gelu(F.linear(r[0], r[1], r[2]), approximate="tanh" if kind == "tanh" else "none"),
                      r[3], r[4]) + r[5]
        yr.backward(g.float())
        assert rel(y, yr) < 2e-2
        for t, tr in zip((x, w1, b1, w2, b2, res), r):
            assert rel(t.grad, tr.grad) < 3e-2, kind


@pytest.mark.parametrize("np_,kvp,hn,rot", [(4, 4, 128, 32), (8, 2, 64, 64), (4, 4, 96, 24)])
def test_qkv_attention_fused(np_, kvp, hn, rot):
    from gpt_neox_b200.ops.fused import qkv_attention
    from gpt_neox_b200.ops.rope import rotary_tables
    torch.manual_seed(12)
    s, b = 300, 2
    width = (np_ + 2 * kvp) * hn
    qkv = bf(s, b, width, grad=True)
    cos, sin = rotary_tables(rot, 512, device=DEV)
    out = qkv_attention(qkv.clone(), num_heads=np_, num_kv_heads=kvp, head_dim=hn, rotary_dim=rot, cos=cos, sin=sin)
    qr = qkv.detach().float().cpu().requires_grad_(True)
    ref = qkv_attention(qr, num_heads=np_, num_kv_heads=kvp, head_dim=hn, rotary_dim=rot, cos=cos.cpu(),
                        sin=sin.cpu())
    assert rel(out.cpu(), ref) < 2e-2
    g = bf(s, b, np_ * hn)
    x = qkv.clone()
    o2 = qkv_attention(x, num_heads=np_, num_kv_heads=kvp, head_dim=hn, rotary_dim=rot, cos=cos, sin=sin)
    (gq,) = torch.autograd.grad(o2, x, g)
    ref.backward(g.float().cpu())
    assert rel(gq.cpu(), qr.grad) < 3e-2


@pytest.mark.parametrize("cfg", [
    dict(b=2, sq=512, sk=512, h=4, hk=4, d=128), dict(b=1, sq=300, sk=300, h=4, hk=2, d=96),
    dict(b=1, sq=384, sk=384, h=2, hk=2, d=64), dict(b=1, sq=512, sk=512, h=2, hk=2, d=128, causal=False),
    dict(b=1, sq=512, sk=512, h=2, hk=2, d=128, window=100), dict(b=1, sq=512, sk=512, h=4, hk=4, d=128, alibi=True),
    dict(b=2, sq=64, sk=320, h=2, hk=1, d=64),
    # cached decoding: one new token (and a short chunk) against a long key sequence
    dict(b=2, sq=1, sk=700, h=4, hk=2, d=128), dict(b=1, sq=5, sk=261, h=2, hk=2, d=64, alibi=True),
    # dropout on the probabilities: the fp32 oracle applies the kernels' own mask
    dict(b=2, sq=512, sk=512, h=4, hk=4, d=128, dropout=0.1), dict(b=1, sq=300, sk=300, h=4, hk=2, d=64, dropout=0.25),
    dict(b=1, sq=384, sk=384, h=2, hk=2, d=128, dropout=0.5, alibi=True, window=200)])
def test_flash_attention(cfg):
    from gpt_neox_b200.ops.attention import alibi_slopes, attention_reference, flash_attention
    torch.manual_seed(13)
    b, sq, sk, h, hk, d = (cfg[k] for k in ("b", "sq", "sk", "h", "hk", "d"))
    causal, window = cfg.get("causal", True), cfg.get("window", -1)
    al = alibi_slopes(h).to(DEV) if cfg.get("alibi") else None
    q, k, v = bf(b, sq, h, d, grad=True), bf(b, sk, hk, d, grad=True), bf(b, sk, hk, d, grad=True)
    drop, seed = cfg.get("dropout", 0.0), 0x1234ABCD5678EF01
    o = flash_attention(q, k, v, causal=causal, window=window, alibi=al, dropout_p=drop, seed=seed)
    g = bf(b, sq, h, d)
    o.backward(g)
    qr, kr, vr = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    oref, _ = attention_reference(qr, kr, vr, causal=causal, window=window, alibi=al, dropout_p=drop, seed=seed)
    oref.backward(g.float())
    assert rel(o, oref) < 2e-2
    assert rel(q.grad, qr.grad) < 3e-2 and rel(k.grad, kr.grad) < 3e-2 and rel(v.grad, vr.grad) < 3e-2


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("b,sq,sk,h,hk,causal,window", [
    (1, 1, 1, 1, 1, True, -1), (2, 63, 65, 2, 1, True, -1), (1, 129, 127, 2, 2, True, -1), (1, 128, 64, 1, 1, False, -1),
    (1, 700, 190, 2, 1, True, -1),            # query rows and whole tiles that see no key
    (1, 190, 700, 2, 2, True, 60),            # keys that no query row sees
    (3, 257, 257, 40, 40, True, -1),          # several items per CTA, single-block ones among them
    (2, 640, 640, 32, 4, True, 200)])         # grouped keys: a CTA's items run over several query heads
def test_flash_attention_backward_tiles(b, sq, sk, h, hk, causal, window, d):
    """The persistent backward kernels at the edges of their tiles, items and blocks, against the fp32 oracle.  A gradient is a
    sum of products of values rounded to 16 bits (P or dS, relative 2^-9 or 2^-12 each, and O inside delta), rounded itself:
    three roundings of unit eps."""
    from gpt_neox_b200.ops.attention import attention_reference, flash_attention
    torch.manual_seed(29)
    q, k, v = bf(b, sq, h, d, grad=True), bf(b, sk, hk, d, grad=True), bf(b, sk, hk, d, grad=True)
    g = bf(b, sq, h, d)
    got = torch.autograd.grad(flash_attention(q, k, v, causal=causal, window=window), (q, k, v), g)
    # (written out: autograd through the oracle's softmax has NaN for rows that see no key)
    qd, kd, vd, gd = (t.detach().double() for t in (q, k, v, g))
    _, lse = attention_reference(qd, kd, vd, causal=causal, window=window)
    heads = lambda t: t.repeat_interleave(h // hk, 2)
    pos = torch.arange(sq, device=DEV)[:, None] + sk - sq - torch.arange(sk, device=DEV)[None]
    seen = ((pos >= 0) if causal else torch.ones_like(pos, dtype=torch.bool)) & ((pos <= window) | (window < 0))
    scores = torch.einsum("bqhd,bkhd->bhqk", qd, heads(kd)) / d ** 0.5
    p = torch.where(seen, (scores - lse[..., None]).exp(), 0.0)
    dp = torch.einsum("bqhd,bkhd->bhqk", gd, heads(vd))
    ds = p * (dp - (p * dp).sum(-1, keepdim=True)) / d ** 0.5
    per_kv = lambda t: t.unflatten(2, (hk, h // hk)).sum(3)
    want = (torch.einsum("bhqk,bkhd->bqhd", ds, heads(kd)), per_kv(torch.einsum("bhqk,bqhd->bkhd", ds, qd)),
            per_kv(torch.einsum("bhqk,bqhd->bkhd", p, gd)))
    eps = 2 ** -8 if DT == torch.bfloat16 else 2 ** -11
    for x, y in zip(got, want):
        assert x.isfinite().all()
        # (one key: the true gradients of q and k are zero and what is left is the rounding of O against dP, of size |dO| |v|)
        assert (x.double() - y).norm() <= 3 * eps * (y.norm() + d ** 0.5 * x.numel() ** 0.5 * (sk == 1))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("form", ["causal", "full", "window", "alibi", "alibi_full", "dropout", "sparse", "scale0"])
@pytest.mark.parametrize("b,s,h,hk", [
    (1, 190, 3, 3),             # fewer tiles than SMs
    (3, 400, 40, 40),           # several items per SM
    (5, 400, 40, 20),           # more than four, two query heads per key head
    (128, 72, 3, 1)])           # several single-block items per SM
def test_flash_attention_backward_routes(b, s, h, hk, form, d):
    """Every form at sizes on both sides of the choice between persistent kernels and one CTA per tile, against the fp32
    oracle's autograd: three roundings of unit eps, as above."""
    from gpt_neox_b200.models.sparse_attention import block_layout
    from gpt_neox_b200.ops.attention import BlockLayout, alibi_slopes, attention_reference, flash_attention
    torch.manual_seed(30)
    kw = {"full": dict(causal=False), "window": dict(window=130), "alibi": dict(alibi=alibi_slopes(h).to(DEV)),
          "alibi_full": dict(alibi=alibi_slopes(h).to(DEV), causal=False), "dropout": dict(dropout_p=0.1, seed=5),
          "scale0": dict(scale=0.0)}.get(form, {})
    if form == "sparse":
        kw = dict(block_layout=BlockLayout(block_layout("bigbird", (s + 31) // 32, {
            "num_sliding_window_blocks": 3, "num_global_blocks": 1, "num_random_blocks": 1, "block": 32}, seed=3), 32))
    ts = [bf(b, s, n, d, grad=True) for n in (h, hk, hk)]
    g = bf(b, s, h, d)
    got = torch.autograd.grad(flash_attention(*ts, **kw), ts, g)
    ref = [t.detach().float().requires_grad_() for t in ts]
    want = torch.autograd.grad(attention_reference(*ref, **kw)[0], ref, g.float())
    eps = 2 ** -8 if DT == torch.bfloat16 else 2 ** -11
    for x, y in zip(got, want):
        assert (x.float() - y).norm() <= 3 * eps * y.norm() + 1e-6


@pytest.mark.parametrize("d", [8, 56, 64, 72, 128])
@pytest.mark.parametrize("b,s,h", [(1, 1, 1), (2, 63, 3), (3, 129, 5), (1, 700, 40)])
def test_flash_attention_backward_output_gradient_layouts(b, s, h, d):
    """The layouts of the output's gradient (heads together, each head's rows together, rows on 16-byte boundaries only, one
    broadcast row) take different forms of the kernel that sums O * dO over a row; all add in the same order."""
    from gpt_neox_b200.ops.attention import flash_attention
    torch.manual_seed(31)
    ts = [bf(b, s, h, d, grad=True) for _ in range(3)]
    grads = lambda g: torch.autograd.grad(flash_attention(*ts), ts, g)
    g = bf(b, s, h, d)
    by_head = g.transpose(1, 2).contiguous().transpose(1, 2)
    room = torch.full((b, s, h, d + 8 if d % 16 == 0 else d), float("nan"), device=DEV, dtype=DT)
    room[..., :d] = g
    row = g[:1, :1, :1].expand(b, s, h, d)
    for one, other in ((g, by_head), (g, room[..., :d]), (row.contiguous(), row)):
        for x, y in zip(grads(one), grads(other)):
            assert torch.equal(x, y)


@pytest.mark.parametrize("env", [{"NEOX_ATTN_FWD_SHAPE": "1"}, {"NEOX_ATTN_FWD_SHAPE": "3"}], ids=["fwd_shape1", "fwd_shape3"])
def test_flash_attention_selectable_kernel_shapes(env):
    """The kernel shapes that an environment variable selects instead of the defaults (read once per process, hence a
    child process): the dense, dropout and block-sparse cases of this file under each of them."""
    import os
    import subprocess
    import sys
    if "_dtype" in globals() and DT != torch.bfloat16:
        pytest.skip("one operand type is enough for the shape selection")
    cmd = [sys.executable, "-m", "pytest", "-q", "-x", "-m", "gpu", os.path.abspath(__file__), "-k",
           "(test_flash_attention or test_block_sparse_flash_attention) and not selectable and not varlen and not backward"]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=900, env=dict(os.environ, **env))
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
    assert " passed" in r.stdout


@pytest.mark.parametrize("kind,cfg,block,sq,sk", [
    ("sparse_fixed", {"num_local_blocks": 4, "num_global_blocks": 1}, 16, 640, 640),
    ("bigbird", {"num_sliding_window_blocks": 3, "num_global_blocks": 1, "num_random_blocks": 1}, 32, 512, 512),
    ("bslongformer", {"num_sliding_window_blocks": 3, "global_block_indices": [0]}, 64, 1024, 1024),
    ("local", {"num_local_blocks": 2}, 128, 1024, 1024),
    ("sparse_variable", {"local_window_blocks": [2, 4], "global_block_indices": [0]}, 16, 3, 500)])
def test_block_sparse_flash_attention(kind, cfg, block, sq, sk):
    """The five block-sparse layouts inside the flash kernels (key tiles without a live block are skipped, the rest
    masked per sub-block), forward and backward, against the fp32 oracle with the same token mask; the last case is
    cached decoding (3 new tokens against 500 keys)."""
    from gpt_neox_b200.models.sparse_attention import block_layout
    from gpt_neox_b200.ops.attention import BlockLayout, attention_reference, flash_attention
    torch.manual_seed(17)
    nb = (max(sq, sk) + block - 1) // block
    lay = BlockLayout(block_layout(kind, nb, dict(cfg, block=block), seed=3), block)
    rows, anyt = lay.tables(sq, sk, DEV)
    if sq >= 512:
        assert int((anyt == 0).sum()) > 0                     # some tiles really are skipped
    b, h, hk, d = 2, 4, 2, 64
    q, k, v = bf(b, sq, h, d, grad=True), bf(b, sk, hk, d, grad=True), bf(b, sk, hk, d, grad=True)
    o = flash_attention(q, k, v, causal=True, block_layout=lay)
    g = bf(b, sq, h, d)
    o.backward(g)
    qr, kr, vr = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    oref, _ = attention_reference(qr, kr, vr, causal=True, block_layout=lay)
    oref.backward(g.float())
    assert rel(o, oref) < 2e-2
    assert rel(q.grad, qr.grad) < 3e-2 and rel(k.grad, kr.grad) < 3e-2 and rel(v.grad, vr.grad) < 3e-2


def test_flash_attention_varlen_matches_per_sequence_oracle():
    """Packed sequences of unequal length (and unequal query / key lengths: cached decoding): each attends to itself only."""
    from gpt_neox_b200.ops.attention import attention_reference, flash_attention_varlen
    torch.manual_seed(31)
    lq, lk, h, hk, d = [130, 1, 257, 64], [130, 300, 257, 200], 4, 2, 64
    cq = [0] + torch.tensor(lq).cumsum(0).tolist()
    ck = [0] + torch.tensor(lk).cumsum(0).tolist()
    q, k, v = bf(cq[-1], h, d, grad=True), bf(ck[-1], hk, d, grad=True), bf(ck[-1], hk, d, grad=True)
    o = flash_attention_varlen(q, k, v, cq, torch.tensor(ck))
    g = bf(cq[-1], h, d)
    o.backward(g)
    qr, kr, vr = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    refs = [attention_reference(qr[cq[i]:cq[i + 1]][None], kr[ck[i]:ck[i + 1]][None], vr[ck[i]:ck[i + 1]][None])[0][0]
            for i in range(4)]
    oref = torch.cat(refs, 0)
    oref.backward(g.float())
    assert rel(o, oref) < 2e-2
    assert rel(q.grad, qr.grad) < 3e-2 and rel(k.grad, kr.grad) < 3e-2 and rel(v.grad, vr.grad) < 3e-2


def test_attention_dropout_mask_statistics_and_seed_dependence():
    """The mask is a pure function of (seed, batch, head, q, k): the keep rate matches 1 - p (p in steps of 1/256),
    rows and columns are not correlated, and another seed gives another mask."""
    from gpt_neox_b200.ops.attention import dropout_keep_mask, dropout_threshold
    for p in (0.1, 0.5):
        m = dropout_keep_mask(2, 3, 256, 384, p, 77, DEV).float()
        want = 1.0 - dropout_threshold(p) / 256.0
        assert abs(m.mean().item() - want) < 4e-3
        assert (m.mean(dim=-1) - want).abs().max().item() < 0.15 and (m.mean(dim=-2) - want).abs().max().item() < 0.17
        assert (m[0, 0] != m[0, 1]).float().mean().item() > 0.1            # heads differ
        m2 = dropout_keep_mask(2, 3, 256, 384, p, 78, DEV).float()
        assert (m != m2).float().mean().item() > 0.1                       # seeds differ


def test_qkv_attention_dropout_matches_the_oracle_with_the_same_mask():
    from gpt_neox_b200.ops.fused import qkv_attention
    from gpt_neox_b200.ops.rope import rotary_tables
    torch.manual_seed(21)
    s, b, np_, hn, rot = 256, 2, 4, 64, 16
    qkv = bf(s, b, 3 * np_ * hn, grad=True)
    cos, sin = rotary_tables(rot, 512, device=DEV)
    kw = dict(num_heads=np_, num_kv_heads=np_, head_dim=hn, rotary_dim=rot, dropout_p=0.2, seed=99)
    x = qkv.clone()
    out = qkv_attention(x, cos=cos, sin=sin, **kw)
    qr = qkv.detach().float().cpu().requires_grad_(True)
    ref = qkv_attention(qr, cos=cos.cpu(), sin=sin.cpu(), **kw)
    assert rel(out.cpu(), ref) < 2e-2
    g = bf(s, b, np_ * hn)
    (gq,) = torch.autograd.grad(out, x, g)
    ref.backward(g.float().cpu())
    assert rel(gq.cpu(), qr.grad) < 3e-2


def test_device_error_word_roundtrip():
    """The host can pre-set and read back the device error word (the fault-injection hook used by
    the failure-detection tests; no GPU wait is ever made to run out for it)."""
    from gpt_neox_b200.ops import _lib
    assert _lib.read_device_error(clear=True) == 0
    _lib.check(_lib.lib().nx_poison_device_error(0x301))
    with pytest.raises(_lib.DeviceWaitTimeout):
        _lib.raise_on_device_error()
    assert _lib.read_device_error(clear=False) == 0


def test_bias_and_norm_gradients_accumulate_straight_into_main_grad():
    """With an fp32 ``main_grad`` on the parameters (what the engine installs) the norm and bias-gradient kernels add
    into it themselves: nothing reaches ``.grad``, and two backward passes leave twice the fp32 reference there."""
    from gpt_neox_b200.ops.gemm import linear
    from gpt_neox_b200.ops.norm import dual_layer_norm
    torch.manual_seed(21)
    rows, H, N = 640, 1024, 768
    x = bf(rows, H, grad=True)
    params = {"g1": (1 + 0.1 * torch.randn(H, device=DEV)).to(DT), "b1": bf(H, scale=0.1), "g2": (1 + 0.1 * torch.randn(H, device=DEV)).to(DT),
              "b2": bf(H, scale=0.1), "w": bf(N, H, scale=0.05), "b": bf(N, scale=0.1)}
    for p in params.values():
        p.requires_grad_(True)
        p.main_grad = torch.zeros(p.shape, device=DEV, dtype=torch.float32)
    g = bf(rows, N)
    g2 = bf(rows, H)
    for _ in range(2):
        y1, y2 = dual_layer_norm(x, params["g1"], params["b1"], params["g2"], params["b2"], 1e-5)
        out = linear(y1, params["w"], params["b"])
        torch.autograd.backward([out, y2], [g, g2])
    ref = {k: v.detach().float().requires_grad_(True) for k, v in params.items()}
    xr = x.detach().float().requires_grad_(True)
    r1 = F.layer_norm(xr, (H,), ref["g1"], ref["b1"], 1e-5)
    r2 = F.layer_norm(xr, (H,), ref["g2"], ref["b2"], 1e-5)
    ro = F.linear(r1.to(DT).float(), ref["w"], ref["b"])
    torch.autograd.backward([ro, r2], [g.float(), g2.float()])
    for k, p in params.items():
        assert p.grad is None, k
        assert rel(p.main_grad, 2 * ref[k].grad) < 2e-2, k


@pytest.mark.parametrize("hn,rot,np_,kvp", [(64, 16, 12, 12), (128, 32, 4, 4), (128, 128, 8, 2), (64, 64, 3, 1)])
def test_rotate_qk_matches_the_per_tensor_kernel_and_writes_the_cache(hn, rot, np_, kvp):
    from gpt_neox_b200.ops.fused import _qkv_views
    from gpt_neox_b200.ops.rope import _launch_qk, _qk_ok, apply_rotary, rotary_tables, rotate_qk_
    torch.manual_seed(3)
    s, b, pos0 = 5, 3, 7
    cos, sin = rotary_tables(rot, 64, device=DEV)
    qkv = bf(s, b, (np_ + 2 * kvp) * hn)
    q, k, v = _qkv_views(qkv, np_, kvp, hn)
    want_q, want_k, want_v = apply_rotary(q, cos, sin, rot, pos0), apply_rotary(k, cos, sin, rot, pos0), v.clone()
    keep = qkv.clone()
    cache = torch.zeros(2, 9, b, kvp, hn, device=DEV, dtype=DT)
    assert _qk_ok(rot, hn, q, k, v, cache[0], cache[1])
    _launch_qk(q, k, cos, sin, rot, pos0, False, v=v, k_out=cache[0, 4:], v_out=cache[1, 4:])
    assert torch.equal(q, want_q) and torch.equal(cache[0, 4:], want_k) and torch.equal(cache[1, 4:], want_v)
    assert torch.equal(k, _qkv_views(keep, np_, kvp, hn)[1]) and not cache[:, :4].any()      # k itself is left alone
    q2, k2, v2 = _qkv_views(keep, np_, kvp, hn)
    rotate_qk_(q2, k2, cos, sin, rot, pos0, False)
    assert torch.equal(q2, want_q) and torch.equal(k2, want_k) and torch.equal(v2, want_v)


@pytest.mark.parametrize("hn,rot,np_,kvp", [(64, 16, 12, 12), (128, 128, 8, 2), (64, 48, 3, 1)])
def test_rotate_qk_out_of_place_leaves_the_projection_alone(hn, rot, np_, kvp):
    from gpt_neox_b200.ops.fused import _qkv_views
    from gpt_neox_b200.ops.rope import _launch_qk, apply_rotary, rotary_tables
    torch.manual_seed(4)
    cos, sin = rotary_tables(rot, 64, device=DEV)
    qkv = bf(5, 3, (np_ + 2 * kvp) * hn)
    keep = qkv.clone()
    q, k, v = _qkv_views(qkv, np_, kvp, hn)
    out, cache = torch.empty(q.shape, device=DEV, dtype=DT), torch.empty(2, 5, 3, kvp, hn, device=DEV, dtype=DT)
    _launch_qk(q, k, cos, sin, rot, 7, False, v=v, q_out=out, k_out=cache[0], v_out=cache[1])
    assert torch.equal(qkv, keep) and torch.equal(out, apply_rotary(q, cos, sin, rot, 7))
    assert torch.equal(cache[0], apply_rotary(k, cos, sin, rot, 7)) and torch.equal(cache[1], v)


@pytest.mark.parametrize("rows,H", [(1, 8), (9, 248), (17, 264), (1001, 1032), (8, 2048), (601, 2048), (3, 2056), (33, 512),
                                    (1001, 520), (300, 768), (5, 776)])
@pytest.mark.parametrize("form", ["dual", "layer", "rms"])
def test_norm_row_sizes(rows, H, form):
    """Row lengths around what a lane, a warp and the warp-per-row form take; every gradient in the parameters' type."""
    from gpt_neox_b200.ops.norm import dual_layer_norm, layer_norm, rms_norm
    torch.manual_seed(4)
    x, ps = bf(rows, H, scale=2.0, grad=True), [bf(H, grad=True) for _ in range({"dual": 4, "layer": 2, "rms": 1}[form])]
    xr, pr = x.detach().double().requires_grad_(True), [p.detach().double().requires_grad_(True) for p in ps]
    if form == "dual":
        ys, yr = dual_layer_norm(x, *ps), [F.layer_norm(xr, (H,), *pr[i:i + 2], 1e-5) for i in (0, 2)]
    elif form == "layer":
        ys, yr = [layer_norm(x, *ps)], [F.layer_norm(xr, (H,), *pr, 1e-5)]
    else:
        ys, yr = [rms_norm(x, *ps, eps=1e-5)], [pr[0] * xr * torch.rsqrt(xr.square().mean(-1, keepdim=True) + 1e-5)]
    gs = [bf(rows, H) for _ in ys]
    got = torch.autograd.grad(ys, [x] + ps, gs)
    want = torch.autograd.grad(yr, [xr] + pr, [g.double() for g in gs])
    tol = 2 ** -7 if DT == torch.bfloat16 else 2 ** -10          # one rounding to the output type
    for a, r in zip(list(ys) + list(got), yr + list(want)):
        assert a.dtype == DT and rel(a, r) < tol
    with torch.no_grad():                                        # without autograd: the same kernel, the same bits
        again = {"dual": lambda: dual_layer_norm(x, *ps), "layer": lambda: [layer_norm(x, *ps)],
                 "rms": lambda: [rms_norm(x, *ps, eps=1e-5)]}[form]()
    assert all(torch.equal(a, y) for a, y in zip(again, ys))


def test_norm_parameter_shared_by_both_norms_and_frozen_parameters():
    from gpt_neox_b200.ops.norm import dual_layer_norm
    torch.manual_seed(5)
    x, w, b = bf(40, 256, grad=True), bf(256, grad=True), bf(256)
    y1, y2 = dual_layer_norm(x, w, b, w, b)
    g1, g2 = bf(40, 256), bf(256 * 40).view(40, 256)
    dx, dw = torch.autograd.grad([y1, y2], [x, w], [g1, g2])
    xr, wr = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    yr = F.layer_norm(xr, (256,), wr, b.double(), 1e-5)
    rx, rw = torch.autograd.grad([yr, yr], [xr, wr], [g1.double(), g2.double()])
    assert rel(dx, rx) < 2e-2 and rel(dw, rw) < 2e-2


def test_norm_parameter_shared_by_both_norms_adds_to_its_main_grad_twice():
    """Both norms' sums have to arrive in one fp32 buffer, for the weight and for the bias."""
    from gpt_neox_b200.ops.norm import dual_layer_norm
    torch.manual_seed(6)
    H = 2048
    x, w, b = bf(300, H, grad=True), bf(H, grad=True), bf(H, grad=True)
    for p in (w, b):
        p.main_grad = torch.zeros(H, device=DEV)
    g1, g2 = bf(300, H), bf(300, H)
    xr, wr, br = (t.detach().double().requires_grad_(True) for t in (x, w, b))
    yr = F.layer_norm(xr, (H,), wr, br, 1e-5)
    want = torch.autograd.grad([yr, yr], [wr, br], [g1.double(), g2.double()])
    for n in range(1, 4):
        torch.autograd.backward(dual_layer_norm(x, w, b, w, b), [g1, g2])
        assert w.grad is None and b.grad is None
        for p, r in zip((w, b), want):
            assert ((p.main_grad - n * r).abs().max() / (n * r).abs().max()).item() < 1e-4


@pytest.mark.parametrize("b,h,hk,sk,d,window,alibi", [
    (1, 1, 1, 1, 128, -1, False), (2, 4, 4, 127, 64, -1, False), (3, 12, 3, 129, 64, -1, True),
    (1, 32, 4, 2049, 128, -1, False), (2, 6, 2, 1000, 40, 700, False), (8, 32, 32, 777, 128, -1, False),
    (1, 16, 1, 4097, 72, 1023, True), (20, 32, 32, 300, 128, -1, False), (1, 3, 1, 511, 96, 0, False)])
def test_one_query_attention(b, h, hk, sk, d, window, alibi):
    """One query row per head against a cache in [seq, batch, head, dim] memory: every cluster size, group size and
    remainder of the split-key kernel.  Only the output is rounded to 16 bits (2^-9 / 2^-12 of its size)."""
    from gpt_neox_b200.ops.attention import _fwd, alibi_slopes, attention_reference
    torch.manual_seed(21)
    al = alibi_slopes(h).to(DEV) if alibi else None
    q = bf(1, b, h, d).permute(1, 0, 2, 3)
    cache = bf(2, sk + 3, b, hk, d)                              # a longer buffer: the keys are a view of its front
    k, v = (t[:sk].permute(1, 0, 2, 3) for t in cache)
    o, lse = _fwd(q, k, v, 1.0 / math.sqrt(d), True, window, al)
    ref, rl = attention_reference(q.double(), k.double(), v.double(), window=window, alibi=al)
    assert o.dtype == DT and rel(o, ref) < (2 ** -7 if DT == torch.bfloat16 else 2 ** -10)
    torch.testing.assert_close(lse[:, :, 0], (rl[:, :, 0] / math.log(2.0)).float(), rtol=1e-4, atol=1e-4)
    assert torch.isinf(lse[:, :, 1:]).all() and (lse[:, :, 1:] > 0).all()


@pytest.mark.parametrize("sk,h,hk", [(5, 4, 4), (300, 4, 4), (3000, 4, 4), (300, 16, 2), (3000, 32, 4)])
def test_one_query_attention_passes_nan_and_inf_on(sk, h, hk):
    """Non-finite scores and values in the split-key kernel, in the first, a middle and the last split: the outputs that are
    NaN or infinite are those of the same query in a call of two rows (the tile kernel), in the other heads nothing is."""
    from gpt_neox_b200.ops.attention import _fwd
    torch.manual_seed(22)
    base = [bf(1, n, m, 128) for n, m in ((1, h), (sk, hk), (sk, hk))]
    run = lambda q, k, v: _fwd(q, k, v, 128 ** -0.5, False, -1, None)[0][0, -1]
    for which, value in ((0, math.nan), (0, math.inf), (1, math.nan), (1, math.inf), (1, -math.inf), (2, math.nan),
                         (2, -math.inf)):
        for at in (0, sk // 2, sk - 1):
            q, k, v = ts = [t.clone() for t in base]
            ts[which][0, min(at, ts[which].shape[1] - 1), 1, 7] = value
            one, two = run(q, k, v), run(torch.cat([q, q], 1), k, v)
            assert torch.equal(one.isnan(), two.isnan()) and torch.equal(one.isinf(), two.isinf()), (which, value, at)
            hit = slice(1, 2) if which == 0 else slice(h // hk, 2 * (h // hk))
            assert not math.isnan(value) or one[hit].isnan().any(-1).all()
            one[hit] = 0
            assert one.isfinite().all()


@pytest.mark.parametrize("rows,H", [(1, 8), (3, 2056), (600, 768)])
@pytest.mark.parametrize("ba,bm", [(True, True), (False, True), (False, False)])
def test_branch_sum_rounds_once(rows, H, ba, bm):
    from gpt_neox_b200.ops.elementwise import branch_sum
    torch.manual_seed(23)
    x, a, m = bf(rows, H, scale=100.0), bf(rows, H), bf(rows, H)
    b1, b2 = bf(H) if ba else None, bf(H) if bm else None
    got = branch_sum(x, a, b1, m, b2)
    p, q = (t.float() if b is None else t.float() + b.float() for t, b in ((a, b1), (m, b2)))
    assert torch.equal(got, (x.float() + p + q).to(DT))


@pytest.mark.parametrize("s,at,d,window", [(256, 40, 128, -1), (200, 130, 64, -1), (300, 290, 128, 100), (130, 0, 64, -1)])
def test_a_nan_row_leaves_the_values_it_does_not_see_alone(s, at, d, window):
    """A query row of NaN: the gradients of the values it attends to are NaN, those of the keys that the causal mask, the
    window or the end of the sequence hides from it are what they are without that row (its probabilities there are 0)."""
    from gpt_neox_b200.ops.attention import flash_attention
    torch.manual_seed(24)
    q, k, v, g = bf(1, s, 2, d), bf(1, s, 2, d, grad=True), bf(1, s, 2, d, grad=True), bf(1, s, 2, d)
    q[0, at, 1] = math.nan
    (dv,) = torch.autograd.grad(flash_attention(q, k, v, window=window), [v], g)
    pos = torch.arange(s, device=DEV)
    seen = (pos <= at) & (pos >= (at - window if window >= 0 else 0))
    assert dv[0, seen, 1].isnan().all() and dv[0, ~seen, 1].isfinite().all() and dv[0, :, 0].isfinite().all()


@pytest.mark.parametrize("sq,sk,scale", [(200, 70, None), (129, 1, None), (140, 140, 0.0), (130, 200, -0.02)])
def test_attention_gradients_of_rows_without_keys_and_odd_scales(sq, sk, scale):
    """More queries than keys (the first rows see none), scale 0 and a negative one."""
    from gpt_neox_b200.ops.attention import attention_reference, flash_attention
    torch.manual_seed(25)
    ts = [bf(2, n, 3, 64, grad=True) for n in (sq, sk, sk)]
    ref = [t.detach().double().requires_grad_(True) for t in ts]
    g = bf(2, sq, 3, 64)
    live = slice(max(0, sq - sk), sq)
    y, r = flash_attention(*ts, scale=scale), attention_reference(ref[0][:, live], *ref[1:], scale=scale)[0]
    assert not y[:, :live.start].any() and rel(y[:, live], r) < 2e-2
    for a, b in zip(torch.autograd.grad(y, ts, g), torch.autograd.grad(r, ref, g[:, live].to(r.dtype))):
        assert (a.float() - b.float()).abs().max() <= 2e-2 * b.float().abs().max() + 1e-6


@pytest.mark.parametrize("b,h,hk,sk,d", [(14, 32, 32, 781, 128), (18, 32, 32, 4100, 128), (33, 32, 32, 523, 128),
                                         (1, 16, 2, 65, 128), (3, 16, 2, 129, 64), (40, 16, 2, 40, 64), (5, 24, 3, 700, 128)])
def test_one_query_attention_splits_and_head_groups(b, h, hk, sk, d):
    """Thirds, quarters and halves of the keys where one round of CTAs would leave places empty, and one, two, four and
    eight heads per CTA: against the tile kernel, which computes the same row as the last of two."""
    from gpt_neox_b200.ops.attention import _fwd
    torch.manual_seed(26)
    q, k, v = bf(b, 1, h, d), bf(b, sk, hk, d), bf(b, sk, hk, d)
    one, lse = _fwd(q, k, v, d ** -0.5, False, -1, None)
    two, lse2 = _fwd(torch.cat([q, q], 1), k, v, d ** -0.5, False, -1, None)
    # the tile kernel rounds its probabilities to 16 bits: each output within one unit of their weighted sum
    assert rel(one[:, 0], two[:, 1]) < (2 ** -6 if DT == torch.bfloat16 else 2 ** -9)
    torch.testing.assert_close(lse[:, :, 0], lse2[:, :, 1], rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("H", [64, 520, 768, 2048])
@pytest.mark.parametrize("form", ["dual", "rms"])
def test_a_nan_stays_in_its_row_of_a_norm(H, form):
    from gpt_neox_b200.ops.norm import dual_layer_norm, rms_norm
    torch.manual_seed(27)
    x, w = bf(40, H), bf(H)
    x[7, H - 1], x[19, 0], x[20, 3] = math.nan, math.inf, -math.inf
    ys = dual_layer_norm(x, w, w, w, w) if form == "dual" else [rms_norm(x, w, eps=1e-5)]
    bad = torch.zeros(40, dtype=torch.bool, device=DEV)
    bad[[7, 19, 20]] = True
    for y in ys:
        assert y[~bad].isfinite().all() and y[7].isnan().all()
        # an infinite element: the mean of a LayerNorm is infinite; an RMS norm divides by infinity (0, and inf * 0 = NaN)
        assert y[19].isnan().all() if form == "dual" else (y[19, 0].isnan() and not y[19, 1:].any())


def test_branch_sum_of_other_types_shapes_and_alignments():
    """What the kernel does not take goes to PyTorch: a branch of another type, one that broadcasts, one on an odd address."""
    from gpt_neox_b200.ops.elementwise import branch_sum
    torch.manual_seed(28)
    x, a, m, b = bf(3, 2, 64), bf(3, 2, 64), bf(3, 2, 64), bf(64)
    want = (x.float() + (a.float() + b.float()) + m.float())
    odd = torch.empty(3 * 2 * 64 + 1, device=DEV, dtype=DT)[1:].view(3, 2, 64).copy_(a)
    oddb = torch.empty(65, device=DEV, dtype=DT)[1:].copy_(b)
    assert torch.equal(branch_sum(x, odd, oddb, m.transpose(0, 1).contiguous().transpose(0, 1), None), want.to(DT))
    wide = branch_sum(x, a.float(), b, m, None)
    assert wide.dtype == torch.float32 and rel(wide, want) < 1e-2
    none = torch.zeros((), device=DEV, dtype=DT)
    assert rel(branch_sum(x, a, b, none, None), want - m.float()) < 1e-2
    cpu = branch_sum(*(t.cpu() for t in (x, a, b, m)), None)
    assert rel(cpu.to(DEV), want) < 2e-2


@pytest.mark.parametrize("captured", [False, True], ids=["eager", "graph"])
@pytest.mark.parametrize("rows,h,f", [(1, 512, 256), (4, 1024, 2816), (64, 768, 1024)])
def test_dependent_launches_see_what_the_kernel_before_wrote(rows, h, f, captured):
    """Kernels that may begin while the one before them runs (few-rows GEMM, gated activation, norm): every input, the weights
    too, is written by the kernel right before.  The same chain with a synchronisation after every launch gives the same bits."""
    from gpt_neox_b200.ops.elementwise import gated_act
    from gpt_neox_b200.ops.gemm import gemm
    from gpt_neox_b200.ops.norm import layer_norm
    torch.manual_seed(5)
    x, w1, w2, g, b = bf(rows, h), bf(2 * f, h, scale=0.05), bf(h, f, scale=0.05), bf(h), bf(h)
    step = torch.zeros((), device=DEV, dtype=DT)

    def chain(pause):
        step.add_(0.25)
        outs = []
        y = x * step
        for _ in range(3):
            pause()
            a, c = w1 * step, w2 * step
            pause()
            u = gemm(y, a)
            pause()
            u = gated_act(u, "swiglu")
            pause()
            u = gemm(u, c)
            pause()
            y = layer_norm(u, g, b)
            pause()
            outs += [u, y]
        return outs

    with torch.no_grad():
        want = []
        for _ in range(6):
            want.append([t.clone() for t in chain(torch.cuda.synchronize)])
        step.zero_()
        if captured:
            graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                chain(lambda: None)
            torch.cuda.current_stream().wait_stream(side)
            with torch.cuda.graph(graph):
                outs = chain(lambda: None)
            step.zero_()
        for ref in want:
            if captured:
                graph.replay()
            else:
                outs = chain(lambda: None)
            for got, r in zip(outs, ref):
                assert torch.equal(got, r)


@pytest.mark.parametrize("wide", [False, True], ids=["16bit", "fp32"])
@pytest.mark.parametrize("M,N,off,pad", [(256, 256, 0, 0), (300, 264, 0, 8), (513, 520, 8, 0), (700, 272, 8, 16), (260, 776, 0, 4)])
def test_pair_gemm_rows_on_16_and_32_byte_boundaries(M, N, off, pad, wide):
    """Result, side operands and sums whose rows start on 32-byte boundaries and on 16-byte ones only (a base or a leading
    dimension that is no multiple of 32 bytes), at column counts that cut tiles of 256 and pieces of 32 and 16: the fp32
    product of 64 terms of order 1 (sums 2 ** -18 off at most), rounded once per 16-bit step."""
    from gpt_neox_b200.ops.gemm import gemm
    if pad == 4 and not wide:
        pytest.skip("16-bit rows are multiples of 16 bytes")
    torch.manual_seed(31)
    K, eps = 64, 2.0 ** -8 if DT == torch.bfloat16 else 2.0 ** -11
    mk = lambda *s: torch.randn(*s, device=DEV).to(DT)

    def place(dtype, like=None):           # [M, N] inside rows of N + pad, `off` elements behind a 32-byte boundary
        t = torch.zeros(off + M * (N + pad) + 32, device=DEV, dtype=dtype)[off:off + M * (N + pad)].view(M, N + pad)[:, :N]
        return t if like is None else t.copy_(like)

    a, b = mk(M, K), mk(N, K)
    z = a.double() @ b.double().t()
    if wide:
        out = place(torch.float32, torch.randn(M, N, device=DEV))
        want = out.double() + z
        got = gemm(a, b, out=out, accumulate=True)
        assert (got.double() - want).abs().max() <= 2 ** -18 * 64
        assert (gemm(a, b, out=place(torch.float32)).double() - z).abs().max() <= 2 ** -18 * 64
        return
    near = lambda got, want, steps=1: (got.double() - want).abs().sub(steps * eps * want.abs()).max() <= 2 ** -12
    assert near(gemm(a, b, out=place(DT)), z)
    res = place(DT, mk(M, N))
    assert near(gemm(a, b, out=place(DT), residual=res), z + res.double())
    assert near(gemm(a, b, out=place(DT), dgelu_aux=res, dgelu="mul"), z * res.double())
    out = place(DT, res)
    assert near(gemm(a, b, out=out, accumulate=True), z + res.double())
    deriv, act = place(DT), place(DT)
    gemm(a, b, out=act, gelu="erf", aux_out=deriv, aux_deriv=True)
    x = z.detach().requires_grad_()
    y = torch.nn.functional.gelu(x)
    assert near(act, y) and near(deriv, torch.autograd.grad(y.sum(), x)[0])

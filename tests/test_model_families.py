"""RWKV-6, gMLP / aMLP and mixed stacks build and train through the public training entry on CPU;
kernel numerics of the WKV recurrence on the GPU."""
import math

import pytest
import torch

from common import run_distributed, tiny_config
from test_mamba import _train


@pytest.mark.parametrize("name,over", [
    ("rwkv", dict(attention_config=[[["rwkv"], 2]], pos_emb="none", gpt_j_residual=False, hidden_size=64,
                  num_attention_heads=2)),
    ("gmlp", dict(attention_config=[[["gmlp"], 2]], pos_emb="none", gpt_j_residual=False)),
    ("amlp", dict(attention_config=[[["amlp"], 2]], pos_emb="none", gpt_j_residual=False, gmlp_attn_dim=16)),
    ("mixed", dict(attention_config=[[["global"], 1], [["mamba"], 1]], num_layers=2, gpt_j_residual=False)),
])
def test_family_trains_on_cpu(name, over):
    cfg = tiny_config(**{**dict(use_cpu_initialization=True), **over})
    losses = run_distributed(_train, 1, cfg, 6)[0]
    assert all(l == l and l < 20 for l in losses), losses


def test_wkv_decay_gradient_identity():
    """dL/dw obtained from gr and gk by the reverse cumulative sum equals autograd's."""
    from gpt_neox_b200.ops.wkv import decay_grad_from_gr_gk, wkv6_reference
    torch.manual_seed(0)
    B, T, H, N = 2, 10, 2, 8
    C = H * N
    r, k, v = (torch.randn(B, T, C, requires_grad=True) for _ in range(3))
    w = (torch.randn(B, T, C) - 1).requires_grad_(True)
    u = torch.randn(H, N, requires_grad=True)
    y = wkv6_reference(r, k, v, w, u)
    gy = torch.randn_like(y)
    gr, gk, gv, gw, gu = torch.autograd.grad(y, (r, k, v, w, u), gy)
    gw2, gu2 = decay_grad_from_gr_gk(r.detach(), k.detach(), v.detach(), w.detach(), u.detach(), gy, gr, gk)
    torch.testing.assert_close(gw2, gw, rtol=1e-3, atol=1e-4)
    torch.testing.assert_close(gu2, gu, rtol=1e-3, atol=1e-4)


@pytest.mark.gpu
@pytest.mark.parametrize("T,H,N", [(300, 3, 64), (128, 2, 32), (50, 1, 64)])
def test_wkv6_kernel(T, H, N):
    from gpt_neox_b200.ops.wkv import wkv6, wkv6_reference
    torch.manual_seed(2)
    B, C, dev = 2, H * N, "cuda"
    mk = lambda: (torch.randn(T, B, C, device=dev) * 0.5).bfloat16().transpose(0, 1)
    r, k, v = mk(), mk(), mk()
    w = (torch.randn(T, B, C, device=dev) * 0.5 - 1.5).bfloat16().transpose(0, 1)
    u = (torch.randn(H, N, device=dev) * 0.3).bfloat16()
    leaves = [t.detach().clone().requires_grad_(True) for t in (r, k, v, w, u)]
    ref = [t.detach().float().clone().requires_grad_(True) for t in (r, k, v, w, u)]
    y = wkv6(*leaves)
    yr = wkv6_reference(*ref)
    gy = (torch.randn(B, T, C, device=dev) * 0.5).bfloat16()
    y.backward(gy)
    yr.backward(gy.float())
    scale = yr.abs().max().item()
    assert (y.float() - yr).abs().max().item() <= 0.02 * scale + 1e-2
    for n, a, b in zip("rkvwu", leaves, ref):
        s = b.grad.abs().max().item() + 1e-6
        err = (a.grad.float() - b.grad).abs().max().item()
        assert err <= 0.04 * s + 1e-2, f"grad {n}: err {err} scale {s}"


def test_sparse_layouts_are_causal_and_have_their_patterns():
    from gpt_neox_b200.models.sparse_attention import block_layout, token_mask
    nb = 16
    fixed = block_layout("sparse_fixed", nb, {"num_local_blocks": 4, "num_global_blocks": 1})
    assert fixed[5, 4] and fixed[5, 7] and not fixed[5, 8 + 1]          # dense inside window [4, 8)
    assert fixed[9, 3] and fixed[15, 7] and not fixed[9, 2]               # window summaries (last block) are global
    local = block_layout("local", nb, {"num_sliding_window_blocks": 4})
    assert local[6, 4] and local[6, 6] and not local[6, 3] and not local[6, 7]
    bb = block_layout("bigbird", nb, {})
    assert bb[10, 0] and bb[0, 10] and bb[10, 9] and bb[10, 11]
    m = token_mask("bslongformer", 100, {"block": 16})
    assert m.shape == (1, 1, 100, 100)
    allowed = ~m[0, 0]
    assert not torch.triu(allowed, 1).any()                               # causal
    assert allowed.diagonal().all() and allowed[:, 0].all()               # self and the global first block


@pytest.mark.parametrize("kind", ["local", "sparse_fixed", "sparse_variable", "bigbird", "bslongformer"])
def test_sparse_attention_types_train_on_cpu(kind):
    cfg = tiny_config(use_cpu_initialization=True, attention_config=[[[kind], 2]], sparsity_config={"block": 4})
    losses = run_distributed(_train, 1, cfg, 3)[0]
    assert all(l == l for l in losses)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,H,N,pad", [(1, 1, 1, 64, 0), (2, 17, 3, 32, 0), (1, 333, 2, 64, 0), (40, 48, 12, 64, 0),
                                         (1, 130, 1, 32, 4), (3, 64, 2, 64, 8)])
def test_wkv6_chunks_and_layouts(B, T, H, N, pad, dtype):
    """Sub-block remainders, one chunk (many heads) and many (few heads), views whose rows are not 16-byte aligned."""
    from gpt_neox_b200.ops.wkv import wkv6, wkv6_reference
    torch.manual_seed(7)
    C = H * N
    mk = lambda m=0.0: (torch.randn(T, B, C + pad, device="cuda") * 0.5 + m).to(dtype)[..., pad:].transpose(0, 1)
    leaves = [t.detach().requires_grad_(True) for t in (mk(), mk(), mk(), mk(-1.5))]
    leaves.append((torch.randn(H, N, device="cuda") * 0.3).to(dtype).requires_grad_(True))
    ref = [t.detach().float().clone().requires_grad_(True) for t in leaves]
    gy = (torch.randn(B, T, C, device="cuda") * 0.5).to(dtype)
    y = wkv6(*leaves)
    got = torch.autograd.grad(y, leaves, gy)
    yr = wkv6_reference(*ref)
    want = torch.autograd.grad(yr, ref, gy.float(), allow_unused=True)       # (T = 1: nothing decays)
    want = [torch.zeros_like(t) if r is None else r for t, r in zip(ref, want)]
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
    for a, r in zip((y,) + got, [yr] + want):                   # one rounding to 16 bits; fp32 sums on both sides
        assert (a.float() - r).abs().max().item() <= 2 * eps * r.abs().max().item() + 1e-3


@pytest.mark.parametrize("B,T,H,counts", [(4, 2048, 24, (12, 9)), (8, 2048, 16, (8, 10)), (2, 4096, 32, (16, 13)),
                                          (40, 512, 12, (1, 4)), (4, 300, 24, (10, 4)), (10, 400, 24, (3, 1)), (1, 10, 4, (1, 1))])
def test_wkv6_chunks_go_by_the_head_size(B, T, H, counts):
    """Heads of 32 go step by step, with CTAs of half the size: on 148 SMs the counts that were measured to be the best ones or
    within 7 % of them, not those of heads of 64 in blocks."""
    from gpt_neox_b200.ops import _lib
    lib = _lib.lib(torch.bfloat16)
    if lib.nx_sm_count() != 148:
        pytest.skip("the counts are those of 148 SMs")
    assert (lib.nx_wkv6_head_chunks(B, T, H, 32), lib.nx_wkv6_head_chunks(B, T, H, 64)) == counts
    assert lib.nx_wkv6_chunks(B, T, H) == counts[1]
    assert _lib.lib(torch.float16).nx_wkv6_head_chunks(B, T, H, 32) == counts[0]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,H", [(1, 517, 5), (4, 300, 24), (2, 1000, 3)])
def test_wkv6_heads_of_32_in_many_chunks(B, T, H, dtype):
    """32, 10 and 32 chunks on 148 SMs, the last one ragged."""
    test_wkv6_chunks_and_layouts(B, T, H, 32, 0, dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("B,T,H,N", [(96, 40, 2, 64), (1, 900, 2, 64), (3, 400, 1, 32)])
def test_wkv6_gradients_repeat_bit_for_bit(B, T, H, N):
    """Many sequences, and one cut into many chunks: the gradient of u is a sum over both, in a fixed order."""
    from gpt_neox_b200.ops.wkv import wkv6, wkv6_reference
    torch.manual_seed(9)
    mk = lambda m=0.0: (torch.randn(B, T, H * N, device="cuda") * 0.5 + m).bfloat16().requires_grad_(True)
    leaves = [mk(), mk(), mk(), mk(-1.5), (torch.randn(H, N, device="cuda") * 0.3).requires_grad_(True)]
    g = torch.randn(B, T, H * N, device="cuda").bfloat16()
    runs = [torch.autograd.grad(wkv6(*leaves), leaves, g) for _ in range(8)]
    for r in runs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(runs[0], r))
    ref = [t.detach().double().requires_grad_(True) for t in leaves]
    r, k, v, w, u = ref
    s = (g.double() * v).view(B, T, H, N).sum(-1, keepdim=True)
    want = ((r * k).view(B, T, H, N) * s).sum((0, 1))
    err = (runs[0][4].double() - want).norm() / want.norm()
    assert err < 1e-5, err.item()                  # fp32 sums of B * T products of 16-bit inputs


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,H", [(1, 15, 1), (2, 16, 3), (1, 33, 2), (45, 50, 10), (1, 600, 2), (64, 15, 4), (24, 33, 4),
                                   (3, 129, 1)])
@pytest.mark.parametrize("w", [-12.0, -1.0, 2.0, 6.0])
def test_wkv6_blocks_of_steps(B, T, H, w, dtype):
    """Heads of 64 in blocks of 16 steps: short blocks, one chunk and many, decays from 1 - 6e-6 to an underflowing one, against
    64 bits.  One rounding to 16 bits; inside, the sums are of fp32 precision: as many terms as steps and channels."""
    from gpt_neox_b200.ops.wkv import wkv6
    torch.manual_seed(11)
    N = 64
    mk = lambda m=0.0: (torch.randn(B, T, H * N, device="cuda") * 0.5 + m).to(dtype)
    leaves = [t.requires_grad_(True) for t in (mk(), mk(), mk(), mk(w))]
    leaves.append((torch.randn(H, N, device="cuda") * 0.3).to(dtype).requires_grad_(True))
    gy = mk()
    y = wkv6(*leaves)
    got = (y,) + torch.autograd.grad(y, leaves, gy)
    ref = [t.detach().double().requires_grad_(True) for t in leaves]
    r, k, v, e = (t.view(B, T, H, N) for t in ref[:4])
    S, ys = torch.zeros(B, H, N, N, device="cuda", dtype=torch.float64), []
    for t in range(T):
        kv = k[:, t, :, :, None] * v[:, t, :, None, :]
        ys.append((r[:, t, :, :, None] * (ref[4][None, :, :, None] * kv + S)).sum(-2))
        S = torch.exp(-torch.exp(e[:, t]))[..., None] * S + kv
    yr = torch.stack(ys, 1).view(B, T, H * N)
    want = (yr,) + torch.autograd.grad(yr, ref, gy.double())
    eps = 2 ** -9 if dtype == torch.bfloat16 else 2 ** -12
    for n, (a, b) in enumerate(zip(got, want)):
        # (fp16: results below 2^-14 are subnormal, rounded to 2^-25)
        lim = eps * b.norm() + (2 ** -20 * b.abs().max() + 2 ** -25) * b.numel() ** 0.5
        if n == 4:
            # The decay gradient is ew times a running difference of r gr and k gk, which cancel: what fp32 leaves of it is a
            # last bit of the sizes of all terms behind a step.  (Plain fp32 sums stay below 0.1 of that; at w = 6, where the
            # gradient itself is 0, it is the whole bound.)
            size = _wkv6_sweeps(*(t.detach().abs() for t in leaves[:3]), leaves[3].detach(), leaves[4].detach().abs(), gy.abs())
            terms = leaves[0].detach().abs() * size[1] + leaves[1].detach().abs() * size[2]
            fp32 = 2 ** -24 * (ref[3].detach().exp() * terms.double().flip(1).cumsum(1).flip(1)).norm()
            assert fp32 <= (0.05 * b.norm() if w < 6 else 5e-2 * b.numel() ** 0.5)
            lim = eps * b.norm() + 2 ** -25 * b.numel() ** 0.5 + fp32
        assert (a.double() - b).norm() <= lim, n


@pytest.mark.gpu
@pytest.mark.parametrize("what,value", [(0, float("nan")), (1, float("nan")), (2, float("inf")), (3, float("nan"))])
@pytest.mark.parametrize("at", [0, 40, 331])
def test_wkv6_passes_nan_and_inf_on(what, value, at):
    """A non-finite r, k, v or w in the first, a middle and the last chunk of a sequence: the outputs that are not finite are
    those of the sequential statement."""
    from gpt_neox_b200.ops.wkv import wkv6, wkv6_reference
    torch.manual_seed(10)
    T, H, N = 333, 2, 64
    ts = [(torch.randn(2, T, H * N, device="cuda") * 0.5 - (3.0 if i == 3 else 0.0)).bfloat16() for i in range(4)]
    ts[what][1, at, 70] = value
    u = (torch.randn(H, N, device="cuda") * 0.3).bfloat16()
    got, want = wkv6(*ts, u), wkv6_reference(*(t.float() for t in ts), u.float())
    assert torch.equal(got.isfinite(), want.isfinite())
    assert got.isfinite().all() == want.isfinite().all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,H", [(32, 512, 12), (8, 2048, 16)])        # chunks of 512 and of 208 steps (fp16: 512 and 688)
@pytest.mark.parametrize("w", [-12.0, -1.0])
def test_wkv6_long_sweeps(B, T, H, w, dtype):
    """Many blocks of steps in one CTA, with decays that keep the state and that forget it, against 64 bits: all results, and the
    steps at the far ends of both sweeps, where what every block leaves out would have added up."""
    from gpt_neox_b200.ops.wkv import wkv6
    torch.manual_seed(14)
    N, n = 64, 2                                   # (sequences and heads that are checked)
    mk = lambda m=0.0: (torch.randn(B, T, H * N, device="cuda") * 0.5 + m).to(dtype)
    leaves = [t.requires_grad_() for t in (mk(), mk(), mk(), mk(w), (torch.randn(H, N, device="cuda") * 0.3).to(dtype))]
    gy = mk()
    y = wkv6(*leaves)
    got = (y.detach(),) + torch.autograd.grad(y, leaves, gy)
    part = [t.detach()[:n, :, :n * N].double() for t in leaves[:4]] + [leaves[4].detach()[:n].double(), gy[:n, :, :n * N].double()]
    want = _wkv6_sweeps(*part)
    size = _wkv6_sweeps(*(t if i == 3 else t.abs() for i, t in enumerate(part)))
    terms = part[0].abs() * size[1] + part[1].abs() * size[2]
    size = (*size[:4], part[3].exp() * terms.flip(1).cumsum(1).flip(1))
    eps = 2 ** -9 if dtype == torch.bfloat16 else 2 ** -12
    for i, (a, b, c) in enumerate(zip(got, want, size)):
        a = a[:n, :, :n * N].double()
        for t in (slice(None), slice(0, 16), slice(T - 16, T)):
            # one rounding; in front of it fp32, and the decays' own error times the steps that remember it
            lim = eps * b[:, t].norm() + 2 ** -24 * c[:, t].norm() + 2 ** -25 * b[:, t].numel() ** 0.5
            assert (a[:, t] - b[:, t]).norm() <= lim, (i, t)


@pytest.mark.gpu
@pytest.mark.parametrize("B,T,H", [(32, 512, 12), (8, 2048, 16), (27, 2048, 16)])      # chunks of 512, 208 and 2048 steps
@pytest.mark.parametrize("w", [-12.0, -6.0, -1.0])
def test_wkv6_row_sums_have_fp32_precision(B, T, H, w):
    """The gradient of r before it is rounded, which the decay gradient is made of: an error of a last bit per step of a chunk
    that adds up like noise, and no drift that grows with the steps.  A chunk's start comes by one product and one exponential
    (two last bits) from the chunk before, likewise noise: about 1 per chunk.  (Without that, 8.3 units of 2 ** -24 at w = -6 in
    ten chunks of 208 steps are above the 8.2 that the steps alone give.)"""
    from gpt_neox_b200.ops import _lib
    torch.manual_seed(15)
    N, C = 64, H * 64
    r, k, v, gy = ((torch.randn(B, T, C, device="cuda") * 0.5).bfloat16() for _ in range(4))
    w = (torch.randn(B, T, C, device="cuda") * 0.5 + w).bfloat16()
    u = torch.randn(H, N, device="cuda") * 0.3
    lib, P = _lib.lib(r), _lib.ptr
    nc = lib.nx_wkv6_chunks(B, T, H)
    f32 = lambda *s: torch.empty(s, device="cuda")
    local, start, rstart, sumew = f32(B, H, nc, N, N), f32(B, H, nc, N, N), f32(B, H, nc, N, N), f32(B, H, nc, N)
    y, gr, gk, gv, gw = (torch.empty_like(r) for _ in range(5))
    gr32, gu, gu_part = f32(B, T, C), f32(H, N), f32(B, nc, H, N)
    lay = (r.stride(0), r.stride(1))
    _lib.check(lib.nx_wkv6_fwd(P(r), P(k), P(v), P(w), *lay, P(u), P(y), *lay, P(local), P(start), P(sumew), B, T, H, N,
                               _lib.stream()), "nx_wkv6_fwd")
    _lib.check(lib.nx_wkv6_bwd(P(r), P(k), P(v), P(w), P(gy), *lay, P(u), P(gr), P(gk), P(gv), P(gw), P(gr32), P(gu), P(gu_part),
                               *lay, P(local), P(start), P(rstart), P(sumew), B, T, H, N, _lib.stream()), "nx_wkv6_bwd")
    part = [t[:1, :, :2 * N].double() for t in (r, k, v, w)]
    want = _wkv6_sweeps(*part, u[:2].double(), gy[:1, :, :2 * N].double())[1]
    err = gr32[:1, :, :2 * N].double() - want
    steps = -(-(-(-T // 16)) // nc) * 16
    assert err.norm() <= 2 ** -24 * (steps ** 0.5 / 2 + (nc - 1) ** 0.5 + 1) * want.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("B,T,H", [(27, 2048, 16), (16, 700, 12), (40, 512, 12), (8, 333, 16)])
@pytest.mark.parametrize("w", [-12.0, -1.0])
def test_wkv6_chunks_of_all_lengths(B, T, H, w):
    """On 148 SMs one chunk of 2048 steps, two of 352, four of 128 and three of 112, ragged ones among them: what
    test_wkv6_long_sweeps asks for, of sequences whose reverse sweeps begin with the products of two states."""
    test_wkv6_long_sweeps(B, T, H, w, torch.bfloat16)


def _wkv6_sweeps(r, k, v, w, u, gy):
    """y and the gradients of r, k, v, w, u as two sweeps form them, one step after the other, in fp32 (64 bits for 64-bit inputs)."""
    B, T, _ = r.shape
    H, N = u.shape
    wide = lambda t: t if t.dtype == torch.float64 else t.float()
    r, k, v, w, gy = (wide(t).reshape(B, T, H, N) for t in (r, k, v, w, gy))
    u, ew = wide(u), -torch.exp(w)
    S, out = r.new_zeros(B, H, N, N), [[] for _ in range(5)]
    dot = lambda a, b: (a * b).sum(-1, keepdim=True)
    for t in range(T):
        st = dot(gy[:, t], v[:, t])
        out[0].append((r[:, t, :, :, None] * S).sum(-2) + dot(r[:, t] * u, k[:, t]) * v[:, t])
        out[1].append((S * gy[:, t, :, None]).sum(-1) + u * k[:, t] * st)
        S = torch.exp(ew[:, t])[..., None] * S + k[:, t, :, :, None] * v[:, t, :, None]
    G, Q, gu = torch.zeros_like(S), torch.zeros_like(r[:, 0]), torch.zeros_like(r[:, 0])
    for t in reversed(range(T)):
        st = dot(gy[:, t], v[:, t])
        row = (G * v[:, t, :, None]).sum(-1)
        gk = row + u * r[:, t] * st
        out[2].append(gk)
        out[3].append((k[:, t, :, :, None] * G).sum(-2) + dot(k[:, t] * u, r[:, t]) * gy[:, t])
        out[4].append((Q - k[:, t] * row) * ew[:, t])
        Q = Q + r[:, t] * out[1][t] - k[:, t] * gk
        gu = gu + r[:, t] * k[:, t] * st
        G = torch.exp(ew[:, t])[..., None] * G + r[:, t, :, :, None] * gy[:, t, :, None]
    y, gr = (torch.stack(x, 1).flatten(2) for x in out[:2])
    gk, gv, gw = (torch.stack(x[::-1], 1).flatten(2) for x in out[2:])
    return y, gr, gk, gv, gw, gu.sum(0)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,H", [(1, 100, 2), (1, 200, 2), (45, 50, 10)])       # step by step; many chunks and one
@pytest.mark.parametrize("positive", [True, False])
@pytest.mark.parametrize("what", [0, 1, 2, 4])                           # r, k, v, the gradient of y
def test_wkv6_infinities_are_those_of_single_steps(what, positive, B, T, H, dtype):
    """An infinite value gives infinities and NaN where sums of one step after the other give them, no more."""
    from gpt_neox_b200.ops.wkv import wkv6
    torch.manual_seed(12)
    N = 64
    ts = [(torch.randn(B, T, H * N, device="cuda") * 0.5 - (3.0 if i == 3 else 0.0)).to(dtype) for i in range(5)]
    u = (torch.randn(H, N, device="cuda") * 0.3).to(dtype)
    if positive:
        u, ts = u.abs(), [t if i == 3 else t.abs() for i, t in enumerate(ts)]
    ts[what][0, 21, 70] = math.inf
    leaves = [t.requires_grad_() for t in (*ts[:4], u)]
    y = wkv6(*leaves)
    got = (y.detach(),) + torch.autograd.grad(y, leaves, ts[4])
    gr, gk, gv, gw, gu = got[1:]
    want = _wkv6_sweeps(*(t.detach() for t in ts[:4]), u.detach(), ts[4])
    for n, (a, b) in enumerate(zip((y, gr, gk, gv, gw, gu), want)):
        if n == 4 and B == 1:
            continue                    # (the running difference starts anew in every chunk)
        b = b.to(dtype)
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isposinf(), b.isposinf()) \
            and torch.equal(a.isneginf(), b.isneginf()), n


@pytest.mark.gpu
@pytest.mark.parametrize("B,T", [(1, 24), (64, 48), (1, 150)])
@pytest.mark.parametrize("scales", [(2.0 ** 100, 2.0 ** 100, 2.0 ** -100, 2.0 ** -90),      # r k and gy v overflow, k v does not
                                    (2.0 ** -100, 2.0 ** 100, 2.0 ** 27, 2.0 ** -20)])       # a state above bf16's largest value
def test_wkv6_finite_extremes(scales, B, T):
    """Steps whose own products stay in fp32's range give finite results."""
    from gpt_neox_b200.ops.wkv import wkv6
    torch.manual_seed(13)
    H, N = 1, 64
    r, k, v, gy = (torch.full((B, T, N), c, device="cuda").bfloat16() for c in scales)
    if scales[2] > 1:
        k[:, 2:], v[:, 0], v[:, 1] = 0, 1.9921875 * 2.0 ** 27, 1.5 * 2.0 ** 19        # the state: 1.998 * 2 ** 127
    w, u = torch.full_like(r, -30.0), torch.zeros(H, N, device="cuda").bfloat16()
    leaves = [t.requires_grad_() for t in (r, k, v, w, u)]
    y = wkv6(*leaves)
    gr, gk, gv, gw, gu = torch.autograd.grad(y, leaves, gy)
    want = _wkv6_sweeps(*(t.detach() for t in (r, k, v, w, u)), gy)
    for n, (a, b) in enumerate(zip((y, gr, gk, gv), want)):
        assert b.isfinite().all()
        assert (a.float() - b).abs().max() <= 2 ** -7 * b.abs().max(), n

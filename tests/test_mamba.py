"""Mamba: model-level CPU checks and kernel numerics against the fp32 PyTorch recurrences."""
import pytest
import torch

from common import run_distributed, tiny_config


def _train(rank, world, cfg, steps):
    from gpt_neox_b200 import parallel as mpu
    from gpt_neox_b200 import training
    from gpt_neox_b200.config import NeoXArgs
    torch.set_num_threads(2)
    mpu.destroy_model_parallel()
    a = NeoXArgs.from_dict(dict(cfg, global_num_gpus=world, train_iters=steps, lr_decay_iters=steps))
    a.configure_distributed_args()
    a.build_tokenizer()
    losses = []
    training.collect_loss_for_unit_test = lambda l: losses.append(float(l))
    training.pretrain(a)
    return losses


def test_mamba_model_trains_on_cpu():
    cfg = tiny_config(attention_config=[[["mamba"], 2]], pos_emb="none", gpt_j_residual=False, norm="rmsnorm",
                      use_cpu_initialization=True, optimizer={"type": "Adam", "params": {"lr": 3e-3}})
    losses = run_distributed(_train, 1, cfg, 12)[0]
    assert all(l == l for l in losses)
    assert min(losses[6:]) < losses[0]


def test_mamba_tp2_sp_runs_on_cpu():
    cfg = tiny_config(attention_config=[[["mamba"], 2]], pos_emb="none", gpt_j_residual=False, norm="rmsnorm",
                      use_cpu_initialization=True, model_parallel_size=2, sequence_parallel=True)
    out = run_distributed(_train, 2, cfg, 3)
    assert out[0] == pytest.approx(out[1], rel=1e-6)


def test_conv_reference_is_causal():
    from gpt_neox_b200.ops.mamba import causal_conv1d_silu
    x = torch.randn(1, 10, 4)
    w, b = torch.randn(4, 4), torch.randn(4)
    y0 = causal_conv1d_silu(x, w, b)
    x2 = x.clone()
    x2[:, 6:] += 1.0
    y1 = causal_conv1d_silu(x2, w, b)
    assert torch.equal(y0[:, :6], y1[:, :6])


@pytest.mark.gpu
@pytest.mark.parametrize("L,D,W,bias", [(200, 192, 4, True), (64, 64, 3, False)])
def test_conv1d_silu_kernel(L, D, W, bias):
    from gpt_neox_b200.ops.mamba import causal_conv1d_silu, causal_conv1d_silu_reference
    torch.manual_seed(0)
    B = 3
    base = torch.randn(L, B, 2 * D, device="cuda", dtype=torch.bfloat16)
    x = base[..., :D].transpose(0, 1).detach().requires_grad_(True)      # strided [b, l, d] view
    w = (torch.randn(D, W, device="cuda") * 0.5).bfloat16().requires_grad_(True)
    b = torch.randn(D, device="cuda").bfloat16().requires_grad_(True) if bias else None
    y = causal_conv1d_silu(x, w, b)
    g = torch.randn(B, L, D, device="cuda", dtype=torch.bfloat16)
    y.backward(g)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    br = b.detach().float().requires_grad_(True) if bias else None
    yr = causal_conv1d_silu_reference(xr, wr, br)
    yr.backward(g.float())
    torch.testing.assert_close(y.float(), yr, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(x.grad.float(), xr.grad, rtol=3e-2, atol=3e-2)
    torch.testing.assert_close(w.grad.float(), wr.grad, rtol=3e-2, atol=0.15)
    if bias:
        torch.testing.assert_close(b.grad.float(), br.grad, rtol=3e-2, atol=0.15)


@pytest.mark.gpu
@pytest.mark.parametrize("L,D,use_z", [(300, 128, True), (128, 96, True), (40, 64, False)])
def test_selective_scan_kernel(L, D, use_z):
    from gpt_neox_b200.ops.mamba import selective_scan, selective_scan_reference
    torch.manual_seed(1)
    B, N = 2, 16
    dev = "cuda"
    mk = lambda *s: (torch.randn(*s, device=dev) * 0.5).bfloat16()
    x, dt, z = mk(B, L, D), mk(B, L, D), mk(B, L, D)
    bc = mk(L, B, 2 * N + 8)
    Bm, Cm = bc[..., 8:8 + N].transpose(0, 1), bc[..., 8 + N:].transpose(0, 1)    # strided views
    A = -(torch.rand(D, N, device=dev) * 4 + 0.5)
    Dp = torch.randn(D, device=dev)
    dtb = torch.randn(D, device=dev) * 0.5 - 2.0
    leaves = [t.detach().clone().requires_grad_(True) for t in (x, dt, A, Bm, Cm, Dp, z, dtb)]
    ref = [t.detach().clone().float().requires_grad_(True) for t in (x, dt, A, Bm, Cm, Dp, z, dtb)]
    y = selective_scan(leaves[0], leaves[1], leaves[2], leaves[3], leaves[4], leaves[5],
                       leaves[6] if use_z else None, leaves[7])
    yr = selective_scan_reference(ref[0], ref[1], ref[2], ref[3], ref[4], ref[5], ref[6] if use_z else None, ref[7])
    g = torch.randn(B, L, D, device=dev).bfloat16()
    y.backward(g)
    yr.backward(g.float())
    torch.testing.assert_close(y.float(), yr, rtol=3e-2, atol=3e-2)
    names = ["x", "dt", "A", "B", "C", "D", "z", "dt_bias"]
    for n, a, r in zip(names, leaves, ref):
        if n == "z" and not use_z:
            continue
        scale = r.grad.abs().max().item() + 1e-6
        err = (a.grad.float() - r.grad).abs().max().item()
        assert err <= 0.03 * scale + 1e-3, f"grad {n}: err {err} vs scale {scale}"


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("L,D,W,off", [(1, 8, 4, 0), (15, 64, 4, 0), (67, 264, 2, 0), (129, 40, 4, 4), (33, 36, 3, 0),
                                       (130, 8, 1, 2)])
def test_conv1d_silu_tiles_and_alignments(L, D, W, off, dtype):
    """Time-tile remainders, and channel counts / offsets that the 8- and 4-channel forms take or leave to the
    one-channel form."""
    from gpt_neox_b200.ops.mamba import causal_conv1d_silu, causal_conv1d_silu_reference
    torch.manual_seed(3)
    x = torch.randn(L, 2, D + 8, device="cuda").to(dtype)[..., off:off + D].transpose(0, 1).detach().requires_grad_(True)
    w = (torch.randn(D, W, device="cuda") * 0.5).to(dtype).requires_grad_(True)
    b = torch.randn(D, device="cuda").to(dtype).requires_grad_(True)
    g = torch.randn(2, L, D, device="cuda").to(dtype)
    y = causal_conv1d_silu(x, w, b)
    got = torch.autograd.grad(y, (x, w, b), g)
    ref = [t.detach().float().requires_grad_(True) for t in (x, w, b)]
    yr = causal_conv1d_silu_reference(*ref)
    want = torch.autograd.grad(yr, ref, g.float())
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
    for a, r in zip((y,) + got, (yr,) + want):                  # one rounding to 16 bits; fp32 sums on both sides
        assert (a.float() - r).abs().max().item() <= 2 * eps * r.abs().max().item() + 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,L,D", [(1, 1, 32), (2, 31, 40), (1, 33, 36), (1, 700, 64), (2, 257, 8), (40, 96, 136)])
def test_selective_scan_blocks_and_chunks(B, L, D, dtype):
    """Block and chunk remainders, one chunk (many channels) and many (few channels), channel counts that the 16-byte
    staging takes or not; forward with and without the states for the backward."""
    from gpt_neox_b200.ops.mamba import selective_scan, selective_scan_reference
    torch.manual_seed(6)
    mk = lambda *s: (torch.randn(*s, device="cuda") * 0.5).to(dtype)
    xz, bc = mk(L, B, 2 * D), mk(L, B, 40)
    x, z, dt = xz[..., :D].transpose(0, 1), xz[..., D:].transpose(0, 1), mk(L, B, D).transpose(0, 1)
    Bm, Cm = bc[..., 3:19].transpose(0, 1), bc[..., 19:35].transpose(0, 1)
    A, Dp = -(torch.rand(D, 16, device="cuda") * 4 + 0.5), torch.randn(D, device="cuda")
    dtb = torch.randn(D, device="cuda") * 0.5 - 2.0
    leaves = [t.detach().requires_grad_(True) for t in (x, dt, A, Bm, Cm, Dp, z, dtb)]
    ref = [t.detach().float().clone().requires_grad_(True) for t in leaves]
    g = mk(B, L, D)
    y = selective_scan(*leaves)
    got = torch.autograd.grad(y, leaves, g)
    yr = selective_scan_reference(*ref)
    want = torch.autograd.grad(yr, ref, g.float())
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
    for a, r in zip((y,) + got, (yr,) + want):
        assert (a.float() - r).abs().max().item() <= 2 * eps * r.abs().max().item() + 1e-4
    with torch.no_grad():
        assert torch.equal(selective_scan(*leaves), y)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,L,D,off,use_z", [(1, 1, 1, 0, True), (2, 3, 2, 0, False), (1, 5, 15, 0, True), (2, 32, 17, 1, True),
                                             (1, 36, 63, 0, False), (3, 65, 66, 1, True), (1, 130, 64, 0, False),
                                             (1, 997, 129, 0, True)])
def test_selective_scan_pairs_and_segments(B, L, D, off, use_z, dtype):
    """Odd channel counts and bases (a quad's second channel dead or read by itself), warps and CTAs with few live channels,
    segments of four and blocks of 32 that the length cuts, B and C on 8-byte boundaries, one chunk and many, no gate, no D."""
    from gpt_neox_b200.ops.mamba import selective_scan, selective_scan_reference
    torch.manual_seed(7)
    mk = lambda *s: (torch.randn(*s, device="cuda") * 0.5).to(dtype)
    xz, bc = mk(L, B, 2 * D + off), mk(L, B, 32)
    x, z, dt = xz[..., off:off + D].transpose(0, 1), xz[..., off + D:].transpose(0, 1), mk(L, B, D).transpose(0, 1)
    dt = (dt.float() * 8 - 2).to(dtype)          # both branches of the softplus, and steps that forget everything
    A, dtb = -(torch.rand(D, 16, device="cuda") * 4 + 0.5), torch.randn(D, device="cuda") * 0.5 - 2.0
    Dp = torch.randn(D, device="cuda") if use_z else None
    args = [x, dt, A, bc[..., :16].transpose(0, 1), bc[..., 16:].transpose(0, 1), Dp, z if use_z else None, dtb]
    leaves = [None if t is None else t.detach().requires_grad_(True) for t in args]
    ref = [None if t is None else t.detach().float().clone().requires_grad_(True) for t in leaves]
    g = mk(B, L, D)
    y, yr = selective_scan(*leaves), selective_scan_reference(*ref)
    got = torch.autograd.grad(y, [t for t in leaves if t is not None], g)
    want = torch.autograd.grad(yr, [t for t in ref if t is not None], g.float())
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
    for a, r in zip((y,) + got, (yr,) + want):                  # one rounding to 16 bits; fp32 sums on both sides
        assert (a.float() - r).abs().max().item() <= 2 * eps * r.abs().max().item() + 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("lo,hi,units", [(-40.0, -10.0, 16), (-10.0, -5.0, 4), (-5.0, -3.0, 1.8), (-3.0, -1.0, 1.25), (-1.0, 0.0, 1),
                                         (0.0, 1.0, 1), (1.0, 20.0, 0.5), (20.0, 60.0, 0.25)])
def test_selective_scan_softplus_has_fp32_precision(lo, hi, units):
    """The step that the scan forms from dt + dt_bias, in fp32: without decay the state behind one step of input 1 is that step.
    Root mean square of the relative error against 64 bits, in units of 2 ** -24: below one where the roundings of log(1 + e) are
    all there is, more where the argument's rounding before the exponential (|v| units at most, a third on average) counts, less
    where v itself is nearly all of the result.  (2 artanh(e / (2 + e)) with a division had 1.22 and 1.4 in (-1, 0) and (-3, -1).)"""
    from gpt_neox_b200.ops import mamba
    torch.manual_seed(5)
    D, L = 1 << 16, 33
    v = torch.empty(D, device="cuda").uniform_(lo, hi)
    zeros = lambda *s: torch.zeros(s, device="cuda", dtype=torch.float16)
    x, B = zeros(1, L, D), zeros(1, L, 16)
    x[:, 0], B[..., 0] = 1, 1
    _, states = mamba._scan_forward(x, zeros(1, L, D), torch.zeros(D, 16, device="cuda"), B, zeros(1, L, 16), None, None, v, True)
    want = torch.log1p(torch.exp(-v.double().abs())) + v.double().clamp(min=0)
    err = states[0, 1, :, 0].double() / want - 1
    assert err.square().mean().sqrt() <= units * 2 ** -24


@pytest.mark.gpu
def test_selective_scan_softplus_at_the_ends():
    from gpt_neox_b200.ops import mamba
    v = torch.tensor([float("inf"), float("-inf"), float("nan"), 0.0, -200.0, 3e38, -3e38, 88.0], device="cuda")
    zeros = lambda *s: torch.zeros(s, device="cuda", dtype=torch.float16)
    x, B = zeros(1, 33, 8), zeros(1, 33, 16) + 1
    x[:, 0] = 1
    out, states = mamba._scan_forward(x, zeros(1, 33, 8), torch.full((8, 16), -1.0, device="cuda"), B, B / 16, None, None, v, True)
    y = out[0, 0].float()                          # the step itself, rounded to fp16 (16 states with a sixteenth each)
    assert y[0].isposinf() and y[1] == 0 and y[2].isnan() and abs(y[3] - 0.6931) < 5e-4
    assert y[4] == 0 and y[5].isposinf() and y[6] == 0 and y[7] == 88


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,L,D", [(1, 22, 8), (3, 129, 2052), (2, 707, 1536), (4, 2501, 1544)])
def test_conv1d_silu_steps_per_thread(B, L, D, dtype):
    """4, 8, 16 and 32 steps a thread forward, and 5, 5, 13 and 21 backward (on 148 SMs), with ragged ends."""
    from gpt_neox_b200.ops.mamba import causal_conv1d_silu, causal_conv1d_silu_reference
    torch.manual_seed(8)
    mk = lambda *s: (torch.randn(*s, device="cuda") * 0.5).to(dtype).requires_grad_()
    x, w, b, g = mk(B, L, D), mk(D, 4), mk(D), mk(B, L, D).detach()
    ref = [t.detach().double().requires_grad_() for t in (x, w, b)]
    y = causal_conv1d_silu(x, w, b)
    yr = torch.nn.functional.silu(torch.nn.functional.conv1d(ref[0].transpose(1, 2), ref[1][:, None], ref[2], padding=3,
                                                             groups=D)[..., :L].transpose(1, 2))
    eps = 2 ** -8 if dtype == torch.bfloat16 else 2 ** -11
    for a, r in zip((y,) + torch.autograd.grad(y, [x, w, b], g), (yr,) + torch.autograd.grad(yr, ref, g.double())):
        # one rounding to 16 bits; fp32 sums over B L steps for the taps and the bias
        assert ((a.double() - r).abs() <= eps * r.abs() + 2 ** -20 * (B * L) ** 0.5).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,L,D,off,use_z", [(500, 1, 33, 0, True), (480, 3, 34, 0, False), (480, 5, 47, 0, True), (460, 37, 49, 1, True),
                                             (480, 36, 63, 0, True), (250, 97, 129, 0, False), (460, 40, 64, 1, False)])
def test_selective_scan_two_channels_a_quad(B, L, D, off, use_z, dtype):
    """The same with so many sequences that a quad has two channels, the second one dead or read by itself."""
    from gpt_neox_b200.ops import _lib
    assert _lib.lib(dtype).nx_scan_tiles(B, L, D) == -(-D // 64)
    test_selective_scan_pairs_and_segments(B, L, D, off, use_z, dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("what,value", [("x", float("nan")), ("dt", float("nan")), ("B", float("nan")), ("C", float("inf")),
                                        ("z", float("nan")), ("x", float("inf"))])
@pytest.mark.parametrize("at", [0, 37, 255, 299])
def test_selective_scan_passes_nan_and_inf_on(what, value, at):
    """A non-finite input in the first, a middle and the last chunk of a sequence: the outputs that are not finite are those
    of the sequential statement (its own channel and the steps after it)."""
    from gpt_neox_b200.ops.mamba import selective_scan, selective_scan_reference
    torch.manual_seed(12)
    L, D = 300, 40
    mk = lambda *s: (torch.randn(*s, device="cuda") * 0.5).bfloat16()
    t = dict(x=mk(2, L, D), dt=mk(2, L, D), B=mk(2, L, 16), C=mk(2, L, 16), z=mk(2, L, D))
    t[what][1, at, 3] = value
    A, Dp, bias = -(torch.rand(D, 16, device="cuda") + 0.5), torch.randn(D, device="cuda"), torch.zeros(D, device="cuda") - 3
    args = lambda c: (c(t["x"]), c(t["dt"]), A, c(t["B"]), c(t["C"]), Dp, c(t["z"]), bias)
    got, want = selective_scan(*args(lambda u: u)), selective_scan_reference(*args(lambda u: u.float()))
    assert torch.equal(got.isfinite(), want.isfinite()) and not got.isfinite().all()

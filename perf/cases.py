"""Performance cases: the calls a training or generation program makes most, through the public entry points.

Every kind of case is one layer or block of the configurations under ``configs/`` (or, for ``generate``, a whole small
model) at the sizes those configurations use.  ``listed()`` names twelve of them; ``draw(rng)`` gives further ones from
the same ranges: hidden sizes, head counts and vocabularies of the configurations, any number of tokens, bf16 and fp16
where both are configured.  Forward and backward run in one pass for the training kinds and the pass returns the
outputs and every gradient; the decoding kinds run without autograd, as generation does.
"""
import contextlib
import io
import math

import torch
import torch.nn.functional as F

from gpt_neox_b200.ops import attention, cross_entropy, elementwise, fused, gemm, mamba, moe, norm, optim, rope, wkv

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


# ---------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one layer's attention of the 6.9B configuration at its training shape (sequence 2048, micro-batch 4)
        dict(name="attention_train", kind="attention", dtype="bf16", seq=2048, batch=4, heads=32, kv=32, dim=128, rot=32,
             window=-1),
        # grouped-query attention with a sliding window (the 7B mistral configuration), a sequence that no tile divides
        dict(name="attention_train_gqa_window", kind="attention", dtype="bf16", seq=5003, batch=1, heads=32, kv=8,
             dim=128, rot=128, window=4096),
        # one layer's attention while generating: one new token per sequence against its cache
        dict(name="attention_decode", kind="decode", dtype="bf16", keys=1543, batch=8, heads=32, kv=32, dim=128),
        # the MLP block of the 6.9B configuration, forward and backward with the residual add
        dict(name="mlp_train", kind="mlp", dtype="bf16", tokens=8192, hidden=4096, ffn=16384),
        # the gated MLP of the 7B llama configuration while generating for a few sequences
        dict(name="mlp_decode", kind="gated_mlp_decode", dtype="bf16", tokens=4, hidden=4096, ffn=11008),
        # both LayerNorms of a parallel-residual block with the residual stream, forward and backward (1.4B width)
        dict(name="norm_train", kind="norm", dtype="bf16", form="dual", tokens=8192, hidden=2048),
        # language-model head and loss of the 6.9B configuration
        dict(name="head_loss_train", kind="head", dtype="bf16", tokens=8192, hidden=4096, vocab=50432),
        # the dropless-MoE feed-forward layer of the 125M configuration (8 experts, top 2)
        dict(name="moe_train", kind="moe", dtype="bf16", tokens=16384, hidden=768, ffn=3072, experts=8, topk=2),
        # conv + selective scan of the 130M Mamba configuration (fp16, as configured)
        dict(name="mamba_train", kind="mamba", dtype="fp16", seq=2048, batch=4, inner=1536),
        # the WKV recurrence of the 170M RWKV configuration
        dict(name="wkv_train", kind="wkv", dtype="bf16", seq=512, batch=32, heads=12, head_size=64),
        # gradient norm, clip coefficient and AdamW over one rank's flat shard (the 1.4B model over 8 ranks)
        dict(name="optimizer_step", kind="adamw", dtype="bf16", elements=176_800_000),
        # whole-model generation with the 160M configuration: a prompt, then cached single-token steps; logits out
        dict(name="generate", kind="generate", dtype="bf16", layers=12, hidden=768, heads=12, batch=4, prompt=100, steps=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "decode", "mlp", "gated_mlp_decode", "norm", "head", "moe", "mamba", "wkv", "adamw",
                       "generate"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16"])
    if kind in ("attention", "decode"):
        heads, dim = rng.choice([(12, 64), (16, 64), (16, 128), (32, 128)])
        kv = rng.choice([heads, heads, heads // 4])
        if kind == "decode":
            return dict(kind=kind, dtype=dtype, keys=_log(rng, 16, 8192), batch=_log(rng, 1, 32), heads=heads, kv=kv, dim=dim)
        seq = _log(rng, 128, 4096)
        return dict(kind=kind, dtype=dtype, seq=seq, batch=_log(rng, 1, max(1, 8192 // seq)), heads=heads, kv=kv, dim=dim,
                    rot=rng.choice([dim, dim // 4]), window=rng.choice([-1, -1, -1, seq // 2]))
    if kind == "mlp":
        hidden = rng.choice([512, 768, 1024, 2048, 4096])
        return dict(kind=kind, dtype=dtype, tokens=_log(rng, 256, 8192), hidden=hidden, ffn=4 * hidden)
    if kind == "gated_mlp_decode":
        hidden, ffn = rng.choice([(2048, 5632), (4096, 11008), (4096, 14336), (5120, 13824)])
        return dict(kind=kind, dtype=dtype, tokens=_log(rng, 1, 64), hidden=hidden, ffn=ffn)
    if kind == "norm":
        return dict(kind=kind, dtype=dtype, form=rng.choice(["dual", "layer", "rms"]), tokens=_log(rng, 64, 16384),
                    hidden=rng.choice([512, 768, 1024, 2048, 2560, 4096, 5120, 6144]))
    if kind == "head":
        return dict(kind=kind, dtype="bf16", tokens=_log(rng, 256, 8192), hidden=rng.choice([512, 768, 1024, 2048, 4096]),
                    vocab=rng.choice([32000, 50304, 50432]))
    if kind == "moe":
        hidden = rng.choice([512, 768, 1024])
        return dict(kind=kind, dtype=dtype, tokens=_log(rng, 512, 16384), hidden=hidden, ffn=4 * hidden,
                    experts=rng.choice([4, 8, 16]), topk=rng.choice([1, 2]))
    if kind == "mamba":
        seq = _log(rng, 128, 4096)
        return dict(kind=kind, dtype=dtype, seq=seq, batch=_log(rng, 1, max(1, 8192 // seq)),
                    inner=rng.choice([1536, 2048, 3072]))
    if kind == "wkv":
        seq = _log(rng, 64, 2048)
        return dict(kind=kind, dtype="bf16", seq=seq, batch=_log(rng, 1, max(1, 16384 // seq)), heads=rng.choice([8, 12, 16]),
                    head_size=64)
    if kind == "adamw":
        return dict(kind=kind, dtype=dtype, elements=8 * _log(rng, 20_000, 22_000_000))
    hidden, heads = rng.choice([(512, 8), (768, 12), (1024, 16)])
    return dict(kind=kind, dtype=dtype, layers=rng.choice([6, 12]), hidden=hidden, heads=heads, batch=_log(rng, 1, 8),
                prompt=_log(rng, 16, 512), steps=rng.choice([4, 8, 16]))


# -------------------------------------------------------------------------------------------------------------- inputs
def prepare(case, seed):
    c, g = case, torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * (seed + 1))
    dt = DTYPES[c["dtype"]]

    def rand(*shape, std=1.0, dtype=dt, grad=False):
        t = torch.empty(shape, device="cuda", dtype=torch.float32).normal_(0.0, std, generator=g).to(dtype)
        return t.requires_grad_() if grad else t

    return globals()["_prepare_" + c["kind"]](c, seed, rand, g)


def _prepare_attention(c, seed, rand, g):
    width = (c["heads"] + 2 * c["kv"]) * c["dim"]
    cos, sin = rope.rotary_tables(c["rot"], c["seq"], device="cuda")
    return dict(case=c, qkv=rand(c["seq"], c["batch"], width, grad=True), cos=cos, sin=sin,
                gout=rand(c["seq"], c["batch"], c["heads"] * c["dim"]))


def _prepare_decode(c, seed, rand, g):
    # [seq, batch, heads, dim] memory, as the layers keep their caches; the kernel takes [batch, seq, heads, dim] views
    perm = lambda t: t.permute(1, 0, 2, 3)
    return dict(case=c, q=perm(rand(1, c["batch"], c["heads"], c["dim"])),
                k=perm(rand(c["keys"], c["batch"], c["kv"], c["dim"])),
                v=perm(rand(c["keys"], c["batch"], c["kv"], c["dim"])))


def _prepare_mlp(c, seed, rand, g):
    t, h, f = c["tokens"], c["hidden"], c["ffn"]
    return dict(case=c, x=rand(t, h, grad=True), w1=rand(f, h, std=0.02, grad=True), b1=rand(f, std=0.02, grad=True),
                w2=rand(h, f, std=0.02, grad=True), b2=rand(h, std=0.02, grad=True), residual=rand(t, h, grad=True),
                gout=rand(t, h))


def _prepare_gated_mlp_decode(c, seed, rand, g):
    t, h, f = c["tokens"], c["hidden"], c["ffn"]
    return dict(case=c, x=rand(t, 1, h), w1=rand(2 * f, h, std=0.02), w2=rand(h, f, std=0.02))


def _prepare_norm(c, seed, rand, g):
    t, h, dual = c["tokens"], c["hidden"], c["form"] == "dual"
    s = dict(case=c, x=rand(t, h, std=2.0, grad=True), gouts=[rand(t, h) for _ in range(3 if dual else 2)])
    names = {"dual": ("w1", "b1", "w2", "b2"), "layer": ("w1", "b1"), "rms": ("w1",)}[c["form"]]
    s["params"] = [(rand(h, std=0.1).float() + (1.0 if n[0] == "w" else 0.0)).to(s["x"].dtype).requires_grad_()
                   for n in names]
    return s


def _prepare_head(c, seed, rand, g):
    # targets as a text has them: frequent and rare tokens (roughly Zipf)
    u = torch.empty(c["tokens"], device="cuda").uniform_(0.0, 1.0, generator=g)
    labels = torch.clamp((c["vocab"] ** u - 1.0).long(), max=c["vocab"] - 1)
    return dict(case=c, x=rand(c["tokens"], c["hidden"], grad=True), w=rand(c["vocab"], c["hidden"], std=0.02, grad=True),
                labels=labels, gout=torch.full((c["tokens"],), 1.0 / c["tokens"], device="cuda"))


def _prepare_moe(c, seed, rand, g):
    t, h, f, e, k = c["tokens"], c["hidden"], c["ffn"], c["experts"], c["topk"]
    # a router that prefers some experts a little, as a trained one does
    score = torch.empty(t, e, device="cuda").normal_(0.0, 1.0, generator=g)
    score += torch.empty(e, device="cuda").normal_(0.0, 0.5, generator=g)
    weights, indices = torch.topk(torch.softmax(score, -1), k)
    return dict(case=c, x=rand(t, h, grad=True), weights=weights.to(DTYPES[c["dtype"]]).requires_grad_(), indices=indices,
                w1=rand(e * f, h, std=0.02, grad=True), w2=rand(e * f, h, std=0.02, grad=True), gout=rand(t, h))


def _prepare_mamba(c, seed, rand, g):
    # the block's own layouts: x | z halves of one projection, B | C columns of another, time-major memory
    L, b, d = c["seq"], c["batch"], c["inner"]
    rank = d // 32
    xz, dbl = rand(L, b, 2 * d), rand(L, b, rank + 32)
    leaf = lambda t: t.transpose(0, 1).detach().requires_grad_()
    dt0 = torch.exp(torch.empty(d, device="cuda").uniform_(math.log(1e-3), math.log(0.1), generator=g))
    return dict(case=c, x=leaf(xz[..., :d]), z=leaf(xz[..., d:]), dt=leaf(rand(L, b, d, std=0.5)),
                B=leaf(dbl[..., rank:rank + 16]), C=leaf(dbl[..., rank + 16:]),
                conv_w=rand(d, 4, std=0.3, grad=True), conv_b=rand(d, std=0.1, grad=True),
                A=(-torch.arange(1, 17, device="cuda", dtype=torch.float32).repeat(d, 1)).requires_grad_(),
                D=torch.ones(d, device="cuda", requires_grad=True),
                dt_bias=(dt0 + torch.log(-torch.expm1(-dt0))).requires_grad_(),
                gout=rand(L, b, d).transpose(0, 1))


def _prepare_wkv(c, seed, rand, g):
    T, b, H, N = c["seq"], c["batch"], c["heads"], c["head_size"]
    leaf = lambda t: t.transpose(0, 1).detach().requires_grad_()
    ramp = (-6 + 5 * (torch.arange(H * N, device="cuda") / (H * N - 1)) ** 1.3).to(DTYPES[c["dtype"]])
    return dict(case=c, r=leaf(rand(T, b, H * N)), k=leaf(rand(T, b, H * N)), v=leaf(rand(T, b, H * N)),
                w=leaf(ramp + rand(T, b, H * N, std=0.3)), u=rand(H, N, std=0.3, grad=True),
                gout=rand(T, b, H * N).transpose(0, 1))


def _prepare_adamw(c, seed, rand, g):
    n = c["elements"]
    p = rand(n, std=0.02, dtype=torch.float32)
    return dict(case=c, p=p, m=rand(n, std=1e-4, dtype=torch.float32), v=rand(n, std=1e-4, dtype=torch.float32).square_(),
                g=rand(n, std=1e-4), lp=p.to(DTYPES[c["dtype"]]), acc=torch.zeros(2, device="cuda"),
                scale=torch.zeros(2, device="cuda"), skip=torch.zeros(1, device="cuda", dtype=torch.int32))


def _prepare_generate(c, seed, rand, g):
    from gpt_neox_b200 import parallel as mpu
    from gpt_neox_b200 import training
    from gpt_neox_b200.config import NeoXArgs
    from gpt_neox_b200.initialize import initialize_megatron
    length = 1024
    config = dict(
        num_layers=c["layers"], hidden_size=c["hidden"], num_attention_heads=c["heads"], seq_length=length,
        max_position_embeddings=length, pos_emb="rotary", rotary_pct=0.25, gpt_j_residual=True, no_weight_tying=True,
        norm="layernorm", attention_config=[[["flash"], c["layers"]]], bias_gelu_fusion=True, pipe_parallel_size=0,
        train_micro_batch_size_per_gpu=c["batch"], train_iters=10, lr_decay_iters=10, global_num_gpus=1, num_workers=0,
        precision="bfloat16" if c["dtype"] == "bf16" else "fp16", dataset_impl="synthetic", synthetic_vocab_size=50277,
        tokenizer_type="HFTokenizer", init_method="small_init", output_layer_init_method="wang_init", seed=seed + 1,
        optimizer={"type": "Adam", "params": {"lr": 6e-4, "betas": [0.9, 0.95], "eps": 1e-8}})
    with contextlib.redirect_stdout(io.StringIO()):
        args = NeoXArgs.from_dict(config)
        args.configure_distributed_args()
        args.build_tokenizer()
        mpu.destroy_model_parallel()
        initialize_megatron(args)
        model = training.get_model(args, use_cache=True)
    model.eval()
    model.inference_mode(use_cache=True)
    n = c["prompt"] + c["steps"]
    tokens = torch.randint(0, 50277, (c["batch"], n), device="cuda", generator=g)
    positions = torch.arange(n, device="cuda")[None].expand(c["batch"], -1)
    pieces = [slice(0, c["prompt"])] + [slice(i, i + 1) for i in range(c["prompt"], n)]
    return dict(case=c, model=model, tokens=tokens,
                feeds=[(tokens[:, p].contiguous(), positions[:, p].contiguous()) for p in pieces])


# -------------------------------------------------------------------------------------------------------------- passes
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state, state["case"])


def _run_attention(s, c):
    y = fused.qkv_attention(s["qkv"], num_heads=c["heads"], num_kv_heads=c["kv"], head_dim=c["dim"], rotary_dim=c["rot"],
                            cos=s["cos"], sin=s["sin"], window=c["window"])
    return [y.detach()] + list(torch.autograd.grad(y, [s["qkv"]], s["gout"]))


def _run_decode(s, c):
    with torch.no_grad():
        return attention.flash_attention(s["q"], s["k"], s["v"])


def _run_mlp(s, c):
    leaves = [s[n] for n in ("x", "w1", "b1", "w2", "b2", "residual")]
    y = fused.mlp_gelu(*leaves)
    return [y.detach()] + list(torch.autograd.grad(y, leaves, s["gout"]))


def _run_gated_mlp_decode(s, c):
    with torch.no_grad():
        return gemm.linear(elementwise.gated_act(gemm.linear(s["x"], s["w1"]), "swiglu"), s["w2"])


def _run_norm(s, c):
    x, p = s["x"], s["params"]
    if c["form"] == "dual":
        ys = norm.dual_layer_norm(x, *p, carry=True)
    elif c["form"] == "layer":
        ys = norm.layer_norm(x, *p, carry=True)
    else:
        ys = norm.rms_norm(x, *p, eps=1e-5, carry=True)
    return [y.detach() for y in ys[1:]] + list(torch.autograd.grad(ys, [x] + p, s["gouts"]))


def _run_head(s, c):
    loss = cross_entropy.vocab_parallel_cross_entropy(gemm.linear(s["x"], s["w"]), s["labels"])
    return [loss.detach()] + list(torch.autograd.grad(loss, [s["x"], s["w"]], s["gout"]))


def _run_moe(s, c):
    leaves = [s[n] for n in ("x", "weights", "w1", "w2")]
    y = moe.experts_gelu(leaves[0], leaves[1], s["indices"], leaves[2], leaves[3], c["experts"])
    return [y.detach()] + list(torch.autograd.grad(y, leaves, s["gout"]))


MAMBA_LEAVES = ("x", "z", "dt", "B", "C", "conv_w", "conv_b", "A", "D", "dt_bias")


def _run_mamba(s, c):
    u = mamba.causal_conv1d_silu(s["x"], s["conv_w"], s["conv_b"])
    y = mamba.selective_scan(u, s["dt"], s["A"], s["B"], s["C"], D=s["D"], z=s["z"], dt_bias=s["dt_bias"])
    return [y.detach()] + list(torch.autograd.grad(y, [s[n] for n in MAMBA_LEAVES], s["gout"]))


def _run_wkv(s, c):
    leaves = [s[n] for n in ("r", "k", "v", "w", "u")]
    y = wkv.wkv6(*leaves)
    return [y.detach()] + list(torch.autograd.grad(y, leaves, s["gout"]))


ADAMW = dict(lr=1e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=100)


def _run_adamw(s, c):
    s["acc"].zero_()
    optim.sumsq_(s["g"], s["acc"])
    optim.clip_coef_(s["acc"], 1.0, 1.0, s["scale"], s["skip"])
    optim.adamw_step_(s["p"], s["m"], s["v"], s["g"], s["lp"], grad_scale=s["scale"], skip=s["skip"], **ADAMW)
    return [s["p"], s["m"], s["v"], s["lp"], s["scale"]]


def _run_generate(s, c):
    model = s["model"]
    model.clear_cache()
    with torch.no_grad():
        return [model((tokens, positions, None))[:, -1] for tokens, positions in s["feeds"]]


# --------------------------------------------------------------------------------- what a pass cannot do without
def _pairs(c):
    """(query, key) pairs of one causal head, a window keeping the nearest window + 1 keys."""
    s, w = c["seq"], c["window"]
    if w < 0 or w + 1 >= s:
        return s * (s + 1) // 2
    return (w + 1) * (w + 2) // 2 + (s - w - 1) * (w + 1)


def work(case):
    c, kind = case, case["kind"]
    if kind == "attention":
        rows = c["seq"] * c["batch"]
        return {"bytes": 2 * rows * c["dim"] * 2 * (2 * c["heads"] + 2 * c["kv"]),
                "flops": 14 * c["batch"] * c["heads"] * c["dim"] * _pairs(c)}
    if kind == "decode":
        return {"bytes": 2 * c["batch"] * c["dim"] * 2 * (c["heads"] + c["keys"] * c["kv"]),
                "flops": 4 * c["batch"] * c["heads"] * c["dim"] * c["keys"]}
    if kind == "mlp":
        t, h, f = c["tokens"], c["hidden"], c["ffn"]
        return {"bytes": 2 * (6 * t * h + 4 * h * f + 2 * (h + f)), "flops": 12 * t * h * f}
    if kind == "gated_mlp_decode":
        t, h, f = c["tokens"], c["hidden"], c["ffn"]
        return {"bytes": 2 * (2 * t * h + 3 * h * f), "flops": 6 * t * h * f}
    if kind == "norm":
        t, h, dual = c["tokens"], c["hidden"], c["form"] == "dual"
        return {"bytes": 2 * t * h * (7 if dual else 5), "flops": (30 if dual else 20) * t * h}
    if kind == "head":
        t, h, v = c["tokens"], c["hidden"], c["vocab"]
        return {"bytes": 2 * (2 * t * h + 2 * v * h) + 16 * t, "flops": 6 * t * h * v}
    if kind == "moe":
        t, h, f, e, k = (c[n] for n in ("tokens", "hidden", "ffn", "experts", "topk"))
        return {"bytes": 2 * (4 * t * h + 4 * e * f * h + 2 * t * k) + 8 * t * k, "flops": 12 * t * k * h * f}
    if kind == "mamba":
        t, d = c["seq"] * c["batch"], c["inner"]
        return {"bytes": 2 * t * (8 * d + 64), "flops": t * d * 16 * 24}
    if kind == "wkv":
        t, ch = c["seq"] * c["batch"], c["heads"] * c["head_size"]
        return {"bytes": 2 * t * ch * 10, "flops": 20 * t * ch * c["head_size"]}
    if kind == "adamw":
        return {"bytes": 28 * c["elements"], "flops": 16 * c["elements"]}
    h, n, vocab = c["hidden"], c["layers"], 50304
    weights = n * 12 * h * h + vocab * h
    tokens = c["batch"] * (c["prompt"] + c["steps"])
    cache = 2 * 2 * n * h * c["batch"] * (c["prompt"] + c["steps"] // 2)
    return {"bytes": 2 * weights * (1 + c["steps"]) + cache * c["steps"], "flops": 2 * weights * tokens}


# ---------------------------------------------------------------------------------------------------------- tolerances
def tolerance(case):
    c, half = case, case["dtype"] == "fp16"
    # bf16 keeps 8 bits of a number, fp16 11: what changes between correct implementations is the rounding of stored
    # 16-bit values and of the intermediate ones that an implementation keeps in 16 bits (probabilities, activations)
    rel = {"attention": 1.2e-2, "decode": 1.0e-2, "mlp": 1.2e-2, "gated_mlp_decode": 1.2e-2, "norm": 1.0e-2,
           "head": 1.5e-2, "moe": 1.5e-2, "mamba": 1.5e-2, "wkv": 1.0e-2, "generate": 2.5e-2}
    if c["kind"] == "adamw":
        # the fp32 state differs by the rounding of one update, the 16-bit copy by its last bit for the few elements
        # that land on the other side of a rounding boundary
        return {"rel": 2e-5}
    return {"rel": rel[c["kind"]] / (4 if half else 1)}


# --------------------------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    if case["kind"] == "adamw" and case["elements"] > 200_000_000:
        return None
    s = prepare(case, seed)
    return globals()["_exact_" + case["kind"]](s, case)


def _double(t):
    return t.detach().double().requires_grad_(t.requires_grad)


def _grads(ys, leaves, gouts):
    return [g.detach() for g in torch.autograd.grad(ys, leaves, gouts)]


def _rotate(x, cos, sin, rot):
    half = rot // 2
    c, s = cos.double()[:x.shape[0], None, None], sin.double()[:x.shape[0], None, None]
    a, b = x[..., :half], x[..., half:rot]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., rot:]], -1)


def _softmax_attention(q, k, v, window=-1):
    """[s, heads, d] of one sequence, queries at the end of the keys."""
    rep = q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1)
    scores = torch.einsum("qhd,khd->hqk", q, k) / math.sqrt(q.shape[-1])
    qp = torch.arange(q.shape[0], device=q.device)[:, None] + k.shape[0] - q.shape[0]
    kp = torch.arange(k.shape[0], device=q.device)[None]
    dead = kp > qp
    if window >= 0:
        dead = dead | (kp < qp - window)
    return torch.einsum("hqk,khd->qhd", torch.softmax(scores.masked_fill(dead, float("-inf")), -1), v)


def _split_heads(qkv, heads, kv, dim):
    s, b = qkv.shape[:2]
    if heads == kv:
        return qkv.view(s, b, heads, 3 * dim).split(dim, -1)
    return [t.reshape(s, b, -1, dim) for t in qkv.split([heads * dim, kv * dim, kv * dim], -1)]


def _exact_attention(s, c):
    qkv, group = _double(s["qkv"]), c["heads"] // c["kv"]
    q, k, v = _split_heads(qkv, c["heads"], c["kv"], c["dim"])
    q, k = _rotate(q, s["cos"], s["sin"], c["rot"]), _rotate(k, s["cos"], s["sin"], c["rot"])
    flat = [t.detach().requires_grad_() for t in (q, k, v)]
    gout = s["gout"].double().view(c["seq"], c["batch"], c["heads"], c["dim"])
    out, grads = torch.empty_like(gout), [torch.empty_like(t) for t in flat]
    for b in range(c["batch"]):                     # a few heads of one sequence at a time: the scores fit in memory
        for h in range(0, c["kv"], 4):
            piece = [t[:, b, n * h:n * (h + 4)] for t, n in zip(flat, (group, 1, 1))]
            y = _softmax_attention(*piece, window=c["window"])
            out[:, b, group * h:group * (h + 4)] = y.detach()
            for t, n, gr in zip(grads, (group, 1, 1), torch.autograd.grad(y, piece, gout[:, b, group * h:group * (h + 4)])):
                t[:, b, n * h:n * (h + 4)] = gr
    return [out.view(c["seq"], c["batch"], -1)] + _grads([q, k, v], [qkv], grads)


def _exact_decode(s, c):
    q, k, v = (s[n].double() for n in ("q", "k", "v"))
    return torch.stack([_softmax_attention(q[b], k[b], v[b]) for b in range(c["batch"])])


def _exact_mlp(s, c):
    leaves = [_double(s[n]) for n in ("x", "w1", "b1", "w2", "b2", "residual")]
    x, w1, b1, w2, b2, r = leaves
    y = F.linear(F.gelu(F.linear(x, w1, b1)), w2, b2) + r
    return [y.detach()] + _grads(y, leaves, s["gout"].double())


def _exact_gated_mlp_decode(s, c):
    value, gate = F.linear(s["x"].double(), s["w1"].double()).chunk(2, -1)
    return F.linear(value * F.silu(gate), s["w2"].double())


def _exact_norm(s, c):
    x, p = _double(s["x"]), [_double(t) for t in s["params"]]
    if c["form"] == "rms":
        ys = [x, p[0] * x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5)]
    else:
        ys = [x] + [F.layer_norm(x, x.shape[-1:], p[i], p[i + 1], 1e-5) for i in range(0, len(p), 2)]
    return [y.detach() for y in ys[1:]] + _grads(ys, [x] + p, [t.double() for t in s["gouts"]])


def _exact_head(s, c):
    x, w = _double(s["x"]), _double(s["w"])
    loss = F.cross_entropy(F.linear(x, w), s["labels"], reduction="none")
    return [loss.detach()] + _grads(loss, [x, w], s["gout"].double())


def _exact_moe(s, c):
    x, gates, w1, w2 = (_double(s[n]) for n in ("x", "weights", "w1", "w2"))
    f, y = c["ffn"], torch.zeros_like(x)
    for e in range(c["experts"]):
        token, slot = torch.nonzero(s["indices"] == e, as_tuple=True)
        h = F.gelu(F.linear(x[token], w1[e * f:(e + 1) * f])) @ w2[e * f:(e + 1) * f]
        y = y.index_add(0, token, h * gates[token, slot][:, None])
    return [y.detach()] + _grads(y, [x, gates, w1, w2], s["gout"].double())


def _exact_mamba(s, c):
    v = {n: _double(s[n]) for n in MAMBA_LEAVES}
    u = F.conv1d(v["x"].transpose(1, 2), v["conv_w"].unsqueeze(1), v["conv_b"], padding=3, groups=c["inner"])
    u = F.silu(u[..., :c["seq"]]).transpose(1, 2)
    dt = F.softplus(v["dt"] + v["dt_bias"])
    h, ys = u.new_zeros(c["batch"], c["inner"], 16), []
    # unbind once: indexing each step would make its backward write a whole zero tensor per step
    for ut, dtt, bt, ct in zip(u.unbind(1), dt.unbind(1), v["B"].unbind(1), v["C"].unbind(1)):
        h = torch.exp(dtt[..., None] * v["A"]) * h + (dtt * ut)[..., None] * bt[:, None]
        ys.append((h * ct[:, None]).sum(-1))
    y = (torch.stack(ys, 1) + v["D"] * u) * F.silu(v["z"])
    return [y.detach()] + _grads(y, [v[n] for n in MAMBA_LEAVES], s["gout"].double())


def _exact_wkv(s, c):
    leaves = [_double(s[n]) for n in ("r", "k", "v", "w", "u")]
    b, T, H, N = c["batch"], c["seq"], c["heads"], c["head_size"]
    ys, grads = [], [torch.zeros_like(t) for t in leaves]
    for h in range(0, H, 4):                        # four heads at a time: the states of every step fit in memory
        n = min(4, H - h)
        part = [t.detach()[..., h * N:(h + n) * N].reshape(b, T, n, N).requires_grad_() for t in leaves[:4]]
        u = leaves[4].detach()[h:h + n].requires_grad_()
        S, rows = u.new_zeros(b, n, N, N), []
        for r, k, v, w in zip(*(t.unbind(1) for t in part)):
            kv = k[..., :, None] * v[..., None, :]
            rows.append((r[..., None] * (u[..., None] * kv + S)).sum(-2))
            S = torch.exp(-torch.exp(w))[..., None] * S + kv
        y = torch.stack(rows, 1)
        ys.append(y.detach().reshape(b, T, n * N))
        got = torch.autograd.grad(y, part + [u], s["gout"].double()[..., h * N:(h + n) * N].reshape(b, T, n, N))
        for t, gr in zip(grads[:4], got):
            t[..., h * N:(h + n) * N] = gr.reshape(b, T, n * N)
        grads[4][h:h + n] = got[4]
    return [torch.cat(ys, -1)] + grads


def _exact_adamw(s, c):
    a = ADAMW
    p, m, v, g = (s[n].double() for n in ("p", "m", "v", "g"))
    total = g.square().sum().sqrt()
    coef = torch.clamp(1.0 / (total + 1e-6), max=1.0)
    g *= coef
    m.mul_(a["beta1"]).add_(g, alpha=1 - a["beta1"])
    v.mul_(a["beta2"]).addcmul_(g, g, value=1 - a["beta2"])
    p.mul_(1 - a["lr"] * a["weight_decay"])
    p.addcdiv_(m, (v / (1 - a["beta2"] ** a["step"])).sqrt() + a["eps"], value=-a["lr"] / (1 - a["beta1"] ** a["step"]))
    return [p, m, v, p.to(s["lp"].dtype).double(), torch.stack([coef, total])]


def _exact_generate(s, c):
    w = {n.split(".", 1)[1]: t.double() for n, t in s["model"].state_dict().items() if t.is_floating_point()}
    width, heads, n = c["hidden"], c["heads"], s["tokens"].shape[1]
    dim = width // heads
    rot = dim // 4
    inv = 1.0 / (10000.0 ** (torch.arange(0, rot, 2, device="cuda", dtype=torch.float64) / rot))
    angle = torch.outer(torch.arange(n, device="cuda", dtype=torch.float64), inv)
    ln = lambda t, name: F.layer_norm(t, (width,), w[name + ".weight"], w[name + ".bias"], 1e-5)
    lin = lambda t, name: F.linear(t, w[name + ".weight"], w[name + ".bias"])
    x = w["0.word_embeddings.weight"][s["tokens"].t()]                          # [s, b, h]
    for i in range(c["layers"]):
        at = "%d." % (i + 2)
        q, k, v = _split_heads(lin(ln(x, at + "input_layernorm"), at + "attention.query_key_value"), heads, heads, dim)
        q, k = (_rotate(t, angle.cos(), angle.sin(), rot) for t in (q, k))
        ctx = torch.stack([_softmax_attention(q[:, b], k[:, b], v[:, b]) for b in range(c["batch"])], 1)
        mid = F.gelu(lin(ln(x, at + "post_attention_layernorm"), at + "mlp.linear1"), approximate="tanh")
        x = x + lin(ctx.reshape(n, c["batch"], width), at + "attention.dense") + lin(mid, at + "mlp.linear2")
    last = c["layers"] + 3
    logits = F.linear(ln(x, "%d.norm" % last), w["%d.final_linear.weight" % (last + 1)])
    return [logits[i] for i in range(c["prompt"] - 1, n)]

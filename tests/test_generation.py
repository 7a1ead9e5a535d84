"""Text generation on CPU: sampling filters, stop sequences, and KV-cache decoding == full recompute."""
import pytest
import torch

from common import tiny_config


def _model(**over):
    from gpt_neox_b200 import parallel as mpu
    from gpt_neox_b200 import training
    from gpt_neox_b200.config import NeoXArgs
    from gpt_neox_b200.initialize import initialize_megatron
    cfg = tiny_config(use_cpu_initialization=True, attention_config=[[["global"], 2]], **over)
    a = NeoXArgs.from_dict(cfg)
    a.configure_distributed_args()
    a.build_tokenizer()
    mpu.destroy_model_parallel()
    initialize_megatron(a)
    m = training.get_model(a, use_cache=True)
    return a, m


def test_filter_logits_topk_topp():
    from gpt_neox_b200.text_generation_utils import filter_logits
    logits = torch.tensor([[1.0, 2.0, 3.0, 4.0], [4.0, 3.0, 2.0, 1.0]])
    out = filter_logits(logits.clone(), top_k=2)
    assert torch.isinf(out[0, :2]).all() and torch.isfinite(out[0, 2:]).all()
    assert torch.isinf(out[1, 2:]).all() and torch.isfinite(out[1, :2]).all()
    p = torch.tensor([[0.5, 0.3, 0.15, 0.05]]).log()
    out = filter_logits(p.clone(), top_p=0.7)
    assert torch.isfinite(out[0, :2]).all() and torch.isinf(out[0, 2:]).all()


def test_pad_batch_and_stop_tokens():
    from gpt_neox_b200.text_generation_utils import pad_batch, stop_tokens_in_completion
    toks, lens = pad_batch([[1, 2, 3], [4]], pad_id=0, pad_len=5)
    assert toks == [[1, 2, 3, 0, 0], [4, 0, 0, 0, 0]] and lens == [3, 1]
    with pytest.raises(ValueError):
        pad_batch([[1] * 6], pad_id=0, pad_len=5)
    ctx = torch.tensor([[5, 6, 7, 8, 0]])
    assert stop_tokens_in_completion([torch.tensor([7, 8])], ctx, 0, 3)
    assert not stop_tokens_in_completion([torch.tensor([6, 8])], ctx, 0, 3)


@pytest.mark.parametrize("over", [dict(), dict(pos_emb="learned"), dict(gpt_j_residual=False, num_kv_heads=2),
                                  dict(pos_emb="sinusoidal"), dict(pos_emb="alibi"), dict(sliding_window_width=4),
                                  dict(pos_emb="rpe", rpe_num_buckets=8, rpe_max_distance=16)])
def test_kv_cache_decoding_matches_recompute(over):
    from gpt_neox_b200.text_generation_utils import stream_tokens
    a, m = _model(**over)
    prompts = [[5, 9, 11, 3], [7, 2]]
    outs = []
    for recompute in (True, False):
        m.inference_mode(use_cache=not recompute)
        m.clear_cache()
        last = None
        for last in stream_tokens(a, m, prompts, maximum_tokens=6, recompute=recompute, eos_token_id=10 ** 6):
            pass
        outs.append(last[0][:, :10].clone())
    assert torch.equal(outs[0], outs[1]), (outs[0], outs[1])
    assert torch.equal(outs[0][0, :4], torch.tensor([5, 9, 11, 3]))


def test_generate_samples_from_prompt_returns_records():
    from gpt_neox_b200.text_generation_utils import generate_samples_from_prompt
    a, m = _model()
    m.inference_mode(use_cache=True)

    class _Tok:
        eod = 0

        def tokenize(self, s):
            return [min(ord(c), 99) for c in s] or [0]

        def detokenize(self, ids):
            return "".join(chr(33 + (i % 60)) for i in ids)
    a.tokenizer = _Tok()
    m.clear_cache()
    out = generate_samples_from_prompt(a, m, ["ab", ""], maximum_tokens=4, temperature=0.8, top_k=5)
    assert len(out) == 2 and all(set(r) >= {"context", "text", "length", "finished", "message"} for r in out)
    assert out[0]["length"] <= 4


def test_eval_adapter_loglikelihood_matches_direct_computation():
    from gpt_neox_b200.eval_tasks import EvalHarnessAdapter
    a, m = _model()

    class _Tok:
        eod = 0
        eod_id = 0

        def tokenize(self, s):
            return [3 + (ord(c) % 90) for c in s]

        def detokenize(self, ids):
            return "".join(chr(40 + (i % 50)) for i in ids)
    a.tokenizer = _Tok()
    ad = EvalHarnessAdapter(m, None, a, batch_size=2)
    reqs = [("hello wor", "ld"), ("", "abc"), ("a much longer context string", " x")]
    got = ad.loglikelihood(reqs)
    m.inference_mode(use_cache=False)
    for (ctx, cont), (ll, greedy) in zip(reqs, got):
        c = [0] if ctx == "" else a.tokenizer.tokenize(ctx)
        t = a.tokenizer.tokenize(cont)
        full = torch.tensor([c + t])
        pos = torch.arange(full.shape[1] - 1)[None]
        from gpt_neox_b200.utils.common import get_attn_mask
        with torch.no_grad():
            logits = m((full[:, :-1], pos, get_attn_mask(full.shape[1] - 1, "cpu", None)))
        lp = torch.log_softmax(logits.float(), -1)[0, -len(t):]
        want = lp.gather(1, torch.tensor(t)[:, None]).sum().item()
        assert ll == pytest.approx(want, rel=1e-4, abs=1e-4)
        assert greedy == bool((lp.argmax(-1) == torch.tensor(t)).all())
    assert len(ad.loglikelihood_rolling([("some document text " * 5,)])) == 1


def test_recurrent_stacks_decode_by_recompute():
    """Mamba / RWKV blocks keep no state between calls, so asking for cached decoding must still run the whole
    prefix: same tokens as an explicit recompute."""
    from gpt_neox_b200 import parallel as mpu
    from gpt_neox_b200 import training
    from gpt_neox_b200.config import NeoXArgs
    from gpt_neox_b200.initialize import initialize_megatron
    from gpt_neox_b200.text_generation_utils import stream_tokens
    a = NeoXArgs.from_dict(tiny_config(use_cpu_initialization=True, attention_config=[[["rwkv"], 2]],
                                       num_attention_heads=1))
    a.configure_distributed_args()
    a.build_tokenizer()
    mpu.destroy_model_parallel()
    initialize_megatron(a)
    m = training.get_model(a, use_cache=True)
    outs = []
    for recompute in (True, False):
        m.inference_mode(use_cache=not recompute)
        m.clear_cache()
        last = None
        for last in stream_tokens(a, m, [[5, 9, 11, 3], [7, 2]], maximum_tokens=6, recompute=recompute,
                                  eos_token_id=10 ** 6):
            pass
        outs.append(last[0][:, :10].clone())
    assert torch.equal(outs[0], outs[1])


def test_sinusoidal_table_rows_follow_position_ids():
    from gpt_neox_b200.models.positional_embeddings import SinusoidalPositionalEmbedding
    e = SinusoidalPositionalEmbedding(8, precision=torch.float32)
    full = e(torch.arange(6)[None])                     # [1, 6, 8]
    one = e(torch.tensor([[4]]))                        # the row a cached decoding step asks for
    torch.testing.assert_close(one[0, 0], full[0, 4])


def _generate(rank, world, cfg, recompute):
    from gpt_neox_b200 import parallel as mpu
    from gpt_neox_b200 import training
    from gpt_neox_b200.config import NeoXArgs
    from gpt_neox_b200.initialize import initialize_megatron
    from gpt_neox_b200.text_generation_utils import stream_tokens
    torch.set_num_threads(1)
    mpu.destroy_model_parallel()
    a = NeoXArgs.from_dict(dict(cfg, global_num_gpus=world))
    a.configure_distributed_args()
    a.build_tokenizer()
    initialize_megatron(a)
    model, _, _, _ = training.setup_model_and_optimizer(neox_args=a, use_cache=True)
    model.eval()
    net = getattr(model, "module", model)
    net.inference_mode(use_cache=not recompute)
    net.clear_cache()
    last = None
    for last in stream_tokens(a, model, [[5, 9, 11, 3], [7, 2]], maximum_tokens=6, recompute=recompute,
                              eos_token_id=10 ** 6):
        pass
    return last[0][:, :10].tolist()


def test_greedy_generation_is_the_same_under_tensor_and_pipeline_parallelism():
    """Same master weights (CPU initialisation) and the same padded vocabulary: one rank, two tensor-parallel ranks
    and two pipeline stages (whose engine re-runs the prefix instead of using the KV cache) emit the same tokens."""
    from common import run_distributed
    base = dict(use_cpu_initialization=True, make_vocab_size_divisible_by=64, attention_config=[[["global"], 2]],
                optimizer=None, no_load_optim=True)
    one = run_distributed(_generate, 1, tiny_config(**base), False)[0]
    tp2 = run_distributed(_generate, 2, tiny_config(model_parallel_size=2, **base), False)[0]
    pp2 = run_distributed(_generate, 2, tiny_config(pipe_parallel_size=2, **base), False)[0]
    assert one[0][:4] == [5, 9, 11, 3] and one[1][:2] == [7, 2]
    assert tp2 == one and pp2 == one


def _loglikelihoods(rank, world, cfg, reqs):
    from gpt_neox_b200 import parallel as mpu
    from gpt_neox_b200 import training
    from gpt_neox_b200.config import NeoXArgs
    from gpt_neox_b200.eval_tasks.eval_adapter import EvalHarnessAdapter
    from gpt_neox_b200.initialize import initialize_megatron
    from gpt_neox_b200.text_generation_utils import forward_model
    torch.set_num_threads(1)
    mpu.destroy_model_parallel()
    a = NeoXArgs.from_dict(dict(cfg, global_num_gpus=world))
    a.configure_distributed_args()
    a.build_tokenizer()
    initialize_megatron(a)
    model, _, _, _ = training.setup_model_and_optimizer(neox_args=a, use_cache=False)
    ad = EvalHarnessAdapter(model, forward_model, a, batch_size=2)
    return [(round(float(l), 3), bool(g)) for l, g in ad.loglikelihood(reqs)]


def test_eval_adapter_scores_are_layout_independent():
    """Requests of different lengths (so the batches have different shapes, which the pipeline stages must
    re-announce to each other): one rank, two pipeline stages and two tensor-parallel ranks give the same scores."""
    from common import run_distributed
    base = dict(use_cpu_initialization=True, make_vocab_size_divisible_by=64, attention_config=[[["global"], 2]],
                optimizer=None, no_load_optim=True, tokenizer_type="CharLevelTokenizer", dataset_impl="gpt2")
    reqs = [("hello wor", "ld"), ("", "abc"), ("some longer context here", " and a continuation"), ("x", "y")]
    one = run_distributed(_loglikelihoods, 1, tiny_config(**base), reqs)[0]
    pp2 = run_distributed(_loglikelihoods, 2, tiny_config(pipe_parallel_size=2, **base), reqs)[0]
    tp2 = run_distributed(_loglikelihoods, 2, tiny_config(model_parallel_size=2, **base), reqs)[0]
    assert len(one) == 4 and all(l < 0 for l, _ in one)
    assert pp2 == one and tp2 == one


def _run_local_eval(rank, world, cfg, task_dir):
    import os
    from gpt_neox_b200 import parallel as mpu
    from gpt_neox_b200 import training
    from gpt_neox_b200.config import NeoXArgs
    from gpt_neox_b200.eval_tasks import run_eval_harness
    from gpt_neox_b200.initialize import initialize_megatron
    from gpt_neox_b200.text_generation_utils import forward_model
    torch.set_num_threads(1)
    os.environ["NEOX_EVAL_TASK_DIR"] = task_dir
    mpu.destroy_model_parallel()
    a = NeoXArgs.from_dict(dict(cfg, global_num_gpus=world))
    a.configure_distributed_args()
    a.build_tokenizer()
    initialize_megatron(a)
    model, _, _, _ = training.setup_model_and_optimizer(neox_args=a, use_cache=False)
    return run_eval_harness(model, forward_model, a, batch_size=2, eval_tasks=["choice", "lastword", "wiki"])


def test_eval_harness_runs_end_to_end_on_local_task_files(tmp_path):
    """``run_eval_harness`` (what ``eval.py`` and the in-training evaluation call) on three task files of the three
    request types, without the lm_eval package: metrics of the harness's shape, identical on one rank and on two
    pipeline stages, and a task with no local file asks for lm_eval by name."""
    import json
    from common import run_distributed
    rows = [{"query": f"the number after {i} is", "choices": [f" {i + 1}", f" {i + 2}", " zero"], "gold": i % 3}
            for i in range(6)]
    (tmp_path / "choice.jsonl").write_text("\n".join(json.dumps(r) for r in rows))
    (tmp_path / "lastword.jsonl").write_text("\n".join(json.dumps({"text": f"row {i} ends with the word stop"})
                                                       for i in range(4)))
    (tmp_path / "wiki.jsonl").write_text(json.dumps({"document": "a short document of a few words " * 3}))
    base = dict(use_cpu_initialization=True, make_vocab_size_divisible_by=64, attention_config=[[["global"], 2]],
                optimizer=None, no_load_optim=True, tokenizer_type="CharLevelTokenizer", dataset_impl="gpt2")
    one = run_distributed(_run_local_eval, 1, tiny_config(**base), str(tmp_path))[0]
    res = one["results"]
    assert set(res) == {"choice", "lastword", "wiki"}
    assert 0.0 <= res["choice"]["acc"] <= 1.0 and 0.0 <= res["choice"]["acc_norm"] <= 1.0
    assert res["lastword"]["ppl"] > 1.0 and 0.0 <= res["lastword"]["acc"] <= 1.0
    assert res["wiki"]["byte_perplexity"] > 1.0 and res["wiki"]["bits_per_byte"] > 0.0
    pp2 = run_distributed(_run_local_eval, 2, tiny_config(pipe_parallel_size=2, **base), str(tmp_path))[0]
    for task in res:
        for metric, v in res[task].items():
            assert pp2["results"][task][metric] == pytest.approx(v, rel=1e-4), (task, metric)
    from gpt_neox_b200.eval_tasks import local_tasks
    assert local_tasks.resolve("hellaswag") is None


def test_growing_cache_keeps_every_continuation_apart():
    """The in-place growth of a layer's cache against plain concatenation: steps, a second continuation of an older
    cache, another layer's cache, a caller's own tensor, and growth past the buffer's room."""
    import torch
    from gpt_neox_b200.models import kv_cache

    class Layer:
        pass

    torch.manual_seed(0)
    layer, other = Layer(), Layer()

    def step(owner, past, rows):
        new = torch.randn(2, rows, 2, 3, 4)
        want = new if past is None else torch.cat((torch.stack((past[0], past[1])), new), dim=1)
        got = kv_cache.extend(owner, past, rows, new[0])
        got[:, got.shape[1] - rows:].copy_(new)
        assert torch.equal(got, want)
        return got, want.clone()

    seen = [step(layer, None, 5)]
    for rows in (1, 1, 3, 1):
        seen.append(step(layer, seen[-1][0], rows))
    assert seen[1][0].data_ptr() == seen[4][0].data_ptr()               # grown in place
    fork = step(layer, seen[2][0], 2)                                   # an older cache: a copy
    again = step(layer, seen[4][0], 1)                                  # no longer the last one returned: a copy
    cross = step(other, again[0], 1)                                    # another layer's
    own = step(layer, torch.randn(2, 7, 2, 3, 4), 1)                    # a caller's tensor
    pair = step(layer, (own[0][0], own[0][1]), 1)                       # (k, v) instead of one tensor
    big = step(layer, pair[0], 2000)                                    # more than the buffer has room for
    last = step(layer, big[0], 1)
    for got, want in seen + [fork, again, cross, own, pair, big, last]:
        assert torch.equal(got, want)
    empty = step(layer, torch.empty(2, 0, 2, 3, 4), 4)
    assert empty[0].shape[1] == 4


@pytest.mark.gpu
@pytest.mark.parametrize("over", [dict(), dict(num_kv_heads=2, rotary_pct=1.0), dict(pos_emb="alibi"),
                                  dict(gpt_j_residual=False, norm="rmsnorm", rotary_pct=0.5)])
def test_cached_steps_match_the_whole_prefix_on_the_gpu(over):
    """Prompt + single-token steps through the growing cache (in place, no autograd, fused rotary write) against one
    uncached pass over the whole sequence."""
    import torch
    from common import tiny_config
    from test_model_gpu import _build
    base = dict(num_layers=2, hidden_size=256, num_attention_heads=4, seq_length=512, max_position_embeddings=512,
                synthetic_vocab_size=1000, attention_config=[[["flash"], 2]], distributed_backend="nccl",
                precision="bfloat16", pipe_parallel_size=0)
    base.update(over)
    _, model = _build(tiny_config(**base))
    model.eval()
    tokens = torch.randint(0, 1000, (2, 300), device="cuda")
    pos = torch.arange(300, device="cuda")[None].expand(2, -1)
    with torch.no_grad():
        full = model((tokens, pos, None)).float()
        model.inference_mode(use_cache=True)
        model.clear_cache()
        got, at = [], 0
        for n in [20, 1, 1, 7] + [1] * 5 + [256, 1, 1]:          # the 256-row step outgrows the first buffer
            got.append(model((tokens[:, at:at + n].contiguous(), pos[:, at:at + n].contiguous(), None)).float())
            at += n
    got = torch.cat(got, dim=1)
    err = (got - full[:, :at]).norm() / full[:, :at].norm()
    assert err < 2e-2, err.item()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["bfloat16", "fp16"])
@pytest.mark.parametrize("over", [dict(), dict(num_kv_heads=2, rotary_pct=1.0), dict(bias_gelu_fusion=True),
                                  dict(sliding_window_width=16), dict(use_bias_in_attn_linear=False,
                                                                      use_bias_in_mlp=False)])
def test_a_layer_in_one_call_gives_the_bits_of_the_op_by_op_path(over, precision, monkeypatch):
    """A hook on a submodule sends the layer down the op-by-op path; without it one native call launches the same
    kernels."""
    from test_model_gpu import _build
    base = dict(num_layers=2, hidden_size=256, num_attention_heads=4, seq_length=512, max_position_embeddings=512,
                synthetic_vocab_size=1000, attention_config=[[["flash"], 2]], distributed_backend="nccl",
                precision=precision, pipe_parallel_size=0)
    base.update(over)
    _, model = _build(tiny_config(**base))
    model.eval()
    model.inference_mode(use_cache=True)
    tokens = torch.randint(0, 1000, (3, 330), device="cuda")
    pos = torch.arange(330, device="cuda")[None].expand(3, -1)
    from gpt_neox_b200.models import transformer
    native, call = [], transformer.layer_infer
    monkeypatch.setattr(transformer, "layer_infer", lambda *a, **k: (native.append(1), call(*a, **k))[1])

    def steps():
        model.clear_cache()
        out, at = [], 0
        with torch.no_grad():
            for n in (40, 1, 1, 5, 1, 270, 1):
                out.append(model((tokens[:, at:at + n].contiguous(), pos[:, at:at + n].contiguous(), None)))
                at += n
        layers = [m for m in model.modules() if type(m).__name__.startswith("ParallelTransformerLayer")]
        return out + [l.layer_past.clone() for l in layers]

    one = steps()
    assert len(native) == 14                            # 2 layers x 7 steps
    mlps = [m for m in model.modules() if type(m).__name__ == "ParallelMLP"]
    calls = []
    handles = [m.register_forward_hook(lambda *a: calls.append(1)) for m in mlps]
    ops = steps()
    for h in handles:
        h.remove()
    assert len(native) == 14 and len(calls) == 14 and len(one) == len(ops)
    assert all(torch.equal(a, b) for a, b in zip(one, ops))


@pytest.mark.gpu
@pytest.mark.parametrize("hidden,heads", [(768, 12), (1024, 8)])
def test_products_in_one_launch_give_the_bits_of_two(hidden, heads, monkeypatch):
    """Few rows: query / key / value with the MLP's first product, and dense with its second one, in one launch each, with
    different numbers of splits (dense 2, down 8) - at both sides of every row count the kernel is built for, and of the
    128 from which they are launched by themselves: six launches a layer with both pairs, eight with none."""
    from test_model_gpu import _build
    from gpt_neox_b200.models import transformer
    from gpt_neox_b200.ops.gemm import LAUNCHES
    launches, call = [], transformer.layer_infer

    def counted(*a, **k):
        before = LAUNCHES["n"]
        out = call(*a, **k)
        launches.append(LAUNCHES["n"] - before)
        return out
    monkeypatch.setattr(transformer, "layer_infer", counted)
    _, model = _build(tiny_config(num_layers=1, hidden_size=hidden, num_attention_heads=heads, seq_length=512,
                                  max_position_embeddings=512, synthetic_vocab_size=1000, pipe_parallel_size=0,
                                  attention_config=[[["flash"], 1]], distributed_backend="nccl", precision="bfloat16"))
    model.inference_mode(use_cache=True)
    mlp = next(m for m in model.modules() if type(m).__name__ == "ParallelMLP")
    tokens = torch.randint(0, 1000, (1, 512), device="cuda")
    pos = torch.arange(512, device="cuda")[None]

    rows = (1, 15, 16, 17, 32, 33, 64, 65, 96, 128, 130)

    def steps():
        model.clear_cache()
        out, at = [], 0
        with torch.no_grad():
            for n in rows:
                out.append(model((tokens[:, at:at + n].contiguous(), pos[:, at:at + n].contiguous(), None)))
                at += n
                if at > 300:
                    model.clear_cache()
                    at = 0
        return out

    one = steps()
    # (128 rows of 768 -> 768 go to the other kernel, whose tiles are enough there)
    assert launches == [6] * 9 + [8 if hidden == 768 else 6, 8]
    handle = mlp.register_forward_hook(lambda *a: None)
    ops = steps()
    handle.remove()
    assert len(launches) == len(rows)                   # (the second run went op by op)
    assert all(torch.equal(a, b) for a, b in zip(one, ops)) and all(t.isfinite().all() for t in one)


@pytest.mark.gpu
@pytest.mark.parametrize("precision,x,branch,want", [("bfloat16", 1024.0, 3.0, 1032.0), ("fp16", 16384.0, 6.0, 16400.0)])
@pytest.mark.parametrize("hook", [False, True])
@pytest.mark.parametrize("rows", [1, 130, 300])
def test_a_generation_step_rounds_the_residual_stream_once(precision, x, branch, want, hook, rows):
    """Attention and MLP add less than half a unit in the last place of the residual stream each, and more than half
    together (all matrices zero, so that the branches are their last biases): with the sum rounded once the stream moves,
    with a rounding after each branch it does not.  One native call and op by op."""
    import torch
    from gpt_neox_b200.models.transformer import ParallelTransformerLayer
    from test_model_gpu import _build
    _, model = _build(tiny_config(num_layers=2, hidden_size=256, num_attention_heads=4, seq_length=512,
                                  max_position_embeddings=512, synthetic_vocab_size=1000, pipe_parallel_size=0,
                                  attention_config=[[["flash"], 2]], distributed_backend="nccl", precision=precision))
    model.inference_mode(use_cache=True)
    layer = next(m for m in model.modules() if isinstance(m, ParallelTransformerLayer))
    for n, p in layer.named_parameters():
        torch.nn.init.constant_(p, branch if n in ("attention.dense.bias", "mlp.linear2.bias") else 0.0)
    if hook:
        layer.mlp.register_forward_hook(lambda *a: None)
    t = torch.full((rows, 1, 256), x, device="cuda", dtype=next(layer.parameters()).dtype)
    with torch.no_grad():
        out = ParallelTransformerLayer.forward(layer, t)
    assert (out == want).all()


@pytest.mark.gpu
def test_a_generation_step_leaves_the_projection_output_as_a_hook_saw_it():
    import torch
    from test_model_gpu import _build
    _, model = _build(tiny_config(num_layers=2, hidden_size=256, num_attention_heads=4, seq_length=512,
                                  max_position_embeddings=512, synthetic_vocab_size=1000, pipe_parallel_size=0,
                                  attention_config=[[["flash"], 2]], distributed_backend="nccl", precision="bfloat16"))
    model.inference_mode(use_cache=True)
    kept = []
    for m in model.modules():
        if type(m).__name__ == "ParallelSelfAttention":
            m.query_key_value.register_forward_hook(lambda m, i, o: kept.append((o[0], o[0].clone())))
    tokens = torch.randint(0, 1000, (2, 20), device="cuda")
    pos = torch.arange(20, device="cuda")[None].expand(2, -1)
    with torch.no_grad():
        for at in (slice(0, 19), slice(19, 20)):
            model((tokens[:, at].contiguous(), pos[:, at].contiguous(), None))
    assert len(kept) == 4 and all(torch.equal(a, b) for a, b in kept)


@pytest.mark.gpu
def test_hooks_see_the_modules_own_outputs_while_generating():
    """Hooks on the attention, its output projection and the MLP fire, and see what the modules return when called alone:
    the branch without the residual stream, and the bias beside it."""
    import torch
    from test_model_gpu import _build
    _, model = _build(tiny_config(num_layers=2, hidden_size=256, num_attention_heads=4, seq_length=512,
                                  max_position_embeddings=512, synthetic_vocab_size=1000, pipe_parallel_size=0,
                                  attention_config=[[["flash"], 2]], distributed_backend="nccl", precision="bfloat16"))
    for n, p in model.named_parameters():
        if n.endswith("bias"):
            torch.nn.init.normal_(p, std=0.3)
    model.inference_mode(use_cache=True)
    tokens = torch.randint(0, 1000, (2, 20), device="cuda")
    pos = torch.arange(20, device="cuda")[None].expand(2, -1)
    run = lambda: [model((tokens[:, a].contiguous(), pos[:, a].contiguous(), None)) for a in (slice(0, 19), slice(19, 20))]
    with torch.no_grad():
        plain = run()
        seen = []
        layers = [m for m in model.modules() if type(m).__name__.startswith("ParallelTransformerLayer")]
        handles = [m.register_forward_hook(lambda m, i, o: seen.append((m, i, o)))
                   for l in layers for m in (l.attention, l.attention.dense, l.mlp)]
        model.clear_cache()
        hooked = run()
        for h in handles:
            h.remove()
        assert len(seen) == 2 * 2 * 3
        for m, i, o in seen:
            name = type(m).__name__
            assert o[1] is {"ParallelSelfAttention": lambda: m.dense.bias, "RowParallelLinear": lambda: m.bias,
                            "ParallelMLP": lambda: m.linear2.bias}[name]()
            if name != "ParallelSelfAttention":
                assert len(i) == 1 and torch.equal(m(i[0])[0], o[0])
    assert all(torch.equal(a, b) for a, b in zip(plain, hooked))


@pytest.mark.gpu
@pytest.mark.parametrize("name,where", [(n, w) for n in ("attention", "attention.query_key_value", "attention.dense", "mlp")
                                        for w in ("instance", "class")]
                         + [(n, "parametrized") for n in ("input_layernorm", "attention.dense", "mlp.linear1")])
def test_a_replaced_forward_is_called_while_generating(name, where, monkeypatch):
    """Modules that generation calls: a forward replaced on one instance or on the class runs, and a weight that is computed
    on access (a parametrization, whose value lives as long as the access) is used."""
    import torch
    from torch.nn.utils import parametrize
    from test_model_gpu import _build
    _, model = _build(tiny_config(num_layers=2, hidden_size=256, num_attention_heads=4, seq_length=512,
                                  max_position_embeddings=512, synthetic_vocab_size=1000, pipe_parallel_size=0,
                                  attention_config=[[["flash"], 2]], distributed_backend="nccl", precision="bfloat16"))
    model.inference_mode(use_cache=True)
    layers = [m for m in model.modules() if type(m).__name__.startswith("ParallelTransformerLayer")]
    target = layers[0].get_submodule(name)
    tokens = torch.randint(0, 1000, (2, 20), device="cuda")
    pos = torch.arange(20, device="cuda")[None].expand(2, -1)
    calls = []
    with torch.no_grad():
        want = model((tokens, pos, None))
        if where == "parametrized":
            class Count(torch.nn.Module):
                def forward(self, w):
                    calls.append(target)
                    return w * 1
            parametrize.register_parametrization(target, "weight", Count())
            calls.clear()
        else:
            owner = target if where == "instance" else type(target)
            old = owner.forward
            monkeypatch.setattr(owner, "forward", lambda *a, **k: (calls.append(a[0] if where == "class" else target), old(*a, **k))[1],
                                raising=False)
        model.clear_cache()
        got = model((tokens, pos, None))
    assert any(c is target for c in calls) and torch.equal(got, want)


@pytest.mark.parametrize("past,shape", [((2, 3, 1, 2, 4), (4, 2, 4)), ((2, 3, 4, 1, 4), (4, 2, 4)), ((2, 3, 4, 2, 1), (4, 2, 4)),
                                        ((2, 3, 4, 2, 8), (4, 2, 4)), ((2, 3, 2, 4), (4, 2, 4))])
def test_a_cache_of_another_shape_is_refused(past, shape):
    """As concatenating it was: no broadcast of a stale cache over this step's batch or heads."""
    import torch
    from gpt_neox_b200.models import kv_cache

    class Layer:
        pass
    for p in (torch.zeros(past), tuple(torch.zeros(past))):
        with pytest.raises(RuntimeError):
            kv_cache.extend(Layer(), p, 1, torch.zeros((1,) + shape))
    with pytest.raises(RuntimeError):                       # keys and values of different lengths
        kv_cache.extend(Layer(), (torch.zeros((3,) + shape), torch.zeros((2,) + shape)), 1, torch.zeros((1,) + shape))
    layer = Layer()                                         # and the layer's own last cache, after the batch has changed
    last = kv_cache.extend(layer, None, 2, torch.zeros((1,) + shape))
    with pytest.raises(RuntimeError):
        kv_cache.extend(layer, last, 1, torch.zeros((1, 1) + shape[1:]))


def test_a_cache_of_inference_mode_is_continued_outside_it():
    import torch
    from gpt_neox_b200.models import kv_cache

    class Layer:
        pass
    torch.manual_seed(1)
    layer, rows = Layer(), [torch.randn(2, n, 2, 3, 4) for n in (3, 1, 1, 1)]

    def step(past, new):
        got = kv_cache.extend(layer, past, new.shape[1], new[0])
        got[:, got.shape[1] - new.shape[1]:].copy_(new)
        return got
    with torch.inference_mode():
        first = step(None, rows[0])
    with torch.no_grad():
        second = step(first, rows[1])
    with torch.inference_mode():
        third = step(second, rows[2])
    with torch.no_grad():
        last = step(third, rows[3])
    assert torch.equal(last, torch.cat(rows, 1)) and torch.equal(first, rows[0]) and torch.equal(third, torch.cat(rows[:3], 1))


@pytest.mark.gpu
def test_a_captured_step_does_not_share_its_cache_with_what_follows():
    """A step captured in a graph on the stream of the eager ones: an eager continuation of its cache, and the cache it started from, keep their rows when
    the graph is replayed on other inputs."""
    import torch
    from gpt_neox_b200.models import kv_cache

    class Layer:
        pass
    layer, like = Layer(), torch.zeros(1, 2, 3, 8, device="cuda")

    def step(past, value):
        got = kv_cache.extend(layer, past, 1, like)
        got[:, got.shape[1] - 1:].copy_(value)
        return got
    value = torch.full((), 2.0, device="cuda")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        first = step(None, torch.ones((), device="cuda"))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            captured = step(first, value)
        graph.replay()
        after = step(captured, torch.full((), 3.0, device="cuda"))
        branch = step(first, torch.full((), 4.0, device="cuda"))
        value.fill_(9.0)
        graph.replay()
    torch.cuda.synchronize()
    for got, want in ((first, [1]), (captured, [1, 9]), (after, [1, 2, 3]), (branch, [1, 4])):
        assert got[0, :, 0, 0, 0].tolist() == want and got.shape[1] == len(want)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["query_key_value", "dense"])
def test_a_module_in_place_of_a_linear_is_called_while_generating(name):
    """An adapter that wraps a projection has none of the parallel linears' attributes."""
    import torch
    from test_model_gpu import _build
    _, model = _build(tiny_config(num_layers=2, hidden_size=256, num_attention_heads=4, seq_length=512,
                                  max_position_embeddings=512, synthetic_vocab_size=1000, pipe_parallel_size=0,
                                  attention_config=[[["flash"], 2]], distributed_backend="nccl", precision="bfloat16"))
    model.inference_mode(use_cache=True)

    class Adapter(torch.nn.Module):
        def __init__(self, inner):
            super().__init__()
            self.inner = inner

        def forward(self, x):
            calls.append(1)
            return self.inner(x)
    calls = []
    tokens = torch.randint(0, 1000, (2, 20), device="cuda")
    pos = torch.arange(20, device="cuda")[None].expand(2, -1)
    layer = next(m for m in model.modules() if type(m).__name__.startswith("ParallelTransformerLayer"))
    with torch.no_grad():
        want = model((tokens, pos, None))
        setattr(layer.attention, name, Adapter(getattr(layer.attention, name)))
        model.clear_cache()
        got = model((tokens, pos, None))
    assert calls == [1] and torch.equal(got, want)

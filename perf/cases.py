"""The work that a user of interattn_b200 has it do, as measurable cases.

Four kinds of call, through the public entry points:

* ``step``       one decode-attention layer-step of a paged batch: ``ops.DecodeAttention.step`` (or ``step_host`` when
                 the query and the output live in host memory).  Block selection, paged attention, merge.
* ``reference``  the same layer-step under the reference project's own name and calling convention, one sequence over a
                 contiguous cache: ``reference_api._condition_block_decode_output_fused_triton``.
* ``summaries``  the block summaries of freshly prefilled prompts: ``ops.build_summaries`` (paged batch) or
                 ``reference_api._build_prompt_blocks`` (one sequence, contiguous cache).
* ``model``      a whole Llama decode step over a static cache, ``llama_step.FusedLlamaStep.step``, eager or captured
                 into a CUDA graph, on a few layers of the full-size architecture.

Data: seeded N(0, 1) queries, keys and values, the key channels scaled by a log-normal(0, 0.5) factor (key outliers);
page tables are random permutations of the pool; weights are random.
"""

import math
import types

import torch

from interattn_b200 import llama_decode, llama_step, ops, reference_api

PAGE = 16
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}

# What a step case is when nothing else is said: the Llama-3-8B attention geometry, top-k routing, selected blocks only.
STEP = {"kind": "step", "dtype": "bf16", "q_heads": 32, "kv_heads": 8, "head_dim": 128, "block": 64, "suffix": 0,
        "rule": "top_k", "rep_mode": "sparse_only", "k_bar": "f32", "host": False}
MODEL = {"kind": "model", "layers": 4, "block": 64, "top_k": 64}


def listed():
    return [
        # The smallest call: the fp32 configuration that also runs on a CPU (two short sequences).  All latency.
        dict(STEP, name="step_f32_small", dtype="f32", batch=2, q_heads=8, kv_heads=2, head_dim=64, lo=1024, hi=1024, k=4),
        # Small heads (head_dim 64), a ragged batch of short prompts with a few generated tokens, hybrid attention.
        dict(STEP, name="step_d64_ragged", batch=8, head_dim=64, lo=500, hi=8000, k=16, suffix=37, rep_mode="hybrid"),
        # The headline: Llama-3-8B attention geometry, batch 16 at 32k context, top-64 of 512 blocks.
        dict(STEP, name="step_8b_32k", batch=16, lo=32768, hi=32768, k=64),
        # The same call by a program that keeps query and output in pinned host memory.
        dict(STEP, name="step_8b_32k_host", batch=16, lo=32768, hi=32768, k=64, host=True),
        # A layer of the batch-32 decode half way through its generation, in the reference's own (hybrid) mode.
        dict(STEP, name="step_8b_8k_hybrid", batch=32, lo=8192, hi=8192, k=64, suffix=128, rep_mode="hybrid"),
        # Few very long sequences: 2048 blocks each, little to attend, much to score.
        dict(STEP, name="step_8b_128k", batch=4, lo=131072, hi=131072, k=32),
        # Llama-3-70B attention geometry, a large ragged batch from 1k to 64k tokens.
        dict(STEP, name="step_70b_ragged", batch=64, q_heads=64, lo=1024, hi=65536, k=48),
        # What the reference's generation loop calls per layer and token: one sequence, epsilon rule, hybrid.
        {"kind": "reference", "name": "reference_eps_8k", "dtype": "bf16", "q_heads": 32, "kv_heads": 8, "head_dim": 128,
         "block": 64, "tokens": 8192, "suffix": 33, "share": 0.125},
        # End of prefill of the headline batch: 2 GiB of keys and values summarised.
        {"kind": "summaries", "name": "summaries_8b_32k", "api": "paged", "dtype": "bf16", "kv_heads": 8, "head_dim": 128,
         "block": 64, "batch": 16, "lo": 32768, "hi": 32768},
        # The same for one short prompt of odd length under the reference's name.
        {"kind": "summaries", "name": "summaries_odd_4099", "api": "reference", "dtype": "bf16", "kv_heads": 8,
         "head_dim": 128, "block": 64, "batch": 1, "lo": 4099, "hi": 4099},
        # Batched generation: four full-size layers, 32 sequences at 8192 tokens, the step captured into a CUDA graph.
        dict(MODEL, name="model_b32_8k", batch=32, tokens=8192, suffix=128, graph=True),
        # Interactive generation: one sequence at 7001 tokens, launched eagerly.
        dict(MODEL, name="model_b1_7k", batch=1, tokens=7001, suffix=40, graph=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["reference"] + ["summaries"] * 2 + ["model"])
    if kind == "reference":
        return {"kind": "reference", "dtype": "bf16", "q_heads": 32, "kv_heads": 8, "head_dim": 128, "block": 64,
                "tokens": _log_int(rng, 1000, 32768), "suffix": _log_int(rng, 1, 300),
                "share": rng.choice([0.0625, 0.125, 0.25])}
    if kind == "summaries":
        if rng.random() < 0.4:
            n = _log_int(rng, 500, 32768)
            return {"kind": "summaries", "api": "reference", "dtype": "bf16", "kv_heads": 8, "head_dim": 128, "block": 64,
                    "batch": 1, "lo": n, "hi": n}
        hi = _log_int(rng, 1000, 32768)
        return {"kind": "summaries", "api": "paged", "dtype": "bf16", "kv_heads": 8, "head_dim": rng.choice([64, 128, 128]),
                "block": rng.choice([32, 64, 64]), "batch": _log_int(rng, 1, 16), "lo": max(1, int(hi * rng.uniform(0.3, 1.0))),
                "hi": hi}
    if kind == "model":
        batch = _log_int(rng, 1, 32)
        return dict(MODEL, layers=rng.choice([2, 3, 4]), batch=batch, tokens=_log_int(rng, 1000, 8192),
                    suffix=_log_int(rng, 1, 200), graph=rng.random() < 0.5)
    shape = rng.choice(["f32", "d64", "d128", "d128", "d128", "d128"])
    c = dict(STEP, suffix=rng.choice([0, _log_int(rng, 1, 300)]), rep_mode=rng.choice(["sparse_only", "sparse_only", "hybrid"]))
    if shape == "f32":
        hi = _log_int(rng, 500, 8192)
        c.update(dtype="f32", batch=_log_int(rng, 1, 8), q_heads=rng.choice([8, 16]), kv_heads=2, head_dim=64, hi=hi,
                 lo=max(1, int(hi * rng.uniform(0.5, 1.0))), k=_log_int(rng, 2, 16))
        return c
    group = rng.choice([1, 4, 4, 4, 8])
    if shape == "d64":
        hi = _log_int(rng, 1000, 16384)
        c.update(batch=_log_int(rng, 1, 32), head_dim=64, q_heads=8 * group)
    else:
        hi = _log_int(rng, 1000, 131072)
        # the pool of a drawn case stays below that of the largest listed one
        c.update(batch=_log_int(rng, 1, max(1, min(64, 2000000 // hi))), q_heads=8 * rng.choice([4, 4, 8]),
                 k_bar=rng.choice(["f32", "f32", "bf16"]), host=rng.random() < 0.15)
    c.update(hi=hi, lo=max(1, int(hi * rng.uniform(0.05, 1.0))), k=_log_int(rng, 8, 64))
    if rng.random() < 0.2:
        c.update(rule="eps", k=0, share=rng.choice([0.0625, 0.125, 0.25]))
    return c


def _lengths(case):
    """The sequences' prompt lengths: spread over [lo, hi], the same for every seed so that the work is too."""
    b, lo, hi = case["batch"], case["lo"], case["hi"]
    if lo == hi or b == 1:
        return [hi] * b
    # a fixed scramble of evenly spread odd lengths: no order that a kernel could profit from
    return [hi if i == 0 else lo + ((i * 40503 + 977) * (hi - lo) // 65536) % (hi - lo + 1) for i in range(b)]


def _randn(shape, gen, dtype, scale=None):
    """N(0, 1) in ``dtype``; a pool of many GB is filled in pieces."""
    out = torch.empty(shape, device="cuda", dtype=dtype)
    flat = out.view(shape[0], -1)
    rows = max(1, (1 << 27) // max(1, flat.shape[1]))
    for at in range(0, shape[0], rows):
        x = torch.randn((min(rows, shape[0] - at),) + tuple(shape[1:]), generator=gen, device="cuda")
        if scale is not None:
            x *= scale
        out[at:at + rows] = x.to(dtype)
    return out


def _key_scale(gen, head_dim):
    return torch.exp(0.5 * torch.randn((head_dim,), generator=gen, device="cuda"))


def _paged(case, gen):
    lens, suffix = _lengths(case), case.get("suffix", 0)
    pages = [(n + suffix + PAGE - 1) // PAGE for n in lens]
    total, d = sum(pages), case["head_dim"]
    shape = (total, case["kv_heads"], PAGE, d)
    k = _randn(shape, gen, DTYPES[case["dtype"]], _key_scale(gen, d))
    v = _randn(shape, gen, DTYPES[case["dtype"]])
    perm = torch.randperm(total, generator=gen, device="cuda").to(torch.int32)
    table = torch.zeros((len(lens), max(pages)), dtype=torch.int32, device="cuda")
    at = 0
    for b, n in enumerate(pages):
        table[b, :n] = perm[at:at + n]
        at += n
    prefix = torch.tensor(lens, dtype=torch.int32, device="cuda")
    return ops.PagedKV(k, v, table, prefix, prefix + suffix)


def _blocks(tokens, block):
    return max(1, (tokens + block - 1) // block)


def _score_threshold(score, n_blocks, share):
    """An epsilon that keeps about ``share`` of the blocks: what a user tunes it for."""
    kept = [s[..., :n].reshape(-1) for s, n in zip(score, n_blocks)]
    return float(torch.quantile(torch.cat(kept)[:1 << 20], 1.0 - share))


def _prepare_step(case, gen):
    kv = _paged(case, gen)
    nb = [_blocks(n, case["block"]) for n in _lengths(case)]
    summ = ops.build_summaries(kv, case["block"], max_blocks=max(nb), k_bar_dtype=DTYPES[case["k_bar"]])
    shape = (case["batch"], case["q_heads"], case["head_dim"])
    q = torch.randn(shape, generator=gen, device="cuda").to(DTYPES[case["dtype"]])
    if case["rule"] == "eps":
        score = ops.select_blocks(q, summ, kv.prefix_lens, top_k=1, want=("score",))[2]["score"]
        rule = {"eps": _score_threshold(score, nb, case["share"])}
    else:
        rule = {"top_k": case["k"]}
    step = ops.DecodeAttention(kv, summ, case["q_heads"], rep_mode=case["rep_mode"], **rule)
    state = types.SimpleNamespace(kind="step", step=step, q=q, host=case["host"])
    if case["host"]:
        state.q = q.cpu().pin_memory()
        state.out = torch.empty_like(state.q).pin_memory()
    return state


def _prepare_reference(case, gen):
    n, s, d, hkv = case["tokens"], case["suffix"], case["head_dim"], case["kv_heads"]
    shape = (hkv, (n + s + 63) // 64 * 64, d)   # a static cache: room behind the suffix
    k = _randn(shape, gen, DTYPES[case["dtype"]], _key_scale(gen, d))
    v = _randn(shape, gen, DTYPES[case["dtype"]])
    prefix = reference_api._build_prompt_blocks(k[:, :n], v[:, :n], case["block"])
    q = torch.randn((hkv, case["q_heads"] // hkv, 1, d), generator=gen, device="cuda").to(DTYPES[case["dtype"]])
    length = torch.tensor([n], dtype=torch.int32, device="cuda")
    kv = ops.PagedKV(*llama_decode.cache_as_pool(k[None], v[None]), length, length)
    nb = _blocks(n, case["block"])
    score = ops.select_blocks(q.reshape(1, case["q_heads"], d), ops.build_summaries(kv, case["block"], max_blocks=nb),
                              length, top_k=1, want=("score",))[2]["score"]
    eps = _score_threshold(score, [nb], case["share"])
    args = dict(q_grouped=q, prompt_prefix=prefix, k_suffix=k[:, n:n + s], v_suffix=v[:, n:n + s],
                suffix_len_dev=torch.tensor(s, dtype=torch.int32, device="cuda"), eps=eps, page_size=case["block"],
                store_selected=False, output_dtype=q.dtype, workspace={})
    return types.SimpleNamespace(kind="reference", args=args)


def _prepare_summaries(case, gen):
    if case["api"] == "paged":
        kv = _paged(case, gen)
        nb = _blocks(max(_lengths(case)), case["block"])
        out = ops.BlockSummaries.empty(kv.batch, kv.n_kv_heads, nb, kv.head_dim, kv.k_pool.dtype, kv.k_pool.device,
                                       case["block"])
        return types.SimpleNamespace(kind="summaries_paged", kv=kv, out=out, block=case["block"])
    shape = (case["kv_heads"], case["hi"], case["head_dim"])
    k = _randn(shape, gen, DTYPES[case["dtype"]], _key_scale(gen, case["head_dim"]))
    v = _randn(shape, gen, DTYPES[case["dtype"]])
    return types.SimpleNamespace(kind="summaries_reference", k=k, v=v, block=case["block"])


def _prepare_model(case, gen, seed):
    model = llama_decode.build_random_llama("llama3-8b", n_layers=case["layers"], seed=seed)
    cfg, b = model.config, case["batch"]
    length = (case["tokens"] + case["suffix"] + PAGE) // PAGE * PAGE
    hkv, d = cfg.num_key_value_heads, cfg.head_dim
    prefix = torch.full((b,), case["tokens"], dtype=torch.int32, device="cuda")
    seq = prefix + case["suffix"]
    cache = types.SimpleNamespace(layers=[])
    attention = []
    for _ in range(case["layers"]):
        keys = _randn((b, hkv, length, d), gen, torch.bfloat16, _key_scale(gen, d))
        values = _randn((b, hkv, length, d), gen, torch.bfloat16)
        cache.layers.append(types.SimpleNamespace(keys=keys, values=values))
        k_pool, v_pool, table = llama_decode.cache_as_pool(keys, values)
        kv = ops.PagedKV(k_pool, v_pool, table, prefix, seq)
        summ = ops.build_summaries(kv, case["block"], max_blocks=_blocks(case["tokens"], case["block"]))
        attention.append(ops.DecodeAttention(kv, summ, cfg.num_attention_heads, top_k=case["top_k"]))
    step = llama_step.FusedLlamaStep(model, cache, attention, seq, length)
    first = torch.randint(0, cfg.vocab_size, (b, 1), generator=gen, device="cuda")
    state = types.SimpleNamespace(kind="model", step=step, first=first, tokens=first.clone(), graph=None)
    if case["graph"]:
        _model_pass(state)   # a captured step has run before: every lazy set-up is behind it
        torch.cuda.synchronize()
        state.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state.graph):
            _model_pass(state)
    return state


def _model_pass(state):
    state.tokens.copy_(state.first)   # the token to decode; step() leaves the next one in its place
    state.step.step(state.tokens)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "step":
        return _prepare_step(case, gen)
    if case["kind"] == "reference":
        return _prepare_reference(case, gen)
    if case["kind"] == "summaries":
        return _prepare_summaries(case, gen)
    return _prepare_model(case, gen, seed)


def run(state):
    if state.kind == "step":
        step = state.step
        if state.host:
            return step.step_host(state.q, state.out)
        out = step.step(state.q)
        return {"out": out, "count": step.sel_count, "blocks": step.sel_idx}
    if state.kind == "reference":
        return reference_api._condition_block_decode_output_fused_triton(**state.args)[0]
    if state.kind == "summaries_paged":
        s = ops.build_summaries(state.kv, state.block, out=state.out)
        return [s.k_bar, s.k_max, s.k_min, s.v_bar, s.v_norm_max]
    if state.kind == "summaries_reference":
        p = reference_api._build_prompt_blocks(state.k, state.v, state.block)
        return [p[name] for name in ("k_bar", "k_max", "k_min", "v_bar", "v_norm_max")]
    if state.graph is not None:
        state.graph.replay()
    else:
        _model_pass(state)
    # The greedy tokens are left out: among 128256 bf16 logits the two largest often differ by one rounding or not at
    # all, so that another summation order picks another one.
    return state.step.logits


def _attention_work(case, lens, suffix, picked, hybrid):
    """Bytes and operations of one layer-step: every block's summary, the picked blocks' tokens and the suffix once."""
    d, hkv, g = case["head_dim"], case["kv_heads"], case["q_heads"] // case["kv_heads"]
    e = DTYPES[case["dtype"]].itemsize
    k_bar = 2 if case.get("k_bar") == "bf16" else 4
    n_bytes = flops = 0
    for n in lens:
        nb = _blocks(n, case["block"])
        tokens = min(picked(nb) * case["block"], n) + suffix
        n_bytes += hkv * (nb * (d * (k_bar + 2 * e) + 4) + tokens * 2 * d * e + (nb * d * e if hybrid else 0) + 2 * g * d * e)
        flops += hkv * g * d * (nb * 6 + tokens * 4 + (nb * 2 if hybrid else 0))
    return n_bytes, flops


def work(case):
    if case["kind"] == "step":
        eps = case["rule"] == "eps"
        picked = (lambda nb: int(nb * case["share"])) if eps else (lambda nb: min(case["k"], nb))
        b, f = _attention_work(case, _lengths(case), case["suffix"], picked, case["rep_mode"] == "hybrid")
    elif case["kind"] == "reference":
        b, f = _attention_work(case, [case["tokens"]], case["suffix"], lambda nb: int(nb * case["share"]), True)
    elif case["kind"] == "summaries":
        d, e = case["head_dim"], DTYPES[case["dtype"]].itemsize
        lens = _lengths(case)
        n = sum(lens)
        nb = sum(_blocks(x, case["block"]) for x in lens)
        b = case["kv_heads"] * (n * 2 * d * e + nb * (d * (4 + 3 * e) + 4))
        f = case["kv_heads"] * n * d * 6
    else:
        p = llama_decode.PRESETS["llama3-8b"]
        h, inter, hkv, d = p["hidden_size"], p["intermediate_size"], p["num_key_value_heads"], p["head_dim"]
        layer = h * (p["num_attention_heads"] + 2 * hkv) * d + p["num_attention_heads"] * d * h + 3 * h * inter
        weights = case["layers"] * layer + p["vocab_size"] * h
        one = {"head_dim": d, "kv_heads": hkv, "q_heads": p["num_attention_heads"], "dtype": "bf16", "block": case["block"]}
        b, f = _attention_work(one, [case["tokens"]] * case["batch"], case["suffix"], lambda nb: min(case["top_k"], nb), False)
        b = 2 * weights + case["layers"] * b + 2 * case["batch"] * p["vocab_size"]
        f = 2 * weights * case["batch"] + case["layers"] * f
    return {"bytes": b, "flops": f}


def tolerance(case):
    if case["kind"] == "summaries":
        # means against 64-bit sums: 1e-8, the stored bf16 means all equal; one that rounds the other way is 8e-6
        return {"rel": 1e-5}
    if case["kind"] == "model":
        # four layers with their projections summed in fp32 or fp64 instead of by the library: logits 1.3e-2 apart
        return {"rel": 3e-2}
    # Against the same step in 64 bits (24 cases): 2.7e-7 in fp32, 2.2e-3 in bf16, the same blocks picked everywhere.
    # One block picked otherwise (two scores within a rounding of each other) moves part of a pair's index list.
    return {"rel": 1.5e-6 if case["dtype"] == "f32" else 8e-3, "differ": 0.002}

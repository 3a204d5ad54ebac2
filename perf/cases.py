"""What the speed of this framework is measured on.

The engine is a stack of Llama decoder layers (and, through the same parts, of other designs') between a token
table and an output head, stepped by one function over a paged cache.  A case is one of its pieces as a program
calls it: a layer on a step's tokens (decode steps of many requests, prompts, mixtures of both, in bfloat16 and in
true 32-bit), the output head, the sampler, a recurrent memory; two cases are whole models stepped through
``ModelRunner.step`` with given tokens, logits out.  Sizes are those of the configurations the engine is specified
on: the small one of the tests (hidden 128, 4 heads of 32), and Llama 3.2 1B, Llama 3.2 3B and Llama 3.1 8B, with
random weights (N(0, 0.02), norms near 1).
"""
from __future__ import annotations

import math

import torch

DEV = "cuda:0"

SIZES = {
    "tiny": dict(num_hidden_layers=3, hidden_size=128, num_attention_heads=4, num_key_value_heads=1, head_dim=32,
                 intermediate_size=320, vocab_size=512, rms_norm_eps=1e-6, tie_word_embeddings=False,
                 factor=32.0, original=64),
    "1b": dict(num_hidden_layers=16, hidden_size=2048, num_attention_heads=32, num_key_value_heads=8, head_dim=64,
               intermediate_size=8192, vocab_size=128256, rms_norm_eps=1e-5, tie_word_embeddings=True,
               factor=32.0, original=8192),
    "3b": dict(num_hidden_layers=28, hidden_size=3072, num_attention_heads=24, num_key_value_heads=8, head_dim=128,
               intermediate_size=8192, vocab_size=128256, rms_norm_eps=1e-5, tie_word_embeddings=True,
               factor=32.0, original=8192),
    "8b": dict(num_hidden_layers=32, hidden_size=4096, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
               intermediate_size=14336, vocab_size=128256, rms_norm_eps=1e-5, tie_word_embeddings=False,
               factor=8.0, original=8192),
}
LAYER_VOCAB = 2048            # token table of a case that runs one layer
MEMORY = dict(width=2048, heads=16, dim=128)


def listed():
    return [
        # The small model in 32-bit: four requests of 1, 9, 40 and 70 tokens in portions of 24, then 12 tokens
        # each.  What a check of a change or a small model's user runs: steps of a few microseconds of work.
        dict(name="small_model_answers", kind="model", model="tiny", dtype="float32", requests=4, longest=70,
             tokens=12, page=8, portion=24),
        # The headline of the engine: 8 requests at 4,096 tokens of context, decoded token by token at 1B sizes
        # (their prompts are in the prefix tree: an answer is asked for again, or a conversation goes on).
        dict(name="answers_1b_8", kind="model", model="1b", dtype="bfloat16", requests=8, longest=4065, tokens=16,
             page=16, portion=0),
        # One layer of a decode step under load: 64 requests at 1B sizes, contexts up to 4,096.
        dict(name="decode_1b_64", kind="layer", model="1b", dtype="bfloat16", singles=64, shortest=1024, longest=4095,
             portion=0, at=0),
        # ... 64 streams at 8B sizes a little beyond prompts of 1,024 tokens.
        dict(name="decode_8b_64", kind="layer", model="8b", dtype="bfloat16", singles=64, shortest=1024, longest=1152,
             portion=0, at=0),
        # ... continuous batching at 3B sizes: the second 512 tokens of a prompt beside 31 requests that decode.
        dict(name="mixed_3b", kind="layer", model="3b", dtype="bfloat16", singles=31, shortest=150, longest=2100,
             portion=512, at=512),
        # One layer on a prompt of 2,048 tokens at 1B sizes (the headline's other half).
        dict(name="prompt_1b_2048", kind="layer", model="1b", dtype="bfloat16", singles=0, shortest=0, longest=0,
             portion=2048, at=0),
        # One layer on a later portion of a long prompt at 8B sizes, an odd number of tokens.
        dict(name="prompt_8b_long", kind="layer", model="8b", dtype="bfloat16", singles=0, shortest=0, longest=0,
             portion=2011, at=4096),
        # The output head over a vocabulary of 128,256 for 64 requests.
        dict(name="head_1b_64", kind="head", model="1b", dtype="bfloat16", rows=64),
        # Sampling 128 rows over that vocabulary: greedy, temperature, top-k, top-p and both, as requests ask for.
        dict(name="sample_128", kind="sample", rows=128, vocab=128256),
        # The true 32-bit path at 1B sizes: a prompt, and a decode step.
        dict(name="prompt_1b_32bit", kind="layer", model="1b", dtype="float32", singles=0, shortest=0, longest=0,
             portion=500, at=0),
        dict(name="decode_1b_32bit", kind="layer", model="1b", dtype="float32", singles=8, shortest=300, longest=1500,
             portion=0, at=0),
        # A recurrent memory of the Ridotar design (one decay a head) on a prompt beside requests that decode.
        dict(name="memory_prompt", kind="memory", dtype="bfloat16", singles=3, portion=1500),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model", "model", "decode", "decode", "decode", "prompt", "prompt", "mixed", "mixed", "head", "sample",
                       "prompt32", "decode32", "memory"])
    if kind == "model":
        if rng.random() < 0.5:
            return dict(kind="model", model="tiny", dtype=rng.choice(["float32", "float32", "bfloat16"]),
                        requests=rng.randint(1, 4), longest=rng.randint(10, 90), tokens=rng.randint(4, 12), page=8,
                        portion=rng.choice([16, 24, 32]))
        return dict(kind="model", model="1b", dtype="bfloat16", requests=_log(rng, 1, 8),
                    longest=16 * rng.randint(16, 254) + 1, tokens=rng.randint(6, 12), page=16, portion=0)
    if kind in ("decode", "mixed", "prompt"):
        c = dict(kind="layer", model=rng.choice(["1b", "3b", "8b"]), dtype="bfloat16", singles=0, shortest=0,
                 longest=0, portion=0, at=0)
        if kind != "prompt":
            c["longest"] = _log(rng, 150, 4000 if c["model"] == "1b" else 1200)
            c["shortest"] = rng.randint(16, c["longest"])
            c["singles"] = _log(rng, 17, 64) if kind == "decode" else rng.randint(4, 60)
        if kind == "mixed":
            c["portion"], c["at"] = _log(rng, 33, 700), rng.choice([0, 0, 256, 511])
        if kind == "prompt":
            c["portion"], c["at"] = _log(rng, 130, 1900), rng.choice([0, 0, 512, 1000, 2048])
        return c
    if kind == "head":
        return dict(kind="head", model=rng.choice(["1b", "3b", "8b"]), dtype="bfloat16", rows=rng.randint(1, 64))
    if kind == "sample":
        return dict(kind="sample", rows=rng.randint(101, 127), vocab=rng.choice([32000, 50257, 128256]))
    if kind == "prompt32":
        return dict(kind="layer", model="1b", dtype="float32", singles=0, shortest=0, longest=0,
                    portion=_log(rng, 40, 480), at=rng.choice([0, 0, 300]))
    if kind == "decode32":
        longest = rng.randint(100, 1500)
        return dict(kind="layer", model="1b", dtype="float32", singles=rng.randint(1, 16),
                    shortest=rng.randint(16, longest), longest=longest, portion=0, at=0)
    return dict(kind="memory", dtype="bfloat16", singles=rng.randint(0, 6), portion=_log(rng, 100, 1450))


# ------------------------------------------------------------------ inputs
def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def _config_dict(model, **other):
    s = dict(SIZES[model], **other)
    factor, original = s.pop("factor"), s.pop("original")
    return dict(s, architectures=["LlamaForCausalLM"], rope_theta=500000.0, max_position_embeddings=131072,
                rope_scaling=dict(rope_type="llama3", factor=factor, low_freq_factor=1.0, high_freq_factor=4.0,
                                  original_max_position_embeddings=original))


def _generator(seed, more=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * (seed + 1) + more)


def _weights(cfg, dtype, seed, head=True):
    """The checkpoint's tensors, from the seed."""
    g = _generator(seed)
    H, I, hd = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    q, kv = cfg["num_attention_heads"] * hd, cfg["num_key_value_heads"] * hd

    def matrix(n, k):
        return torch.empty(n, k, dtype=dtype, device=DEV).normal_(0.0, 0.02, generator=g)

    def norm():
        return 1.0 + torch.empty(H, dtype=torch.float32, device=DEV).normal_(0.0, 0.1, generator=g)

    t = {"model.embed_tokens.weight": matrix(cfg["vocab_size"], H), "model.norm.weight": norm()}
    if not cfg["tie_word_embeddings"]:
        t["lm_head.weight"] = matrix(cfg["vocab_size"], H)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        t[p + "input_layernorm.weight"], t[p + "post_attention_layernorm.weight"] = norm(), norm()
        for name, (n, k) in (("self_attn.q_proj", (q, H)), ("self_attn.k_proj", (kv, H)), ("self_attn.v_proj", (kv, H)),
                             ("self_attn.o_proj", (H, q)), ("mlp.gate_proj", (I, H)), ("mlp.up_proj", (I, H)),
                             ("mlp.down_proj", (H, I))):
            t[p + name + ".weight"] = matrix(n, k)
    return t


def _lengths(n, lo, hi):
    """n lengths from lo to hi, spread evenly and in no order."""
    if n == 1:
        return [hi]
    return [lo + (hi - lo) * ((7 * i + 3) % n) // (n - 1) for i in range(n)]


def _entries(case):
    """(tokens already cached, new tokens) of each request of a layer's step: single tokens first."""
    e = [(n, 1) for n in _lengths(case["singles"], case["shortest"], case["longest"])] if case["singles"] else []
    return e + ([(case["at"], case["portion"])] if case["portion"] else [])


def _tokens(n, vocab, seed, more):
    return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(977 * seed + more)).tolist()


def _plan(case, seed):
    """The prompts of a model case and the tokens that follow each."""
    vocab = SIZES[case["model"]]["vocab_size"]
    n, longest = case["requests"], case["longest"]
    if case["portion"]:
        lens = [1 + (longest - 1) * i * (i + 1) // max(1, n * (n - 1)) for i in range(n)]
    else:
        lens = [longest] * n
    return ([_tokens(k, vocab, seed, 10 + i) for i, k in enumerate(lens)],
            [_tokens(case["tokens"], vocab, seed, 500 + i) for i in range(n)])


def _portions(case, prompts, more):
    """The steps of a model case with portions: request -> tokens, and whether its last token's logits are wanted."""
    left = [list(p) for p in prompts]
    next_token = [0] * len(prompts)
    steps = []
    while any(k < len(m) for k, m in zip(next_token, more)):
        step = []
        for i in range(len(prompts)):
            if left[i]:
                step.append((i, left[i][:case["portion"]], len(left[i]) <= case["portion"]))
                left[i] = left[i][case["portion"]:]
            elif next_token[i] < len(more[i]):
                step.append((i, [more[i][next_token[i]]], True))
                next_token[i] += 1
        steps.append(step)
    return steps


def _runner(case, cfg, tensors, pages, requests, tokens, longest, page=16):
    from llm_singularity_b200.config.llama import LlamaConfig
    from llm_singularity_b200.engine.runner import ModelRunner
    return ModelRunner(config=LlamaConfig.from_dict(cfg), tensors=tensors, dtype=case["dtype"], device=DEV,
                       page_size=page, num_pages=pages, max_requests=requests, max_tokens_per_step=max(tokens, 64),
                       max_model_len=longest)


def _cached(case, cfg, seed, length, i):
    """Keys and values a request already has in the cache: [kv heads, length, head size] each."""
    shape = (2, cfg["num_key_value_heads"], length, cfg["head_dim"])
    return torch.empty(shape, dtype=_dtype(case), device=DEV).normal_(0.0, 0.9, generator=_generator(seed, 7 + i))


def _logits_of(seed, rows, vocab):
    """Logits as trained models give them: most of the weight on a few tokens."""
    return torch.empty(rows, vocab, dtype=torch.float32, device=DEV).normal_(0.0, 3.0, generator=_generator(seed, 3))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return _prepare_sample(case, seed)
    if kind == "memory":
        return _prepare_memory(case, seed)
    from llm_singularity_b200.engine import StepEntry
    if kind == "model":
        cfg = _config_dict(case["model"])
        prompts, more = _plan(case, seed)
        longest = max(map(len, prompts)) + case["tokens"] + 1
        pages = 2 + sum(-(-(len(p) + case["tokens"] + 1) // case["page"]) for p in prompts)
        runner = _runner(case, cfg, _weights(cfg, _dtype(case), seed), pages + 8, len(prompts), 2048, longest + 16, case["page"])
        state = dict(case=case, runner=runner, prompts=prompts)
        if case["portion"]:
            state["steps"] = [[(i, StepEntry(i, toks, [len(toks) - 1] if want else [])) for i, toks, want in step]
                              for step in _portions(case, prompts, more)]
            return state
        from llm_singularity_b200.cache.prefix import RadixPrefixCache
        tree = state["tree"] = RadixPrefixCache(runner.cache)
        for i, p in enumerate(prompts):
            runner.open(i)
            for s in range(0, len(p) - 1, 2048):
                runner.step([StepEntry(i, p[s:min(s + 2048, len(p) - 1)], [])])
            tree.insert(p[:-1], i)
            runner.close(i)
        feed = [[p[-1]] + m[:-1] for p, m in zip(prompts, more)]
        state["steps"] = [[(i, StepEntry(i, [f[s]], [0])) for i, f in enumerate(feed)] for s in range(case["tokens"])]
        return state
    if kind == "head":
        cfg = _config_dict(case["model"], num_hidden_layers=1, tie_word_embeddings=True)
        runner = _runner(case, cfg, _weights(cfg, _dtype(case), seed), 4, 1, 64, 64)
        g = _generator(seed, 5)
        T, H = case["rows"], cfg["hidden_size"]
        return dict(case=case, head=runner.model.head,
                    stream=torch.empty(T, H, dtype=torch.float32, device=DEV).normal_(0.0, 1.0, generator=g),
                    delta=torch.empty(T, H, dtype=_dtype(case), device=DEV).normal_(0.0, 0.3, generator=g),
                    rows=torch.arange(T, dtype=torch.int32, device=DEV))
    # one layer of a step
    cfg = _config_dict(case["model"], num_hidden_layers=1, vocab_size=LAYER_VOCAB, tie_word_embeddings=True)
    entries = _entries(case)
    T = sum(n for _, n in entries)
    pages = sum(-(-(s + n) // 16) for s, n in entries)
    runner = _runner(case, cfg, _weights(cfg, _dtype(case), seed), pages, len(entries), T,
                     max(s + n for s, n in entries) + 16)
    cache = runner.cache
    view = cache.view(0)
    for i, (s, n) in enumerate(entries):
        runner.open(i)
        cache.reserve(i, s + n)
        cache.commit(i, s)
        if s:
            held = -(-s // 16)
            ids = torch.tensor(cache.pages_of(i)[:held], dtype=torch.long, device=DEV)
            kv = torch.nn.functional.pad(_cached(case, cfg, seed, s, i), (0, 0, 0, held * 16 - s))
            kv = kv.view(2, cfg["num_key_value_heads"], held, 16, cfg["head_dim"]).transpose(1, 2)
            view.k_pages[ids], view.v_pages[ids] = kv[0], kv[1]
    step = [StepEntry(i, _tokens(n, LAYER_VOCAB, seed, 20 + i), []) for i, (_, n) in enumerate(entries)]
    ctx, _ = runner.prepare_context(step, [s for s, _ in entries])
    return dict(case=case, model=runner.model, ctx=ctx, view=cache.view(0, ctx), runner=runner)


def _prepare_sample(case, seed):
    from llm_singularity_b200.parts.base import Runtime
    from llm_singularity_b200.sampling import Sampler, SamplingParams
    kinds = [dict(temperature=0.0), dict(temperature=0.8), dict(temperature=0.8, top_k=50),
             dict(temperature=1.0, top_p=0.9), dict(temperature=0.7, top_k=40, top_p=0.95), dict(temperature=0.6, top_p=0.95)]
    params = [SamplingParams(seed=seed * 1000 + r, **kinds[r % len(kinds)]) for r in range(case["rows"])]
    return dict(case=case, sampler=Sampler(Runtime(DEV, torch.bfloat16)), params=params,
                draws=[5 + r % 90 for r in range(case["rows"])], logits=_logits_of(seed, case["rows"], case["vocab"]))


def _decays():
    return [1.0 - 2.0 ** (-5 - 3 * h / MEMORY["heads"]) for h in range(MEMORY["heads"])]


def _memory_tensors(case, seed):
    g = _generator(seed)
    H, n = MEMORY["width"], MEMORY["heads"] * MEMORY["dim"]
    T, dt = case["singles"] + case["portion"], _dtype(case)
    w = {k: torch.empty(n, H, dtype=dt, device=DEV).normal_(0.0, 0.02, generator=g) for k in "qkvg"}
    w["o"] = torch.empty(H, n, dtype=dt, device=DEV).normal_(0.0, 0.02, generator=g)
    w["norm"] = 1.0 + torch.empty(n, dtype=torch.float32, device=DEV).normal_(0.0, 0.1, generator=g)
    x = torch.empty(T, H, dtype=dt, device=DEV).normal_(0.0, 1.0, generator=g)
    s = torch.empty(case["singles"] + 1, MEMORY["heads"], MEMORY["dim"], MEMORY["dim"], device=DEV).normal_(0.0, 1.0, generator=g)
    s[-1].zero_()                                      # (the prompt begins here)
    return w, x, s


def _prepare_memory(case, seed):
    from llm_singularity_b200.config.specs import LinearRecurrenceSpec
    from llm_singularity_b200.engine.batch import ContextBuilder
    from llm_singularity_b200.parts.base import MIXERS, Runtime
    w, x, s = _memory_tensors(case, seed)
    rt = Runtime(DEV, _dtype(case))
    spec = LinearRecurrenceSpec(hidden_size=MEMORY["width"], num_heads=MEMORY["heads"], key_dim=MEMORY["dim"],
                                value_dim=MEMORY["dim"], gate="fixed_decay", decay=tuple(_decays()), q_activation="silu",
                                k_activation="silu", v_activation="silu", out_norm="all", out_gate=True, eps=1e-6)
    part = MIXERS.build(spec, rt)
    part.load(w)
    cache_spec = part.cache_spec()
    storage = cache_spec.allocate(rt, 16, None, s.shape[0])
    tokens = [[0]] * case["singles"] + [[0] * case["portion"]]
    ctx, _ = ContextBuilder(DEV, x.shape[0], s.shape[0]).build(
        tokens, [100 + i for i in range(case["singles"])] + [0], list(range(s.shape[0])), [[]] * len(tokens))
    return dict(case=case, part=part, x=x, ctx=ctx, view=cache_spec.view(storage, None), begin=s)


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["case"]["kind"]
    if kind == "layer":
        model, ctx = state["model"], state["ctx"]
        stream = model.embedding.forward(ctx.token_ids)
        delta = model.blocks[0].forward(stream, None, ctx, state["view"], True)
        return [stream, delta, state["view"].k_pages, state["view"].v_pages]
    if kind == "head":
        return state["head"].forward(state["stream"], state["delta"], state["rows"])
    if kind == "sample":
        return state["sampler"].sample(state["logits"], state["params"], state["draws"])
    if kind == "memory":
        state["view"].state.copy_(state["begin"])
        y = state["part"].forward(state["x"], state["ctx"], state["view"])
        return [y, state["view"].state]
    runner, prompts = state["runner"], state["prompts"]
    tree, paths = state.get("tree"), {}
    for i, p in enumerate(prompts):
        runner.open(i)
        if tree is not None:
            paths[i] = tree.match(p)
            tree.adopt(i, paths[i])
    logits = []
    for step in state["steps"]:
        out = runner.step([e for _, e in step])
        if out.shape[0]:
            logits.append(out.clone())               # (a decode step's rows are the runner's own)
    for i in range(len(prompts)):
        if tree is not None:
            tree.release(paths[i])
        runner.close(i)
    return logits


# ------------------------------------------------------------------ what a pass cannot do without
def _layer_work(model, dtype, entries):
    s = SIZES[model]
    esize = 4 if dtype == "float32" else 2
    H, I, hd, nh, nkv = (s[k] for k in ("hidden_size", "intermediate_size", "head_dim", "num_attention_heads",
                                        "num_key_value_heads"))
    weights = (nh + 2 * nkv) * hd * H + nh * hd * H + 3 * I * H
    T = sum(n for _, n in entries)
    keys = sum(s0 * n + n * (n + 1) // 2 for s0, n in entries)           # (query, key) pairs of a head
    kv = sum(s0 + n for s0, n in entries) * 2 * nkv * hd * esize
    return weights * esize + kv, 2 * T * weights + 4 * nh * hd * keys


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": 4 * case["rows"] * (case["vocab"] + 1), "flops": 2 * case["rows"] * case["vocab"]}
    if kind == "memory":
        H, n, d = MEMORY["width"], MEMORY["heads"] * MEMORY["dim"], MEMORY["dim"]
        T, slots = case["singles"] + case["portion"], case["singles"] + 1
        return {"bytes": 2 * 5 * n * H + 2 * 2 * T * H + 2 * 4 * slots * n * d, "flops": 2 * T * 5 * n * H + 4 * T * n * d}
    s = SIZES[case["model"]]
    esize = 4 if case["dtype"] == "float32" else 2
    H, V = s["hidden_size"], s["vocab_size"]
    if kind == "head":
        T = case["rows"]
        return {"bytes": V * H * esize + T * H * 6 + 4 * T * V, "flops": 2 * T * V * H}
    if kind == "layer":
        entries = _entries(case)
        T = sum(n for _, n in entries)
        b, f = _layer_work(case["model"], case["dtype"], entries)
        return {"bytes": b + T * H * (4 + 2 * esize), "flops": f}
    prompts, more = _plan(case, 0)
    total_b = total_f = 0
    if case["portion"]:
        held = [0] * len(prompts)
        steps = [[(i, len(toks), want) for i, toks, want in step] for step in _portions(case, prompts, more)]
    else:
        held = [len(p) - 1 for p in prompts]
        steps = [[(i, 1, True) for i in range(len(prompts))]] * case["tokens"]
    for step in steps:
        b, f = _layer_work(case["model"], case["dtype"], [(held[i], n) for i, n, _ in step])
        wanted = sum(1 for _, _, want in step if want)
        total_b += s["num_hidden_layers"] * b + (V * H * esize + 4 * wanted * V if wanted else 0)
        total_f += s["num_hidden_layers"] * f + 2 * wanted * V * H
        for i, n, _ in step:
            held[i] += n
    return {"bytes": total_b, "flops": total_f}


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        return {"rel": 0.0, "differ": 0.01}           # a draw that falls on the edge of two tokens
    if kind == "model":
        return {"rel": 1e-5} if case["dtype"] == "float32" else {"rel": 0.03}
    if kind == "memory":
        return {"rel": 1e-2}
    if kind == "head":
        return {"rel": 5e-3}
    # (against 64 bits: up to 6.3e-6 in 32 bits, angles of positions beyond 1,000 among it; 1e-2 in bfloat16)
    return {"rel": 2.5e-5} if case["dtype"] == "float32" else {"rel": 1.5e-2}


# ------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()


def _inv_freq(cfg):
    half = cfg["head_dim"] // 2
    f = 500000.0 ** (-torch.arange(half, dtype=torch.float64, device=DEV) / half)
    rs = cfg["rope_scaling"]
    length = 2 * math.pi / f
    low = rs["original_max_position_embeddings"] / rs["low_freq_factor"]
    high = rs["original_max_position_embeddings"] / rs["high_freq_factor"]
    smooth = (rs["original_max_position_embeddings"] / length - rs["low_freq_factor"]) \
        / (rs["high_freq_factor"] - rs["low_freq_factor"])
    mid = (1 - smooth) * f / rs["factor"] + smooth * f
    return torch.where(length > low, f / rs["factor"], torch.where(length < high, f, mid))


def _rotate(x, positions, inv):
    """x [T, heads, size]: dims i and i + size / 2 are a pair."""
    a = positions.double()[:, None] * inv
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    half = x.shape[-1] // 2
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _layer64(h, w, cfg, inv, spans, caches):
    """One layer in place on the stream h: (stream with attention added, feed-forward's output).  ``spans``: (first row,
    tokens, tokens cached) of each request; ``caches``: [2, kv heads, cached, size] or None, replaced by the longer one."""
    T = h.shape[0]
    nh, nkv, hd, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    x = _rms(h, w["input_layernorm"], eps)
    pos = torch.cat([torch.arange(s, s + n, device=DEV) for _, n, s in spans])
    q = _rotate((x @ w["self_attn.q_proj"].double().T).view(T, nh, hd), pos, inv)
    k = _rotate((x @ w["self_attn.k_proj"].double().T).view(T, nkv, hd), pos, inv)
    v = (x @ w["self_attn.v_proj"].double().T).view(T, nkv, hd)
    out = torch.empty(T, nh, hd, dtype=torch.float64, device=DEV)
    for r, (t0, n, s) in enumerate(spans):
        keys, vals = k[t0:t0 + n].transpose(0, 1), v[t0:t0 + n].transpose(0, 1)
        if caches[r] is not None:
            keys, vals = torch.cat([caches[r][0].double(), keys], 1), torch.cat([caches[r][1].double(), vals], 1)
        caches[r] = (keys, vals)
        for g in range(nkv):
            qg = q[t0:t0 + n, g * (nh // nkv):(g + 1) * (nh // nkv)].transpose(0, 1)          # [group, n, hd]
            sc = (qg @ keys[g].T) / math.sqrt(hd)
            if n > 1:
                sc.masked_fill_(torch.arange(s + n, device=DEV) > torch.arange(s, s + n, device=DEV)[:, None], -math.inf)
            out[t0:t0 + n, g * (nh // nkv):(g + 1) * (nh // nkv)] = (torch.softmax(sc, -1) @ vals[g]).transpose(0, 1)
    h = h + out.view(T, nh * hd) @ w["self_attn.o_proj"].double().T
    x = _rms(h, w["post_attention_layernorm"], eps)
    gate = x @ w["mlp.gate_proj"].double().T
    return h, (gate * torch.sigmoid(gate) * (x @ w["mlp.up_proj"].double().T)) @ w["mlp.down_proj"].double().T


def _of_layer(t, i):
    p = f"model.layers.{i}."
    return {k[len(p):-len(".weight")]: v for k, v in t.items() if k.startswith(p)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return None                                    # (whole numbers)
    if kind == "memory":
        return _exact_memory(case, seed)
    if kind == "head":
        cfg = _config_dict(case["model"], num_hidden_layers=1, tie_word_embeddings=True)
        t = _weights(cfg, _dtype(case), seed)
        g = _generator(seed, 5)
        T, H = case["rows"], cfg["hidden_size"]
        x = torch.empty(T, H, dtype=torch.float32, device=DEV).normal_(0.0, 1.0, generator=g).double()
        x = x + torch.empty(T, H, dtype=_dtype(case), device=DEV).normal_(0.0, 0.3, generator=g).double()
        return _rms(x, t["model.norm.weight"], cfg["rms_norm_eps"]) @ t["model.embed_tokens.weight"].double().T
    if kind == "layer":
        cfg = _config_dict(case["model"], num_hidden_layers=1, vocab_size=LAYER_VOCAB, tie_word_embeddings=True)
        t = _weights(cfg, _dtype(case), seed)
        spans, caches, ids = [], [], []
        for i, (s, n) in enumerate(_entries(case)):
            spans.append((len(ids), n, s))
            caches.append(_cached(case, cfg, seed, s, i) if s else None)
            ids += _tokens(n, LAYER_VOCAB, seed, 20 + i)
        h = t["model.embed_tokens.weight"][torch.tensor(ids, device=DEV)].double()
        return [*_layer64(h, _of_layer(t, 0), cfg, _inv_freq(cfg), spans, caches), None, None]
    # a whole model: request by request, every token's logits that the steps ask for
    cfg = _config_dict(case["model"])
    t = _weights(cfg, _dtype(case), seed)
    inv = _inv_freq(cfg)
    prompts, more = _plan(case, seed)
    layers = [_of_layer(t, i) for i in range(cfg["num_hidden_layers"])]
    head = t["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"].double().T
    rows = []
    for p, m in zip(prompts, more):
        last = m if case["portion"] else m[:-1]
        ids = torch.tensor(p + last, device=DEV)
        h, d = t["model.embed_tokens.weight"][ids].double(), 0.0
        for w in layers:
            h, d = _layer64(h + d, w, cfg, inv, [(0, len(ids), 0)], [None])
        rows.append(_rms((h + d)[len(p) - 1:], t["model.norm.weight"], cfg["rms_norm_eps"]) @ head)
    if not case["portion"]:
        return [torch.stack([r[s] for r in rows]) for s in range(case["tokens"])]
    out, seen = [], [0] * len(prompts)
    for step in _portions(case, prompts, more):
        wanted = [i for i, _, want in step if want]
        if wanted:
            out.append(torch.stack([rows[i][seen[i]] for i in wanted]))
        for i in wanted:
            seen[i] += 1
    return out


def _exact_memory(case, seed):
    w, x, s = _memory_tensors(case, seed)
    x, n, d = x.double(), MEMORY["heads"], MEMORY["dim"]
    q, k, v = (torch.nn.functional.silu(x @ w[c].double().T).view(-1, n, d) for c in "qkv")
    decay = torch.tensor(_decays(), dtype=torch.float64, device=DEV)
    o, states = [], []
    spans = [(i, 1) for i in range(case["singles"])] + [(case["singles"], case["portion"])]
    for r, (t0, T) in enumerate(spans):
        S = s[r].double()                              # [heads, value, key]
        at = torch.arange(T, device=DEV, dtype=torch.float64)
        rows = torch.empty(T, n, d, dtype=torch.float64, device=DEV)
        new = torch.empty_like(S)
        for h in range(n):
            qh, kh, vh = (z[t0:t0 + T, h] for z in (q, k, v))
            fade = torch.where(at[:, None] >= at, decay[h] ** (at[:, None] - at).clamp(min=0), 0.0)
            rows[:, h] = ((qh @ kh.T) * fade) @ vh + (decay[h] ** (at + 1))[:, None] * (qh @ S[h].T)
            new[h] = decay[h] ** T * S[h] + (vh * (decay[h] ** (T - 1 - at))[:, None]).T @ kh
        o.append(rows)
        states.append(new)
    y = _rms(torch.cat(o).view(-1, n * d), w["norm"], 1e-6) * torch.sigmoid(x @ w["g"].double().T)
    return [y @ w["o"].double().T, torch.stack(states)]

"""What is timed of this package, by what a program has it do.

The kinds of cases:

* ``serve``: a whole Qwen3 model of a few layers through ``ModelRunner.step``, as a trace is replayed: the prompts
  of some requests in one step, then steps of one given token each, logits of every step.  bfloat16 at the 8B layer
  sizes, and the 32-bit path at the 0.6B sizes (where programs check logits).
* ``mlp``: a gated feed-forward part (gate | up product, SwiGLU, down product into the residual) over the rows of a
  step, from one decoded token to a prompt portion of 4,096.
* ``attention``: ``CudaKernels.attention`` over the paged cache: prompts, portions of prompts after a context, and
  decode steps of many requests of different lengths; with Gitipel's capped scores; in both element types.
* ``experts``: the routed feed-forward of Pitudra, Dogetar and Pafivik for choices already made.
* ``delta_rule`` (Gitipel), ``channel_delta`` (Pafivik), ``state_space`` (Dogetar): the recurrences with a state per
  request, over prompts and over decode steps.

Sizes are those of ``bench.py``'s designs (widths 1,024, 2,048 and 4,096 with their heads) and of Qwen3 0.6B and 8B.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch

DEV = "cuda:0"
PAGE = 16
VOCAB = 151936
# (width, attention heads, kv heads, head size, feed-forward)
SIZES = {"small": (1024, 16, 8, 64, 3072), "medium": (2048, 16, 8, 128, 6144), "large": (4096, 32, 8, 128, 12288),
         "qwen3-0.6b": (1024, 16, 8, 128, 3072), "qwen3-8b": (4096, 32, 8, 128, 12288)}
TYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
# the models' constants: Gitipel's decay scale, what is added under a key's root
DECAY_SCALE, KEY_EPS = 0.606531, 1e-6
RANK, STATE, GROUPS, STATE_HEAD = 64, 128, 8, 64


def listed():
    return [
        # a small serving batch at the 8B sizes: eight prompts at once, then sixteen tokens of each
        dict(name="serve 8b bf16", kind="serve", dtype="bfloat16", size="qwen3-8b", layers=4, requests=8, prompt=512, steps=16),
        # the 32-bit path, as used to check logits of a small model
        dict(name="serve 0.6b fp32", kind="serve", dtype="float32", size="qwen3-0.6b", layers=4, requests=4, prompt=200, steps=8),
        # a prompt portion through the feed-forward of an 8B layer, rows that fill no whole tile
        dict(name="mlp prompt bf16", kind="mlp", dtype="bfloat16", size="qwen3-8b", rows=2000),
        # a short prompt through the same part in 32-bit
        dict(name="mlp prompt fp32", kind="mlp", dtype="float32", size="qwen3-0.6b", rows=300),
        # one long prompt, and a decode step of a full server
        dict(name="attention prompt bf16", kind="attention", dtype="bfloat16", size="qwen3-8b", seqs=1, query=2048, context=0, softcap=0.0),
        dict(name="attention decode bf16", kind="attention", dtype="bfloat16", size="qwen3-8b", seqs=64, query=1, context=4095, softcap=0.0),
        # Gitipel's capped scores over a few prompts
        dict(name="attention capped bf16", kind="attention", dtype="bfloat16", size="medium", seqs=4, query=700, context=0, softcap=30.0),
        # prompts of the 32-bit path
        dict(name="attention prompt fp32", kind="attention", dtype="float32", size="qwen3-0.6b", seqs=3, query=400, context=0, softcap=0.0),
        # a prompt through Gitipel's recurrence, several through Pafivik's, a decode step through Dogetar's
        dict(name="delta rule prompt", kind="delta_rule", dtype="bfloat16", size="medium", seqs=1, query=2048),
        dict(name="channel delta prompts", kind="channel_delta", dtype="bfloat16", size="medium", seqs=4, query=600),
        dict(name="state space decode", kind="state_space", dtype="bfloat16", size="medium", seqs=64, query=1),
        # a prompt through eight experts, two a token
        dict(name="experts prompt", kind="experts", size="medium", rows=2048, experts=8, top=2),
    ]


def _log(rng, low, high):
    """A whole number between the two, spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["serve", "mlp", "mlp", "attention", "attention", "attention", "experts", "delta_rule",
                       "channel_delta", "state_space"])
    exact_path = rng.random() < 0.35
    dtype = "float32" if exact_path else "bfloat16"
    width = rng.choice(["small", "medium", "large"])
    if kind == "serve":
        if exact_path:
            return dict(kind=kind, dtype=dtype, size="qwen3-0.6b", layers=rng.randint(2, 4), requests=rng.randint(1, 8),
                        prompt=_log(rng, 16, 300), steps=rng.randint(2, 8))
        requests = _log(rng, 1, 32)
        return dict(kind=kind, dtype=dtype, size=rng.choice(["qwen3-0.6b", "qwen3-8b"]), layers=rng.randint(2, 4),
                    requests=requests, prompt=_log(rng, 16, max(32, min(600, 3000 // requests))), steps=rng.randint(4, 16))
    if kind == "mlp":
        if exact_path:
            return dict(kind=kind, dtype=dtype, size=rng.choice(["small", "medium"]), rows=_log(rng, 1, 1200))
        return dict(kind=kind, dtype=dtype, size=width, rows=_log(rng, 1, 4096))
    if kind == "attention":
        capped = 30.0 if rng.random() < 0.3 else 0.0
        if rng.random() < 0.5:                               # a decode step
            return dict(kind=kind, dtype=dtype, size=width, seqs=_log(rng, 1, 16 if exact_path else 96), query=1,
                        context=_log(rng, 64, 2000 if exact_path else 8000), softcap=capped)
        query = _log(rng, 64, 600 if exact_path else 3000)
        return dict(kind=kind, dtype=dtype, size=width, seqs=rng.randint(1, 4), query=query,
                    context=0 if rng.random() < 0.6 else _log(rng, 64, 800 if exact_path else 6000), softcap=capped)
    if kind == "experts":
        return dict(kind=kind, size=width, rows=_log(rng, 1, 4096), experts=8, top=rng.choice([1, 2, 2, 3]))
    if rng.random() < 0.4:                                   # a decode step of a recurrence
        return dict(kind=kind, dtype=dtype, size=width, seqs=_log(rng, 1, 96), query=1)
    seqs = rng.randint(1, 6)
    return dict(kind=kind, dtype=dtype, size=width, seqs=seqs, query=_log(rng, 16, 3000 // seqs))


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) + 12345)


def _normal(g, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device=DEV) * std).to(dtype)


def _uniform(g, low, high, *shape):
    return torch.rand(*shape, generator=g, device=DEV) * (high - low) + low


def _lengths(case, most, least):
    """A length for each sequence: the first the longest, the others anywhere from a quarter of it.  (The case's
    own, whatever the seed: outputs of two seeds have the same shape.)"""
    g = torch.Generator().manual_seed(99 + most)
    low = max(least, most // 4)
    return [most] + [int(torch.randint(low, most + 1, (1,), generator=g)) for _ in range(case["seqs"] - 1)]


def _ints(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _starts(lens):
    out = [0]
    for n in lens:
        out.append(out[-1] + n)
    return out


def _qwen3_config(case):
    width, heads, kv, dim, ff = SIZES[case["size"]]
    return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "attention_bias": False, "hidden_act": "silu",
            "rope_scaling": None, "torch_dtype": "bfloat16", "num_hidden_layers": case["layers"], "hidden_size": width,
            "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": dim, "intermediate_size": ff,
            "vocab_size": VOCAB, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "max_position_embeddings": 40960,
            "tie_word_embeddings": case["size"] == "qwen3-0.6b", "use_sliding_window": False, "sliding_window": None}


def _qwen3_tensors(case, seed):
    """(name, tensor) of a random model: matrices N(0, 0.02), norm weights near one."""
    width, heads, kv, dim, ff = SIZES[case["size"]]
    g = _generator(seed)
    dtype = TYPES[case["dtype"]]

    def matrix(rows, cols):
        # (values that bfloat16 holds, whatever the run's type: a checkpoint's)
        return _normal(g, rows, cols, std=0.02, dtype=torch.bfloat16).to(dtype)

    def vector(n):
        return _uniform(g, 0.9, 1.1, n).to(torch.bfloat16).to(dtype)

    yield "model.embed_tokens.weight", matrix(VOCAB, width)
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        yield p + "input_layernorm.weight", vector(width)
        for role, rows in (("q", heads * dim), ("k", kv * dim), ("v", kv * dim)):
            yield p + f"self_attn.{role}_proj.weight", matrix(rows, width)
        yield p + "self_attn.q_norm.weight", vector(dim)
        yield p + "self_attn.k_norm.weight", vector(dim)
        yield p + "self_attn.o_proj.weight", matrix(width, heads * dim)
        yield p + "post_attention_layernorm.weight", vector(width)
        yield p + "mlp.gate_proj.weight", matrix(ff, width)
        yield p + "mlp.up_proj.weight", matrix(ff, width)
        yield p + "mlp.down_proj.weight", matrix(width, ff)
    yield "model.norm.weight", vector(width)
    if case["size"] != "qwen3-0.6b":
        yield "lm_head.weight", matrix(VOCAB, width)


def _serve_tokens(case, seed):
    """Token ids of every request: its prompt, then one a step."""
    g = torch.Generator().manual_seed(99)
    lens = [case["prompt"]] + [int(torch.randint(16, case["prompt"] + 1, (1,), generator=g)) for _ in range(case["requests"] - 1)]
    g = torch.Generator().manual_seed(int(seed) + 7)
    return [torch.randint(0, VOCAB, (n + case["steps"],), generator=g).tolist() for n in lens], lens


def _attention_inputs(case, seed):
    width, heads, kv, dim, _ = SIZES[case["size"]]
    dtype = TYPES[case["dtype"]]
    g = _generator(seed)
    if case["query"] == 1:
        ctx = _lengths(case, case["context"] + 1, 1)
        q_lens = [1] * len(ctx)
    else:
        q_lens = _lengths(case, case["query"], 16)
        ctx = [n + case["context"] for n in q_lens]
    pages = [-(-n // PAGE) for n in ctx]
    order = torch.randperm(sum(pages), generator=g, device=DEV).to(torch.int32)
    table = torch.zeros(len(ctx), max(pages), dtype=torch.int32, device=DEV)
    at = 0
    for s, n in enumerate(pages):
        table[s, :n] = order[at:at + n]
        at += n
    shape = (sum(pages), kv, PAGE, dim)
    keys, values = _normal(g, *shape, dtype=dtype), _normal(g, *shape, dtype=dtype)
    q = _normal(g, sum(q_lens), heads * dim, dtype=dtype)
    return q, keys, values, table, q_lens, ctx


def _delta_inputs(case, seed):
    width = SIZES[case["size"]][0]
    heads, d = width // 64, 64
    g = _generator(seed)
    lens = _lengths(case, case["query"], 1)
    T = sum(lens)
    proj = _normal(g, T, 5 * width + RANK, dtype=TYPES[case["dtype"]])
    logits = _normal(g, T, width, std=2.0)
    decay_bias, removal_bias = _uniform(g, -6.0, 0.0, width), _uniform(g, -2.0, 2.0, width)
    state = _normal(g, len(lens), heads, d, d, std=0.5)
    return proj, logits, decay_bias, removal_bias, state, lens, heads, d


def _channel_inputs(case, seed):
    width, _, _, d, _ = SIZES[case["size"]]
    heads = width // d
    g = _generator(seed)
    lens = _lengths(case, case["query"], 1)
    T = sum(lens)
    dtype = TYPES[case["dtype"]]
    qkv = _normal(g, T, 3 * width, dtype=dtype)
    logits, beta = _normal(g, T, width, std=2.0), _normal(g, T, heads, dtype=dtype)
    a_log, dt_bias = _uniform(g, -2.0, 1.0, heads), _uniform(g, -4.0, -1.0, width)
    state = _normal(g, len(lens), heads, d, d, std=0.5)
    return qkv, logits, beta, a_log, dt_bias, state, lens, heads, d


def _state_space_inputs(case, seed):
    width = SIZES[case["size"]][0]
    heads = width // STATE_HEAD
    g = _generator(seed)
    lens = _lengths(case, case["query"], 1)
    T = sum(lens)
    dtype = TYPES[case["dtype"]]
    xbc = _normal(g, T, width + 2 * GROUPS * STATE, std=0.5, dtype=dtype)
    dt = _normal(g, T, heads, dtype=dtype)
    dt_bias, a_log, skip = _uniform(g, -3.0, 0.0, heads), _uniform(g, -1.0, 1.5, heads), _uniform(g, 0.9, 1.1, heads)
    state = _normal(g, len(lens), heads, STATE_HEAD, STATE, std=0.5)
    return xbc, dt, dt_bias, a_log, skip, state, lens, heads


def _expert_inputs(case, seed):
    width, _, _, _, ff = SIZES[case["size"]]
    E, F, top, T = case["experts"], ff // 2, case["top"], case["rows"]
    g = _generator(seed)
    x = _normal(g, T, width, dtype=torch.bfloat16)
    gate = _normal(g, E, F, width, std=0.02, dtype=torch.bfloat16)
    up = _normal(g, E, F, width, std=0.02, dtype=torch.bfloat16)
    down = _normal(g, E, width, F, std=0.02, dtype=torch.bfloat16)
    scores = _normal(g, T, E)
    best = scores.topk(top, dim=1)
    return x, gate, up, down, best.indices.to(torch.int32).contiguous(), torch.softmax(best.values, 1).contiguous()


def prepare(case, seed):
    from chibillm_b200.engine.batch import Workspace
    from chibillm_b200.engine.runner import make_runtime
    kind = case["kind"]
    if kind == "serve":
        return _prepare_serve(case, seed)
    k = make_runtime(case.get("dtype", "bfloat16"), DEV)
    s = SimpleNamespace(case=case, kernels=k.kernels)
    if kind == "mlp":
        from chibillm_b200.config.spec import GatedMLPSpec
        from chibillm_b200.parts.base import make_feed_forward
        width, _, _, _, ff = SIZES[case["size"]]
        names = {"gate_proj": "gate", "up_proj": "up", "down_proj": "down"}
        s.part = make_feed_forward(GatedMLPSpec(kind="gated_mlp", hidden_size=width, intermediate_size=ff), names, k)
        x, gate, up, down, s.residual = _mlp_inputs(case, seed)
        s.x = x
        s.part.bind({"gate": gate, "up": up, "down": down})
        s.out = torch.empty_like(s.residual)
        s.ctx = SimpleNamespace(workspace=Workspace(torch.device(DEV)))
    elif kind == "attention":
        s.q, s.keys, s.values, s.table, q_lens, ctx = _attention_inputs(case, seed)
        s.out = torch.empty_like(s.q)
        s.q_start, s.ctx_len = _ints(_starts(q_lens)), _ints(ctx)
        s.seq_of_token = _ints([i for i, n in enumerate(q_lens) for _ in range(n)])
        s.positions = _ints([c - n + j for n, c in zip(q_lens, ctx) for j in range(n)])
        s.most, s.least, s.longest = max(q_lens), min(q_lens), max(ctx)
    elif kind == "experts":
        x, gate, up, down, s.chosen, s.share = _expert_inputs(case, seed)
        s.x, s.down = x, down
        s.up = torch.stack([s.kernels.interleave_expert_gate_up(a, b) for a, b in zip(gate, up)]).contiguous()
        pairs, F, D = s.chosen.numel(), down.shape[2], x.shape[1]
        s.route = torch.empty(s.kernels.route_words(pairs, case["experts"]), dtype=torch.int32, device=DEV)
        s.act = torch.empty(pairs, F, dtype=torch.bfloat16, device=DEV)
        s.y, s.sorted_x = torch.empty(pairs, D, device=DEV), torch.empty(pairs, D, dtype=torch.bfloat16, device=DEV)
        s.out = torch.empty(x.shape[0], D, device=DEV)
    else:
        if kind == "delta_rule":
            s.proj, s.logits, s.decay_bias, s.removal_bias, s.state, lens, s.heads, s.d = _delta_inputs(case, seed)
            s.out = torch.empty_like(s.logits)
        elif kind == "channel_delta":
            s.qkv, s.logits, s.beta, s.a_log, s.dt_bias, s.state, lens, s.heads, s.d = _channel_inputs(case, seed)
            s.out = torch.empty_like(s.logits)
        else:
            s.xbc, s.dt, s.dt_bias, s.a_log, s.skip, s.state, lens, s.heads = _state_space_inputs(case, seed)
            s.out = torch.empty(s.xbc.shape[0], s.heads * STATE_HEAD, device=DEV)
        s.q_start, s.slots, s.most = _ints(_starts(lens)), _ints(list(range(len(lens)))), max(lens)
    return s


def _mlp_inputs(case, seed):
    width, _, _, _, ff = SIZES[case["size"]]
    g = _generator(seed)
    dtype = TYPES[case["dtype"]]
    x = _normal(g, case["rows"], width, dtype=dtype)
    gate, up = _normal(g, ff, width, std=0.02, dtype=dtype), _normal(g, ff, width, std=0.02, dtype=dtype)
    return x, gate, up, _normal(g, width, ff, std=0.02, dtype=dtype), _normal(g, case["rows"], width)


def _prepare_serve(case, seed):
    from chibillm_b200.config.registry import find_architecture
    from chibillm_b200.engine.batch import StepEntry
    from chibillm_b200.engine.model import DecoderModel
    from chibillm_b200.engine.runner import ModelRunner, make_runtime
    config = _qwen3_config(case)
    arch = find_architecture(config)
    spec = arch.model_spec(arch.read_config(config))
    runtime = make_runtime(case["dtype"], DEV, spec=spec)
    model = DecoderModel(spec, runtime)
    model.bind(dict(_qwen3_tensors(case, seed)))
    tokens, lens = _serve_tokens(case, seed)
    runner = ModelRunner(model, runtime, PAGE, pool_tokens=sum(len(t) + PAGE for t in tokens), max_requests=case["requests"])
    plan = [[StepEntry(i, t[:n], [n - 1]) for i, (t, n) in enumerate(zip(tokens, lens))]]
    for j in range(case["steps"]):
        plan.append([StepEntry(i, [t[n + j]], [0]) for i, (t, n) in enumerate(zip(tokens, lens))])
    return SimpleNamespace(case=case, runner=runner, plan=plan)


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s.case["kind"]
    if kind == "serve":
        logits = [s.runner.step(entries, check=False).clone() for entries in s.plan]
        for e in s.plan[0]:
            s.runner.end(e.request_id)
        return logits
    k = s.kernels
    if kind == "mlp":
        s.out.copy_(s.residual)                              # (the residual stream, which the part adds into)
        left = s.part.forward(s.x, s.out, s.ctx)
        if left is not None:
            left.add_into(s.out)
        return s.out
    if kind == "attention":
        _, heads, kv, d, _ = SIZES[s.case["size"]]
        k.attention(s.q, s.keys, s.values, s.out, s.table, s.q_start, s.ctx_len, s.seq_of_token, s.positions, heads, kv, d,
                    PAGE, d ** -0.5, None, s.most, s.longest, min_q_len=s.least, softcap=s.case["softcap"] or None)
        return s.out
    if kind == "experts":
        k.chosen_experts(s.x, s.chosen, s.share, s.up, s.down, s.out, s.route, s.act, s.y, "silu", s.sorted_x, gated=True,
                         interleaved=True, overwrite=True)
        return s.out
    if kind == "delta_rule":
        k.delta_rule(s.proj, s.logits, s.decay_bias, s.removal_bias, s.state, s.out, s.q_start, s.slots, s.heads, s.d, RANK,
                     DECAY_SCALE, KEY_EPS, s.most)
    elif kind == "channel_delta":
        k.channel_delta(s.qkv, s.logits, s.beta, s.a_log, s.dt_bias, s.state, s.out, s.q_start, s.slots, s.heads, s.heads,
                        s.d, s.d, KEY_EPS, s.d ** -0.5, s.most)
    else:
        k.state_space_scan(s.xbc, s.dt, s.dt_bias, s.a_log, s.skip, s.state, s.out, s.q_start, s.slots, s.heads, GROUPS,
                           STATE_HEAD, STATE)
    return s.out, s.state                                    # the requests' states go on from pass to pass


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    width, heads, kv, dim, ff = SIZES[case["size"]]
    size = 2 if case.get("dtype", "bfloat16") == "bfloat16" else 4
    if kind == "serve":
        layer = width * (heads + 2 * kv) * dim + heads * dim * width + 3 * width * ff
        lens = _serve_tokens(case, 0)[1]
        rows = sum(lens)
        steps, live = case["steps"], case["requests"]
        per_key = case["layers"] * 2 * kv * dim * size
        weights = case["layers"] * layer + VOCAB * width
        keys = sum(rows + live * j for j in range(steps + 1))
        pairs = sum(n * (n + 1) / 2 for n in lens) + sum(rows + live * j for j in range(1, steps + 1))
        flops = 2 * case["layers"] * layer * (rows + live * steps) + 2 * VOCAB * width * live * (steps + 1) \
            + 4 * case["layers"] * heads * dim * pairs
        return {"bytes": (steps + 1) * weights * size + keys * per_key + 4 * VOCAB * live * (steps + 1), "flops": flops}
    if kind == "mlp":
        rows = case["rows"]
        return {"bytes": size * (3 * width * ff + rows * width) + 8 * rows * width, "flops": 6 * rows * width * ff}
    if kind == "attention":
        if case["query"] == 1:
            ctx, lens = _lengths(case, case["context"] + 1, 1), [1] * case["seqs"]
        else:
            lens = _lengths(case, case["query"], 16)
            ctx = [n + case["context"] for n in lens]
        pairs = sum(n * (c - n) + n * (n + 1) / 2 for n, c in zip(lens, ctx))
        return {"bytes": size * dim * (2 * kv * sum(ctx) + 2 * heads * sum(lens)), "flops": 4 * heads * dim * pairs}
    if kind == "experts":
        F, pairs = ff // 2, case["rows"] * case["top"]
        used = case["experts"] * (1 - (1 - case["top"] / case["experts"]) ** case["rows"])
        return {"bytes": 2 * 3 * used * width * F + 6 * case["rows"] * width + 8 * pairs, "flops": 6 * pairs * width * F}
    T = sum(_lengths(case, case["query"], 1))
    if kind == "delta_rule":
        return {"bytes": T * (4 * width * size + 8 * width) + 8 * case["seqs"] * width * 64, "flops": 9 * T * width * 64}
    if kind == "channel_delta":
        return {"bytes": T * (3 * width * size + 8 * width) + 8 * case["seqs"] * width * dim, "flops": 7 * T * width * dim}
    return {"bytes": T * ((width + 2 * GROUPS * STATE) * size + 4 * width) + 8 * case["seqs"] * width * STATE,
            "flops": 5 * T * width * STATE}


def tolerance(case):
    """About four times the error against 64-bit arithmetic that the path shows, or the rounding of its types."""
    if case.get("dtype", "bfloat16") == "float32" and case["kind"] in ("serve", "mlp", "attention"):
        return {"rel": 1e-5}
    return {"serve": {"rel": 4e-2}, "mlp": {"rel": 1e-2}, "attention": {"rel": 1e-2}, "experts": {"rel": 1e-2},
            "delta_rule": {"rel": 1e-5}, "channel_delta": {"rel": 1e-5}, "state_space": {"rel": 1e-5}}[case["kind"]]


# ------------------------------------------------------------------ the same in 64 bits
def _exact_serve(case, seed):
    width, heads, kv, dim, _ = SIZES[case["size"]]
    tokens, lens = _serve_tokens(case, seed)
    w = dict(_qwen3_tensors(case, seed))
    ids = torch.tensor([i for t in tokens for i in t], device=DEV)
    sizes = [len(t) for t in tokens]
    starts = _starts(sizes)
    position = torch.cat([torch.arange(n, device=DEV) for n in sizes]).to(torch.float32)
    # (angles as the model defines them: 32-bit position times 32-bit frequency)
    freq = 1.0 / (1000000.0 ** (torch.arange(0, dim, 2, device=DEV, dtype=torch.float64) / dim))
    angle = (position[:, None] * freq.float()).double()
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def norm(x, weight):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * weight.double()

    def linear(x, name):
        return x @ w[name].double().t()

    def rotate(x):
        a, b = x[..., :dim // 2], x[..., dim // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    x = w["model.embed_tokens.weight"][ids].double()
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        h = norm(x, w[p + "input_layernorm.weight"])
        q = rotate(norm(linear(h, p + "self_attn.q_proj.weight").view(-1, heads, dim), w[p + "self_attn.q_norm.weight"]))
        k = rotate(norm(linear(h, p + "self_attn.k_proj.weight").view(-1, kv, dim), w[p + "self_attn.k_norm.weight"]))
        v = linear(h, p + "self_attn.v_proj.weight").view(-1, kv, dim)
        o = torch.cat([_exact_attention(q[a:b], k[a:b], v[a:b], dim ** -0.5, 0.0) for a, b in zip(starts, starts[1:])])
        x = x + linear(o, p + "self_attn.o_proj.weight")
        h = norm(x, w[p + "post_attention_layernorm.weight"])
        x = x + linear(torch.nn.functional.silu(linear(h, p + "mlp.gate_proj.weight")) * linear(h, p + "mlp.up_proj.weight"),
                       p + "mlp.down_proj.weight")
    x = norm(x, w["model.norm.weight"])
    head = w["lm_head.weight" if "lm_head.weight" in w else "model.embed_tokens.weight"].double()
    del w
    return [x[torch.tensor([a + n - 1 + j for a, n in zip(starts, lens)], device=DEV)] @ head.t() for j in range(case["steps"] + 1)]


def _exact_attention(q, k, v, scale, softcap):
    """q [n, heads, d] at the last n places of k, v [keys, kv heads, d]; [n, heads d]."""
    n, heads, d = q.shape
    keys, kv = k.shape[:2]
    group = heads // kv
    hidden = torch.arange(keys, device=DEV)[None] > torch.arange(keys - n, keys, device=DEV)[:, None]
    out = torch.empty(n, heads, d, dtype=torch.float64, device=DEV)
    for h in range(heads):
        s = q[:, h] @ k[:, h // group].t() * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        out[:, h] = torch.softmax(s.masked_fill(hidden, -math.inf), -1) @ v[:, h // group]
    return out.view(n, heads * d)


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return _exact_serve(case, seed)
    if kind == "mlp":
        x, gate, up, down, residual = _mlp_inputs(case, seed)
        x = x.double()
        act = torch.nn.functional.silu(x @ gate.double().t()) * (x @ up.double().t())
        return residual.double() + act @ down.double().t()
    if kind == "attention":
        _, heads, kv, d, _ = SIZES[case["size"]]
        q, keys, values, table, q_lens, ctx = _attention_inputs(case, seed)
        out, at = [], 0
        for s, (n, c) in enumerate(zip(q_lens, ctx)):
            pages = table[s, :-(-c // PAGE)].long()
            k = keys[pages].transpose(1, 2).reshape(-1, kv, d)[:c].double()
            v = values[pages].transpose(1, 2).reshape(-1, kv, d)[:c].double()
            out.append(_exact_attention(q[at:at + n].view(n, heads, d).double(), k, v, d ** -0.5, case["softcap"]))
            at += n
        return torch.cat(out)
    if kind == "experts":
        x, gate, up, down, chosen, share = _expert_inputs(case, seed)
        x = x.double()
        out = torch.zeros_like(x)
        for e in range(case["experts"]):
            t, s = torch.nonzero(chosen == e, as_tuple=True)
            act = torch.nn.functional.silu(x[t] @ gate[e].double().t()) * (x[t] @ up[e].double().t())
            out.index_add_(0, t, share[t, s].double()[:, None] * (act @ down[e].double().t()))
        return out
    return _exact_recurrence(case, seed)


def _exact_recurrence(case, seed):
    """Token by token, all sequences that still have tokens at once."""
    kind = case["kind"]
    if kind == "delta_rule":
        proj, logits, decay_bias, removal_bias, state, lens, H, d = _delta_inputs(case, seed)
        width = H * d
        r, k, v, _, a = (p.double().view(-1, H, d) for p in proj[:, :5 * width].split(width, 1))
        decay = torch.exp(-DECAY_SCALE * torch.sigmoid(logits.double() + decay_bias.double())).view(-1, H, d)
        rate = torch.sigmoid(a + removal_bias.double().view(H, d))
        unit = k / torch.sqrt(k.square().sum(-1, keepdim=True) + KEY_EPS)
        S = state.double()                                   # [seqs, heads, value, key]

        def turn(S, t):
            removed = torch.einsum("shvk,shk->shv", S, unit[t])
            S = S * decay[t][:, :, None] - removed[..., None] * (rate[t] * unit[t])[:, :, None] + v[t][..., None] * k[t][:, :, None]
            return S, torch.einsum("shvk,shk->shv", S, r[t])
    elif kind == "channel_delta":
        qkv, logits, beta, a_log, dt_bias, state, lens, H, d = _channel_inputs(case, seed)
        q, k, v = (p.double().view(-1, H, d) for p in qkv.split(H * d, 1))
        q = q / torch.sqrt(q.square().sum(-1, keepdim=True) + KEY_EPS) * d ** -0.5
        k = k / torch.sqrt(k.square().sum(-1, keepdim=True) + KEY_EPS)
        b = torch.sigmoid(beta.double())
        decay = torch.exp(-a_log.double().exp()[:, None]
                          * torch.nn.functional.softplus(logits.double() + dt_bias.double()).view(-1, H, d))
        S = state.double()                                   # [seqs, heads, key, value]

        def turn(S, t):
            S = S * decay[t][..., None]
            u = b[t][..., None] * (v[t] - torch.einsum("shkv,shk->shv", S, k[t]))
            S = S + k[t][..., None] * u[:, :, None]
            return S, torch.einsum("shkv,shk->shv", S, q[t])
    else:
        xbc, dt, dt_bias, a_log, skip, state, lens, H = _state_space_inputs(case, seed)
        width = H * STATE_HEAD
        x = xbc[:, :width].double().view(-1, H, STATE_HEAD)
        B, C = (p.double().view(-1, GROUPS, STATE).repeat_interleave(H // GROUPS, 1) for p in xbc[:, width:].split(GROUPS * STATE, 1))
        step = torch.nn.functional.softplus(dt.double() + dt_bias.double())
        decay = torch.exp(-a_log.double().exp() * step)
        S = state.double()                                   # [seqs, heads, value, state]

        def turn(S, t):
            S = S * decay[t][..., None, None] + (step[t][..., None] * x[t])[..., None] * B[t][:, :, None]
            return S, torch.einsum("shvn,shn->shv", S, C[t]) + skip.double()[:, None] * x[t]

    starts = torch.tensor(_starts(lens)[:-1], device=DEV)
    out = torch.empty(sum(lens), S.shape[1], S.shape[3] if kind == "channel_delta" else S.shape[2], dtype=torch.float64, device=DEV)
    for j in range(max(lens)):
        live = torch.tensor([i for i, n in enumerate(lens) if n > j], device=DEV)
        t = starts[live] + j
        new, o = turn(S[live], t)
        S[live] = new
        out[t] = o
    return out.reshape(sum(lens), -1), S

"""Workloads of the engine, from a model's weights and given token ids to logits, through the public entry points.

A pass is what a program does with a batch of requests: it admits them, hands the step function (``Engine.step``) their
prompts in portions under a token budget beside one token of every request that is past its prompt (the order that the
scheduler plans in), keeps the float32 logits of every place it asked for, and ends the requests.  Token ids after
the prompt are given too, as when a recorded conversation is replayed or a continuation is scored: two correct
implementations that choose different tokens at a near tie would otherwise not compute the same thing.  The smallest
workload goes through ``LLM.generate`` and returns the tokens that it chose.

Model sizes are the package's own presets.  Weights, token ids and prompts are random, made from a seed.  The designs with
routed experts are left out: in bfloat16 a router's near ties move whole rows of the result, which says nothing about
an implementation; their matrix products, attention and norms are the kernels that are run here.
"""
import json
import math
import os
import random

import numpy as np
import torch

PRESETS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "infer_b200", "models", "presets")
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


def _case(name, model, dtype, requests, shortest, longest, new, budget, how="replay"):
    """requests: how many at once; shortest, longest: the range of their prompts' lengths; new: tokens after the prompt, one
    step each; budget: tokens of a step at most."""
    c = dict(model=model, dtype=dtype, requests=requests, shortest=shortest, longest=longest, new=new, budget=budget, how=how)
    return dict(c, name=name) if name else c


def listed():
    return [
        # The smallest call of all: a tiny model through LLM.generate, greedy, in float32, prompts that cross page boundaries.
        _case("tiny-generate", "tiny-b", "float32", 4, 1, 70, 24, 512, "generate"),
        # The time to the first token of a short question.
        _case("first-token-33", "qwen2.5-1.5b", "bfloat16", 1, 33, 33, 0, 2048),
        # One user in a conversation: a prompt of ordinary, odd length, then single tokens, one request at a time.
        _case("chat-1", "qwen2.5-1.5b", "bfloat16", 1, 301, 301, 64, 2048),
        # The benchmark's batch: eight requests at 2,048-token contexts, decoding together.
        _case("decode-8", "qwen2.5-1.5b", "bfloat16", 8, 2048, 2048, 64, 2048),
        # A half-filled server: a number of requests that is no power of two, with short prompts of different lengths.
        _case("decode-21", "qwen2.5-1.5b", "bfloat16", 21, 20, 400, 48, 1024),
        # A full server: 64 requests of different lengths.
        _case("decode-64", "qwen2.5-1.5b", "bfloat16", 64, 64, 384, 32, 2048),
        # The benchmark's prompt.
        _case("prompt-2048", "qwen2.5-1.5b", "bfloat16", 1, 2048, 2048, 0, 2048),
        # A long document, in portions, of a length that is no multiple of a page or a tile.
        _case("prompt-15873", "qwen2.5-1.5b", "bfloat16", 1, 15873, 15873, 0, 4096),
        # Continuous batching of a larger model: requests decode while others' prompts are still being read in portions of 512.
        _case("serve-7b", "qwen2.5-7b", "bfloat16", 8, 128, 1536, 16, 512),
        # The largest model, one request.
        _case("chat-14b", "qwen2.5-14b", "bfloat16", 1, 1500, 1500, 16, 2048),
        # The true 32-bit path: prompts and single tokens of a few requests.
        _case("float32", "qwen2.5-1.5b", "float32", 3, 100, 300, 8, 512),
        # The design with a recurrence beside attention: prompts, then single tokens.
        _case("recurrence-6", "ruvenex-1.5b", "bfloat16", 6, 200, 700, 32, 2048),
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _cost(c):
    """About the seconds that a pass takes at the rates of the engine's kernels: to keep drawn cases below the largest listed one."""
    w = work(c)
    return w["bytes"] / 3e12 + w["flops"] / (6e14 if c["dtype"] == "bfloat16" else 5e12)


def draw(rng):
    """One more case of the same ranges: sizes of requests, prompts and continuations over their logarithm, every kind of case as
    often as it is listed."""
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(("tiny", "first", "chat", "decode", "decode", "decode", "prompt", "serve", "large", "float32", "recurrence"))
        if kind == "tiny":
            return _case(None, rng.choice(("tiny-a", "tiny-b")), "float32", rng.randint(1, 8), 1, rng.randint(5, 90), rng.randint(8, 32), 512, "generate")
        model, dtype, n, lo, hi, new, budget = "qwen2.5-1.5b", "bfloat16", 1, 1, 1, 0, rng.choice((512, 1024, 2048, 4096))
        if kind == "first":
            lo = hi = _between(rng, 1, 512)
        elif kind == "chat":
            lo = hi = _between(rng, 16, 2048)
            new = _between(rng, 16, 96)
        elif kind == "decode":
            n = _between(rng, 2, 64)
            hi = _between(rng, 32, 2048)
            lo, new = max(1, hi // rng.randint(1, 16)), _between(rng, 16, 96)
        elif kind == "prompt":
            lo = hi = _between(rng, 512, 16000)
        elif kind == "serve":
            model, n, hi, new, budget = "qwen2.5-7b", _between(rng, 2, 12), _between(rng, 128, 2048), _between(rng, 8, 24), rng.choice((512, 1024))
            lo = max(1, hi // 8)
        elif kind == "large":
            model, new = "qwen2.5-14b", _between(rng, 4, 24)
            lo = hi = _between(rng, 64, 2048)
        elif kind == "float32":
            dtype, n, hi, new, budget = "float32", _between(rng, 1, 8), _between(rng, 16, 384), _between(rng, 4, 12), 512
            lo = max(1, hi // 4)
        else:
            model, n, hi, new = "ruvenex-1.5b", _between(rng, 1, 12), _between(rng, 32, 2048), _between(rng, 8, 64)
            lo = max(1, hi // 4)
        c = _case(None, model, dtype, n, lo, hi, new, budget)
        if _cost(c) <= most and n * (new + 1) <= 3000:
            return c


# ------------------------------------------------------------------------------------------------ what a case says

def _config(case):
    with open(os.path.join(PRESETS, case["model"] + ".json"), encoding="utf-8") as f:
        return json.load(f)


def _lengths(case):
    """The prompts' lengths: the case's alone, whatever the seed."""
    r = random.Random("%d %d %d" % (case["requests"], case["shortest"], case["longest"]))
    return [r.randint(case["shortest"], case["longest"]) for _ in range(case["requests"])]


def _steps(case):
    """The steps of a pass. A step is a list of (request, first position, tokens, whether the last place's logits are wanted): one token of
    every request that is past its prompt, then what the budget leaves for prompts, oldest request first."""
    prompts, new = _lengths(case), case["new"]
    at, steps = [0] * len(prompts), []
    while any(a < p + new for a, p in zip(at, prompts)):
        step = [(r, a, 1, True) for r, (a, p) in enumerate(zip(at, prompts)) if p <= a < p + new]
        room = case["budget"] - len(step)
        for r, (a, p) in enumerate(zip(at, prompts)):
            if a < p and room > 0:
                n = min(room, p - a)
                step.append((r, a, n, a + n == p))
                room -= n
        for r, a, n, _ in step:
            at[r] = a + n
        steps.append(step)
    return steps


def _shapes(case, cfg):
    """Every tensor of the model's checkpoint: (name, shape, kind of values)."""
    if case["model"].startswith("ruvenex"):
        W, V = cfg["width"], cfg["vocab"]
        out = [("embed", (V, W), "matrix"), ("head", (V, W), "matrix"), ("final.norm", (W,), "norm")]
        for i, l in enumerate(cfg["layers"]):
            p, a, r, ff = "l%d." % i, l["mixer"]["left"], l["mixer"]["right"], l["mlp"]["ff"]
            for x, n in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"])):
                out += [(p + "mix.left." + x, (n, W), "matrix"), (p + "mix.left." + x + ".conv", (n, a["conv"]), "filter")]
            out += [(p + "norm1", (W,), "norm"), (p + "mix.left.g", (a["heads"], W), "matrix"), (p + "mix.left.o", (W, a["heads"] * a["vdim"]), "matrix")]
            nq, nv = r["heads"] * r["dim"], r["heads"] * r["vdim"]
            out += [(p + "mix.right.q", (nq, W), "matrix"), (p + "mix.right.f", (nq, W), "matrix"), (p + "mix.right.f.b", (nq,), "wide"),
                    (p + "mix.right.lower", (nq,), "bound"), (p + "mix.right.v", (nv, W), "matrix"), (p + "mix.right.norm", (r["vdim"],), "norm"),
                    (p + "mix.right.o", (W, nv), "matrix"), (p + "mlp.up", (ff, W), "matrix"), (p + "mlp.down", (W, ff), "matrix")]
            for g in ("rg1", "rg2"):
                out += [(p + g, (W, W), "matrix"), (p + g + ".b", (W,), "bias")]
        return out
    H, I, V = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"]
    hd = H // cfg["num_attention_heads"]
    out = [("model.embed_tokens.weight", (V, H), "table"), ("model.norm.weight", (H,), "norm")]
    if not cfg["tie_word_embeddings"]:
        out.append(("lm_head.weight", (V, H), "matrix"))
    for i in range(cfg["num_hidden_layers"]):
        p = "model.layers.%d." % i
        for x, n in (("q", cfg["num_attention_heads"] * hd), ("k", cfg["num_key_value_heads"] * hd), ("v", cfg["num_key_value_heads"] * hd)):
            out += [(p + "self_attn.%s_proj.weight" % x, (n, H), "matrix"), (p + "self_attn.%s_proj.bias" % x, (n,), "bias")]
        out += [(p + "self_attn.o_proj.weight", (H, H), "into"), (p + "mlp.gate_proj.weight", (I, H), "matrix"),
                (p + "mlp.up_proj.weight", (I, H), "matrix"), (p + "mlp.down_proj.weight", (H, I), "into"),
                (p + "input_layernorm.weight", (H,), "norm"), (p + "post_attention_layernorm.weight", (H,), "norm")]
    return out


def _weights(case, cfg, seed):
    """The checkpoint, as models are initialised: matrices N(0, 0.02) at 1,536 features (rows longer than that smaller in proportion), the two
    of a layer that add to the stream divided by the root of how many do, a token table that the layers' sum outgrows two- to threefold, norm
    weights 1 + N(0, 0.1), filters that keep a channel's scale, bounds in [0, 0.9). (Without the second and third, a bfloat16 pass of 48 layers
    is 8 % off the exact one, whatever the implementation.)"""
    dtype = DTYPES[case["dtype"]]
    size = 0.8 / math.sqrt(cfg.get("hidden_size") or cfg["width"])
    spread = {"matrix": size, "into": size / math.sqrt(2.0 * (cfg.get("num_hidden_layers") or 1)), "table": 0.25, "bias": 0.02, "norm": 0.1,
              "filter": 0.3, "wide": 1.0}
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    out = {}
    for name, shape, kind in _shapes(case, cfg):
        w = torch.empty(shape, dtype=dtype, device="cuda")
        if kind == "bound":
            w.uniform_(0.0, 0.9, generator=gen)
        else:
            w.normal_(1.0 if kind == "norm" else 0.0, spread[kind], generator=gen)
            if kind == "filter":
                w[:, -1] += 1.0
        out[name] = w
    return out


def _tokens(case, cfg, seed):
    """The token ids of every request: its prompt and, for a replay, its continuation."""
    rng = np.random.default_rng(int(seed))
    V = cfg.get("vocab_size") or cfg["vocab"]
    more = 0 if case["how"] == "generate" else case["new"]
    return [rng.integers(0, V, n + more).tolist() for n in _lengths(case)]


def prepare(case, seed):
    """A loaded model and its cache, the requests' token ids, and a place for the logits."""
    from infer_b200 import LLM, Engine, StepEntry
    from infer_b200.config import parse_config
    import infer_b200.models  # noqa: F401  (registers the architectures)
    cfg = _config(case)
    arch, typed = parse_config(cfg)
    spec = arch.to_spec(typed)
    weights, tokens = _weights(case, cfg, seed), _tokens(case, cfg, seed)
    longest = case["longest"] + case["new"]
    if case["how"] == "generate":
        llm = LLM(None, dtype=case["dtype"], spec=spec, weights=weights, slots=case["requests"], max_seq=longest, max_batch_tokens=case["budget"])
        return {"llm": llm, "prompts": tokens, "new": case["new"]}
    room = sum(-(-(n + case["new"]) // 16) * 16 for n in _lengths(case))
    engine = Engine(spec, weights, dtype=case["dtype"], max_tokens=room, max_requests=case["requests"], max_seq_len=longest)
    steps, rows = [], 0
    for step in _steps(case):
        entries = [StepEntry(r, tokens[r][a:a + n], [n - 1] if want else []) for r, a, n, want in step]
        wanted = sum(want for _, _, _, want in step)
        steps.append((entries, rows, rows + wanted))
        rows += wanted
    logits = torch.empty((rows, spec.vocab_size), dtype=torch.float32, device="cuda")
    return {"engine": engine, "requests": range(case["requests"]), "steps": steps, "logits": logits}


def run(state):
    if "llm" in state:
        return np.array(state["llm"].generate(state["prompts"], max_new=state["new"], eos_id=-1))
    engine, logits = state["engine"], state["logits"]
    for r in state["requests"]:
        engine.add_request(r)
    for entries, first, end in state["steps"]:
        out = engine.step(entries)
        if end > first:
            logits[first:end].copy_(out)
    for r in state["requests"]:
        engine.end_request(r)
    return logits


# ------------------------------------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Every step reads the weights once (a later step is another call), the earlier positions of its requests once, and a
    recurrence's state; it writes new positions and the wanted logits. Operations: the matrix products of every token, the output
    matrix where logits are wanted, scores and sums of attention over the positions that a token sees."""
    cfg = _config(case)
    item = 2 if case["dtype"] == "bfloat16" else 4
    ruvenex = case["model"].startswith("ruvenex")
    shapes = _shapes(case, cfg)
    table = "embed" if ruvenex else "model.embed_tokens.weight"
    layers = [(n, s) for n, s, _ in shapes if n not in (table, "head", "lm_head.weight")]
    per_token = 2 * sum(s[0] * s[1] for _, s in layers if len(s) == 2)
    weight_bytes = item * sum(math.prod(s) for _, s in layers)
    state = 0
    if ruvenex:
        V, H, n_layers, a, r = cfg["vocab"], cfg["width"], len(cfg["layers"]), cfg["layers"][0]["mixer"]["left"], cfg["layers"][0]["mixer"]["right"]
        heads, dims, kv = a["heads"], a["dim"] + a["vdim"], a["kv_heads"] * (a["dim"] + a["vdim"])
        state = n_layers * r["heads"] * r["dim"] * r["vdim"]
        per_token += 5 * state
    else:
        V, H, n_layers, heads = cfg["vocab_size"], cfg["hidden_size"], cfg["num_hidden_layers"], cfg["num_attention_heads"]
        dims = 2 * (H // heads)
        kv = cfg["num_key_value_heads"] * dims
    total_bytes = total_flops = 0
    for step in _steps(case) if case["how"] == "replay" else _generate_steps(case):
        wanted = sum(w for _, _, _, w in step)
        total_bytes += weight_bytes + (V * H * item if wanted else 0) + 4 * V * wanted
        total_flops += 2 * V * H * wanted
        for _, first, n, _ in step:
            total_bytes += H * item * n + n_layers * kv * item * (first + n) + 8 * state
            total_flops += per_token * n + 2 * heads * dims * n_layers * (n * first + n * (n + 1) // 2)
    return {"bytes": total_bytes, "flops": total_flops}


def _generate_steps(case):
    """All prompts in one step, then one token of every request per step: each prompt's last place already chooses a token."""
    prompts = _lengths(case)
    yield [(r, 0, n, True) for r, n in enumerate(prompts)]
    for i in range(case["new"] - 1):
        yield [(r, n + i, 1, True) for r, n in enumerate(prompts)]


def tolerance(case):
    if case["how"] == "generate":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 2e-5}
    return {"rel": 0.02}


# ------------------------------------------------------------------------------------------------ the same in 64 bits

F = torch.float64


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _linear(x, w, b=None, rows=4096):
    w = w.to(F).T
    y = torch.cat([x[i:i + rows] @ w for i in range(0, x.shape[0], rows)])
    return y if b is None else y + b.to(F)


def _attention(q, k, v, scale):
    """q [T, H, d], k [T, G, d], v [T, G, dv] of one request -> [T, H, dv]: position t sees positions up to t."""
    T, H, _ = q.shape
    G = k.shape[1]
    out = torch.empty((T, H, v.shape[2]), dtype=F, device=q.device)
    for i in range(0, T, 1024):
        j = min(T, i + 1024)
        unseen = torch.arange(j, device=q.device)[None, :] > torch.arange(i, j, device=q.device)[:, None]
        for h in range(H):
            g = h // (H // G)
            s = (q[i:j, h] @ k[:j, g].T * scale).masked_fill_(unseen, float("-inf"))
            out[i:j, h] = torch.softmax(s, dim=-1) @ v[:j, g]
    return out


def _angles(base, dims, position, exponents):
    """Rotation angles: both designs state them as float32 products of position and frequency; their cosines and sines."""
    freq = 1.0 / torch.pow(torch.tensor(float(base), dtype=torch.float32), exponents) if exponents.dtype == torch.float32 else \
        torch.pow(torch.tensor(float(base), dtype=F), -exponents).to(torch.float32)
    a = (position.cpu().to(torch.float32)[:, None] * freq[None, :]).to(F).to(position.device)
    return torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]


def _qwen2(cfg, W, ids, position, spans):
    """The stream after the last norm, for the rows of all requests (spans: each request's first row and end)."""
    nh, nkv, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["rms_norm_eps"]
    hd = cfg["hidden_size"] // nh
    cos, sin = _angles(cfg["rope_theta"], hd, position, torch.arange(hd // 2, dtype=torch.float32) * 2.0 / float(hd))

    def turn(x):
        a, b = x[..., :hd // 2], x[..., hd // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)
    h = W["model.embed_tokens.weight"][ids].to(F)
    for i in range(cfg["num_hidden_layers"]):
        p = "model.layers.%d." % i
        n = _rms(h, eps) * W[p + "input_layernorm.weight"].to(F)
        q, k, v = (_linear(n, W[p + "self_attn.%s_proj.weight" % x], W[p + "self_attn.%s_proj.bias" % x]).view(len(ids), -1, hd) for x in "qkv")
        q, k = turn(q), turn(k)
        ctx = torch.cat([_attention(q[a:b], k[a:b], v[a:b], 1.0 / math.sqrt(hd)) for a, b in spans])
        h = h + _linear(ctx.reshape(len(ids), -1), W[p + "self_attn.o_proj.weight"])
        n = _rms(h, eps) * W[p + "post_attention_layernorm.weight"].to(F)
        g = _linear(n, W[p + "mlp.gate_proj.weight"])
        g = g / (1.0 + torch.exp(-g)) * _linear(n, W[p + "mlp.up_proj.weight"])
        h = h + _linear(g, W[p + "mlp.down_proj.weight"])
    return _rms(h, eps) * W["model.norm.weight"].to(F)


def _filtered(u, w, spans):
    """y[t] = sum_j w[:, j] u[t - (taps - 1) + j] within each request, zeros before it."""
    w, y = w.to(F), torch.zeros_like(u)
    taps = w.shape[1]
    for a, b in spans:
        for j in range(taps):
            back = taps - 1 - j
            if b - a > back:
                y[a + back:b] += u[a:b - back] * w[:, j]
    return y


def _recurrence(q, f, v, spans):
    """S <- diag(f) S + (1 - f) v^T, o = S^T q per request and head; requests side by side, the shorter ones padded behind their end."""
    n, longest = len(spans), max(b - a for a, b in spans)
    side = [torch.zeros((longest, n) + x.shape[1:], dtype=F, device=x.device) for x in (q, f, v)]
    for x, y in zip((q, f, v), side):
        for r, (a, b) in enumerate(spans):
            y[:b - a, r] = x[a:b]
    q2, f2, v2 = side
    S = torch.zeros((n,) + q.shape[1:] + (v.shape[2],), dtype=F, device=q.device)
    o = torch.empty_like(v2)
    for t in range(longest):
        S = torch.addcmul((1.0 - f2[t])[..., None] * v2[t][:, :, None, :], f2[t][..., None], S)
        o[t] = torch.matmul(q2[t][:, :, None, :], S)[:, :, 0]
    return torch.cat([o[:b - a, r] for r, (a, b) in enumerate(spans)])


def _ruvenex(cfg, W, ids, position, spans):
    eps, T = cfg["norm"]["eps"], len(ids)
    x = W["embed"][ids].to(F) * cfg["embedding"]["scale"]
    for i, l in enumerate(cfg["layers"]):
        p, a, r = "l%d." % i, l["mixer"]["left"], l["mixer"]["right"]
        n = _rms(x, eps) * W[p + "norm1"].to(F)
        q, k, v = (_filtered(_linear(n, W[p + "mix.left." + c]), W[p + "mix.left." + c + ".conv"], spans) for c in "qkv")
        q, k, v = q.view(T, -1, a["dim"]), k.view(T, -1, a["dim"]), _rms(v.view(T, -1, a["vdim"]), eps)
        m = a["rot"]["dims"]
        cos, sin = _angles(a["rot"]["base"], m, position, 2.0 * torch.arange(m // 2, dtype=F) / m)
        for y in (q, k):
            even, odd = y[..., 0:m:2].clone(), y[..., 1:m:2].clone()
            y[..., 0:m:2], y[..., 1:m:2] = even * cos - odd * sin, odd * cos + even * sin
        ctx = torch.cat([_attention(q[s:e], k[s:e], v[s:e], a["scale"]) for s, e in spans])
        ctx = ctx * torch.sigmoid(_linear(n, W[p + "mix.left.g"]))[:, :, None]
        left = _linear(ctx.reshape(T, -1), W[p + "mix.left.o"])
        z = _linear(n, W[p + "mix.right.q"])
        low = W[p + "mix.right.lower"].to(F)
        f = low + (1.0 - low) * torch.sigmoid(_linear(n, W[p + "mix.right.f"], W[p + "mix.right.f.b"]))
        o = _recurrence((z * torch.sigmoid(z)).view(T, r["heads"], r["dim"]), f.view(T, r["heads"], r["dim"]),
                        _linear(n, W[p + "mix.right.v"]).view(T, r["heads"], r["vdim"]), spans)
        right = _linear((_rms(o, eps) * W[p + "mix.right.norm"].to(F)).reshape(T, -1), W[p + "mix.right.o"])
        z = _linear(n, W[p + "mlp.up"])
        z = 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))
        gate = [torch.sigmoid(_linear(n, W[p + g], W[p + g + ".b"])) for g in ("rg1", "rg2")]
        x = x + gate[0] * (l["mixer"]["left_scale"] * left + l["mixer"]["right_scale"] * right) + gate[1] * _linear(z, W[p + "mlp.down"])
    return _rms(x, eps) * W["final.norm"].to(F)


def _logits(case, cfg, W, tokens, wanted):
    """The logits of (request, position) pairs of whole sequences."""
    spans, at = [], 0
    for t in tokens:
        spans.append((at, at + len(t)))
        at += len(t)
    ids = torch.tensor([x for t in tokens for x in t], device="cuda")
    position = torch.cat([torch.arange(len(t), device="cuda") for t in tokens])
    ruvenex = case["model"].startswith("ruvenex")
    rows = (_ruvenex if ruvenex else _qwen2)(cfg, W, ids, position, spans)
    rows = rows[torch.tensor([spans[r][0] + p for r, p in wanted], device="cuda")]
    head = W["head"] if ruvenex else W["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"]
    return torch.cat([_linear(rows, head[i:i + 32768]) for i in range(0, head.shape[0], 32768)], dim=1)


@torch.no_grad()
def exact(case, seed):
    """What ``run`` returns, from whole sequences in float64: no cache, no portions."""
    cfg = _config(case)
    W, tokens = _weights(case, cfg, seed), _tokens(case, cfg, seed)
    if case["how"] == "generate":
        tokens, chosen = [list(t) for t in tokens], [[] for _ in tokens]
        for _ in range(case["new"]):
            best = _logits(case, cfg, W, tokens, [(r, len(t) - 1) for r, t in enumerate(tokens)]).argmax(dim=1).tolist()
            for t, c, b in zip(tokens, chosen, best):
                t.append(b)
                c.append(b)
        return np.array(chosen)
    return _logits(case, cfg, W, tokens, [(r, a + n - 1) for step in _steps(case) for r, a, n, want in step if want])

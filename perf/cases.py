"""The engine's work as its users give it: prompts, decoding, bursts of requests, over model sizes and types.

A case is a dict of plain values; `prepare` builds the engine with random weights and brings the requests to where the
pass begins, `run` makes one pass through the public entry points (`Engine.step`, `DecodeGraphPool`), `exact` says in plain
torch and 64 bits what the logits are.  Four kinds of pass:

  prompt   whole prompts in one `Engine.step`, the last place's logits of each (time to the first token)
  decode   a few steps of a captured decode step: the tokens go up, the step is replayed, the selected tokens come back, as in
           `LLM.step`; what the model is fed next is given (scoring a known continuation), so that a pass can be repeated
  burst    requests through a budget of tokens a step: portions of prompts beside the decoded tokens of the requests before
           them, one `Engine.step` each, which is what the scheduler makes of a burst of requests
  turn     prompts in one step, then captured decode steps of the same requests (models whose state moves on with every token)

Logits are kept through the step's tensor sink, the trace's own way to them; each step's are copied once.
"""
import math
import random
import zlib

import numpy as np
import torch

# ------------------------------------------------------------------------------------------------------ the cases
BF16, FP32 = "bfloat16", "float32"
F = torch.float64


def _case(kind, model, dtype, batch, low, high, steps=0, page=64, budget=0, top_k=0, spread=1):
    """`batch` requests with prompts of low..high tokens (`spread` draws the lengths), `steps` decode steps behind them,
    `budget` tokens a step in a burst, `top_k` > 0: seeded sampling among that many at temperature 0.8, else greedy."""
    return {"kind": kind, "model": model, "dtype": dtype, "batch": batch, "low": low, "high": high, "steps": steps, "page": page,
            "budget": budget, "top_k": top_k, "spread": spread}


def listed():
    named = {
        # one person at a chat: the shortest step there is; latency and launches decide
        "decode one": _case("decode", "qwen2.5-1.5b", BF16, 1, 317, 317, steps=8, page=16),
        # the headline shape: eight requests with 2,048-token prompts
        "decode 8 at 2048": _case("decode", "qwen2.5-1.5b", BF16, 8, 2048, 2048, steps=8),
        # a server in the middle of its day: an odd number of requests of all ages, sampled
        "decode 41 ragged": _case("decode", "qwen2.5-1.5b", BF16, 41, 64, 2048, steps=4, top_k=50),
        # few long conversations on the larger model: weights and cache both stream
        "decode long 7b": _case("decode", "qwen2.5-7b", BF16, 4, 6144, 6144, steps=4),
        # a short question: time to the first token of 45 tokens
        "prompt 45": _case("prompt", "qwen2.5-1.5b", BF16, 1, 45, 45, page=16),
        # the headline prompt
        "prompt 2048": _case("prompt", "qwen2.5-1.5b", BF16, 1, 2048, 2048),
        # requests of assorted lengths arriving at once, prompts in portions of 512 beside decoded tokens
        "burst 7b": _case("burst", "qwen2.5-7b", BF16, 9, 128, 1536, budget=512),
        # the 32-bit path, with which people check a model or a checkpoint: a prompt, and decoding
        "prompt 333 float32": _case("prompt", "qwen2.5-1.5b", FP32, 1, 333, 333, page=16),
        "decode 2 float32": _case("decode", "qwen2.5-1.5b", FP32, 2, 300, 300, steps=4, page=16),
        # latent attention with routed experts: a prompt, and decoding
        "latent experts prompt": _case("prompt", "gedalix-16b-layers", BF16, 1, 2048, 2048),
        "latent experts decode": _case("decode", "gedalix-16b-layers", BF16, 8, 500, 2048, steps=8),
        # attention beside a gated delta rule: four questions answered at once
        "delta rule turn": _case("turn", "matidra-3b-layers", BF16, 4, 200, 1000, steps=8),
    }
    return [dict(case, name=name) for name, case in named.items()]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    spread = rng.randrange(1, 1 << 20)
    page = rng.choice((16, 64))
    what = rng.choice(("decode", "decode", "decode", "prompt", "prompt", "burst", "float32", "latent", "delta"))
    if what == "decode":
        model = rng.choice(("qwen2.5-1.5b", "qwen2.5-1.5b", "qwen2.5-7b"))
        batch = _spread(rng, 1, 64)
        high = _spread(rng, 64, max(128, min(6144, 24000 // batch)))
        return _case("decode", model, BF16, batch, max(32, int(high * rng.uniform(0.1, 1.0))), high, steps=4, page=page,
                     top_k=rng.choice((0, 0, 50)), spread=spread)
    if what == "prompt":
        batch = rng.choice((1, 1, 1, 2, 5))
        high = max(16, _spread(rng, 16, 3000) // batch)
        return _case("prompt", rng.choice(("qwen2.5-1.5b", "qwen2.5-7b")), BF16, batch, max(8, int(high * rng.uniform(0.3, 1.0))), high,
                     page=page, spread=spread)
    if what == "burst":
        return _case("burst", rng.choice(("qwen2.5-1.5b", "qwen2.5-7b")), BF16, rng.randint(3, 9), 64, _spread(rng, 256, 1400),
                     budget=rng.choice((256, 512, 1024)), page=page, spread=spread)
    if what == "float32":
        high = _spread(rng, 16, 500)
        if rng.random() < 0.5:
            return _case("prompt", "qwen2.5-1.5b", FP32, 1, high, high, page=page, spread=spread)
        return _case("decode", "qwen2.5-1.5b", FP32, rng.randint(1, 8), max(16, high // 2), high, steps=4, page=page, spread=spread)
    if what == "latent":
        if rng.random() < 0.5:
            high = _spread(rng, 100, 2048)
            return _case("prompt", "gedalix-16b-layers", BF16, 1, high, high, page=page, spread=spread)
        high = _spread(rng, 100, 2048)
        return _case("decode", "gedalix-16b-layers", BF16, _spread(rng, 1, 32), max(50, high // 3), high, steps=4, page=page, spread=spread)
    high = _spread(rng, 100, 1500)
    return _case("turn", "matidra-3b-layers", BF16, rng.randint(1, 8), max(50, high // 4), high, steps=rng.choice((4, 8)), page=page, spread=spread)


# ---------------------------------------------------------------------------------------- what a case holds, in numbers
def _prompt_lengths(case):
    rng = random.Random(case["spread"])
    return [case["high"] if case["low"] == case["high"] else _spread(rng, case["low"], case["high"]) for _ in range(case["batch"])]


def _burst_plan(case):
    """Steps as lists of (request, first place, count, whether the last place's logits are wanted): every step decodes a token of
    each request whose prompt is in, then fills the budget with portions of the prompts that wait; ends with the last prompt."""
    prompts = _prompt_lengths(case)
    done = [0] * len(prompts)
    plan = []
    while any(d < n for d, n in zip(done, prompts)):
        step, left = [], case["budget"]
        for i, n in enumerate(prompts):
            if done[i] >= n:
                step.append((i, done[i], 1, True))
                done[i] += 1
                left -= 1
        for i, n in enumerate(prompts):
            if done[i] < n and left > 0 and not any(s[0] == i for s in step):
                count = min(left, n - done[i])
                step.append((i, done[i], count, done[i] + count == n))
                done[i] += count
                left -= count
        plan.append(step)
    return plan, done


def _total_lengths(case):
    if case["kind"] == "burst":
        return _burst_plan(case)[1]
    return [n + case["steps"] for n in _prompt_lengths(case)]


def _config(case):
    from microllm_rocm_b200.config import find_preset
    return find_preset(case["model"])[1]


def _token_ids(case, seed, vocab):
    rng = np.random.RandomState((int(seed) * 7919 + 13) % (1 << 31))
    return [rng.randint(0, vocab, n).tolist() for n in _total_lengths(case)]


# ------------------------------------------------------------------------------------------------------ the weights
class _Weights:
    """Random weights: a tensor's values follow from the seed and its name."""

    def __init__(self, seed, dtype):
        self.seed, self.dtype = int(seed), torch.bfloat16 if dtype == BF16 else torch.float32

    def tensor(self, name, shape):
        """The tensor as a checkpoint of this type holds it."""
        std, one = self.kind(name)
        generator = torch.Generator("cuda").manual_seed((self.seed << 32) + zlib.crc32(name.encode()))
        out = torch.empty(shape, dtype=self.dtype, device="cuda").normal_(0.0, std, generator=generator)
        return out.add_(1.0) if one else out

    def __call__(self, name, *shape):
        return self.tensor(name, shape).to(F)

    @staticmethod
    def kind(name):
        """(standard deviation, whether one is added) of a tensor.  A router's weights are those of one that is sure of its choice,
        as trained ones are: between experts that weigh the same, rounding to bf16 would choose."""
        last = name.rsplit(".", 1)[-1]
        if name.endswith(("norm1.b", "norm2.b", "final.norm.b", "a2", "g2")):
            return 0.1, False
        if last == "router":
            return 0.08, False
        if last == "sink":
            return 1.0, False
        if last in ("conv", "A_log", "dt_bias"):
            return 0.5, False
        if last in ("norm", "norm1", "norm2", "ls1", "ls2") or name.endswith("norm.weight"):
            return 0.1, True
        return 0.02, False


def _engine(case, cfg, seed, pages):
    from microllm_rocm_b200.config.registry import architecture_for
    from microllm_rocm_b200.engine.loading import make_engine, prepare_kernels, require_gpu, resolve_dtype
    from microllm_rocm_b200.parts.base import Runtime
    from microllm_rocm_b200.parts.build import build_model
    model = build_model(architecture_for(cfg).build_spec(cfg), Runtime(require_gpu(), resolve_dtype(case["dtype"])))
    prepare_kernels(model)
    weights = _Weights(seed, case["dtype"])
    made = {}
    for name, spec in model.expected_tensors().items():
        made[name] = weights.tensor(name, tuple(spec.shape))
        if spec.role == "vector":
            made[name] = made[name].float()
    model.bind(made)
    return make_engine(model, case["page"], pages, max(64, case["batch"]))


# ------------------------------------------------------------------------------------------------------ preparation
class State:
    pass


def _steps_of_prompts(engine, ids, prompts, portion=2048):
    """Bring the prompts into the cache, a portion of one of them a step."""
    from microllm_rocm_b200.engine.step import StepEntry
    for rid, prompt in zip(ids, prompts):
        for at in range(0, len(prompt), portion):
            engine.step([StepEntry(rid, prompt[at:at + portion], [])])


def _load(s):
    s.graph.load(s.ids, [t[n] for t, n in zip(s.tokens, s.lengths)], s.lengths, s.configs, [0] * len(s.ids))


def _capture(s):
    """The captured decode step of these requests, its logits kept."""
    from microllm_rocm_b200.engine.decode_graph import DecodeGraphPool
    steps = s.case["steps"]
    for rid, n in zip(s.ids, s.lengths):
        if not s.engine.cache.reserve(rid, n + steps):
            raise RuntimeError("no pages for the requests")
    s.pool = DecodeGraphPool(s.engine)
    s.graph = s.pool.get(s.ids, headroom_tokens=steps)
    s.kept = {}
    s.graph.ctx.tensor_sink = lambda name, tensor: s.kept.__setitem__(name, tensor) if name == "logits" else None
    _load(s)
    s.pool.ensure_captured(s.graph)


def prepare(case, seed):
    from microllm_rocm_b200.sampling import GenerationConfig
    s = State()
    s.case, cfg = case, _config(case)
    s.lengths = _prompt_lengths(case)
    s.tokens = _token_ids(case, seed, cfg.vocab_size)
    pages = sum(-(-len(t) // case["page"]) for t in s.tokens) + 2
    s.engine = _engine(case, cfg, seed, pages)
    s.ids = [f"request {i}" for i in range(case["batch"])]
    s.configs = [GenerationConfig(max_new_tokens=1 + case["steps"], temperature=0.8 if case["top_k"] else 0.0, top_k=case["top_k"], seed=i)
                 for i in range(case["batch"])]
    if case["kind"] == "decode":
        for rid in s.ids:
            s.engine.cache.add(rid)
        _steps_of_prompts(s.engine, s.ids, [t[:n] for t, n in zip(s.tokens, s.lengths)])
        _capture(s)
    elif case["kind"] == "turn":
        _prompt_pass(s)
        _capture(s)
        for rid in s.ids:
            s.engine.cache.release(rid)
    elif case["kind"] == "burst":
        s.plan = _burst_plan(case)[0]
    return s


# ------------------------------------------------------------------------------------------------------ one pass
def _prompt_pass(s):
    from microllm_rocm_b200.engine.step import StepEntry
    for rid in s.ids:
        s.engine.cache.add(rid)
    return s.engine.step([StepEntry(rid, t[:n], [n - 1]) for rid, t, n in zip(s.ids, s.tokens, s.lengths)])


def _decode_pass(s):
    batch, picked, logits = len(s.ids), [], []
    _load(s)
    for k in range(s.case["steps"]):
        if k:
            s.graph.upload_tokens([t[n + k] for t, n in zip(s.tokens, s.lengths)])
        s.graph.replay()
        logits.append(s.kept["logits"][:batch].clone())
        picked.append(s.graph.read_tokens())
    return {"tokens": np.array(picked, dtype=np.int64), "logits": logits}


def run(state):
    from microllm_rocm_b200.engine.step import StepEntry
    s = state
    kind, cache = s.case["kind"], s.engine.cache
    if kind == "decode":
        return _decode_pass(s)
    if kind == "prompt":
        out = _prompt_pass(s)
    elif kind == "turn":
        prompt = _prompt_pass(s)
        for rid, n in zip(s.ids, s.lengths):
            cache.reserve(rid, n + s.case["steps"])
        out = dict(_decode_pass(s), prompt=prompt)
    else:
        for rid in s.ids:
            cache.add(rid)
        out = []
        for step in s.plan:
            logits = s.engine.step([StepEntry(s.ids[i], s.tokens[i][a:a + n], [n - 1] if wants else []) for i, a, n, wants in step])
            if any(wants for _, _, _, wants in step):
                out.append(logits)
    for rid in s.ids:
        cache.release(rid)
    return out


# ---------------------------------------------------------------------- what a pass cannot do without (bytes, operations)
def _model_numbers(case):
    """(weights every step reads, bytes of a cached token over all layers, operations of a token's products, operations of one
    (token, key) pair over all layers, (experts, chosen, bytes of one, operations of one, layers) or None, head elements)."""
    cfg, item = _config(case), 2 if case["dtype"] == BF16 else 4
    if case["model"].startswith("qwen"):
        h, d, layers = cfg.hidden_size, cfg.head_size, cfg.num_hidden_layers
        q, kv = cfg.num_attention_heads * d, cfg.num_key_value_heads * d
        n = layers * (h * (q + 2 * kv) + q * h + 3 * h * cfg.intermediate_size)
        return n * item, layers * 2 * kv * item, 2 * n, layers * 4 * q, None, cfg.vocab_size * h
    raw = cfg.to_dict()
    h, n, row, pair, experts = raw["width"], 0, 0, 0, None
    for layer in raw["layers"]:
        m, mlp = layer["mixer"], layer["mlp"]
        if layer["type"] == "latent_attention":
            H, dk, r = m["heads"], m["dim"] + m["rot_dim"], m["kv_rank"]
            n += h * (H * dk + r + m["rot_dim"]) + r * H * (m["dim"] + m["vdim"]) + 2 * H * m["vdim"] * h + h * mlp["router"]["experts"]
            n += 3 * h * mlp["shared"]["ff"]
            row += (r + m["rot_dim"]) * item
            pair += 2 * H * (dk + m["vdim"])          # the cheaper of the two forms, keys and values per head
            one = 3 * h * mlp["expert"]["ff"]
            experts = (mlp["router"]["experts"], mlp["router"]["top"], one * item, 2 * one, (experts[4] if experts else 0) + 1)
            continue
        soft = m["left"] if layer["type"] == "parallel" else m
        q, k, v = soft["heads"] * soft["dim"], soft["kv_heads"] * soft["dim"], soft["kv_heads"] * soft["vdim"]
        o = soft["heads"] * soft["vdim"]
        n += h * (q + k + o) + 3 * h * mlp["ff"]
        row += (k + v) * item
        pair += 2 * (q + o)
        if layer["type"] == "parallel":
            r = m["right"]
            q, o = r["kv_heads"] * r["dim"], r["heads"] * r["vdim"]
            n += h * (v + o) + h * (2 * q + 2 * o + r["heads"]) + (h + r["heads"] * r["dim"]) * r["a_rank"] + (h + o) * r["g_rank"]
            n += 3 * r["heads"] * r["dim"] * r["vdim"]                # a token's update of the state and its read-out
    return n * item, row, 2 * n, pair, experts, raw["vocab"] * h


def work(case):
    weights, row, flops, pair, experts, head = _model_numbers(case)
    item = 2 if case["dtype"] == BF16 else 4
    vocab = _config(case).vocab_size
    lengths = _prompt_lengths(case)
    steps = []                                          # per step: (tokens, (token, key) pairs, cached tokens read, wanted rows)
    if case["kind"] in ("prompt", "turn"):
        steps.append((sum(lengths), sum(n * (n + 1) // 2 for n in lengths), sum(lengths), len(lengths)))
    if case["kind"] in ("decode", "turn"):
        for k in range(case["steps"]):
            keys = sum(n + k + 1 for n in lengths)
            steps.append((len(lengths), keys, keys, len(lengths)))
    if case["kind"] == "burst":
        for step in _burst_plan(case)[0]:
            steps.append((sum(s[2] for s in step), sum(s[2] * s[1] + s[2] * (s[2] + 1) // 2 for s in step), sum(s[1] + s[2] for s in step),
                          sum(1 for s in step if s[3])))
    total = {"bytes": 0.0, "flops": 0.0}
    for tokens, pairs, keys, rows in steps:
        total["bytes"] += weights + head * item + row * keys + 4 * rows * vocab
        total["flops"] += tokens * flops + pairs * pair + 2 * rows * head
        if experts:
            count, top, each_bytes, each_flops, layers = experts
            total["bytes"] += layers * each_bytes * count * (1 - (1 - top / count) ** tokens)
            total["flops"] += layers * each_flops * top * tokens
    return total


def tolerance(case):
    """About four times what the path showed against `exact` (2-norms: 9e-6 with 32-bit sums; rounding to bf16 around every product:
    0.017, 0.037 at the larger width, 0.003 where every sublayer's result is normalised, 0.05 where experts are chosen, whose
    weights amplify what came before; the largest of some million differences is five times the 2-norm).  `differ`: greedy picks among 150,000 random logits meet near ties, and a
    draw among the 50 largest follows every change of their order."""
    if case["dtype"] == FP32:
        rel = 9e-6
    else:
        rel = {"qwen2.5-1.5b": 0.017, "qwen2.5-7b": 0.037, "matidra-3b-layers": 0.0035, "gedalix-16b-layers": 0.05}[case["model"]]
    return {"rel": 4 * rel, "max": min(0.9, 20 * rel), "differ": 0.5 if case["top_k"] else 0.2}


# ------------------------------------------------------------------------------------- the same in 64 bits, plain torch
def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _rows(x, f, rows=4096):
    return torch.cat([f(x[a:a + rows]) for a in range(0, x.shape[0], rows)], 0)


def _silu(x):
    return x * torch.sigmoid(x)


def _swiglu(x, gate, up, down):
    return _rows(x, lambda r: (_silu(r @ gate.T) * (r @ up.T)) @ down.T)


def _turn_half(x, positions, base, dims):
    half = dims // 2
    f = base ** (-2.0 * torch.arange(half, dtype=F, device=x.device) / dims)
    a = (positions.to(F)[:, None] * f)[:, None, :]
    cos, sin = torch.cos(a), torch.sin(a)
    out = x.clone()
    u, v = x[..., :half], x[..., half:dims]
    out[..., :half] = u * cos - v * sin
    out[..., half:dims] = v * cos + u * sin
    return out


def _softmax_attention(q, k, v, scale, spans, sink=None):
    """q [N, H, dk], k [N, G, dk], v [N, G, dv]; each span of rows is a sequence of its own."""
    H, G = q.shape[1], k.shape[1]
    out = torch.empty(q.shape[0], H, v.shape[2], dtype=F, device=q.device)
    for a, b in spans:
        hidden = torch.ones(b - a, b - a, dtype=torch.bool, device=q.device).triu(1)
        for h in range(H):
            g = h // (H // G)
            s = (q[a:b, h] @ k[a:b, g].T * scale).masked_fill_(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(b - a, 1)], 1)
            out[a:b, h] = torch.softmax(s, -1)[:, :b - a] @ v[a:b, g]
    return out


def _qwen(cfg, w, ids, positions, spans, wanted):
    h, d, eps = cfg.hidden_size, cfg.head_size, cfg.rms_norm_eps
    H, G, ff = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.intermediate_size
    N = ids.shape[0]
    x = w("model.embed_tokens.weight", cfg.vocab_size, h)[ids]
    for i in range(cfg.num_hidden_layers):
        p = f"model.layers.{i}."
        y = _rms(x, eps) * w(p + "input_layernorm.weight", h)
        q, k, v = ((y @ w(p + f"self_attn.{n}_proj.weight", c * d, h).T + w(p + f"self_attn.{n}_proj.bias", c * d)).view(N, c, d)
                   for n, c in (("q", H), ("k", G), ("v", G)))
        q, k = _turn_half(q, positions, cfg.rope_theta, d), _turn_half(k, positions, cfg.rope_theta, d)
        x = x + _softmax_attention(q, k, v, d ** -0.5, spans).view(N, H * d) @ w(p + "self_attn.o_proj.weight", h, H * d).T
        y = _rms(x, eps) * w(p + "post_attention_layernorm.weight", h)
        x = x + _swiglu(y, w(p + "mlp.gate_proj.weight", ff, h), w(p + "mlp.up_proj.weight", ff, h), w(p + "mlp.down_proj.weight", h, ff))
    head = w("model.embed_tokens.weight" if cfg.tie_word_embeddings else "lm_head.weight", cfg.vocab_size, h)
    return (_rms(x[wanted], eps) * w("model.norm.weight", h)) @ head.T


def _gedalix(cfg, w, ids, positions, spans, wanted):
    raw = cfg.to_dict()
    h, eps, mult, N = raw["width"], raw["norm"]["eps"], raw["residual_mult"], ids.shape[0]
    x = w("embed", raw["vocab"], h)[ids] * raw["embedding"]["scale"] + w("pos", raw["max_positions"], h)[positions]
    for i, layer in enumerate(raw["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        H, dim, rot, vdim, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        y = _rms(x, eps) * w(p + "norm1", h)
        q = (y @ w(p + "mix.q", H * (dim + rot), h).T).view(N, H, dim + rot)
        both = y @ w(p + "mix.dkv", rank + rot, h).T
        c = _rms(both[:, :rank], eps) * w(p + "mix.dkv.norm", rank)
        turn = lambda t: _turn_half(t, positions, m["rot"]["base"], m["rot"]["dims"])  # noqa: E731
        q = torch.cat([q[..., :dim], turn(q[..., dim:])], -1)
        k = torch.cat([(c @ w(p + "mix.uk", H * dim, rank).T).view(N, H, dim), turn(both[:, None, rank:]).expand(N, H, rot)], -1)
        v = (c @ w(p + "mix.uv", H * vdim, rank).T).view(N, H, vdim)
        o = _softmax_attention(q, k, v, m["scale"], spans, w(p + "mix.sink", H)).view(N, H * vdim)
        o = (o * torch.sigmoid(y @ w(p + "mix.g", H * vdim, h).T)) @ w(p + "mix.o", h, H * vdim).T
        x = x + mult * o * w(p + "ls1", h)
        y = _rms(x, eps) * w(p + "norm2", h)
        E, top, ff, sff = mlp["router"]["experts"], mlp["router"]["top"], mlp["expert"]["ff"], mlp["shared"]["ff"]
        best = torch.topk(y @ w(p + "mlp.router", E, h).T + w(p + "mlp.router.b", E), top, dim=-1)
        share = torch.softmax(best.values, -1)
        out = _swiglu(y, w(p + "mlp.shared.gate", sff, h), w(p + "mlp.shared.up", sff, h), w(p + "mlp.shared.down", h, sff))
        out = out * torch.sigmoid(y @ w(p + "mlp.shared.sg", 1, h).T)
        for e in range(E):
            rows, which = (best.indices == e).nonzero(as_tuple=True)
            if rows.numel():
                t = p + f"mlp.e{e}."
                out.index_add_(0, rows, share[rows, which, None] * _swiglu(y[rows], w(t + "gate", ff, h), w(t + "up", ff, h), w(t + "down", h, ff)))
        x = x + mult * out * w(p + "ls2", h)
    return (_rms(x[wanted], eps) * w("final.norm", h)) @ w("head", raw["vocab"], h).T


def _layer_norm(x, w, b, eps):
    mean = x.mean(-1, keepdim=True)
    return (x - mean) * torch.rsqrt(((x - mean) ** 2).mean(-1, keepdim=True) + eps) * w + b


def _convolve(x, taps, spans):
    n, out = taps.shape[1], torch.empty_like(x)
    for a, b in spans:
        padded = torch.nn.functional.pad(x[a:b], (0, 0, n - 1, 0))
        out[a:b] = sum(padded[j:j + b - a] * taps[:, j] for j in range(n))
    return out


def _turn_pairs(x, positions, rot):
    dims, base, s = rot["dims"], rot["base"], rot.get("scaling")
    f, size = [base ** (-2.0 * i / dims) for i in range(dims // 2)], 1.0
    if s:
        where = lambda turns: dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(where(s["fast"])), 0), min(math.ceil(where(s["slow"])), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        f, size = [v / s["factor"] * r + v * (1.0 - r) for v, r in zip(f, ramp)], 0.1 * math.log(s["factor"]) + 1.0
    a = (positions.to(F)[:, None] * torch.tensor(f, dtype=F, device=x.device))[:, None, :]
    cos, sin = torch.cos(a) * size, torch.sin(a) * size
    out = x.clone()
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    out[..., 0:dims:2] = u * cos - v * sin
    out[..., 1:dims:2] = v * cos + u * sin
    return out


def _delta_rule(q, k, v, g, beta, spans):
    """q, k, g [N, H, dk], v [N, H, dv], beta [N, H]: the sequences side by side, token by token."""
    B, T = len(spans), max(b - a for a, b in spans)

    def side_by_side(t):
        out = torch.zeros(T, B, *t.shape[1:], dtype=F, device=t.device)
        for i, (a, b) in enumerate(spans):
            out[:b - a, i] = t[a:b]
        return out
    qs, ks, vs, gs, bs = (side_by_side(t) for t in (q, k, v, g, beta))
    S = torch.zeros(B, q.shape[1], q.shape[2], v.shape[2], dtype=F, device=q.device)
    o = torch.empty(T, B, v.shape[1], v.shape[2], dtype=F, device=q.device)
    for t in range(T):
        S = S * gs[t][..., None]
        u = bs[t][..., None] * (vs[t] - (ks[t][:, :, None, :] @ S)[:, :, 0])
        S = S + ks[t][..., None] * u[:, :, None, :]
        o[t] = (qs[t][:, :, None, :] @ S)[:, :, 0]
    return torch.cat([o[:b - a, i] for i, (a, b) in enumerate(spans)], 0)


def _matidra(cfg, w, ids, positions, spans, wanted):
    raw = cfg.to_dict()
    h, eps, alpha, N = raw["width"], raw["norm"]["eps"], raw["postln_alpha"], ids.shape[0]

    def soft(x, p, m, conv):
        H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k = x @ w(p + "q", H * dk, h).T, x @ w(p + "k", G * dk, h).T
        v = x @ w(p + "v", G * dv, h).T if conv else k
        if conv:
            q, k, v = (_convolve(t, w(p + n + ".conv", t.shape[1], m["conv"]), spans) for t, n in ((q, "q"), (k, "k"), (v, "v")))
        q, k, v = _rms(q.view(N, H, dk), eps) * w(p + "q.norm", dk), _rms(k.view(N, G, dk), eps) * w(p + "k.norm", dk), v.view(N, G, dv)
        if m.get("rot"):
            q, k = _turn_pairs(q, positions, m["rot"]), _turn_pairs(k, positions, m["rot"])
        if m.get("q_temp"):
            q = q * (1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((positions.to(F) + 1) / m["q_temp"]["every"]) + 1.0))[:, None, None]
        o = _softmax_attention(q, k, v, m["scale"], spans).view(N, H * dv)
        if conv:
            o = o * torch.sigmoid(x @ w(p + "g", H * dv, h).T)
        return o @ w(p + "o", h, H * dv).T

    def delta(x, p, m):
        H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(_convolve(x @ w(p + n, c, h).T, w(p + n + ".conv", c, m["conv"]), spans)).view(N, -1, d)
                   for n, c, d in (("q", G * dk, dk), ("k", G * dk, dk), ("v", H * dv, dv)))
        unit = lambda t: t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k = ((unit(t) * f).repeat_interleave(H // G, 1) for t, f in ((q, dk ** -0.5), (k, 1.0)))
        beta = torch.sigmoid(x @ w(p + "b", H, h).T)
        pre = (x @ w(p + "a1", m["a_rank"], h).T) @ w(p + "a2", H * dk, m["a_rank"]).T + w(p + "dt_bias", H * dk)
        g = torch.exp(-torch.exp(w(p + "A_log", H))[None, :, None] * torch.nn.functional.softplus(pre).view(N, H, dk))
        o = _rms(_delta_rule(q, k, v, g, beta, spans), eps) * w(p + "norm", dv)
        o = o * torch.sigmoid((x @ w(p + "g1", m["g_rank"], h).T) @ w(p + "g2", H * dv, m["g_rank"]).T).view(N, H, dv)
        return o.reshape(N, H * dv) @ w(p + "o", h, H * dv).T

    x = w("embed", raw["vocab"], h)[ids]
    for i, layer in enumerate(raw["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        if layer["type"] == "attention":
            mixed = soft(x, p + "mix.", m, False)
        else:
            mixed = m["left_scale"] * soft(x, p + "mix.left.", m["left"], True) + m["right_scale"] * delta(x, p + "mix.right.", m["right"])
        x = _layer_norm(alpha * x + mixed, w(p + "norm1", h), w(p + "norm1.b", h), eps)
        gate, up, down = w(p + "mlp.gate", ff, h), w(p + "mlp.up", ff, h), w(p + "mlp.down", h, ff)
        y = (torch.nn.functional.gelu(x @ gate.T, approximate="tanh") * (x @ up.T)) @ down.T
        x = _layer_norm(alpha * x + y, w(p + "norm2", h), w(p + "norm2.b", h), eps)
    return _layer_norm(x[wanted], w("final.norm", h), w("final.norm.b", h), eps) @ w("head", raw["vocab"], h).T


def exact(case, seed):
    cfg, device = _config(case), torch.device("cuda")
    tokens, lengths = _token_ids(case, seed, cfg.vocab_size), _prompt_lengths(case)
    starts = [0]
    for t in tokens:
        starts.append(starts[-1] + len(t))
    spans = list(zip(starts, starts[1:]))
    if case["kind"] == "burst":
        groups = [[starts[i] + a + n - 1 for i, a, n, wants in step if wants] for step in _burst_plan(case)[0]]
        groups = [g for g in groups if g]
    else:
        groups = [[a + n - 1 for a, n in zip(starts, lengths)]] if case["kind"] != "decode" else []
        groups += [[a + n + k for a, n in zip(starts, lengths)] for k in range(case["steps"])]
    flat = lambda lists: torch.tensor([v for one in lists for v in one], dtype=torch.int64, device=device)  # noqa: E731
    model = _qwen if case["model"].startswith("qwen") else _gedalix if case["model"].startswith("gedalix") else _matidra
    logits = model(cfg, _Weights(seed, case["dtype"]), flat(tokens), flat([range(b - a) for a, b in spans]), spans, flat(groups))
    parts = list(torch.split(logits, [len(g) for g in groups]))
    if case["kind"] == "prompt":
        return parts[0]
    if case["kind"] == "burst":
        return parts
    if case["kind"] == "turn":
        return {"prompt": parts[0], "tokens": None, "logits": parts[1:]}
    return {"tokens": None, "logits": parts}

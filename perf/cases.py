"""The work that a user of the framework has it do, as cases that can be timed and compared.

A case is a small dict of plain values.  Its kind ("what") is one of

  generate   a whole Llama model (the 1B preset) through ModelRunner.step: the prompts of a batch in one step, then a
             number of steps of one given token per request (a trace replay), every step's logits kept; the requests end
  layer      one mixer of a model as the runner builds it, forward over a step's tokens: grouped-query attention over
             the paged cache (prompts, portions behind a cached prefix, single tokens), attention with biases and normed
             queries and keys, the gated delta rule, lightning attention, retention
  sample     a batch of logit rows through the Sampler

`portions` lists a step's requests as "new@cached" tokens.  Sizes are those of the shipped presets and of the shapes that
bench.py and the kernel benchmarks use; `draw` gives other sizes of the same ranges.
"""
import math

import numpy as np
import torch

from nanoinfer_b200.config import LayerRun, LayerSpec, MixerSpec, ModelConfig, NormSpec, PositionSpec, config_from_dict, preset
from nanoinfer_b200.config.model_config import EmbeddingSpec, HeadSpec
from nanoinfer_b200.config.registry import architecture
from nanoinfer_b200.engine.step import ModelRunner, StepEntry
from nanoinfer_b200.sampling import Sampler, SamplingParams
from nanoinfer_b200.weights.plan import tensor_plan

PAGE = 16
F64 = torch.float64
TAPS = 4                 # of the gated delta rule's convolution
EPS = 1e-5


# ---- the cases -------------------------------------------------------------------------------------------------------

def listed():
    return [
        # one user waiting for a short answer: the latency of single-token steps, weights read once per token
        {"name": "generate_one", "what": "generate", "dtype": "bfloat16", "portions": "33@0", "steps": 16},
        # the headline batch: eight requests of uneven prompts answered together
        {"name": "generate_eight", "what": "generate", "dtype": "bfloat16", "steps": 16,
         "portions": "212@0,37@0,301@0,128@0,90@0,256@0,17@0,175@0"},
        # the true 32-bit path, as replays for exact logits use it
        {"name": "generate_f32", "what": "generate", "dtype": "float32", "steps": 8, "portions": "120@0,57@0"},
        # a prompt of 2,048 tokens through an attention layer of the 1B shape
        {"name": "attention_prompt", "what": "layer", "kind": "attention", "dtype": "bfloat16", "width": 2048,
         "heads": 32, "kv_heads": 8, "dim": 64, "portions": "2048@0"},
        # chunked prefill of a busy server at the 8B shape: portions of prompts behind what is cached already, one answer token
        {"name": "attention_portions", "what": "layer", "kind": "attention", "dtype": "bfloat16", "width": 4096,
         "heads": 32, "kv_heads": 8, "dim": 128, "portions": "512@3072,512@1024,1@777,377@0,512@4608"},
        # 32 requests decoding at the 3B shape, contexts of all lengths
        {"name": "attention_decode", "what": "layer", "kind": "attention", "dtype": "bfloat16", "width": 3072,
         "heads": 24, "kv_heads": 8, "dim": 128,
         "portions": ",".join("1@%d" % (301 + 97 * i) for i in range(32))},
        # prompts through an attention layer of the 32-bit path (1B shape)
        {"name": "attention_f32", "what": "layer", "kind": "attention", "dtype": "float32", "width": 2048,
         "heads": 32, "kv_heads": 8, "dim": 64, "portions": "701@0,130@0,256@384"},
        # attention with biases, normed queries and keys, half of a head rotated: a long prompt and a portion
        {"name": "normed_attention_prompt", "what": "layer", "kind": "normed_qk_attention", "dtype": "bfloat16", "width": 2048,
         "heads": 16, "kv_heads": 8, "dim": 128, "portions": "1537@0,511@512"},
        # the gated delta rule over prompts of uneven lengths, one of them continued
        {"name": "delta_prompt", "what": "layer", "kind": "gated_delta", "dtype": "bfloat16", "width": 2048,
         "heads": 16, "kv_heads": 16, "dim": 128, "portions": "1201@0,847@512"},
        # lightning attention over a prompt
        {"name": "lightning_prompt", "what": "layer", "kind": "lightning", "dtype": "bfloat16", "width": 2048,
         "heads": 16, "kv_heads": 16, "dim": 128, "portions": "2048@0"},
        # retention (rotated 32-bit queries and keys) over prompts
        {"name": "retention_prompt", "what": "layer", "kind": "retention", "dtype": "bfloat16", "width": 2048,
         "heads": 8, "kv_heads": 8, "dim": 128, "portions": "1100@0,948@300"},
        # the token of every request of a batch drawn with top-k and top-p: once per step of a server
        {"name": "sample_eight", "what": "sample", "rows": 8, "vocab": 128256, "top_k": 50, "top_p": 0.9},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _prompts(rng, total, most):
    """Portions of `total` tokens in all over at most `most` requests, some behind a cached prefix."""
    n = rng.randint(1, most)
    cuts = sorted(rng.sample(range(16, max(total - 15, 17 + n)), n - 1)) if n > 1 and total > 64 else []
    sizes = [b - a for a, b in zip([0] + cuts, cuts + [total])]
    return ",".join("%d@%d" % (max(s, 1), rng.choice((0, 0, _spread(rng, 16, 2048)))) for s in sizes)


def draw(rng):
    what = rng.choice(("generate", "generate_f32", "attention", "attention", "decode", "attention_f32", "normed_qk_attention",
                       "gated_delta", "lightning", "retention", "sample"))
    if what == "sample":
        return {"what": "sample", "rows": _spread(rng, 1, 64), "vocab": rng.choice((32000, 50257, 128256)),
                "top_k": rng.choice((-1, 20, 50, 200)), "top_p": rng.choice((1.0, 0.8, 0.9, 0.95))}
    if what in ("generate", "generate_f32"):
        f32 = what == "generate_f32"
        n = rng.randint(1, 3) if f32 else _spread(rng, 1, 10)
        return {"what": "generate", "dtype": "float32" if f32 else "bfloat16", "steps": rng.randint(5, 8 if f32 else 16),
                "portions": ",".join("%d@0" % _spread(rng, 5, 90 if f32 else 200) for _ in range(n))}
    case = {"what": "layer", "kind": what, "dtype": "bfloat16"}
    if what in ("attention", "decode", "attention_f32"):
        case["kind"] = "attention"
        case["width"], case["heads"], case["kv_heads"], case["dim"] = rng.choice(((2048, 32, 8, 64), (3072, 24, 8, 128), (4096, 32, 8, 128)))
        if what == "decode":
            case["portions"] = ",".join("1@%d" % _spread(rng, 40, 4096) for _ in range(_spread(rng, 4, 64)))
        elif what == "attention":
            case["portions"] = _prompts(rng, _spread(rng, 200, 3000), 5)
        else:
            case["dtype"] = "float32"
            case["portions"] = _prompts(rng, _spread(rng, 20, 1000), 3)
        return case
    case["width"] = rng.choice((1024, 2048))
    case["heads"] = case["kv_heads"] = case["width"] // rng.choice((128, 256))
    case["dim"] = 128
    if what == "normed_qk_attention":
        case["kv_heads"] = max(case["heads"] // 2, 1)
    case["portions"] = _prompts(rng, _spread(rng, 100, 3000), 4)
    return case


# ---- inputs ----------------------------------------------------------------------------------------------------------

def _portions(case):
    return [tuple(int(x) for x in p.split("@")) for p in case["portions"].split(",")]


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape, std=1.0):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * std


def _raw_llama():
    raw = dict(preset("llama-3.2-1b"))
    raw["max_position_embeddings"] = 8192
    return raw


def _decays(case):
    """One fixed decay per head, from heads that forget within a few tokens to heads that hardly do."""
    n = case["heads"]
    if case["kind"] == "retention":
        return tuple(1.0 - 2.0 ** (-5.0 - 3.0 * h / n) for h in range(n))
    return tuple(math.exp(-2.0 ** (-8.0 * (h + 1) / n)) for h in range(n))


def _layer_config(case):
    kind, h, g, d, width = case["kind"], case["heads"], case["kv_heads"], case["dim"], case["width"]
    scale, none = d ** -0.5, PositionSpec(kind="none")
    if kind == "attention":
        mixer = MixerSpec(kind=kind, num_heads=h, num_kv_heads=g, head_dim=d, softmax_scale=scale,
                          position=PositionSpec(kind="rope", theta=500000.0, rotary_dim=d, pairing="half"))
    elif kind == "normed_qk_attention":
        mixer = MixerSpec(kind=kind, num_heads=h, num_kv_heads=g, head_dim=d, softmax_scale=scale,
                          position=PositionSpec(kind="rope_yarn", theta=10000.0, rotary_dim=d // 2, pairing="half"),
                          extra=(("value_dim", d), ("norm_eps", EPS), ("bias", True), ("qk_norm", True)))
    elif kind == "gated_delta":
        mixer = MixerSpec(kind=kind, num_heads=h, num_kv_heads=g, head_dim=d, position=none,
                          extra=(("value_dim", d), ("conv_taps", TAPS), ("norm_eps", EPS)))
    elif kind == "lightning":
        mixer = MixerSpec(kind=kind, num_heads=h, num_kv_heads=h, head_dim=d, position=none,
                          extra=(("value_dim", d), ("decay", _decays(case)), ("norm_eps", EPS)))
    else:
        mixer = MixerSpec(kind="retention", num_heads=h, num_kv_heads=h, head_dim=d,
                          position=PositionSpec(kind="rope_yarn", theta=10000.0, rotary_dim=d, pairing="half"),
                          extra=(("value_dim", d), ("decay", _decays(case)), ("norm_eps", EPS)))
    norm = NormSpec(kind="rmsnorm", eps=EPS)
    layer = LayerSpec(mixer=mixer, feed_forward=None, mixer_norm=norm, ffn_norm=None, arrangement="pre_norm")
    return ModelConfig(architecture="Tazulix", hidden_size=width, vocab_size=256, max_position_embeddings=1 << 20,
                       layers=(layer,), schedule=(LayerRun(layer=0),), final_norm=norm,
                       embedding=EmbeddingSpec(kind="table"), head=HeadSpec(kind="linear", tied=False))


def _mixer_weights(case, g):
    """The mixer's tensors by slot, in the stored type: projections that keep activations of order one."""
    kind, h, kv, d, width = case["kind"], case["heads"], case["kv_heads"], case["dim"], case["width"]
    w = lambda n, k: _randn(g, n, k, std=k ** -0.5)
    out = {"q": w(h * d if kind != "gated_delta" else kv * d, width), "k": w(kv * d, width),
           "v": w((kv if "attention" in kind else h) * d, width), "o": w(width, h * d)}
    if kind == "normed_qk_attention":
        out.update({"q.b": _randn(g, h * d, std=0.2), "k.b": _randn(g, kv * d, std=0.2), "v.b": _randn(g, kv * d, std=0.2),
                    "q.norm": 1 + _randn(g, h * d, std=0.2), "k.norm": 1 + _randn(g, kv * d, std=0.2)})
    elif kind == "gated_delta":
        step = torch.exp(torch.rand(h, generator=g, device="cuda") * math.log(100.0) + math.log(0.001))
        out.update({"g": w(h * d, width), "a": w(h, width), "b": w(h, width), "norm": 1 + _randn(g, d, std=0.2),
                    "A_log": torch.log(1 + 15 * torch.rand(h, generator=g, device="cuda")), "dt_bias": torch.log(torch.expm1(step))})
        out.update({s + ".conv": _randn(g, out[s].shape[0], TAPS, std=0.5) for s in ("q", "k", "v")})
    elif kind in ("lightning", "retention"):
        out["g"] = w(h * d, width)
        if kind == "lightning":
            out["norm"] = 1 + _randn(g, h * d, std=0.2)
    return {k: v.to(_dtype(case)) for k, v in out.items()}


def _state_size(case):
    h, d = case["heads"], case["dim"]
    if case["kind"] == "gated_delta":
        return h * d * d + (TAPS - 1) * (2 * case["kv_heads"] * d + h * d)
    return h * d * d


def _layer_inputs(case, seed):
    """(weights by slot, x, cached keys and values per request, starting states): everything that the seed decides."""
    g = _generator(seed)
    weights = _mixer_weights(case, g)
    portions = _portions(case)
    x = _randn(g, sum(n for n, _ in portions), case["width"]).to(_dtype(case))
    cached, start = [], None
    if "attention" in case["kind"]:
        cached = [tuple(_randn(g, c, case["kv_heads"], case["dim"]).to(_dtype(case)) for _ in range(2)) for _, c in portions]
    else:
        start = torch.stack([_randn(g, _state_size(case), std=0.2 if c else 0.0) for _, c in portions])
    return weights, x, cached, start


def _llama_weights(case, seed):
    config = config_from_dict(_raw_llama())
    g = _generator(seed)
    out = {}
    for p in tensor_plan(config):
        t = 1 + _randn(g, *p.shape, std=0.1) if p.init == "ones" else _randn(g, *p.shape, std=0.02)
        out[p.name] = t.to(_dtype(case))
    return config, out


def _tokens(case, seed):
    """Per request: its prompt and the tokens that follow, one per step."""
    rs = np.random.RandomState(seed % (1 << 32))
    return [rs.randint(0, 128256, n + case["steps"]).tolist() for n, _ in _portions(case)]


def prepare(case, seed):
    if case["what"] == "sample":
        g = _generator(seed)
        n = case["rows"]
        params = [SamplingParams(temperature=0.7 + 0.05 * (r % 8), top_k=case["top_k"], top_p=case["top_p"], seed=r) for r in range(n)]
        return {"what": "sample", "sampler": Sampler(case["vocab"], torch.device("cuda:0")), "logits": _randn(g, n, case["vocab"], std=3.0),
                "params": params, "seeds": [seed * 64 + r for r in range(n)], "indices": [17 + r for r in range(n)]}
    portions = _portions(case)
    if case["what"] == "generate":
        config, weights = _llama_weights(case, seed)
        longest = max(n for n, _ in portions) + case["steps"]
        runner = ModelRunner(config, weights, dtype=case["dtype"], page_size=PAGE, max_requests=len(portions),
                             num_pages=sum(-(-(n + case["steps"]) // PAGE) + 1 for n, _ in portions),
                             max_tokens_per_request=-(-longest // PAGE) * PAGE)
        state = {"what": "generate", "runner": runner, "tokens": _tokens(case, seed), "prompts": [n for n, _ in portions], "steps": case["steps"]}
        for _ in range(4):               # a server has met its step shapes before: recurring ones are replayed from graphs
            run(state)
        return state
    weights, x, cached, start = _layer_inputs(case, seed)
    config = _layer_config(case)
    g = _generator(seed + 1)
    name = architecture(config.architecture).tensor_name
    named = {p.name: _randn(g, *p.shape) for p in tensor_plan(config) if p.scope[-1] != "mixer"}
    named.update({name(("layer", 0, "mixer"), slot): t for slot, t in weights.items()})
    most = max(n + c for n, c in portions)
    runner = ModelRunner(config, named, dtype=case["dtype"], page_size=PAGE, max_requests=len(portions),
                         num_pages=sum(-(-(n + c) // PAGE) for n, c in portions), max_tokens_per_request=-(-most // PAGE) * PAGE)
    for i in range(len(portions)):
        if runner.admit(i) != i:
            raise RuntimeError("requests admitted in order take the state rows in order")
    for at in range(0, max(c for _, c in portions), 512):        # prompts grew in turns, so their pages lie mixed
        behind = [StepEntry(i, [0] * min(512, c - at)) for i, (_, c) in enumerate(portions) if c > at]
        runner.build_context(behind)
    ctx = runner.build_context([StepEntry(i, [0] * n) for i, (n, _) in enumerate(portions)])
    cache = runner.caches[0]
    for i, kv in enumerate(cached):
        n = kv[0].shape[0]
        j = torch.arange(n, device="cuda")
        page = ctx.block_tables[0][i].long()[j // PAGE]
        for plane, rows in zip((cache.pages["k"], cache.pages["v"]), kv):
            plane[page, :, j % PAGE] = rows
    return {"what": "layer", "runner": runner, "mixer": runner.model.blocks[0].mixer, "ctx": ctx, "cache": cache, "x": x, "start": start}


# ---- one pass --------------------------------------------------------------------------------------------------------

def run(state):
    if state["what"] == "sample":
        return state["sampler"].sample(state["logits"], state["params"], state["seeds"], state["indices"])
    if state["what"] == "layer":
        cache = state["cache"]
        if state["start"] is None:
            y = state["mixer"].forward(state["x"], state["ctx"], cache)
            return {"y": y, "keys": cache.pages["k"], "values": cache.pages["v"]}
        cache.state.copy_(state["start"])            # new requests start from zero, continued ones from where they stood
        return {"y": state["mixer"].forward(state["x"], state["ctx"], cache), "state": cache.state}
    runner, tokens, prompts = state["runner"], state["tokens"], state["prompts"]
    logits = [runner.step([StepEntry(i, t[:n], [n - 1]) for i, (t, n) in enumerate(zip(tokens, prompts))]).clone()]
    for s in range(state["steps"]):
        logits.append(runner.step([StepEntry(i, [t[n + s]], [0]) for i, (t, n) in enumerate(zip(tokens, prompts))]).clone())
    for i in range(len(tokens)):
        runner.end(i)
    return logits


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

def work(case):
    if case["what"] == "sample":
        return {"bytes": 4 * case["rows"] * (case["vocab"] + 1), "flops": 0}
    size = 4 if case["dtype"] == "float32" else 2
    portions = _portions(case)
    new = sum(n for n, _ in portions)
    pairs = sum(n * c + n * (n + 1) // 2 for n, c in portions)                # (query, key) pairs of causal attention
    if case["what"] == "generate":
        raw = _raw_llama()
        d, ff, layers, vocab = raw["hidden_size"], raw["intermediate_size"], raw["num_hidden_layers"], raw["vocab_size"]
        kv, hd = raw["num_key_value_heads"] * raw["head_dim"], raw["num_attention_heads"] * raw["head_dim"]
        layer = d * (2 * hd + 2 * kv + 3 * ff)
        steps, b = case["steps"], len(portions)
        pairs += sum(steps * n + steps * (steps + 1) // 2 for n, _ in portions)
        kept = sum(steps * n + steps * (steps + 1) // 2 + n + steps for n, _ in portions)
        return {"bytes": size * ((steps + 1) * (layers * layer + vocab * d) + layers * 2 * kv * kept) + 4 * (steps + 1) * b * vocab,
                "flops": 2 * (new + steps * b) * layers * layer + 2 * (steps + 1) * b * vocab * d + 4 * pairs * hd * layers}
    h, g, d, width = case["heads"], case["kv_heads"], case["dim"], case["width"]
    hd, gd = h * d, g * d
    out = size if case["kind"] in ("attention", "gated_delta") else 4
    io = new * width * (size + out)
    if "attention" in case["kind"]:
        weights = width * (2 * hd + 2 * gd)
        kept = sum(n + c for n, c in portions)
        return {"bytes": io + size * (weights + 2 * gd * kept), "flops": 2 * new * weights + 4 * pairs * hd}
    weights = width * (3 * hd + 2 * gd + (2 * h if case["kind"] == "gated_delta" else 0))
    per_token = (8 if case["kind"] == "gated_delta" else 4) * h * d * d
    return {"bytes": io + size * weights + 8 * len(portions) * _state_size(case), "flops": new * (2 * weights + per_token)}


def tolerance(case):
    if case["what"] == "sample":
        return "exact"                   # thresholds are exact and masses fixed-point: the same logits give the same token
    if case["what"] == "generate":
        return {"rel": 4e-5} if case["dtype"] == "float32" else {"rel": 7e-2}      # 16 layers: 0.9e-5 / 1.9e-2 from the exact logits
    if case["dtype"] == "float32":
        return {"rel": 1e-5}             # 1.5e-6 from the exact result
    return {"rel": 1.6e-2}               # 0.2e-2 (lightning) to 0.42e-2 (attention)


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------

def _rms(x, gain, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * (1.0 if gain is None else gain)


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, pos, freq):
    """x [T, H, d] with the pairs (i, i + n) of its first 2 n = 2 len(freq) dimensions turned by float32(pos * freq)."""
    n = freq.numel()
    angle = (pos.to(torch.float32)[:, None] * freq.to(torch.float32)[None, :]).to(F64)[:, None, :]
    a, b, rest = x[..., :n], x[..., n:2 * n], x[..., 2 * n:]
    return torch.cat([a * torch.cos(angle) - b * torch.sin(angle), a * torch.sin(angle) + b * torch.cos(angle), rest], dim=-1)


def _frequencies(dims, theta):
    i = torch.arange(dims // 2, dtype=F64, device="cuda")
    return torch.pow(torch.tensor(theta, dtype=F64, device="cuda"), -2.0 * i / dims).to(torch.float32)


def _llama_frequencies(raw):
    """float32, by the llama3 rule: long waves slowed down by the factor, a blend between the two bounds."""
    f32, rs, n = np.float32, raw["rope_scaling"], raw["head_dim"]
    out = []
    for i in range(n // 2):
        f = f32(1.0) / np.power(f32(raw["rope_theta"]), f32(2 * i) / f32(n), dtype=f32)
        wave = f32(2.0) * f32(math.pi) / f
        lo, hi, old = f32(rs["low_freq_factor"]), f32(rs["high_freq_factor"]), f32(rs["original_max_position_embeddings"])
        if wave >= old / lo:
            f = f / f32(rs["factor"])
        elif wave > old / hi:
            s = (old / wave - lo) / (hi - lo)
            f = (f32(1.0) - s) * f / f32(rs["factor"]) + s * f
        out.append(f)
    return torch.tensor(np.array(out, dtype=f32), device="cuda")


def _attend(q, k, v, first):
    """Causal attention: q [T, H, d] at positions first .. over k, v [first + T, G, d]; scores by d^-1/2."""
    t, h, d = q.shape
    group = h // k.shape[1]
    hidden = torch.arange(k.shape[0], device="cuda")[None, :] > first + torch.arange(t, device="cuda")[:, None]
    out = torch.empty_like(q)
    for a in range(h):
        s = (q[:, a] @ k[:, a // group].T) * d ** -0.5
        out[:, a] = torch.softmax(s.masked_fill_(hidden, -math.inf), dim=-1) @ v[:, a // group]
    return out


def _stored_as_halves(k, n):
    """Cached keys lie with the two numbers of a rotated pair side by side: back to (i, i + n / 2)."""
    return torch.cat([k[..., 0:n:2], k[..., 1:n:2], k[..., n:]], dim=-1)


def _exact_attention(case, w, x, cached):
    h, g, d = case["heads"], case["kv_heads"], case["dim"]
    normed = case["kind"] == "normed_qk_attention"
    q, k, v = (x @ w[s].T for s in "qkv")
    if normed:
        q, k, v = _rms(q + w["q.b"], w["q.norm"], EPS), _rms(k + w["k.b"], w["k.norm"], EPS), v + w["v.b"]
    freq = _frequencies(d // 2, 10000.0) if normed else _plain_rope(d)
    out, at = [], 0
    for (n, c), (ck, cv) in zip(_portions(case), cached):
        pos = c + torch.arange(n, device="cuda")
        mine = slice(at, at + n)
        qr = _rotate(q[mine].view(n, h, d), pos, freq)
        kr = _rotate(k[mine].view(n, g, d), pos, freq)
        ck = ck.to(F64) if normed else _stored_as_halves(ck.to(F64), d)
        out.append(_attend(qr, torch.cat([ck, kr]), torch.cat([cv.to(F64), v[mine].view(n, g, d)]), c).reshape(n, h * d))
        at += n
    return {"y": torch.cat(out) @ w["o"].T, "keys": None, "values": None}


def _plain_rope(d):
    f32 = np.float32
    return torch.tensor(np.array([f32(1.0) / np.power(f32(500000.0), f32(2 * i) / f32(d), dtype=f32) for i in range(d // 2)], dtype=f32),
                        device="cuda")


def _exact_linear(case, w, x, start):
    """Lightning attention and retention as one masked product per request and head."""
    h, d, retention = case["heads"], case["dim"], case["kind"] == "retention"
    q, k, v, z = (x @ w[s].T for s in ("q", "k", "v", "g"))
    if not retention:
        q, k, v = _silu(q), _silu(k), _silu(v)
    decay = torch.tensor(_decays(case), dtype=torch.float32, device="cuda").to(F64)
    out, states, at = [], [], 0
    for (n, c), s0 in zip(_portions(case), start.to(F64)):
        qr, kr, vr = (t[at:at + n].view(n, h, d) for t in (q, k, v))
        if retention:
            pos = c + torch.arange(n, device="cuda")
            freq = _frequencies(d, 10000.0)
            qr, kr = _rotate(qr, pos, freq), _rotate(kr, pos, freq) * d ** -0.5
        i = torch.arange(n, device="cuda", dtype=F64)
        s0, o, end = s0.view(h, d, d), torch.empty(n, h, d, dtype=F64, device="cuda"), []
        for a in range(h):
            m = torch.pow(decay[a], (i[:, None] - i[None, :]).clamp(min=0)).tril()
            o[:, a] = (qr[:, a] @ kr[:, a].T * m) @ vr[:, a] + torch.pow(decay[a], i + 1)[:, None] * (qr[:, a] @ s0[a])
            end.append(torch.pow(decay[a], torch.tensor(float(n), dtype=F64, device="cuda")) * s0[a]
                       + (kr[:, a] * torch.pow(decay[a], n - 1 - i)[:, None]).T @ vr[:, a])
        out.append(o)
        states.append(torch.stack(end).reshape(-1))
        at += n
    o = torch.cat(out)
    y = _rms(o, None, EPS).reshape(-1, h * d) * _silu(z) if retention else \
        _rms(o.reshape(-1, h * d), w["norm"], EPS) * torch.sigmoid(z)
    return {"y": y @ w["o"].T, "state": torch.stack(states)}


def _exact_delta(case, w, x, start):
    h, g, d = case["heads"], case["kv_heads"], case["dim"]
    inputs = torch.cat([x @ w[s].T for s in "qkv"], dim=1)
    taps = torch.cat([w[s + ".conv"] for s in "qkv"])
    decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a"].T + w["dt_bias"]))
    beta, z = torch.sigmoid(x @ w["b"].T), x @ w["g"].T
    out, states, at = [], [], 0
    for (n, _), s0 in zip(_portions(case), start.to(F64)):
        history = torch.cat([s0[h * d * d:].view(TAPS - 1, -1), inputs[at:at + n]])
        conv = _silu(sum(history[j:j + n] * taps[:, j] for j in range(TAPS)))
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
        q = (unit(conv[:, :g * d].view(n, g, d)) * d ** -0.5).repeat_interleave(h // g, dim=1)
        k = unit(conv[:, g * d:2 * g * d].view(n, g, d)).repeat_interleave(h // g, dim=1)
        v = conv[:, 2 * g * d:].view(n, h, d)
        s, o = s0[:h * d * d].view(h, d, d).clone(), torch.empty(n, h, d, dtype=F64, device="cuda")
        for t in range(n):
            s *= decay[at + t][:, None, None]
            e = beta[at + t][:, None] * (v[t] - torch.einsum("hd,hdv->hv", k[t], s))
            s += k[t][:, :, None] * e[:, None, :]
            o[t] = torch.einsum("hd,hdv->hv", q[t], s)
        out.append(o)
        states.append(torch.cat([s.reshape(-1), history[n:].reshape(-1)]))
        at += n
    y = (_rms(torch.cat(out), w["norm"], EPS)).reshape(-1, h * d) * _silu(z)
    return {"y": y @ w["o"].T, "state": torch.stack(states)}


def _exact_generate(case, seed):
    raw = _raw_llama()
    _, weights = _llama_weights(case, seed)
    h, g, d, eps = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"], raw["rms_norm_eps"]
    freq = _llama_frequencies(raw)
    rows = []
    tokens, prompts = _tokens(case, seed), [n for n, _ in _portions(case)]
    table = weights["model.embed_tokens.weight"]
    xs = [table[torch.tensor(t, device="cuda")].to(F64) for t in tokens]
    for i in range(raw["num_hidden_layers"]):
        w = {k: v.to(F64) for k, v in weights.items() if k.startswith("model.layers.%d." % i)}
        get = lambda s: w["model.layers.%d.%s.weight" % (i, s)]
        for j, x in enumerate(xs):
            n, pos = x.shape[0], torch.arange(x.shape[0], device="cuda")
            a = _rms(x, get("input_layernorm"), eps)
            q, k, v = (a @ get("self_attn.%s_proj" % s).T for s in "qkv")
            att = _attend(_rotate(q.view(n, h, d), pos, freq), _rotate(k.view(n, g, d), pos, freq), v.view(n, g, d), 0)
            x = x + att.reshape(n, h * d) @ get("self_attn.o_proj").T
            a = _rms(x, get("post_attention_layernorm"), eps)
            xs[j] = x + (_silu(a @ get("mlp.gate_proj").T) * (a @ get("mlp.up_proj").T)) @ get("mlp.down_proj").T
    last = torch.stack([x[n - 1:n + case["steps"]] for x, n in zip(xs, prompts)], dim=1)          # [steps + 1, requests, width]
    last = _rms(last, weights["model.norm.weight"].to(F64), eps)
    rows = torch.cat([last @ table[a:a + 16384].to(F64).T for a in range(0, table.shape[0], 16384)], dim=-1)
    return list(rows)


def exact(case, seed):
    if case["what"] == "sample":
        return None                       # token ids: see tolerance
    if case["what"] == "generate":
        return _exact_generate(case, seed)
    weights, x, cached, start = _layer_inputs(case, seed)
    w, x = {k: v.to(F64) for k, v in weights.items()}, x.to(F64)
    if start is None:
        return _exact_attention(case, w, x, cached)
    return (_exact_delta if case["kind"] == "gated_delta" else _exact_linear)(case, w, x, start)

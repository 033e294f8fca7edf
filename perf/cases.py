"""The work this engine is timed on: one whole generation and the layers its models are made of.

A layer is built as an engine builds it (``build_part`` on a part's description, weights by tensor name, a step's context and
a view of the cache) and called as the decoder calls it. Sizes are those of ``llama-3.2-1b`` and of the layer sizes that
``bench.py --design`` uses (widths 1,024 / 2,048 / 4,096). Every layer reads unit-variance inputs and weights of the spread
the random-weights mode uses, which gives projections of about unit size.
"""
from __future__ import annotations

import hashlib
import math

import numpy as np
import torch

from serve_b200 import Engine, EngineConfig, StepEntry, load_preset
from serve_b200.cache.manager import CacheView
from serve_b200.config.spec import PartSpec
from serve_b200.engine import BatchShape, Runtime, StepContext
from serve_b200.kernels import load_kernels
from serve_b200.parts.base import build_part

DEVICE = "cuda:0"
PAGE = 64
F64 = torch.float64

# width -> (heads of 128, experts, experts per token, expert width)
WIDTHS = {1024: (8, 32, 2, 512), 2048: (16, 64, 4, 768), 4096: (32, 64, 8, 512)}
# width -> (heads, kv heads, head size, feed-forward) of the Llama presets
LLAMA = {2048: (32, 8, 64, 8192), 3072: (24, 8, 128, 8192), 4096: (32, 8, 128, 14336)}


def listed():
    return [
        # a batch of short chats: eight prompts of about 256 tokens in one step, then fifteen decoding steps; all logits
        {"name": "llama_generate_8x256", "kind": "llama", "requests": 8, "prompt": 256, "new": 16},
        # one long prompt through a Llama attention layer (prefill)
        {"name": "attention_prompt_2048", "kind": "attention", "dtype": "bfloat16", "width": 2048, "requests": 1, "tokens": 2048, "context": 0},
        # the same layer in a busy decoding step: 64 requests of many lengths
        {"name": "attention_decode_64", "kind": "attention", "dtype": "bfloat16", "width": 2048, "requests": 64, "tokens": 1, "context": 2176},
        # the same layer in the true 32-bit mode, eight requests decoding
        {"name": "attention_decode_8_f32", "kind": "attention", "dtype": "float32", "width": 2048, "requests": 8, "tokens": 1, "context": 2048},
        # one user, one token: the smallest call, a dense feed-forward that only reads its weights
        {"name": "mlp_decode_1", "kind": "mlp", "dtype": "bfloat16", "width": 2048, "tokens": 1},
        # routed experts with a shared one, on a long prompt and in a decoding step of eight requests
        {"name": "experts_prompt_2048", "kind": "experts", "dtype": "bfloat16", "width": 2048, "tokens": 2048, "router": "softmax"},
        {"name": "experts_decode_8", "kind": "experts", "dtype": "bfloat16", "width": 2048, "tokens": 8, "router": "softmax"},
        # attention behind a window that keeps the first tokens, with a sink and normalised queries and keys, on a prompt
        {"name": "window_prompt_2048", "kind": "window", "dtype": "bfloat16", "width": 2048, "requests": 1, "tokens": 2048, "context": 0,
         "window": 1024, "keep": 4},
        # latent attention (one cached row a token for all heads) behind a window: a prompt, and a decoding step
        {"name": "latent_prompt_2048", "kind": "latent", "dtype": "bfloat16", "width": 2048, "requests": 1, "tokens": 2048, "context": 0,
         "window": 1024},
        {"name": "latent_decode_8", "kind": "latent", "dtype": "bfloat16", "width": 2048, "requests": 8, "tokens": 1, "context": 2048,
         "window": 1024},
        # gated delta rule (a matrix state per head) over one long prompt
        {"name": "delta_prompt_2048", "kind": "delta", "dtype": "bfloat16", "width": 2048, "requests": 1, "tokens": 2048, "rate": "head"},
        # linear attention with a fixed decay per head over eight prompts side by side
        {"name": "lightning_8x256", "kind": "lightning", "dtype": "bfloat16", "width": 2048, "requests": 8, "tokens": 256},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["llama", "attention", "attention", "mlp", "mlp", "experts", "experts", "window", "window", "latent", "latent", "delta",
                       "delta", "lightning"])
    if kind == "llama":
        return {"kind": kind, "requests": rng.randint(1, 8), "prompt": _log(rng, 8, 256), "new": rng.randint(2, 12)}
    dtype = "float32" if rng.random() < 0.15 else "bfloat16"
    if kind in ("mlp", "experts"):
        width = rng.choice(sorted(LLAMA if kind == "mlp" else WIDTHS))
        case = {"kind": kind, "dtype": dtype, "width": width, "tokens": _log(rng, 1, 512 if dtype == "float32" else 4096)}
        if kind == "experts":
            case["router"] = rng.choice(["softmax", "sigmoid"])
        return case
    width = rng.choice([2048, 2048, 3072] if kind == "attention" else [1024, 2048])
    most = 1024 if dtype == "float32" else 3072
    if kind in ("delta", "lightning"):
        requests = _log(rng, 1, 16)
        case = {"kind": kind, "dtype": dtype, "width": width, "requests": requests, "tokens": _log(rng, 2, max(2, most // requests))}
        if kind == "delta":
            case["rate"] = rng.choice(["head", "channel"])
        return case
    if rng.random() < 0.5:                                   # a decoding step
        requests = _log(rng, 1, 64)
        case = {"kind": kind, "dtype": dtype, "width": width, "requests": requests, "tokens": 1, "context": _log(rng, 16, 4000 if requests < 32 else 2500)}
    else:                                                    # prompts, or portions of prompts
        requests = _log(rng, 1, 8)
        case = {"kind": kind, "dtype": dtype, "width": width, "requests": requests, "tokens": _log(rng, 2, max(2, most // requests)),
                "context": rng.choice([0, 0, _log(rng, 1, 1024)])}
    if kind != "attention":
        case["window"] = _log(rng, 64, 2048)
    if kind == "window":
        case["keep"] = rng.choice([0, 4, 16])
    return case


# ---- what a case is made of -------------------------------------------------------------------------------------------
def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _lengths(case):
    """(tokens each request brings, tokens it had before): no two requests alike, the first the longest."""
    n, t, c = case["requests"], case["tokens"], case.get("context", 0)
    new = [t - (i * 7919) % (t // 3 + 1) if i else t for i in range(n)]
    had = [c - (i * 104729) % (c // 2 + 1) if i else c for i in range(n)]
    return new, had


def _generator(seed, name):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:8], "little") & 0x7FFFFFFFFFFFFFFF)
    return g


def _normal(seed, name, shape, std, dtype=torch.float32):
    t = torch.randn(tuple(shape), generator=_generator(seed, name), dtype=torch.float32, device=DEVICE) * std
    return t.to(dtype)


def _uniform(seed, name, shape, low, high):
    return low + (high - low) * torch.rand(tuple(shape), generator=_generator(seed, name), dtype=torch.float32, device=DEVICE)


def _yarn():
    return {"kind": "yarn", "factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}


def _spec(case):
    """(family, part description) of a layer case."""
    kind, w = case["kind"], case["width"]
    if kind == "attention":
        heads, kv, d, _ = LLAMA[w]
        return "mixer", PartSpec("attention", {"hidden": w, "heads": heads, "kv_heads": kv, "head_dim": d,
                                               "position": PartSpec("rotary", {"rotary_dim": d, "theta": 500000.0, "pairing": "half"})})
    if kind == "mlp":
        return "feed_forward", PartSpec("swiglu", {"hidden": w, "intermediate": LLAMA[w][3]})
    heads, experts, top, ff = WIDTHS[w]
    if kind == "experts":
        if case["router"] == "softmax":
            return "feed_forward", PartSpec("routed_experts", {
                "hidden": w, "experts": experts, "top": top, "ff": ff, "score": "softmax", "renormalise": True, "renormalise_eps": 1e-20,
                "scale_input": False, "activation": "swiglu", "shared": {"ff": ff, "gated": True}})
        return "feed_forward", PartSpec("routed_experts", {
            "hidden": w, "experts": experts, "top": top, "ff": ff, "score": "sigmoid", "renormalise": False, "scale_input": True,
            "activation": "clamped_swish", "limit": 7.0, "alpha": 1.702})
    if kind == "window":
        return "mixer", PartSpec("rotary_sink_attention", {
            "hidden": w, "heads": heads, "kv_heads": max(1, heads // 4), "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "bias": True,
            "qk_norm_eps": 1e-5, "sink": True, "window": case["window"], "keep_first": case["keep"],
            "position": PartSpec("rotary", {"rotary_dim": 64, "theta": 500000.0, "pairing": "half", "scaling": {"kind": "linear", "factor": 4.0}})})
    if kind == "latent":
        return "mixer", PartSpec("latent_attention", {
            "hidden": w, "heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 192, "scale": 192 ** -0.5, "rot_base": 10000.0,
            "rot_dims": 64, "pairing": "half", "eps": 1e-5, "rot_scaling": _yarn(), "window": case["window"]})
    if kind == "delta":
        extra = ({"decay_per": "head", "low_rank": False, "gate": "silu"} if case["rate"] == "head" else {"rank": 64})
        return "mixer", PartSpec("gated_delta", dict({"hidden": w, "heads": heads, "kv_heads": heads // 2 if case["rate"] == "head" else heads,
                                                      "dim": 128, "vdim": 128, "taps": 4, "eps": 1e-5}, **extra))
    return "mixer", PartSpec("lightning", {"hidden": w, "heads": heads, "dim": 128, "vdim": 128, "eps": 1e-5,
                                           "decay": [1.0 - 2.0 ** (-5.0 - 4.0 * h / heads) for h in range(heads)]})


def _tensor(case, seed, name, shape):
    """A layer's weight as the weight file holds it: vectors float, matrices in the compute type."""
    if name.endswith("norm"):
        return 1.0 + _normal(seed, name, shape, 0.1)
    if name == "A_log":                                       # decay rates spread as trained models have them
        return _uniform(seed, name, shape, 1.0, 16.0).log()
    if name == "dt_bias":                                     # softplus(dt_bias) between 0.001 and 0.1
        dt = _uniform(seed, name, shape, math.log(1e-3), math.log(1e-1)).exp()
        return dt + torch.log(-torch.expm1(-dt))
    if name.endswith(".b") or name == "sink":
        return _normal(seed, name, shape, 0.5)
    if name.endswith(".conv"):
        return _normal(seed, name, shape, 0.5, _dtype(case))
    return _normal(seed, name, shape, 1.0 / math.sqrt(shape[-1]), _dtype(case))


def _shapes(case):
    return {d.name: tuple(d.shape) for d in _describe(case).tensor_decls()}


def _describe(case):
    family, spec = _spec(case)
    return build_part(family, spec, Runtime.describe_only())


def _input(case, seed, tokens):
    return _normal(seed, "input", (tokens, case["width"]), 1.0, _dtype(case))


def _pages(case, seed, new, had):
    """Pages dealt out at random, as a server's pool hands them out after a while: [requests, blocks]."""
    blocks = [-(-(a + b) // PAGE) for a, b in zip(new, had)]
    order = np.random.RandomState(int(seed) & 0x7FFFFFFF).permutation(sum(blocks) + 3)
    table = np.full((len(new), max(blocks)), -1, dtype=np.int32)
    at = 0
    for i, n in enumerate(blocks):
        table[i, :n] = order[at: at + n]
        at += n
    return table, sum(blocks) + 3


def _cached(case, seed, pages, heads, dim):
    """Keys (and values) of the tokens before this step."""
    k = _normal(seed, "keys", (pages, heads, PAGE, dim), 1.0, _dtype(case))
    return k, k if case["kind"] == "latent" else _normal(seed, "values", (pages, heads, PAGE, dim), 1.0, _dtype(case))


def prepare(case, seed):
    if case["kind"] == "llama":
        r, prompt, new = case["requests"], case["prompt"], case["new"]
        eng = Engine.from_config(load_preset("llama-3.2-1b"), seed=seed, norm_std=0.1, engine_config=EngineConfig(
            page_size=PAGE, num_pages=r * (-(-(prompt + new) // PAGE) + 1), max_slots=r, max_tokens_per_step=4096, max_context=4096))
        return {"case": case, "engine": eng, "tokens": _tokens(case, seed)}
    dtype = _dtype(case)
    family, spec = _spec(case)
    kernels = load_kernels(DEVICE, (), verbose=False)
    part = build_part(family, spec, Runtime(kernels, DEVICE, dtype))
    part.load({d.name: _tensor(case, seed, d.name, d.shape) if d.role == "vector" else _tensor(case, seed, d.name, d.shape).to(dtype)
               for d in part.tensor_decls()})
    if family == "feed_forward":
        return {"case": case, "part": part, "kernels": kernels, "h": _input(case, seed, case["tokens"])}
    new, had = _lengths(case)
    rows, total = len(new), sum(new)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEVICE)
    cu = np.concatenate([[0], np.cumsum(new)])
    row_of = np.repeat(np.arange(rows), new)
    order = sorted(range(rows), key=lambda i: -new[i])
    decode = total == rows
    shape = BatchShape(rows, total, max(new), min(new), max(a + b for a, b in zip(new, had)), decode,
                       rows_by_q=None if decode else ints(order), neg_q_sorted=None if decode else tuple(-new[i] for i in order))
    need = part.cache_need()
    table, pages = _pages(case, seed, new, had) if need.has_pages else (np.zeros((rows, 1), np.int32), 0)
    k, v = _cached(case, seed, pages, need.kv_heads, need.head_dim) if need.has_pages else (None, None)
    states = {name: torch.zeros((rows,) + tuple(s), dtype=torch.float32, device=DEVICE) for name, s in need.states}
    ctx = StepContext(
        rt=part.rt, shape=shape, tokens=ints([0] * total),
        positions=ints((np.arange(total) - cu[row_of] + np.array(had)[row_of]).tolist()), token_row=ints(row_of.tolist()), cu_q=ints(cu.tolist()),
        kv_len=ints([a + b for a, b in zip(new, had)]), slots=ints(list(range(rows))), logit_rows=ints([0]),
        block_tables=[torch.from_numpy(table).to(DEVICE)])
    view = CacheView(group=0, k=k, v=v, page_size=PAGE, writes=True, window=need.window, states=states)
    return {"case": case, "part": part, "kernels": kernels, "h": _input(case, seed, total), "ctx": ctx, "view": view}


def _tokens(case, seed):
    """Per request: its prompt's ids and the ids decoded after it (given, as a replayed trace gives them)."""
    rs = np.random.RandomState(int(seed) & 0x7FFFFFFF)
    return [rs.randint(0, 128256, case["prompt"] - (i * 31) % (case["prompt"] // 3 + 1) + case["new"] - 1).tolist() for i in range(case["requests"])]


def run(state):
    case = state["case"]
    if case["kind"] == "llama":
        eng, ids, new = state["engine"], state["tokens"], case["new"]
        portions = [t[: len(t) - new + 1] for t in ids]
        out = [eng.step([StepEntry(i, p, [len(p) - 1]) for i, p in enumerate(portions)]).clone()]
        for j in range(new - 1):
            out.append(eng.step([StepEntry(i, [t[len(t) - new + 1 + j]], [0]) for i, t in enumerate(ids)]).clone())
        for i in range(len(ids)):
            eng.end(i)
        return out
    part, h = state["part"], state["h"]
    if "ctx" not in state:
        with state["kernels"].on_current_stream():
            return part.forward(h, None)
    ctx, view = state["ctx"], state["view"]
    ctx.memo.clear()                                          # (a step starts with nothing derived from its arrays)
    for s in view.states.values():
        s.zero_()                                             # (as when a request gets its slot)
    with state["kernels"].on_current_stream():
        out = part.forward(h, ctx, view)
    if view.states:
        return {"out": out, **view.states}
    return {"out": out, "k": view.k} if view.v is view.k else {"out": out, "k": view.k, "v": view.v}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def _weights(case):
    return sum(math.prod(s) for s in _shapes(case).values())


def _hit(tokens, experts, top):
    """Experts that a step of this many tokens is expected to choose."""
    return experts * (1.0 - (1.0 - top / experts) ** tokens)


def _pairs_read(case):
    """Key/query pairs, and keys of a request that any of its queries reads."""
    new, had = _lengths(case)
    window, keep = case.get("window") or 1 << 30, case.get("keep", 0)
    pairs = read = 0
    for a, b in zip(new, had):
        p = np.arange(b, a + b)
        kept = np.minimum(keep, np.maximum(0, p + 1 - window))
        pairs += int((np.minimum(p + 1, window) + kept).sum())
        read += min(a + b, window + a - 1 + keep)
    return pairs, read


def work(case):
    if case["kind"] == "llama":
        ids = [case["prompt"] - (i * 31) % (case["prompt"] // 3 + 1) for i in range(case["requests"])]
        layers = 16 * (2048 * (2048 + 1024) + 2048 * 2048 + 3 * 2048 * 8192)
        head = 2048 * 128256
        new, r = case["new"], case["requests"]
        tokens = sum(ids) + r * (new - 1)
        pairs = sum(n * (n + 1) // 2 + sum(n + j + 1 for j in range(new - 1)) for n in ids)
        kv = 16 * 2 * 1024 * 2                                # bytes of keys and values a cached token has
        read = sum(sum(n + j + 1 for j in range(new - 1)) for n in ids)
        return {"bytes": 2 * new * (layers + head) + kv * (tokens + read) + 4 * 128256 * r * new,
                "flops": 2 * layers * tokens + 2 * head * r * new + 16 * 4 * 2048 * pairs}
    e = _dtype(case).itemsize
    w, params = case["width"], _weights(case)
    if case["kind"] == "mlp":
        t = case["tokens"]
        return {"bytes": e * (params + 2 * t * w), "flops": 2 * params * t}
    if case["kind"] == "experts":
        _, experts, top, ff = WIDTHS[w]
        t = case["tokens"]
        each, extra = 3 * w * ff, params - experts * 3 * w * ff
        return {"bytes": e * (int(_hit(t, experts, top) * each) + extra + 2 * t * w), "flops": 2 * t * (top * each + extra)}
    new, had = _lengths(case)
    t = sum(new)
    io = e * (params + 2 * t * w)
    if case["kind"] in ("attention", "window", "latent"):
        pairs, read = _pairs_read(case)
        if case["kind"] == "latent":
            heads = WIDTHS[w][0]
            return {"bytes": io + e * 256 * read, "flops": 2 * params * t + 2 * heads * (256 + 192) * pairs}
        heads, kv, d = LLAMA[w][:3] if case["kind"] == "attention" else (WIDTHS[w][0], max(1, WIDTHS[w][0] // 4), 128)
        return {"bytes": io + e * 2 * kv * d * read, "flops": 2 * params * t + 4 * heads * d * pairs}
    heads = WIDTHS[w][0]
    per = 8 if case["kind"] == "delta" else 5                 # operations an element of the state needs for a token
    return {"bytes": io + 4 * heads * 128 * 128 * len(new), "flops": 2 * params * t + per * heads * 128 * 128 * t}


def tolerance(case):
    return TOLERANCE[case["kind"]][0 if _dtype(case) == torch.bfloat16 else 1]


# Largest relative error another correct implementation may show (bfloat16, float32): about four times what the path differs
# from its 64-bit form (measured: llama 0.02; bfloat16 layers 0.0015 to 0.005; float32 layers 3e-7 to 1.4e-6).
TOLERANCE = {
    "llama": ({"rel": 8e-2}, {"rel": 1e-4}),
    "attention": ({"rel": 1.6e-2}, {"rel": 5e-6}),
    "mlp": ({"rel": 1.4e-2}, {"rel": 6e-6}),
    "experts": ({"rel": 1.4e-2}, {"rel": 1e-5}),
    "window": ({"rel": 1e-2}, {"rel": 1e-5}),
    "latent": ({"rel": 2e-2}, {"rel": 5e-6}),
    "delta": ({"rel": 2e-2}, {"rel": 1e-5}),
    "lightning": ({"rel": 1.4e-2}, {"rel": 5e-6}),
}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------
def _rms(x, weight, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * (1.0 if weight is None else weight)


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, positions, inv_freq, mult=1.0):
    """x [T, H, D]: pairs (i, i + n) of the first 2 n elements turned; angles are float32 numbers by definition."""
    n = inv_freq.numel()
    angle = (positions.float()[:, None] * inv_freq.float()[None]).to(F64)[:, None]
    c, s = angle.cos() * mult, angle.sin() * mult
    a, b = x[..., :n], x[..., n: 2 * n]
    return torch.cat([a * c - b * s, a * s + b * c, x[..., 2 * n:]], -1)


def _inv_freq(dims, theta, scaling=None):
    f = 1.0 / (theta ** (torch.arange(0, dims, 2).float() / dims))
    if scaling is None:
        return f.to(DEVICE)
    if scaling["kind"] == "linear":
        return (f / scaling["factor"]).to(DEVICE)
    if scaling["kind"] == "yarn":
        pair = lambda turns: dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(theta))
        lo, hi = max(math.floor(pair(scaling["fast"])), 0), min(math.ceil(pair(scaling["slow"])), dims - 1)
        i = torch.arange(dims // 2, dtype=F64)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        g = theta ** (-2.0 * i / dims)
        return (g / scaling["factor"] * ramp + g * (1.0 - ramp)).float().to(DEVICE)
    wave = 2 * math.pi / f                                    # the llama3 rule
    lo, hi, old = scaling["low_freq_factor"], scaling["high_freq_factor"], scaling["original_max_position_embeddings"]
    smooth = (old / wave - lo) / (hi - lo)
    mixed = (1 - smooth) * f / scaling["factor"] + smooth * f
    return torch.where(wave < old / hi, f, torch.where(wave > old / lo, f / scaling["factor"], mixed)).to(DEVICE)


def _attend(q, k, v, scale, first, window=None, keep=0, sink=None):
    """q [T, H, D] at positions first..; k [S, G, D], v [S, G, E] -> [T, H, E]; a block of queries at a time."""
    t, h, _ = q.shape
    s, g, _ = k.shape
    out = torch.empty((t, h, v.shape[-1]), dtype=F64, device=q.device)
    j = torch.arange(s, device=q.device)
    kh, vh = k.permute(1, 2, 0), v.transpose(0, 1)            # [G, D, S], [G, S, E]
    for a in range(0, t, 256):
        qs = q[a: a + 256]
        n = qs.shape[0]
        i = first + a + torch.arange(n, device=q.device)[:, None]
        see = j[None] <= i
        if window:
            see &= (i - j[None] < window) | (j[None] < keep)
        z = (qs.reshape(n, g, h // g, -1).permute(1, 2, 0, 3) @ kh[:, None]) * scale           # [G, H/G, n, S]
        z = z.masked_fill(~see, -math.inf)
        m = z.amax(-1, keepdim=True)
        if sink is not None:
            m = torch.maximum(m, sink.view(g, h // g, 1, 1))
        p = (z - m).exp()
        den = p.sum(-1, keepdim=True) + (0.0 if sink is None else (sink.view(g, h // g, 1, 1) - m).exp())
        out[a: a + n] = ((p / den) @ vh[:, None]).permute(2, 0, 1, 3).reshape(n, h, -1)
    return out


def _rows_before(pool, table, n):
    """The first n cached rows of a request: [n, heads, dim]."""
    p = torch.arange(n, device=DEVICE)
    pages = torch.from_numpy(table.astype(np.int64)).to(DEVICE)[p // PAGE]
    return pool[pages, :, p % PAGE].to(F64)


def _exact_llama(case, seed):
    cfg = load_preset("llama-3.2-1b")
    w = lambda name, shape: _normal(seed, name, shape, 0.02, torch.bfloat16).to(F64)
    norm = lambda name: 1.0 + _normal(seed, name, (2048,), 0.1).to(F64)
    ids, new = _tokens(case, seed), case["new"]
    flat = torch.tensor([t for r in ids for t in r], device=DEVICE)
    at = np.concatenate([[0], np.cumsum([len(r) for r in ids])]).tolist()
    positions = torch.cat([torch.arange(len(r), device=DEVICE) for r in ids])
    inv = _inv_freq(64, cfg.rope_theta, {"kind": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                                         "original_max_position_embeddings": 8192})
    table = _normal(seed, "model.embed_tokens.weight", (128256, 2048), 0.02, torch.bfloat16)
    x = table[flat].to(F64)
    for layer in range(16):
        p = f"model.layers.{layer}."
        h = _rms(x, norm(p + "input_layernorm.weight"), 1e-5)
        q = _rotate((h @ w(p + "self_attn.q_proj.weight", (2048, 2048)).T).view(-1, 32, 64), positions, inv)
        k = _rotate((h @ w(p + "self_attn.k_proj.weight", (512, 2048)).T).view(-1, 8, 64), positions, inv)
        v = (h @ w(p + "self_attn.v_proj.weight", (512, 2048)).T).view(-1, 8, 64)
        a = torch.cat([_attend(q[s:e], k[s:e], v[s:e], 0.125, 0) for s, e in zip(at, at[1:])])
        x = x + a.reshape(-1, 2048) @ w(p + "self_attn.o_proj.weight", (2048, 2048)).T
        h = _rms(x, norm(p + "post_attention_layernorm.weight"), 1e-5)
        g = _silu(h @ w(p + "mlp.gate_proj.weight", (8192, 2048)).T) * (h @ w(p + "mlp.up_proj.weight", (8192, 2048)).T)
        x = x + g @ w(p + "mlp.down_proj.weight", (2048, 8192)).T
    rows = [e - new + j for j in range(new) for e in at[1:]]
    logits = _rms(x[rows], norm("model.norm.weight"), 1e-5) @ table.to(F64).T
    r = len(ids)
    return [logits[j * r: (j + 1) * r].float() for j in range(new)]


def _softplus(x):
    return torch.nn.functional.softplus(x, beta=1.0, threshold=1e9)


def _padded(x, at):
    """[T, ...] -> [R, longest, ...] with zeros after each request's end."""
    n = [e - s for s, e in zip(at, at[1:])]
    out = x.new_zeros((len(n), max(n)) + tuple(x.shape[1:]))
    for i, (s, e) in enumerate(zip(at, at[1:])):
        out[i, : e - s] = x[s:e]
    return out


def _packed(x, at):
    return torch.cat([x[i, : e - s] for i, (s, e) in enumerate(zip(at, at[1:]))])


def _exact_recurrence(case, seed, x, t):
    new, _ = _lengths(case)
    at = np.concatenate([[0], np.cumsum(new)]).tolist()
    heads = WIDTHS[case["width"]][0]
    rows = len(new)
    live = _padded(x.new_ones((x.shape[0], 1)), at)[..., None]                 # [R, L, 1, 1]
    s = x.new_zeros((rows, heads, 128, 128))
    states = {}
    if case["kind"] == "lightning":
        q, k, v = (_padded(_silu(x @ t[n].T).view(-1, heads, 128), at) for n in "qkv")
        decay = torch.tensor([1.0 - 2.0 ** (-5.0 - 4.0 * i / heads) for i in range(heads)], dtype=torch.float32, device=DEVICE).to(F64)
        keep = torch.where(live > 0, decay.view(1, 1, heads, 1), torch.ones_like(decay).view(1, 1, heads, 1))
        y = torch.empty_like(v)
        for i in range(v.shape[1]):
            s = keep[:, i, :, :, None] * s + k[:, i, :, :, None] * v[:, i, :, None]
            y[:, i] = (s * q[:, i, :, :, None]).sum(2)
        o = _rms(_packed(y, at).reshape(x.shape[0], -1), t["norm"], 1e-5) * torch.sigmoid(x @ t["g"].T)
        return {"out": (o @ t["o"].T).float(), "state": s.float()}
    per_head = case["rate"] == "head"
    kv = heads // 2 if per_head else heads
    proj = torch.cat([x @ t[n].T for n in "qkv"], -1)
    w = torch.cat([t[n + ".conv"] for n in "qkv"], 0)                          # [C, 4]
    padded = _padded(proj, at)
    c = sum(torch.nn.functional.pad(padded, (0, 0, 3 - j, 0))[:, : padded.shape[1]] * w[:, j] for j in range(4))
    c = _silu(c)
    tail = torch.stack([torch.nn.functional.pad(proj[a:b], (0, 0, 3, 0))[-3:] for a, b in zip(at, at[1:])])
    qk = kv * 128
    unit = lambda z: z * torch.rsqrt(z.square().sum(-1, keepdim=True) + 1e-6)
    many = lambda z: unit(z.unflatten(-1, (kv, 128))).repeat_interleave(heads // kv, dim=2)
    q, k, v = many(c[..., :qk]) * 128 ** -0.5, many(c[..., qk: 2 * qk]) * live, c[..., 2 * qk:].unflatten(-1, (heads, 128))
    beta = _padded(torch.sigmoid(x @ t["b"].T), at)
    if per_head:
        rate, gate = (x @ t["rate"].T)[..., None], x @ t["gate"].T
        bias, act = t["dt_bias"].view(heads, 1), _silu
    else:
        rate, gate = (x @ t["a1"].T @ t["a2"].T).view(-1, heads, 128), x @ t["g1"].T @ t["g2"].T
        bias, act = t["dt_bias"].view(heads, 128), torch.sigmoid
    g = _padded(-t["A_log"].exp().view(heads, 1) * _softplus(rate + bias), at) * live
    g = g.exp()
    y = torch.empty_like(v)
    for i in range(v.shape[1]):
        s = g[:, i, :, :, None] * s
        u = beta[:, i, :, None] * (v[:, i] - (s * k[:, i, :, :, None]).sum(2))
        s = s + k[:, i, :, :, None] * u[:, :, None]
        y[:, i] = (s * q[:, i, :, :, None]).sum(2)
    o = _rms(_packed(y, at), t["norm"], 1e-5).reshape(x.shape[0], -1) * act(gate)
    states = {"state": s.float(), "conv_tail": tail.float()}
    return {"out": (o @ t["o"].T).float(), **states}


def _exact_experts(case, x, t):
    _, experts, top, _ = WIDTHS[case["width"]]
    z = x @ t["router"].T
    plain = case["router"] == "sigmoid"
    score = torch.sigmoid(z) if plain else torch.softmax(z, -1)
    w, idx = score.sort(dim=-1, descending=True, stable=True)
    w, idx = w[:, :top], idx[:, :top]
    if not plain:
        w = w / w.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(experts):
        tok, place = (idx == e).nonzero(as_tuple=True)
        if tok.numel() == 0:
            continue
        wt = w[tok, place][:, None]
        h = x[tok] * wt if plain else x[tok]
        g, u = h @ t[f"e{e}.gate"].T, h @ t[f"e{e}.up"].T
        if plain:
            g = g.clamp(max=7.0)
            a = g * torch.sigmoid(1.702 * g) * (u.clamp(-7.0, 7.0) + 1.0)
            wt = 1.0
        else:
            a = _silu(g) * u
        out.index_add_(0, tok, (a @ t[f"e{e}.down"].T) * wt)
    if not plain:
        shared = (_silu(x @ t["shared.gate"].T) * (x @ t["shared.up"].T)) @ t["shared.down"].T
        out = out + torch.sigmoid(x @ t["shared.sg"].T) * shared
    return out.float()


def _exact_attention(case, seed, x, t):
    new, had = _lengths(case)
    at = np.concatenate([[0], np.cumsum(new)]).tolist()
    kind, w = case["kind"], case["width"]
    table, pages = _pages(case, seed, new, had)
    positions = torch.cat([torch.arange(b, a + b, device=DEVICE) for a, b in zip(new, had)])
    sink, window, keep = None, case.get("window"), case.get("keep", 0)
    if kind == "attention":
        heads, kv, d, _ = LLAMA[w]
        inv, scale = _inv_freq(d, 500000.0), d ** -0.5
        # cached keys have rotary partners side by side
        near = torch.stack([torch.arange(d // 2), torch.arange(d // 2) + d // 2], 1).reshape(-1).to(DEVICE)
        q = _rotate((x @ t["q_proj.weight"].T).view(-1, heads, d), positions, inv)[..., near]
        k = _rotate((x @ t["k_proj.weight"].T).view(-1, kv, d), positions, inv)[..., near]
        v = (x @ t["v_proj.weight"].T).view(-1, kv, d)
    elif kind == "window":
        heads, kv, d = WIDTHS[w][0], max(1, WIDTHS[w][0] // 4), 128
        inv, scale, sink = _inv_freq(64, 500000.0, {"kind": "linear", "factor": 4.0}), d ** -0.5, t["sink"]
        q = _rms(x @ t["q"].T + t["q.b"], t["q.norm"], 1e-5).view(-1, heads, d)
        k = _rms(x @ t["k"].T + t["k.b"], t["k.norm"], 1e-5).view(-1, kv, d)
        q, k, v = _rotate(q, positions, inv), _rotate(k, positions, inv), (x @ t["v"].T + t["v.b"]).view(-1, kv, d)
    else:
        heads, kv, d = WIDTHS[w][0], 1, 256
        inv, scale, mult = _inv_freq(64, 10000.0, _yarn()), 192 ** -0.5, 0.1 * math.log(8.0) + 1.0
        q = (x @ t["q"].T).view(-1, heads, 192)
        q_rot = _rotate(q[..., 128:], positions, inv, mult)
        row = x @ t["dkv"].T
        c = _rms(row[:, :192], t["dkv.norm"], 1e-5)
        k = torch.cat([c, _rotate(row[:, None, 192:], positions, inv, mult)[:, 0]], -1)[:, None]
        v = c[:, None]
        q = torch.cat([torch.einsum("thd,hdr->thr", q[..., :128], t["uk"].view(heads, 128, 192)), q_rot], -1)
    k_pool, v_pool = _cached(case, seed, pages, kv, d)
    parts = []
    for i, (s, e) in enumerate(zip(at, at[1:])):
        ks = torch.cat([_rows_before(k_pool, table[i], had[i]), k[s:e]])
        vs = torch.cat([_rows_before(v_pool, table[i], had[i])[..., : v.shape[-1]], v[s:e]])
        parts.append(_attend(q[s:e], ks, vs, scale, had[i], window, keep, sink))
    a = torch.cat(parts)
    if kind == "attention":
        out = a.reshape(x.shape[0], -1) @ t["o_proj.weight"].T
    elif kind == "window":
        out = a.reshape(x.shape[0], -1) @ t["o"].T + t["o.b"]
    else:
        out = torch.einsum("thr,hvr->thv", a, t["uv"].view(heads, 128, 192)).reshape(x.shape[0], -1) @ t["o"].T
    return {"out": out.float(), "k": None} if kind == "latent" else {"out": out.float(), "k": None, "v": None}


def exact(case, seed):
    if case["kind"] == "llama":
        return _exact_llama(case, seed)
    t = {name: _tensor(case, seed, name, shape).to(F64) for name, shape in _shapes(case).items()}
    if case["kind"] in ("mlp", "experts"):
        x = _input(case, seed, case["tokens"]).to(F64)
        if case["kind"] == "experts":
            return _exact_experts(case, x, t)
        return ((_silu(x @ t["gate_proj.weight"].T) * (x @ t["up_proj.weight"].T)) @ t["down_proj.weight"].T).float()
    x = _input(case, seed, sum(_lengths(case)[0])).to(F64)
    if case["kind"] in ("delta", "lightning"):
        return _exact_recurrence(case, seed, x, t)
    return _exact_attention(case, seed, x, t)

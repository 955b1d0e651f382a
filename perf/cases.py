"""What the speed of this framework is measured on: steps of whole decoders through the step function, and single layers.

A step is what a server asks for again and again: ``StepExecutor.step`` over requests that already hold a context, beside a new
prompt or without one. The single layers are the ones in which the seven architectures differ, each called as a model calls it, at
the layer sizes of ``bench.py`` (widths 1,024 and 2,048) over the prompts of one step.

Every case is a dict of plain values: ``kind`` names the path, ``width``, ``lengths`` (tokens a request, "2048,777"), ``batch``
(requests that decode), ``context`` (tokens that each holds), ``portion`` (tokens of a new prompt in the same step).
"""
import math

import torch
import torch.nn.functional as F

from roost_b200.cache.manager import CacheManager, build_groups
from roost_b200.cache.storage import CacheStorage
from roost_b200.config.lovurax import LovuraxConfig
from roost_b200.config.qwen3 import Qwen3Config
from roost_b200.config.spec import (GatedLinearAttentionSpec, LatentAttentionSpec, Mamba1Spec, Mamba2Spec, PositionSpec, RoutedMlpSpec,
                                    SigmoidAttentionSpec, SinkAttentionSpec)
from roost_b200.engine.batch import BatchBuilder
from roost_b200.engine.executor import StepEntry, StepExecutor
from roost_b200.engine.model import Model, parameter_declarations
from roost_b200.kernels import library
from roost_b200.parts import Runtime
from roost_b200.parts.base import FEED_FORWARDS, MIXERS

PAGE = 16
EPS = 1e-6
F64 = torch.float64


def listed():
    return [
        # one user waiting for the next token of a small model: latency, launches and gaps are the time
        {"name": "decode 0.6b batch 1", "kind": "qwen3", "size": "0.6b", "layers": 28, "dtype": "bfloat16", "batch": 1, "context": 1000, "portion": 0},
        # a server's decode step at the sizes of the framework's headline figure, a share of the layers
        {"name": "decode 8b batch 8", "kind": "qwen3", "size": "8b", "layers": 4, "dtype": "bfloat16", "batch": 8, "context": 4001, "portion": 0},
        # a server's mixed step under a budget of 512 tokens: a portion of a new prompt beside the requests that decode
        {"name": "mixed step 0.6b", "kind": "qwen3", "size": "0.6b", "layers": 8, "dtype": "bfloat16", "batch": 31, "context": 900, "portion": 481},
        # the 32-bit path, which fidelity runs use: a prompt beside two requests that decode
        {"name": "mixed step 0.6b float32", "kind": "qwen3", "size": "0.6b", "layers": 2, "dtype": "float32", "batch": 2, "context": 500, "portion": 510},
        # a decode step of a decoder with retention, sigmoid weights and a latent attention
        {"name": "decode retention design", "kind": "lovurax", "width": 1024, "layers": 4, "dtype": "bfloat16", "batch": 8, "context": 1000, "portion": 0},
        # single layers over the prompts of a step
        {"name": "latent attention", "kind": "latent", "width": 2048, "window": 2048, "lengths": "2048,1000"},
        {"name": "attention with a sink", "kind": "sink", "width": 2048, "window": 0, "lengths": "1500,500,2048"},
        {"name": "attention, sigmoid weights", "kind": "sigmoid", "width": 1024, "window": 0, "lengths": "2048,777"},
        {"name": "state space, matrix state", "kind": "mamba2", "width": 2048, "lengths": "2048,1037,1011"},
        {"name": "selective scan", "kind": "mamba1", "width": 1024, "lengths": "2048,300"},
        {"name": "gated linear attention", "kind": "gla", "width": 2048, "lengths": "3000,1096"},
        {"name": "routed experts", "kind": "experts", "width": 2048, "lengths": "2048"},
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["qwen3", "qwen3", "lovurax", "latent", "sink", "sigmoid", "mamba2", "mamba1", "gla", "experts"])
    if kind == "qwen3":
        f32 = rng.random() < 0.25
        return {"kind": kind, "size": "0.6b" if f32 else rng.choice(["0.6b", "8b"]), "layers": rng.randint(1, 2 if f32 else 4),
                "dtype": "float32" if f32 else "bfloat16", "batch": _spread(rng, 1, 4 if f32 else 32), "context": _spread(rng, 64, 700 if f32 else 3000),
                "portion": rng.choice([0, _spread(rng, 17, 512)])}
    if kind == "lovurax":
        return {"kind": kind, "width": 1024, "layers": 4, "dtype": "bfloat16", "batch": _spread(rng, 1, 16), "context": _spread(rng, 64, 1500),
                "portion": rng.choice([0, _spread(rng, 17, 512)])}
    rows = rng.choice([1, 1, 2, 3])
    total = _spread(rng, 200, 3000)
    cuts = sorted(rng.sample(range(1, total), rows - 1))
    lengths = [b - a for a, b in zip([0] + cuts, cuts + [total])]
    case = {"kind": kind, "width": rng.choice([1024, 2048]), "lengths": ",".join(map(str, lengths))}
    if kind == "latent":
        case["window"] = rng.choice([0, _spread(rng, 256, 2048)])
    if kind in ("sink", "sigmoid"):
        case["window"] = rng.choice([0, _spread(rng, 128, 1024)]) if kind == "sink" else 0
    return case


def _lengths(c):
    return [int(v) for v in c["lengths"].split(",")]


# ------------------------------------------------------------------------------------------------------------- sizes of the paths
def _qwen3_config(c):
    sizes = {"0.6b": dict(hidden_size=1024, num_attention_heads=16, intermediate_size=3072, tie_word_embeddings=True),
             "8b": dict(hidden_size=4096, num_attention_heads=32, intermediate_size=12288, tie_word_embeddings=False)}[c["size"]]
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=c["layers"], num_key_value_heads=8, head_dim=128,
                vocab_size=151936, rope_theta=1000000.0, rms_norm_eps=EPS, max_position_embeddings=40960, torch_dtype="bfloat16", **sizes)


def _decays(heads):
    return [1.0 - 2.0 ** (-5 - 3 * h / max(heads - 1, 1)) for h in range(heads)]


def _lovurax_config(c):
    W, dim = c["width"], 64 if c["width"] < 2048 else 128
    retention = {"type": "retention", "mixer": {"heads": W // 128, "dim": 64, "vdim": 128, "rot": {"dims": 64, "base": 10000.0}, "decay": _decays(W // 128)}}
    attention = {"type": "attention", "mixer": {"heads": 16, "kv_heads": 4, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "q_temp": {"coef": 0.2, "every": 512}}}
    latent = {"type": "latent_attention", "mixer": {"heads": 16, "dim": dim, "vdim": dim, "kv_rank": W // 4, "scale": dim ** -0.5}}
    order = (retention, attention, attention, latent)
    return {"architecture": "Lovurax", "vocab": 32768, "width": W, "norm": {"eps": EPS}, "logit_scale": 1.0,
            "layers": [dict(order[i % 4], mlp={"kind": "dense", "ff": 4 * W}) for i in range(c["layers"])]}


def _model_spec(c):
    if c["kind"] == "qwen3":
        cfg = _qwen3_config(c)
        return Qwen3Config.from_dict(cfg).to_spec(cfg["tie_word_embeddings"])
    return LovuraxConfig.from_dict(_lovurax_config(c)).to_spec()


def _part_spec(c):
    W, dim, kind = c["width"], 64 if c["width"] < 2048 else 128, c["kind"]
    if kind == "latent":
        window = c["window"] or None
        return LatentAttentionSpec(hidden=W, num_heads=16, nope_dim=dim, rope_dim=dim // 2, v_dim=dim, kv_rank=W // 4, scale=(1.5 * dim) ** -0.5, window=window,
                                   cache_window=window, latent_eps=EPS, position=PositionSpec(kind="rope_neox", rotary_dim=dim // 2, theta=1000000.0))
    if kind == "sink":
        return SinkAttentionSpec(hidden=W, num_heads=16, num_kv_heads=4, head_dim=dim, v_dim=dim, scale=dim ** -0.5, sink=True, unit_norm_eps=EPS,
                                 window=c["window"] or None, position=PositionSpec(kind="rope_interleaved", rotary_dim=dim, theta=1000000.0))
    if kind == "sigmoid":
        return SigmoidAttentionSpec(hidden=W, num_heads=16, num_kv_heads=4, head_dim=dim, v_dim=dim, scale=dim ** -0.5, qk_norm_eps=EPS, temp_coef=0.2,
                                    temp_every=512, slopes=tuple(2.0 ** (-8.0 * (h + 1) / 16) for h in range(16)), head_bias=True, output_gate=True)
    if kind == "mamba2":
        groups = 8 if W >= 2048 else 1
        return Mamba2Spec(hidden=W, num_heads=W // 32, head_dim=64, state=128, groups=groups, conv_taps=4, norm_groups=groups, eps=EPS)
    if kind == "mamba1":
        return Mamba1Spec(hidden=W, inner=2 * W, state=16, dt_rank=W // 16, conv_taps=4)
    if kind == "gla":
        return GatedLinearAttentionSpec(hidden=W, num_heads=W // 128, head_dim=64, v_dim=128, tau=16.0, decay_rank=16, eps=EPS)
    big = W >= 2048
    return RoutedMlpSpec(hidden=W, experts=64 if big else 32, top=6 if big else 4, expert_intermediate=768 if big else 512,
                         shared_intermediate=1536 if big else 1024, activation="silu", score="sigmoid", weight_on="input")


def _part_class(c):
    return (FEED_FORWARDS if c["kind"] == "experts" else MIXERS).get(_part_spec(c).kind)


# ------------------------------------------------------------------------------------------------------------- inputs from a seed
def _generator(seed, n):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + n * 7919 + 17) % (1 << 62))


def _draw_parameter(decl, gen, dtype):
    """Values such as trained weights have: matrices N(0, 0.02), vectors around one, rates and biases as their part declares them."""
    out = torch.empty(decl.shape, dtype=dtype if decl.role == "matrix" else torch.bfloat16, device="cuda")
    if decl.init is not None and decl.init[0] == "uniform":
        return out.uniform_(decl.init[1], decl.init[2], generator=gen)
    mean, std = (decl.init[1], decl.init[2]) if decl.init is not None else ((0.0, 0.02) if decl.role == "matrix" else (1.0, 0.1))
    return out.normal_(mean, std, generator=gen)


def _model_parameters(c, seed):
    gen, dtype = _generator(seed, 1), getattr(torch, c["dtype"])
    return {scope: {k: _draw_parameter(d, gen, dtype) for k, d in sorted(decls.items())} for scope, decls in sorted(parameter_declarations(_model_spec(c)).items())}


def _part_parameters(c, seed):
    gen = _generator(seed, 2)
    return {k: _draw_parameter(d, gen, torch.bfloat16) for k, d in sorted(_part_class(c).parameters(_part_spec(c)).items())}


def _tokens(c, seed):
    """(token lists of the requests that decode, one more token than their context each; the new prompt)"""
    g = torch.Generator().manual_seed(int(seed) * 31 + 5)
    vocab = 151936 if c["kind"] == "qwen3" else 32768
    ids = torch.randint(0, vocab, (c["batch"], c["context"] + 1), generator=g).tolist()
    return ids, torch.randint(0, vocab, (c["portion"],), generator=g).tolist()


def _hidden(c, seed):
    """The normed input of a layer."""
    return torch.randn((sum(_lengths(c)), c["width"]), generator=_generator(seed, 3), device="cuda").to(torch.bfloat16)


# ------------------------------------------------------------------------------------------------------------- preparing and running
def prepare(case, seed):
    return _prepare_step(case, seed) if case["kind"] in ("qwen3", "lovurax") else _prepare_part(case, seed)


def run(state):
    return _run_step(state) if "executor" in state else _run_part(state)


def _prepare_step(c, seed):
    """A running server: the model is loaded and every request holds its context. As there, a step's sizes have come before."""
    model = Model(_model_spec(c), Runtime(getattr(torch, c["dtype"]), "cuda", library.load()))
    model.load(_model_parameters(c, seed))
    pages = c["batch"] * (c["context"] // PAGE + 2) + c["portion"] // PAGE + 2
    ex = StepExecutor(model, page_size=PAGE, num_pages=pages, max_requests=c["batch"] + 1)
    held, new = _tokens(c, seed)
    for r, ids in enumerate(held):
        for at in range(0, c["context"], 2048):
            ex.step([StepEntry(r, ids[at : min(at + 2048, c["context"])])])
    state = {"executor": ex, "context": c["context"], "entries": [StepEntry(r, [ids[-1]], [0]) for r, ids in enumerate(held)]}
    if new:
        state["entries"].append(StepEntry("new", new, [len(new) - 1]))
    states = [t.clone() for g, t in zip(ex.groups, ex.storage.tensors) if g.kind == "state"]
    for _ in range(2):
        _run_step(state)
    for t, old in zip([t for g, t in zip(ex.groups, ex.storage.tensors) if g.kind == "state"], states):
        t.copy_(old)
    return state


def _run_step(state):
    """One step; the requests then stand where they stood, so that the next pass is a step of the same sizes."""
    ex = state["executor"]
    logits = ex.step(state["entries"])
    for e in state["entries"]:
        if e.request_id == "new":
            ex.finish("new")
        else:
            ex.cache.commit(e.request_id, state["context"])
    return logits


def _prepare_part(c, seed):
    """One layer of a step over the prompts ``lengths``: its weights, its cache, the step's tables, the normed input."""
    runtime = Runtime(torch.bfloat16, "cuda", library.load())
    part = (FEED_FORWARDS if c["kind"] == "experts" else MIXERS).build(_part_spec(c), runtime)
    part.load(_part_parameters(c, seed))
    state = {"part": part, "x": _hidden(c, seed), "cache": None, "batch": None}
    if c["kind"] == "experts":
        return state
    lengths = _lengths(c)
    groups = build_groups([part.cache_need()], PAGE)
    manager = CacheManager(groups, [sum(n // PAGE + 1 for n in lengths) if g.kind == "paged" else len(lengths) for g in groups])
    storage = CacheStorage(groups, [p.capacity for p in manager.pools], torch.bfloat16, "cuda")
    rows = [(manager.extend(r, n), 0, [0] * n, []) for r, n in enumerate(lengths)]
    state["batch"] = BatchBuilder("cuda", manager).build(rows, 1)
    state["cache"] = storage.view(0)
    return state


def _run_part(state):
    """The layer's output, and what it leaves in its cache: a request's recurrent state, or the pages of keys and values. A pass over
    the same state again is the next portion of the same requests for a recurrence, and the same portion for an attention."""
    cache = state["cache"]
    if cache is None:
        return {"y": state["part"](state["x"], state["batch"])}
    y = state["part"](state["x"], state["batch"], cache)
    if cache.kind == "state":
        return {"y": y, "cache": cache.state[:-1]}
    return {"y": y, "cache": cache.k_pool}


# ------------------------------------------------------------------------------------------------------------- what a pass cannot do without
def _causal_pairs(n, window):
    return n * (n + 1) // 2 if not window or n <= window else window * (window + 1) // 2 + (n - window) * window


def work(case):
    c = case
    if c["kind"] == "qwen3":
        cfg, elem = _qwen3_config(c), 4 if c["dtype"] == "float32" else 2
        H, I, Q, KV = cfg["hidden_size"], cfg["intermediate_size"], cfg["num_attention_heads"] * 128, 1024
        layer = (Q + 2 * KV) * H + H * Q + 3 * H * I
        T, S = c["batch"] + c["portion"], c["batch"] + (1 if c["portion"] else 0)
        pairs = c["batch"] * (c["context"] + 1) + _causal_pairs(c["portion"], 0)
        weights = c["layers"] * layer + 151936 * H
        cache = c["layers"] * 2 * KV * (c["batch"] * c["context"] + T)
        return {"bytes": elem * (weights + cache) + 4 * S * 151936, "flops": 2.0 * T * c["layers"] * layer + 2.0 * S * 151936 * H + 4.0 * pairs * Q * c["layers"]}
    if c["kind"] == "lovurax":
        W, dim, B, S = c["width"], 64 if c["width"] < 2048 else 128, c["batch"], c["batch"] + (1 if c["portion"] else 0)
        T, r = B + c["portion"], W // 4
        pairs = B * (c["context"] + 1) + _causal_pairs(c["portion"], 0)
        weights, state, flops = 32768 * W, 0.0, 2.0 * S * 32768 * W
        for i in range(c["layers"]):
            m = {0: 4 * W * W, 1: 2 * 16 * dim * W + 2 * 4 * dim * W + 16 * dim * W, 2: 2 * 16 * dim * W + 2 * 4 * dim * W + 16 * dim * W,
                 3: 16 * dim * W + r * W + 2 * 16 * dim * r + 16 * W + W * 16 * dim}[i % 4]
            m += 2 * 4 * W * W + 2 * W * W
            weights += m
            flops += 2.0 * T * m
            if i % 4 == 0:
                state += 2 * 4 * S * (W // 128) * 64 * 128
                flops += 4.0 * T * (W // 128) * 64 * 128
            else:
                entry = r if i % 4 == 3 else 2 * 4 * dim
                state += 2 * entry * (B * c["context"] + T)
                flops += 4.0 * pairs * 16 * dim
        return {"bytes": 2.0 * weights + state + 4.0 * S * 32768, "flops": flops}
    T, W, s = sum(_lengths(c)), c["width"], _part_spec(c)
    weights = sum(math.prod(d.shape) for d in _part_class(c).parameters(s).values())
    moved = 2.0 * weights + 4.0 * T * W
    if c["kind"] == "experts":
        used = T * s.top * 3 * s.expert_intermediate * W + T * 3 * s.shared_intermediate * W + T * s.experts * W
        return {"bytes": moved, "flops": 2.0 * used}
    flops = 2.0 * T * sum(math.prod(d.shape) for d in _part_class(c).parameters(s).values() if d.role == "matrix")
    if c["kind"] in ("latent", "sink", "sigmoid"):
        pairs = sum(_causal_pairs(n, c["window"]) for n in _lengths(c))
        entry = s.kv_rank + s.rope_dim if c["kind"] == "latent" else 2 * s.num_kv_heads * s.head_dim
        qk = s.nope_dim + s.rope_dim if c["kind"] == "latent" else s.head_dim
        return {"bytes": moved + 2.0 * T * entry, "flops": flops + 2.0 * pairs * s.num_heads * (qk + s.v_dim)}
    entries = {"mamba2": lambda: s.num_heads * s.head_dim * s.state, "mamba1": lambda: s.inner * s.state,
               "gla": lambda: s.num_heads * s.head_dim * s.v_dim}[c["kind"]]()
    return {"bytes": moved + 8.0 * entries * len(_lengths(c)), "flops": flops + 4.0 * T * entries}


def tolerance(case):
    """Sums in 32 bits over 32-bit values: about 1e-5; a decoder or a layer whose activations are rounded to bfloat16: what the rounding
    of each intermediate gives, measured against 64 bits and about four times that between two correct forms at most."""
    if case.get("dtype") == "float32":
        return {"rel": 1.2e-5}
    return {"rel": 0.02 if case["kind"] in ("qwen3", "lovurax") else 0.012}


# ------------------------------------------------------------------------------------------------------------- in 64 bits
def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "qwen3":
            return _exact_qwen3(case, seed)
        if case["kind"] == "lovurax":
            return _exact_lovurax(case, seed)
        w = {k: v.to(F64) for k, v in _part_parameters(case, seed).items()}
        x, s, at, ys, states = _hidden(case, seed).to(F64), _part_spec(case), 0, [], []
        if case["kind"] == "experts":
            return {"y": _experts(x, w, s)}
        layer = {"latent": _latent, "sink": _sink, "sigmoid": _sigmoid, "mamba2": _mamba2, "mamba1": _mamba1, "gla": _gla}[case["kind"]]
        for n in _lengths(case):
            y, left = layer(x[at : at + n], w, s)
            ys.append(y)
            states.append(left)
            at += n
        return {"y": torch.cat(ys), "cache": torch.stack(states) if states[0] is not None else None}


def _unit(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _turned(x, dims, theta, interleaved=False):
    """x [T, ..., n] with its first ``dims`` numbers turned in pairs by position times frequency."""
    half = dims // 2
    freq = float(theta) ** (-2.0 * torch.arange(half, dtype=F64, device=x.device) / dims)
    a = (torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * freq).reshape([x.shape[0]] + [1] * (x.dim() - 2) + [half])
    u, v = (x[..., 0:dims:2], x[..., 1:dims:2]) if interleaved else (x[..., :half], x[..., half:dims])
    p, q = u * torch.cos(a) - v * torch.sin(a), v * torch.cos(a) + u * torch.sin(a)
    turned = torch.stack([p, q], -1).flatten(-2) if interleaved else torch.cat([p, q], -1)
    return torch.cat([turned, x[..., dims:]], -1)


def _visible(T, first, n, window, device):
    """Which of the first T keys the queries first .. first + n - 1 see."""
    i, j = torch.arange(first, first + n, device=device)[:, None], torch.arange(T, device=device)[None]
    return (j <= i) & (j > i - window) if window else j <= i


def _attend(q, k, v, scale, window, weigh):
    """q [n, H, d] of the last n positions over k, v [T, G, d]; ``weigh`` turns a head's scores (masked by -inf) into weights."""
    (n, H, _), (T, G, _) = q.shape, k.shape
    out = torch.empty((n, H, v.shape[-1]), dtype=F64, device=q.device)
    for lo in range(0, n, 1024):
        part = q[lo : lo + 1024]
        see = _visible(T, T - n + lo, part.shape[0], window, q.device)
        for h in range(H):
            g = h * G // H
            s = (part[:, h] @ k[:, g].T * scale).masked_fill(~see, -math.inf)
            out[lo : lo + 1024, h] = weigh(s, h, T - n + lo) @ v[:, g]
    return out


def _softmax(s, h, first):
    return torch.softmax(s, -1)


def _sink(x, w, s):
    T, H, G, d = x.shape[0], s.num_heads, s.num_kv_heads, s.head_dim
    q, k, v = (x @ w["qkv"].T).split([H * d, G * d, G * d], -1)
    q, k = (_unit(_turned(t.reshape(T, -1, d), d, 1000000.0, interleaved=True)) for t in (q, k))
    none = torch.zeros((T, 1), dtype=F64, device=x.device)
    weigh = lambda t, h, first: torch.softmax(torch.cat([t, none[: t.shape[0]]], -1), -1)[:, :-1]   # noqa: E731  a key of score 0 without a value
    return _attend(q, k, v.reshape(T, G, d), s.scale, s.window, weigh).reshape(T, -1) @ w["out"].T, None


def _sigmoid_weights(slopes, bias):
    def weigh(t, h, first):
        i, j = torch.arange(first, first + t.shape[0], device=t.device, dtype=F64)[:, None], torch.arange(t.shape[1], device=t.device, dtype=F64)[None]
        return torch.sigmoid(t - slopes[h] * (i - j) + bias[h])
    return weigh


def _sigmoid_parts(x, w, s):
    T, H, G, d = x.shape[0], s.num_heads, s.num_kv_heads, s.head_dim
    q, k, v, g = (x @ w["qkv"].T).split([H * d, G * d, G * d, H * d], -1)
    temp = 1.0 + s.temp_coef * torch.log(torch.div(torch.arange(1, T + 1, device=x.device), s.temp_every, rounding_mode="floor").to(F64) + 1.0)
    q = _unit(q.reshape(T, H, d)) * w["q_norm"] * temp[:, None, None]
    return q, _unit(k.reshape(T, G, d)) * w["k_norm"], v.reshape(T, G, d), g


def _sigmoid(x, w, s):
    q, k, v, g = _sigmoid_parts(x, w, s)
    o = _attend(q, k, v, s.scale, 0, _sigmoid_weights(s.slopes, w["head_bias"]))
    return (o.reshape(x.shape[0], -1) * torch.sigmoid(g)) @ w["out"].T, None


def _latent(x, w, s):
    T, H = x.shape[0], s.num_heads
    down = x @ w["dkv"].T
    c = _unit(down[:, : s.kv_rank]) * w["latent_norm"]
    q = (x @ w["q"].T).reshape(T, H, -1)
    k, v = (c @ w["uk"].T).reshape(T, H, -1), (c @ w["uv"].T).reshape(T, H, -1)
    if s.rope_dim:
        shared = _turned(down[:, s.kv_rank :], s.rope_dim, 1000000.0)[:, None].expand(T, H, s.rope_dim)
        q = torch.cat([q[..., : s.nope_dim], _turned(q[..., s.nope_dim :], s.rope_dim, 1000000.0)], -1)
        k = torch.cat([k, shared], -1)
    o = _attend(q, k, v, s.scale, s.window, _softmax)
    if s.head_gate:
        o = o * torch.sigmoid(x @ w["head_gate"].T)[..., None]
    return o.reshape(T, -1) @ w["out"].T, None


def _convolved(x, w, taps):
    padded = F.pad(x, (0, 0, taps - 1, 0))
    return F.silu(sum(padded[k : k + x.shape[0]] * w["conv"][:, k] for k in range(taps)) + w["conv_bias"])


def _mamba2(x, w, s):
    T, H, P, N, G = x.shape[0], s.num_heads, s.head_dim, s.state, s.groups
    z, raw, dt = (x @ w["in"].T).split([H * P, H * P + 2 * G * N, H], -1)
    xs, B, C = _convolved(raw, w, s.conv_taps).split([H * P, G * N, G * N], -1)
    xs, (B, C) = xs.reshape(T, H, P), (t.reshape(T, G, N).repeat_interleave(H // G, 1) for t in (B, C))
    dt = F.softplus(dt + w["dt_bias"])
    fade, S, ys = torch.exp(-torch.exp(w["A_log"]) * dt), torch.zeros((H, N, P), dtype=F64, device=x.device), []
    for t in range(T):
        S = fade[t][:, None, None] * S + (dt[t][:, None] * B[t])[:, :, None] * xs[t][:, None]
        ys.append(torch.einsum("hnp,hn->hp", S, C[t]))
    y = (torch.stack(ys) + w["D"][:, None] * xs).reshape(T, -1) * F.silu(z)
    y = _unit(y.reshape(T, s.norm_groups, -1)).reshape(T, -1) * w["norm"]
    return y @ w["out"].T, torch.cat([S.transpose(1, 2).flatten(), F.pad(raw, (0, 0, s.conv_taps - 1, 0))[-(s.conv_taps - 1):].flatten()])


def _mamba1(x, w, s):
    T = x.shape[0]
    raw, z = (x @ w["in"].T).split([s.inner, s.inner], -1)
    xs = _convolved(raw, w, s.conv_taps)
    dt, B, C = (xs @ w["x"].T).split([s.dt_rank, s.state, s.state], -1)
    dt, A = F.softplus(dt @ w["dt"].T + w["dt_bias"]), -torch.exp(w["A_log"])
    S, ys = torch.zeros((s.inner, s.state), dtype=F64, device=x.device), []
    for t in range(T):
        S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * xs[t])[:, None] * B[t]
        ys.append(S @ C[t])
    y = (torch.stack(ys) + w["D"] * xs) * F.silu(z)
    return y @ w["out"].T, torch.cat([S.flatten(), F.pad(raw, (0, 0, s.conv_taps - 1, 0))[-(s.conv_taps - 1):].flatten()])


def _gla(x, w, s):
    T, H, d, dv = x.shape[0], s.num_heads, s.head_dim, s.v_dim
    q, k, v, g, a1 = (x @ w["in"].T).split([H * d, H * d, H * dv, H * dv, s.decay_rank], -1)
    q, k, v = q.reshape(T, H, d) * d ** -0.5, k.reshape(T, H, d), v.reshape(T, H, dv)
    fade = torch.sigmoid(a1 @ w["decay"].T + w["decay_bias"]).pow(1.0 / s.tau).reshape(T, H, d)
    S, ys = torch.zeros((H, d, dv), dtype=F64, device=x.device), []
    for t in range(T):
        S = fade[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None]
        ys.append(torch.einsum("hdv,hd->hv", S, q[t]))
    y = (_unit(torch.stack(ys)) * w["norm"]).reshape(T, -1) * F.silu(g)
    return y @ w["out"].T, S.flatten()


def _experts(x, w, s):
    E, H = s.experts, s.hidden
    score = torch.sigmoid(x @ w["router"].T)
    chosen = torch.topk(score, s.top, -1).indices
    gate, up, down = w["gate"].reshape(E, -1, H), w["up"].reshape(E, -1, H), w["down"].reshape(E, H, -1)
    g, u = w["shared_gate_up"].chunk(2)
    y = (F.silu(x @ g.T) * (x @ u.T)) @ w["shared_down"].T
    for e in range(E):
        t = (chosen == e).any(-1).nonzero()[:, 0]
        rows = x[t] * score[t, e : e + 1]
        y.index_add_(0, t, (F.silu(rows @ gate[e].T) * (rows @ up[e].T)) @ down[e].T)
    return y


def _wide(params, scope):
    return {k: v.to(F64) for k, v in params.get(scope, {}).items()}


def _sequences(c, seed):
    held, new = _tokens(c, seed)
    return held + ([new] if new else [])


def _exact_qwen3(c, seed):
    cfg, params, d, G = _qwen3_config(c), _model_parameters(c, seed), 128, 8
    H, rows, rotate = cfg["num_attention_heads"], _sequences(c, seed), lambda t: _turned(t, d, cfg["rope_theta"])
    table = params["embed"]["table"]
    hs = [table[torch.tensor(ids, device="cuda")].to(F64) for ids in rows]
    for i in range(c["layers"]):
        m, f = _wide(params, f"blocks.{i}.mixer"), _wide(params, f"blocks.{i}.feed_forward")
        n1, n2 = (_wide(params, f"blocks.{i}.{k}")["weight"] for k in ("input_norm", "post_mixer_norm"))
        last = i == c["layers"] - 1
        for r, h in enumerate(hs):
            q, k, v = (_unit(h) * n1 @ m["qkv"].T).reshape(h.shape[0], H + 2 * G, d).split([H, G, G], 1)
            q, k = rotate(_unit(q) * m["q_norm"]), rotate(_unit(k) * m["k_norm"])
            if last:       # only the last token's logits are wanted
                q, h = q[-1:], h[-1:]
            h = h + _attend(q, k, v, d ** -0.5, 0, _softmax).reshape(q.shape[0], -1) @ m["out"].T
            g, u = (_unit(h) * n2 @ f["gate_up"].T).chunk(2, -1)
            hs[r] = h + (F.silu(g) * u) @ f["down"].T
    head = table if cfg["tie_word_embeddings"] else params["lm_head"]["weight"]
    return _unit(torch.cat(hs)) * params["final_norm"]["weight"].to(F64) @ head.to(F64).T


def _exact_lovurax(c, seed):
    spec, params = _model_spec(c), _model_parameters(c, seed)
    table, out = params["embed"]["table"].to(F64), []
    for ids in _sequences(c, seed):
        h = table[torch.tensor(ids, device="cuda")]
        for i, b in enumerate(spec.blocks):
            w = {k: _wide(params, f"blocks.{i}.{k}") for k in ("input_norm", "mixer", "mixer_connection", "post_mixer_norm", "feed_forward", "feed_forward_connection")}
            n = _unit(h) * w["input_norm"]["weight"]
            y = {"retention": _retention, "sigmoid_attention": _sigmoid, "latent_attention": _latent}[b.mixer.kind](n, w["mixer"], b.mixer)[0]
            h = h + y * torch.sigmoid(n @ w["mixer_connection"]["gate"].T + w["mixer_connection"]["gate_bias"])
            n = _unit(h) * w["post_mixer_norm"]["weight"]
            z, act = n @ w["feed_forward"]["up"].T, w["feed_forward"]["act"]
            low = torch.clamp(z, max=0.0)
            z = torch.where(z > 0, F.softplus(act[0]) * z * z, (0.5 + F.softplus(act[1])) * (torch.expm1(low) - low)) + 0.5 * z
            h = h + (z @ w["feed_forward"]["down"].T) * torch.sigmoid(n @ w["feed_forward_connection"]["gate"].T + w["feed_forward_connection"]["gate_bias"])
        out.append(_unit(h[-1:]) * params["final_norm"]["weight"].to(F64) @ table.T)
    return torch.cat(out)


def _retention(x, w, s):
    """Every pair of tokens at once: o_t = sum_u decay^(t - u) (q_t . k_u) v_u."""
    T, H, d, dv = x.shape[0], s.num_heads, s.head_dim, s.v_dim
    q, k, v, g = (x @ w["in"].T).split([H * d, H * d, H * dv, H * dv], -1)
    q, k = (_turned(t.reshape(T, H, d), 64, 10000.0) for t in (q, k))
    i = torch.arange(T, device=x.device, dtype=F64)
    out = torch.empty((T, H, dv), dtype=F64, device=x.device)
    for h in range(H):
        fade = torch.exp(math.log(s.decay[h]) * (i[:, None] - i[None])).tril()
        out[:, h] = (q[:, h] @ k[:, h].T * d ** -0.5 * fade) @ v.reshape(T, H, dv)[:, h]
    return (_unit(out).reshape(T, -1) * F.silu(g)) @ w["out"].T, None

"""The work that this framework is measured on: its layers, one by one, and its decode steps.

A *layer* case runs one part (a mixer over the paged cache or a state, a feed-forward) the way a block of a
model does: the part is built from its ``PartSpec``, bound to weights and run with a ``StepContext`` on normed
rows; what it returns joins the float residual stream in the norm that follows.  A *step* case is a whole call
of the step function (``ModelRunner.step``) of a model whose layers are the named preset's first ones.

Sizes are those of the presets (``kvforge_b200.PRESETS``), a step's token budget (2,048) and the contexts and
batches that ``bench.py`` and the tests use, with ragged ones among them.
"""

from __future__ import annotations

import math

import numpy as np
import torch
from dataclasses import replace

from kvforge_b200 import PRESETS
from kvforge_b200.config.engine_config import CacheConfig
from kvforge_b200.engine.core import EngineCore, spec_from_config
from kvforge_b200.engine.runtime import QueryTiles, Runtime, StepContext
from kvforge_b200.engine.step import BatchItem
from kvforge_b200.parts.base import LayerCache, PartSpec, build_part
from kvforge_b200.parts.model import DecoderModel
from kvforge_b200.weights.random_init import random_weights

PAGE = 16  # tokens a page, the default of the engine's configuration
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
FEED_FORWARDS = ("gated_mlp", "routed_experts")
NORM_EPS = 1e-5
INIT_STD = 0.03  # matrices of layer cases: scores of order one, as in a trained layer


def listed() -> list[dict]:
    layer = dict(call="layer", dtype="bfloat16", requests=1, past=0)
    return [
        # a decode step of a small chat model for a handful of users: every generated token pays for it
        dict(name="step-decode-8", call="step", model="llama-3.2-1b", layers=16, requests=8, past=4095),
        # a decode step of a busy server, the mixers alone: attention with a bias under a window, latent attention
        dict(name="step-decode-64-mixers", call="step", model="setenex-1b", layers=4, requests=64, past=2300),
        # the last portion of a long prompt: grouped-query attention over what the portions before it left
        dict(layer, name="attention-portion", model="llama-3.2-1b", part="paged_attention", tokens=2047, past=6145),
        # the feed-forward of a whole prompt, the largest share of the flops of a dense model
        dict(layer, name="feed-forward-prompt", model="llama-3.2-1b", part="gated_mlp", tokens=2048),
        # two prompts of unequal length behind a little context: attention with a bias by distance and kept first tokens
        dict(layer, name="biased-attention-prompt", model="setenex-1b", part="paged_attention", tokens=2048, requests=2, past=300),
        # a whole prompt through attention over one latent a token
        dict(layer, name="latent-attention-prompt", model="sonalix-1b", part="latent_attention", tokens=2048),
        # a whole prompt through attention whose heads talk
        dict(layer, name="talking-attention-prompt", model="gukirax-1b", part="talking_attention", tokens=2048),
        # a whole prompt through the delta rule, state from zero
        dict(layer, name="delta-rule-prompt", model="mopilorn-1b", part="gated_delta_rule", tokens=2048),
        # a whole prompt through the state space, state from zero
        dict(layer, name="state-space-prompt", model="ritizen-1b", part="state_space", tokens=2048),
        # a full step's tokens through routed experts
        dict(layer, name="experts-prompt", model="setenex-1b", part="routed_experts", tokens=2048),
        # the one token of a single user through gated experts: the smallest call
        dict(layer, name="experts-decode-1", model="sonalix-1b", part="routed_experts", tokens=1),
        # a ragged portion in true 32-bit, what exact replay and debugging run
        dict(layer, name="feed-forward-float32", model="llama-3.2-1b", part="gated_mlp", tokens=515, dtype="float32"),
    ]


# parts and the presets that have them
_DRAWN = [
    ("paged_attention", ("llama-3.2-1b", "llama-3.2-3b", "llama-3.1-8b", "setenex-1b", "sonalix-1b")),
    ("gated_mlp", ("llama-3.2-1b", "llama-3.2-3b", "llama-3.1-8b")),
    ("latent_attention", ("setenex-1b", "sonalix-1b")),
    ("talking_attention", ("gukirax-1b", "gukirax-3b")),
    ("gated_delta_rule", ("mopilorn-1b", "mopilorn-3b")),
    ("state_space", ("ritizen-1b", "ritizen-3b")),
    ("routed_experts", ("setenex-1b", "sonalix-1b", "gukirax-1b")),
]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    if rng.random() < 0.2:
        model, layers = rng.choice([("llama-3.2-1b", 8), ("setenex-1b", 4)])
        return dict(call="step", model=model, layers=layers, requests=_log_uniform(rng, 1, 64), past=_log_uniform(rng, 100, 4095))
    part, models = rng.choice(_DRAWN)
    case = dict(call="layer", model=rng.choice(models), part=part, dtype="bfloat16")
    case["requests"] = rng.choice([1, 1, 1, 2, 3, 5, 8])
    case["tokens"] = _log_uniform(rng, max(130, 20 * case["requests"]), 2048)
    case["past"] = 0
    if part in ("paged_attention", "latent_attention", "talking_attention") and rng.random() < 0.5:
        case["past"] = _log_uniform(rng, 16, 4095 if part == "paged_attention" else 1500)
    if part in ("gated_mlp", "paged_attention") and rng.random() < 0.25:
        case.update(dtype="float32", tokens=min(case["tokens"], 400), past=min(case["past"], 500))
        case["requests"] = min(case["requests"], 5)
        if case["model"] == "llama-3.1-8b":
            case["model"] = "llama-3.2-1b"
    if part == "gated_delta_rule" and case["model"] == "mopilorn-3b":
        case["tokens"] = min(case["tokens"], 1500)
    if part == "talking_attention" and case["model"] == "gukirax-3b":
        case["tokens"] = min(case["tokens"], 1100)
    if part == "routed_experts":
        case["requests"] = 1
        if rng.random() < 0.5:
            case["tokens"] = case["requests"] = _log_uniform(rng, 1, 64)
    return case


# ------------------------------------------------------------------ inputs


def _generator(seed: int, salt: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed * 1000003 + salt)


def _part_spec(case: dict) -> PartSpec:
    """The first mixer or feed-forward of that kind in the preset's layers."""
    for layer in spec_from_config(PRESETS[case["model"]]).layers:
        for key in ("mixer", "ffn"):
            spec = layer.block.params.get(key)
            if spec is not None and spec.kind == case["part"]:
                return spec
    raise ValueError(f"{case['model']} has no {case['part']}")


def _fill(decl, g: torch.Generator, dtype: torch.dtype) -> torch.Tensor:
    z = torch.randn(decl.shape, generator=g, dtype=torch.float32, device="cuda")
    if decl.init == "ones":
        z = 1.0 + 0.1 * z
    elif decl.init in ("conv", "small"):
        z = 0.5 * z
    elif decl.init == "eye":
        z = torch.eye(*decl.shape, device="cuda") + 0.1 * z
    elif decl.init == "unit":
        z = torch.rand(decl.shape, generator=g, dtype=torch.float32, device="cuda")
    elif decl.init == "wide":
        z = z * decl.shape[-1] ** -0.5
    else:
        z = INIT_STD * z
    return z.to(dtype) if decl.kind == "matrix" else z


def _declared(part) -> dict:
    out = dict(type(part).weight_decls(part.params))
    for sub in part.sub_parts():  # a shared expert: its tensors under its own prefix
        out.update({"shared." + k: v for k, v in _declared(sub).items()})
    return out


def _weights(part, case: dict, seed: int) -> dict:
    g = _generator(seed, 1)
    return {name: _fill(decl, g, DTYPES[case["dtype"]]) for name, decl in sorted(_declared(part).items())}


def _bind(part, weights: dict, rt) -> None:
    for sub in part.sub_parts():
        _bind(sub, {k[len("shared.") :]: v for k, v in weights.items() if k.startswith("shared.")}, rt)
    part.bind({k: v for k, v in weights.items() if not k.startswith("shared.")}, rt)


def _lengths(case: dict) -> tuple[list[int], list[int]]:
    """(new tokens, tokens in the cache before them) of every request: unequal where there are several."""
    r, n = case["requests"], case["tokens"]
    shares = [2 * i + 1 for i in range(r)]
    new = [max(1, n * s // sum(shares)) for s in shares]
    new[-1] += n - sum(new)
    return new, [case["past"] * (r - i) // r for i in range(r)]


def _rows(case: dict, seed: int, width: int) -> tuple[torch.Tensor, torch.Tensor]:
    """Normed rows as a norm leaves them and the float residual stream beside them."""
    g = _generator(seed, 2)
    x = torch.randn((case["tokens"], width), generator=g, device="cuda").to(DTYPES[case["dtype"]])
    return x, 0.5 * torch.randn((case["tokens"], width), generator=g, device="cuda")


def _pages(case: dict, seed: int, need) -> dict:
    """Pages of keys and values in shuffled order, holding what earlier steps left, and every request's table."""
    new, past = _lengths(case)
    g = _generator(seed, 3)
    per = [-(-(n + p) // PAGE) for n, p in zip(new, past)]
    order = torch.randperm(sum(per) + 8, generator=g, device="cuda").tolist()
    tables, at = [], 0
    for m in per:
        tables.append(order[at : at + m])
        at += m
    shape, dtype = (sum(per) + 8, need.kv_heads, PAGE), DTYPES[case["dtype"]]
    k = torch.randn((*shape, need.head_dim), generator=g, device="cuda").to(dtype)
    v = k if need.v_in_k else torch.randn((*shape, need.value_dim), generator=g, device="cuda").to(dtype)
    return {"k": k, "v": v, "tables": tables}


def _step_context(case: dict, rt, tables: list[list[int]]) -> StepContext:
    new, past = _lengths(case)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    starts = np.concatenate([[0], np.cumsum(new)])
    ends = [p + n for p, n in zip(past, new)]
    positions = [p + i for p, n in zip(past, new) for i in range(n)]
    slots = [t[(p + i) // PAGE] * PAGE + (p + i) % PAGE for t, p, n in zip(tables, past, new) for i in range(n)] if tables else [-1] * case["tokens"]
    width = max([len(t) for t in tables] or [1])
    tiles = {}
    for tq in rt.query_tile_sizes if max(new) > 1 else ():
        every = sorted(((b, q) for b, n in enumerate(new) for q in range(0, n, tq)), key=lambda t: -(past[t[0]] + min(new[t[0]], t[1] + tq)))
        multi = [t for t in every if new[t[0]] > 1]
        tiles[tq] = QueryTiles(i32(every).reshape(-1), len(every), i32(multi).reshape(-1), len(multi), sum(n == 1 for n in new))
    return StepContext(
        rt=rt, num_tokens=case["tokens"], num_seqs=case["requests"], token_ids=i32([0] * case["tokens"]), positions=i32(positions),
        query_start_loc=i32(starts.tolist()), context_lens=i32(ends), state_slots=i32(list(range(case["requests"]))), logit_rows=i32([0]),
        num_logit_rows=0, block_tables=[i32([t + [0] * (width - len(t)) for t in tables])] if tables else [i32([[0]])], slot_mappings=[i32(slots)],
        max_query_len=max(new), max_context_len=max(ends), block_size=PAGE, h_query_start_loc=starts, h_context_lens=np.array(ends),
        h_state_slots=np.arange(case["requests"]), query_tiles=tiles,
    )  # fmt: skip


def _step_spec(case: dict):
    """The preset's first layers, without their feed-forwards where these are experts (their choice turns with a rounding)."""
    spec = spec_from_config(PRESETS[case["model"]])
    layers = spec.layers[: case["layers"]]
    layers = [replace(s, block=PartSpec(s.block.kind, {**s.block.params, "ffn": None})) if s.block.params["ffn"].kind == "routed_experts" else s for s in layers]
    return replace(spec, layers=layers, execution=[], pass_offsets=0)


def _step_past(case: dict) -> list[int]:
    """Tokens in every request's cache: spread from half the largest to the largest."""
    r = case["requests"]
    return [case["past"] - (case["past"] // 2) * i // max(1, r - 1) for i in range(r)]


def _prepare_step(case: dict, seed: int) -> dict:
    past = _step_past(case)
    blocks = sum(-(-(p + 1) // PAGE) for p in past) + 8
    core = EngineCore(
        _step_spec(case), dtype="bfloat16", seed=seed, cache=CacheConfig(block_size=PAGE, num_blocks=blocks, watermark=0.0),
        max_num_seqs=case["requests"], max_num_batched_tokens=256, max_model_len=max(past) + 16, cuda_graphs=True,
    )  # fmt: skip
    g = _generator(seed, 4)
    for t in {id(t): t for t in core.pool.k + core.pool.v}.values():
        t.copy_(0.7 * torch.randn(t.shape, generator=g, device="cuda"))
    tokens = torch.randint(0, core.spec.vocab_size, (case["requests"],), generator=g, device="cuda").tolist()
    items = []
    for i, p in enumerate(past):
        core.block_manager.allocate(f"r{i}", p + 1)
        core.state_slots.allocate(f"r{i}")
        items.append(BatchItem(f"r{i}", [tokens[i]], p, "last"))
    return {"core": core, "items": items, "tokens": tokens}


def prepare(case: dict, seed: int):
    if case["call"] == "step":
        return _prepare_step(case, seed)
    spec = _part_spec(case)
    mixer = case["part"] not in FEED_FORWARDS
    part = build_part("mixer" if mixer else "ffn", spec, "")
    new, past = _lengths(case)
    rt = Runtime("cuda", DTYPES[case["dtype"]], case["tokens"], case["requests"], max(n + p for n, p in zip(new, past)))
    _bind(part, _weights(part, case, seed), rt)
    width = int(spec.params["hidden_size"])
    norm = build_part("norm", PartSpec("rmsnorm", {"dim": width, "eps": NORM_EPS}), "")
    norm.bind({"weight": torch.ones(width, device="cuda")}, rt)
    x, stream = _rows(case, seed, width)
    cache, tables = None, []
    if mixer and part.cache_need().kind != "none":
        pages = _pages(case, seed, part.cache_need())
        cache, tables = LayerCache(pages["k"], pages["v"], 0), pages["tables"]
    elif mixer:
        cache = LayerCache(None, None, -1, True, torch.zeros((case["requests"], *part.state_shape()), device="cuda"))
    ctx = _step_context(case, rt, tables)
    ctx.residual = torch.empty_like(stream)
    return {"part": part, "norm": norm, "ctx": ctx, "x": x, "stream": stream, "cache": cache, "conv": getattr(part, "conv_floats", 0)}


# ------------------------------------------------------------------ one pass


def run(state):
    if "core" in state:
        core = state["core"]
        return {"logits": core.runner.step(state["items"]), "keys": core.pool.k, "values": core.pool.v}
    ctx, part, cache = state["ctx"], state["part"], state["cache"]
    ctx.residual.copy_(state["stream"])
    if cache is None:
        y = part.forward(ctx, state["x"])
    else:
        if cache.state is not None:
            cache.state.zero_()  # a new request's slot, as the engine hands it out
        y = part.forward(ctx, state["x"], cache)
    rows = state["norm"].forward(ctx, ctx.residual, y)
    out = {"rows": rows, "stream": ctx.residual}
    if cache is not None and cache.state is not None:
        out["inputs"], out["matrix"] = cache.state[:, : state["conv"]], cache.state[:, state["conv"] :]
    elif cache is not None:
        out["keys"] = cache.k
        if cache.v is not cache.k:
            out["values"] = cache.v
    return out


# ------------------------------------------------------------------ what a pass cannot do without


def _visible(case: dict, window: int | None) -> tuple[int, int]:
    """(query-key pairs, tokens whose keys are read) of a causal pass under a window."""
    new, past = _lengths(case)
    pairs = reads = 0
    for n, p in zip(new, past):
        seen = np.arange(p + 1, p + n + 1)
        pairs += int((np.minimum(seen, window) if window else seen).sum())
        reads += min(n + p, n + window) if window else n + p
    return pairs, reads


def work(case: dict) -> dict:
    if case["call"] == "step":
        return _work_step(case)
    p = dict(_part_spec(case).params)
    size = 4 if case["dtype"] == "float32" else 2
    n, w = case["tokens"], int(p["hidden_size"])
    part = build_part("ffn" if case["part"] in FEED_FORWARDS else "mixer", PartSpec(case["part"], p), "")
    decls = _declared(part)
    matrices = sum(math.prod(d.shape) for d in decls.values() if d.kind == "matrix")
    flops, bytes_ = 2 * n * matrices, size * matrices
    if case["part"] == "routed_experts":
        one = sum(math.prod(d.shape) for name, d in decls.items() if name.startswith("e0."))
        shared = sum(math.prod(d.shape) for name, d in decls.items() if name.startswith("shared.") and d.kind == "matrix")
        e, top = int(p["experts"]), int(p["top"])
        flops = 2 * n * (top * one + shared + e * w)
        bytes_ = size * (min(e, n * top) * one + shared) + 4 * e * w
    bytes_ += n * w * (2 * size + 8)  # rows in and out, the stream in and out
    if case["part"] in ("paged_attention", "talking_attention", "latent_attention"):
        pairs, reads = _visible(case, p.get("window"))
        h, d = int(p["num_heads"]), int(p["head_dim"])
        if case["part"] == "latent_attention":
            # scores and values over every head's own keys and values, made once a token from the latent
            flops += 2 * pairs * h * (d + int(p["rot_dim"]) + int(p["v_head_dim"]))
            bytes_ += size * (reads + n) * (int(p["kv_rank"]) + int(p["rot_dim"]))
        else:
            dv = int(p.get("v_head_dim") or d)
            flops += 2 * pairs * h * (d + dv) + (2 * pairs * h * h if case["part"] == "talking_attention" else 0)
            bytes_ += size * (reads + n) * int(p["num_kv_heads"]) * (d + dv)
    elif case["part"] == "gated_delta_rule":
        h, d, dv = int(p["num_heads"]), int(p["head_dim"]), int(p["v_head_dim"])
        flops += 7 * n * h * d * dv
        bytes_ += 8 * case["requests"] * h * d * dv
    elif case["part"] == "state_space":
        h, d, dv = int(p["num_heads"]), int(p["state_dim"]), int(p["v_head_dim"])
        flops += 5 * n * h * d * dv
        bytes_ += 8 * case["requests"] * h * d * dv
    return {"bytes": bytes_, "flops": flops}


def _work_step(case: dict) -> dict:
    spec, past = _step_spec(case), _step_past(case)
    r = case["requests"]
    model = DecoderModel(spec)
    matrices = sum(math.prod(d.shape) for name, d in model.expected_weights().items() if d.kind == "matrix" and name != spec.embedding_name)
    bytes_, flops = 2 * matrices + 4 * r * spec.vocab_size, 2 * r * matrices
    for layer in spec.layers:
        p = layer.block.params["mixer"].params
        seen = sum(min(x + 1, int(p["window"])) if p.get("window") else x + 1 for x in past)
        if "kv_rank" in p:
            bytes_ += 2 * seen * (int(p["kv_rank"]) + int(p["rot_dim"]))
            flops += 2 * seen * int(p["num_heads"]) * (2 * int(p["kv_rank"]) + int(p["rot_dim"]))
        else:
            bytes_ += 4 * seen * int(p["num_kv_heads"]) * int(p["head_dim"])
            flops += 4 * seen * int(p["num_heads"]) * int(p["head_dim"])
    return {"bytes": bytes_, "flops": flops}


def tolerance(case: dict):
    """About four times what the paths show against ``exact``: bfloat16 rounds the projections, the cached rows, the
    inner activations and the normed rows (2.3e-3 of the result for a layer, 4.1e-3 where a convolution and a gated
    read-out come on top, 1.5e-2 for the logits of sixteen layers, 1.7e-3 for those of four mixers over a wide
    stream); 32-bit shows the order of its sums (2.2e-6)."""
    if case["call"] == "step":
        return {"rel": 6e-2 if case["model"] == "llama-3.2-1b" else 8e-3}
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 1.6e-2 if case["part"] in ("gated_delta_rule", "state_space") else 1e-2}


# ------------------------------------------------------------------ the same numbers in 64 bits


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _frequencies(position) -> tuple[torch.Tensor | None, bool]:
    """Angular frequencies of a rotary encoding and whether its pairs are neighbours."""
    if position is None:
        return None, False
    q = position.params
    dims = int(q.get("rotary_dim") or q["head_dim"])
    f = float(q["theta"]) ** (-torch.arange(0, dims, 2, dtype=torch.float64, device="cuda") / dims)
    s = q.get("scaling")
    if s:  # long wavelengths are slowed by the factor, short ones stay, those between are blended
        turns = float(s["original_max_position_embeddings"]) * f / (2 * math.pi)
        mix = ((turns - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])).clamp(0, 1)
        f = (1 - mix) * f / s["factor"] + mix * f
    return f, bool(q.get("interleaved", False))


def _turn(x, positions, f, neighbours):
    """``x [T, heads, d]`` with the pairs of its first dims turned."""
    if f is None:
        return x
    ang = positions[:, None, None] * f
    c, s, m = ang.cos(), ang.sin(), f.numel()
    y = x.clone()
    if neighbours:
        a, b = x[..., 0 : 2 * m : 2], x[..., 1 : 2 * m : 2]
        y[..., 0 : 2 * m : 2], y[..., 1 : 2 * m : 2] = a * c - b * s, b * c + a * s
    else:
        a, b = x[..., :m], x[..., m : 2 * m]
        y[..., :m], y[..., m : 2 * m] = a * c - b * s, b * c + a * s
    return y


def _bias_by_distance(rel, far: int, dist):
    rows = rel.shape[0]
    half = rows // 2
    n = torch.arange(far + 1, dtype=torch.float64, device=rel.device).clamp(min=1)
    steps = half + torch.floor(torch.log(n / half) / math.log(far / half) * (rows - half)).long()
    bucket = torch.where(torch.arange(far + 1, device=rel.device) < half, torch.arange(far + 1, device=rel.device), steps.clamp(max=rows - 1))
    return rel[bucket[dist.clamp(0, far)]]


def _attend(p, w, q, k, v, start: int):
    """``q [T, H, d]`` at positions ``start ..`` over keys ``[J, G, d]`` from position 0 on."""
    t, h, _ = q.shape
    scale = float(p.get("scale") or 1.0 / math.sqrt(int(p["head_dim"])))
    out = q.new_empty(t, h, v.shape[-1])
    j = torch.arange(k.shape[0], device="cuda")[None, :]
    for lo in range(0, t, 512):
        i = torch.arange(start + lo, start + min(t, lo + 512), device="cuda")[:, None]
        seen = j <= i
        if p.get("window"):
            seen = seen & ((i - j < int(p["window"])) | (j < int(p.get("keep_first") or 0)))
        for head in range(h):
            s = q[lo : lo + 512, head] @ k[:, head // (h // k.shape[1])].T * scale
            if p.get("distance_bias"):
                s = s + _bias_by_distance(w["rel"][:, head].double(), int(p["distance_bias"]["far"]), i - j)
            if p.get("softcap"):
                s = p["softcap"] * torch.tanh(s / p["softcap"])
            s = s.masked_fill(~seen, -math.inf)
            if p.get("sink"):
                s = torch.cat([s, w["sink"][head].double().expand(s.shape[0], 1)], dim=1)
            out[lo : lo + 512, head] = torch.softmax(s, dim=-1)[:, : k.shape[0]] @ v[:, head // (h // k.shape[1])]
    return out.reshape(t, -1)


def _cached(pool, table, count):
    """Rows ``[count, heads, d]`` of a request's first positions."""
    return pool[torch.tensor(table, device="cuda")].transpose(1, 2).reshape(-1, pool.shape[1], pool.shape[3])[:count].double()


def _exact_attention(p, w, x, start, past_k, past_v):
    h, g, d = int(p["num_heads"]), int(p["num_kv_heads"]), int(p["head_dim"])
    q, k, v = (x @ w[n + "_proj.weight"].double().T for n in "qkv")
    q, k, v = q.view(-1, h, d), k.view(-1, g, d), v.view(-1, g, int(p.get("v_head_dim") or d))
    if p.get("qk_norm"):
        q = _rms(q, p["qk_norm"]["eps"]) * w["q_norm.weight"].double()
        k = _rms(k, p["qk_norm"]["eps"]) * w["k_norm.weight"].double()
    f, neighbours = _frequencies(p.get("position"))
    pos = torch.arange(start, start + x.shape[0], dtype=torch.float64, device="cuda")
    q, k = _turn(q, pos, f, neighbours), _turn(k, pos, f, neighbours)
    o = _attend(p, w, q, torch.cat([past_k, k]), torch.cat([past_v, v]), start)
    return o @ w["o_proj.weight"].double().T


def _exact_latent(p, w, x, start, past, _):
    h, d, dr, dv, r = (int(p[k]) for k in ("num_heads", "head_dim", "rot_dim", "v_head_dim", "kv_rank"))
    t = x.shape[0]
    if p.get("q_rank"):
        q = (_rms(x @ w["dq"].double().T, p["eps"]) * w["dq.norm"].double()) @ w["uq"].double().T
    else:
        q = x @ w["q"].double().T
    q = q.view(t, h, d + dr)
    down = x @ w["dkv"].double().T
    f, neighbours = _frequencies(p.get("position"))
    pos = torch.arange(start, start + t, dtype=torch.float64, device="cuda")
    c = torch.cat([past[:, 0, :r], _rms(down[:, :r], p["eps"]) * w["dkv.norm"].double()])
    turned = torch.cat([past[:, 0, r:], _turn(down[:, None, r:], pos, f, neighbours)[:, 0]])
    q = torch.cat([q[..., :d], _turn(q[..., d:], pos, f, neighbours)], dim=-1)
    k = torch.cat([(c @ w["uk"].double().T).view(-1, h, d), turned[:, None].expand(-1, h, dr)], dim=-1)
    o = _attend(p, w, q, k, (c @ w["uv"].double().T).view(-1, h, dv), start)
    if p.get("gate"):
        gate = torch.sigmoid(x @ w["g"].double().T)
        o = o * gate if gate.shape[1] == h * dv else (o.view(t, h, dv) * gate[:, :, None]).view(t, -1)
    return o @ w["o"].double().T


def _exact_talking(p, w, x, start, past_k, past_v):
    h, g, d = int(p["num_heads"]), int(p["num_kv_heads"]), int(p["head_dim"])
    dv, t = int(p.get("v_head_dim") or d), x.shape[0]
    q, k = (x @ w["q_proj.weight"].double().T).view(t, h, d), (x @ w["k_proj.weight"].double().T).view(t, g, d)
    v = k[..., :dv]
    f, neighbours = _frequencies(p.get("position"))
    pos = torch.arange(start, start + t, dtype=torch.float64, device="cuda")
    q, k = (_rms(_turn(y, pos, f, neighbours), p["qk_norm"]["eps"]) for y in (q, k))
    k, v = torch.cat([past_k, k]), torch.cat([past_v, v])
    out = x.new_empty(t, h, dv)
    j = torch.arange(k.shape[0], device="cuda")[None, :]
    for lo in range(0, t, 256):
        i = torch.arange(start + lo, start + min(t, lo + 256), device="cuda")[:, None]
        s = torch.stack([q[lo : lo + 256, a] @ k[:, a // (h // g)].T for a in range(h)]) * float(p["scale"])
        s = torch.einsum("ab,bij->aij", w["talk"].double(), s).masked_fill(j > i, -math.inf)
        s = torch.cat([s, w["sink"].double()[:, None, None].expand(h, s.shape[1], 1)], dim=2)
        s = torch.softmax(s, dim=-1)[..., : k.shape[0]]
        for a in range(h):
            out[lo : lo + 256, a] = s[a] @ v[:, a // (h // g)]
    return out.reshape(t, -1) @ w["o_proj.weight"].double().T


def _conv(x, taps, bias=None):
    """``taps [C, n]``, the last column for the token itself; zeros before the start."""
    n = taps.shape[1]
    y = sum(torch.nn.functional.pad(x, (0, 0, b, 0))[: x.shape[0]] * taps[:, n - 1 - b] for b in range(n))
    return y if bias is None else y + bias


def _exact_delta(p, w, x):
    h, g, d, dv = (int(p[k]) for k in ("num_heads", "num_kv_heads", "head_dim", "v_head_dim"))
    t = x.shape[0]
    w = {k: v.double() for k, v in w.items()}
    silu = torch.nn.functional.silu
    q, k, v = (silu(_conv(x @ w[n].T, w[n + ".conv"])) for n in "qkv")
    unit = lambda y: y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q = (unit(q.view(t, g, d)) * d**-0.5).repeat_interleave(h // g, dim=1)
    k = unit(k.view(t, g, d)).repeat_interleave(h // g, dim=1)
    v, beta = v.view(t, h, dv), torch.sigmoid(x @ w["b"].T)
    a = ((x @ w["a1"].T) @ w["a2"].T if "a1" in w else x @ w["a"].T) + w["dt_bias"]
    decay = torch.exp(-torch.exp(w["A_log"])[None, :, None] * torch.nn.functional.softplus(a.view(t, h, -1)))
    s, read = x.new_zeros(h, d, dv), x.new_empty(t, h, dv)
    for n in range(t):
        s = s * decay[n][:, :, None]
        u = beta[n][:, None] * (v[n] - torch.bmm(k[n][:, None], s)[:, 0])
        s = torch.baddbmm(s, k[n][:, :, None], u[:, None])
        read[n] = torch.bmm(q[n][:, None], s)[:, 0]
    gate = (x @ w["g1"].T) @ w["g2"].T if "g1" in w else x @ w["g"].T
    gate = (silu(gate) if p.get("gate", "silu") == "silu" else torch.sigmoid(gate)).view(t, h, dv)
    return (_rms(read, float(p["eps"])) * w["norm"] * gate).reshape(t, -1) @ w["o"].T, s


def _exact_state_space(p, w, x):
    h, dv, n_state, g = (int(p[k]) for k in ("num_heads", "v_head_dim", "state_dim", "groups"))
    t, inner = x.shape[0], h * dv
    w = {k: v.double() for k, v in w.items()}
    y = x @ w["in"].T
    z, xbc, dt = y[:, :inner], y[:, inner : 2 * inner + 2 * g * n_state], y[:, 2 * inner + 2 * g * n_state :]
    xbc = torch.nn.functional.silu(_conv(xbc, w["conv"], w["conv.b"]))
    xs = xbc[:, :inner].view(t, h, dv)
    b, c = (xbc[:, lo : lo + g * n_state].view(t, g, n_state).repeat_interleave(h // g, dim=1) for lo in (inner, inner + g * n_state))
    dt = torch.nn.functional.softplus(dt + w["dt_bias"])
    decay = torch.exp(-torch.exp(w["A_log"]) * dt)
    s, read = x.new_zeros(h, n_state, dv), x.new_empty(t, h, dv)
    for n in range(t):
        s = torch.baddbmm(s * decay[n][:, None, None], b[n][:, :, None], (dt[n][:, None] * xs[n])[:, None])
        read[n] = torch.bmm(c[n][:, None], s)[:, 0]
    read = (read + w["D"][:, None] * xs).reshape(t, inner) * torch.nn.functional.silu(z)
    parts = int(p["norm_groups"])
    return (_rms(read.view(t, parts, -1), float(p["eps"])).reshape(t, inner) * w["norm"]) @ w["o"].T, s


def _exact_feed_forward(w, x):
    gate, up = x @ w["gate_proj.weight"].double().T, x @ w["up_proj.weight"].double().T
    return (torch.nn.functional.silu(gate) * up) @ w["down_proj.weight"].double().T


def _exact_experts(p, w, x):
    e, top = int(p["experts"]), int(p["top"])
    z = x @ w["router"].double().T
    if p.get("router_bias"):
        z = z + w["router.b"].double()
    score = p.get("score", "sigmoid")
    s = z if score == "chosen_softmax" else torch.softmax(z, -1) if score == "softmax" else torch.sigmoid(z)
    choice = s + w["correction"].double() if p.get("correction", True) else s
    groups = int(p.get("groups") or 1)
    if groups > 1:
        rank = choice.view(-1, groups, e // groups).topk(min(2, e // groups), dim=-1).values.sum(-1)
        keep = torch.zeros_like(rank, dtype=torch.bool).scatter_(1, rank.topk(int(p["keep"]), dim=-1).indices, True)
        choice = choice.masked_fill(~keep.repeat_interleave(e // groups, dim=1), -math.inf)
    ids = choice.topk(top, dim=-1).indices
    wts = s.gather(1, ids)
    if score == "chosen_softmax":
        wts = torch.softmax(wts, -1)
    elif p.get("normalize", True):
        wts = wts / (wts.sum(-1, keepdim=True) + 1e-20)

    out = torch.zeros_like(x)
    for i in range(e):
        rows, place = (ids == i).nonzero(as_tuple=True)
        if rows.numel() == 0:
            continue
        u = x[rows] @ w[f"e{i}.up"].double().T
        if p.get("activation") == "gated":
            a = p["gated"]
            gate = (x[rows] @ w[f"e{i}.gate"].double().T).clamp(max=a["limit"])
            u = gate * torch.sigmoid(a["alpha"] * gate) * (u.clamp(-a["limit"], a["limit"]) + a["shift"])
        elif p.get("activation", "gelu") == "gelu":
            u = 0.5 * u * (1 + torch.erf(u / math.sqrt(2.0)))
        else:
            u = torch.relu(u) ** 2
        out.index_add_(0, rows, wts[rows, place][:, None] * (u @ w[f"e{i}.down"].double().T))
    if p.get("shared") is not None:
        out = out + torch.relu(x @ w["shared.up"].double().T) ** 2 @ w["shared.down"].double().T
    return out


def _exact_step(case: dict, seed: int):
    state = _prepare_step(case, seed)
    core, spec = state["core"], _step_spec(case)
    model = DecoderModel(spec)
    skip = (spec.lm_head_name,) if spec.tie_word_embeddings else ()
    w = random_weights(model.expected_weights(), seed, torch.bfloat16, "cuda", skip=skip)
    past = _step_past(case)

    def norm(x, part):
        weight = w[part.tensor_name("weight")].double()
        return _rms(x, float(part.params["eps"])) * (1 + weight if part.params.get("one_plus") else weight)

    x = w[spec.embedding_name][torch.tensor(state["tokens"], device="cuda")].double()
    if spec.embedding is not None:
        x = x * float(spec.embedding.params.get("scale", 1.0))
    for idx, block in enumerate(model.blocks):
        mixer = block.mixer_part()
        local = {n: w[mixer.tensor_name(n)] for n in type(mixer).weight_decls(mixer.params)}
        first = block.norm1 if hasattr(block, "norm1") else block.norm
        rows, cache = norm(x, first), core.pool.caches[idx]
        f = _exact_latent if mixer.kind == "latent_attention" else _exact_attention
        y = []
        for i, n in enumerate(past):
            table = core.block_manager.get_block_table(f"r{i}", cache.group)
            y.append(f(mixer.params, local, rows[i : i + 1], n, _cached(cache.k, table, n), _cached(cache.v, table, n)))
        x = x + torch.cat(y)
        if block.ffn is not None:
            local = {n: w[block.ffn.tensor_name(n)] for n in type(block.ffn).weight_decls(block.ffn.params)}
            x = x + _exact_feed_forward(local, norm(x, block.norm2))
    head = w[spec.embedding_name] if spec.tie_word_embeddings or spec.lm_head_name not in w else w[spec.lm_head_name]
    return {"logits": norm(x, model.final_norm) @ head.double().T, "keys": [None] * len(core.pool.k), "values": [None] * len(core.pool.v)}


def exact(case: dict, seed: int):
    if case["call"] == "step":
        return _exact_step(case, seed)
    spec = _part_spec(case)
    p = spec.params
    mixer = case["part"] not in FEED_FORWARDS
    part = build_part("mixer" if mixer else "ffn", spec, "")
    w = _weights(part, case, seed)
    x, stream = _rows(case, seed, int(p["hidden_size"]))
    x, stream = x.double(), stream.double()
    out = {}
    if case["part"] == "gated_mlp":
        y = _exact_feed_forward(w, x)
    elif case["part"] == "routed_experts":
        y = _exact_experts(p, w, x)
    else:
        new, past = _lengths(case)
        rows = x.split(new)
        if part.cache_need().kind == "none":
            f = _exact_delta if case["part"] == "gated_delta_rule" else _exact_state_space
            parts = [f(p, w, r) for r in rows]
            y = torch.cat([a for a, _ in parts])
            out = {"inputs": None, "matrix": torch.stack([s.reshape(-1) for _, s in parts])}
        else:
            pages = _pages(case, seed, part.cache_need())
            f = {"paged_attention": _exact_attention, "latent_attention": _exact_latent, "talking_attention": _exact_talking}[case["part"]]
            y = torch.cat([f(p, w, r, n, _cached(pages["k"], t, n), _cached(pages["v"], t, n)) for r, n, t in zip(rows, past, pages["tables"])])
            out = {"keys": None, "values": None} if pages["v"] is not pages["k"] else {"keys": None}
    stream = stream + y
    return {"rows": _rms(stream, NORM_EPS), "stream": stream, **out}

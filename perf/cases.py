"""The work that programs have this package do, as cases that can be timed and compared.

A case is a dict of plain values; its ``kind`` names one of the families below.  Two families are whole calls
(`ModelRunner.step` over a request's life); the others are single layers through the parts or the ``ops`` functions that
a decoder is put together from, at the sizes of the configurations in this repository (layer sizes of Qwen2.5-0.5B, 1.5B
and 7B, the mixers and experts of the other decoders at those sizes, head sizes from 16 to 256).
"""

from __future__ import annotations

import json
import math
import tempfile
from pathlib import Path

import numpy as np
import torch

from slipstream_b200 import ops
from slipstream_b200.cache import CacheManager, GroupLayout, PagedStore
from slipstream_b200.engine.context import StepEntry, build_context
from slipstream_b200.engine.runner import ModelRunner
from slipstream_b200.parts import LayerBinding, PagedAttention, RotaryEncoding, Runtime, SwiGLUFeedForward
from slipstream_b200.parts.base import CacheSpec
from slipstream_b200.parts.experts import RoutedExperts
from slipstream_b200.parts.recurrent import MatrixMemoryMixer
from slipstream_b200.parts.state_space import StateSpaceMixer
from slipstream_b200.weights.random_init import random_weights_on_device

DEVICE = torch.device("cuda:0")
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
PAGE = 16

# layer sizes by name; every family below draws from these
SIZES = {
    "0.5b": dict(vocab=151936, width=896, heads=14, kv_heads=2, dim=64, ff=4864, theta=1e6, tied=True),
    "1.5b": dict(vocab=151936, width=1536, heads=12, kv_heads=2, dim=128, ff=8960, theta=1e6, tied=True),
    "7b": dict(vocab=152064, width=3584, heads=28, kv_heads=4, dim=128, ff=18944, theta=1e6, tied=False),
}


def listed() -> list[dict]:
    return [
        # one user, a short question, a small model: every token is a step of one row, bound by latency and launches
        dict(name="generate_0.5b_one_request", kind="generate", size="0.5b", layers=24, requests=1, prompt=17, steps=16),
        # a server under load: ragged prompts arrive together, then all requests decode side by side
        dict(name="generate_7b_layers_16_requests", kind="generate", size="7b", layers=4, requests=16, prompt=3001, steps=12),
        # prompt portions of three requests, two of them behind what earlier steps cached, heads of 128
        dict(name="attention_prompt_heads_of_128", kind="attention", heads=28, kv_heads=4, dim=128, requests=3, tokens=2050,
             cached=3000, window=0, decode=False),
        # the same path for a head size and a mask of other decoders: 96 elements a head under a sliding window
        dict(name="attention_prompt_heads_of_96_window", kind="attention", heads=16, kv_heads=4, dim=96, requests=2, tokens=1531,
             cached=700, window=1024, decode=False),
        # a decode step of many requests at the contexts a chat reaches
        dict(name="attention_decode_48_requests", kind="attention", heads=28, kv_heads=4, dim=128, requests=48, tokens=48,
             cached=90000, window=0, decode=True),
        # routed feed-forward under a prompt portion, and under a decode step, where the touched weights are the work
        dict(name="experts_prompt", kind="experts", width=3584, ff=4736, experts=8, top=2, tokens=1999, gated=True, on_input=True),
        dict(name="experts_decode", kind="experts", width=3584, ff=4736, experts=8, top=2, tokens=12, gated=True, on_input=True),
        # recurrent mixers over prompt portions that start from what earlier steps left in the state
        dict(name="state_space_prompt", kind="state_space", width=3584, heads=112, head_dim=64, state=128, groups=8, requests=2,
             tokens=2045),
        dict(name="matrix_memory_prompt", kind="matrix_memory", width=3584, heads=28, dim=128, value_dim=128, requests=2,
             tokens=1900),
        # the true 32-bit path (trace replay): a layer's two branches under a prompt, and under a few decoded tokens
        dict(name="float32_layer_prompt", kind="float32_layer", size="7b", requests=2, tokens=777, cached=300, decode=False),
        dict(name="float32_layer_decode", kind="float32_layer", size="1.5b", requests=4, tokens=4, cached=2000, decode=True),
        # the end of every sampled step: 64 rows of logits, a different chain of filters in each
        dict(name="sample_64_rows", kind="sample", rows=64, vocab=152064),
    ]


def _log(rng, low: int, high: int) -> int:
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng) -> dict:
    kind = rng.choice(["generate", "attention", "attention", "experts", "experts", "state_space", "matrix_memory",
                       "float32_layer", "float32_layer", "sample"])
    if kind == "generate":
        size = rng.choice(list(SIZES))
        layers = rng.randint(2, {"0.5b": 24, "1.5b": 12, "7b": 4}[size])
        requests = _log(rng, 1, 16)
        return dict(kind=kind, size=size, layers=layers, requests=requests, prompt=requests * _log(rng, 5, 180) + rng.randint(0, 7),
                    steps=rng.randint(3, 12))
    if kind == "attention":
        kv_heads = rng.choice([1, 2, 4, 8])
        heads, dim = kv_heads * rng.choice([1, 2, 4, 7]), rng.choice([32, 64, 64, 80, 96, 128, 128, 192, 256])
        window = rng.choice([0, 0, 0, 512, 1024])
        if rng.random() < 0.5:
            requests = _log(rng, 1, 48)
            return dict(kind=kind, heads=heads, kv_heads=kv_heads, dim=dim, requests=requests, tokens=requests,
                        cached=requests * _log(rng, 100, 1800), window=window, decode=True)
        requests = rng.randint(1, 4)
        return dict(kind=kind, heads=heads, kv_heads=kv_heads, dim=dim, requests=requests, tokens=requests * _log(rng, 33, 700),
                    cached=requests * rng.choice([0, _log(rng, 20, 1200)]), window=window, decode=False)
    if kind == "experts":
        width, wide = rng.choice([(896, 1216), (1536, 2240), (3584, 4736), (2048, 1032)])
        experts = rng.choice([8, 8, 16, 32])
        tokens = _log(rng, 1, 64) if rng.random() < 0.5 else _log(rng, 65, 1900)
        gated = rng.random() < 0.7
        return dict(kind=kind, width=width, ff=wide if experts <= 8 else wide // 16 * 8, experts=experts, top=rng.randint(1, 4), tokens=tokens,
                    gated=gated, on_input=gated and rng.random() < 0.5)
    if kind == "state_space":
        groups = rng.choice([1, 2, 8])
        requests = rng.randint(1, 6)
        return dict(kind=kind, width=rng.choice([896, 1536, 3584]), heads=groups * rng.randint(2, 14), head_dim=rng.choice([32, 64, 64, 128]),
                    state=rng.choice([16, 64, 128, 128, 256]), groups=groups, requests=requests,
                    tokens=requests * (1 if rng.random() < 0.25 else _log(rng, 9, 340)) + (0 if requests > 1 else rng.randint(0, 3)))
    if kind == "matrix_memory":
        requests, dim = rng.randint(1, 6), rng.choice([64, 64, 128, 128, 96, 256])
        return dict(kind=kind, width=rng.choice([896, 1536, 3584]), heads=rng.randint(4, 28), dim=dim, value_dim=rng.choice([dim, dim, 64]),
                    requests=requests, tokens=requests * (1 if rng.random() < 0.25 else _log(rng, 9, 310)))
    if kind == "float32_layer":
        if rng.random() < 0.5:
            requests = _log(rng, 1, 24)
            return dict(kind=kind, size=rng.choice(list(SIZES)), requests=requests, tokens=requests, cached=requests * _log(rng, 20, 1000), decode=True)
        requests = rng.randint(1, 3)
        return dict(kind=kind, size=rng.choice(list(SIZES)), requests=requests, tokens=requests * _log(rng, 20, 250),
                    cached=requests * rng.choice([0, _log(rng, 20, 500)]), decode=False)
    return dict(kind=kind, rows=_log(rng, 1, 64), vocab=rng.choice([152064, 151936, 32000, 50257]))


# --------------------------------------------------------------------------- what the families share

def _shares(total: int, parts: int) -> list[int]:
    """``total`` in ``parts`` uneven parts, the same for everybody: request i gets about (2 + i % 5) shares."""
    weights = np.array([2 + i % 5 for i in range(parts)], dtype=np.float64)
    cuts = np.floor(np.cumsum(weights) / weights.sum() * (total - parts) + 1e-9).astype(int)
    return [int(c) + 1 for c in np.diff(np.concatenate([[0], cuts]))] if total >= parts else [1] * parts


def _token_counts(case: dict) -> list[int]:
    return _shares(case["tokens"], case["requests"])


def _cached_counts(case: dict) -> list[int]:
    """Cached tokens per request; in a prompt step the first request is a new one where there are several."""
    n = case["requests"]
    if not case.get("cached"):
        return [0] * n
    if case["decode"] or n == 1:
        return _shares(case["cached"], n)
    return [0, *_shares(case["cached"], n - 1)]


def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _normal(g: torch.Generator, *shape: int, std: float = 1.0, mean: float = 0.0, dtype: torch.dtype = BF16) -> torch.Tensor:
    t = torch.empty(shape, dtype=F32, device=DEVICE)
    return (t.normal_(0.0, std, generator=g) + mean).to(dtype)


def _draw_weights(specs, g: torch.Generator, dtype: torch.dtype, special: dict | None = None) -> dict[str, torch.Tensor]:
    """Matrices that keep the scale of what passes through them, vectors as their part asks; ``special``: (std, mean) by
    the end of a tensor's name."""
    out = {}
    for s in specs:
        std, mean = s.init[1], 1.0 if s.init[0] == "one_plus_normal" else 0.0
        if len(s.shape) == 2 and s.kind != "vector":
            std = s.shape[1] ** -0.5
        for end, (sd, mn) in (special or {}).items():
            if s.name.endswith(end):
                std, mean = sd, mn
        out[s.name] = _normal(g, *s.shape, std=std, mean=mean, dtype=dtype)
    return out


def _step_context(specs: list[CacheSpec], tokens: list[int], cached: list[int]):
    """A step of ``tokens[i]`` new tokens behind ``cached[i]`` of request i: its context and the layouts of its pages."""
    layouts = [GroupLayout(s, 1) for s in specs]
    pages = sum(-(-(t + c) // PAGE) for t, c in zip(tokens, cached))
    longest = max(t + c for t, c in zip(tokens, cached))
    cache = CacheManager(layouts, [pages] * len(layouts), [PAGE] * len(layouts), len(tokens), longest + 1)
    for i, c in enumerate(cached):
        cache.admit(i)
        if c:
            cache.reserve(i, c)
            cache.commit(i, c)
    ctx = build_context([StepEntry(i, [0] * t, []) for i, t in enumerate(tokens)], cache, 2, DEVICE)
    return cache, layouts, ctx


def _page_rows(cache: CacheManager, kv: torch.Tensor, request: int, count: int) -> tuple[torch.Tensor, torch.Tensor]:
    """A request's first ``count`` cached keys and values, [count, kv heads, dim] in 64 bits."""
    table = torch.tensor(cache.get(request).tables[0], device=DEVICE)
    at = torch.arange(count, device=DEVICE)
    rows = kv[table[at // PAGE], :, :, at % PAGE].to(F64)  # [count, 2, kv heads, dim]
    return rows[:, 0], rows[:, 1]


def _attend(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float, window: int = 0) -> torch.Tensor:
    """Causal attention of the last rows of a request: q [n, heads, dim], k and v [length, kv heads, dim]."""
    n, heads, dim = q.shape
    length, kv_heads = k.shape[:2]
    pos = torch.arange(length - n, length, device=q.device)[:, None]
    key = torch.arange(length, device=q.device)[None]
    hidden = (key > pos) | ((key <= pos - window) if window else torch.zeros_like(key > pos))
    out = torch.empty(n, heads, v.shape[2], dtype=F64, device=q.device)
    for h in range(heads):
        scores = (q[:, h] @ k[:, h // (heads // kv_heads)].T * scale).masked_fill(hidden, -math.inf)
        out[:, h] = torch.softmax(scores, dim=-1) @ v[:, h // (heads // kv_heads)]
    return out.reshape(n, -1)


def _rms(x: torch.Tensor, eps: float) -> torch.Tensor:
    return x * torch.rsqrt(x.square().mean(dim=-1, keepdim=True) + eps)


def _rotate(x: torch.Tensor, positions: torch.Tensor, theta: float) -> torch.Tensor:
    """Rotary positions over [n, heads, dim], half-split pairs.  The angles are float32 products, as the model defines
    them; their sines and everything after are 64-bit."""
    half = x.shape[-1] // 2
    inv_freq = 1.0 / (theta ** (torch.arange(0, 2 * half, 2, dtype=F32) / (2 * half)))
    angle = (positions.to(F32)[:, None] * inv_freq.to(x.device)[None]).to(F64)[:, None, :]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], dim=-1)


# --------------------------------------------------------------------------- generate: a request's life through the model runner

def _generate_parts(case: dict, seed: int):
    z = SIZES[case["size"]]
    rng = np.random.RandomState(seed)
    prompts = [rng.randint(0, z["vocab"], n).tolist() for n in _shares(case["prompt"], case["requests"])]
    answers = rng.randint(0, z["vocab"], (case["steps"], case["requests"])).tolist()
    config = dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", vocab_size=z["vocab"], hidden_size=z["width"],
                  num_hidden_layers=case["layers"], intermediate_size=z["ff"], num_attention_heads=z["heads"],
                  num_key_value_heads=z["kv_heads"], head_dim=z["dim"], rms_norm_eps=1e-6, rope_theta=z["theta"],
                  max_position_embeddings=4096, tie_word_embeddings=z["tied"], torch_dtype="bfloat16")
    return z, prompts, answers, config


def _generate_runner(case: dict, config: dict, seed: int) -> ModelRunner:
    with tempfile.TemporaryDirectory() as folder:
        (Path(folder) / "config.json").write_text(json.dumps(config))
        return ModelRunner(folder, page_size=PAGE, num_pages=case["requests"] * (case["steps"] // PAGE + 2) + case["prompt"] // PAGE + 8,
                           max_num_seqs=case["requests"], max_model_len=4096, load_format="random", seed=seed)


def _generate_prepare(case: dict, seed: int):
    _, prompts, answers, config = _generate_parts(case, seed)
    return dict(runner=_generate_runner(case, config, seed), prompts=prompts, answers=answers)


def _generate_run(state):
    """Prompts in steps of at most 2,048 tokens, then one given token per request and step; the logits of every step."""
    runner, prompts = state["runner"], state["prompts"]
    logits, entries, held = [], [], 0
    for i, tokens in enumerate(prompts):
        if entries and held + len(tokens) > 2048:
            logits.append(runner.step(entries))
            entries, held = [], 0
        entries.append(StepEntry(i, tokens, [len(tokens) - 1]))
        held += len(tokens)
    logits.append(runner.step(entries))
    for tokens in state["answers"]:
        logits.append(runner.step([StepEntry(i, [t], [0]) for i, t in enumerate(tokens)]))
    for i in range(len(prompts)):
        runner.release(i)
    return {"prompts": torch.cat(logits[: len(logits) - len(state["answers"])]), "steps": logits[-len(state["answers"]):]}


def _generate_exact(case: dict, seed: int):
    z, prompts, answers, config = _generate_parts(case, seed)
    runner = _generate_runner(dict(case, prompt=1, requests=1), config, seed)  # only its list of weights is used
    weights = random_weights_on_device(runner.model.weight_specs(), Runtime(DEVICE, BF16), seed)
    del runner
    heads, kv_heads, dim = z["heads"], z["kv_heads"], z["dim"]
    tokens = [p + [a[i] for a in answers] for i, p in enumerate(prompts)]
    starts = np.concatenate([[0], np.cumsum([len(t) for t in tokens])])
    positions = torch.cat([torch.arange(len(t), device=DEVICE) for t in tokens])
    x = weights["model.embed_tokens.weight"][torch.tensor(sum(tokens, []), device=DEVICE)].to(F64)
    for layer in range(case["layers"]):
        w = {k[len(f"model.layers.{layer}."):]: t.to(F64) for k, t in weights.items() if k.startswith(f"model.layers.{layer}.")}
        y = _rms(x, 1e-6) * w["input_layernorm.weight"]
        q, k, v = (y @ w[f"self_attn.{r}_proj.weight"].T + w[f"self_attn.{r}_proj.bias"] for r in "qkv")
        q, k, v = q.view(-1, heads, dim), k.view(-1, kv_heads, dim), v.view(-1, kv_heads, dim)
        q, k = _rotate(q, positions, z["theta"]), _rotate(k, positions, z["theta"])
        mixed = torch.cat([_attend(q[a:b], k[a:b], v[a:b], dim ** -0.5) for a, b in zip(starts[:-1], starts[1:])])
        x = x + mixed @ w["self_attn.o_proj.weight"].T
        y = _rms(x, 1e-6) * w["post_attention_layernorm.weight"]
        x = x + (torch.nn.functional.silu(y @ w["mlp.gate_proj.weight"].T) * (y @ w["mlp.up_proj.weight"].T)) @ w["mlp.down_proj.weight"].T
    x = _rms(x, 1e-6) * weights["model.norm.weight"].to(F64)
    head = weights["model.embed_tokens.weight" if z["tied"] else "lm_head.weight"].to(F64)
    last = torch.tensor([starts[i] + len(p) - 1 for i, p in enumerate(prompts)], device=DEVICE)
    return {"prompts": x[last] @ head.T, "steps": [x[last + 1 + s] @ head.T for s in range(case["steps"])]}


def _generate_work(case: dict) -> dict:
    z = SIZES[case["size"]]
    h, d = z["width"], z["dim"]
    layer = h * (2 * z["heads"] + 2 * z["kv_heads"]) * d + 3 * h * z["ff"]
    passes = -(-case["prompt"] // 2048) + case["steps"]
    rows = case["requests"] * (1 + case["steps"])
    tokens = case["prompt"] + case["requests"] * case["steps"]
    keys = sum(p * (p + 1) // 2 + sum(p + 1 + s for s in range(case["steps"])) for p in _shares(case["prompt"], case["requests"]))
    cached = case["layers"] * 4 * z["kv_heads"] * d * (case["prompt"] * (1 + case["steps"]) + case["requests"] * case["steps"] ** 2 // 2)
    return {"bytes": 2 * passes * (case["layers"] * layer + z["vocab"] * h) + cached + 4 * rows * z["vocab"],
            "flops": 2 * tokens * case["layers"] * layer + 4 * keys * z["heads"] * d * case["layers"] + 2 * rows * z["vocab"] * h}


# --------------------------------------------------------------------------- attention over pages

def _attention_state(case: dict, seed: int):
    g = _generator(seed)
    heads, kv_heads, dim = case["heads"], case["kv_heads"], case["dim"]
    tokens, cached = _token_counts(case), _cached_counts(case)
    cache, layouts, ctx = _step_context([CacheSpec(kv_heads, dim)], tokens, cached)
    kv = PagedStore(layouts, BF16, DEVICE, [[]], len(tokens)).kv[0][0]
    kv.copy_(_normal(g, *kv.shape))  # keys and values of the step itself among them, as behind the page write
    qkv = _normal(g, sum(tokens), (heads + 2 * kv_heads) * dim)
    return cache, dict(case=case, ctx=ctx, kv=kv, qkv=qkv, out=torch.empty(sum(tokens), heads * dim, dtype=BF16, device=DEVICE))


def _attention_run(state):
    case, ctx = state["case"], state["ctx"]
    ops.paged_attention(state["qkv"], state["out"], state["kv"], ctx.groups[0].block_tables, ctx, case["heads"], case["kv_heads"],
                        case["dim"], case["dim"] ** -0.5, window=case["window"])
    return state["out"]


def _attention_exact(case: dict, seed: int):
    cache, s = _attention_state(case, seed)
    q = s["qkv"][:, : case["heads"] * case["dim"]].reshape(-1, case["heads"], case["dim"]).to(F64)
    out, row = [], 0
    for i, (t, c) in enumerate(zip(_token_counts(case), _cached_counts(case))):
        k, v = _page_rows(cache, s["kv"], i, t + c)
        out.append(_attend(q[row: row + t], k, v, case["dim"] ** -0.5, case["window"]))
        row += t
    return torch.cat(out)


def _seen_keys(tokens: list[int], cached: list[int], window: int) -> tuple[int, int]:
    """(pairs of query and key, keys that any query of their request sees)"""
    pairs = keys = 0
    for t, c in zip(tokens, cached):
        seen = np.arange(c + 1, c + t + 1)
        pairs += int(np.minimum(seen, window).sum() if window else seen.sum())
        keys += min(t + c, t + window - 1) if window else t + c
    return pairs, keys


def _attention_work(case: dict) -> dict:
    pairs, keys = _seen_keys(_token_counts(case), _cached_counts(case), case["window"])
    return {"bytes": 2 * case["dim"] * (2 * case["tokens"] * case["heads"] + 2 * keys * case["kv_heads"]),
            "flops": 4 * pairs * case["heads"] * case["dim"]}


# --------------------------------------------------------------------------- routed experts

def _experts_weights(case: dict, seed: int):
    part = RoutedExperts("moe", case["width"], case["ff"], case["experts"], case["top"], renormalize=True,
                         weight_on_input=case["on_input"], gated=case["gated"])
    g = _generator(seed)
    return part, _draw_weights(part.weight_specs(), g, BF16), _normal(g, case["tokens"], case["width"])


def _experts_prepare(case: dict, seed: int):
    part, weights, x = _experts_weights(case, seed)
    part.bind(weights, Runtime(DEVICE, BF16))
    return dict(part=part, x=x)


def _experts_run(state):
    return state["part"].forward(state["x"], None)


def _experts_exact(case: dict, seed: int):
    _, w, x = _experts_weights(case, seed)
    x = x.to(F64)
    scores, ids = torch.topk(torch.sigmoid(x @ w["moe.gate.weight"].to(F64).T), case["top"], dim=-1)
    scores = scores / scores.sum(dim=-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        row, place = torch.nonzero(ids == e, as_tuple=True)
        gate, up, down = (w[f"moe.experts.{e}.{r}_proj.weight"].to(F64) if r != "gate" or case["gated"] else None for r in ("gate", "up", "down"))
        weight = scores[row, place][:, None]
        a = x[row] * weight if case["on_input"] else x[row]
        y = a @ up.T
        y = (torch.nn.functional.silu(a @ gate.T) * y if case["gated"] else torch.relu(y).square()) @ down.T
        out.index_add_(0, row, y if case["on_input"] else y * weight)
    return out


def _experts_work(case: dict) -> dict:
    matrices = 3 if case["gated"] else 2
    touched = case["experts"] * (1.0 - (1.0 - case["top"] / case["experts"]) ** case["tokens"])  # with an even router
    return {"bytes": 2 * (touched * matrices * case["width"] * case["ff"] + case["experts"] * case["width"] + 2 * case["tokens"] * case["width"]),
            "flops": 2 * case["tokens"] * (case["top"] * matrices * case["width"] * case["ff"] + case["experts"] * case["width"])}


# --------------------------------------------------------------------------- recurrent mixers

def _recurrent_prepare(part, special: dict, case: dict, seed: int, state_std: dict):
    g = _generator(seed)
    weights = _draw_weights(part.weight_specs(), g, BF16, special)
    tokens = _token_counts(case)
    cache, _, ctx = _step_context([], tokens, [0] * len(tokens))
    x = _normal(g, sum(tokens), case["width"])
    state = {s.name: _normal(g, len(tokens), *s.shape, std=state_std[s.name], dtype=F32) for s in part.state_specs()}
    slots = [cache.get(i).slot for i in range(len(tokens))]
    return weights, dict(part=part, ctx=ctx, x=x, layer=LayerBinding(state=state)), slots


def _recurrent_run(state):
    out = state["part"].forward(state["x"], state["ctx"], state["layer"])
    return {"out": out, **state["layer"].state}


def _state_space(case: dict, seed: int):
    part = StateSpaceMixer("ssm", case["width"], case["heads"], case["head_dim"], case["state"], case["groups"], taps=4,
                           norm_groups=1, norm_eps=1e-6)
    special = {"dt_bias": (0.5, -1.0), "A_log": (0.5, -0.5), "conv1d.weight": (0.5, 0.0), "conv1d.bias": (0.2, 0.0)}
    return _recurrent_prepare(part, special, case, seed, {"conv": 1.0, "ssm": 0.3})


def _matrix_memory(case: dict, seed: int):
    part = MatrixMemoryMixer("cell", case["width"], case["heads"], case["dim"], case["value_dim"], gate_cap=15.0, norm_eps=1e-6)
    special = {"i.b": (0.5, 0.0), "f.b": (1.0, 3.0)}  # gates that forget slowly, as trained ones do
    return _recurrent_prepare(part, special, case, seed, {"memory": 0.3, "peak": 0.5})


def _bound(made):
    weights, state, _ = made
    state["part"].bind(weights, Runtime(DEVICE, BF16))
    return state


def _scan(decay: torch.Tensor, add_k: torch.Tensor, add_v: torch.Tensor, read: torch.Tensor, start: torch.Tensor):
    """``S <- decay_t S + add_k_t add_v_t^T`` head by head, ``y_t = S_t^T read_t``: decay [n, h], add_k and read [n, h, a],
    add_v [n, h, b], start [h, a, b]; 64 tokens at a time.  Returns (y [n, h, b], the last S)."""
    out, state = [], start
    for i in range(0, decay.shape[0], 64):
        c = decay[i: i + 64].log().cumsum(dim=0).T  # [h, t]
        k, v, q = (t[i: i + 64].transpose(0, 1) for t in (add_k, add_v, read))
        gap = (c[:, :, None] - c[:, None, :]).tril()
        scores = (q @ k.transpose(1, 2) * gap.exp()).tril()
        out.append((scores @ v + (q * c.exp()[..., None]) @ state).transpose(0, 1))
        state = c[:, -1].exp()[:, None, None] * state + (k * (c[:, -1:] - c).exp()[..., None]).transpose(1, 2) @ v
    return torch.cat(out), state


def _state_space_exact(case: dict, seed: int):
    w, s, slots = _state_space(case, seed)
    w = {k[len("ssm."):]: t.to(F64) for k, t in w.items()}
    heads, p, n, groups = case["heads"], case["head_dim"], case["state"], case["groups"]
    inner = heads * p
    proj = s["x"].to(F64) @ w["in_proj.weight"].T
    z, xbc, dt = proj[:, :inner], proj[:, inner: -heads], torch.nn.functional.softplus(proj[:, -heads:] + w["dt_bias"])
    conv, ssm = s["layer"].state["conv"].to(F64), s["layer"].state["ssm"].to(F64)
    out, row = [], 0
    for t, slot in zip(_token_counts(case), slots):
        past = torch.cat([conv[slot], xbc[row: row + t]])
        mixed = torch.nn.functional.silu(sum(past[j: j + t] * w["conv1d.weight"][:, j] for j in range(4)) + w["conv1d.bias"])
        conv[slot] = past[-3:]
        x = mixed[:, :inner].reshape(t, heads, p)
        b, c = (mixed[:, inner + i * groups * n: inner + (i + 1) * groups * n].reshape(t, groups, n).repeat_interleave(heads // groups, dim=1)
                for i in range(2))
        step = dt[row: row + t]
        y, last = _scan((-w["A_log"].exp() * step).exp(), b, step[..., None] * x, c, ssm[slot].transpose(1, 2))
        ssm[slot] = last.transpose(1, 2)
        out.append((y + w["D"][:, None] * x).reshape(t, inner))
        row += t
    y = _rms(torch.cat(out) * torch.nn.functional.silu(z), 1e-6) * w["norm.weight"]
    return {"out": y @ w["out_proj.weight"].T, "conv": conv, "ssm": ssm}


def _matrix_memory_exact(case: dict, seed: int):
    w, s, slots = _matrix_memory(case, seed)
    w = {k[len("cell."):]: t.to(F64) for k, t in w.items()}
    heads, d, v = case["heads"], case["dim"], case["value_dim"]
    x = s["x"].to(F64)
    q, k, val = ((x @ w[r].T).reshape(-1, heads, d if r != "v" else v) for r in ("q", "k", "v"))
    gate_i = 15.0 * torch.tanh((x @ w["i"].T + w["i.b"]) / 15.0)
    gate_f = torch.nn.functional.logsigmoid(15.0 * torch.tanh((x @ w["f"].T + w["f.b"]) / 15.0))
    memory, peak = s["layer"].state["memory"].to(F64), s["layer"].state["peak"].to(F64)
    out, row = [], 0
    for t, slot in zip(_token_counts(case), slots):
        at = slice(row, row + t)
        peaks, m = [], peak[slot]
        for f, i in zip(gate_f[at].cpu(), gate_i[at].cpu()):
            m = torch.maximum(f + m.cpu(), i)
            peaks.append(m)
        peaks = torch.stack(peaks).to(DEVICE)
        before = torch.cat([peak[slot][None], peaks[:-1]])
        grown = torch.exp(gate_i[at] - peaks)[..., None] * torch.cat([val[at], torch.ones_like(val[at][..., :1])], dim=-1)
        y, last = _scan(torch.exp(gate_f[at] + before - peaks), k[at], grown, q[at] * d ** -0.5, memory[slot].transpose(1, 2))
        memory[slot], peak[slot] = last.transpose(1, 2), peaks[-1]
        out.append(y[..., :v] / (torch.maximum(y[..., v].abs(), torch.exp(-peaks)) + 1e-6)[..., None])
        row += t
    o = _rms(torch.cat(out), 1e-6).reshape(-1, heads * v) * w["norm"] * torch.sigmoid(x @ w["g"].T)
    return {"out": o @ w["o"].T, "memory": memory, "peak": peak}


def _state_space_work(case: dict) -> dict:
    inner, gn = case["heads"] * case["head_dim"], case["groups"] * case["state"]
    weights = case["width"] * (3 * inner + 2 * gn + case["heads"])
    cell = case["heads"] * case["head_dim"] * case["state"]
    return {"bytes": 2 * weights + 4 * case["tokens"] * case["width"] + 8 * case["requests"] * (cell + 3 * (inner + 2 * gn)),
            "flops": 2 * case["tokens"] * weights + 5 * case["tokens"] * cell}


def _matrix_memory_work(case: dict) -> dict:
    d, v = case["dim"], case["value_dim"]
    weights = case["width"] * case["heads"] * (2 * d + 3 * v + 2)
    return {"bytes": 2 * weights + 4 * case["tokens"] * case["width"] + 8 * case["requests"] * case["heads"] * d * (v + 1),
            "flops": 2 * case["tokens"] * weights + 5 * case["tokens"] * case["heads"] * d * (v + 1)}


# --------------------------------------------------------------------------- the two branches of a float32 layer

def _float32_layer(case: dict, seed: int):
    z = SIZES[case["size"]]
    mixer = PagedAttention("attn", z["width"], z["heads"], z["kv_heads"], z["dim"], RotaryEncoding(z["dim"], z["theta"]))
    ffn = SwiGLUFeedForward("mlp", z["width"], z["ff"])
    g = _generator(seed)
    weights = _draw_weights(mixer.weight_specs() + ffn.weight_specs(), g, F32)
    tokens, cached = _token_counts(case), _cached_counts(case)
    cache, layouts, ctx = _step_context([mixer.cache_spec()], tokens, cached)
    kv = PagedStore(layouts, F32, DEVICE, [[]], len(tokens)).kv[0][0]
    kv.copy_(_normal(g, *kv.shape, dtype=F32))
    x = _normal(g, sum(tokens), z["width"], dtype=F32)
    return cache, weights, dict(mixer=mixer, ffn=ffn, ctx=ctx, x=x, layer=LayerBinding(kv=kv, group=0))


def _float32_layer_prepare(case: dict, seed: int):
    _, weights, state = _float32_layer(case, seed)
    for part in (state["mixer"], state["mixer"].position_encoding, state["ffn"]):
        part.bind(weights, Runtime(DEVICE, F32))
    return state


def _float32_layer_run(state):
    return {"mixer": state["mixer"].forward(state["x"], state["ctx"], state["layer"]),
            "feed_forward": state["ffn"].forward(state["x"], state["ctx"])}


def _float32_layer_exact(case: dict, seed: int):
    z = SIZES[case["size"]]
    cache, w, s = _float32_layer(case, seed)
    w = {k: t.to(F64) for k, t in w.items()}
    x = s["x"].to(F64)
    q, k, v = ((x @ w[f"attn.{r}_proj.weight"].T + w[f"attn.{r}_proj.bias"]).view(x.shape[0], -1, z["dim"]) for r in "qkv")
    mixed, row = [], 0
    for i, (t, c) in enumerate(zip(_token_counts(case), _cached_counts(case))):
        at, pos = slice(row, row + t), torch.arange(c, c + t, device=DEVICE)
        old_k, old_v = _page_rows(cache, s["layer"].kv, i, c)
        mixed.append(_attend(_rotate(q[at], pos, z["theta"]), torch.cat([old_k, _rotate(k[at], pos, z["theta"])]),
                             torch.cat([old_v, v[at]]), z["dim"] ** -0.5))
        row += t
    gate, up = x @ w["mlp.gate_proj.weight"].T, x @ w["mlp.up_proj.weight"].T
    return {"mixer": torch.cat(mixed) @ w["attn.o_proj.weight"].T,
            "feed_forward": (torch.nn.functional.silu(gate) * up) @ w["mlp.down_proj.weight"].T}


def _float32_layer_work(case: dict) -> dict:
    z = SIZES[case["size"]]
    weights = z["width"] * ((2 * z["heads"] + 2 * z["kv_heads"]) * z["dim"] + 3 * z["ff"])
    pairs, keys = _seen_keys(_token_counts(case), _cached_counts(case), 0)
    return {"bytes": 4 * (weights + 3 * case["tokens"] * z["width"] + 2 * keys * z["kv_heads"] * z["dim"]),
            "flops": 2 * case["tokens"] * weights + 4 * pairs * z["heads"] * z["dim"]}


# --------------------------------------------------------------------------- sampling

def _sample_prepare(case: dict, seed: int):
    """Logits with a few likely tokens over a broad tail, and rows that ask for arg-max, top-k, top-p, min-p, a repetition
    penalty or several of them."""
    g, m, v = _generator(seed), case["rows"], case["vocab"]
    logits = _normal(g, m, v, std=2.0, dtype=F32)
    logits[torch.arange(m, device=DEVICE)[:, None], torch.randint(0, v, (m, 12), generator=g, device=DEVICE)] += 9.0
    row = np.arange(m)
    as_dev = lambda a, dtype: torch.tensor(np.ascontiguousarray(a, dtype=dtype), device=DEVICE)  # noqa: E731
    seen = torch.zeros(m, (v + 31) // 32, dtype=torch.int32, device=DEVICE)
    for i in range(m):
        if i % 4 == 3:
            ops.mark_seen(seen[i], torch.randint(0, v, (300,), generator=g, device=DEVICE, dtype=torch.int32), v)
    return dict(logits=logits, params=dict(
        temperature=as_dev(np.where(row % 8 == 7, 0.0, 0.7 + 0.1 * (row % 5)), "f4"),
        top_k=as_dev(np.where(row % 3 == 1, 40, -1), "i4"), top_p=as_dev(np.where(row % 2 == 0, 0.9, 1.0), "f4"),
        min_p=as_dev(np.where(row % 5 == 4, 0.05, 0.0), "f4"), penalty=as_dev(np.where(row % 4 == 3, 1.1, 1.0), "f4"),
        seeds=as_dev(1000003 * seed + row, "i8"), draws=as_dev(row % 17, "i8"),
        slots=as_dev(np.where(row % 4 == 3, row, -1), "i4"), seen=seen))


def _sample_run(state):
    return ops.sample(state["logits"], **state["params"])


def _sample_work(case: dict) -> dict:
    return {"bytes": 4 * case["rows"] * case["vocab"], "flops": 0}


# --------------------------------------------------------------------------- the families

_PREPARE = {
    "generate": _generate_prepare,
    "attention": lambda case, seed: _attention_state(case, seed)[1],
    "experts": _experts_prepare,
    "state_space": lambda case, seed: _bound(_state_space(case, seed)),
    "matrix_memory": lambda case, seed: _bound(_matrix_memory(case, seed)),
    "float32_layer": _float32_layer_prepare,
    "sample": _sample_prepare,
}
_RUN = {"generate": _generate_run, "attention": _attention_run, "experts": _experts_run, "state_space": _recurrent_run,
        "matrix_memory": _recurrent_run, "float32_layer": _float32_layer_run, "sample": _sample_run}
_EXACT = {"generate": _generate_exact, "attention": _attention_exact, "experts": _experts_exact, "state_space": _state_space_exact,
          "matrix_memory": _matrix_memory_exact, "float32_layer": _float32_layer_exact}
_WORK = {"generate": _generate_work, "attention": _attention_work, "experts": _experts_work, "state_space": _state_space_work,
         "matrix_memory": _matrix_memory_work, "float32_layer": _float32_layer_work, "sample": _sample_work}

# About four times what the path shows against `exact`: rounding of 16-bit activations, weights kept as they are; 32-bit
# sums in the float32 layer; tokens drawn from the same filters are the same.
_TOLERANCE = {
    "generate": {"rel": 0.03},
    "attention": {"rel": 1e-2},
    "experts": {"rel": 1.5e-2},
    "state_space": {"rel": 2e-2},
    "matrix_memory": {"rel": 2e-2},
    "float32_layer": {"rel": 1e-5},
    "sample": "exact",
}


def prepare(case: dict, seed: int):
    with torch.inference_mode():
        return dict(kind=case["kind"], made=_PREPARE[case["kind"]](case, seed))


@torch.inference_mode()
def run(state):
    return _RUN[state["kind"]](state["made"])


@torch.inference_mode()
def exact(case: dict, seed: int):
    make = _EXACT.get(case["kind"])
    return make(case, seed) if make is not None else None


def work(case: dict) -> dict:
    return _WORK[case["kind"]](case)


def tolerance(case: dict):
    return _TOLERANCE[case["kind"]]

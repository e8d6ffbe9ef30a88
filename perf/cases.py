"""The work this engine is measured on: layers alone at the sizes of its model shapes, and one whole serving pass.

Kinds of cases (every layer is built through its registry and called as the model's layers call it):

  mlp        the SwiGLU feed-forward of the Llama shapes, from one decoded token to a whole prompt
  prompt     grouped-query attention over the paged cache for portions of prompts, some behind a history in the cache
  decode     the same mixer for a batch of single tokens at mixed context lengths
  delta, lightning, memory, space
             the recurrent mixers (gated delta rule, lightning attention, matrix memory, state space) on new prompts;
             their outputs and the state they leave behind
  experts    routed gated experts beside a shared one
  serve      requests created, their prompts run in one step, tokens decoded one by one from captured graphs with the
             logits of every step, requests released: the whole model through `Stepper`

Inputs are seeded: normed activations and weights normal, projections scaled so that activations stay of order one.
"""
from __future__ import annotations

import math

import torch

from cisr_b200 import Model, StepEntry, Stepper, parts
from cisr_b200.cache import CacheManager
from cisr_b200.config import LlamaConfig, PartSpec
from cisr_b200.config.presets import preset_dict
from cisr_b200.engine.batch import PinnedRing
from cisr_b200.engine.step import prepare_step
from cisr_b200.ops import build as kernel_build

# layer sizes of the presets: width, feed-forward, query heads, key heads, head size, rotary base
LLAMA = {"smollm2-135m": (576, 1536, 9, 3, 64, 100000.0), "smollm2-1.7b": (2048, 8192, 32, 32, 64, 130000.0),
         "llama-3.1-8b": (4096, 14336, 32, 8, 128, 500000.0)}
# experts, chosen per token, dense width they share, by model width (the shapes of `bench.py --designs`)
ROUTED = {1024: (16, 4, 2048), 2048: (32, 4, 4096), 4096: (64, 8, 8192)}
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
PAGE = 16


def listed():
    return [
        # one decode step of a few users on the smallest shape: launches and latency
        {"name": "mlp 4 tokens 135m", "kind": "mlp", "shape": "smollm2-135m", "tokens": 4, "dtype": "bfloat16"},
        # a portion of a prompt as a token budget cuts it
        {"name": "mlp 200 tokens 8b", "kind": "mlp", "shape": "llama-3.1-8b", "tokens": 200, "dtype": "bfloat16"},
        # a whole prompt on the largest shape
        {"name": "mlp 2048 tokens 8b", "kind": "mlp", "shape": "llama-3.1-8b", "tokens": 2048, "dtype": "bfloat16"},
        # one long prompt on the largest shape
        {"name": "prompt 4096 8b", "kind": "prompt", "shape": "llama-3.1-8b", "requests": 1, "tokens": 4096, "history": 0, "dtype": "bfloat16"},
        # portions of several prompts, each behind an earlier portion, lengths of no tile
        {"name": "prompt ragged 1.7b", "kind": "prompt", "shape": "smollm2-1.7b", "requests": 4, "tokens": 2533, "history": 611, "dtype": "bfloat16"},
        # the float mode of the engine
        {"name": "prompt 1000 135m float", "kind": "prompt", "shape": "smollm2-135m", "requests": 1, "tokens": 1000, "history": 0, "dtype": "float32"},
        # a server's decode step: many users, contexts of mixed length
        {"name": "decode 48 x 3000 8b", "kind": "decode", "shape": "llama-3.1-8b", "requests": 48, "context": 3000, "dtype": "bfloat16"},
        # new prompts through the recurrent mixers of the other designs
        {"name": "delta 2048", "kind": "delta", "width": 2048, "requests": 1, "tokens": 2048},
        {"name": "lightning 2048", "kind": "lightning", "width": 2048, "requests": 1, "tokens": 2048},
        {"name": "memory 3 x 700", "kind": "memory", "width": 2048, "requests": 3, "tokens": 2100},
        # a whole prompt through routed experts
        {"name": "experts 2048", "kind": "experts", "width": 4096, "tokens": 2048},
        # eight users of the smallest shape: prompts, then a reply token by token
        {"name": "serve 8 x 100 + 24", "kind": "serve", "shape": "smollm2-135m", "requests": 8, "tokens": 100, "new": 24},
    ]


def spread(rng, low, high):
    """A whole number between low and high, even over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["mlp", "mlp", "prompt", "prompt", "decode", "delta", "lightning", "memory", "space", "experts", "serve"])
    if kind == "mlp":
        dtype = "float32" if rng.random() < 0.15 else "bfloat16"
        return {"kind": kind, "shape": rng.choice(sorted(LLAMA)), "tokens": spread(rng, 1, 512 if dtype == "float32" else 2048), "dtype": dtype}
    if kind == "prompt":
        if rng.random() < 0.2:
            return {"kind": kind, "shape": "smollm2-135m", "requests": rng.randint(1, 3), "tokens": spread(rng, 64, 1000),
                    "history": rng.choice([0, spread(rng, 16, 500)]), "dtype": "float32"}
        requests = spread(rng, 1, 8)
        return {"kind": kind, "shape": rng.choice(sorted(LLAMA)), "requests": requests, "tokens": spread(rng, 16 * requests, 4000),
                "history": rng.choice([0, spread(rng, 16, 2000)]), "dtype": "bfloat16"}
    if kind == "decode":
        return {"kind": kind, "shape": rng.choice(sorted(LLAMA)), "requests": spread(rng, 1, 64), "context": spread(rng, 64, 4000), "dtype": "bfloat16"}
    if kind == "experts":
        return {"kind": kind, "width": rng.choice(sorted(ROUTED)), "tokens": spread(rng, 1, 2048)}
    if kind == "serve":
        return {"kind": kind, "shape": "smollm2-135m", "requests": spread(rng, 1, 8), "tokens": spread(rng, 16, 400), "new": rng.randint(8, 24)}
    return {"kind": kind, "width": rng.choice([1024, 2048]), "requests": rng.randint(1, 3), "tokens": spread(rng, 96, 2048)}


# ---------------------------------------------------------------- inputs, made from the seed alone
def generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + stream)


def normal(shape, seed, stream, dtype, std=1.0, mean=0.0):
    return (torch.randn(shape, generator=generator(seed, stream), device="cuda") * std + mean).to(dtype)


def lengths(case):
    """Portion lengths of a step's requests: uneven shares of the tokens."""
    n, total = case["requests"], case["tokens"]
    weights = [3 + (5 * i + 2) % 7 for i in range(n)]
    got = [max(2, total * w // sum(weights)) for w in weights]
    got[0] += total - sum(got)
    return got


def contexts(case):
    """Context lengths of a decode batch, this step's token included: a third to all of the longest, mixed."""
    n, longest = case["requests"], case["context"]
    return [max(1, longest - (longest * 2 // 3) * ((7 * i) % n) // n) for i in range(n)]


def histories(case):
    if case["kind"] == "decode":
        return [c - 1 for c in contexts(case)]
    return [case["history"] * (2 + i) // (1 + case["requests"]) if case["history"] else 0 for i in range(case["requests"])]


def dtype_of(case):
    return DTYPES[case.get("dtype", "bfloat16")]


def part_of(case):
    kind, dtype = case["kind"], dtype_of(case)
    if kind == "mlp":
        width, ff = LLAMA[case["shape"]][:2]
        return parts.build_part(parts.FEED_FORWARDS, PartSpec("swiglu", {"hidden_size": width, "intermediate_size": ff}), dtype, kind)
    if kind in ("prompt", "decode"):
        width, _, heads, kv_heads, dim, base = LLAMA[case["shape"]]
        return parts.build_part(parts.MIXERS, PartSpec("gqa_attention", {
            "hidden_size": width, "num_heads": heads, "num_kv_heads": kv_heads, "head_dim": dim,
            "position": PartSpec("rotary_half", {"theta": base, "dim": dim})}), dtype, kind)
    width = case["width"]
    if kind == "experts":
        experts, top, dense = ROUTED[width]
        ff = dense // (top + 1) // 64 * 64
        return parts.build_part(parts.FEED_FORWARDS, PartSpec("routed_experts", {
            "hidden_size": width, "expert_size": ff, "experts": experts, "top": top, "activation": "gated_clamp", "limit": 7.0,
            "scores": "softmax", "renormalize": True, "shared": {"size": ff, "limit": 7.0, "scaled": False}}), dtype, kind)
    heads = width // 64
    if kind == "delta":
        spec = PartSpec("gated_delta", {"hidden_size": width, "num_heads": heads, "num_kv_heads": heads // 4, "key_dim": 64, "value_dim": 64,
                                        "conv": 4, "eps": 1e-5})
    elif kind == "lightning":
        spec = PartSpec("lightning", {"hidden_size": width, "num_heads": heads // 2, "key_dim": 128, "value_dim": 128, "eps": 1e-5,
                                      "decay": [1.0 - 2.0 ** -(5.0 + 3.0 * i / (heads // 2)) for i in range(heads // 2)]})
    elif kind == "memory":
        spec = PartSpec("matrix_memory", {"hidden_size": width, "num_heads": width // 256, "key_dim": 128, "value_dim": 256, "gate_cap": 15.0, "eps": 1e-5})
    else:
        spec = PartSpec("state_space", {"hidden_size": width, "num_heads": heads // 2, "value_dim": 64, "state_dim": 128, "groups": 1, "conv": 4,
                                        "norm_groups": 1, "eps": 1e-5})
    return parts.build_part(parts.MIXERS, spec, dtype, kind)


def tensors_for(needs, seed, dtype):
    """Seeded tensors by name: matrices scaled by their fan-in (or as the part asks), vectors around one (or as it asks)."""
    out = {}
    for i, name in enumerate(sorted(needs)):
        need = needs[name]
        if need.alias is not None:
            continue
        if need.role == "vector":
            mean, std, kept = (1.0 if need.init_mean is None else need.init_mean), (0.1 if need.init_std is None else need.init_std), torch.float32
        else:
            mean, std, kept = 0.0, (need.shape[-1] ** -0.5 if need.init_std is None else need.init_std), dtype
        out[name] = normal(need.shape, seed, 10 + i, kept, std, mean)
    return out


def activations(case, seed):
    width = LLAMA[case["shape"]][0] if "shape" in case else case["width"]
    tokens = case["requests"] if case["kind"] == "decode" else case["tokens"]
    return normal((tokens, width), seed, 1, dtype_of(case))


def history_rows(case, seed, request, n):
    """Keys and values an earlier step left in the cache, [2, n, key heads, head size]."""
    _, _, _, kv_heads, dim, _ = LLAMA[case["shape"]]
    return normal((2, n, kv_heads, dim), seed, 5000 + request, dtype_of(case))


def conversations(case, seed):
    """Prompt and reply tokens of a serving pass, [request][tokens]."""
    vocab = preset_dict(case["shape"])["vocab_size"]
    lens = [max(2, case["tokens"] * (6 + (3 * i) % 5) // 8) for i in range(case["requests"])]
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, vocab, (n,), generator=g).tolist() for n in lens], torch.randint(0, vocab, (case["requests"], case["new"]), generator=g).tolist()


def model_tensors(model, seed):
    return tensors_for(model.tensor_needs(), seed, torch.bfloat16)


# ---------------------------------------------------------------- the framework's side
def prepare(case, seed):
    kind, dtype = case["kind"], dtype_of(case)
    if kind == "serve":
        raw = preset_dict(case["shape"])
        model = Model(LlamaConfig.from_dict(raw).to_spec(), dtype, config=raw, device=torch.device("cuda", torch.cuda.current_device()))
        model.compile_kernels()
        model.load_tensors(model_tensors(model, seed))
        prompts, replies = conversations(case, seed)
        pages = sum(-(-(len(p) + case["new"]) // PAGE) for p in prompts) + 8
        return {"kind": kind, "stepper": Stepper(model, n_pages=pages, page_size=PAGE, max_slots=8, graph=True), "prompts": prompts, "replies": replies}
    part = part_of(case)
    kernel_build.compile_many([job for p in part.planning_parts() for job in p.kernel_jobs()])
    part.load(tensors_for(part.tensor_needs(), seed, dtype))
    state = {"kind": kind, "part": part, "h": activations(case, seed)}
    if kind in ("mlp", "experts"):
        return state
    device = torch.device("cuda", torch.cuda.current_device())
    portions = [1] * case["requests"] if kind == "decode" else lengths(case)
    before = histories(case) if kind in ("prompt", "decode") else [0] * len(portions)
    pages = sum(-(-(a + b) // PAGE) for a, b in zip(portions, before)) + 8
    cache = CacheManager([part.cache_use()], pages, PAGE, len(portions), 8192, dtype=dtype, device=device)
    for r, n in enumerate(before):
        cache.create(r)
        if n:
            cache.reserve([(r, n)])
            cache.commit(r, n)
            binding, table = cache.binding(0), cache.requests[r].tables[0]
            rows = torch.nn.functional.pad(history_rows(case, seed, r, n), (0, 0, 0, 0, 0, -n % PAGE))
            rows = rows.view(2, len(table), PAGE, *rows.shape[2:]).transpose(2, 3)
            at = torch.tensor(table, device=device)
            binding.k[at], binding.v[at] = rows[0], rows[1]
    ring = PinnedRing()
    ctx, _, _ = prepare_step(cache, ring, device, [StepEntry(r, [0] * n) for r, n in enumerate(portions)], 1, planners=part.planning_parts())
    state.update(ctx=ctx, cache=cache, ring=ring, requests=len(portions))
    return state


def run(state):
    kind = state["kind"]
    if kind in ("mlp", "experts"):
        return state["part"].forward(state["h"], None)
    if kind == "serve":
        stepper, prompts, replies = state["stepper"], state["prompts"], state["replies"]
        keys = range(len(prompts))
        for r in keys:
            stepper.create(r)
        logits = [stepper.step([StepEntry(r, prompts[r], [len(prompts[r]) - 1]) for r in keys]).clone()]
        for i in range(len(replies[0])):
            logits.append(stepper.step([StepEntry(r, [replies[r][i]], [0]) for r in keys]).clone())
        for r in keys:
            stepper.release(r)
        return torch.stack(logits)
    cache, ctx = state["cache"], state["ctx"]
    ctx.shared.clear()                       # position tables belong to a step
    state["part"].begin_step(ctx)
    if kind in ("prompt", "decode"):
        return state["part"].forward(state["h"], ctx, cache.binding(0))
    for r in reversed(range(state["requests"])):       # new requests: their states begin at zero
        cache.release(r)
    for r in range(state["requests"]):
        cache.create(r)
    binding = cache.binding(0)
    return state["part"].forward(state["h"], ctx, binding), binding.state[[cache.slot(r) for r in range(state["requests"])]]


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind, size = case["kind"], 4 if case.get("dtype") == "float32" else 2
    if kind == "serve":
        raw = preset_dict(case["shape"])
        width, ff, heads, kv_heads, dim, _ = LLAMA[case["shape"]]
        weights = raw["num_hidden_layers"] * (width * dim * (2 * heads + 2 * kv_heads) + 3 * width * ff) + raw["vocab_size"] * width
        prompts, _ = conversations(case, 0)
        total = sum(map(len, prompts))
        kv = raw["num_hidden_layers"] * 2 * kv_heads * dim * size
        steps, n = case["new"], case["requests"]
        cache = sum(kv * (steps * len(p) + steps * (steps + 1) // 2) for p in prompts)
        logits = (steps + 1) * n * raw["vocab_size"] * 4
        head = raw["vocab_size"] * width
        pairs = sum((len(p) + steps) ** 2 // 2 for p in prompts)
        return {"bytes": (steps + 1) * weights * size + cache + kv * (total + n * steps) + logits,
                "flops": 2 * (weights - head) * (total + n * steps) + 2 * head * n * (steps + 1) + raw["num_hidden_layers"] * 4 * heads * dim * pairs}
    if kind == "mlp":
        width, ff = LLAMA[case["shape"]][:2]
        return {"bytes": 3 * width * ff * size + case["tokens"] * width * (size + 4), "flops": 6 * width * ff * case["tokens"]}
    if kind in ("prompt", "decode"):
        width, _, heads, kv_heads, dim, _ = LLAMA[case["shape"]]
        portions = [1] * case["requests"] if kind == "decode" else lengths(case)
        before = histories(case)
        tokens, cached = sum(portions), sum(before)
        pairs = sum(n * b + n * (n + 1) // 2 for n, b in zip(portions, before))
        matrix = width * dim * (2 * heads + 2 * kv_heads)
        return {"bytes": matrix * size + tokens * width * (size + 4) + (cached + tokens) * 2 * kv_heads * dim * size,
                "flops": 2 * matrix * tokens + 4 * heads * dim * pairs}
    width, tokens = case["width"], case["tokens"]
    if kind == "experts":
        experts, top, dense = ROUTED[width]
        ff = dense // (top + 1) // 64 * 64
        used = min(experts, top * tokens)
        return {"bytes": 3 * (used + 1) * width * ff * size + experts * width * size + tokens * width * (size + 4),
                "flops": tokens * (6 * (top + 1) * width * ff + 2 * experts * width)}
    heads = width // 64
    if kind == "delta":
        hd, dk, dv, columns, inner = heads, 64, 64, 2 * (heads // 4) * 64 + 2 * width + 2 * heads, width
    elif kind == "lightning":
        hd, dk, dv, columns, inner = heads // 2, 128, 128, 4 * width, width
    elif kind == "memory":
        hd, dk, dv, columns, inner = width // 256, 128, 256, 3 * width + 2 * (width // 256), width
    else:
        hd, dk, dv, columns, inner = heads // 2, 128, 64, width + 256 + heads // 2, width // 2
    per_token = (6 if kind == "delta" else 4) * hd * dk * dv        # the state's update and the read-out
    return {"bytes": width * (columns + inner) * size + tokens * width * (size + 4) + case["requests"] * hd * dk * dv * 4,
            "flops": tokens * (2 * width * (columns + inner) + per_token)}


def tolerance(case):
    """About four times the distance from the 64-bit result that the sizes above showed (0.0017 for products of bfloat16
    operands with one rounding between them, 0.0033 where attention adds its own, 0.0092 through thirty layers, 1e-6 in float)."""
    kind = case["kind"]
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    if kind == "serve":
        return {"rel": 4e-2, "max": 0.4}
    if kind == "experts":            # two experts with nearly the same score may change places for a token
        return {"rel": 1.5e-2}
    return {"rel": 1.4e-2 if kind in ("prompt", "decode") else 8e-3, "max": 0.15}


# ---------------------------------------------------------------- the same in 64 bits, in plain torch
def silu(x):
    return x * torch.sigmoid(x)


def rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def rotate(x, first, base):
    dim = x.shape[-1]
    angle = (first + torch.arange(x.shape[0], device="cuda", dtype=torch.float64))[:, None] * base ** (
        -torch.arange(dim // 2, device="cuda", dtype=torch.float64) * 2.0 / dim)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., :dim // 2], x[..., dim // 2:]
    return torch.cat((a * cos - b * sin, b * cos + a * sin), dim=-1)


def attention(q, k, v):
    """q [T, heads, dim] at the last T of the S positions of k, v [S, key heads, dim]."""
    n, heads, dim = q.shape
    out = torch.empty_like(q)
    hidden = torch.ones(n, k.shape[0], dtype=torch.bool, device="cuda").triu(k.shape[0] - n + 1)
    for h in range(heads):
        g = h // (heads // k.shape[1])
        scores = (q[:, h] @ k[:, g].T).mul_(dim ** -0.5).masked_fill_(hidden, float("-inf"))
        out[:, h] = torch.softmax(scores, dim=-1) @ v[:, g]
    return out


def short_conv(x, taps):
    """Causal convolution over time per channel: x [T, C], taps [C, K], the last the current token's."""
    k = taps.shape[1]
    padded = torch.cat((x.new_zeros(k - 1, x.shape[1]), x))
    return sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(k))


def exact_prompt(case, seed, w):
    _, _, heads, kv_heads, dim, base = LLAMA[case["shape"]]
    h = activations(case, seed).double()
    portions = [1] * case["requests"] if case["kind"] == "decode" else lengths(case)
    rows, at = [], 0
    for r, (n, before) in enumerate(zip(portions, histories(case))):
        x = h[at:at + n]
        at += n
        q = rotate((x @ w["q_proj.weight"].T).view(n, heads, dim), before, base)
        k = rotate((x @ w["k_proj.weight"].T).view(n, kv_heads, dim), before, base)
        v = (x @ w["v_proj.weight"].T).view(n, kv_heads, dim)
        if before:
            old = history_rows(case, seed, r, before).double()
            k, v = torch.cat((old[0], k)), torch.cat((old[1], v))
        rows.append(attention(q, k, v).reshape(n, heads * dim) @ w["o_proj.weight"].T)
    return torch.cat(rows)


def exact_recurrent(case, x, w):
    """One request from a zero state: (the output operand of the last projection, the state row as the engine lays it out)."""
    kind, n, width = case["kind"], x.shape[0], case["width"]
    eps, heads = 1e-5, width // 64
    zeros = lambda *shape: torch.zeros(shape, dtype=torch.float64, device="cuda")
    rows = []
    if kind == "delta":
        groups, d = heads // 4, 64
        raw = torch.cat([x @ w[c].T for c in ("q", "k", "v")], dim=1)
        mixed = silu(short_conv(raw, torch.cat([w[c + ".conv"] for c in ("q", "k", "v")])))
        q, k, v = mixed[:, :groups * d].view(n, groups, d), mixed[:, groups * d:2 * groups * d].view(n, groups, d), mixed[:, 2 * groups * d:].view(n, heads, d)
        q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5).repeat_interleave(4, dim=1)
        k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(4, dim=1)
        beta = torch.sigmoid(x @ w["b"].T)[..., None]
        decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a"].T + w["dt_bias"]))[..., None, None]
        S = zeros(heads, d, d)
        for t in range(n):
            S = decay[t] * S
            u = beta[t] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            rows.append(torch.einsum("hkv,hk->hv", S, q[t]))
        out = rms(torch.stack(rows), eps) * w["norm"] * silu((x @ w["g"].T).view(n, heads, d))
        kept = torch.cat((zeros(3, raw.shape[1]), raw))[-3:]
        return out.reshape(n, -1), torch.cat((S.reshape(-1), kept.reshape(-1)))
    if kind == "lightning":
        heads, d = heads // 2, 128
        q, k, v = (silu(x @ w[c].T).view(n, heads, d) for c in ("q", "k", "v"))
        decay = torch.tensor([1.0 - 2.0 ** -(5.0 + 3.0 * i / heads) for i in range(heads)], dtype=torch.float32, device="cuda").double()[:, None, None]
        S = zeros(heads, d, d)
        for t in range(n):
            S = decay * S + k[t][:, :, None] * v[t][:, None, :]
            rows.append(torch.einsum("hkv,hk->hv", S, q[t]))
        o = torch.stack(rows).reshape(n, -1)
        return rms(o, eps) * w["norm"] * torch.sigmoid(x @ w["g"].T), S.transpose(1, 2).reshape(-1)
    if kind == "memory":
        heads, d, dv, cap = width // 256, 128, 256, 15.0
        q, k = (x @ w["q"].T).view(n, heads, d) * d ** -0.5, (x @ w["k"].T).view(n, heads, d)
        v = (x @ w["v"].T).view(n, heads, dv)
        i = cap * torch.tanh((x @ w["i"].T + w["i.b"]) / cap)
        f = torch.nn.functional.logsigmoid(cap * torch.tanh((x @ w["f"].T + w["f.b"]) / cap))
        S, norm, m = zeros(heads, d, dv), zeros(heads, d), zeros(heads)
        for t in range(n):
            top = torch.maximum(f[t] + m, i[t])
            keep, gain = torch.exp(f[t] + m - top)[:, None], torch.exp(i[t] - top)[:, None]
            S = keep[..., None] * S + (gain * k[t])[:, :, None] * v[t][:, None, :]
            norm, m = keep * norm + gain * k[t], top
            scale = torch.maximum((norm * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
            rows.append(torch.einsum("hkv,hk->hv", S, q[t]) / scale[:, None])
        o = rms(torch.stack(rows), eps).reshape(n, -1) * w["norm"] * torch.sigmoid(x @ w["g"].T)
        row = torch.cat((S.reshape(-1), norm.reshape(-1), m))
        return o, torch.cat((row, zeros(-row.numel() % 4)))
    heads, d, dv = heads // 2, 128, 64
    inner = heads * dv
    z, rest, dt = (x @ w["in"].T).split([inner, inner + 2 * d, heads], dim=1)
    mixed = silu(short_conv(rest, w["conv"]) + w["conv.b"])
    xs, B, C = mixed[:, :inner].view(n, heads, dv), mixed[:, inner:inner + d], mixed[:, inner + d:]
    dt = torch.nn.functional.softplus(dt + w["dt_bias"])
    keep = torch.exp(-torch.exp(w["A_log"]) * dt)[..., None, None]
    S = zeros(heads, d, dv)
    for t in range(n):
        S = keep[t] * S + B[t][None, :, None] * (dt[t][:, None] * xs[t])[:, None, :]
        rows.append(torch.einsum("hkv,k->hv", S, C[t]) + w["D"][:, None] * xs[t])
    o = rms(torch.stack(rows).reshape(n, -1) * silu(z), eps) * w["norm"]
    row = torch.cat((S.reshape(-1), torch.cat((zeros(3, rest.shape[1]), rest))[-3:].reshape(-1)))
    return o, torch.cat((row, zeros(-row.numel() % 4)))


def exact_experts(case, x, w):
    experts, top, _ = ROUTED[case["width"]]
    gated = lambda h, gate, up, down: (lambda g, u: (g * torch.sigmoid(1.702 * g) * (u + 1)) @ down.T)((h @ gate.T).clamp(max=7.0), (h @ up.T).clamp(-7.0, 7.0))
    scores = torch.softmax(x @ w["router.weight"].double().T, dim=-1)
    chosen = scores.topk(top, dim=-1)
    weight = chosen.values / (chosen.values.sum(-1, keepdim=True) + 1e-20)
    out = gated(x, *(w[f"shared.{c}"].double() for c in ("gate", "up", "down")))
    for e in range(experts):
        token, place = (chosen.indices == e).nonzero(as_tuple=True)
        if token.numel():
            mats = (w[f"experts.{e}.{c}.weight"].double() for c in ("gate", "up", "down"))
            out.index_add_(0, token, weight[token, place][:, None] * gated(x[token], *mats))
    return out


def exact_serve(case, seed):
    raw = preset_dict(case["shape"])
    _, _, heads, kv_heads, dim, base = LLAMA[case["shape"]]
    w = model_tensors(Model(LlamaConfig.from_dict(raw).to_spec(), torch.bfloat16, config=raw), seed)
    w = {k: v.double() for k, v in w.items()}
    prompts, replies = conversations(case, seed)
    out = torch.empty(case["new"] + 1, len(prompts), raw["vocab_size"], dtype=torch.float64, device="cuda")
    for r, (prompt, reply) in enumerate(zip(prompts, replies)):
        x = w["model.embed_tokens.weight"][torch.tensor(prompt + reply, device="cuda")]
        n = x.shape[0]
        for i in range(raw["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = rms(x, raw["rms_norm_eps"]) * w[p + "input_layernorm.weight"]
            q = rotate((h @ w[p + "self_attn.q_proj.weight"].T).view(n, heads, dim), 0, base)
            k = rotate((h @ w[p + "self_attn.k_proj.weight"].T).view(n, kv_heads, dim), 0, base)
            v = (h @ w[p + "self_attn.v_proj.weight"].T).view(n, kv_heads, dim)
            x = x + attention(q, k, v).reshape(n, -1) @ w[p + "self_attn.o_proj.weight"].T
            h = rms(x, raw["rms_norm_eps"]) * w[p + "post_attention_layernorm.weight"]
            x = x + (silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
        last = rms(x[len(prompt) - 1:], raw["rms_norm_eps"]) * w["model.norm.weight"]
        out[:, r] = last @ w["model.embed_tokens.weight"].T
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return exact_serve(case, seed)
    w = tensors_for(part_of(case).tensor_needs(), seed, dtype_of(case))
    x = activations(case, seed).double()
    if kind == "experts":
        return exact_experts(case, x, w)
    w = {k: v.double() for k, v in w.items()}
    if kind == "mlp":
        return (silu(x @ w["gate_proj.weight"].T) * (x @ w["up_proj.weight"].T)) @ w["down_proj.weight"].T
    if kind in ("prompt", "decode"):
        return exact_prompt(case, seed, w)
    outs, states, at = [], [], 0
    for n in lengths(case):
        out, state = exact_recurrent(case, x[at:at + n], w)
        at += n
        outs.append(out @ w["o"].T)
        states.append(state)
    return torch.cat(outs), torch.stack(states)

"""What the speed of this library is measured on: whole requests through the engine's step function, and single layers
through the parts' own entry points, over the sizes that this repository's benchmark and tests use.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare(case, seed)`` makes what a
program holds before the call (weights, caches, a planned step), ``run(state)`` is one call and returns what it computed,
``exact(case, seed)`` the same in 64 bits by plain tensor operations, ``work(case)`` the bytes and operations the call cannot
do without and ``tolerance(case)`` how far two correct implementations of equal precision may lie apart.
"""
import math

import torch

from llmplayer_b200.cache import SequenceCache
from llmplayer_b200.config import config_from_dict
from llmplayer_b200.engine.engine import Engine
from llmplayer_b200.engine.model import Model
from llmplayer_b200.engine.options import EngineOptions
from llmplayer_b200.engine.step import SequenceStep, StepContext, Workspace
from llmplayer_b200.parts import BLOCKS, FEED_FORWARDS, MIXERS
from llmplayer_b200.parts.base import Runtime
from llmplayer_b200.parts.specs import (BIAS, GAIN, AttentionSpec, BlockSpec, ExpertRoutingSpec, GatedDeltaRuleSpec,
                                        GatedLinearAttentionSpec, LatentAttentionSpec, LowRankDecaySpec, MixtureSpec, NormSpec,
                                        PositionSpec, SwiGLUSpec)

DEV = "cuda:0"
PAGE = 64           # positions per page of the cache
EPS = 1e-5

# width -> (heads, key/value heads, head size, feed-forward width): the Llama shapes of the benchmark (1B, 3B, 8B) and the
# smaller one that its hybrid designs are compared with
LLAMA = {1024: (8, 2, 128, 2816), 2048: (32, 8, 64, 8192), 3072: (24, 8, 128, 8192), 4096: (32, 8, 128, 14336)}
# width -> (heads, latent (dim, rot_dim, vdim, rank), linear attention (heads, dim, vdim), feed-forward width): the
# benchmark's hybrid sizes
HYBRID = {1024: (8, (64, 32, 64, 256), (4, 64, 256), 4096), 2048: (16, (128, 64, 128, 512), (8, 128, 256), 8192),
          4096: (32, (128, 64, 128, 512), (16, 128, 256), 14336)}


def listed():
    return [
        # One short question to a small model: latency, launches and the host path of the step function.
        {"name": "request_llama_one", "kind": "request", "design": "llama", "width": 2048, "layers": 4, "sequences": 1,
         "prompt": 23, "steps": 12},
        # A batch of requests to the hybrid design (a recurrence among latent-attention layers).
        {"name": "request_hybrid_batch", "kind": "request", "design": "ramupel", "width": 2048, "layers": 4, "sequences": 8,
         "prompt": 300, "steps": 16},
        # A layer of the 1B shape over a long prompt: the benchmark's prefill.
        {"name": "block_prompt", "kind": "block", "dtype": "bfloat16", "width": 2048, "sequences": 1, "cached": 0, "new": 2048},
        # A layer of the 8B shape in a decode step of a serving batch, sequences of unequal lengths.
        {"name": "block_decode", "kind": "block", "dtype": "bfloat16", "width": 4096, "sequences": 64, "cached": 2500, "new": 1},
        # The float32 path (exact replays of traces): a prompt, and a step of a few sequences.
        {"name": "block_f32_prompt", "kind": "block", "dtype": "float32", "width": 2048, "sequences": 1, "cached": 0, "new": 509},
        {"name": "block_f32_decode", "kind": "block", "dtype": "float32", "width": 2048, "sequences": 4, "cached": 700, "new": 1},
        # Latent attention: a batch of two prompts of unequal lengths, and a decode step over cached rows.
        {"name": "latent_prompt", "kind": "latent", "width": 2048, "sequences": 2, "cached": 0, "new": 1100},
        {"name": "latent_decode", "kind": "latent", "width": 2048, "sequences": 32, "cached": 1500, "new": 1},
        # Recurrent layers over prompts: linear attention with a decay per key channel, and a delta rule.
        {"name": "linear_prompt", "kind": "linear", "width": 2048, "sequences": 1, "new": 2048},
        {"name": "delta_prompt", "kind": "delta", "width": 2048, "sequences": 3, "new": 777},
        # Routed experts beside a shared one, over a prompt.
        {"name": "mixture_prompt", "kind": "mixture", "width": 2048, "experts": 8, "top": 2, "expert_size": 2048,
         "shared_size": 2048, "tokens": 2048},
        # Attention with capped scores, unit-norm heads, biases and a sink, its weights kept at float32 precision.
        {"name": "capped_prompt", "kind": "capped", "width": 2048, "sequences": 1, "cached": 0, "new": 2048},
    ]


def _spread(rng, lo, hi):
    """A whole number between the two, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["request", "block", "block", "latent", "linear", "delta", "mixture", "capped"])
    if kind == "request":
        n = _spread(rng, 1, 16)
        return {"kind": kind, "design": rng.choice(["llama", "ramupel"]), "width": rng.choice([1024, 2048]),
                "layers": rng.randint(2, 4), "sequences": n, "prompt": _spread(rng, 5, min(400, 2000 // n)),
                "steps": rng.randint(4, 16)}
    if kind == "mixture":
        experts = rng.choice([8, 16, 32])
        return {"kind": kind, "width": rng.choice([1024, 2048]), "experts": experts, "top": rng.randint(1, 4),
                "expert_size": rng.choice([512, 1024, 2048]), "shared_size": rng.choice([0, 1024]),
                "tokens": _spread(rng, 8, 2048)}
    if kind in ("linear", "delta"):
        n = _spread(rng, 1, 4)
        return {"kind": kind, "width": rng.choice([1024, 2048]), "sequences": n, "new": _spread(rng, 40, 2048 // n)}
    decode = rng.random() < 0.5
    n = _spread(rng, 1, 64) if decode else _spread(rng, 1, 4)
    sizes = {"sequences": n, "cached": _spread(rng, 16, 2500) if decode else 0, "new": 1 if decode else _spread(rng, 33, 2048 // n)}
    if kind == "block":
        dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
        if dtype == "float32":       # exact replays are short
            sizes["sequences"] = n = min(n, 8)
            if not decode:
                sizes["new"] = min(sizes["new"], 512 // n)
        return dict({"kind": kind, "dtype": dtype, "width": rng.choice([1024, 2048] if dtype == "float32" else sorted(LLAMA))}, **sizes)
    return dict({"kind": kind, "width": rng.choice([1024, 2048])}, **sizes)


# ---------------------------------------------------------------------------------------------------- inputs
def _lengths(count, longest):
    """Unequal lengths of a batch: the first is the longest, the last about half of it."""
    return [max(1, longest - longest * i // (2 * count)) for i in range(count)]


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * seed + 17)
    return g


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32)


def _weights(specs, g, dtype):
    """Tensors of the given specifications: maps that keep the size of what they multiply, gains around one, and small
    additive vectors."""
    out = {}
    for name, spec in specs.items():
        shape = spec.concrete()
        if spec.kind == GAIN:
            t = 1.0 + 0.1 * _normal(g, *shape)
        elif name.endswith("dwa"):           # weights of the sum over depth
            t = 0.5 + 0.1 * _normal(g, *shape)
        elif name.endswith("dt_bias"):       # time constants of some ten to a hundred tokens
            t = 0.5 * _normal(g, *shape) - 4.0
        elif spec.kind == BIAS:
            t = 0.1 * _normal(g, *shape)
        elif name.endswith(".conv"):
            t = 0.5 * _normal(g, *shape)
        elif name.startswith("embed") or "embed_tokens" in name:
            t = 0.02 * _normal(g, *shape)
        else:
            t = _normal(g, *shape) * shape[-1] ** -0.5
        out[name] = t.to(dtype)
    return out


def _step(cache, slots, counts, workspace):
    """The description of a step that brings ``counts[i]`` new tokens to ``slots[i]``."""
    cache.reserve(slots, counts)
    sequences, start = [], 0
    for slot, n in zip(slots, counts):
        sequences.append(SequenceStep(slot, start, n, cache.length(slot)))
        start += n
    return StepContext(workspace, sequences, [0] * start, cache.page_tables(slots), [])


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _part(case):
    """The layer of a case, built from its specification."""
    d, kind = case["width"], case["kind"]
    if kind == "block":
        H, G, hd, F = LLAMA[d]
        mixer = AttentionSpec(d, H, G, hd, hd ** -0.5, PositionSpec("rope", hd, hd, 500000.0), q="q", k="k", v="v", o="o")
        return BLOCKS.build(BlockSpec(NormSpec(d, EPS, "norm1"), mixer, NormSpec(d, EPS, "norm2"),
                                      SwiGLUSpec(d, F, "gate", "up", "down")))
    if kind == "mixture":
        routing = ExpertRoutingSpec(num_experts=case["experts"], top=case["top"], groups=4, keep_groups=max(2, case["top"] * 4 // case["experts"]),
                                    router="router")
        return FEED_FORWARDS.build(MixtureSpec(d, case["expert_size"], routing, "", shared_size=case["shared_size"],
                                               shared_prefix="shared." if case["shared_size"] else None))
    H, (dn, dr, dv, rank), (gh, gk, gv), _ = HYBRID[d]
    if kind == "latent":
        return MIXERS.build(LatentAttentionSpec(d, H, dn, dr, dv, rank, (dn + dr) ** -0.5, EPS, PositionSpec("rope", dr, dr, 10000.0),
                                                q="q", kv_down="dkv", latent_norm="dkv.norm", k_up="uk", v_up="uv", o="o", out_gate="g"))
    if kind == "linear":
        return MIXERS.build(GatedLinearAttentionSpec(d, gh, gk, gv, EPS, LowRankDecaySpec(16.0, "a1", "a2", "a2.b"),
                                                     q="q", k="k", v="v", gate="g", out_norm="norm", o="o"))
    if kind == "delta":
        return MIXERS.build(GatedDeltaRuleSpec(d, gh, gh, gk, gk, 4, EPS, q="q", k="k", v="v", q_conv="q.conv", k_conv="k.conv",
                                               v_conv="v.conv", strength="b", decay="a1", decay_up="a2", a_log="A_log",
                                               dt_bias="dt_bias", gate="g1", gate_up="g2", gate_activation="sigmoid",
                                               out_norm="norm", o="o"))
    hd = d // H                                     # capped attention, four query heads to a key head
    return MIXERS.build(AttentionSpec(d, H, H // 4, hd, 4.0 * hd ** -0.5, PositionSpec("rope", hd, hd, 10000.0, pairing="interleaved"),
                                      q="q", k="k", v="v", o="o", q_bias="q.b", k_bias="k.b", v_bias="v.b", unit_norm_eps=EPS,
                                      softcap=30.0, sink="sink", exact_weights=True))


def _model_config(case):
    d, layers = case["width"], case["layers"]
    if case["design"] == "llama":
        H, G, hd, F = LLAMA[d]
        return {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": layers, "hidden_size": d, "num_attention_heads": H,
                "num_key_value_heads": G, "head_dim": hd, "intermediate_size": F, "vocab_size": 32000, "rope_theta": 500000.0,
                "rms_norm_eps": EPS, "tie_word_embeddings": True, "max_position_embeddings": 4096}
    H, (dn, dr, dv, rank), (gh, gk, gv), F = HYBRID[d]
    latent = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": F},
              "mixer": {"heads": H, "dim": dn, "rot_dim": dr, "vdim": dv, "kv_rank": rank, "scale": (dn + dr) ** -0.5,
                        "rot": {"base": 10000.0, "dims": dr}}}
    linear = {"type": "gla", "mlp": {"kind": "dense", "ff": F}, "mixer": {"heads": gh, "dim": gk, "vdim": gv, "tau": 16.0}}
    return {"architecture": "Ramupel", "vocab": 32000, "width": d, "embedding": {"scale": float(d) ** 0.5}, "norm": {"eps": EPS},
            "layers": [latent if i % 4 else linear for i in range(layers)]}


def _request_inputs(case, seed):
    config = config_from_dict(_model_config(case))
    model = Model(config.layout())
    g = _generator(seed)
    weights = _weights(model.tensor_specs(), g, torch.bfloat16)
    lengths = _lengths(case["sequences"], case["prompt"])
    ids = torch.randint(0, 32000, (case["sequences"], max(lengths) + case["steps"]), generator=g, device=DEV).tolist()
    prompts = [row[:n] for row, n in zip(ids, lengths)]
    forced = [row[n:n + case["steps"]] for row, n in zip(ids, lengths)]
    return config, model, weights, prompts, forced


def _layer_inputs(case, seed):
    """(part, weights, stream [T, width] float32, cached rows or None, new tokens per sequence, cached per sequence)."""
    part = _part(case)
    g = _generator(seed)
    weights = _weights(part.tensor_specs(), g, _dtype(case))
    if case["kind"] == "mixture":
        return part, weights, _normal(g, case["tokens"], case["width"]), None, [], []
    n = case["sequences"]
    new = [1] * n if case["new"] == 1 else _lengths(n, case["new"])
    cached = _lengths(n, case["cached"]) if case.get("cached") else [0] * n
    x = _normal(g, sum(new), case["width"])
    rows = None
    if sum(cached):
        d = case["width"]
        if case["kind"] == "latent":
            _, (_, dr, _, rank), _, _ = HYBRID[d]
            rows = [_normal(g, c, rank + dr).to(_dtype(case)) for c in cached]
        else:
            G, hd = (LLAMA[d][1], LLAMA[d][2]) if case["kind"] == "block" else (HYBRID[d][0] // 4, d // HYBRID[d][0])
            rows = [_normal(g, 2, G, c, hd).to(_dtype(case)) for c in cached]
    return part, weights, x, rows, new, cached


def _fill(pages, table, rows):
    """Cached rows ([rows, width], or [2, heads, rows, head size]) into the pages of one sequence."""
    n = rows.shape[-2]
    for i, page in enumerate(table):
        lo, hi = i * PAGE, min(n, (i + 1) * PAGE)
        if lo < hi:
            pages[page][..., :hi - lo, :] = rows[..., lo:hi, :]


def prepare(case, seed):
    if case["kind"] == "request":
        config, model, weights, prompts, forced = _request_inputs(case, seed)
        runtime = Runtime(device=torch.device(DEV), dtype="bfloat16")
        model.load(weights, runtime)
        longest = -(-(case["prompt"] + case["steps"]) // PAGE) * PAGE
        engine = Engine(config, model, runtime, max_tokens=longest * len(prompts), max_slots=len(prompts),
                        context_length=longest, options=EngineOptions(dtype="bfloat16"))
        return {"case": case, "engine": engine, "prompts": prompts, "forced": forced}
    part, weights, x, rows, new, cached = _layer_inputs(case, seed)
    runtime = Runtime(device=torch.device(DEV), dtype="float32" if _dtype(case) == torch.float32 else "bfloat16")
    part.load(weights, runtime)
    state = {"case": case, "part": part, "x": x, "workspace": Workspace(torch.device(DEV))}
    if case["kind"] == "mixture":
        state["ctx"] = StepContext(state["workspace"], [], [0] * x.shape[0], [], [])
        state["normed"] = x.to(torch.bfloat16)
        return state
    room = sum(-(-(n + c) // PAGE) * PAGE for n, c in zip(new, cached))
    cache = SequenceCache([part.cache_request()], max_tokens=room, max_slots=len(new), kv_dtype=runtime.kv_dtype, device=DEV)
    slots = [cache.acquire() for _ in new]
    if rows is not None:
        cache.reserve(slots, cached)
        for table, held in zip(cache.page_tables(slots)[0], rows):
            _fill(cache.view(0).pages, table, held)
        cache.commit(slots, cached)
    state.update(cache=cache, slots=slots, ctx=_step(cache, slots, new, state["workspace"]), normed=x.to(runtime.act_dtype))
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "request":
        engine, prompts, forced = state["engine"], state["prompts"], state["forced"]
        slots = [engine.acquire() for _ in prompts]
        logits = [engine.step(list(zip(slots, prompts)), [[len(p) - 1] for p in prompts]).clone()]
        for i in range(len(forced[0])):
            logits.append(engine.step([(s, [f[i]]) for s, f in zip(slots, forced)], [[0]] * len(slots)).clone())
        for s in slots:
            engine.release(s)
        return {"logits": torch.stack(logits)}
    stream = state["x"].clone()                     # the residual stream, which a layer changes in place
    part, ctx = state["part"], state["ctx"]
    if kind == "mixture":
        part.forward(ctx, state["normed"], stream)
        return {"stream": stream}
    cache = state["cache"]
    view = cache.view(0)
    if kind == "block":
        part.forward(ctx, view, stream)
        return {"stream": stream, "cache": view.pages}
    if kind in ("linear", "delta"):                 # new sequences take the slots: their states start at zero
        for s in state["slots"]:
            cache.release(s)
        for _ in state["slots"]:
            cache.acquire()
        part.forward(ctx, view, state["normed"], stream)
        return {"stream": stream, "state": view.rows}
    part.forward(ctx, view, state["normed"], stream)
    return {"stream": stream, "cache": view.pages}


# ---------------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x, gain=None, eps=EPS):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if gain is None else y * gain


def _layer_norm(x, gain):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * gain


def _silu(z):
    return z * torch.sigmoid(z)


def _softplus(z):
    return torch.nn.functional.softplus(z)


def _rotate(v, positions, base, neighbours=False):
    """v [T, heads, n]: pairs (i, i + n/2), or neighbouring ones, turned by position * base^(-2i/n)."""
    n = v.shape[-1]
    f = torch.tensor([base ** (-2.0 * i / n) for i in range(n // 2)], dtype=torch.float32).to(v.device).double()
    angle = positions.double()[:, None, None] * f
    cos, sin = torch.cos(angle), torch.sin(angle)
    a, b = (v[..., 0::2], v[..., 1::2]) if neighbours else (v[..., :n // 2], v[..., n // 2:])
    a, b = a * cos - b * sin, b * cos + a * sin
    return torch.stack([a, b], dim=-1).flatten(-2) if neighbours else torch.cat([a, b], dim=-1)


def _attend(q, k, v, first, scale, softcap=None, sink=None):
    """q [T, H, n] at positions first .. over k, v [S, G, n] from position 0."""
    T, H, _ = q.shape
    S, G, _ = k.shape
    out = torch.empty(T, H, v.shape[-1], dtype=q.dtype, device=q.device)
    hidden = torch.arange(S, device=q.device)[None, :] > first + torch.arange(T, device=q.device)[:, None]
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].T * scale
        if softcap is not None:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(hidden, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], dim=1)
        out[:, h] = torch.softmax(s, dim=-1)[:, :S] @ v[:, h * G // H]
    return out


def _latent_exact(h, q, down, gate, w, sizes, base, first, held, p=""):
    """From the projections of one sequence's new tokens; ``held``: its cached rows or None."""
    H, dn, dr, dv, rank = sizes
    pos = first + torch.arange(h.shape[0], device=h.device)
    rows = torch.cat([_rms(down[:, :rank], w[p + "dkv.norm"]), _rotate(down[:, None, rank:], pos, base)[:, 0]], dim=1)
    if held is not None:
        rows = torch.cat([held, rows], dim=0)
    q = q.reshape(-1, H, dn + dr)
    q = torch.cat([q[..., :dn], _rotate(q[..., dn:], pos, base)], dim=-1)
    k = torch.cat([(rows[:, :rank] @ w[p + "uk"].T).reshape(-1, H, dn), rows[:, None, rank:].expand(-1, H, -1)], dim=-1)
    v = (rows[:, :rank] @ w[p + "uv"].T).reshape(-1, H, dv)
    out = _attend(q, k, v, first, (dn + dr) ** -0.5) * torch.sigmoid(gate)[:, :, None]
    return out.reshape(-1, H * dv) @ w[p + "o"].T


def _linear_exact(h, w, sizes, p=""):
    """Linear attention of one sequence from a zero state: (output, state [heads, value, key])."""
    H, dk, dv = sizes
    T = h.shape[0]
    q = (h @ w[p + "q"].T).reshape(T, H, dk) * dk ** -0.5
    k = (h @ w[p + "k"].T).reshape(T, H, dk)
    v = (h @ w[p + "v"].T).reshape(T, H, dv)
    a = (torch.sigmoid(h @ w[p + "a1"].T @ w[p + "a2"].T + w[p + "a2.b"]) ** (1 / 16.0)).reshape(T, H, dk)
    S = torch.zeros(H, dv, dk, dtype=h.dtype, device=h.device)
    o = torch.empty(T, H, dv, dtype=h.dtype, device=h.device)
    for t in range(T):
        S = S * a[t][:, None, :] + v[t][:, :, None] * k[t][:, None, :]
        o[t] = torch.matmul(S, q[t][:, :, None])[:, :, 0]
    o = _rms(o, w[p + "norm"]).reshape(T, H * dv) * _silu(h @ w[p + "g"].T)
    return o @ w[p + "o"].T, S


def _delta_exact(h, w, sizes):
    """The delta rule of one sequence from a zero state: (output, state [heads, value, key])."""
    H, dk, dv = sizes
    T = h.shape[0]

    def conv(name):
        u = h @ w[name].T
        taps = w[name + ".conv"]
        u = torch.cat([torch.zeros(taps.shape[1] - 1, u.shape[1], dtype=u.dtype, device=u.device), u], dim=0)
        return _silu(sum(u[j:j + T] * taps[:, j] for j in range(taps.shape[1]))).reshape(T, H, -1)

    q, k, v = conv("q"), conv("k"), conv("v")
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    beta = torch.sigmoid(h @ w["b"].T)
    z = h @ w["a1"].T @ w["a2"].T + w["dt_bias"]
    g = torch.exp(-torch.exp(w["A_log"])[None, :, None] * _softplus(z).reshape(T, H, dk))
    S = torch.zeros(H, dv, dk, dtype=h.dtype, device=h.device)
    o = torch.empty(T, H, dv, dtype=h.dtype, device=h.device)
    for t in range(T):
        S = S * g[t][:, None, :]
        u = beta[t][:, None] * (v[t] - torch.matmul(S, k[t][:, :, None])[:, :, 0])
        S = S + u[:, :, None] * k[t][:, None, :]
        o[t] = torch.matmul(S, q[t][:, :, None])[:, :, 0]
    gate = torch.sigmoid(h @ w["g1"].T @ w["g2"].T).reshape(T, H, dv)
    return (_rms(o, w["norm"]) * gate).reshape(T, H * dv) @ w["o"].T, S


def _mixture_exact(h, w, case):
    E, groups = case["experts"], 4
    keep = max(2, case["top"] * 4 // E)
    scores = torch.sigmoid(h @ w["router"].T)
    by_group = scores.reshape(-1, groups, E // groups)
    best = by_group.topk(min(2, E // groups), dim=-1).values.sum(-1).topk(keep, dim=-1).indices
    open_group = torch.zeros(h.shape[0], groups, dtype=torch.bool, device=h.device).scatter_(1, best, True)
    chosen = scores.masked_fill(~open_group.repeat_interleave(E // groups, dim=1), -1.0).topk(case["top"], dim=-1)
    weights = torch.zeros_like(scores).scatter_(1, chosen.indices, chosen.values / chosen.values.sum(-1, keepdim=True))

    def expert(x, p):
        return (_silu(x @ w[p + "gate"].T) * (x @ w[p + "up"].T)) @ w[p + "down"].T

    out = expert(h, "shared.") if case["shared_size"] else torch.zeros_like(h)
    for e in range(E):
        rows = weights[:, e].nonzero()[:, 0]
        out[rows] += weights[rows, e, None] * expert(h[rows], f"e{e}.")
    return out


def _llama_layer(x, w, sizes, first, held, names):
    """One Llama layer on one sequence's new tokens; ``held`` [2, G, cached, hd] or None."""
    H, G, hd, _ = sizes
    T = x.shape[0]
    pos = first + torch.arange(T, device=x.device)
    h = _rms(x, w[names["norm1"]])
    q = _rotate((h @ w[names["q"]].T).reshape(T, H, hd), pos, 500000.0)
    k = _rotate((h @ w[names["k"]].T).reshape(T, G, hd), pos, 500000.0)
    v = (h @ w[names["v"]].T).reshape(T, G, hd)
    if held is not None:
        k, v = torch.cat([held[0].transpose(0, 1), k]), torch.cat([held[1].transpose(0, 1), v])
    x = x + _attend(q, k, v, first, hd ** -0.5).reshape(T, H * hd) @ w[names["o"]].T
    h = _rms(x, w[names["norm2"]])
    return x + (_silu(h @ w[names["gate"]].T) * (h @ w[names["up"]].T)) @ w[names["down"]].T


_BARE = {n: n for n in ("norm1", "q", "k", "v", "o", "norm2", "gate", "up", "down")}


def _llama_names(i):
    p = f"model.layers.{i}."
    return {"norm1": p + "input_layernorm.weight", "norm2": p + "post_attention_layernorm.weight",
            **{n: p + f"self_attn.{n}_proj.weight" for n in "qkvo"}, **{n: p + f"mlp.{n}_proj.weight" for n in ("gate", "up", "down")}}


def _request_exact(case, w, tokens):
    """Logits of one sequence's tokens."""
    d = case["width"]
    ids = torch.tensor(tokens, device=DEV)
    if case["design"] == "llama":
        x = w["model.embed_tokens.weight"][ids]
        for i in range(case["layers"]):
            x = _llama_layer(x, w, LLAMA[d], 0, None, _llama_names(i))
        return _rms(x, w["model.norm.weight"]) @ w["model.embed_tokens.weight"].T
    H, (dn, dr, dv, rank), gla, _ = HYBRID[d]
    streams = [w["embed"][ids] * float(d) ** 0.5]
    x = streams[0]
    for i in range(case["layers"]):
        p = f"l{i}."
        m = p + "mix."
        h = _layer_norm(x, w[p + "norm1"])
        if i % 4:
            y = _latent_exact(h, h @ w[m + "q"].T, h @ w[m + "dkv"].T, h @ w[m + "g"].T, w, (H, dn, dr, dv, rank), 10000.0, 0, None, m)
        else:
            y, _ = _linear_exact(h, w, gla, m)
        z = h @ w[p + "mlp.up"].T
        a, b = _softplus(w[p + "mlp.act"][0]), _softplus(w[p + "mlp.act"][1])
        z = torch.where(z > 0, a * z * z + z / 2, (0.5 + b) * (torch.expm1(z.clamp(max=0)) - z) + z / 2)
        y = y * torch.sigmoid(h @ w[p + "rg1"].T + w[p + "rg1.b"])
        y = y + (z @ w[p + "mlp.down"].T) * torch.sigmoid(h @ w[p + "rg2"].T + w[p + "rg2.b"])
        streams.append(x + y)
        x = sum(w[p + "dwa"][j] * s for j, s in enumerate(streams))
    return _layer_norm(x, w["final.norm"]) @ w["embed"].T


def exact(case, seed):
    if case["kind"] == "request":
        _, _, weights, prompts, forced = _request_inputs(case, seed)
        w = {n: t.double() for n, t in weights.items()}
        rows = [_request_exact(case, w, p + f)[len(p) - 1:len(p) + len(f)] for p, f in zip(prompts, forced)]
        return {"logits": torch.stack(rows, dim=1)}
    part, weights, x, held, new, cached = _layer_inputs(case, seed)
    w = {n: t.double() for n, t in weights.items()}
    kind, d = case["kind"], case["width"]
    h = x.to(_dtype(case)).double()                 # what the layer is given
    x = x.double()
    if kind == "mixture":
        return {"stream": x + _mixture_exact(h, w, case)}
    out, states, start = [], [], 0
    for i, n in enumerate(new):
        xi, hi = x[start:start + n], h[start:start + n]
        kept = None if held is None else held[i].double()
        start += n
        if kind == "block":
            out.append(_llama_layer(xi, w, LLAMA[d], cached[i], kept, _BARE))
            continue
        H, (dn, dr, dv, rank), gla, _ = HYBRID[d]
        if kind == "latent":
            y = _latent_exact(hi, hi @ w["q"].T, hi @ w["dkv"].T, hi @ w["g"].T, w, (H, dn, dr, dv, rank), 10000.0, cached[i], kept)
        elif kind == "linear":
            y, S = _linear_exact(hi, w, gla)
            states.append(S)
        elif kind == "delta":
            y, S = _delta_exact(hi, w, (gla[0], gla[1], gla[1]))
            states.append(S)
        else:
            G, hd = H // 4, d // H
            pos = cached[i] + torch.arange(n, device=x.device)
            q = _rms(_rotate((hi @ w["q"].T + w["q.b"]).reshape(n, H, hd), pos, 10000.0, True))
            k = _rms(_rotate((hi @ w["k"].T + w["k.b"]).reshape(n, G, hd), pos, 10000.0, True))
            v = (hi @ w["v"].T + w["v.b"]).reshape(n, G, hd)
            if kept is not None:
                k, v = torch.cat([kept[0].transpose(0, 1), k]), torch.cat([kept[1].transpose(0, 1), v])
            y = _attend(q, k, v, cached[i], 4.0 * hd ** -0.5, 30.0, w["sink"]).reshape(n, H * hd) @ w["o"].T
        out.append(xi + y)
    result = {"stream": torch.cat(out)}
    if kind in ("linear", "delta"):
        result["state"] = torch.stack(states)
    else:
        result["cache"] = None
    return result


# ---------------------------------------------------------------------------------------------------- work, tolerance
def work(case):
    d, kind = case["width"], case["kind"]
    e = 4 if case.get("dtype") == "float32" else 2
    if kind == "mixture":
        T, E, top = case["tokens"], case["experts"], case["top"]
        one = 3 * d * case["expert_size"]
        shared = 3 * d * case["shared_size"]
        touched = min(E, T * top)
        return {"bytes": 2 * (touched * one + shared + E * d) + T * d * (2 + 8), "flops": 2 * T * (top * one + shared + E * d)}
    n = case["sequences"]
    if kind == "request":
        steps = case["steps"]
        H, G, hd, F = LLAMA[d]
        layer = d * (2 * H + 2 * G) * hd + 3 * d * F
        if case["design"] == "ramupel":
            H, (dn, dr, dv, rank), _, F = HYBRID[d]
            layer = d * (H * (dn + dr) + rank + dr + H * dv) + H * rank * (dn + dv) + 2 * d * F + 2 * d * d
        params = case["layers"] * layer + 32000 * d
        tokens = sum(_lengths(n, case["prompt"]))
        return {"bytes": (steps + 1) * (2 * params + 4 * n * 32000),
                "flops": 2 * case["layers"] * layer * (tokens + n * steps) + 2 * 32000 * d * n * (steps + 1)}
    new = [1] * n if case["new"] == 1 else _lengths(n, case["new"])
    cached = _lengths(n, case["cached"]) if case.get("cached") else [0] * n
    T = sum(new)
    pairs = sum(a * c + a * (a + 1) // 2 for a, c in zip(new, cached))      # (query, key) pairs
    stream = 2 * 4 * T * d
    if kind == "block":
        H, G, hd, F = LLAMA[d]
        params = d * (2 * H + 2 * G) * hd + 3 * d * F
        return {"bytes": e * (params + 2 * G * hd * (T + sum(cached))) + stream, "flops": 2 * T * params + 4 * pairs * H * hd}
    H, (dn, dr, dv, rank), (gh, gk, gv), _ = HYBRID[d]
    if kind == "latent":
        params = d * (H * (dn + dr) + rank + dr + H + H * dv) + H * rank * (dn + dv)
        heads = 2 * pairs * H * ((dn + dr + dv) if not sum(cached) else (2 * rank + dr))
        return {"bytes": 2 * (params + (rank + dr) * (T + sum(cached))) + 2 * T * d + stream, "flops": 2 * T * params + heads}
    if kind == "capped":
        hd = d // H
        params = d * (2 * H + 2 * (H // 4)) * hd
        return {"bytes": 2 * (params + 2 * (H // 4) * hd * (T + sum(cached))) + 2 * T * d + stream,
                "flops": 2 * T * params + 4 * pairs * H * hd}
    if kind == "delta":
        gv = gk
    params = gh * (2 * gk + 3 * gv) * d
    return {"bytes": 2 * params + 2 * T * d + stream + 4 * n * gh * gk * gv, "flops": 2 * T * params + 6 * T * gh * gk * gv}


def tolerance(case):
    """About four times what the layers' results lie off the 64-bit ones: float32 sums, or bfloat16 operands between float32
    sums; through several layers the latter's rounding adds up."""
    if case.get("dtype") == "float32":
        return {"rel": 5e-6, "max": 1e-3}
    kind = "latent_decode" if case["kind"] == "latent" and case["new"] == 1 else case["kind"]
    rel = {"request": 3e-2, "block": 7e-3, "latent": 1.5e-3, "latent_decode": 5e-4, "linear": 3.5e-3, "delta": 3.5e-3,
           "mixture": 5e-3, "capped": 1e-2}[kind]
    return {"rel": rel, "max": 0.3}

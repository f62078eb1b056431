"""The library's work by layer, at the sizes of its own configurations, tests and benchmark: what a serving program calls
for prompts and for single tokens of a running batch.

A case is one call of a public entry point on the tensors that the layer meets there: whole steps of a Qwen3 model
(``Engine.step``), decode attention over the paged cache, the gated feed-forward, routed experts, the recurrences of the
Movudra, Sagupel and Tebozen designs behind their short convolution (prompts and single tokens), attention through a latent
(prompts; single tokens scored against the cached rows), and differential attention with two score maps (prompts, single
tokens).  Sequences of a batch have unequal lengths.  The 32-bit engine, whose kernels are there to check the bfloat16 ones,
is not timed; the recurrences are 32-bit in both engines.
"""
from __future__ import annotations

import math

import torch

from questwend_b200 import Engine, StepEntry
from questwend_b200.cache.manager import CacheManager
from questwend_b200.config.registry import config_from_dict
from questwend_b200.engine.engine import build_step_context
from questwend_b200.kernels import ops
from questwend_b200.parts.base import KVSpec, PartSpec, Runtime, StateSpec
from questwend_b200.parts.registry import build_part

BF, F32, F64 = torch.bfloat16, torch.float32, torch.float64
GOLDEN = 0.6180339887498949
EPS = 1e-6

# Qwen3-0.6B layer sizes (the benchmark's small model) with four layers and its whole vocabulary
QWEN = {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "num_hidden_layers": 4, "hidden_size": 1024,
        "intermediate_size": 3072, "num_attention_heads": 16, "num_key_value_heads": 8, "head_dim": 128, "vocab_size": 151936,
        "rope_theta": 1e6, "rms_norm_eps": EPS, "tie_word_embeddings": True}
# the recurrences: Mamba-2 (Movudra), the delta rule with a decay per key channel (Movudra) or per head (Sagupel), the mLSTM
SSM = {"heads": 64, "vdim": 64, "state": 128, "groups": 8}
MEMORIES = ((4, 256, 512), (16, 128, 128))
CONV_TAPS = 4
GATE_CAP, TINY = 15.0, 1e-6
# latent attention (Movudra, Tebozen) and differential attention (Punolix: a cap; Tebozen: a window and a gate per head)
LATENT = {"heads": 16, "dim": 128, "rot": 64, "vdim": 128, "rank": 512}
MAPS = {"heads": 16, "kv_heads": 4, "dim": 64, "vdim": 128}
LAM, DIFF = 0.6, 0.8
EXPERTS = {"width": 2048, "ff": 1408, "experts": 64, "top": 6, "shared": 2816}


# ----------------------------------------------------------------------------- cases
def listed():
    return [
        # five prompts of unequal lengths through a whole model in one step, a logit row for each
        {"name": "qwen3-5-prompts", "kind": "qwen3", "tokens": 3001, "seqs": 5},
        # one decode step's attention of a batch of 8 at Qwen3-8B heads, norm, rotation and cache write included
        {"name": "gqa-decode-8x4096", "kind": "gqa_decode", "seqs": 8, "ctx": 4096, "heads": 32, "kv_heads": 8},
        # the feed-forward of a decode step of 8 at Qwen3-8B sizes: three matrices streamed
        {"name": "gated-mlp-8", "kind": "gated_mlp", "tokens": 8, "width": 4096, "ff": 12288},
        # router and experts of a decode step of 8
        {"name": "experts-8", "kind": "experts", "tokens": 8},
        # recurrent layers on prompts: one long one, and unequal ones together; the second starts from a state
        {"name": "ssm-prompt-2048", "kind": "ssm", "tokens": 2048, "seqs": 1, "started": False},
        {"name": "delta-3-prompts", "kind": "delta", "tokens": 2900, "seqs": 3, "per_head": False, "started": True},
        {"name": "mlstm-prompt-4096", "kind": "mlstm", "tokens": 4096, "seqs": 1, "memory": 0, "started": False},
        # one token of one sequence through a recurrence: the smallest call of a decode step
        {"name": "ssm-step-1", "kind": "ssm", "tokens": 1, "seqs": 1, "started": True},
        # a prompt through latent attention, and a decode step of 8 over its cached rows
        {"name": "latent-prompt-4096", "kind": "latent_prompt", "tokens": 4096, "seqs": 1, "window": 0, "sink": False, "gate": True},
        {"name": "latent-decode-8x4096", "kind": "latent_decode", "seqs": 8, "ctx": 4096, "window": 0, "sink": True},
        # differential attention: a long prompt with capped scores, and a decode step of 8
        {"name": "maps-prompt-8192", "kind": "maps_prompt", "tokens": 8192, "seqs": 1, "softcap": 50.0, "window": 0, "gate": False},
        {"name": "maps-decode-8x8192", "kind": "maps_decode", "seqs": 8, "ctx": 8192, "softcap": 0.0, "window": 0, "gate": True},
    ]


def _log(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["qwen3", "gqa_decode", "gated_mlp", "experts", "ssm", "delta", "mlstm", "step", "latent_prompt",
                       "latent_decode", "maps_prompt", "maps_decode"])
    if kind == "qwen3":
        tokens = _log(rng, 32, 4096)
        return {"kind": kind, "tokens": tokens, "seqs": rng.randint(1, min(8, tokens // 16))}
    if kind == "gqa_decode":
        seqs = _log(rng, 1, 64)
        heads, kv_heads = rng.choice([(16, 8), (32, 8), (64, 8)])
        return {"kind": kind, "seqs": seqs, "ctx": _log(rng, 64, min(16384, 131072 // seqs)), "heads": heads, "kv_heads": kv_heads}
    if kind == "gated_mlp":
        width, ff = rng.choice([(1024, 3072), (2048, 6144), (4096, 12288)])
        return {"kind": kind, "tokens": _log(rng, 1, 2048), "width": width, "ff": ff}
    if kind == "experts":
        return {"kind": kind, "tokens": _log(rng, 1, 2048)}
    if kind == "step":                                  # single tokens of a batch through one of the recurrences
        kind, seqs = rng.choice(["ssm", "delta", "mlstm"]), _log(rng, 1, 64)
        case = {"kind": kind, "tokens": seqs, "seqs": seqs, "started": True}
        case.update({"per_head": rng.random() < 0.5} if kind == "delta" else {"memory": rng.randrange(2)} if kind == "mlstm" else {})
        return case
    if kind in ("ssm", "delta", "mlstm"):
        tokens = _log(rng, 100, 4096)
        case = {"kind": kind, "tokens": tokens, "seqs": rng.randint(1, min(4, tokens // 32)), "started": rng.random() < 0.3}
        case.update({"per_head": rng.random() < 0.3} if kind == "delta" else {"memory": rng.randrange(2)} if kind == "mlstm" else {})
        return case
    if kind == "latent_prompt":
        tokens = _log(rng, 64, 6144)
        return {"kind": kind, "tokens": tokens, "seqs": rng.randint(1, min(4, tokens // 32)), "window": rng.choice([0, 0, 1024, 4096]),
                "sink": rng.random() < 0.5, "gate": rng.random() < 0.5}
    if kind == "maps_prompt":
        tokens = _log(rng, 64, 6144)
        return {"kind": kind, "tokens": tokens, "seqs": rng.randint(1, min(4, tokens // 32)), "softcap": rng.choice([0.0, 50.0]),
                "window": rng.choice([0, 0, 1024]), "gate": rng.random() < 0.5}
    seqs = _log(rng, 1, 32)
    case = {"kind": kind, "seqs": seqs, "ctx": _log(rng, 64, min(16384, 65536 // seqs)), "window": rng.choice([0, 0, 1024])}
    case.update({"sink": rng.random() < 0.5} if kind == "latent_decode" else {"softcap": rng.choice([0.0, 50.0]), "gate": rng.random() < 0.5})
    return case


# ----------------------------------------------------------------------------- lengths, random tensors, steps
def _cut(total, parts):
    """``total`` in ``parts`` unequal whole pieces of at least 1."""
    weight = [0.5 + (i * GOLDEN) % 1.0 for i in range(parts)]
    ends = [0] + [int(round(total * sum(weight[:i + 1]) / sum(weight))) for i in range(parts)]
    return [b - a for a, b in zip(ends, ends[1:])]


def _lengths(case):
    """New tokens of each sequence, and what it holds before them."""
    n = case["seqs"]
    if "ctx" in case:
        return [1] * n, [max(1, int(case["ctx"] * (0.5 + (i * GOLDEN) % 1.0))) if n > 1 else case["ctx"] for i in range(n)]
    return _cut(case["tokens"], n), [0] * n


class _Draw:
    def __init__(self, seed):
        self.dev = torch.device("cuda:0")
        self.gen = torch.Generator(device=self.dev).manual_seed(seed)

    def normal(self, *shape, dtype=F32, std=1.0):
        return (torch.randn(shape, generator=self.gen, device=self.dev) * std).to(dtype)

    def uniform(self, low, high, *shape):
        return torch.rand(shape, generator=self.gen, device=self.dev) * (high - low) + low


def _step(unit, new, before, device):
    """A cache with one layer run of these needs, filled up to ``before``, and the step that brings ``new`` tokens."""
    longest = max(n + b for n, b in zip(new, before))
    cache = CacheManager([unit], sum(-(-(n + b) // 64) * 64 for n, b in zip(new, before)), len(new) + 1, longest, BF, device)
    slots = cache.open(len(new))
    if any(before):
        build_step_context(cache, [StepEntry(s, [0] * b, []) for s, b in zip(slots, before)], 8, device)
        for s, b in zip(slots, before):
            cache.advance(s, b)
    ctx = build_step_context(cache, [StepEntry(s, [0] * n, []) for s, n in zip(slots, new)], 8, device)[0]
    return cache, cache.unit_cache(0), ctx


def _fill(unit, r):
    unit.k_pool.copy_(r.normal(*unit.k_pool.shape, dtype=BF))
    if unit.v_pool is not None:
        unit.v_pool.copy_(r.normal(*unit.v_pool.shape, dtype=BF))


def _write_strengths(r, n):
    """Biases under softplus for step sizes spread over 0.001 to 0.1, as such layers are initialised."""
    dt = torch.exp(r.uniform(math.log(1e-3), math.log(0.1), n))
    return dt + torch.log(-torch.expm1(-dt))


# ----------------------------------------------------------------------------- what a program has before the call
def _qwen3_weights(r):
    c, D, F = QWEN, QWEN["hidden_size"], QWEN["intermediate_size"]
    nq, nk = c["num_attention_heads"] * c["head_dim"], c["num_key_value_heads"] * c["head_dim"]
    w = {"model.embed_tokens.weight": r.normal(c["vocab_size"], D, dtype=BF, std=0.02), "model.norm.weight": r.uniform(0.9, 1.1, D)}
    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for name, shape in (("self_attn.q_proj", (nq, D)), ("self_attn.k_proj", (nk, D)), ("self_attn.v_proj", (nk, D)),
                            ("self_attn.o_proj", (D, nq)), ("mlp.gate_proj", (F, D)), ("mlp.up_proj", (F, D)), ("mlp.down_proj", (D, F))):
            w[p + name + ".weight"] = r.normal(*shape, dtype=BF, std=0.02)
        for name, n in (("input_layernorm", D), ("post_attention_layernorm", D), ("self_attn.q_norm", c["head_dim"]), ("self_attn.k_norm", c["head_dim"])):
            w[p + name + ".weight"] = r.uniform(0.9, 1.1, n)
    return w


def _qwen3_prompts(case, r):
    ids = torch.randint(0, QWEN["vocab_size"], (case["tokens"],), generator=r.gen, device=r.dev).tolist()
    out, at = [], 0
    for n in _lengths(case)[0]:
        out.append(ids[at:at + n])
        at += n
    return out


def _prepare_qwen3(case, r):
    weights = _qwen3_weights(r)
    prompts = _qwen3_prompts(case, r)
    engine = Engine(config_from_dict(QWEN), weights, BF, r.dev, max_tokens=case["tokens"] + 64 * case["seqs"], max_batch=case["seqs"])
    return {"engine": engine, "prompts": prompts}


def _prepare_gqa_decode(case, r):
    new, before = _lengths(case)
    H, G = case["heads"], case["kv_heads"]
    cache, unit, ctx = _step((KVSpec(G, 128), None, None), new, before, r.dev)
    _fill(unit, r)
    freq = 1e6 ** (-2.0 * torch.arange(64, dtype=F64) / 128)
    cos, sin = ops.rope_table(ctx.tok_pos, freq.to(r.dev))
    return {"cache": cache, "unit": unit, "ctx": ctx, "qkv": r.normal(case["seqs"], (H + 2 * G) * 128), "cos": cos, "sin": sin,
            "qw": r.uniform(0.9, 1.1, 128), "kw": r.uniform(0.9, 1.1, 128)}


def _prepare_gated_mlp(case, r):
    D, F = case["width"], case["ff"]
    part = build_part("feed_forward", PartSpec("gated_mlp", {"hidden_size": D, "intermediate_size": F}), Runtime(r.dev, BF))
    weights = {t.name: r.normal(*t.shape, dtype=BF, std=0.02) for t in part.tensors()}
    state = {"x": r.normal(case["tokens"], D, dtype=BF), "part": part, "plain": dict(weights)}
    part.bind(weights)
    return state


def _prepare_experts(case, r):
    e = EXPERTS
    part = build_part("feed_forward", PartSpec("routed_experts", {
        "hidden_size": e["width"], "expert_size": e["ff"], "experts": e["experts"], "top": e["top"], "gated": False,
        "activation": "relu2", "scores": "sigmoid", "weight_on": "input", "shared_size": e["shared"]}), Runtime(r.dev, BF))
    weights = {t.name: r.normal(*t.shape, dtype=BF, std=0.02) for t in part.tensors()}
    state = {"x": r.normal(case["tokens"], e["width"], dtype=BF), "part": part, "plain": dict(weights)}
    part.bind(weights)
    return state


def _prepare_ssm(case, r):
    new, before = _lengths(case)
    H, P, N, G = (SSM[k] for k in ("heads", "vdim", "state", "groups"))
    inner = H * P
    C = inner + 2 * G * N
    cache, unit, ctx = _step((None, (StateSpec((CONV_TAPS - 1, C)), StateSpec((H, P, N))), None), new, before, r.dev)
    tail, state = unit.state
    if case["started"]:
        tail.copy_(r.normal(*tail.shape))
        state.copy_(r.normal(*state.shape))
    return {"cache": cache, "ctx": ctx, "tail": tail, "state": state, "proj": r.normal(case["tokens"], inner + C + H),
            "conv_w": r.uniform(-0.5, 0.5, C, CONV_TAPS), "conv_b": r.uniform(-0.5, 0.5, C), "dt_bias": _write_strengths(r, H),
            "a_log": torch.log(r.uniform(1.0, 16.0, H)), "d": torch.ones(H, device=r.dev)}


def _prepare_delta(case, r):
    new, before = _lengths(case)
    H, K, P, per_head = 16, 128, 128, case["per_head"]
    Hk = 4 if per_head else 16
    C = 2 * Hk * K + H * P
    n_decay = H if per_head else H * K
    cache, unit, ctx = _step((None, (StateSpec((CONV_TAPS - 1, C)), StateSpec((H, P, K))), None), new, before, r.dev)
    tail, state = unit.state
    if case["started"]:
        tail.copy_(r.normal(*tail.shape))
        state.copy_(r.normal(*state.shape, std=0.3))
    return {"cache": cache, "ctx": ctx, "tail": tail, "state": state, "proj": r.normal(case["tokens"], C + H), "key_heads": Hk,
            "a_raw": r.normal(case["tokens"], n_decay), "conv_w": r.uniform(-0.5, 0.5, C, CONV_TAPS),
            "dt_bias": _write_strengths(r, n_decay), "a_log": torch.log(r.uniform(1.0, 16.0, H)), "per_head": per_head}


def _prepare_mlstm(case, r):
    new, before = _lengths(case)
    H, K, P = MEMORIES[case["memory"]]
    cache, unit, ctx = _step((None, (StateSpec((H, P + 1, K)), StateSpec((H, P + 1))), None), new, before, r.dev)
    state, m = unit.state
    if case["started"]:
        state.copy_(r.normal(*state.shape, std=0.5))
        m.copy_(r.uniform(0.0, 2.0, m.shape[0], H, 1).expand(m.shape))
    return {"cache": cache, "ctx": ctx, "state": state, "m": m, "size": (H, K, P), "i_bias": r.normal(H, std=0.1),
            "f_bias": r.uniform(3.0, 6.0, H), "proj": r.normal(case["tokens"], H * (2 * K + 2 * P) + -(-2 * H // 8) * 8)}


def _prepare_latent_prompt(case, r):
    new, before = _lengths(case)
    H, d, R, P, L = (LATENT[k] for k in ("heads", "dim", "rot", "vdim", "rank"))
    T = case["tokens"]
    _, _, ctx = _step((KVSpec(1, L + R, case["window"], values=False), None, None), new, before, r.dev)
    return {"ctx": ctx, "q": r.normal(T, H, d + R, dtype=BF), "k": r.normal(T, H * d, dtype=BF), "rows": r.normal(T, L + R, dtype=BF),
            "v": r.normal(T, H * P, dtype=BF), "sink": r.normal(H) if case["sink"] else None, "gate": r.normal(T, H) if case["gate"] else None,
            "window": case["window"]}


def _prepare_latent_decode(case, r):
    new, before = _lengths(case)
    H, R, L = (LATENT[k] for k in ("heads", "rot", "rank"))
    cache, unit, ctx = _step((KVSpec(1, L + R, case["window"], values=False), None, None), new, before, r.dev)
    _fill(unit, r)
    # a query taken into the latent space: 128 values times a matrix with entries of a few hundredths
    return {"cache": cache, "unit": unit, "ctx": ctx, "q_abs": r.normal(H, case["seqs"], L, std=0.3), "q_rot": r.normal(case["seqs"], H, R),
            "sink": r.normal(H) if case["sink"] else None, "window": case["window"]}


def _prepare_maps(case, r):
    new, before = _lengths(case)
    H, G, d, P = (MAPS[k] for k in ("heads", "kv_heads", "dim", "vdim"))
    cache, unit, ctx = _step((KVSpec(G, 2 * d, case["window"], value_dim=P), None, None), new, before, r.dev)
    _fill(unit, r)
    T = sum(new)
    return {"cache": cache, "unit": unit, "ctx": ctx, "q": r.normal(T, H, 2 * d, dtype=BF), "gate": r.normal(T, H) if case["gate"] else None,
            "softcap": case["softcap"], "window": case["window"]}


def prepare(case, seed):
    make = {"qwen3": _prepare_qwen3, "gqa_decode": _prepare_gqa_decode, "gated_mlp": _prepare_gated_mlp, "experts": _prepare_experts,
            "ssm": _prepare_ssm, "delta": _prepare_delta, "mlstm": _prepare_mlstm, "latent_prompt": _prepare_latent_prompt,
            "latent_decode": _prepare_latent_decode, "maps_prompt": _prepare_maps, "maps_decode": _prepare_maps}[case["kind"]]
    return {"kind": case["kind"], "case": case, **make(case, _Draw(seed))}


# ----------------------------------------------------------------------------- one pass
def _run_qwen3(s):
    slots = s["engine"].open_sequences(len(s["prompts"]))
    logits = s["engine"].step([StepEntry(slot, p, [len(p) - 1]) for slot, p in zip(slots, s["prompts"])])
    s["engine"].close_sequences(slots)
    return logits


def _run_gqa_decode(s):
    c, ctx, unit = s["case"], s["ctx"], s["unit"]
    return ops.attn_decode_fused(s["qkv"], s["qw"], s["kw"], s["cos"], s["sin"], EPS, unit.k_pool, unit.v_pool, ctx.page_tables[unit.group_id],
                                 ctx.seq_len, 128 ** -0.5, ctx.max_len, c["heads"], c["kv_heads"], 128)


def _run_ffn(s):
    return s["part"].forward(s["x"], None)


def _run_ssm(s):
    H, P, N, G = (SSM[k] for k in ("heads", "vdim", "state", "groups"))
    inner = H * P
    C = inner + 2 * G * N
    xbc = ops.short_conv(s["proj"], inner, C, s["conv_w"], s["conv_b"], s["tail"], s["ctx"])
    y = ops.ssm_scan(xbc, s["proj"], inner + C, s["dt_bias"], s["a_log"], s["d"], s["state"], s["ctx"], H, P, N, G)
    return y, s["state"], s["tail"]


def _run_delta(s):
    H, K, P, Hk = 16, 128, 128, s["key_heads"]
    C = 2 * Hk * K + H * P
    qkv = ops.short_conv(s["proj"], 0, C, s["conv_w"], None, s["tail"], s["ctx"])
    o = ops.delta_rule(qkv, s["proj"], C, s["a_raw"], s["dt_bias"], s["a_log"], s["state"], s["ctx"], H, Hk, K, P, EPS, K ** -0.5,
                       per_head=s["per_head"])
    return o, s["state"], s["tail"]


def _run_mlstm(s):
    H, K, P = s["size"]
    at = H * (2 * K + 2 * P)
    raw, divisor = ops.mlstm_scan(s["proj"], at, at + H, s["i_bias"], s["f_bias"], GATE_CAP, s["state"], s["m"], s["ctx"], H, K, P, K ** -0.5, TINY)
    return raw, divisor, s["state"], s["m"]


def _run_latent_prompt(s):
    H, d, R, P = (LATENT[k] for k in ("heads", "dim", "rot", "vdim"))
    return ops.latent_prefill(s["q"], s["k"], s["rows"], s["v"], s["ctx"], s["sink"], (d + R) ** -0.5, s["window"], H, d, R, P, gate=s["gate"])


def _run_latent_decode(s):
    unit = s["unit"]
    return ops.latent_attention(s["q_abs"], s["q_rot"], unit.k_pool, s["ctx"].page_tables[unit.group_id], s["ctx"], s["sink"],
                                (LATENT["dim"] + LATENT["rot"]) ** -0.5, s["window"])


def _run_maps(s):
    unit = s["unit"]
    return ops.maps_attention(s["q"], unit.k_pool, unit.v_pool, s["ctx"].page_tables[unit.group_id], s["ctx"], 2, MAPS["dim"] ** -0.5,
                              softcap=s["softcap"], lam=LAM, norm_out=True, eps=1e-5, out_scale=1.0 - DIFF, window=s["window"], gate=s["gate"])


_RUN = {"qwen3": _run_qwen3, "gqa_decode": _run_gqa_decode, "gated_mlp": _run_ffn, "experts": _run_ffn, "ssm": _run_ssm, "delta": _run_delta,
        "mlstm": _run_mlstm, "latent_prompt": _run_latent_prompt, "latent_decode": _run_latent_decode, "maps_prompt": _run_maps,
        "maps_decode": _run_maps}


def run(state):
    return _RUN[state["kind"]](state)


# ----------------------------------------------------------------------------- bytes, operations, tolerances
def _pairs(case):
    """Visible (query, key) pairs of the step, and visible keys of single tokens."""
    window, total = case.get("window", 0), 0
    for n, b in zip(*_lengths(case)):
        full = n * (2 * b + n + 1) // 2
        hidden = max(0, b + n - window) if window else 0            # tokens with more than a window of keys: what they don't see
        first = max(0, b + 1 - window) if window else 0
        total += full - (hidden * (hidden + 1) // 2 - (first * (first - 1) // 2 if first else 0) if window else 0)
    return total


def work(case):
    kind, B = case["kind"], case.get("seqs", 1)
    T = case.get("tokens", B)
    if kind == "qwen3":
        c, D = QWEN, QWEN["hidden_size"]
        per = D * 128 * (2 * c["num_attention_heads"] + 2 * c["num_key_value_heads"]) + 3 * D * c["intermediate_size"]
        n, V = c["num_hidden_layers"], c["vocab_size"]
        kv = n * T * 2 * c["num_key_value_heads"] * 128
        return {"bytes": 2 * (n * per + V * D + kv) + 4 * B * V, "flops": 2 * n * per * T + 4 * n * c["num_attention_heads"] * 128 * _pairs(case) + 2 * B * V * D}
    if kind == "gqa_decode":
        H, G, keys = case["heads"], case["kv_heads"], _pairs(case)
        return {"bytes": 4 * keys * G * 128 + B * (4 * (H + 2 * G) * 128 + 2 * H * 128), "flops": 4 * H * 128 * keys}
    if kind == "gated_mlp":
        D, F = case["width"], case["ff"]
        return {"bytes": 6 * D * F + T * D * 6, "flops": 6 * T * D * F}
    if kind == "experts":
        e = EXPERTS
        used = e["experts"] * (1 - (1 - e["top"] / e["experts"]) ** T)      # the experts that T tokens choose, on average
        per = 2 * e["width"] * e["ff"]
        return {"bytes": 2 * (used * per + 2 * e["width"] * e["shared"] + e["experts"] * e["width"]) + 6 * T * e["width"],
                "flops": 2 * T * (e["top"] * per + 2 * e["width"] * e["shared"] + e["experts"] * e["width"])}
    if kind == "ssm":
        H, P, N, G = (SSM[k] for k in ("heads", "vdim", "state", "groups"))
        return {"bytes": 4 * (T * (2 * H * P + 2 * G * N + H) + 2 * B * H * P * N), "flops": T * H * P * N * 4}
    if kind == "delta":
        H, K, P, Hk = 16, 128, 128, 4 if case["per_head"] else 16
        return {"bytes": 4 * (T * (2 * Hk * K + 2 * H * P + H + (H if case["per_head"] else H * K)) + 2 * B * H * P * K), "flops": T * H * P * K * 6}
    if kind == "mlstm":
        H, K, P = MEMORIES[case["memory"]]
        return {"bytes": 4 * (T * H * (2 * K + 2 * P + 3) + 2 * B * H * (P + 1) * K), "flops": T * H * 4 * K * (P + 1)}
    if kind == "latent_prompt":
        H, d, R, P = (LATENT[k] for k in ("heads", "dim", "rot", "vdim"))
        return {"bytes": 2 * T * (H * (2 * d + R + 2 * P) + R), "flops": 2 * H * (d + R + P) * _pairs(case)}
    if kind == "latent_decode":
        H, R, L = (LATENT[k] for k in ("heads", "rot", "rank"))
        return {"bytes": 2 * _pairs(case) * (L + R) + B * H * (4 * (L + R) + 2 * L), "flops": 2 * H * (2 * L + R) * _pairs(case)}
    H, G, d, P = (MAPS[k] for k in ("heads", "kv_heads", "dim", "vdim"))
    n_new = sum(_lengths(case)[0])
    rows = _pairs(case) if kind == "maps_decode" else T
    return {"bytes": 2 * (rows * G * (2 * d + P) + n_new * H * (2 * d + P)), "flops": 2 * H * 2 * (d + P) * _pairs(case)}


def tolerance(case):
    # 32-bit recurrences: sums of a few thousand terms in another order; the rest: bfloat16 operands and results
    if case["kind"] in ("ssm", "delta", "mlstm"):
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "qwen3":
        return {"rel": 0.025, "max": 0.25}
    return {"rel": 0.01, "max": 0.1}


# ----------------------------------------------------------------------------- the same in 64 bits
def _d(t):
    return t.to(F64)


def _rms(x, w, eps=EPS):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turn(x, pos, base):
    """Halves of the last axis turned as pairs by pos * base^(-2i/n); x [T, H, n]."""
    n = x.shape[-1]
    angle = pos[:, None, None] * base ** (-2.0 * torch.arange(n // 2, dtype=F64, device=x.device) / n)
    a, b = x[..., :n // 2], x[..., n // 2:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], -1)


def _attend(q, k, v, scale, before=0, window=0, softcap=0.0, sink=None):
    """One head: q [n, d] at positions before .. before + n - 1, k and v of all positions."""
    out, at = [], torch.arange(len(k), device=q.device)
    for i in range(0, len(q), 2048):
        pos = before + torch.arange(i, min(i + 2048, len(q)), device=q.device)[:, None]
        s = q[i:i + 2048] @ k.T * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill((at > pos) | ((at <= pos - window) if window else False), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.expand(len(s), 1)], 1)
        p = torch.softmax(s, 1)
        out.append((p[:, :-1] if sink is not None else p) @ v)
    return torch.cat(out)


def _cached(pool, table, n):
    """The first n rows of one sequence, [heads, n, size]."""
    pages = _d(pool[table[:-(-n // 64)].long()])
    return pages.permute(1, 0, 2, 3).reshape(pool.shape[1], -1, pool.shape[3])[:, :n]


def _exact_qwen3(case, r):
    w, c = _qwen3_weights(r), QWEN
    H, G, hd = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"]
    rows = []
    for prompt in _qwen3_prompts(case, r):
        n = len(prompt)
        pos = torch.arange(n, dtype=F64, device=r.dev)
        h = _d(w["model.embed_tokens.weight"][torch.tensor(prompt, device=r.dev)])
        for i in range(c["num_hidden_layers"]):
            g = lambda name: _d(w[f"model.layers.{i}.{name}.weight"])                   # noqa: B023
            x = _rms(h, g("input_layernorm"))
            q = _turn(_rms((x @ g("self_attn.q_proj").T).view(n, H, hd), g("self_attn.q_norm")), pos, c["rope_theta"])
            k = _turn(_rms((x @ g("self_attn.k_proj").T).view(n, G, hd), g("self_attn.k_norm")), pos, c["rope_theta"])
            v = (x @ g("self_attn.v_proj").T).view(n, G, hd)
            att = torch.cat([_attend(q[:, a], k[:, a // (H // G)], v[:, a // (H // G)], hd ** -0.5) for a in range(H)], 1)
            h = h + att @ g("self_attn.o_proj").T
            x = _rms(h, g("post_attention_layernorm"))
            h = h + (torch.nn.functional.silu(x @ g("mlp.gate_proj").T) * (x @ g("mlp.up_proj").T)) @ g("mlp.down_proj").T
        rows.append(_rms(h[-1:], _d(w["model.norm.weight"])))
    return torch.cat(rows) @ _d(w["model.embed_tokens.weight"]).T


def _exact_gqa_decode(case, s):
    H, G, unit, ctx = case["heads"], case["kv_heads"], s["unit"], s["ctx"]
    table, out = ctx.page_tables[unit.group_id], []
    for b, n in enumerate(x + 1 for x in _lengths(case)[1]):
        q, k, v = _d(s["qkv"][b]).view(-1, 128).split([H, G, G])
        pos = torch.tensor([n - 1.0], dtype=F64, device=q.device)
        q, k = (_turn(_rms(t, _d(wt))[None], pos, 1e6)[0] for t, wt in ((q, s["qw"]), (k, s["kw"])))
        keys, vals = _cached(unit.k_pool, table[b], n), _cached(unit.v_pool, table[b], n)
        keys[:, -1], vals[:, -1] = k, v
        out.append(torch.cat([_attend(q[h:h + 1], keys[h // (H // G)], vals[h // (H // G)], 128 ** -0.5, before=n - 1) for h in range(H)], 1))
    return torch.cat(out)


def _exact_gated_mlp(case, s):
    w = {k.split("_proj")[0]: _d(v) for k, v in s["plain"].items()}
    x = _d(s["x"])
    return (torch.nn.functional.silu(x @ w["gate"].T) * (x @ w["up"].T)) @ w["down"].T


def _exact_experts(case, s):
    e, w, x = EXPERTS, s["plain"], _d(s["x"])
    weight, chosen = torch.sigmoid(x @ _d(w["router"]).T).topk(e["top"], 1)
    out = torch.relu(x @ _d(w["shared.up"]).T).square() @ _d(w["shared.down"]).T
    for i in range(e["experts"]):
        t, k = (chosen == i).nonzero(as_tuple=True)
        if len(t):
            out.index_add_(0, t, torch.relu((weight[t, k][:, None] * x[t]) @ _d(w[f"e{i}.up"]).T).square() @ _d(w[f"e{i}.down"]).T)
    return out


def _exact_conv(x, w, bias, tail):
    """x [n, C] of one sequence, silu of the convolution with the taps before; and the new tail."""
    taps = w.shape[1]
    full = torch.cat([tail, x])
    y = sum(full[j:j + len(x)] * w[:, j] for j in range(taps)) + (bias if bias is not None else 0.0)
    return torch.nn.functional.silu(y), full[-(taps - 1):]


def _sequences(case, s):
    at = 0
    for slot, n in zip(s["ctx"].slots.tolist(), _lengths(case)[0]):
        yield slot, at, at + n
        at += n


def _exact_ssm(case, s):
    H, P, N, G = (SSM[k] for k in ("heads", "vdim", "state", "groups"))
    inner = H * P
    C = inner + 2 * G * N
    proj, state, tail = _d(s["proj"]), _d(s["state"]), _d(s["tail"])
    a, out = -torch.exp(_d(s["a_log"])), torch.zeros(len(proj), inner, dtype=F64, device=proj.device)
    for slot, t0, t1 in _sequences(case, s):
        xbc, tail[slot] = _exact_conv(proj[t0:t1, inner:inner + C], _d(s["conv_w"]), _d(s["conv_b"]), tail[slot])
        x, b, c = xbc[:, :inner].view(-1, H, P), *(xbc[:, inner + i * G * N:inner + (i + 1) * G * N].view(-1, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
        dt = torch.nn.functional.softplus(proj[t0:t1, inner + C:inner + C + H] + _d(s["dt_bias"]), threshold=100.0)
        decay, S = torch.exp(a * dt), state[slot].clone()
        for t in range(t1 - t0):
            S = decay[t, :, None, None] * S + (dt[t, :, None] * x[t])[:, :, None] * b[t][:, None, :]
            out[t0 + t] = ((S @ c[t][:, :, None])[..., 0] + _d(s["d"])[:, None] * x[t]).reshape(-1)
        state[slot] = S
    return out, state, tail


def _exact_delta(case, s):
    H, K, P, Hk = 16, 128, 128, s["key_heads"]
    C = 2 * Hk * K + H * P
    proj, state, tail = _d(s["proj"]), _d(s["state"]), _d(s["tail"])
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + EPS)
    rate = torch.exp(_d(s["a_log"]))[:, None]
    out = torch.zeros(len(proj), H * P, dtype=F64, device=proj.device)
    for slot, t0, t1 in _sequences(case, s):
        qkv, tail[slot] = _exact_conv(proj[t0:t1, :C], _d(s["conv_w"]), None, tail[slot])
        q, k = (unit(qkv[:, i * Hk * K:(i + 1) * Hk * K].view(-1, Hk, K)).repeat_interleave(H // Hk, 1) for i in (0, 1))
        q, v = q * K ** -0.5, qkv[:, 2 * Hk * K:].view(-1, H, P)
        beta = torch.sigmoid(proj[t0:t1, C:C + H])
        decay = torch.exp(-rate * torch.nn.functional.softplus(_d(s["a_raw"][t0:t1]) + _d(s["dt_bias"]), threshold=100.0).view(t1 - t0, H, -1))
        S = state[slot].clone()                                             # [H, P, K]
        for t in range(t1 - t0):
            S = S * decay[t][:, None, :]
            u = beta[t, :, None] * (v[t] - (S @ k[t][:, :, None])[..., 0])
            S = S + u[:, :, None] * k[t][:, None, :]
            out[t0 + t] = (S @ q[t][:, :, None]).reshape(-1)
        state[slot] = S
    return out, state, tail


def _exact_mlstm(case, s):
    H, K, P = s["size"]
    proj, state, m = _d(s["proj"]), _d(s["state"]), _d(s["m"])
    at = H * (2 * K + 2 * P)
    cap = lambda z: GATE_CAP * torch.tanh(z / GATE_CAP)
    i, f = cap(proj[:, at:at + H] + _d(s["i_bias"])), torch.nn.functional.logsigmoid(cap(proj[:, at + H:at + 2 * H] + _d(s["f_bias"])))
    q, k, v = (proj[:, a:a + H * n].view(-1, H, n) for a, n in ((0, K), (H * K, K), (2 * H * K, P)))
    v = torch.cat([v, torch.ones_like(v[..., :1])], -1)
    raw, divisor = torch.zeros(len(proj), H * P, dtype=F64, device=proj.device), torch.zeros(len(proj), H, dtype=F64, device=proj.device)
    for slot, t0, t1 in _sequences(case, s):
        S, last = state[slot].clone(), m[slot, :, 0].clone()
        for t in range(t0, t1):
            top = torch.maximum(last + f[t], i[t])
            S = torch.exp(last + f[t] - top)[:, None, None] * S + (torch.exp(i[t] - top)[:, None] * v[t])[:, :, None] * k[t][:, None, :]
            y, last = (S @ q[t][:, :, None])[..., 0] * K ** -0.5, top
            raw[t], divisor[t] = y[:, :P].reshape(-1), torch.maximum(y[:, P].abs(), torch.exp(-top)) + TINY
        state[slot], m[slot] = S, last[:, None]
    return raw, divisor, state, m


def _exact_latent_prompt(case, s):
    H, d, R, P = (LATENT[k] for k in ("heads", "dim", "rot", "vdim"))
    out, at = [], 0
    for n in _lengths(case)[0]:
        q, k, v = (s[x][at:at + n].view(n, H, -1) for x in ("q", "k", "v"))
        rot = s["rows"][at:at + n, -R:]
        o = torch.stack([_attend(_d(q[:, h]), _d(torch.cat([k[:, h], rot], 1)), _d(v[:, h]), (d + R) ** -0.5, window=case["window"],
                                 sink=_d(s["sink"][h]) if case["sink"] else None) for h in range(H)], 1)
        out.append((o * torch.sigmoid(_d(s["gate"][at:at + n]))[..., None] if case["gate"] else o).reshape(n, H * P))
        at += n
    return torch.cat(out)


def _exact_latent_decode(case, s):
    L, unit, out = LATENT["rank"], s["unit"], []
    table = s["ctx"].page_tables[unit.group_id]
    for b, n in enumerate(x + 1 for x in _lengths(case)[1]):
        rows, q = _cached(unit.k_pool, table[b], n)[0], torch.cat([_d(s["q_abs"][:, b]), _d(s["q_rot"][b])], 1)
        out.append(torch.cat([_attend(q[h:h + 1], rows, rows[:, :L], (LATENT["dim"] + LATENT["rot"]) ** -0.5, before=n - 1, window=case["window"],
                                      sink=_d(s["sink"][h]) if case["sink"] else None) for h in range(len(q))]))
    return torch.stack(out, 1)


def _exact_maps(case, s):
    H, G, d, P = (MAPS[k] for k in ("heads", "kv_heads", "dim", "vdim"))
    unit, out, at = s["unit"], [], 0
    table = s["ctx"].page_tables[unit.group_id]
    for b, (n, before) in enumerate(zip(*_lengths(case))):
        keys, vals = _cached(unit.k_pool, table[b], n + before), _cached(unit.v_pool, table[b], n + before)
        heads = []
        for h in range(H):
            k, v, q = keys[h // (H // G)], vals[h // (H // G)], _d(s["q"][at:at + n, h])
            a = [_attend(q[:, m * d:(m + 1) * d], k[:, m * d:(m + 1) * d], v, d ** -0.5, before, case["window"], case["softcap"]) for m in (0, 1)]
            heads.append(_rms(a[0] - LAM * a[1], 1.0 - DIFF, 1e-5))
        o = torch.stack(heads, 1)
        out.append((o * torch.sigmoid(_d(s["gate"][at:at + n]))[..., None] if case["gate"] else o).reshape(n, H * P))
        at += n
    return torch.cat(out)


def exact(case, seed):
    if case["kind"] == "qwen3":
        return _exact_qwen3(case, _Draw(seed))
    make = {"gqa_decode": _exact_gqa_decode, "gated_mlp": _exact_gated_mlp, "experts": _exact_experts, "ssm": _exact_ssm,
            "delta": _exact_delta, "mlstm": _exact_mlstm, "latent_prompt": _exact_latent_prompt, "latent_decode": _exact_latent_decode, "maps_prompt": _exact_maps, "maps_decode": _exact_maps}
    return make[case["kind"]](case, prepare(case, seed))

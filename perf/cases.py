"""What the library's speed is measured on: steps of its decoders, through ``LanguageModel.step``.

A case is a model (a decoder and a size of ``camelid_b200.benchmark``), a compute type, a number of sequences, the range
of their prompts' lengths (``low`` to ``high`` tokens, spread evenly, odd lengths among them), a number of single-token
``steps``, and where a pass begins:

* ``begin: "cache"``: the prompts stand in the cache; a pass runs ``steps`` single-token steps and rolls the cache back.
* ``begin: "prompt"``: a pass takes slots, runs all prompts in one step, then ``steps`` single-token steps, and gives the
  slots back: a request from its first token to its last.

The tokens are given, as when a text is scored or a trace is replayed, so the outputs are float32 logits: of each
prompt's last ``kept`` positions, and of every single-token step. ``exact`` makes the same logits in 64 bits from the
weights alone. Where rows are routed to experts, the norm behind the feed-forwards of two decoders (Nudusun, Zulozen with
experts) turns a near-tie that another rounding breaks the other way into a tenth of the row, so that two correct
implementations can lie further apart than a comparison allows; routed experts are therefore measured in the Ramopel
decoder, which has no such norm, and Zulozen with dense feed-forwards. The models are drawn on the device with a fixed seed and kept while cases ask for them; prompts and
tokens come from the case's seed.
"""
from __future__ import annotations

import math
import re

import numpy as np
import torch

import camelid_b200
from camelid_b200 import StepEntry, benchmark
from camelid_b200.engine.model import DecoderModel
from camelid_b200.weights.random_init import random_tensor

WEIGHTS_SEED = 7
F64 = torch.float64


def listed():
    bf16, prompt, cache = {"dtype": "bfloat16"}, {"begin": "prompt", "kept": 1}, {"begin": "cache", "kept": 0}
    return [
        # one user's next token: the smallest call, bound by the chain of launches
        {"name": "llama 1b next token of 1", "model": "llama", "size": "1b", **bf16, "batch": 1, "low": 511, "high": 511, "steps": 1, **cache},
        # the benchmark's own decode step: 8 sequences behind prompts of 2,048 tokens
        {"name": "llama 1b next token of 8", "model": "llama", "size": "1b", **bf16, "batch": 8, "low": 2048, "high": 2048, "steps": 1, **cache},
        # a busy service: 64 sequences of unequal length
        {"name": "llama 1b next token of 64", "model": "llama", "size": "1b", **bf16, "batch": 64, "low": 65, "high": 2047, "steps": 1, **cache},
        # the benchmark's own prompt
        {"name": "llama 1b prompt of 2048", "model": "llama", "size": "1b", **bf16, "batch": 1, "low": 2048, "high": 2048, "steps": 0, **prompt},
        # a batch of unequal prompts in one step of the widest layers: the largest call
        {"name": "llama wide 16 prompts", "model": "llama", "size": "wide", **bf16, "batch": 16, "low": 64, "high": 1601, "steps": 0, **prompt},
        # the 32-bit path, short requests: what a trace replay against the reference runs
        {"name": "llama 1b float32 4 requests", "model": "llama", "size": "1b", "dtype": "float32", "batch": 4, "low": 37, "high": 300, "steps": 8, **prompt},
        # the other decoders: a long prompt of one user and a short answer, or several users' requests together
        {"name": "fomatar long request", "model": "fomatar", "size": "medium", **bf16, "batch": 1, "low": 2048, "high": 2048, "steps": 8, **prompt},
        {"name": "fomatar 4 requests", "model": "fomatar", "size": "small", **bf16, "batch": 4, "low": 130, "high": 901, "steps": 16, **prompt},
        {"name": "zulozen 8 requests", "model": "zulozen", "size": "medium", **bf16, "batch": 8, "low": 100, "high": 700, "steps": 8, **prompt},
        {"name": "kizezen long request", "model": "kizezen", "size": "medium", **bf16, "batch": 1, "low": 2048, "high": 2048, "steps": 8, **prompt},
        {"name": "ramopel 2 requests", "model": "ramopel", "size": "small", **bf16, "batch": 2, "low": 500, "high": 1500, "steps": 8, **prompt},
        {"name": "zabunex 4 requests", "model": "zabunex", "size": "medium", **bf16, "batch": 4, "low": 130, "high": 901, "steps": 16, **prompt},
    ]


def _between(rng, low, high):
    """A whole number between the two, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    model = rng.choice(("llama", "llama", "llama", "fomatar", "zulozen", "kizezen", "ramopel", "zabunex"))
    if model == "llama" and rng.random() < 0.6:                             # the next token of 1 to 64 sequences
        batch = _between(rng, 1, 64)
        high = _between(rng, 32, min(4000, 70000 // batch))
        return {"model": model, "size": rng.choice(("1b", "1b", "medium", "wide")), "dtype": "bfloat16", "batch": batch,
                "low": rng.randint(max(1, high // 8), high), "high": high, "steps": rng.choice((1, 1, 2, 4)), "begin": "cache", "kept": 0}
    if model == "llama":
        dtype = rng.choice(("bfloat16", "bfloat16", "float32"))
        batch = _between(rng, 1, 16 if dtype == "bfloat16" else 4)
        high = _between(rng, 16, min(4000, (12000 if dtype == "bfloat16" else 600) // batch))
        return {"model": model, "size": "1b" if dtype == "float32" else rng.choice(("1b", "medium", "wide")), "dtype": dtype, "batch": batch,
                "low": rng.randint(max(1, high // 8), high), "high": high, "steps": rng.choice((0, 0, 8)), "begin": "prompt", "kept": 1}
    batch = _between(rng, 1, 8)
    high = _between(rng, 16, min(3000, 4000 // batch))
    return {"model": model, "size": "small" if model == "ramopel" else rng.choice(("small", "medium")), "dtype": "bfloat16", "batch": batch,
            "low": rng.randint(max(1, high // 4), high), "high": high, "steps": rng.choice((0, 4, 8, 16)), "begin": "prompt", "kept": 1}


# ---- the calls --------------------------------------------------------------------------------------------------
def _config(case):
    if case["model"] == "llama":
        return benchmark.config_for(2) if case["size"] == "1b" else benchmark.llama_config_like(case["size"])
    if case["model"] == "zulozen":
        return benchmark.zulozen_config_like_kizezen(case["size"])
    return getattr(benchmark, case["model"] + "_config_for")(case["size"])


def _lengths(case):
    n, low, high = case["batch"], min(case["low"], case["high"]), case["high"]
    spread = [low + (high - low) * i // max(n - 1, 1) for i in range(n)] if n > 1 else [high]
    return spread[::2] + spread[1::2][::-1]                                   # neither sorted nor by turns


def _vocab(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def _tokens(case, seed):
    """(each sequence's prompt, the tokens of the single-token steps [steps][sequence])"""
    rng = np.random.default_rng([int(seed), 11])
    vocab = _vocab(_config(case))
    return ([rng.integers(0, vocab, size=n).tolist() for n in _lengths(case)],
            rng.integers(0, vocab, size=(case["steps"], case["batch"])).tolist())


_kept = {}                                   # the one model that cases are asking for


def _model(case):
    key = (case["model"], case["size"], case["dtype"])
    if key not in _kept:
        _kept.clear()
        _kept[key] = camelid_b200.from_random(_config(case), seed=WEIGHTS_SEED, dtype=case["dtype"])
    return _kept[key]


def _wanted(case, n):
    return list(range(max(0, n - case["kept"]), n))


def prepare(case, seed):
    lm = _model(case)
    prompts, fed = _tokens(case, seed)
    cache = lm.new_cache(sum((len(p) + case["steps"] + 63) // 64 * 64 for p in prompts), max_slots=len(prompts))
    state = {"case": case, "lm": lm, "cache": cache, "prompts": prompts, "fed": fed}
    if case["begin"] == "cache":
        state["slots"] = [cache.alloc_slot() for _ in prompts]
        for s, p in zip(state["slots"], prompts):                             # one at a time: a small workspace
            lm.step(cache, [StepEntry(s, p, [])])
        lm.model.drop_graphs(cache)
    return state


def run(state):
    case, lm, cache, prompts = state["case"], state["lm"], state["cache"], state["prompts"]
    out = {}
    if case["begin"] == "cache":
        slots = state["slots"]
    else:
        slots = [cache.alloc_slot() for _ in prompts]
        out["prompts"] = lm.step(cache, [StepEntry(s, p, _wanted(case, len(p))) for s, p in zip(slots, prompts)])
    if state["fed"]:
        # a step's logits lie in a buffer that the next step writes
        out["steps"] = torch.stack([lm.step(cache, [StepEntry(s, [t], [0]) for s, t in zip(slots, row)]).clone() for row in state["fed"]])
    for s, p in zip(slots, prompts):
        if case["begin"] == "cache":
            cache.truncate(s, len(p))
        else:
            cache.free_slot(s)
    return out


def tolerance(case):
    # float32: 8e-6 off the 64-bit logits as measured, four times that. bfloat16: every kernel rounds the rows it hands on
    # (one part in 256), which after 16 layers leaves 0.018 against the 64-bit logits and 0.016 between two settings of
    # the kernels (the 1B shape; 0.005 to 0.014 for the others)
    return {"rel": 4e-5} if case["dtype"] == "float32" else {"rel": 3e-2}


# ---- what a pass cannot do without ------------------------------------------------------------------------------
def _specs(case):
    return DecoderModel.from_config(_config(case), dtype=case["dtype"], device="cpu").tensor_specs()


def _layers(cfg):
    """Per layer and attention or recurrence in it: (kind, query heads, channels of cached rows per position, channels
    multiplied per head and pair of positions, what limits the keys, elements of the state)."""
    if "layers" not in cfg:
        D = cfg["head_dim"]
        return [("keys", cfg["num_attention_heads"], 2 * cfg["num_key_value_heads"] * D, 2 * D, None, 0)] * cfg["num_hidden_layers"]
    out = []
    for L in cfg["layers"]:
        parts = [L["mixer"]] if "left" not in L["mixer"] else [L["mixer"]["left"], L["mixer"]["right"]]
        for m in parts:
            H, D = m["heads"], m.get("dim", m.get("state"))
            Dv = m.get("vdim", D)
            if "kv_rank" in m:
                out.append(("keys", H, 0 if m.get("kv_from") is not None else m["kv_rank"] + m["rot_dim"], D + m["rot_dim"] + Dv, m.get("mask"), 0))
            elif L["type"] in ("attention",) or m is L["mixer"].get("left"):
                out.append(("keys", H, m["kv_heads"] * (D + Dv), D + Dv, m.get("mask"), 0))
            else:
                out.append(("state", H, 0, 0, None, H * D * Dv))
    return out


def _seen(position, mask, blocks):
    if not mask:
        return position + 1
    if blocks:
        return position % mask["size"] + 1
    return min(position + 1, mask["size"] + mask.get("keep_first", 0))


def work(case):
    cfg, elem = _config(case), 2 if case["dtype"] == "bfloat16" else 4
    matrices = experts = head = 0
    for name, spec in _specs(case).items():
        n = math.prod(spec.shape)
        if name in ("head", "lm_head.weight") or (name == "model.embed_tokens.weight" and cfg.get("tie_word_embeddings")):
            head = n
        elif len(spec.shape) == 2 and not name.endswith(("conv", ".rel")) and name not in ("embed", "bigram", "model.embed_tokens.weight"):
            if re.search(r"\.e\d+\.", name):
                experts += n
            else:
                matrices += n
    routers = [L["mlp"]["router"] for L in cfg.get("layers", []) if (L.get("mlp") or {}).get("kind") == "moe"]
    share = routers[0]["top"] / routers[0]["experts"] if routers else 0.0
    blocks = case["model"] in ("zulozen", "zabunex")
    lengths = _lengths(case)
    steps = [] if case["begin"] == "cache" else [[(0, n) for n in lengths]]
    steps += [[(n + i, 1) for n in lengths] for i in range(case["steps"])]
    total = flops = 0.0
    for step in steps:
        rows, wanted = sum(n for _, n in step), sum(min(n, max(1, case["kept"])) for _, n in step)
        total += elem * (matrices + head + experts * (1.0 - (1.0 - share) ** rows)) + 4 * wanted * _vocab(cfg)
        flops += 2.0 * rows * (matrices + experts * share) + 2.0 * wanted * head
        for kind, H, cached, per_pair, mask, state in _layers(cfg):
            for start, n in step:
                if kind == "keys":
                    pairs = sum(_seen(start + i, mask, blocks) for i in range(n))
                    total += elem * cached * (n + (_seen(start, mask, blocks) if start else 0))
                    flops += 2.0 * pairs * H * per_pair
                else:
                    total += 8 * state
                    flops += 6.0 * n * state
    return {"bytes": total, "flops": flops}


# ---- the same logits in 64 bits ---------------------------------------------------------------------------------
class _Weights:
    """The model's tensors by name, each drawn when it is asked for, in 64 bits."""

    def __init__(self, case):
        self.specs, self.dtype = _specs(case), torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32

    def __call__(self, name):
        return random_tensor(name, self.specs[name], WEIGHTS_SEED, self.dtype, "cuda").to(F64)

    def rows(self, name, index):
        return random_tensor(name, self.specs[name], WEIGHTS_SEED, self.dtype, "cuda")[index].to(F64)

    def under(self, prefix):
        return lambda name: self(prefix + name)


def _norm(x, w=None, eps=1e-6):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _each(spans, f, *rows):
    """f on every sequence's part of the rows."""
    return torch.cat([f(*(r[a:b] for r in rows)) for a, b in spans])


def _distance(n):
    i = torch.arange(n, device="cuda")
    return i[:, None] - i[None, :]


def _visible(n, mask, blocks=False):
    d = _distance(n)
    see = d >= 0
    if mask and blocks:
        b = torch.arange(n, device="cuda") // mask["size"]
        see &= b[:, None] == b[None, :]
    elif mask:
        see &= (d < mask["size"]) | (torch.arange(n, device="cuda") < mask.get("keep_first", 0))
    return see


def _attend(q, k, v, scale, see, add=None, sink=None):
    """q [n, H, D], k [n, G, D], v [n, G, Dv] -> [n, H, Dv], head by head; ``sink`` [H]: logs of one more term each."""
    out, per = [], q.shape[1] // k.shape[1]
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // per].T) * scale
        if add is not None:
            s = s + add(h)
        s = s.masked_fill(~see, -math.inf)
        z = torch.logsumexp(s, -1, keepdim=True)
        if sink is not None:
            z = torch.logaddexp(z, sink[h])
        out.append(torch.exp(s - z) @ v[:, h // per])
    return torch.stack(out, 1)


def _turn(x, dims, freq, amp=1.0, pairs=False):
    """x [n, heads, channels]: the first ``dims`` channels turned by position * freq."""
    ang = torch.arange(x.shape[0], device="cuda", dtype=F64)[:, None, None] * torch.as_tensor(freq, dtype=F64, device="cuda")
    c, s, out = amp * torch.cos(ang), amp * torch.sin(ang), x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, dims // 2), slice(dims // 2, dims))
    out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return out


def _frequencies(dims, base, scaling=None):
    """(frequencies, amplitude) under no scaling, one factor, scaling by bands or along a ramp."""
    f = np.float64(base) ** (-2.0 * np.arange(dims // 2) / dims)
    if not scaling:
        return f, 1.0
    if "fast" in scaling:
        where = [dims * math.log(scaling["original"] / (2.0 * math.pi * scaling[t])) / (2.0 * math.log(base)) for t in ("fast", "slow")]
        lo, hi = max(math.floor(where[0]), 0), min(math.ceil(where[1]), dims - 1)
        ramp = np.clip((np.arange(dims // 2) - lo) / max(hi - lo, 0.001), 0.0, 1.0)
        return f / scaling["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(scaling["factor"]) + 1.0
    if "high" not in scaling:
        return f / scaling["factor"], 1.0
    turns = scaling["original"] * f / (2.0 * math.pi)                         # within the original length
    s = np.clip((turns - scaling["low"]) / (scaling["high"] - scaling["low"]), 0.0, 1.0)
    return (1.0 - s) * f / scaling["factor"] + s * f, 1.0


def _conv(x, w, bias=0.0):
    taps = w.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(padded[j:j + x.shape[0]] * w[:, j] for j in range(taps)) + bias


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _recur(r, k, v, decay, remove=None, u=None):
    """Per head S <- decay * S - remove (u^T S) + k v^T, out = S^T r, token by token: all [n, H, D] but v [n, H, Dv];
    decay [n, H, D or 1]."""
    S, out = r.new_zeros(r.shape[1], r.shape[2], v.shape[2]), torch.empty_like(v)
    for t in range(r.shape[0]):
        if remove is None:
            S = decay[t].unsqueeze(-1) * S
        else:
            S = decay[t].unsqueeze(-1) * S - remove[t].unsqueeze(-1) * (u[t].unsqueeze(1) @ S)
        S = torch.baddbmm(S, k[t].unsqueeze(-1), v[t].unsqueeze(1))
        out[t] = (r[t].unsqueeze(1) @ S).squeeze(1)
    return out


def _delta(q, k, v, beta, decay):
    """The gated delta rule S <- D S + k beta (v - (D S)^T k)^T as the removal of beta k of what k D finds."""
    share = v.shape[1] // q.shape[1]
    q, k = q.repeat_interleave(share, 1), k.repeat_interleave(share, 1)
    return _recur(q, k * beta.unsqueeze(-1), v, decay, k * beta.unsqueeze(-1), k * decay)


def _memory(q, k, v, gi, gf):
    """The matrix memory with exponential gates and a running maximum that starts at zero."""
    S, m = q.new_zeros(q.shape[1], q.shape[2], v.shape[2]), q.new_zeros(q.shape[1])
    n, out = q.new_zeros(q.shape[1], q.shape[2]), torch.empty_like(v)
    for t in range(q.shape[0]):
        new = torch.maximum(gf[t] + m, gi[t])
        a, b, m = torch.exp(gf[t] + m - new)[:, None], torch.exp(gi[t] - new)[:, None], new
        S = torch.baddbmm(a.unsqueeze(-1) * S, (b * k[t]).unsqueeze(-1), v[t].unsqueeze(1))
        n = a * n + b * k[t]
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        out[t] = (q[t].unsqueeze(1) @ S).squeeze(1) / den[:, None]
    return out


def _silu(z):
    return z * torch.sigmoid(z)


def _clamped(h, w, name, limit):
    g, u = (h @ w(name + ".gate").T).clamp(max=limit), (h @ w(name + ".up").T).clamp(-limit, limit)
    return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(name + ".down").T


def _experts(h, chosen, weights, count, expert):
    """Sum of the chosen experts; ``expert(e, rows, their weights)``."""
    out = torch.zeros_like(h)
    for e in range(count):
        row, place = torch.nonzero(chosen == e, as_tuple=True)
        if len(row):
            out.index_add_(0, row, expert(e, h[row], weights[row, place].unsqueeze(1)))
    return out


def _llama(case, cfg, w, ids, spans):
    H, G, D, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    sc = cfg["rope_scaling"]
    bands = {"factor": sc["factor"], "low": sc["low_freq_factor"], "high": sc["high_freq_factor"], "original": sc["original_max_position_embeddings"]} if sc else None
    freq, _ = _frequencies(D, cfg["rope_theta"], bands)
    x = w.rows("model.embed_tokens.weight", ids)
    for i in range(cfg["num_hidden_layers"]):
        t = w.under(f"model.layers.{i}.")
        h = _norm(x, t("input_layernorm.weight"), eps)

        def attention(q, k, v):
            n = q.shape[0]
            q, k = _turn(q.reshape(n, H, D), D, freq), _turn(k.reshape(n, G, D), D, freq)
            return _attend(q, k, v.reshape(n, G, D), D ** -0.5, _visible(n, None)).reshape(n, -1)
        y = _each(spans, attention, *(h @ t(f"self_attn.{c}_proj.weight").T for c in "qkv"))
        x = x + y @ t("self_attn.o_proj.weight").T
        h = _norm(x, t("post_attention_layernorm.weight"), eps)
        x = x + (_silu(h @ t("mlp.gate_proj.weight").T) * (h @ t("mlp.up_proj.weight").T)) @ t("mlp.down_proj.weight").T
    return _norm(x, w("model.norm.weight"), eps), "model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"


def _fomatar(case, cfg, w, ids, spans):
    eps, bg = cfg["norm"]["eps"], cfg["embedding"]["bigram"]

    def bigram(t):
        return torch.cat([t.new_full((1,), bg["buckets"]), (t[:-1] * bg["mul_prev"] + t[1:] * bg["mul_cur"]) % bg["buckets"]])
    x = w.rows("embed", ids) + w.rows("bigram", _each(spans, bigram, ids))
    for i, L in enumerate(cfg["layers"]):
        p = w.under(f"l{i}.")
        shift = p("shift")
        h = _each(spans, lambda r: r + (torch.cat([torch.zeros_like(r[:1]), r[:-1]]) - r) * shift, _norm(x, p("norm1"), eps))
        if L["type"] == "parallel":
            t, m = w.under(f"l{i}.mix.left."), L["mixer"]["left"]
            H, G, D, Dv, r1, r2 = m["heads"], m["kv_heads"], m["dim"], m["vdim"], t("r1"), t("r2")

            def attention(q, k, v):
                n = q.shape[0]
                far = _distance(n).clamp(min=0).to(F64)
                return _attend(q, k, v, m["scale"], _visible(n, m["mask"]), add=lambda hd: -r1[hd] * torch.log1p(r2[hd] * far)).reshape(n, -1)
            y = _each(spans, attention, _norm((h @ t("q").T).view(-1, H, D), t("q.norm"), eps),
                      _norm((h @ t("k").T).view(-1, G, D), t("k.norm"), eps), (h @ t("v").T).view(-1, G, Dv))
            left = _norm((y * torch.sigmoid(h @ t("g").T)) @ t("o").T, t("out"), eps)
            t, m = w.under(f"l{i}.mix.right."), L["mixer"]["right"]
            H, D, Dv, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
            gi = cap * torch.tanh((h @ t("i").T + t("i.b")) / cap)
            gf = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ t("f").T + t("f.b")) / cap))
            y = _each(spans, _memory, (h @ t("q").T).view(-1, H, D) * D ** -0.5, (h @ t("k").T).view(-1, H, D), (h @ t("v").T).view(-1, H, Dv), gi, gf)
            y = _norm(y, None, eps).reshape(-1, H * Dv) * t("norm")
            x = x + 0.5 * (left + _norm((y * torch.sigmoid(h @ t("g").T)) @ t("o").T, t("out"), eps))
        else:
            t, m = w.under(f"l{i}.mix."), L["mixer"]
            H, G, D, Dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            q, k, v = (_silu(_each(spans, lambda r, taps=t(c + ".conv"): _conv(r, taps), h @ t(c).T)) for c in "qkv")
            rate = torch.nn.functional.softplus((h @ t("a1").T) @ t("a2").T + t("dt_bias")).view(-1, H, D)
            y = _each(spans, _delta, _unit(q.view(-1, G, D)) * D ** -0.5, _unit(k.view(-1, G, D)), v.view(-1, H, Dv),
                      torch.sigmoid(h @ t("b").T), torch.exp(-torch.exp(t("A_log"))[:, None] * rate))
            y = _norm(y, t("norm"), eps).reshape(-1, H * Dv) * torch.sigmoid((h @ t("g1").T) @ t("g2").T)
            x = x + y @ t("o").T
        if L.get("mlp"):
            h = _norm(x, p("norm2"), eps)
            x = x + torch.nn.functional.gelu(h @ p("mlp.up").T, approximate="tanh") @ p("mlp.down").T
    return _norm(x, w("final.norm"), eps), "head"


def _zulozen(case, cfg, w, ids, spans):
    eps, x = cfg["norm"]["eps"], w.rows("embed", ids)
    for i, L in enumerate(cfg["layers"]):
        p, t, m = w.under(f"l{i}."), w.under(f"l{i}.mix."), L["mixer"]
        H, G, D, Dv, rot = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["rot"]
        freq, _ = _frequencies(rot["dims"], rot["base"])
        h = _norm(x, p("norm1"), eps)
        sink = t("sink")

        def attention(q, k, v):
            n = q.shape[0]
            q, k = (_turn(u.reshape(n, -1, D), rot["dims"], freq, pairs=True) for u in (q, k))
            return _attend(q, k, v.reshape(n, G, Dv), m["scale"], _visible(n, m["mask"], True), sink=sink)
        y = _each(spans, attention, _norm(h @ t("q").T, t("q.norm"), eps), _norm(h @ t("k").T, t("k.norm"), eps), h @ t("v").T)
        y = (y * torch.sigmoid(h @ t("g").T).unsqueeze(-1)).reshape(-1, H * Dv) @ t("o").T
        x = x + cfg["residual_mult"] * _norm(y, p("norm1b"), eps)
        y = torch.relu(_norm(x, p("norm2"), eps) @ p("mlp.up").T + p("mlp.up.b")) ** 2 @ p("mlp.down").T + p("mlp.down.b")
        x = x + cfg["residual_mult"] * _norm(y, p("norm2b"), eps)
    return _norm(x, w("final.norm"), eps), "head"


def _latent(q, c, k_turned, t, m, freq, amp, sink):
    """One sequence: query rows, normed latent rows and turned key rows -> [n, H, Dv]."""
    n, H, D, R = q.shape[0], m["heads"], m["dim"], m["rot_dim"]
    q = q.reshape(n, H, D + R)
    q = torch.cat([q[..., :D], _turn(q[..., D:], R, freq, amp, pairs=True)], -1)
    k = torch.cat([(c @ t("uk").T).view(n, H, D), _turn(k_turned.unsqueeze(1), R, freq, amp, pairs=True).expand(n, H, R)], -1)
    return _attend(q, k, (c @ t("uv").T).view(n, H, -1), m["scale"], _visible(n, m.get("mask")), sink=sink)


def _kizezen(case, cfg, w, ids, spans):
    eps, x = cfg["norm"]["eps"], w.rows("embed", ids) * cfg["embedding"]["scale"]
    for i, L in enumerate(cfg["layers"]):
        p, t, m = w.under(f"l{i}."), w.under(f"l{i}.mix."), L["mixer"]
        H, D, Dv, rot = m["heads"], m["dim"], m["vdim"], m["rot"]
        freq, amp = _frequencies(rot["dims"], rot["base"], rot.get("scaling"))
        h = _norm(x, p("norm1"), eps)
        if L["type"] == "retention":
            decay = torch.tensor(m["decay"], dtype=F64, device="cuda").view(1, H, 1)

            def retention(q, k, v):
                n = q.shape[0]
                q, k = (_turn(u.reshape(n, H, D), rot["dims"], freq) for u in (q, k))
                return _recur(q, k * D ** -0.5, v.reshape(n, H, Dv), decay.expand(n, H, 1))
            y = _norm(_each(spans, retention, *(h @ t(c).T for c in "qkv")), None, eps).reshape(-1, H * Dv) * _silu(h @ t("g").T)
        elif L["type"] == "attention":
            G, sink = m["kv_heads"], t("sink")

            def attention(q, k, v):
                n = q.shape[0]
                q, k = _turn(q.reshape(n, H, D), rot["dims"], freq), _turn(k.reshape(n, G, D), rot["dims"], freq)
                return _attend(q, k, v.reshape(n, G, Dv), m["scale"], _visible(n, m["mask"]), sink=sink)
            y = _each(spans, attention, _norm(h @ t("q").T + t("q.b"), t("q.norm"), eps), _norm(h @ t("k").T + t("k.b"), t("k.norm"), eps), h @ t("v").T + t("v.b"))
        else:
            down, C, sink = h @ t("dkv").T, m["kv_rank"], t("sink")
            y = _each(spans, lambda q, c, kt: _latent(q, c, kt, t, m, freq, amp, sink), h @ t("q").T, _norm(down[:, :C], t("dkv.norm"), eps), down[:, C:])
        if L["type"] != "retention":
            y = (y * torch.sigmoid(h @ t("g").T).unsqueeze(-1)).reshape(-1, H * Dv)
        x = x + y @ t("o").T
        x = x + torch.nn.functional.gelu(_norm(x, p("norm2"), eps) @ p("mlp.up").T) @ p("mlp.down").T
    return _norm(x, w("final.norm"), eps) * cfg["logit_scale"], "head"


def _ramopel(case, cfg, w, ids, spans):
    eps, x, latents = cfg["norm"]["eps"], w.rows("embed", ids) * cfg["embedding"]["scale"], {}
    for i, L in enumerate(cfg["layers"]):
        p, t, m, f = w.under(f"l{i}."), w.under(f"l{i}.mix."), L["mixer"], L["mlp"]
        H, D = m["heads"], m["dim"]
        h = _norm(x, 1.0 + p("norm1"), eps)
        if L["type"] == "latent_attention":
            freq, amp = _frequencies(m["rot_dim"], m["rot"]["base"])
            if m.get("kv_from") is None:
                down = h @ t("dkv").T
                latents[i] = (_norm(down[:, :m["kv_rank"]], t("dkv.norm"), eps), down[:, m["kv_rank"]:])
            q = _norm(h @ t("dq").T, t("dq.norm"), eps) @ t("uq").T
            y = _each(spans, lambda q, c, kt: _latent(q, c, kt, t, m, freq, amp, None), q, *latents[m.get("kv_from", i)]).reshape(-1, H * m["vdim"])
        else:
            r, k, v = ((h @ t(c).T).view(len(h), H, -1) for c in "rkv")
            decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ t("w1").T) @ t("w2").T + t("w0"))).view(k.shape)
            u = _unit(k)
            y = _each(spans, _recur, r, k, v, decay, torch.sigmoid(h @ t("a").T + t("a.b")).view(k.shape) * u, u)
            y = _norm(y, None, eps).reshape(len(h), -1) * t("norm") * torch.sigmoid(h @ t("g").T)
        y = y @ t("o").T
        h, t = _norm(x, 1.0 + p("norm2"), eps), w.under(f"l{i}.mlp.")
        if f["kind"] == "dense":
            z, act = h @ t("up").T, t("act")
            y = y + (act[0] * _norm(z, None, eps) + act[1] * _norm(z ** 2, None, eps) + act[2] * _norm(z ** 3, None, eps) + act[3]) @ t("down").T
        else:
            best = torch.topk(h @ t("router").T + t("router.b"), f["router"]["top"], -1)
            y = y + _experts(h, best.indices, torch.softmax(best.values, -1), f["router"]["experts"],
                             lambda e, rows, share: share * _clamped(rows, t, f"e{e}", f["expert"]["limit"]))
            y = y + torch.sigmoid(h @ t("shared.sg").T) * _clamped(h, t, "shared", f["shared"]["limit"])
        x = x + y
    return _norm(x, 1.0 + w("final.norm"), eps), "head"


def _zabunex(case, cfg, w, ids, spans):
    eps, x = cfg["norm"]["eps"], w.rows("embed", ids)
    for i, L in enumerate(cfg["layers"]):
        p = w.under(f"l{i}.")
        if L["type"] == "attention":
            t, m = w.under(f"l{i}.mix."), L["mixer"]
            H, G, D, rel, half = m["heads"], m["kv_heads"], m["dim"], t("rel"), m["bias_rows"] // 2

            def attention(q, k, v):
                n = q.shape[0]
                far = _distance(n).clamp(min=0)
                row = half + torch.floor(torch.log(far.clamp(min=1).to(F64) / half) / math.log(m["bias_max"] / half) * half).long()
                row = torch.where(far < half, far, row.clamp(max=2 * half - 1))
                grow = 1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((torch.arange(n, device="cuda", dtype=F64) + 1.0) / m["q_temp"]["every"]) + 1.0)
                return _attend(q * grow[:, None, None], k, v, m["scale"], _visible(n, None), add=lambda hd: rel[:, hd][row], sink=rel.new_zeros(H)).reshape(n, -1)
            k = x @ t("k").T
            y = _each(spans, attention, _norm(x @ t("q").T, t("q.norm"), eps).view(-1, H, D), _norm(k, t("k.norm"), eps).view(-1, G, D), k.view(-1, G, D)) @ t("o").T
        else:
            t, m = w.under(f"l{i}.mix.left."), L["mixer"]["left"]
            H, G, D, Dv, rot = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["rot"]
            freq, _ = _frequencies(rot["dims"], rot["base"], rot.get("scaling"))
            q, k, v = (_each(spans, lambda r, taps=t(c + ".conv"): _conv(r, taps), x @ t(c).T) for c in "qkv")

            def blocks(q, k, v):
                n = q.shape[0]
                q, k = _turn(q.reshape(n, H, D), rot["dims"], freq), _turn(k.reshape(n, G, D), rot["dims"], freq)
                return _attend(q, k, v.reshape(n, G, Dv), m["scale"], _visible(n, m["mask"], True)).reshape(n, -1)
            y = L["mixer"]["left_scale"] * (_each(spans, blocks, _norm(q, t("q.norm"), eps), _norm(k, t("k.norm"), eps), v) @ t("o").T)
            t, m = w.under(f"l{i}.mix.right."), L["mixer"]["right"]
            H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            rows, inner = x @ t("in").T, H * P
            z, u, dt = rows[:, :inner], rows[:, inner:2 * inner + 2 * G * N], rows[:, 2 * inner + 2 * G * N:]
            taps, bias = t("conv"), t("conv.b")
            u = _silu(_each(spans, lambda r: _conv(r, taps, bias), u))
            xs, B, C = u[:, :inner].view(-1, H, P), u[:, inner:inner + G * N].view(-1, G, N), u[:, inner + G * N:].view(-1, G, N)
            dt = torch.nn.functional.softplus(dt + t("dt_bias")).unsqueeze(-1)
            B, C = B.repeat_interleave(H // G, 1) * dt, C.repeat_interleave(H // G, 1)
            s = _each(spans, _recur, C, B, xs, torch.exp(-torch.exp(t("A_log"))[:, None] * dt)) + t("D")[:, None] * xs
            s = _norm((s.reshape(-1, inner) * _silu(z)).view(len(x), m["norm_groups"], -1), None, eps).reshape(-1, inner) * t("norm")
            y = y + L["mixer"]["right_scale"] * (s @ t("o").T)
        x = x + _norm(y, p("norm1"), eps)
        x = x + _norm(torch.relu(x @ p("mlp.up").T) ** 2 @ p("mlp.down").T, p("norm2"), eps)
    return _norm(x, w("final.norm"), eps), "head"


@torch.no_grad()
def exact(case, seed):
    cfg, w = _config(case), _Weights(case)
    prompts, fed = _tokens(case, seed)
    whole = [p + [row[i] for row in fed] for i, p in enumerate(prompts)]
    spans, at = [], 0
    for s in whole:
        spans.append((at, at + len(s)))
        at += len(s)
    x, head = globals()["_" + case["model"]](case, cfg, w, torch.tensor([t for s in whole for t in s], device="cuda"), spans)
    matrix, cap, out = w(head).T, cfg.get("logit_softcap"), {}

    def logits(rows):
        z = x[torch.tensor(rows, device="cuda")] @ matrix
        return cap * torch.tanh(z / cap) if cap else z
    if case["begin"] == "prompt":
        out["prompts"] = logits([a + r for (a, _), p in zip(spans, prompts) for r in _wanted(case, len(p))])
    if fed and case["model"] == "ramopel":
        # A router's near-tie that 16 bits break the other way moves one row by a tenth (0.019 in all against 0.006): with
        # a decision per row, layer and step, how far a run is from 64 bits says whether one fell, not how exact it is.
        out["steps"] = None
    elif fed:
        out["steps"] = torch.stack([logits([a + len(p) + t for (a, _), p in zip(spans, prompts)]) for t in range(len(fed))])
    return out

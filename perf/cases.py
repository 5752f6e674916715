"""Workloads of the library as a program meets them, for timing and for comparing results.

A case is a model (one of the registered decoders, random weights at the sizes the benchmark uses), a batch of prompts of unequal
lengths and a number of tokens that every sequence goes on for.  A pass opens the sequences, runs the prompts in one step and then
one step per further token, and returns the float32 logits after the prompt and after every further token (`kind` "score": the
further tokens are given, as when text is scored or a reply is replayed), or runs `Engine.generate` and returns the tokens (`kind`
"generate").  The model and its engine are loaded once and kept, as a serving program keeps them.
"""
import json
import math
import os
import shutil
import tempfile

import numpy as np
import torch

import velomind_b200 as vm

# ------------------------------------------------------------------------------------------------ the models
LLAMA = {"135m": (30, 576, 9, 3, 1536, 100000.0), "360m": (32, 960, 15, 5, 2560, 100000.0), "1.7b": (24, 2048, 32, 32, 8192, 130000.0)}
WIDE = {1024: dict(heads=16, kv=4, q_rank=384, ff=2816, experts=16, expert_ff=512, shared_ff=1024, n=1),
        2048: dict(heads=32, kv=8, q_rank=768, ff=5632, experts=32, expert_ff=1024, shared_ff=2048, n=2)}
FAMILIES = ("kogilix", "semesun", "vozetar", "zabozen", "depunex")
VOCAB, DIM, LATENT = 32000, 64, 128


def config_of(model):
    """config.json of a model by its name: llama-<size>[-untied], or <family>-<width>."""
    family, size = model.split("-")[:2]
    if family == "llama":
        layers, hidden, heads, kv, ff, theta = LLAMA[size]
        return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "vocab_size": 49152, "hidden_size": hidden, "intermediate_size": ff,
                "num_hidden_layers": layers, "num_attention_heads": heads, "num_key_value_heads": kv, "rms_norm_eps": 1e-5, "rope_theta": theta,
                "max_position_embeddings": 8192, "tie_word_embeddings": not model.endswith("-untied"), "hidden_act": "silu"}
    W = int(size)
    z = WIDE[W]
    n = z["n"]
    att = {"heads": z["heads"], "kv_heads": z["kv"], "dim": DIM, "vdim": DIM, "scale": DIM ** -0.5}
    rot = {"base": 10000.0, "dims": DIM}
    pairs = {"buckets": 100003, "mul_prev": 8191, "mul_cur": 31}
    dense = {"kind": "dense", "ff": z["ff"]}
    moe = {"kind": "moe", "expert": {"ff": z["expert_ff"]}, "router": {"experts": z["experts"], "top": 4}}
    grouped = {"kind": "moe", "expert": {"ff": z["expert_ff"]}, "router": {"experts": z["experts"], "top": 4, "groups": {"count": 2, "keep": 1}}}
    ssm = {"heads": 32 * n, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}
    c = {"architecture": family.capitalize(), "vocab": VOCAB, "width": W, "norm": {"eps": 1e-6}}
    if family == "kogilix":
        lat = {"heads": z["heads"], "dim": DIM, "vdim": DIM, "q_rank": z["q_rank"], "kv_rank": LATENT, "scale": DIM ** -0.5}
        lstm = {"heads": 4 * n, "dim": 128, "vdim": 256, "gate_cap": 15.0}
        moe["shared"] = {"ff": z["shared_ff"]}
        layers = [("latent_attention", lat, dense), ("mlstm", lstm, moe), ("latent_attention", dict(lat, kv_from=0), moe), ("mlstm", lstm, moe)]
    elif family == "semesun":
        att.update(bias_max=4096, bias_rows=32, mask={"size": 1024, "keep_first": 4}, v_mix=True)
        grouped["expert"]["limit"] = 7.0
        grouped["router"].update(identity=2, scale=1.0)
        layers = [("attention", att, dense), ("mamba2", ssm, grouped), ("attention", att, grouped), ("mamba2", ssm, grouped)]
    elif family == "vozetar":
        mask = {"size": 1024, "keep_first": 4}
        att["rot"] = rot
        mem = {"heads": 8 * n, "dim": 64, "vdim": 128}
        decay = [1.0 - 2.0 ** (-5 - 5.0 * i / (8 * n - 1)) for i in range(8 * n)]
        par = {"left": dict(att, mask=mask), "left_scale": 1.0, "right": dict(mem, rot=rot, decay=decay), "right_scale": 1.0}
        par2 = {"left": dict(att, mask=mask, conv=4), "right": dict(mem, tau=16.0, decay_rank=32)}
        grouped["shared"] = {"ff": z["shared_ff"]}
        c.update(streams=3, embedding={"bigram": pairs})
        layers = [("attention", dict(att, conv=3), dense), ("parallel", par, grouped), ("parallel_2", par2, dense), ("parallel", par, grouped)]
    elif family == "zabozen":
        lat = {"heads": z["heads"], "dim": DIM, "rot_dim": 32, "vdim": DIM, "kv_rank": LATENT, "scale": (DIM + 32) ** -0.5, "rot": {"base": 10000.0, "dims": 32}}
        delta = {"heads": 8 * n, "kv_heads": 4 * n, "dim": 128, "vdim": 128, "conv": 4}
        c.update(residual_mult=0.8, logit_softcap=25.0)
        layers = [("attention", dict(att, mask={"size": 1024}), dense), ("latent_attention", lat, dense), ("delta", delta, dense),
                  ("attention", dict(att, mask={"size": 1536}, kv_from=0), dense)]
    else:
        scaled = {"base": 500000.0, "dims": DIM, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
        scan = {"inner": 2048 * n, "dt_rank": 64 * n, "state": 16, "conv": 4}
        par = {"left": dict(att, mask={"size": 1024}, rot=scaled), "left_scale": 0.7, "right": scan, "right_scale": 0.7}
        dense["limit"] = 7.0
        c.update(logit_softcap=30.0, token_side={"dim": 128 * n}, embedding={"scale": W ** 0.5, "bigram": pairs})
        layers = [("mamba2", ssm, dense), ("parallel", par, grouped), ("mamba2", ssm, grouped), ("parallel", par, dense)]
    c["layers"] = [{"type": t, "mixer": m, "mlp": f} for t, m, f in layers]
    return c


def _inverse_softplus(x):
    return x + torch.log(-torch.expm1(-x))


def _tensor(name, spec, cfg, g):
    """One weight in float32 on the GPU: the distribution its kind has in use.  Matrices N(0, 0.02)."""
    shape, last = spec["shape"], name.rsplit(".", 1)[-1]

    def normal(std, mean=0.0):
        return torch.randn(shape, generator=g, device="cuda") * std + mean

    def uniform(a, b):
        return torch.rand(shape, generator=g, device="cuda") * (b - a) + a

    if spec["ones"] or last == "D":
        return uniform(0.9, 1.1)
    if last == "A_log":                                           # decay rates from 1 to 16, as state-space models start
        return torch.log(torch.arange(1, shape[1] + 1, device="cuda").float()).expand(shape) + normal(0.05) if len(shape) == 2 else torch.log(uniform(1.0, 16.0))
    if last == "dt_bias" or name.endswith("dt.b"):                # time steps from 0.001 to 0.1
        return _inverse_softplus(torch.exp(uniform(math.log(1e-3), math.log(1e-1))))
    if name.endswith("mix.f.b"):                                  # forget gates that start open
        return uniform(3.0, 6.0)
    if name.endswith("a2.b"):
        return normal(1.0, 1.0)
    if last == "conv":
        return uniform(-0.5, 0.5)
    if last == "vmix":
        return uniform(0.4, 0.6)
    if last in ("sink", "rel"):
        return normal(0.5)
    if ".hc" in name:                                             # copies that start as one stream: read the mean, keep each, add to all
        if last == "mix":
            return torch.eye(shape[0], device="cuda") + normal(0.02)
        return normal(0.02, 1.0 if last == "out" else 1.0 / shape[0])
    if last in ("embed", "bigram") and "architecture" in cfg:
        return normal((0.1 if last == "bigram" else 1.0 / (cfg.get("embedding") or {}).get("scale", 1.0)) if "side" not in name else 1.0)
    return normal(0.02)


def weights_of(model, dtype):
    """name -> tensor on the GPU in the model's dtype, from a fixed seed.  Tokens lie on the side of a router's rows that four experts
    of one half share, so that the choice of experts has clear gaps (as trained routers have) instead of ties."""
    cfg = config_of(model)
    table = vm.weight_table(cfg)
    g = torch.Generator(device="cuda").manual_seed(20240611)
    w = {n: _tensor(n, s, cfg, g) for n, s in sorted(table.items()) if not s["alias_of"]}
    routers = sorted(n for n in w if n.endswith(".router"))
    if routers:
        rows = torch.cat([w[n] for n in routers])
        q = torch.linalg.qr(rows.T)[0].T                          # [all outputs, width], orthonormal
        e = w["embed"] * (cfg.get("embedding") or {}).get("scale", 1.0)
        at = 0
        e = e - (e @ q.T) @ q
        for n in routers:
            E = w[n].shape[0]
            w[n] = 0.75 * q[at:at + E]
            half = torch.randint(0, 2, (e.shape[0], 1), generator=g, device="cuda")
            score = torch.rand((e.shape[0], E), generator=g, device="cuda") + 2.0 * (torch.arange(E, device="cuda") // (E // 2) == half)
            on = torch.zeros_like(score).scatter_(1, score.topk(4, dim=1).indices, 1.0)
            side = (2.0 * on - 1.0) * (3.0 + 0.3 * torch.randn(score.shape, generator=g, device="cuda"))
            e = e + side @ q[at:at + E]
            at += E
        w["embed"] = e / (cfg.get("embedding") or {}).get("scale", 1.0)
    if model.endswith("-untied"):
        # one token clearly leads to the next, as in text that a trained model is sure of: greedy runs then have no ties
        e = torch.randn(w["model.embed_tokens.weight"].shape, generator=g, device="cuda")
        w["model.embed_tokens.weight"] = e
        w["lm_head.weight"] = torch.empty_like(e).index_copy_(0, torch.randperm(e.shape[0], generator=g, device="cuda"), 0.1 * e)
    return {n: t.to(torch.bfloat16 if dtype == "bfloat16" else torch.float32) for n, t in w.items()}


def _write_model(folder, model, dtype):
    w = weights_of(model, dtype)
    header, at = {}, 0
    for n, t in w.items():
        size = t.numel() * t.element_size()
        header[n] = {"dtype": "BF16" if dtype == "bfloat16" else "F32", "shape": list(t.shape), "data_offsets": [at, at + size]}
        at += size
    blob = json.dumps(header).encode()
    blob += b" " * (-len(blob) % 8)
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(config_of(model), f)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(len(blob).to_bytes(8, "little") + blob)
        for t in w.values():
            f.write(t.reshape(-1).view(torch.uint8).cpu().numpy().data)


_loaded = {}


def _engine(model, dtype):
    """The engine of a model, loaded at its first use and kept until another model is asked for."""
    key = (model, dtype)
    if key not in _loaded:
        _loaded.clear()
        torch.cuda.empty_cache()
        folder = tempfile.mkdtemp(prefix="vm_cases_")
        try:
            _write_model(folder, model, dtype)
            torch.cuda.empty_cache()
            _loaded[key] = vm.Engine(vm.load_model(folder, dtype=dtype), max_tokens=65536, max_slots=64)
        finally:
            shutil.rmtree(folder, ignore_errors=True)
    return _loaded[key]


# ------------------------------------------------------------------------------------------------ the cases
def _case(name, model, batch, shortest, longest, more, kind="score", dtype="bfloat16"):
    return {"name": name, "kind": kind, "model": model, "dtype": dtype, "batch": batch, "shortest": shortest, "longest": longest, "more": more}


def listed():
    return [
        # one user, a short question, the first tokens of the reply: latency and launches
        _case("one_short", "llama-135m", 1, 17, 17, 8),
        # the benchmark's decode shape: eight conversations going on together
        _case("eight_decode", "llama-135m", 8, 512, 512, 32),
        # one long prompt, first token of the reply
        _case("one_prompt", "llama-135m", 1, 2048, 2048, 0),
        # the true 32-bit path: checking or comparing a model
        _case("float32", "llama-135m", 4, 33, 190, 4, dtype="float32"),
        # the middle size with a ragged batch of sixteen
        _case("sixteen_ragged", "llama-360m", 16, 64, 1024, 8),
        # the largest size with long contexts: documents and their continuation
        _case("long_contexts", "llama-1.7b", 4, 1000, 3000, 16),
        # the generation loop with the device sampler and its token feedback
        _case("generate", "llama-135m-untied", 16, 40, 300, 24, kind="generate"),
        # the other decoders, each with its mixers, feed-forwards and caches: prompts and some steps behind them
        _case("kogilix", "kogilix-1024", 1, 2048, 2048, 8),
        _case("semesun", "semesun-1024", 8, 130, 509, 8),
        _case("vozetar", "vozetar-1024", 4, 301, 850, 8),
        _case("zabozen", "zabozen-2048", 2, 1400, 2000, 8),
        _case("depunex", "depunex-1024", 8, 512, 512, 8),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """Any model of the list's families and sizes, 1 to 64 sequences, prompts of 1 to 3,000 tokens, up to 24 further tokens."""
    if rng.random() < 0.45:
        model, most = rng.choice([("llama-135m", 8000), ("llama-135m", 8000), ("llama-360m", 6000), ("llama-1.7b", 3000)])
    else:
        model, most = "%s-%d" % (rng.choice(FAMILIES), rng.choice([1024, 2048])), 5000
    dtype, kind = "bfloat16", "score"
    if rng.random() < 0.12 and model.endswith(("135m", "1024")):
        dtype, most = "float32", 500
    elif model == "llama-135m" and rng.random() < 0.2:
        model, kind = "llama-135m-untied", "generate"
    longest = _log_int(rng, 1, min(most, 3000))
    batch = _log_int(rng, 1, max(1, min(64, most // longest)))
    shortest = _log_int(rng, max(1, longest // 16), longest)
    more = rng.choice([0, 1, 4, 8, 16, 24])
    if dtype == "float32":
        more = min(more, 4)
    c = _case("", model, batch, shortest, longest, max(more, 1) if kind == "generate" else more, kind, dtype)
    del c["name"]
    return c


def _lengths(case):
    """The prompts' lengths: from the longest down to the shortest in even strides, in an order that does not run up or down."""
    B, a, b = case["batch"], case["shortest"], case["longest"]
    up = [b - (b - a) * i // max(1, B - 1) for i in range(B)]
    return up[::2] + up[1::2][::-1]


def _vocab(model):
    return 49152 if model.startswith("llama") else VOCAB


def _tokens(case, seed):
    """Prompts (lists of token ids) and the further tokens [more, batch], uniform as no text is at hand."""
    rng = np.random.default_rng(seed)
    V = _vocab(case["model"])
    return [rng.integers(0, V, n).tolist() for n in _lengths(case)], rng.integers(0, V, (case["more"], case["batch"])).tolist()


def prepare(case, seed):
    engine = _engine(case["model"], case["dtype"])
    prompts, further = _tokens(case, seed)
    state = {"kind": case["kind"], "engine": engine, "prompts": prompts, "further": further, "batch": case["batch"]}
    if case["kind"] == "generate":
        params = vm.SamplingParams(temperature=0.0, max_tokens=case["more"] + 1, stop_tokens=())
        state["requests"] = [vm.Request(p, params, i) for i, p in enumerate(prompts)]
    return state


def run(state):
    engine = state["engine"]
    if state["kind"] == "generate":
        results, _ = engine.generate(state["requests"], max_batch=64)
        return np.array([r.tokens for r in results], dtype=np.int32)
    slots = [engine.open() for _ in state["prompts"]]
    try:
        with torch.cuda.stream(engine.stream):
            out = torch.empty((1 + len(state["further"]), state["batch"], engine.vocab), dtype=torch.float32, device="cuda")
            out[0].copy_(engine.step([vm.Entry(s, p, (len(p) - 1,)) for s, p in zip(slots, state["prompts"])], synchronize=False))
            for i, tokens in enumerate(state["further"]):
                out[i + 1].copy_(engine.step([vm.Entry(s, (t,), (0,)) for s, t in zip(slots, tokens)], synchronize=False))
        engine.synchronize()
    finally:
        for s in slots:
            engine.close(s)
    return out


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Bytes: per step every weight that the step's tokens need once (experts: as many as the pairs can reach), the cached keys and
    values (or the states) it reads and writes, the logits.  Operations: two per weight and token, and the attention's products."""
    cfg, B, size = config_of(case["model"]), case["batch"], 2 if case["dtype"] == "bfloat16" else 4
    table = vm.weight_table(cfg)
    dense = expert = rows = 0
    for n, s in table.items():
        k = int(np.prod(s["shape"]))
        if s["alias_of"] or n.endswith(("embed", "embed_tokens.weight", "bigram", "head", "lm_head.weight")):
            continue
        if ".mlp.e" in n:
            expert += k
        else:
            dense += k
    hidden = cfg.get("hidden_size") or cfg["width"]
    head = _vocab(case["model"]) * hidden
    if "layers" in cfg:
        heads, E, top = WIDE[hidden]["heads"], WIDE[hidden]["experts"], 4
        attn = []                                                 # (window, query and value width of all heads, cached values per token)
        state = 0
        for layer in cfg["layers"]:
            t, m = layer["type"], layer["mixer"]
            for p in ([m] if "left" not in m else [m["left"], m["right"]]):
                if "kv_rank" in p:
                    attn.append((1 << 30, 2 * heads * DIM, LATENT + p.get("rot_dim", 0)))
                elif "scale" in p:
                    attn.append((p["mask"]["size"] if p.get("mask") else 1 << 30, 2 * heads * DIM, 2 * p["kv_heads"] * DIM))
                elif "inner" in p:
                    state += p["inner"] * p["state"]
                else:
                    state += p["heads"] * p["vdim"] * p.get("state", p.get("dim"))
    else:
        E = top = 1
        attn = [(1 << 30, 2 * hidden, 2 * cfg["num_key_value_heads"] * (hidden // cfg["num_attention_heads"]))] * cfg["num_hidden_layers"]
        state = 0
    lengths = _lengths(case)
    total = flops = 0.0
    for step in range(1 + case["more"]):
        T = sum(lengths) if step == 0 else B
        total += size * (dense + head + expert * min(E, T * top) / E + T * hidden)
        flops += 2.0 * T * (dense + expert * top / E + 3 * state) + 2.0 * B * head
        for n in lengths:
            for window, width, cached in attn:
                if step == 0:
                    w = min(window, n)
                    flops += 2.0 * width * (w * (w + 1) / 2 + (n - w) * w)
                    total += size * n * cached
                else:
                    w = min(window, n + step)
                    flops += 2.0 * width * w
                    total += size * cached * w
        total += 4.0 * state * B * (1 if step == 0 else 2)
        total += 4.0 * B * _vocab(case["model"])
    return {"bytes": total, "flops": flops}


def tolerance(case):
    if case["kind"] == "generate":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 4e-4}
    # measured against 64 bits: 0.002 to 0.007, and 0.02 for the 1.7B sizes
    return {"rel": 0.03, "max": 0.5} if "1.7b" in case["model"] else {"rel": 0.02, "max": 0.3}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _lin(x, w, b=None):
    y = x @ w.T
    return y if b is None else y + b


def _unit(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _norm(x, w, eps):
    return _unit(x, eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.logaddexp(x, torch.zeros_like(x))


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _under(w, prefix):
    return {k[len(prefix):]: v for k, v in w.items() if k.startswith(prefix)}


def _heads(x, n):
    return x.reshape(*x.shape[:-1], n, -1)


def _frequencies(rot):
    f = float(rot["base"]) ** (-2.0 * torch.arange(rot["dims"] // 2, dtype=torch.float64, device="cuda") / rot["dims"])
    s = rot.get("scaling")
    if s:
        share = ((s["original"] * f / (2.0 * math.pi) - s["low"]) / (s["high"] - s["low"])).clamp(0.0, 1.0)
        f = (1.0 - share) * f / s["factor"] + share * f
    return f


def _turn(x, rot, pairing="half"):
    """Rotary positions along dimension 1 of x [B, n, heads, d] on the first rot["dims"] values."""
    dims = rot["dims"]
    a = torch.arange(x.shape[1], dtype=torch.float64, device="cuda")[:, None] * _frequencies(rot)
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    y = x.clone()
    i = torch.arange(dims // 2, device="cuda")
    i, j = (2 * i, 2 * i + 1) if pairing == "interleaved" else (i, i + dims // 2)
    y[..., i] = x[..., i] * c - x[..., j] * s
    y[..., j] = x[..., j] * c + x[..., i] * s
    return y


def _attend(q, k, v, scale, window=None, keep_first=0, chunk=None, bias=None, sink=None):
    """q [B, n, H, d], k and v [B, n, G, ...]; `bias` [H, n] by distance; one sequence and one key head at a time."""
    B, n, H, _ = q.shape
    G = k.shape[2]
    i, j = torch.arange(n, device="cuda")[:, None], torch.arange(n, device="cuda")[None]
    seen = j <= i
    if window:
        seen = seen & ((i - j < window) | (j < keep_first))
    if chunk:
        seen = seen & (i // chunk == j // chunk)
    far = (i - j).clamp(min=0)
    out = torch.empty((B, n, H, v.shape[-1]), dtype=torch.float64, device="cuda")
    for b in range(B):
        for h in range(H):
            g = h // (H // G)
            s = (q[b, :, h] @ k[b, :, g].T) * scale
            if bias is not None:
                s = s + bias[h][far]
            s = s.masked_fill(~seen, -math.inf)
            top = s.max(-1, keepdim=True).values
            if sink is not None:
                top = top.clamp(min=float(sink[h]))
            e = torch.exp(s - top)
            total = e.sum(-1, keepdim=True)
            if sink is not None:
                total = total + torch.exp(sink[h] - top)
            out[b, :, h] = (e @ v[b, :, g]) / total
    return out


def _conv(u, taps):
    k = taps.shape[1]
    y = torch.zeros_like(u)
    for back in range(min(k, u.shape[1])):
        y[:, back:] += taps[:, k - 1 - back] * u[:, :u.shape[1] - back]
    return y


def _memory(q, k, v, decay, u=None):
    """S <- decay S + k v^T (with `u` = write strengths: the delta rule), o = S^T q.  q, k, decay [B, n, H, d], v [B, n, H, dv]."""
    S = torch.zeros((*q.shape[:1], *q.shape[2:], v.shape[-1]), dtype=torch.float64, device="cuda")
    o = torch.empty_like(v)
    for t in range(q.shape[1]):
        S = S * decay[:, t, :, :, None]
        val = v[:, t]
        if u is not None:
            val = u[:, t, :, None] * (val - torch.einsum("bhdv,bhd->bhv", S, k[:, t]))
        S = S + k[:, t, :, :, None] * val[:, :, None]
        o[:, t] = torch.einsum("bhdv,bhd->bhv", S, q[:, t])
    return o


# ---- mixers: x [B, n, width] -> [B, n, width]
def _latent(x, w, m, eps, kept, i):
    H, d, r, rank = m["heads"], m["dim"], m.get("rot_dim", 0), m["kv_rank"]
    src = i if m.get("kv_from") is None else m["kv_from"]
    if src == i:
        low = _lin(x, w["dkv"])
        kept[i] = _norm(low[..., :rank], w["dkv.norm"], eps), low[..., None, rank:]
    c, kr = kept[src]
    q = _heads(_lin(_norm(_lin(x, w["dq"]), w["dq.norm"], eps), w["uq"]) if "dq" in w else _lin(x, w["q"]), H)
    k = _heads(_lin(c, w["uk"]), H)
    if r:
        q = torch.cat([q[..., :d], _turn(q[..., d:], m["rot"])], -1)
        k = torch.cat([k, _turn(kr, m["rot"]).expand(*k.shape[:3], r)], -1)
    o = _attend(q, k, _heads(_lin(c, w["uv"]), H), m["scale"])
    if "g" in w:
        o = o * torch.sigmoid(_lin(x, w["g"]))[..., None]
    return _lin(o.flatten(2), w["o"])


def _mlstm(x, w, m, eps):
    H, d, cap = m["heads"], m["dim"], m["gate_cap"]
    q, k, v = _heads(_lin(x, w["q"]), H) / math.sqrt(d), _heads(_lin(x, w["k"]), H), _heads(_lin(x, w["v"]), H)
    gi = cap * torch.tanh(_lin(x, w["i"], w["i.b"]) / cap)
    gf = -_softplus(-cap * torch.tanh(_lin(x, w["f"], w["f.b"]) / cap))
    S = torch.zeros((x.shape[0], H, d, v.shape[-1]), dtype=torch.float64, device="cuda")
    z = torch.zeros_like(S[..., 0])
    top = torch.zeros_like(z[..., 0])
    o = torch.empty_like(v)
    for t in range(x.shape[1]):
        new = torch.maximum(gf[:, t] + top, gi[:, t])
        keep, take = torch.exp(gf[:, t] + top - new)[..., None], torch.exp(gi[:, t] - new)[..., None]
        S = keep[..., None] * S + (take * k[:, t])[..., None] * v[:, t, :, None]
        z, top = keep * z + take * k[:, t], new
        low = torch.maximum((z * q[:, t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        o[:, t] = torch.einsum("bhdv,bhd->bhv", S, q[:, t]) / low[..., None]
    return _lin(_unit(o, eps).flatten(2) * w["norm"] * torch.sigmoid(_lin(x, w["g"])), w["o"])


def _bucket(n, rows, far):
    half = rows // 2
    return n if n < half else min(rows - 1, half + int(math.floor(math.log(n / half) / math.log(far / half) * (rows - half))))


def _biased(x, w, m, eps, kept):
    H, G, n = m["heads"], m["kv_heads"], x.shape[1]
    q, k, v = _norm(_heads(_lin(x, w["q"]), H), w["q.norm"], eps), _norm(_heads(_lin(x, w["k"]), G), w["k.norm"], eps), _heads(_lin(x, w["v"]), G)
    first = kept.setdefault("values", v)
    if first is not v:
        v = (1.0 - w["vmix"]) * v + w["vmix"] * first
    rows = torch.tensor([_bucket(i, m["bias_rows"], m["bias_max"]) for i in range(n)], device="cuda")
    return _lin(_attend(q, k, v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"], bias=w["rel"].T[:, rows]).flatten(2), w["o"])


def _mamba2(x, w, m, eps):
    H, P, N = m["heads"], m["vdim"], m["state"]
    inner = H * P
    p = _lin(x, w["in"])
    z, u, dt = p[..., :inner], _silu(_conv(p[..., inner:2 * inner + 2 * N], w["conv"]) + w["conv.b"]), _softplus(p[..., 2 * inner + 2 * N:] + w["dt_bias"])
    xs, Bm, Cm = _heads(u[..., :inner], H), u[..., inner:inner + N], u[..., inner + N:]
    keep = torch.exp(-torch.exp(w["A_log"]) * dt)
    S = torch.zeros((x.shape[0], H, N, P), dtype=torch.float64, device="cuda")
    y = torch.empty_like(xs)
    for t in range(x.shape[1]):
        S = keep[:, t, :, None, None] * S + Bm[:, t, None, :, None] * (dt[:, t, :, None] * xs[:, t])[:, :, None]
        y[:, t] = torch.einsum("bhnp,bn->bhp", S, Cm[:, t])
    y = (y + w["D"][:, None] * xs).flatten(2) * _silu(z)
    return _lin(_norm(y, w["norm"], eps), w["o"])


def _selective(x, w, m):
    inner, rank, N = m["inner"], m["dt_rank"], m["state"]
    p = _lin(x, w["in"])
    xs, z = _silu(_conv(p[..., :inner], w["conv"]) + w["conv.b"]), p[..., inner:]
    r = _lin(xs, w["x"])
    dt = _softplus(_lin(r[..., :rank], w["dt"]) + w["dt.b"])
    A = -torch.exp(w["A_log"])
    S = torch.zeros((x.shape[0], inner, N), dtype=torch.float64, device="cuda")
    y = torch.empty_like(xs)
    for t in range(x.shape[1]):
        S = torch.exp(dt[:, t, :, None] * A) * S + (dt[:, t] * xs[:, t])[..., None] * r[:, t, None, rank:rank + N]
        y[:, t] = torch.einsum("bcn,bn->bc", S, r[:, t, rank + N:])
    return _lin((y + w["D"] * xs) * _silu(z), w["o"])


def _branch(x, w, m, eps, pairing):
    """Softmax attention with the options that its tensors name; the heads' outputs."""
    q, k = _lin(x, w["q"], w.get("q.b")), _lin(x, w["k"], w.get("k.b"))
    v = _lin(x, w["v"], w.get("v.b")) if "v" in w else None
    if "q.conv" in w:
        q, k, v = _conv(q, w["q.conv"]), _conv(k, w["k.conv"]), None if v is None else _conv(v, w["v.conv"])
    v = k if v is None else v
    if "q.norm" in w:
        q, k = _norm(q, w["q.norm"], eps), _norm(k, w["k.norm"], eps)
    mask = m.get("mask") or {}
    q, k = _turn(_heads(q, m["heads"]), m["rot"], pairing), _turn(_heads(k, m["kv_heads"]), m["rot"], pairing)
    window = {"chunk": mask.get("size")} if "scaling" in m["rot"] else {"window": mask.get("size"), "keep_first": mask.get("keep_first", 0)}
    return _attend(q, k, _heads(v, m["kv_heads"]), m["scale"], sink=w.get("sink"), **window)


def _linear_memory(x, w, m, eps):
    H, d = m["heads"], m["dim"]
    q, k, v = (_heads(_lin(x, w[n]), H) for n in "qkv")
    if "decay" in m:
        q, k = _turn(q, m["rot"]), _turn(k, m["rot"]) * d ** -0.5
        decay = torch.tensor(m["decay"], dtype=torch.float64, device="cuda")[:, None].expand(q.shape)
    else:
        q, decay = q * d ** -0.5, _heads(torch.sigmoid(_lin(_lin(x, w["a1"]), w["a2"], w["a2.b"])) ** (1.0 / m["tau"]), H)
    o = _unit(_memory(q, k, v, decay), eps)
    o = o * w["norm"] if "norm" in w else o
    return _lin(o.flatten(2) * _silu(_lin(x, w["g"])), w["o"])


def _delta(x, w, m, eps):
    H, G, d = m["heads"], m["kv_heads"], m["dim"]
    q, k, v = (_heads(_silu(_conv(_lin(x, w[n]), w[n + ".conv"])), c) for n, c in (("q", G), ("k", G), ("v", H)))
    q, k = (a * torch.rsqrt((a * a).sum(-1, keepdim=True) + 1e-6) for a in (q, k))
    q, k = (a.repeat_interleave(H // G, dim=2) for a in (q * d ** -0.5, k))
    keep = torch.exp(-torch.exp(w["A_log"]) * _softplus(_lin(x, w["a"]) + w["dt_bias"]))[..., None].expand(q.shape)
    o = _memory(q, k, v, keep, u=torch.sigmoid(_lin(x, w["b"])))
    return _lin((_norm(o, w["norm"], eps) * _silu(_heads(_lin(x, w["g"]), H))).flatten(2), w["o"])


def _sloped(x, w, m, eps, kept, i):
    H, G = m["heads"], m["kv_heads"]
    if m.get("kv_from") is None:
        kept[i] = _unit(_heads(_lin(x, w["k"], w["k.b"]), G), eps), _heads(_lin(x, w["v"], w["v.b"]), G)
    k, v = kept[i if m.get("kv_from") is None else m["kv_from"]]
    q = _unit(_heads(_lin(x, w["q"], w["q.b"]), H), eps)
    slope = 2.0 ** (-8.0 * torch.arange(1, H + 1, dtype=torch.float64, device="cuda") / H)
    bias = -slope[:, None] * torch.arange(x.shape[1], dtype=torch.float64, device="cuda")
    return _lin(_attend(q, k, v, m["scale"], m["mask"]["size"], bias=bias).flatten(2), w["o"], w["o.b"])


def _mix(family, kind, x, w, m, eps, kept, i):
    if kind == "latent_attention":
        return _latent(x, w, m, eps, kept, i)
    if kind == "mamba2":
        return _mamba2(x, w, m, eps)
    if kind == "mlstm":
        return _mlstm(x, w, m, eps)
    if kind == "delta":
        return _delta(x, w, m, eps)
    if kind == "attention":
        if family == "semesun":
            return _biased(x, w, m, eps, kept)
        if family == "zabozen":
            return _sloped(x, w, m, eps, kept, i)
        return _lin(_branch(x, w, m, eps, "half").flatten(2) * torch.sigmoid(_lin(x, w["g"])), w["o"], w["o.b"])
    left, right = _under(w, "left."), _under(w, "right.")
    o = _branch(x, left, m["left"], eps, "half" if family == "depunex" else "interleaved")
    if "g" in left:
        o = o * torch.sigmoid(_lin(x, left["g"]))[..., None]
    a = _lin(o.flatten(2), left["o"])
    b = _selective(x, right, m["right"]) if family == "depunex" else _linear_memory(x, right, m["right"], eps)
    if kind == "parallel":
        return m["left_scale"] * a + m["right_scale"] * b
    return 0.5 * (_norm(a, left["out"], eps) + _norm(b, right["out"], eps))


# ---- feed-forwards
def _clamped(x, w, limit):
    g, u = _lin(x, w["gate"]).clamp(max=limit), _lin(x, w["up"]).clamp(-limit, limit)
    return _lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), w["down"])


def _unit_of(family, x, w, f):
    if f.get("limit"):
        return _clamped(x, w, f["limit"])
    if family in ("kogilix", "semesun") and "gate" not in w:
        return _lin(torch.relu(_lin(x, w["up"])) ** 2, w["down"])
    gate = _lin(x, w["gate"])
    return _lin((_gelu(gate) if family == "kogilix" else _silu(gate)) * _lin(x, w["up"]), w["down"])


def _routed(family, x, w, f):
    r, x0 = f["router"], x
    x = x.reshape(-1, x.shape[-1])
    z = _lin(x, w["router"], w.get("router.b"))
    s = choice = z if family == "kogilix" else torch.softmax(z, -1) if family == "semesun" else torch.sigmoid(z)
    if "correction" in w:
        choice = s + w["correction"]
    if r.get("groups"):
        by = choice.reshape(len(x), r["groups"]["count"], -1)
        rank = by.max(-1).values if family == "semesun" else by.topk(2, -1).values.sum(-1)
        kept = torch.zeros_like(rank).scatter_(1, rank.topk(r["groups"]["keep"], -1).indices, 1.0).bool()
        choice = by.masked_fill(~kept[..., None], -math.inf).reshape(choice.shape)
    idx = choice.topk(r["top"], -1).indices
    p = s.gather(1, idx)
    p = torch.softmax(p, -1) if family == "kogilix" else p * r["scale"] if family == "semesun" else p / (p.sum(-1, keepdim=True) + 1e-20) if family == "depunex" else p
    y = torch.zeros_like(x)
    for e in range(w["router"].shape[0]):
        row, place = (idx == e).nonzero(as_tuple=True)
        if len(row):
            out = x[row] if e >= r["experts"] else _unit_of(family, x[row], _under(w, "e%d." % e), f["expert"])
            y.index_add_(0, row, p[row, place, None] * out)
    if f.get("shared"):
        u = _unit_of(family, x, _under(w, "shared."), {})
        y = y + (torch.sigmoid(_lin(x, w["shared.sg"])) * u if "shared.sg" in w else u)
    return y.reshape(x0.shape)


def _feed(family, x, w, f):
    return _unit_of(family, x, w, f) if f["kind"] == "dense" else _routed(family, x, w, f)


# ---- whole models: tokens [B, n] -> logits at `places`, [B, places, vocab]
def _llama(cfg, w, tokens, places):
    eps, H, G = cfg["rms_norm_eps"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
    rot = {"base": cfg["rope_theta"], "dims": cfg["hidden_size"] // H}
    x = w["model.embed_tokens.weight"][tokens]
    for i in range(cfg["num_hidden_layers"]):
        u = _under(w, "model.layers.%d." % i)
        h = _norm(x, u["input_layernorm.weight"], eps)
        q, k, v = (_heads(_lin(h, u["self_attn.%s_proj.weight" % n]), c) for n, c in (("q", H), ("k", G), ("v", G)))
        o = _attend(_turn(q, rot), _turn(k, rot), v, rot["dims"] ** -0.5)
        x = x + _lin(o.flatten(2), u["self_attn.o_proj.weight"])
        h = _norm(x, u["post_attention_layernorm.weight"], eps)
        x = x + _lin(_silu(_lin(h, u["mlp.gate_proj.weight"])) * _lin(h, u["mlp.up_proj.weight"]), u["mlp.down_proj.weight"])
    h = _norm(x.gather(1, places[..., None].expand(-1, -1, x.shape[-1])), w["model.norm.weight"], eps)
    return _lin(h, w.get("lm_head.weight", w["model.embed_tokens.weight"]))


def _listed_layers(cfg, w, tokens, places):
    family, eps, emb = cfg["architecture"].lower(), cfg["norm"]["eps"], cfg.get("embedding") or {}
    x = w["embed"][tokens] * emb.get("scale", 1.0)
    if emb.get("bigram"):
        b = emb["bigram"]
        row = torch.full_like(tokens, b["buckets"])
        row[:, 1:] = (tokens[:, :-1] * b["mul_prev"] + tokens[:, 1:] * b["mul_cur"]) % b["buckets"]
        x = x + w["bigram"][row]
    if family == "depunex":
        w = {n: t + 1.0 if n.endswith(("norm1", "final.norm")) else t for n, t in w.items()}    # stored as the distance from 1
    kept, xs = {}, None
    if family == "vozetar":
        xs = x[None].repeat(cfg["streams"], 1, 1, 1)
    for i, layer in enumerate(cfg["layers"]):
        u = _under(w, "l%d." % i)

        def mix(h):
            return _mix(family, layer["type"], h, _under(u, "mix."), layer["mixer"], eps, kept, i)

        def feed(h):
            return _feed(family, h, _under(u, "mlp."), layer["mlp"])

        if xs is not None:
            for n, fn in (("1", mix), ("2", feed)):
                y = fn(_norm(torch.einsum("s,sbnw->bnw", u["hc%s.in" % n], xs), u["norm" + n], eps))
                xs = torch.einsum("st,sbnw->tbnw", u["hc%s.mix" % n], xs) + u["hc%s.out" % n][:, None, None, None] * y
        elif family == "zabozen":
            x = x + cfg["residual_mult"] * _norm(mix(_norm(x, u["norm1"], eps)), u["norm1b"], eps)
            x = x + cfg["residual_mult"] * _norm(feed(_norm(x, u["norm2"], eps)), u["norm2b"], eps)
        elif family == "depunex":
            h = _norm(x, u["norm1"], eps)
            x = x + mix(h) * u["ls1"] + feed(h) * u["ls2"]
            d = cfg["token_side"]["dim"]
            own = w["side.embed"][:, i * d:(i + 1) * d][tokens]
            x = x + _norm(_lin(_gelu(_lin(x, u["side.gate"])) * own, u["side.proj"]), u["side.norm"], eps)
        else:
            x = x + mix(_norm(x, u["norm1"], eps))
            x = x + feed(_norm(x, u["norm2"], eps))
    x = x if xs is None else xs.sum(0)
    z = _lin(_norm(x.gather(1, places[..., None].expand(-1, -1, x.shape[-1])), w["final.norm"], eps), w["head"] if "head" in w else w["embed"])
    cap = cfg.get("logit_softcap")
    return cap * torch.tanh(z / cap) if cap else z


def exact(case, seed):
    if case["kind"] == "generate":
        return None                                               # whole numbers
    prompts, further = _tokens(case, seed)
    more = case["more"]
    cfg = config_of(case["model"])
    w = weights_of(case["model"], case["dtype"])
    w = {n: t.double() for n, t in w.items()}
    n = max(len(p) for p in prompts) + more
    out = torch.empty((1 + more, case["batch"], _vocab(case["model"])), dtype=torch.float64, device="cuda")
    at = max(1, 16384 // n)                                       # sequences at a time
    for a in range(0, len(prompts), at):
        group = range(a, min(len(prompts), a + at))
        tokens = torch.zeros((len(group), n), dtype=torch.int64)
        for r, b in enumerate(group):
            line = prompts[b] + [further[t][b] for t in range(more)]
            tokens[r, :len(line)] = torch.tensor(line)
        places = torch.tensor([[len(prompts[b]) - 1 + t for t in range(more + 1)] for b in group], device="cuda")
        model = _llama if "layers" not in cfg else _listed_layers
        out[:, a:a + len(group)] = model(cfg, w, tokens.cuda(), places).transpose(0, 1)
    return out

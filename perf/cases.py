"""The work that programs have this library do, as cases that can be measured.

Kinds of pass (``run``), each through the public entry points:

* ``prompt``: new sequences take their prompts in one ``Engine.step``; the logits at every prompt's last place come back;
  the slots are given up again.
* ``decode``: the same, then ``steps`` steps of one given token per sequence (replay of a trace, or decoding with ids that
  another program chose); the logits of every step come back.  Prompts are short or the model small, so that most of the
  pass is the single-token steps.
* ``answer``: ``Engine.generate`` (greedy), then one step that scores what was generated: the logits from which every
  generated token was chosen.  In 32 bits, where greedy tokens are the same for every correct implementation.
* ``sample``: one sampling step of a batch over logits on the device, host ids out.

Sizes of models come from ``rocml_b200.config.CATALOG``: the dense decoder from 0.6 to 8 billion weights, which most of the
library is for, and one of the other decoders (recurrences, differential attention, convolutions) with none of its work decided
by comparisons.  Decoders with routed experts are left out: the experts a token takes are a comparison, so rounding alone moves
whole tokens and no tolerance says anything.

Weights and inputs are random and made from the seed: embeddings, heads and biases N(0, 0.02), matrices N(0, 0.64 / sqrt(inputs)) (which is
N(0, 0.02) at 1,024 inputs; the same deviation at every width would let a wide model amplify rounding as no trained one does), norm
scales 1 + N(0, 0.1), ids uniform.  An engine in a user's program has served requests like the next one, so ``prepare`` runs one pass (this captures the decode graphs).
"""
from __future__ import annotations

import math

import torch

from rocml_b200 import Engine, Model, SamplingParams, StepEntry
from rocml_b200.config import CATALOG, config_from_dict
from rocml_b200.parts import BuildEnv
from rocml_b200.sampling import Sampler, XorShift64Star

DEVICE = "cuda:0"


def listed():
    return [
        # one user, a small model, a short question: nothing but latency and launches
        dict(name="decode 0.6b b1", kind="decode", model="qwen3-0.6b", batch=1, shortest=23, longest=23, steps=40),
        # one user, the benchmark's model: every weight read once a token
        dict(name="decode 8b b1", kind="decode", model="qwen3-8b", batch=1, shortest=61, longest=61, steps=12),
        # a small server's batch with a long history each: a small model's weights beside the cache
        dict(name="decode 1.7b b8", kind="decode", model="qwen3-1.7b", batch=8, shortest=700, longest=1337, steps=48),
        # the benchmark's batch on the benchmark's model
        dict(name="decode 8b b8", kind="decode", model="qwen3-8b", batch=8, shortest=40, longest=150, steps=24),
        # a busy server: as many sequences as the loop takes at once
        dict(name="decode 4b b64", kind="decode", model="qwen3-4b", batch=64, shortest=17, longest=40, steps=16),
        # a short question's first token, an odd number of tokens
        dict(name="prompt 1.7b 61", kind="prompt", model="qwen3-1.7b", batch=1, shortest=61, longest=61),
        # the benchmark's prompt
        dict(name="prompt 8b 2048", kind="prompt", model="qwen3-8b", batch=1, shortest=2048, longest=2048),
        # a document, cut into pieces of at most 4,096 tokens: attention over a long cache
        dict(name="prompt 4b 12001", kind="prompt", model="qwen3-4b", batch=1, shortest=12001, longest=12001),
        # the true 32-bit path: generation and scoring
        dict(name="answer 32-bit b3", kind="answer", model="qwen3-like-2k", batch=3, shortest=24, longest=97, steps=16),
        # a decoder with recurrences: a prompt, and a batch of answers
        dict(name="prompt kemizen 2048", kind="prompt", model="kemizen-2k", batch=1, shortest=2048, longest=2048),
        dict(name="decode kemizen b8", kind="decode", model="kemizen-2k", batch=8, shortest=50, longest=333, steps=32),
        # a sampling step of a mid-size batch with the catalog's preset
        dict(name="sample b16", kind="sample", vocab=151936, batch=16, temperature=0.6, top_k=20, top_p=0.95),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    most = max(_seconds(c) for c in listed())
    while True:
        kind = rng.choice(["prompt", "prompt", "decode", "decode", "decode", "answer", "sample"])
        if kind == "sample":
            case = dict(kind=kind, vocab=rng.choice([32768, 151936]), batch=log_int(1, 64), temperature=round(rng.uniform(0.5, 1.2), 2),
                        top_k=rng.choice([0, 20, 50]), top_p=rng.choice([0.0, 0.9, 0.95]))
        elif kind == "answer":
            case = dict(kind=kind, model="qwen3-like-2k", batch=log_int(1, 8), shortest=log_int(5, 60), longest=log_int(5, 200),
                        steps=log_int(4, 24))
        else:
            case = dict(kind=kind, model=rng.choice(["qwen3-0.6b", "qwen3-1.7b", "qwen3-4b", "qwen3-8b", "kemizen-2k"]))
            if kind == "prompt":
                case.update(batch=log_int(1, 12), shortest=log_int(9, 4000), longest=log_int(9, 12000))
            else:
                case.update(batch=log_int(1, 64), shortest=log_int(5, 1000), longest=log_int(5, 1500), steps=log_int(8, 48))
        if "shortest" in case:
            case["shortest"], case["longest"] = sorted((case["shortest"], case["longest"]))
            if case["batch"] == 1:
                case["shortest"] = case["longest"]
            # a decode pass is mostly single tokens
            if kind == "decode" and sum(_lengths(case)) > 200 * case["steps"]:
                continue
        if _seconds(case) <= most:
            return case


def prepare(case, seed):
    if case["kind"] == "sample":
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        # heavy-tailed rows, a few tokens well above the rest, as trained models give them
        x = torch.randn((case["batch"], case["vocab"]), generator=g, device=DEVICE)
        logits = (2.0 * x + 0.4 * x.abs().pow(2.0)).contiguous()
        p = SamplingParams(temperature=case["temperature"], top_k=case["top_k"] or None, top_p=case["top_p"] or None, seed=seed)
        return dict(case=case, sampler=Sampler(DEVICE, max_batch=64), logits=logits, params=[p] * case["batch"], seed=seed)
    config = CATALOG[case["model"]].config
    wide = torch.float32 if case["kind"] == "answer" else torch.bfloat16
    device = torch.device(DEVICE)
    model = Model(config_from_dict(config).to_model_spec(), BuildEnv(device, wide))
    model.load({name: w.to(wide) for name, w in _weights(config, seed)})
    lengths, steps = _lengths(case), case.get("steps", 0)
    engine = Engine(model, max_tokens=sum((n + steps + 63) // 64 * 64 for n in lengths), max_slots=case["batch"], max_step_tokens=4096)
    state = dict(case=case, engine=engine, prompts=_ids(config, lengths, seed), forced=_ids(config, [steps] * len(lengths), seed + 1),
                 out=torch.empty((1 + steps, len(lengths), _vocab(config)), device=device) if case["kind"] == "decode" else None)
    run(state)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "sample":
        rngs = [XorShift64Star(state["seed"] * 64 + i + 1) for i in range(case["batch"])]
        ids = state["sampler"].sample(state["logits"], state["params"], rngs, [[]] * case["batch"])
        return torch.tensor(ids)
    engine, prompts = state["engine"], state["prompts"]
    if case["kind"] == "answer":
        done = engine.generate(prompts, max_new_tokens=case["steps"], stop_tokens=[], ignore_eos=True)
        slots = [engine.new_sequence() for _ in prompts]
        logits = engine.step([StepEntry(s, p + c.tokens[:-1], list(range(len(p) - 1, len(p) + len(c.tokens) - 1)))
                              for s, p, c in zip(slots, prompts, done)])
        for s in slots:
            engine.release(s)
        return {"tokens": torch.tensor([c.tokens for c in done]), "logits": logits}
    slots = [engine.new_sequence() for _ in prompts]
    logits = engine.step([StepEntry(s, p, [len(p) - 1]) for s, p in zip(slots, prompts)])
    if case["kind"] == "decode":
        out, forced = state["out"], state["forced"]
        out[0].copy_(logits)
        for t in range(case["steps"]):
            logits = engine.step([StepEntry(s, [f[t]], [0]) for s, f in zip(slots, forced)])
            out[t + 1].copy_(logits)
        logits = out
    for s in slots:
        engine.release(s)
    return logits


def work(case):
    nbytes, flops = _work(case)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["kind"] == "answer":
        return {"rel": 1e-5, "max": 1e-4}          # 2.3e-6 off `exact`
    # against `exact` the dense decoder's logits are 0.0053 to 0.0058 off at every size, the other's 0.015 to 0.025
    return {"rel": 0.03, "max": 0.4} if case["model"].startswith("kemizen") else {"rel": 0.02, "max": 0.15}


def exact(case, seed):
    """Whole sequences without a cache in float64."""
    if case["kind"] == "sample":
        return None
    config = CATALOG[case["model"]].config
    weights = dict(_weights(config, seed))
    lengths, steps = _lengths(case), case.get("steps", 0)
    prompts = _ids(config, lengths, seed)
    forward = _exact_kemizen if "layers" in config else _exact_qwen3
    with torch.no_grad():
        if case["kind"] == "prompt":
            return torch.cat(forward(config, weights, prompts, [[n - 1] for n in lengths]))
        if case["kind"] == "decode":
            forced = _ids(config, [steps] * len(lengths), seed + 1)
            got = forward(config, weights, [p + f for p, f in zip(prompts, forced)], [range(n - 1, n + steps) for n in lengths])
            return torch.stack(got, dim=1)
        weights = {k: w.double() for k, w in weights.items()}
        done = [list(p) for p in prompts]
        for _ in range(steps):
            got = forward(config, weights, done, [range(n - 1, len(d)) for n, d in zip(lengths, done)])
            for d, x in zip(done, got):
                d.append(int(x[-1].argmax()))
        return {"tokens": torch.tensor([d[n:] for n, d in zip(lengths, done)]), "logits": torch.cat(got)}


# ---- inputs ------------------------------------------------------------------------------------------

def _vocab(config):
    return config["vocab"] if "layers" in config else config["vocab_size"]


def _lengths(case):
    """The prompts' lengths, spread evenly from the shortest to the longest."""
    n, lo, hi = case["batch"], case["shortest"], case["longest"]
    return [hi] if n == 1 else [lo + (hi - lo) * i // (n - 1) for i in range(n)]


def _ids(config, lengths, seed):
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, _vocab(config), (n,), generator=g).tolist() for n in lengths]


def _shapes(config):
    """(tensor name, shape, kind of values) of a folder of this configuration."""
    if "layers" in config:
        return _kemizen_shapes(config)
    H, I, hd = config["hidden_size"], config["intermediate_size"], config["head_dim"]
    q, kv = config["num_attention_heads"] * hd, config["num_key_value_heads"] * hd
    out = [("model.embed_tokens.weight", (config["vocab_size"], H), "matrix")]
    for i in range(config["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for name, shape in (("q", (q, H)), ("k", (kv, H)), ("v", (kv, H)), ("o", (H, q))):
            out.append((f"{p}self_attn.{name}_proj.weight", shape, "matrix"))
        for name, shape in (("gate", (I, H)), ("up", (I, H)), ("down", (H, I))):
            out.append((f"{p}mlp.{name}_proj.weight", shape, "matrix"))
        for name, n in (("self_attn.q_norm", hd), ("self_attn.k_norm", hd), ("input_layernorm", H), ("post_attention_layernorm", H)):
            out.append((f"{p}{name}.weight", (n,), "scale"))
    out.append(("model.norm.weight", (H,), "scale"))
    if not config["tie_word_embeddings"]:
        out.append(("lm_head.weight", (config["vocab_size"], H), "matrix"))
    return out


def _kemizen_shapes(config):
    W = config["width"]
    out = [("embed", (config["vocab"], W), "matrix"), ("final.norm", (W,), "offset"), ("head", (config["vocab"], W), "matrix")]
    for i, layer in enumerate(config["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        add = lambda name, shape, kind="matrix": out.append((p + name, shape, kind))  # noqa: E731
        if layer["type"] == "mlstm":
            k, v, n = m["heads"] * m["dim"], m["heads"] * m["vdim"], m["heads"]
            for name, shape in (("q", (k, W)), ("k", (k, W)), ("v", (v, W)), ("g", (v, W)), ("i", (n, W)), ("f", (n, W)), ("o", (W, v))):
                add(name, shape)
            add("i.b", (n,)), add("f.b", (n,), "forget"), add("norm", (v,), "scale")
        elif layer["type"] == "attention":
            q, k, v = m["heads"] * 2 * m["dim"], m["kv_heads"] * 2 * m["dim"], m["kv_heads"] * m["vdim"]
            add("q", (q, W)), add("o", (W, m["heads"] * m["vdim"])), add("q.norm", (m["dim"],), "scale")
            if m.get("kv_from") is None:
                add("k", (k, W)), add("v", (v, W)), add("k.norm", (m["dim"],), "scale")
            for name in ("lq1", "lk1", "lq2", "lk2"):
                add(name, (m["dim"],), "offset")
        else:
            left, right = m["left"], m["right"]
            q, k, v = left["heads"] * left["dim"], left["kv_heads"] * left["dim"], left["kv_heads"] * left["vdim"]
            o, n, c = left["heads"] * left["vdim"], right["width"], right["width"] // right["blocks"]
            for name, rows in (("q", q), ("k", k), ("v", v)):
                add(f"left.{name}", (rows, W)), add(f"left.{name}.b", (rows,)), add(f"left.{name}.conv", (rows, left["conv"]), "taps")
            add("left.q.norm", (q,), "scale"), add("left.k.norm", (k,), "scale")
            add("left.g", (o, W)), add("left.o", (W, o)), add("left.o.b", (W,)), add("left.out", (W,), "scale")
            for name in ("y", "x"):
                add(f"right.{name}", (n, W)), add(f"right.{name}.b", (n,))
            add("right.conv", (n, right["conv"]), "taps"), add("right.conv.b", (n,))
            for name in ("ra", "ri"):
                add(f"right.{name}", (right["blocks"], c, c)), add(f"right.{name}.b", (right["blocks"], c))
            add("right.lam", (n,), "decay"), add("right.o", (W, n)), add("right.out", (W,), "scale")
        out.append((f"l{i}.norm1", (W,), "offset"))
        if layer["mlp"] is not None:
            ff = layer["mlp"]["ff"]
            out += [(f"l{i}.norm2", (W,), "offset"), (f"l{i}.mlp.up", (ff, W), "matrix"), (f"l{i}.mlp.down", (W, ff), "matrix")]
    return out


def _weights(config, seed):
    """(name, tensor) of every tensor, in bfloat16."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    #                scale and centre: matrices and biases, norm scales, norm scales around zero, a convolution's taps, forget
    #                gates that keep, and decays of a recurrent unit between 0.9 and 0.999 a token
    values = {"matrix": (0.02, 0.0), "scale": (0.1, 1.0), "offset": (0.1, 0.0), "taps": (0.3, 0.25), "forget": (1.0, 3.0), "decay": (1.0, -5.0)}
    for name, shape, kind in _shapes(config):
        scale, centre = values[kind]
        if kind == "matrix" and len(shape) > 1 and "embed" not in name and "head" not in name:
            scale = 0.64 / math.sqrt(shape[-1])
        yield name, torch.randn(shape, generator=g, device=DEVICE, dtype=torch.bfloat16).mul_(scale).add_(centre)


# ---- what a pass cannot do without ----------------------------------------------------------------------

def _work(case):
    """(bytes, operations): in every step the matrices once, the cache's live rows once, new rows and wanted logits; two operations
    a weight and token (the head's only where logits are wanted), scores and their products with the values under the causal mask
    (or window), and the recurrences' updates."""
    if case["kind"] == "sample":
        n = case["batch"] * case["vocab"]
        return 4 * n + 4 * case["batch"], 3 * n
    config = CATALOG[case["model"]].config
    size = 4 if case["kind"] == "answer" else 2
    vocab = _vocab(config)
    head = vocab * (config["width"] if "layers" in config else config["hidden_size"])
    body = sum(math.prod(shape) for name, shape, _ in _shapes(config) if name not in ("embed", "head", "model.embed_tokens.weight", "lm_head.weight"))
    attention, recurrent = _mixers(config)
    lengths, steps = _lengths(case), case.get("steps", 0)
    totals = [0, 0]

    def step(before, new, wanted):
        totals[0] += (body + (head if wanted else 0)) * size + wanted * vocab * 4
        totals[1] += 2 * body * sum(new) + 2 * head * wanted
        for kv_width, score_width, window in attention:
            for b, n in zip(before, new):
                seen = sum(min(b + j + 1, window) for j in range(n)) if window else n * b + n * (n + 1) // 2
                totals[0] += (min(b, window) if window else b) * kv_width * size + n * kv_width * size
                totals[1] += 2 * seen * score_width
        for entries in recurrent:
            totals[0] += 8 * entries * len(new)
            totals[1] += 4 * entries * sum(new)

    zero = [0] * len(lengths)
    step(zero, lengths, len(lengths))
    for t in range(steps if case["kind"] == "decode" else steps - 1):
        step([n + t for n in lengths], [1] * len(lengths), len(lengths))
    if case["kind"] == "answer":
        step(zero, [n + steps - 1 for n in lengths], steps * len(lengths))
    return totals[0], totals[1]


def _mixers(config):
    """([cached values a token, width of scores and values over all heads, window] of every attention, [state's entries] of every recurrence)."""
    if "layers" not in config:
        hd = config["head_dim"]
        return [(2 * config["num_key_value_heads"] * hd, 2 * config["num_attention_heads"] * hd, None)] * config["num_hidden_layers"], []
    attention, recurrent = [], []
    for layer in config["layers"]:
        m = layer["mixer"]
        if layer["type"] == "mlstm":
            recurrent.append(m["heads"] * m["dim"] * (m["vdim"] + 1))
        elif layer["type"] == "attention":
            attention.append((m["kv_heads"] * (2 * m["dim"] + m["vdim"]), 2 * m["heads"] * (m["dim"] + m["vdim"]),
                              m["mask"]["size"] if m.get("mask") else None))
        else:
            left = m["left"]
            attention.append((left["kv_heads"] * (left["dim"] + left["vdim"]), left["heads"] * (left["dim"] + left["vdim"]), None))
            recurrent.append(m["right"]["width"])
    return attention, recurrent


def _seconds(case):
    """What a pass costs, roughly: for choosing cases."""
    nbytes, flops = _work(case)
    return nbytes / 4e12 + flops / (3e13 if case["kind"] == "answer" else 8e14)


# ---- the same in float64 -----------------------------------------------------------------------------------

def _rms(x, eps, weight=1.0):
    return x / torch.sqrt(x.square().mean(dim=-1, keepdim=True) + eps) * weight


def _rotate(x, inv_freq, magnitude=1.0):
    """x [T, heads, dim]: entries i and i + dim / 2 turn by position * inv_freq[i]."""
    angle = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * inv_freq.to(x.device)
    c, s = torch.cos(angle)[:, None] * magnitude, torch.sin(angle)[:, None] * magnitude
    a, b = x.chunk(2, dim=-1)
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _attend(q, k, v, scale, cap=None, window=None):
    """q [T, heads, dim], k and v [T, groups, dim]: causal, every head over its group's keys, a few thousand queries at a time."""
    T, heads = q.shape[:2]
    out = torch.empty((T, heads, v.shape[2]), dtype=q.dtype, device=q.device)
    for h in range(heads):
        g = h // (heads // k.shape[1])
        for a in range(0, T, 4096):
            b = min(T, a + 4096)
            s = (q[a:b, h] @ k[:b, g].T).mul_(scale)
            if cap is not None:
                s = cap * torch.tanh(s / cap)
            back = torch.arange(a, b, device=q.device)[:, None] - torch.arange(b, device=q.device)
            s.masked_fill_((back < 0) | (back >= window) if window else back < 0, float("-inf"))
            out[a:b, h] = torch.softmax(s, dim=-1) @ v[:b, g]
    return out


def _exact_qwen3(config, weights, sequences, wanted):
    eps, hd = config["rms_norm_eps"], config["head_dim"]
    inv_freq = config["rope_theta"] ** (-torch.arange(0, hd, 2, dtype=torch.float64) / hd)
    table = weights["model.embed_tokens.weight"]
    lengths = [len(s) for s in sequences]
    ids = torch.tensor(sum((list(s) for s in sequences), []), device=DEVICE)
    x = table[ids].double()
    for i in range(config["num_hidden_layers"]):
        w = lambda name: weights[f"model.layers.{i}.{name}.weight"].double()  # noqa: E731,B023
        h = _rms(x, eps, w("input_layernorm"))
        q, k, v = (h @ w(f"self_attn.{n}_proj").T for n in "qkv")
        q, k = (_rms(t.view(len(ids), -1, hd), eps, w(f"self_attn.{n}_norm")) for t, n in ((q, "q"), (k, "k")))
        parts = [_attend(_rotate(a, inv_freq), _rotate(b, inv_freq), c, hd ** -0.5)
                 for a, b, c in zip(q.split(lengths), k.split(lengths), v.view(len(ids), -1, hd).split(lengths))]
        x = x + torch.cat(parts).flatten(1) @ w("self_attn.o_proj").T
        h = _rms(x, eps, w("post_attention_layernorm"))
        x = x + (torch.nn.functional.silu(h @ w("mlp.gate_proj").T) * (h @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T
    head = (table if config["tie_word_embeddings"] else weights["lm_head.weight"]).double()
    norm = weights["model.norm.weight"].double()
    return [_rms(part[list(rows)], eps, norm) @ head.T for part, rows in zip(x.split(lengths), wanted)]


def _exact_kemizen(config, weights, sequences, wanted):
    eps = config["norm"]["eps"]
    weights = {k: w.double() for k, w in weights.items()}
    out = []
    for ids, rows in zip(sequences, wanted):
        x = weights["embed"][torch.tensor(ids, device=DEVICE)] * config["embedding"]["scale"]
        kept = {}
        for i, layer in enumerate(config["layers"]):
            w = {k[len(f"l{i}."):]: t for k, t in weights.items() if k.startswith(f"l{i}.")}
            m = {k[4:]: t for k, t in w.items() if k.startswith("mix.")}
            if layer["type"] == "mlstm":
                y = _exact_memory(x, layer["mixer"], m, eps)
            elif layer["type"] == "attention":
                y = _exact_difference(x, layer["mixer"], m, eps, kept, i)
            else:
                y = _exact_side_by_side(x, layer["mixer"], m, eps)
            x = x + _rms(y, eps, 1.0 + w["norm1"])
            if layer["mlp"] is not None:
                x = x + _rms(torch.nn.functional.gelu(x @ w["mlp.up"].T) @ w["mlp.down"].T, eps, 1.0 + w["norm2"])
        out.append(_rms(x[list(rows)], eps, 1.0 + weights["final.norm"]) @ weights["head"].T)
    return out


def _exact_memory(x, m, w, eps):
    """o_t = sum_s e^(F_t - F_s + i_s) (q_t . k_s) v_s over the running maximum's exponent, F the running sum of the log forget gates."""
    T, n, dim, cap = x.shape[0], m["heads"], m["dim"], m["gate_cap"]
    q = (x @ w["q"].T).view(T, n, dim) * dim ** -0.5
    k, v = (x @ w["k"].T).view(T, n, dim), (x @ w["v"].T).view(T, n, m["vdim"])
    gate_i = cap * torch.tanh((x @ w["i"].T + w["i.b"]) / cap)
    F = torch.cumsum(torch.nn.functional.logsigmoid(cap * torch.tanh((x @ w["f"].T + w["f.b"]) / cap)), dim=0)
    seen = torch.ones((T, T), dtype=torch.bool, device=x.device).tril()
    o = torch.empty_like(v)
    for h in range(n):
        e = (F[:, None, h] - F[None, :, h] + gate_i[None, :, h]).masked_fill(~seen, float("-inf"))
        top = torch.maximum(e.amax(dim=1), F[:, h])          # the maximum starts at 0 and decays with the memory
        s = torch.exp(e - top[:, None]) * (q[:, h] @ k[:, h].T)
        o[:, h] = s @ v[:, h] / (torch.maximum(s.sum(dim=1).abs(), torch.exp(-top)) + 1e-6)[:, None]
    return (_rms(o, eps).flatten(1) * w["norm"] * torch.sigmoid(x @ w["g"].T)) @ w["o"].T


def _exact_difference(x, m, w, eps, kept, i):
    T, heads, groups, dim = x.shape[0], m["heads"], m["kv_heads"], m["dim"]
    rot = m["rot"]
    n, base, sc = rot["dims"], rot["base"], rot["scaling"]
    inv_freq = base ** (-torch.arange(0, n, 2, dtype=torch.float64) / n)
    # between the waves that turn `fast` and `slow` times over the original length, the frequencies blend with the slowed ones
    lo, hi = (n * math.log(sc["original"] / (2 * math.pi * sc[t])) / (2 * math.log(base)) for t in ("fast", "slow"))
    lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), n - 1)
    ramp = ((torch.arange(n // 2, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    inv_freq = inv_freq / sc["factor"] * ramp + inv_freq * (1 - ramp)
    turn = lambda t: _rotate(t, inv_freq, 0.1 * math.log(sc["factor"]) + 1.0)  # noqa: E731
    q = turn(_rms((x @ w["q"].T).view(T, heads * 2, dim), eps, w["q.norm"])).view(T, heads, 2, dim)
    if m.get("kv_from") is None:
        k = turn(_rms((x @ w["k"].T).view(T, groups * 2, dim), eps, w["k.norm"])).view(T, groups, 2, dim)
        kept[i] = k, (x @ w["v"].T).view(T, groups, m["vdim"])
    k, v = kept[i if m.get("kv_from") is None else m["kv_from"]]
    a, b = (_attend(q[:, :, j], k[:, :, j], v, m["scale"], m["softcap"], m["mask"]["size"]) for j in (0, 1))
    factor = torch.exp(w["lq1"] @ w["lk1"]) - torch.exp(w["lq2"] @ w["lk2"]) + m["diff"]
    return (_rms(a - factor * b, eps) * (1 - m["diff"])).flatten(1) @ w["o"].T


def _exact_side_by_side(x, m, w, eps):
    T, left, right = x.shape[0], m["left"], m["right"]
    gelu, softplus = (lambda t: torch.nn.functional.gelu(t, approximate="tanh")), torch.nn.functional.softplus

    def conv(u, taps):
        padded = torch.cat([torch.zeros_like(u[: taps.shape[1] - 1]), u])
        if len(u) < taps.shape[1] - 1:
            padded = torch.cat([u.new_zeros((taps.shape[1] - 1, u.shape[1])), u])
        return sum(padded[j: j + T] * taps[:, j] for j in range(taps.shape[1]))

    rot = left["rot"]
    inv_freq = rot["base"] ** (-torch.arange(0, rot["dims"], 2, dtype=torch.float64) / rot["dims"])
    q, k, v = (conv(x @ w[f"left.{n}"].T + w[f"left.{n}.b"], w[f"left.{n}.conv"]) for n in "qkv")
    q = _rotate(_rms(q, eps, w["left.q.norm"]).view(T, left["heads"], -1), inv_freq)
    k = _rotate(_rms(k, eps, w["left.k.norm"]).view(T, left["kv_heads"], -1), inv_freq)
    o = _attend(q, k, v.view(T, left["kv_heads"], -1), left["scale"]).flatten(1)
    a = (o * torch.sigmoid(x @ w["left.g"].T)) @ w["left.o"].T + w["left.o.b"]

    u = conv(x @ w["right.x"].T + w["right.x.b"], w["right.conv"]) + w["right.conv.b"]
    parts = u.view(T, right["blocks"], -1)
    r, i = (torch.sigmoid(torch.einsum("tbi,boi->tbo", parts, w[f"right.{n}"]) + w[f"right.{n}.b"]).flatten(1) for n in ("ra", "ri"))
    log_a = -8.0 * r * softplus(w["right.lam"])
    decay, add = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * i * u
    s, states = torch.zeros_like(u[0]), []
    for t in range(T):
        s = torch.addcmul(add[t], decay[t], s)
        states.append(s)
    b = (torch.stack(states) * gelu(x @ w["right.y"].T + w["right.y.b"])) @ w["right.o"].T
    return (_rms(a, eps, w["left.out"]) + _rms(b, eps, w["right.out"])) / 2

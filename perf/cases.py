"""What the engine is measured on: steps through `Engine.step` and a run of `LLM.generate`, at the sizes that a user has.

A case names a model of random weights, the data type, and one of five kinds of pass over it:

  decode    every request holds its context and brings one token: one step (the bulk of all serving)
  serve     such requests beside portions of prompts under the scheduler's token budget: one step (serving while requests arrive)
  prompt    whole prompts into fresh slots: one step (prefill)
  reply     whole prompts into fresh slots, then their next tokens one by one: `steps` + 1 steps
  generate  the Python entry point from prompts to chosen tokens, the scheduler and the sampler included

The tokens are given (scoring; only "generate" chooses its own), so what a pass returns does not hang on near-ties. A pass returns the
logits at the wanted places, "generate" the tokens and their logits. The models are the layer sizes that bench.py measures: Llama 3.2 1B,
Llama 3.1 8B (four layers), and three of the other designs with four layers of the same width: Keralorn (windowed softmax attention and
lightning attention), Ganupel (recurrent blocks; sigmoid attention beside HGRN2), Viperax (latent attention over several streams, experts).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from stride_b200 import LLM, Engine, EngineOptions, StepEntry

DEVICE = "cuda:0"
VOCAB = {"llama-1b": 128256, "llama-8b": 128256}     # (the others: 32000)
PAGE = 64                                            # tokens a cache page
CHUNK = 64                                           # the scheduler's portion of a prompt
SCALING = {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}


def _case(name, model, kind, requests, shortest, longest, steps=0, rows=0, dtype="bfloat16"):
    c = {"model": model, "dtype": dtype, "kind": kind, "requests": requests, "shortest": shortest, "longest": longest, "steps": steps, "rows": rows}
    return {"name": name, **c} if name else c


def listed() -> list:
    return [
        # one user's chat, a token at a time: launches and latency
        _case("decode_1", "llama-1b", "decode", 1, 300, 300),
        # the headline: eight requests, 256-token prompts and up to 256 generated tokens behind them
        _case("decode_8", "llama-1b", "decode", 8, 257, 511),
        # a busy server: 64 requests whose contexts reach from a short question to a long document
        _case("decode_64", "llama-1b", "decode", 64, 130, 3900),
        # one request over a book
        _case("decode_long", "llama-1b", "decode", 1, 32768, 32768),
        # a larger model's layers (heads of 128): 128 requests at the contexts of a chat service
        _case("decode_128_8b", "llama-8b", "decode", 128, 224, 544),
        # true 32-bit serving of one request
        _case("decode_1_float32", "llama-1b", "decode", 1, 300, 300, dtype="float32"),
        # requests arrive while eight others decode: a step at the default budget of 256 tokens
        _case("serve_256", "llama-1b", "serve", 8, 257, 511, rows=256),
        # a long prompt at once
        _case("prompt_2048", "llama-1b", "prompt", 1, 2048, 2048),
        # the whole way through the Python entry point: eight prompts, 32 tokens each
        _case("generate_8", "llama-1b", "generate", 8, 90, 250, steps=32),
        # the other designs: a long prompt, ragged prompts side by side, short prompts and their replies
        _case("keralorn_prompt_2048", "keralorn", "prompt", 1, 2048, 2048),
        _case("ganupel_reply_8", "ganupel", "reply", 8, 60, 300, steps=8),
        _case("viperax_prompts_2000", "viperax", "prompt", 3, 333, 1025),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    kind = rng.choice(["decode", "decode", "decode", "serve", "prompt", "prompt", "reply", "generate"])
    if kind == "decode":
        model = rng.choice(["llama-1b", "llama-1b", "llama-8b"])
        dtype = "float32" if model == "llama-1b" and rng.random() < 0.2 else "bfloat16"
        n = _log(rng, 1, 4) if dtype == "float32" else _log(rng, 1, 64 if model == "llama-1b" else 128)
        longest = _log(rng, 100, 600) if dtype == "float32" else _log(rng, 100, min(32768, 128 * 1024 // n) if model == "llama-1b" else 600)
        return _case("", model, kind, n, rng.randint(max(1, longest // 3), longest), longest, dtype=dtype)
    if kind == "serve":
        longest = _log(rng, 200, 1500)
        return _case("", "llama-1b", kind, _log(rng, 1, 64), rng.randint(100, longest), longest, rows=_log(rng, 130, 512))
    if kind == "generate":
        longest = rng.randint(40, 250)
        return _case("", "llama-1b", kind, _log(rng, 1, 8), rng.randint(20, longest), longest, steps=rng.randint(8, 32))
    if kind == "prompt":
        model = rng.choice(["llama-1b", "keralorn", "ganupel", "viperax"])
        n = _log(rng, 1, 8)
        longest = _log(rng, 64, 2048 // n)
        return _case("", model, kind, n, rng.randint(max(1, longest // 3), longest), longest)
    longest = _log(rng, 40, 300)
    return _case("", rng.choice(["keralorn", "ganupel", "viperax"]), kind, _log(rng, 1, 16) if longest < 120 else _log(rng, 1, 6),
                 rng.randint(longest // 3, longest), longest, steps=rng.randint(4, 12))


# ---------------------------------------------------------------------------------------------------- models
def config(case) -> dict:
    model = case["model"]
    if model.startswith("llama"):
        big = model == "llama-8b"
        return {"architectures": ["LlamaForCausalLM"], "hidden_size": 4096 if big else 2048, "intermediate_size": 14336 if big else 8192,
                "num_hidden_layers": 4 if big else 16, "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 128 if big else 64,
                "vocab_size": VOCAB[model], "rope_theta": 500000.0, "rope_scaling": dict(SCALING, factor=8.0 if big else 32.0),
                "tie_word_embeddings": not big and case["kind"] != "generate", "rms_norm_eps": 1e-5, "max_position_embeddings": 131072}
    width, ff, vocab = 2048, 8192, 32000
    decay = [1.0 - 2.0 ** (-3 - h / 3.0) for h in range(16)]
    dense = {"kind": "dense", "ff": ff}
    if model == "keralorn":
        att = {"type": "attention", "mlp": dense,
               "mixer": {"heads": 32, "kv_heads": 8, "dim": 64, "vdim": 64, "scale": 0.125, "mask": {"size": 1024}, "rot": {"dims": 32, "base": 500000.0}}}
        lig = {"type": "lightning", "mlp": dense, "mixer": {"heads": 16, "dim": 128, "vdim": 128, "decay": decay}}
        return {"architecture": "Keralorn", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "layers": [att, lig] * 2}
    if model == "ganupel":
        rec = {"type": "rglru", "mixer": {"width": width, "blocks": 16, "conv": 4}, "mlp": dense}
        par = {"type": "parallel", "mlp": dense,
               "mixer": {"left": {"heads": 32, "kv_heads": 8, "dim": 64, "vdim": 64, "scale": 0.125, "mask": {"size": 1024}, "rot": {"dims": 64, "base": 500000.0}},
                         "right": {"heads": 16, "dim": 128, "vdim": 128}, "left_scale": 1.0, "right_scale": 1.0}}
        return {"architecture": "Ganupel", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "layers": [rec, par] * 2}
    mixer = {"heads": 16, "dim": 128, "vdim": 128, "kv_rank": 512, "scale": 128 ** -0.5, "mask": {"size": 1024}}
    moe = {"kind": "moe", "expert": {"ff": ff // 4}, "router": {"experts": 8, "top": 1}, "shared": {"ff": ff // 4}}
    return {"architecture": "Viperax", "vocab": vocab, "width": width, "streams": 3, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
            "logit_scale": 0.5, "logit_softcap": 15.0,
            "layers": [{"type": "latent_attention", "mlp": moe, "mixer": mixer if i < 2 else dict(mixer, kv_from=1)} for i in range(4)]}


def shapes(case) -> dict:
    """Tensor name -> (shape, form): "matrix" N(0, 0.02), "gain" 1 + N(0, 0.1), "bias" N(0, 0.1), and a few forms of their own."""
    cfg, out = config(case), {}
    if case["model"].startswith("llama"):
        W, F, V = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"]
        kv = cfg["num_key_value_heads"] * cfg["head_dim"]
        out["model.embed_tokens.weight"] = ((V, W), "matrix")
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            out.update({p + "input_layernorm.weight": ((W,), "gain"), p + "post_attention_layernorm.weight": ((W,), "gain"),
                        p + "self_attn.q_proj.weight": ((W, W), "matrix"), p + "self_attn.k_proj.weight": ((kv, W), "matrix"),
                        p + "self_attn.v_proj.weight": ((kv, W), "matrix"), p + "self_attn.o_proj.weight": ((W, W), "matrix"),
                        p + "mlp.gate_proj.weight": ((F, W), "matrix"), p + "mlp.up_proj.weight": ((F, W), "matrix"),
                        p + "mlp.down_proj.weight": ((W, F), "matrix")})
        out["model.norm.weight"] = ((W,), "gain")
        if not cfg["tie_word_embeddings"]:
            out["lm_head.weight"] = ((V, W), "matrix")
        return out
    W, V = cfg["width"], cfg["vocab"]
    plus_one = "bias" if case["model"] == "ganupel" else "gain"          # (Ganupel stores a gain's distance from one)
    out["embed"] = ((V, W), "matrix")
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        for n in (1, 2):
            out[f"{p}norm{n}"] = ((W,), plus_one)
            if case["model"] == "keralorn":
                out[f"{p}norm{n}.b"] = ((W,), "bias")
            if case["model"] == "ganupel":
                out[f"{p}ls{n}"] = ((W,), "gain")
            if case["model"] == "viperax":
                S = cfg["streams"]
                out.update({f"{p}hc{n}.in": ((S,), "gain"), f"{p}hc{n}.out": ((S,), "gain"), f"{p}hc{n}.mix": ((S, S), "identity")})
        x = p + "mix."
        if layer["type"] == "attention":
            out.update({x + "q": ((m["heads"] * m["dim"], W), "matrix"), x + "k": ((m["kv_heads"] * m["dim"], W), "matrix"),
                        x + "o": ((W, m["heads"] * m["dim"]), "matrix")})
        elif layer["type"] == "lightning":
            out.update({x + r: ((m["heads"] * 128, W), "matrix") for r in "qkvg"})
            out.update({x + "o": ((W, m["heads"] * 128), "matrix"), x + "norm": ((m["heads"] * 128,), "gain")})
        elif layer["type"] == "rglru":
            C, B = m["width"], m["blocks"]
            for r in "yx":
                out.update({x + r: ((C, W), "matrix"), x + r + ".b": ((C,), "bias")})
            out.update({x + "conv": ((C, m["conv"]), "taps"), x + "conv.b": ((C,), "bias"), x + "lam": ((C,), "decay"), x + "o": ((W, C), "matrix")})
            for r in ("ra", "ri"):
                out.update({x + r: ((B, C // B, C // B), "matrix"), x + r + ".b": ((B, C // B), "bias")})
        elif layer["type"] == "parallel":
            a, g = m["left"], m["right"]
            D, R = a["dim"], g["heads"] * g["dim"]
            out.update({x + "left.q": ((a["heads"] * D, W), "matrix"), x + "left.k": ((a["kv_heads"] * D, W), "matrix"), x + "left.v": ((a["kv_heads"] * D, W), "matrix"),
                        x + "left.o": ((W, a["heads"] * D), "matrix"), x + "left.pb": ((a["heads"],), "attention_bias"),
                        x + "right.q": ((R, W), "matrix"), x + "right.f": ((R, W), "matrix"), x + "right.v": ((R, W), "matrix"), x + "right.f.b": ((R,), "forget"),
                        x + "right.lower": ((R,), "lower"), x + "right.norm": ((g["vdim"],), "gain"), x + "right.o": ((W, R), "matrix")})
        else:
            R, C = m["heads"] * m["dim"], m["kv_rank"]
            out.update({x + "q": ((R, W), "matrix"), x + "g": ((R, W), "matrix"), x + "uk": ((R, C), "matrix"), x + "uv": ((R, C), "matrix"), x + "o": ((W, R), "matrix"),
                        x + "sink": ((m["heads"],), "bias")})
            if m.get("kv_from") is None:
                out.update({x + "dkv": ((C, W), "matrix"), x + "dkv.norm": ((C,), "gain")})
        f = p + "mlp."
        if mlp["kind"] == "moe":
            F = mlp["expert"]["ff"]
            out[f + "table"] = ((V, 1), "table")
            for e in [f"e{k}." for k in range(mlp["router"]["experts"])] + ["shared."]:
                out.update({f + e + "gate": ((F, W), "matrix"), f + e + "up": ((F, W), "matrix"), f + e + "down": ((W, F), "matrix")})
        else:
            F = mlp["ff"]
            out.update({f + "up": ((F, W), "matrix"), f + "down": ((W, F), "matrix")})
            out.update({f + "gate": ((F, W), "matrix")} if case["model"] == "keralorn" else {f + "act": ((4,), "gain")})
    out["final.norm"] = ((W,), plus_one)
    if case["model"] == "keralorn":
        out["final.norm.b"] = ((W,), "bias")
    out["head"] = ((V, W), "matrix")
    return out


def weights(case, seed: int) -> dict:
    """bfloat16 tensors on the GPU, from the seed. Decays and forget gates lie where trained ones do (close to one)."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed * 2 + 1)
    bf = torch.bfloat16

    def randn(shape, std, mean=0.0, dtype=bf):
        t = torch.empty(shape, dtype=dtype, device=DEVICE)
        return t.normal_(mean, std, generator=gen)

    out = {}
    for name, (shape, form) in shapes(case).items():
        if form == "matrix":
            out[name] = randn(shape, 0.02)
        elif form in ("gain", "bias"):
            out[name] = randn(shape, 0.1, 1.0 if form == "gain" else 0.0)
        elif form == "taps":
            out[name] = randn(shape, 0.5)
        elif form == "identity":
            out[name] = (torch.eye(shape[0], device=DEVICE) + randn(shape, 0.1, dtype=torch.float32)).to(bf)
        elif form == "decay":                        # exp(-8 softplus(lam)) uniform in 0.9 .. 0.999
            soft = -torch.log(torch.empty(shape, device=DEVICE).uniform_(0.9, 0.999, generator=gen)) / 8.0
            out[name] = torch.log(torch.expm1(soft)).to(bf)
        elif form == "forget":
            out[name] = randn(shape, 1.0, 3.0)
        elif form == "lower":
            out[name] = torch.empty(shape, device=DEVICE).uniform_(0.0, 0.5, generator=gen).to(bf)
        elif form == "attention_bias":               # a sigmoid's sum over a context stays of the order of one
            out[name] = randn(shape, 0.5, -5.0)
        else:
            out[name] = torch.randint(0, 8, shape, dtype=torch.int32, device=DEVICE, generator=gen)
    if case["kind"] == "generate":
        # a head whose rows follow the embedding's: the next token is as clear a choice as a trained model's, whatever the last bits are
        order = torch.randperm(VOCAB[case["model"]], device=DEVICE, generator=gen)
        head = torch.empty_like(out["lm_head.weight"])
        head[order] = out["model.embed_tokens.weight"]
        out["lm_head.weight"] = head
        out["model.embed_tokens.weight"] = out["model.embed_tokens.weight"] * 100.0
    return out


# ---------------------------------------------------------------------------------------------------- passes
def lengths(case) -> list:
    """The requests' contexts or prompts, from the shortest to the longest in equal ratios, in an order that mixes them."""
    n, lo, hi = case["requests"], case["shortest"], case["longest"]
    if n == 1:
        return [hi]
    all_ = [round(lo * (hi / lo) ** (i / (n - 1))) for i in range(n)]
    step = next(s for s in range(max(1, int(n * 0.618)), 2 * n + 2) if math.gcd(s, n) == 1)
    return [all_[(i * step) % n] for i in range(n)]


def script(case):
    """(tokens that each request holds in front of the pass, steps of the pass), a step being [(request, first position, tokens, wanted places)]."""
    held, steps = lengths(case), []
    if case["kind"] == "decode":
        steps = [[(i, n, 1, [0]) for i, n in enumerate(held)]]
    elif case["kind"] == "serve":
        steps = [[(i, n, 1, [0]) for i, n in enumerate(held)]]
        left, k = case["rows"] - len(held), 0
        while left > 0:                              # a portion of every further request's prompt; every second one ends its prompt
            count = min(CHUNK, left)
            held = held + [(k % 4) * CHUNK]
            steps[0].append((len(held) - 1, held[-1], count, [count - 1] if k % 2 == 0 else []))
            left, k = left - count, k + 1
    else:
        steps = [[(i, 0, n, [n - 1]) for i, n in enumerate(held)]]
        more = case["steps"] - (1 if case["kind"] == "generate" else 0)      # (a generated token that nobody follows is not fed)
        steps += [[(i, n + s, 1, [0]) for i, n in enumerate(held)] for s in range(more)]
        held = [0] * len(held)
    return held, steps


def totals(case) -> list:
    held, steps = script(case)
    return [max(f + c for st in steps for i, f, c, _ in st if i == r) for r in range(len(held))]


def tokens_of(case, seed: int) -> list:
    gen = torch.Generator().manual_seed(seed * 2)
    return [torch.randint(0, VOCAB.get(case["model"], 32000), (n,), generator=gen).tolist() for n in totals(case)]


def prepare(case, seed: int) -> dict:
    rows = 256 if case["kind"] in ("decode", "generate") else 512 if case["kind"] == "serve" else 2048
    total, toks = totals(case), tokens_of(case, seed)
    held, steps = script(case)
    wanted = max(sum(len(w) for *_, w in st) for st in steps)
    full = 1 << (max(wanted, 1) - 1).bit_length()
    context = max(total) + PAGE
    options = EngineOptions(dtype=case["dtype"], max_rows=rows, max_full_rows=full, max_slots=2 * len(total), page_size=PAGE, max_context=context,
                            kv_pages=2 * sum(-(-n // PAGE) for n in total) + 2)
    engine = Engine(None, options, config=config(case), tensors=weights(case, seed))
    state = {"engine": engine, "kind": case["kind"], "steps": case["steps"]}
    if case["kind"] == "generate":
        state["llm"] = LLM(engine=engine, concurrency=8)
        state["prompts"] = [t[:n] for t, n in zip(toks, lengths(case))]
        return state
    state["plan"] = [[(i, first, toks[i][first:first + count], want) for i, first, count, want in st] for st in steps]
    if len(steps) > 1:
        state["out"] = torch.empty((sum(len(w) for st in steps for *_, w in st), VOCAB.get(case["model"], 32000)), dtype=torch.float32, device=DEVICE)
    state["flying"] = []
    if any(held):
        state["slots"] = [engine.cache.acquire_slot() for _ in held]
        fed = [0] * len(held)
        while any(f < h for f, h in zip(fed, held)):
            left, entries = rows, []
            for i, slot in enumerate(state["slots"]):
                count = min(held[i] - fed[i], left)
                if count > 0:
                    assert engine.cache.ensure(slot, fed[i] + count)
                    entries.append(StepEntry(slot, fed[i], toks[i][fed[i]:fed[i] + count], []))
                    fed[i], left = fed[i] + count, left - count
            engine.step(entries)
    return state


def run(state):
    if state["kind"] == "generate":
        results = state["llm"].generate(state["prompts"], max_new_tokens=state["steps"])
        return {"tokens": np.array([r.tokens for r in results]), "values": np.array([r.values for r in results], dtype=np.float32)}
    engine, cache = state["engine"], state["engine"].cache
    slots = state.get("slots")                       # (held over the passes where the requests have a context already)
    if slots is None:                                # fresh slots; the last pass but one has to be over before its own go back
        if len(state["flying"]) == 2:
            done, old = state["flying"].pop(0)
            done.synchronize()
            for slot in old:
                cache.release_slot(slot)
        slots = [cache.acquire_slot() for _ in state["plan"][0]]
        state["flying"].append((torch.cuda.Event(), slots))
    out, at = state.get("out"), 0
    for step in state["plan"]:
        entries = []
        for i, first, toks, want in step:
            if not cache.ensure(slots[i], first + len(toks)):
                raise RuntimeError("the cache is too small")
            entries.append(StepEntry(slots[i], first, toks, want))
        logits = engine.step(entries)
        if out is not None:
            out[at:at + logits.shape[0]].copy_(logits)
            at += logits.shape[0]
    if "slots" not in state:
        state["flying"][-1][0].record()
    return logits if out is None else out


# ---------------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case) -> dict:
    """Weights are counted once a step (they exceed the L2, and a step cannot begin before the one in front of it has ended), keys, values
    and states once a step, logits once. Products: every matrix for every token, the head for the wanted places, one expert a token."""
    cfg, held_steps = config(case), script(case)[1]
    matrix = head = expert = small = 0
    for name, (shape, form) in shapes(case).items():
        n = math.prod(shape)
        if name in ("head", "lm_head.weight"):
            head = n
        elif name in ("embed", "model.embed_tokens.weight"):
            head = head or n
        elif form == "matrix" and ".mlp.e" in name:
            expert += n
        elif form == "matrix":
            matrix += n
        elif form != "table":
            small += n
    size = 4 if case["dtype"] == "float32" else 2
    width = cfg.get("hidden_size") or cfg["width"]
    if "layers" in cfg:
        kinds = [l["type"] for l in cfg["layers"]]
        att = {"attention": (2 * 8 * 64, 32 * 128, 1024), "parallel": (2 * 8 * 64, 32 * 128, 1024), "latent_attention": (512, 16 * 1024, 1024)}
        mixers = [att[k] for k in kinds if k in att]
        states = sum({"lightning": 16 * 128 * 128, "parallel": 16 * 128 * 128, "rglru": 4 * 2048}.get(k, 0) for k in kinds)
    else:
        D = cfg["head_dim"]
        mixers = [(2 * cfg["num_key_value_heads"] * D, 2 * cfg["num_attention_heads"] * D, 0)] * cfg["num_hidden_layers"]
        states = 0
    total_bytes = total_flops = 0.0
    for step in held_steps:
        rows, places = sum(c for _, _, c, _ in step), sum(len(w) for *_, w in step)
        total_bytes += 2.0 * (matrix + small + (expert * min(1.0, rows / 8.0)) + (head if places else 0)) + rows * width * 2.0
        total_bytes += places * 4.0 * VOCAB.get(case["model"], 32000) + len(step) * 2.0 * 4.0 * states
        total_flops += 2.0 * rows * (matrix + expert / 8.0) + 2.0 * places * head + rows * 5.0 * states
        for row, per_key, window in mixers:
            for _, first, count, _ in step:
                seen = [min(first + j + 1, window or first + j + 1) for j in range(count)]
                total_bytes += size * row * (min(first, window or first) + count)
                total_flops += 2.0 * per_key * sum(seen)
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    """About four times what the engine differs from 64 bits by (0.004 to 0.0085 for the designs of four layers, 5e-6 in 32 bits, 2e-4 for
    the clear choices), and less than that for Llama's sixteen layers in bfloat16 (0.016)."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 1e-3}
    if case["kind"] == "generate":
        return {"rel": 1e-3, "max": 4e-3}
    return {"rel": 0.03, "max": 0.3}


# ---------------------------------------------------------------------------------------------------- the same in 64 bits
F64 = torch.float64


def linear(x, w):
    """x W^T over pieces of the tokens."""
    w = w.to(F64)
    return torch.cat([x[a:a + 16384] @ w.T for a in range(0, x.shape[0], 16384)])


def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def layer_norm(x, gain, eps, bias=0.0):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * gain + bias


def silu(z):
    return z * torch.sigmoid(z)


def gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def rotate(x, dims, base, scaling=None):
    """x [T, heads, D] at positions 0 ..: element i < dims / 2 turns with i + dims / 2. The angle is a product of 32-bit numbers, as the designs have it."""
    half = dims // 2
    f = base ** (-2.0 * torch.arange(half, dtype=F64, device=x.device) / dims)
    if scaling:
        wave, old = 2.0 * math.pi / f, scaling["original_max_position_embeddings"]
        low, high = scaling["low_freq_factor"], scaling["high_freq_factor"]
        part = (old / wave - low) / (high - low)
        f = torch.where(wave > old / low, f / scaling["factor"], torch.where(wave < old / high, f, (1.0 - part) * f / scaling["factor"] + part * f))
    angle = (torch.arange(x.shape[0], device=x.device).to(torch.float32)[:, None] * f.to(torch.float32)[None, :]).to(F64)
    c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], dim=-1)


def attend(q, k, v, scale, window=0, sink=None, sigmoid_bias=None):
    """q [T, H, D], k [T, G, D], v [T, G, V] of one sequence; a query sees the last `window` keys up to its own (0: all). [T, H V]."""
    T, H, _ = q.shape
    G = k.shape[1]
    step = max(16, int(2.5e8 / (H * T)))
    out = []
    for a in range(0, T, step):
        b = min(T, a + step)
        lo = max(0, a - window + 1) if window else 0
        s = torch.einsum("tgrd,sgd->grts", q[a:b].reshape(b - a, G, H // G, -1), k[lo:b]) * scale
        i, j = torch.arange(a, b, device=q.device)[:, None], torch.arange(lo, b, device=q.device)[None, :]
        seen = (j <= i) & (i - j < window) if window else j <= i
        if sigmoid_bias is not None:
            p = torch.sigmoid(s + sigmoid_bias.view(G, H // G, 1, 1)) * seen
        else:
            s = s.masked_fill(~seen, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink.view(G, H // G, 1, 1).expand(G, H // G, b - a, 1)], dim=-1)
            p = torch.softmax(s, dim=-1)[..., :b - lo]
        out.append(torch.einsum("grts,sgv->tgrv", p, v[lo:b]).reshape(b - a, -1))
    return torch.cat(out)


def recurrence(q, k, v, keep):
    """S_t = diag(keep_t) S_(t-1) + k_t v_t^T, o_t = S_t^T q_t per head; q, k [T, H, D], v [T, H, V], keep [T or 1, H, D or 1]."""
    S = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F64, device=q.device)
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = keep[min(t, keep.shape[0] - 1)][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
        out[t] = (S * q[t][:, :, None]).sum(1)
    return out


class Exact:
    """Logits of whole sequences, their tokens laid end to end: x [all tokens, width]."""

    def __init__(self, case, seed):
        self.case, self.cfg, self.w = case, config(case), weights(case, seed)

    def t(self, name):
        return self.w[name].to(F64)

    def each(self, f, *xs):
        """f over every sequence's part of xs."""
        parts, at = [], 0
        for n in self.spans:
            parts.append(f(*(x[at:at + n] for x in xs)))
            at += n
        return torch.cat(parts)

    def logits(self, sequences, wanted):
        """wanted: [(sequence, position)]."""
        self.spans = [len(s) for s in sequences]
        self.ids = torch.tensor([t for s in sequences for t in s], device=DEVICE)
        starts = np.concatenate([[0], np.cumsum(self.spans)])
        rows = torch.tensor([int(starts[s]) + p for s, p in wanted], device=DEVICE)
        return getattr(self, self.case["model"].split("-")[0])(rows)

    def llama(self, rows):
        c, H, G, D, eps = self.cfg, self.cfg["num_attention_heads"], self.cfg["num_key_value_heads"], self.cfg["head_dim"], self.cfg["rms_norm_eps"]
        x = self.w["model.embed_tokens.weight"][self.ids].to(F64)
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = rms(x, eps) * self.t(p + "input_layernorm.weight")
            q, k, v = (linear(h, self.w[f"{p}self_attn.{r}_proj.weight"]).view(-1, n, D) for r, n in (("q", H), ("k", G), ("v", G)))

            def one(q, k, v):
                return attend(rotate(q, D, c["rope_theta"], c["rope_scaling"]), rotate(k, D, c["rope_theta"], c["rope_scaling"]), v, D ** -0.5)
            x = x + linear(self.each(one, q, k, v), self.w[p + "self_attn.o_proj.weight"])
            del q, k, v
            if i == c["num_hidden_layers"] - 1:      # nothing else is read of the last layer
                x = x[rows]
            h = rms(x, eps) * self.t(p + "post_attention_layernorm.weight")
            up, gate, down = (self.w[f"{p}mlp.{r}_proj.weight"].to(F64) for r in ("up", "gate", "down"))
            x = torch.cat([x[a:a + 16384] + (silu(h[a:a + 16384] @ gate.T) * (h[a:a + 16384] @ up.T)) @ down.T for a in range(0, x.shape[0], 16384)])
        return linear(rms(x, eps) * self.t("model.norm.weight"), self.w.get("lm_head.weight", self.w["model.embed_tokens.weight"]))

    def keralorn(self, rows):
        eps = self.cfg["norm"]["eps"]
        x = self.w["embed"][self.ids].to(F64)
        for i, layer in enumerate(self.cfg["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            h = layer_norm(x, self.t(p + "norm1"), eps, self.t(p + "norm1.b"))
            if layer["type"] == "attention":
                q, k = linear(h, self.w[p + "mix.q"]).view(-1, m["heads"], m["dim"]), linear(h, self.w[p + "mix.k"]).view(-1, m["kv_heads"], m["dim"])
                rot = m["rot"]["dims"], m["rot"]["base"]
                y = self.each(lambda q, k: attend(rotate(q, *rot), rotate(k, *rot), k, m["scale"], m["mask"]["size"]), q, k)
            else:
                q, k, v = (silu(linear(h, self.w[p + "mix." + r])).view(-1, m["heads"], 128) for r in "qkv")
                keep = torch.tensor(m["decay"], dtype=torch.float32, device=DEVICE).to(F64).view(1, -1, 1)
                y = self.each(lambda q, k, v: recurrence(q, k, v, keep), q, k, v).reshape(x.shape[0], -1)
                y = rms(y, eps) * self.t(p + "mix.norm") * torch.sigmoid(linear(h, self.w[p + "mix.g"]))
            x = x + linear(y, self.w[p + "mix.o"])
            h = layer_norm(x, self.t(p + "norm2"), eps, self.t(p + "norm2.b"))
            x = x + linear(gelu(linear(h, self.w[p + "mlp.gate"])) * linear(h, self.w[p + "mlp.up"]), self.w[p + "mlp.down"])
        return linear(layer_norm(x[rows], self.t("final.norm"), eps, self.t("final.norm.b")), self.w["head"])

    def ganupel(self, rows):
        eps = self.cfg["norm"]["eps"]
        x = self.w["embed"][self.ids].to(F64)
        for i, layer in enumerate(self.cfg["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            h = rms(x, eps) * (1.0 + self.t(p + "norm1"))
            y = self.rglru(h, p + "mix.", m) if layer["type"] == "rglru" else self.side_by_side(h, p + "mix.", m, eps)
            x = x + y * self.t(p + "ls1")
            z = linear(rms(x, eps) * (1.0 + self.t(p + "norm2")), self.w[p + "mlp.up"])
            a, b, c, e = self.t(p + "mlp.act").tolist()
            z = a * rms(z, eps) + b * rms(z ** 2, eps) + c * rms(z ** 3, eps) + e
            x = x + linear(z, self.w[p + "mlp.down"]) * self.t(p + "ls2")
        return linear(rms(x[rows], eps) * (1.0 + self.t("final.norm")), self.w["head"])

    def rglru(self, h, p, m):
        C, B = m["width"], m["blocks"]
        y = gelu(linear(h, self.w[p + "y"]) + self.t(p + "y.b"))
        taps = self.t(p + "conv")

        def conv(u):
            padded = torch.cat([torch.zeros(taps.shape[1] - 1, C, dtype=F64, device=DEVICE), u])
            return self.t(p + "conv.b") + sum(padded[j:j + u.shape[0]] * taps[:, j] for j in range(taps.shape[1]))
        u = self.each(conv, linear(h, self.w[p + "x"]) + self.t(p + "x.b"))
        r, g = (torch.sigmoid(torch.einsum("boi,tbi->tbo", self.t(p + n), u.view(-1, B, C // B)) + self.t(p + n + ".b")).reshape(-1, C) for n in ("ra", "ri"))
        a = torch.exp(-8.0 * r * torch.nn.functional.softplus(self.t(p + "lam")))

        def scan(a, drive):
            S, out = torch.zeros_like(a[0]), torch.empty_like(a)
            for t in range(a.shape[0]):
                S = a[t] * S + drive[t]
                out[t] = S
            return out
        return linear(self.each(scan, a, torch.sqrt(1.0 - a * a) * g * u) * y, self.w[p + "o"])

    def side_by_side(self, h, p, m, eps):
        a, g = m["left"], m["right"]
        q, k, v = (linear(h, self.w[f"{p}left.{r}"]).view(-1, a[n], a["dim"]) for r, n in (("q", "heads"), ("k", "kv_heads"), ("v", "kv_heads")))
        rot = a["rot"]["dims"], a["rot"]["base"]
        left = self.each(lambda q, k, v: attend(rotate(q, *rot), rotate(k, *rot), v, a["scale"], a["mask"]["size"], sigmoid_bias=self.t(p + "left.pb")), q, k, v)
        q, v = silu(linear(h, self.w[p + "right.q"])).view(-1, g["heads"], g["dim"]), linear(h, self.w[p + "right.v"]).view(-1, g["heads"], g["vdim"])
        low = self.t(p + "right.lower")
        f = (low + (1.0 - low) * torch.sigmoid(linear(h, self.w[p + "right.f"]) + self.t(p + "right.f.b"))).view(-1, g["heads"], g["dim"])
        right = rms(self.each(lambda q, v, f: recurrence(q, 1.0 - f, v, f), q, v, f), eps) * self.t(p + "right.norm")
        return m["left_scale"] * linear(left, self.w[p + "left.o"]) + m["right_scale"] * linear(right.reshape(h.shape[0], -1), self.w[p + "right.o"])

    def viperax(self, rows):
        c, eps = self.cfg, self.cfg["norm"]["eps"]
        X = [self.w["embed"][self.ids].to(F64) * c["embedding"]["scale"]] * c["streams"]
        latents = {}

        def around(X, p, norm, f):
            into, out, mix = (self.t(p + n).tolist() for n in (".in", ".out", ".mix"))
            y = f(layer_norm(sum(a * x for a, x in zip(into, X)), self.t(norm), eps))
            return [sum(mix[s][t] * x for s, x in enumerate(X)) + out[t] * y for t in range(len(X))]
        for i, layer in enumerate(c["layers"]):
            p, m = f"l{i}.", layer["mixer"]

            def mixer(h):
                x = p + "mix."
                if m.get("kv_from") is None:
                    latents[i] = rms(linear(h, self.w[x + "dkv"]), eps) * self.t(x + "dkv.norm")
                lat = latents[m.get("kv_from", i)]
                q, k, v = (linear(u, self.w[x + r]).view(-1, m["heads"], 128) for u, r in ((h, "q"), (lat, "uk"), (lat, "uv")))
                sink = self.t(x + "sink")
                y = self.each(lambda q, k, v: attend(q, k, v, m["scale"], m["mask"]["size"], sink=sink), q, k, v)
                return linear(y * torch.sigmoid(linear(h, self.w[x + "g"])), self.w[x + "o"])

            def gated(h, x):
                return linear(silu(linear(h, self.w[x + "gate"])) * linear(h, self.w[x + "up"]), self.w[x + "down"])

            def experts(h):
                x = p + "mlp."
                y, chosen = gated(h, x + "shared."), self.w[x + "table"][self.ids, 0]
                for e in range(layer["mlp"]["router"]["experts"]):
                    at = (chosen == e).nonzero()[:, 0]
                    if at.numel():
                        y[at] += gated(h[at], f"{x}e{e}.")
                return y
            X = around(X, p + "hc1", p + "norm1", mixer)
            X = around(X, p + "hc2", p + "norm2", experts)
        logits = linear(layer_norm(sum(X)[rows], self.t("final.norm"), eps), self.w["head"]) * c["logit_scale"]
        return c["logit_softcap"] * torch.tanh(logits / c["logit_softcap"])


def exact(case, seed: int):
    with torch.no_grad():
        model, toks = Exact(case, seed), tokens_of(case, seed)
        steps = script(case)[1]
        if case["kind"] != "generate":
            return model.logits(toks, [(i, first + j) for st in steps for i, first, _, want in st for j in want])
        # the tokens that the head's rows make clear, checked below by the logits themselves: each is the largest in its row
        head, embed = model.w["lm_head.weight"], model.w["model.embed_tokens.weight"]
        follow = {}
        prompts = [t[:n] for t, n in zip(toks, lengths(case))]
        for s in range(case["steps"]):
            for t in prompts:
                if t[-1] not in follow:
                    follow[t[-1]] = int((head.to(torch.float32) @ embed[t[-1]].to(torch.float32)).argmax())
                t.append(follow[t[-1]])
        n = lengths(case)
        logits = model.logits([t[:-1] for t in prompts], [(i, n[i] - 1 + s) for i in range(len(n)) for s in range(case["steps"])])
        best = logits.max(-1)
        return {"tokens": best.indices.view(len(n), -1).cpu().numpy(), "values": best.values.view(len(n), -1).cpu().numpy()}

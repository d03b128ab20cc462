"""What this framework's speed is measured on: calls of its public entry points at the sizes its users run.

The listed cases are the path of a quantized Llama (the 1B / 8B layer sizes of ``checkpoint.LLAMA_PRESETS``) -- a
feed-forward at one row, at a batch of rows and at a short prompt, a single matrix at a thousand rows, whole layers that
decode a batch over a bf16 and over an 8-bit cache, whole layers that take a prompt, attention alone, a chat turn through the
captured decode engine -- and two of the dense bf16 families through the continuous-batching engine.  ``draw`` gives further
cases of the same kinds with sizes spread over the whole range.

Kinds (``case["kind"]``) and what one pass runs:
    linear   nn.QuantizedLinear on [rows, K]
    mlp      llama.MLP on [rows, hidden]
    decode   llama.TransformerBlock, one new token for each of ``batch`` sequences over ``context`` cached tokens
    prefill  llama.TransformerBlock, ``tokens`` new tokens behind ``offset`` cached ones
    sdpa     ops.scaled_dot_product_attention with the causal mask
    chat     decode.DecodeEngine: a prompt, then ``steps`` decode steps on given tokens
    golitar  engine.HybridEngine: one prompt portion of the delta-rule / differential-attention family
    vokusun  engine.HybridEngine: prompts of several sequences in one step, then decode steps of all of them
"""
from __future__ import annotations

import math

import torch

F64 = torch.float64
BF16 = torch.bfloat16
GROUP = 64

# hidden, feed-forward, query heads, key / value heads, head size, rotary scaling factor
SIZES = {"1b": (2048, 8192, 32, 8, 64, 32.0), "8b": (4096, 14336, 32, 8, 128, 8.0)}
MAX_POSITIONS = 131072
EPS = 1e-5


def listed():
    return [
        # the feed-forward of a 1B model for one token: the smallest call, all latency
        {"name": "mlp_1b_q4_1", "kind": "mlp", "size": "1b", "bits": 4, "rows": 1},
        # an 8B feed-forward for sixteen users decoding together
        {"name": "mlp_8b_q4_16", "kind": "mlp", "size": "8b", "bits": 4, "rows": 16},
        # ... and for a short question, which is more rows than a decode step and fewer than a tile of a prompt
        {"name": "mlp_8b_q4_77", "kind": "mlp", "size": "8b", "bits": 4, "rows": 77},
        # one 8-bit matrix at a prompt portion of a thousand rows
        {"name": "linear_q8_1000", "kind": "linear", "k": 4096, "n": 14336, "bits": 8, "rows": 1000},
        # a layer of an 8-bit 8B model, thirty-two sequences in the middle of their answers (bf16 cache)
        {"name": "decode_8b_q8_b32", "kind": "decode", "size": "8b", "bits": 8, "batch": 32, "context": 2047, "kv_bits": 0},
        # a layer of a 4-bit 8B model, a few long conversations over the 8-bit cache
        {"name": "decode_8b_q4_b5_kv8", "kind": "decode", "size": "8b", "bits": 4, "batch": 5, "context": 7001, "kv_bits": 8},
        # a layer of a 4-bit 8B model taking a whole 8192-token prompt: the largest call
        {"name": "prefill_8b_q4_8192", "kind": "prefill", "size": "8b", "bits": 4, "batch": 1, "tokens": 8192, "offset": 0},
        # a layer of a 1B model (head size 64) taking the rest of a prompt behind a reused prefix
        {"name": "prefill_1b_q4_1531", "kind": "prefill", "size": "1b", "bits": 4, "batch": 1, "tokens": 1531, "offset": 517},
        # causal attention of two 3000-token prompts, no projections
        {"name": "sdpa_d128_3000", "kind": "sdpa", "batch": 2, "heads": 32, "kv_heads": 8, "dim": 128, "tokens": 3000},
        # a chat turn: short question, one user, answer token by token (four of the 8B model's layers and its head)
        {"name": "chat_8b_q4", "kind": "chat", "size": "8b", "bits": 4, "layers": 4, "batch": 1, "prompt": 19, "steps": 24},
        # dense bf16 families: a prompt portion of one, a mixed batch (prompts, then decoding) of the other
        {"name": "golitar_1200", "kind": "golitar", "tokens": 1200},
        {"name": "vokusun_4x", "kind": "vokusun", "batch": 4, "tokens": 330, "steps": 6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "mlp", "mlp", "decode", "decode", "prefill", "prefill", "sdpa", "chat", "golitar", "vokusun"])
    size, bits = rng.choice(["1b", "8b"]), rng.choice([4, 4, 8])
    if kind == "linear":
        return {"kind": kind, "k": rng.choice([2048, 4096, 8192, 14336]), "n": _log_int(rng, 300, 30000), "bits": bits,
                "rows": _log_int(rng, 1, 4096)}
    if kind == "mlp":
        return {"kind": kind, "size": size, "bits": bits, "rows": _log_int(rng, 1, 4096)}
    if kind == "decode":
        return {"kind": kind, "size": size, "bits": bits, "batch": _log_int(rng, 1, 32), "context": _log_int(rng, 50, 6000),
                "kv_bits": rng.choice([0, 8])}
    if kind == "prefill":
        return {"kind": kind, "size": size, "bits": bits, "batch": rng.choice([1, 1, 2]), "tokens": _log_int(rng, 33, 3500),
                "offset": rng.choice([0, 0, _log_int(rng, 10, 2000)])}
    if kind == "sdpa":
        return {"kind": kind, "batch": rng.choice([1, 2, 3]), "heads": 32, "kv_heads": rng.choice([4, 8, 32]),
                "dim": rng.choice([64, 128]), "tokens": _log_int(rng, 50, 4000)}
    if kind == "chat":
        return {"kind": kind, "size": size, "bits": bits, "layers": rng.randint(2, 4), "batch": _log_int(rng, 1, 16),
                "prompt": _log_int(rng, 5, 60), "steps": rng.randint(4, 20)}
    if kind == "golitar":
        return {"kind": kind, "tokens": _log_int(rng, 60, 1600)}
    return {"kind": kind, "batch": rng.randint(1, 4), "tokens": _log_int(rng, 40, 500), "steps": rng.randint(2, 8)}


# ---------------------------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _quantized(g, n, k, bits, gain=1.0):
    """An affine group-quantized matrix as a checkpoint of a U(-1, 1) / sqrt(k) layer holds it: (words, scales, biases)."""
    words = torch.randint(-(1 << 31), 1 << 31, (n, k * bits // 32), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    top = gain / math.sqrt(k)
    spread = 1 - 0.1 * torch.rand((n, k // GROUP), generator=g, device="cuda")
    return words, (2 * top / (2 ** bits - 1) * spread).to(BF16), (-top * spread).to(BF16)


def _normal(g, *shape, std=1.0, dtype=BF16):
    return (std * torch.randn(shape, generator=g, device="cuda")).to(dtype)


def _norm_weight(g, n):
    return (1 + 0.1 * torch.randn(n, generator=g, device="cuda")).to(BF16)


def _llama_args(size, bits, layers=1):
    from proxy_inference_engine_b200.llama import ModelArgs

    hidden, ff, hq, hkv, d, factor = SIZES[size]
    return ModelArgs(hidden_size=hidden, num_hidden_layers=layers, intermediate_size=ff, num_attention_heads=hq,
                     num_key_value_heads=hkv, head_dim=d, vocab_size=128256, rms_norm_eps=EPS, rope_theta=500000.0,
                     max_position_embeddings=MAX_POSITIONS, tie_word_embeddings=size == "1b",
                     rope_scaling={"factor": factor, "low_freq_factor": 1.0, "high_freq_factor": 4.0},
                     quantization={"group_size": GROUP, "bits": bits})


def _put(weights, name, triple):
    weights[name + ".weight"], weights[name + ".scales"], weights[name + ".biases"] = triple


def _layer_weights(g, size, bits):
    """One layer by parameter name.  The query projection has gain 4, so attention is as selective as a trained layer's."""
    hidden, ff, hq, hkv, d, _ = SIZES[size]
    w = {}
    for name, n, k, gain in (("self_attn.q_proj", hq * d, hidden, 4.0), ("self_attn.k_proj", hkv * d, hidden, 1.7),
                             ("self_attn.v_proj", hkv * d, hidden, 1.0), ("self_attn.o_proj", hidden, hq * d, 1.0),
                             ("mlp.gate_proj", ff, hidden, 2.0), ("mlp.up_proj", ff, hidden, 2.0), ("mlp.down_proj", hidden, ff, 1.0)):
        _put(w, name, _quantized(g, n, k, bits, gain))
    w["input_layernorm.weight"], w["post_attention_layernorm.weight"] = _norm_weight(g, hidden), _norm_weight(g, hidden)
    return w


def _golitar_config():
    ff = {"kind": "dense", "ff": 8192}
    delta = {"heads": 16, "kv_heads": 16, "dim": 128, "vdim": 128, "conv": 4}
    attention = {"heads": 16, "kv_heads": 4, "dim": 64, "vdim": 128, "diff": 0.25, "scale": 0.125, "softcap": 40.0,
                 "mask": {"size": 1024}, "rot": {"base": 5e5, "dims": 64}}
    return {"architecture": "Golitar", "vocab": 32000, "width": 2048, "streams": 2, "norm": {"eps": EPS}, "logit_softcap": 30.0,
            "layers": [{"type": "delta", "mlp": ff, "mixer": delta}, {"type": "attention", "mlp": ff, "mixer": attention}]}


def _golitar_weights(g, cfg):
    rnd = lambda *s: torch.rand(s, generator=g, device="cuda") * 2 - 1
    lin = lambda o, i: (rnd(o, i) / math.sqrt(i)).to(BF16)
    W, S = cfg["width"], cfg["streams"]
    w = {"embed": _normal(g, cfg["vocab"], W), "head": lin(cfg["vocab"], W), "final.norm": (0.1 * rnd(W)).to(BF16)}
    for i, ly in enumerate(cfg["layers"]):
        p, q, m = f"l{i}.", f"l{i}.mix.", ly["mixer"]
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        for t in "12":
            w[p + "norm" + t], w[p + f"hc{t}.in"] = (0.1 * rnd(W)).to(BF16), (1 / S + 0.1 * rnd(S)).to(BF16)
            w[p + f"hc{t}.out"] = (1 + 0.2 * rnd(S)).to(BF16)
            w[p + f"hc{t}.mix"] = (torch.eye(S, device="cuda") + 0.1 * rnd(S, S)).to(BF16)
        if ly["type"] == "delta":
            for n, rows in (("q", G * d), ("k", G * d), ("v", H * dv)):
                w[q + n] = lin(rows, W)
                w[q + n + ".conv"] = (rnd(rows, m["conv"]) / 2 + torch.eye(m["conv"], device="cuda")[-1]).to(BF16)
            w[q + "g"], w[q + "b"], w[q + "a"] = lin(H * dv, W), lin(H, W), lin(H, W)
            w[q + "A_log"] = torch.log(0.5 + 4 * torch.rand(H, generator=g, device="cuda")).to(BF16)
            w[q + "dt_bias"], w[q + "norm"] = (rnd(H) - 2).to(BF16), (1 + 0.1 * rnd(dv)).to(BF16)
        else:
            for n, rows in (("q", 2 * H * d), ("k", 2 * G * d), ("v", G * dv)):
                w[q + n], w[q + n + ".b"] = lin(rows, W), (0.1 * rnd(rows)).to(BF16)
            for n in ("q.norm", "k.norm"):
                w[q + n] = (1 + 0.2 * rnd(d)).to(BF16)
            for n in ("lq1", "lk1", "lq2", "lk2"):
                w[q + n] = (0.3 * rnd(d)).to(BF16)
            w[q + "o.b"] = (0.1 * rnd(W)).to(BF16)
        w[q + "o"], w[p + "mlp.up"], w[p + "mlp.down"] = lin(W, H * dv), lin(ly["mlp"]["ff"], W), lin(W, ly["mlp"]["ff"])
    return w


def _vokusun_config():
    ff = {"kind": "dense", "ff": 14336}
    latent = {"heads": 32, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 128, "scale": 192 ** -0.5, "rot": {"base": 1e4, "dims": 64}}
    attention = {"heads": 32, "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 2048, "keep_first": 4},
                 "rot": {"base": 5e4, "dims": 64, "scaling": {"factor": 4.0}}}
    return {"architecture": "Vokusun", "vocab": 32000, "width": 4096, "norm": {"eps": EPS},
            "layers": [{"type": "latent_attention", "mlp": ff, "mixer": latent}, {"type": "attention", "mlp": ff, "mixer": attention}]}


def _vokusun_weights(g, cfg):
    rnd = lambda *s: torch.rand(s, generator=g, device="cuda") * 2 - 1
    lin = lambda o, i: (2 * rnd(o, i) / math.sqrt(i)).to(BF16)
    W = cfg["width"]
    w = {"embed": _normal(g, cfg["vocab"], W), "head": lin(cfg["vocab"], W)}
    names = ["final.norm"] + [f"l{i}.norm{t}" for i in range(len(cfg["layers"])) for t in ("1", "1b", "2", "2b")]
    for name in names:
        w[name], w[name + ".b"] = (1 + 0.2 * rnd(W)).to(BF16), (0.2 * rnd(W)).to(BF16)
    for i, ly in enumerate(cfg["layers"]):
        q, m = f"l{i}.mix.", ly["mixer"]
        H, d = m["heads"], m["dim"]
        if ly["type"] == "latent_attention":
            dr, dv, r = m["rot_dim"], m["vdim"], m["kv_rank"]
            w[q + "q"], w[q + "dkv"], w[q + "dkv.norm"] = lin(H * (d + dr), W), lin(r + dr, W), (1 + 0.2 * rnd(r)).to(BF16)
            w[q + "g"], w[q + "uk"], w[q + "uv"], w[q + "o"] = lin(H, W), lin(H * d, r), lin(H * dv, r), lin(W, H * dv)
        else:
            G = m["kv_heads"]
            w[q + "q"], w[q + "k"], w[q + "o"] = lin(H * d, W), lin(G * d, W), lin(W, H * d)
            w[q + "q.b"], w[q + "k.b"] = (0.5 * rnd(H * d)).to(BF16), (0.5 * rnd(G * d)).to(BF16)
            w[q + "q.norm"], w[q + "k.norm"] = (1 + 0.3 * rnd(d)).to(BF16), (1 + 0.3 * rnd(d)).to(BF16)
        q = f"l{i}.mlp."
        w[q + "gate"], w[q + "up"], w[q + "down"] = lin(ly["mlp"]["ff"], W), lin(ly["mlp"]["ff"], W), lin(W, ly["mlp"]["ff"])
    return w


def _tokens(g, vocab, *shape):
    return torch.randint(0, vocab, shape, generator=g, device="cuda")


def _inputs(case, seed):
    """Everything a pass starts from, as plain tensors: what ``prepare`` loads into the framework and ``exact`` computes on."""
    g, kind = _generator(seed), case["kind"]
    if kind == "linear":
        return {"w": _quantized(g, case["n"], case["k"], case["bits"]), "x": _normal(g, case["rows"], case["k"])}
    if kind == "sdpa":
        b, hq, hkv, d, t = (case[k] for k in ("batch", "heads", "kv_heads", "dim", "tokens"))
        return {"q": _normal(g, b, hq, t, d, std=1.5), "k": _normal(g, b, hkv, t, d, std=1.5), "v": _normal(g, b, hkv, t, d)}
    if kind == "golitar":
        cfg = _golitar_config()
        return {"cfg": cfg, "w": _golitar_weights(g, cfg), "ids": _tokens(g, cfg["vocab"], case["tokens"]).tolist()}
    if kind == "vokusun":
        cfg = _vokusun_config()
        # ragged prompts: sequence i has i * 37 tokens more than the shortest
        ids = [_tokens(g, cfg["vocab"], case["tokens"] + 37 * i + case["steps"]).tolist() for i in range(case["batch"])]
        return {"cfg": cfg, "w": _vokusun_weights(g, cfg), "ids": ids}
    hidden, ff, hq, hkv, d, _ = SIZES[case["size"]]
    if kind == "chat":
        vocab, n = 128256, case["prompt"] + case["steps"]
        w = {}
        for i in range(case["layers"]):
            w.update({f"model.layers.{i}.{k}": v for k, v in _layer_weights(g, case["size"], case["bits"]).items()})
        # embeddings of unit size, as the layers above them are made for
        _put(w, "model.embed_tokens", _quantized(g, vocab, hidden, case["bits"], math.sqrt(hidden)))
        if case["size"] != "1b":
            _put(w, "lm_head", _quantized(g, vocab, hidden, case["bits"]))
        w["model.norm.weight"] = _norm_weight(g, hidden)
        return {"w": w, "ids": _tokens(g, vocab, case["batch"], n).to(torch.int32)}
    if kind == "mlp":
        return {"w": _layer_weights(g, case["size"], case["bits"]), "x": _normal(g, case["rows"], hidden)}
    tokens, past = (1, case["context"]) if kind == "decode" else (case["tokens"], case["offset"])
    b = case["batch"]
    got = {"w": _layer_weights(g, case["size"], case["bits"]), "x": _normal(g, b, tokens, hidden), "k": None, "v": None}
    if past:
        got["k"], got["v"] = _normal(g, b, hkv, past, d), _normal(g, b, hkv, past, d, std=0.6)
    return got


def prepare(case, seed):
    from proxy_inference_engine_b200 import nn, ops

    kind, got = case["kind"], _inputs(case, seed)
    state = {"kind": kind}
    if kind == "linear":
        lin = nn.QuantizedLinear(case["k"], case["n"], bias=False, group_size=GROUP, bits=case["bits"])
        lin.weight, lin.scales, lin.biases = got["w"]
        state.update(layer=lin, x=got["x"])
    elif kind == "sdpa":
        state.update(ops=ops, q=got["q"], k=got["k"], v=got["v"], scale=case["dim"] ** -0.5)
    elif kind == "chat":
        from proxy_inference_engine_b200.checkpoint import build_model
        from proxy_inference_engine_b200.decode import DecodeEngine

        model = build_model(_llama_args(case["size"], case["bits"], case["layers"]), got["w"])
        n = case["prompt"]
        state.update(engine=DecodeEngine(model, batch=case["batch"], max_context=n + case["steps"] + 2),
                     prompt=got["ids"][:, :n].contiguous(), forced=got["ids"][:, n:].t().contiguous())
    elif kind in ("golitar", "vokusun"):
        from proxy_inference_engine_b200.engine import HybridEngine

        if kind == "golitar":
            from proxy_inference_engine_b200.golitar import GolitarArgs as Args, GolitarModel as Model
            lengths = [case["tokens"]]
        else:
            from proxy_inference_engine_b200.vokusun import VokusunArgs as Args, VokusunModel as Model
            lengths = [len(ids) for ids in got["ids"]]
        model = Model(Args.from_dict(got["cfg"]), got["w"], "cuda", "bfloat16")
        state.update(engine=HybridEngine(model, max_tokens=sum(n + 64 for n in lengths), max_seqs=len(lengths)), ids=got["ids"])
        if kind == "vokusun":
            state["steps"] = case["steps"]
    else:
        from proxy_inference_engine_b200.cache import KVCache, QuantizedKVCache
        from proxy_inference_engine_b200.llama import TransformerBlock

        block = TransformerBlock(_llama_args(case["size"], case["bits"]))
        block.load_weights(got["w"])
        if kind == "mlp":
            state.update(layer=block.mlp, x=got["x"])
        else:
            new = got["x"].shape[1]
            past = 0 if got["k"] is None else got["k"].shape[2]
            cache = QuantizedKVCache(capacity=past + new) if case.get("kv_bits") else KVCache(past + new)
            if past:
                cache.update_and_fetch(got["k"], got["v"])
            state.update(layer=block, x=got["x"], cache=cache, new=new, past=past)
            if new > 1:
                state["mask"] = ops.CausalMask(new, past)
    return state


# ---------------------------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind in ("linear", "mlp"):
        return state["layer"](state["x"])
    if kind == "sdpa":
        return state["ops"].scaled_dot_product_attention(state["q"], state["k"], state["v"], scale=state["scale"], mask="causal")
    if kind == "chat":
        engine = state["engine"]
        engine.prefill(state["prompt"])
        logits = [engine.logits.clone()]
        for given in state["forced"]:           # the answer's tokens are given, so that every step's logits can be compared
            engine.tokens.copy_(given)
            engine.step(1)
            logits.append(engine.logits.clone())
        return torch.stack(logits)
    if kind == "golitar":
        out = state["engine"].forward([("a", state["ids"], list(range(0, len(state["ids"]), 8)))])
        state["engine"].finish("a")
        return out
    if kind == "vokusun":
        engine, ids, steps = state["engine"], state["ids"], state["steps"]
        out = [engine.forward([(i, s[:len(s) - steps], None) for i, s in enumerate(ids)])]
        for t in range(steps, 0, -1):
            out.append(engine.forward([(i, [s[len(s) - t]], None) for i, s in enumerate(ids)]))
        for i in range(len(ids)):
            engine.finish(i)
        return torch.stack(out)
    cache = state["cache"]
    out = state["layer"](state["x"], state.get("mask"), cache)
    kept = cache.state
    cache.trim(state["new"])                     # the next pass appends the same tokens again
    return [out, kept]


# ---------------------------------------------------------------------------------------------------- what it costs
def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["rows"], case["n"], case["k"]
        return {"bytes": n * k * _weight_bytes(case["bits"]) + 2 * m * (n + k), "flops": 2 * m * n * k}
    if kind == "sdpa":
        b, hq, hkv, d, t = (case[k] for k in ("batch", "heads", "kv_heads", "dim", "tokens"))
        return {"bytes": 4 * b * (hq + hkv) * t * d, "flops": 4 * b * hq * d * t * (t + 1) // 2}
    if kind == "golitar":
        W, T = 2048, case["tokens"]
        matrices = W * (4 * 2048 + 32) + W * 2048 + W * (2 * 16 * 64 + 2 * 4 * 64 + 4 * 128) + W * 2048 + 4 * W * 8192
        rows = (T + 7) // 8
        keys = sum(min(t + 1, 1024) for t in range(T))
        flops = 2 * T * matrices + 2 * rows * W * 32000 + 16 * T * 6 * 128 * 128 + 2 * 16 * keys * (2 * 64 + 2 * 128)
        return {"bytes": 2 * matrices + 2 * 32000 * W + T * W * 2 + 4 * rows * 32000, "flops": flops}
    if kind == "vokusun":
        W, b, steps = 4096, case["batch"], case["steps"]
        matrices = W * (32 * 192 + 192 + 32) + 2 * 32 * 128 * 128 + W * 4096 + W * (4096 + 1024) + W * 4096 + 6 * W * 14336
        lengths = [case["tokens"] + 37 * i + steps for i in range(b)]
        pairs = sum(n * (n + 1) // 2 for n in lengths)
        flops = 2 * sum(lengths) * matrices + 2 * b * (steps + 1) * W * 32000 + pairs * 32 * (2 * (192 + 128) + 4 * 128)
        return {"bytes": (steps + 1) * (2 * matrices + 2 * 32000 * W + 4 * b * 32000) + 2 * W * sum(lengths), "flops": flops}
    hidden, ff, hq, hkv, d, _ = SIZES[case["size"]]
    per = _weight_bytes(case["bits"])
    attn_w, mlp_w = hidden * d * (2 * hq + 2 * hkv), 3 * hidden * ff
    if kind == "mlp":
        return {"bytes": mlp_w * per + 4 * case["rows"] * hidden, "flops": 2 * case["rows"] * mlp_w}
    token_bytes = 2 * hkv * d * 2                # K and V of one token, bf16
    if kind == "chat":
        b, n, steps, layers, head = case["batch"], case["prompt"], case["steps"], case["layers"], 128256 * hidden
        weights = layers * (attn_w + mlp_w) + head
        ctx = sum(n + i + 1 for i in range(steps))
        flops = 2 * b * (n + steps) * layers * (attn_w + mlp_w) + 2 * b * (steps + 1) * head + 4 * b * layers * hq * d * ctx
        return {"bytes": (steps + 1) * (weights * per + 2 * b * 128256) + layers * b * ctx * token_bytes, "flops": flops}
    new, past = (1, case["context"]) if kind == "decode" else (case["tokens"], case["offset"])
    b = case["batch"]
    if case.get("kv_bits"):
        token_bytes = 2 * hkv * (d + 4 * d // GROUP)
    pairs = new * past + new * (new + 1) // 2
    return {"bytes": (attn_w + mlp_w) * per + 4 * b * new * hidden + b * (past + new) * token_bytes,
            "flops": 2 * b * new * (attn_w + mlp_w) + 4 * b * hq * d * pairs}


def _weight_bytes(bits):
    return bits / 8 + 4 / GROUP


def tolerance(case):
    # bf16 operands and results, fp32 sums; two correct orders of summation differ by the roundings between the operators
    if case["kind"] in ("linear", "sdpa"):
        return {"rel": 0.01, "max": 0.1}
    if case["kind"] == "decode" and case["kv_bits"]:
        return {"rel": 0.02, "max": 0.3, "differ": 0.005}      # a new row's 8-bit codes can move by one
    if case["kind"] in ("mlp", "decode", "prefill"):
        return {"rel": 0.02, "max": 0.3}
    return {"rel": 0.03, "max": 0.5}                           # whole calls: a rounding travels through all that follows


# ---------------------------------------------------------------------------------------------------- in 64 bits
def _dense(triple):
    words, scales, biases = triple
    n, groups = scales.shape
    bits = words.shape[1] * 32 // (groups * GROUP)
    shifts = torch.arange(0, 32, bits, device="cuda", dtype=torch.int32)
    codes = ((words[:, :, None] >> shifts) & (2 ** bits - 1)).reshape(n, groups, GROUP).to(F64)
    return (codes * scales.to(F64)[:, :, None] + biases.to(F64)[:, :, None]).reshape(n, groups * GROUP)


def _apply(x, triple):
    return x @ _dense(triple).t()


def _rms(x, w=None, eps=EPS):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w.to(F64)


def _llama_wavelengths(size):
    _, _, _, _, d, factor = SIZES[size]
    f = torch.tensor(500000.0) ** (torch.arange(0, d, 2, dtype=torch.float32) / d)
    wave = 2 * math.pi * f
    low, high = MAX_POSITIONS / 1.0, MAX_POSITIONS / 4.0
    f = torch.where(wave > low, f * factor, f)
    smooth = (MAX_POSITIONS / wave - 1.0) / 3.0
    return torch.where((wave > high) & (wave < low), f / ((1 - smooth) / factor + smooth), f).to("cuda", F64)


def _rotate_halves(x, first, wavelengths):
    """x [..., L, D]: feature i turns with feature i + D / 2 by position / wavelength."""
    angle = torch.arange(first, first + x.shape[-2], device="cuda", dtype=F64)[:, None] / wavelengths
    c, s = torch.cos(angle), torch.sin(angle)
    a, b = x.chunk(2, -1)
    return torch.cat([a * c - b * s, a * s + b * c], -1)


def _causal(q, k, v, scale, offset=0, window=0, keep=0, cap=0.0):
    """q [H, L, d], k [G, T, d], v [G, T, dv]; query i is at position offset + i."""
    H, L, _ = q.shape
    per = H // k.shape[0]
    i = torch.arange(offset, offset + L, device="cuda")[:, None]
    j = torch.arange(k.shape[1], device="cuda")[None]
    seen = j <= i
    if window:
        seen = seen & ((i - j < window) | (j < keep))
    out = torch.empty((H, L, v.shape[-1]), dtype=F64, device="cuda")
    for h in range(H):
        s = q[h] @ k[h // per].t() * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        out[h] = torch.softmax(s.masked_fill(~seen, -math.inf), -1) @ v[h // per]
    return out


def _silu(x):
    return x * torch.sigmoid(x)


def _exact_mlp(x, w, p=""):
    return _apply(_silu(_apply(x, w[p + "mlp.gate_proj"])) * _apply(x, w[p + "mlp.up_proj"]), w[p + "mlp.down_proj"])


def _exact_block(x, w, size, past_k=None, past_v=None):
    """x [B, L, hidden] behind the cached keys / values -> (y, keys, values) with the new rows appended."""
    _, _, hq, hkv, d, _ = SIZES[size]
    B, L, hidden = x.shape
    first = 0 if past_k is None else past_k.shape[2]
    h = _rms(x, w["input_layernorm.weight"])
    split = lambda y, n: y.view(B, L, n, d).transpose(1, 2)
    wave = _llama_wavelengths(size)
    q = _rotate_halves(split(_apply(h, w["self_attn.q_proj"]), hq), first, wave)
    k = _rotate_halves(split(_apply(h, w["self_attn.k_proj"]), hkv), first, wave)
    v = split(_apply(h, w["self_attn.v_proj"]), hkv)
    if past_k is not None:
        k, v = torch.cat([past_k, k], 2), torch.cat([past_v, v], 2)
    o = torch.stack([_causal(q[b], k[b], v[b], d ** -0.5, first) for b in range(B)])
    x = x + _apply(o.transpose(1, 2).reshape(B, L, hq * d), w["self_attn.o_proj"])
    return x + _exact_mlp(_rms(x, w["post_attention_layernorm.weight"]), w), k, v


def _triples(w):
    """{"name.weight" ...} -> {"name": (words, scales, biases)} beside the norm weights."""
    out = {}
    for name, t in w.items():
        if name.endswith(".scales"):
            p = name[:-7]
            out[p] = (w[p + ".weight"], t, w[p + ".biases"])
        elif name.endswith("norm.weight"):
            out[name] = t
    return out


def _eight_bit(x):
    """What an 8-bit cache in groups of 64 gives back for x: the affine code of each group, scale and bias held in bf16."""
    g = x.reshape(*x.shape[:-1], -1, GROUP)
    lo, hi = g.amin(-1, keepdim=True), g.amax(-1, keepdim=True)
    # the code grid runs from the end of larger magnitude, and that end is moved onto a multiple of the step
    side = lo.abs() > hi.abs()
    step = ((hi - lo) / 255).clamp_min(1e-7)
    step = torch.where(side, step, -step)
    edge = torch.where(side, lo, hi)
    q0 = torch.round(edge / step)
    step = torch.where(q0 != 0, edge / q0, step)
    edge = torch.where(q0 != 0, edge, torch.zeros_like(edge))
    codes = torch.round((g - edge) / step).clamp(0, 255)
    return (codes * step.to(BF16).to(F64) + edge.to(BF16).to(F64)).reshape(x.shape)


def _exact_golitar(cfg, w, ids, wanted):
    w = {k: v.to(F64) for k, v in w.items()}
    offset_norm = lambda x, name: _rms(x) * (1 + w[name])
    xs = w["embed"][torch.tensor(ids, device="cuda")][None].repeat(cfg["streams"], 1, 1)
    T = len(ids)

    def delta(h, p, m):
        H, dk, dv, taps = m["heads"], m["dim"], m["vdim"], m["conv"]
        part = {}
        for n in ("q", "k", "v"):
            z = torch.nn.functional.pad(h @ w[p + n].t(), (0, 0, taps - 1, 0))
            part[n] = _silu(sum(z[j:j + T] * w[p + n + ".conv"][:, j] for j in range(taps))).view(T, H, -1)
        unit = lambda z: z * torch.rsqrt((z * z).sum(-1, keepdim=True) + 1e-6)
        q, k, v = unit(part["q"]) * dk ** -0.5, unit(part["k"]), part["v"]
        beta = torch.sigmoid(h @ w[p + "b"].t())
        decay = torch.exp(-torch.exp(w[p + "A_log"]) * torch.nn.functional.softplus(h @ w[p + "a"].t() + w[p + "dt_bias"]))
        memory, out = torch.zeros((H, dk, dv), dtype=F64, device="cuda"), torch.empty((T, H, dv), dtype=F64, device="cuda")
        for t in range(T):
            memory = memory * decay[t][:, None, None]
            missing = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], memory)[:, 0])
            memory = torch.baddbmm(memory, k[t][:, :, None], missing[:, None])
            out[t] = torch.bmm(q[t][:, None], memory)[:, 0]
        return ((_rms(out) * w[p + "norm"]).reshape(T, -1) * _silu(h @ w[p + "g"].t())) @ w[p + "o"].t()

    def attention(h, p, m):
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = ((h @ w[p + n].t() + w[p + n + ".b"]) for n in ("q", "k", "v"))
        q, k, v = _rms(q.view(T, H, 2, d), w[p + "q.norm"]), _rms(k.view(T, G, 2, d), w[p + "k.norm"]), v.view(T, G, dv)
        freqs = [m["rot"]["base"] ** (-2 * i / d) for i in range(d // 2)]
        maps = []
        for i in (0, 1):
            turn = lambda z: _rotate_neighbours(z[:, :, i].transpose(0, 1), freqs)
            maps.append(_causal(turn(q), turn(k), v.transpose(0, 1), m["scale"], window=m["mask"]["size"], cap=m["softcap"]))
        dot = lambda a, b: torch.exp((w[p + a] * w[p + b]).sum())
        o = maps[0] - (dot("lq1", "lk1") - dot("lq2", "lk2") + m["diff"]) * maps[1]
        return (_rms(o) * (1 - m["diff"])).transpose(0, 1).reshape(T, -1) @ w[p + "o"].t() + w[p + "o.b"]

    def feed_forward(h, p):
        return torch.relu(h @ w[p + "mlp.up"].t()).square() @ w[p + "mlp.down"].t()

    for i, ly in enumerate(cfg["layers"]):
        p = f"l{i}."
        mixer = lambda h: (delta if ly["type"] == "delta" else attention)(h, p + "mix.", ly["mixer"])
        for t, f in (("1", mixer), ("2", lambda h: feed_forward(h, p))):
            y = f(offset_norm(torch.einsum("s,stw->tw", w[p + f"hc{t}.in"], xs), p + "norm" + t))
            xs = torch.einsum("st,sqw->tqw", w[p + f"hc{t}.mix"], xs) + w[p + f"hc{t}.out"][:, None, None] * y
    logits = offset_norm(xs.sum(0), "final.norm")[wanted] @ w["head"].t()
    return cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"])


def _rotate_neighbours(x, freqs):
    """x [heads, T, d]: features 2 i and 2 i + 1 turn together by position * freqs[i]; the rest passes."""
    n = 2 * len(freqs)
    angle = torch.arange(x.shape[1], device="cuda", dtype=F64)[:, None] * torch.tensor(freqs, device="cuda", dtype=F64)
    c, s = torch.cos(angle), torch.sin(angle)
    a, b = x[..., 0:n:2], x[..., 1:n:2]
    return torch.cat([torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2), x[..., n:]], -1)


def _exact_vokusun(cfg, w, ids, wanted):
    """One sequence from its start -> logits of the wanted positions.  w: float64."""
    T = len(ids)

    def norm(x, name):
        c = x - x.mean(-1, keepdim=True)
        return c * torch.rsqrt((c * c).mean(-1, keepdim=True) + EPS) * w[name] + w[name + ".b"]

    def latent(h, p, m):
        H, d, dr, dv, r = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "kv_rank"))
        freqs = [m["rot"]["base"] ** (-2 * i / dr) for i in range(dr // 2)]
        q, low = (h @ w[p + "q"].t()).view(T, H, d + dr).transpose(0, 1), h @ w[p + "dkv"].t()
        c = _rms(low[:, :r], w[p + "dkv.norm"])
        q = torch.cat([q[..., :d], _rotate_neighbours(q[..., d:], freqs)], -1)
        k = torch.cat([(c @ w[p + "uk"].t()).view(T, H, d).transpose(0, 1),
                       _rotate_neighbours(low[None, :, r:], freqs).expand(H, T, dr)], -1)
        o = _causal(q, k, (c @ w[p + "uv"].t()).view(T, H, dv).transpose(0, 1), m["scale"])
        return (o * torch.sigmoid(h @ w[p + "g"].t()).t()[:, :, None]).transpose(0, 1).reshape(T, -1) @ w[p + "o"].t()

    def attention(h, p, m):
        H, G, d, rot = m["heads"], m["kv_heads"], m["dim"], m["rot"]
        freqs = [rot["base"] ** (-2 * i / rot["dims"]) / rot["scaling"]["factor"] for i in range(rot["dims"] // 2)]
        q = (h @ w[p + "q"].t() + w[p + "q.b"]).view(T, H, d).transpose(0, 1)
        v = (h @ w[p + "k"].t() + w[p + "k.b"]).view(T, G, d).transpose(0, 1)
        q, k = _rotate_neighbours(_rms(q, w[p + "q.norm"]), freqs), _rotate_neighbours(_rms(v, w[p + "k.norm"]), freqs)
        o = _causal(q, k, v, m["scale"], window=m["mask"]["size"], keep=m["mask"]["keep_first"])
        return o.transpose(0, 1).reshape(T, -1) @ w[p + "o"].t()

    x = w["embed"][torch.tensor(ids, device="cuda")]
    for i, ly in enumerate(cfg["layers"]):
        p = f"l{i}."
        mixer = latent if ly["type"] == "latent_attention" else attention
        x = x + norm(mixer(norm(x, p + "norm1"), p + "mix.", ly["mixer"]), p + "norm1b")
        h = norm(x, p + "norm2")
        h = torch.nn.functional.gelu(h @ w[p + "mlp.gate"].t(), approximate="tanh") * (h @ w[p + "mlp.up"].t())
        x = x + norm(h @ w[p + "mlp.down"].t(), p + "norm2b")
    return norm(x, "final.norm")[wanted] @ w["head"].t()


def exact(case, seed):
    kind, got = case["kind"], _inputs(case, seed)
    if kind == "linear":
        return _apply(got["x"].to(F64), got["w"])
    if kind == "sdpa":
        q, k, v = (got[n].to(F64) for n in "qkv")
        return torch.stack([_causal(q[b], k[b], v[b], case["dim"] ** -0.5) for b in range(case["batch"])])
    if kind == "golitar":
        return _exact_golitar(got["cfg"], got["w"], got["ids"], list(range(0, case["tokens"], 8)))
    if kind == "vokusun":
        w, steps, rows = {k: v.to(F64) for k, v in got["w"].items()}, case["steps"], []
        for ids in got["ids"]:
            rows.append(_exact_vokusun(got["cfg"], w, ids, list(range(len(ids) - steps - 1, len(ids)))))
        return torch.stack(rows, 1)
    w = _triples(got["w"])
    if kind == "mlp":
        return _exact_mlp(got["x"].to(F64), w)
    if kind == "chat":
        ids = got["ids"].long()
        words, scales, biases = w["model.embed_tokens"]
        x = _dense((words[ids.flatten()], scales[ids.flatten()], biases[ids.flatten()])).view(*ids.shape, -1)
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            x = _exact_block(x, {k[len(p):]: v for k, v in w.items() if k.startswith(p)}, case["size"])[0]
        x = _rms(x[:, case["prompt"] - 1:], w["model.norm.weight"]).transpose(0, 1)
        return _apply(x, w["model.embed_tokens" if case["size"] == "1b" else "lm_head"])
    past = [None if got[n] is None else got[n].to(F64) for n in "kv"]
    if case.get("kv_bits"):
        # the cached rows are 8-bit codes; the row this token appends is one of thousands and is left as it is
        y, _, _ = _exact_block(got["x"].to(F64), w, case["size"], _eight_bit(past[0]), _eight_bit(past[1]))
        return [y, None]
    y, k, v = _exact_block(got["x"].to(F64), w, case["size"], *past)
    return [y, [k, v]]

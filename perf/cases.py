"""What the performance of this engine is measured on: steps of `Engine`, as a serving program issues them.

A case is one step through the engine's public entry points: prompts (add the requests, one step, end them) or decode rows and
mixed batches for a caller that schedules itself (the rows' pages reserved once, StepFunction called without cache management, so
that every pass computes the same step).  Kinds:

  decode            LFM2 model of the named preset, one-token rows over requests that hold `context` positions
  prompt            LFM2 model of the named preset, whole prompts in one step, the last position's logits wanted
  mixed             LFM2 model of the named preset, decode rows beside one portion of a prompt (a continuous batch's step)
  blocks_f32        one convolution block and one attention block of the named preset in the 32-bit path, every position wanted
  attention         one attention block of the named preset, a portion of a long prompt over the positions before it
  delta, state_space, memory, experts_decode
                    the mixers of the other architectures at the sizes of `bench.py`: the gated delta rule, the Mamba-2 mixer, the
                    matrix memory beside routed experts in groups, and decode rows through latent attention, attention with keys
                    as values and ungated routed experts

Whole models draw their weights by the engine's random mode; the kinds of one or two layers get theirs from here, as a model folder
(matrices of standard deviation 1/sqrt(inputs), so that a layer's output is as large as the stream).
"""
import json
import math
import os
import struct
import tempfile

import torch

PRESETS = {     # imparo_b200/config/presets
    "1.2b": dict(width=2048, heads=32, kv_heads=8, ff=8192, layers="ccaccaccacacacac"),
    "700m": dict(width=1536, heads=24, kv_heads=8, ff=6912, layers="ccaccaccacacacac"),
    "350m": dict(width=1024, heads=16, kv_heads=8, ff=4608, layers="ccaccaccacacacac"),
}
HEAD = 64
VOCAB = 65536
SMALL_VOCAB = 1024          # of the kinds of one or two layers: every position's logits come back


def listed():
    return [
        # a single user's chat on the smallest model: launches and latency
        {"name": "decode_350m_b1", "kind": "decode", "model": "350m", "rows": 1, "context": 301},
        # a small server: the benchmark's own decode step
        {"name": "decode_1.2b_b8", "kind": "decode", "model": "1.2b", "rows": 8, "context": 2048},
        # a busy server
        {"name": "decode_1.2b_b64", "kind": "decode", "model": "1.2b", "rows": 64, "context": 2000},
        # a short question
        {"name": "prompt_1.2b_131", "kind": "prompt", "model": "1.2b", "tokens": 131, "prompts": 1},
        # a page of text: the benchmark's own prompt
        {"name": "prompt_1.2b_2048", "kind": "prompt", "model": "1.2b", "tokens": 2048, "prompts": 1},
        # a step of a continuous batch under a budget of 512 tokens
        {"name": "mixed_700m_512", "kind": "mixed", "model": "700m", "rows": 24, "context": 1100, "portion": 488},
        # the 32-bit path, which results are checked with
        {"name": "blocks_f32_1000", "kind": "blocks_f32", "model": "350m", "tokens": 1000, "prompts": 3},
        # a long document, portion by portion
        {"name": "attention_350m_long", "kind": "attention", "model": "350m", "tokens": 4096, "context": 20000},
        # prompts through the recurrent mixers of the other architectures
        {"name": "delta_2048", "kind": "delta", "tokens": 2048, "prompts": 1},
        {"name": "state_space_1999", "kind": "state_space", "tokens": 1999, "prompts": 2},
        {"name": "memory_experts_2048", "kind": "memory", "tokens": 2048, "prompts": 1},
        # decode rows through routed experts and latent attention
        {"name": "experts_decode_b8", "kind": "experts_decode", "rows": 8, "context": 1024},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "mixed", "blocks_f32", "attention", "delta", "state_space", "memory",
                       "experts_decode"])
    model = rng.choice(["1.2b", "700m", "350m"])
    if kind == "decode":
        return {"kind": kind, "model": model, "rows": _log(rng, 1, 64), "context": _log(rng, 60, 2000)}
    if kind == "prompt":
        tokens = _log(rng, 20, 2047)
        return {"kind": kind, "model": model, "tokens": tokens, "prompts": rng.randint(1, min(4, tokens // 10))}
    if kind == "mixed":
        rows = rng.randint(3, 31)
        return {"kind": kind, "model": rng.choice(["700m", "350m"]), "rows": rows, "context": _log(rng, 200, 1500), "portion": 512 - rows}
    if kind == "attention":
        return {"kind": kind, "model": "350m", "tokens": _log(rng, 1000, 4096), "context": _log(rng, 2000, 20000)}
    if kind == "experts_decode":
        return {"kind": kind, "rows": _log(rng, 1, 32), "context": _log(rng, 100, 1200)}
    if kind == "blocks_f32":
        return {"kind": kind, "model": "350m", "tokens": _log(rng, 60, 1000), "prompts": rng.randint(1, 4)}
    return {"kind": kind, "tokens": _log(rng, 300, 2048), "prompts": rng.randint(1, 3)}


# ---- configurations -----------------------------------------------------------------------------------------------

def _lfm2(model, layers, vocab):
    p = PRESETS[model]
    return {"architectures": ["Lfm2ForCausalLM"], "model_type": "lfm2", "vocab_size": vocab, "hidden_size": p["width"],
            "num_hidden_layers": len(layers), "layer_types": ["conv" if c == "c" else "full_attention" for c in layers],
            "num_attention_heads": p["heads"], "num_key_value_heads": p["kv_heads"], "block_ff_dim": p["ff"],
            "block_auto_adjust_ff_dim": False, "conv_L_cache": 3, "conv_bias": False, "rope_theta": 1000000.0, "norm_eps": 1e-5,
            "tie_embedding": True, "max_position_embeddings": 128000}


DELTA = dict(width=1024, heads=8, kv_heads=4, dim=64, vdim=128, taps=4, inner=64, ff=4096, streams=4)
SSM = dict(width=1024, heads=32, vdim=64, state=64, taps=4)
MEMORY = dict(width=1024, heads=8, dim=64, vdim=128, experts=16, top=2, groups=4, keep=2, ff=1024, limit=7.0, cap=10.0)
EXPERTS = dict(width=1024, lat_heads=16, lat_dim=64, rot=32, rank=96, heads=16, kv_heads=4, head=64, window=512, experts=16, top=2,
               groups=4, keep=2, ff=1536, side=128, layers=8)


def _config(case):
    kind = case["kind"]
    if kind in ("decode", "prompt", "mixed"):
        return _lfm2(case["model"], PRESETS[case["model"]]["layers"], VOCAB)
    if kind == "blocks_f32":
        return _lfm2(case["model"], "ca", SMALL_VOCAB)
    if kind == "attention":
        return _lfm2(case["model"], "a", SMALL_VOCAB)
    if kind == "delta":
        d = DELTA
        mixer = {"heads": d["heads"], "kv_heads": d["kv_heads"], "dim": d["dim"], "vdim": d["vdim"], "conv": d["taps"],
                 "decay_rank": d["inner"], "gate_rank": d["inner"]}
        return {"architecture": "Keralix", "vocab": SMALL_VOCAB, "width": d["width"], "norm": {"eps": 1e-5}, "streams": d["streams"],
                "embedding": {"scale": 1.0},
                "layers": [{"type": "channel_delta", "mixer": mixer, "mlp": {"kind": "dense", "ff": d["ff"]}}]}
    if kind == "state_space":
        s = SSM
        mixer = {"heads": s["heads"], "vdim": s["vdim"], "state": s["state"], "groups": 1, "conv": s["taps"], "norm_groups": 1}
        return {"architecture": "Negotar", "vocab": SMALL_VOCAB, "width": s["width"], "norm": {"eps": 1e-5}, "logit_scale": 1.0,
                "layers": [{"type": "mamba2", "mixer": mixer}] * 2}
    if kind == "memory":
        m = MEMORY
        moe = {"kind": "moe", "router": {"experts": m["experts"], "top": m["top"], "scale": 2.5,
                                         "groups": {"count": m["groups"], "keep": m["keep"]}},
               "expert": {"ff": m["ff"], "limit": m["limit"]}, "shared": {"ff": m["ff"], "limit": m["limit"]}}
        mixer = {"heads": m["heads"], "dim": m["dim"], "vdim": m["vdim"], "gate_cap": m["cap"]}
        return {"architecture": "Zepesun", "vocab": SMALL_VOCAB, "width": m["width"], "max_positions": 2048, "norm": {"eps": 1e-5},
                "embedding": {"scale": 1.0}, "layers": [{"type": "mlstm", "mixer": mixer, "mlp": moe}]}
    x = EXPERTS
    lat = {"heads": x["lat_heads"], "dim": x["lat_dim"], "rot_dim": x["rot"], "vdim": x["lat_dim"], "kv_rank": x["rank"],
           "scale": (x["lat_dim"] + x["rot"]) ** -0.5, "mask": {"size": x["window"]},
           "rot": {"base": 500000.0, "dims": x["rot"], "scaling": {"factor": 4.0, "original": 2048, "fast": 32.0, "slow": 1.0}}}
    att = {"heads": x["heads"], "kv_heads": x["kv_heads"], "dim": x["head"], "vdim": x["head"], "scale": x["head"] ** -0.5,
           "rot": {"base": 500000.0, "dims": x["head"], "scaling": {"factor": 4.0}}}
    moe = {"kind": "moe", "router": {"experts": x["experts"], "top": x["top"], "scale": 2.0,
                                     "groups": {"count": x["groups"], "keep": x["keep"]}},
           "expert": {"ff": x["ff"]}, "shared": {"ff": x["ff"]}}
    kinds = []
    for i in range(0, x["layers"], 4):
        kinds += [("latent_attention", lat), ("attention", att), ("attention", att), ("latent_attention", dict(lat, kv_from=i))]
    return {"architecture": "Zinunex", "vocab": 32768, "width": x["width"], "norm": {"eps": 1e-6}, "token_side": {"dim": x["side"]},
            "layers": [{"type": t, "mixer": m, "mlp": moe} for t, m in kinds]}


# ---- weights of the kinds of one or two layers --------------------------------------------------------------------

def _weights(case, seed):
    """name -> tensor on the GPU, as the model folder stores them (matrices bfloat16, or 32-bit for the 32-bit path)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 7 + 1)
    matrix = torch.float32 if case["kind"] == "blocks_f32" else torch.bfloat16
    W = {}

    def mat(name, n, k, std=None):
        W[name] = (torch.randn(n, k, generator=gen, device="cuda") * (k ** -0.5 if std is None else std)).to(matrix)

    def vec(name, *shape, low=0.9, high=1.1):
        W[name] = low + (high - low) * torch.rand(*shape, generator=gen, device="cuda")

    def normal(name, *shape, std):
        W[name] = torch.randn(*shape, generator=gen, device="cuda") * std

    kind = case["kind"]
    if kind in ("blocks_f32", "attention"):
        p = PRESETS[case["model"]]
        H, F = p["width"], p["ff"]
        mat("model.embed_tokens.weight", SMALL_VOCAB, H, 1.0)
        vec("model.embedding_norm.weight", H)
        for i, c in enumerate("ca" if kind == "blocks_f32" else "a"):
            q = f"model.layers.{i}."
            vec(q + "operator_norm.weight", H)
            vec(q + "ffn_norm.weight", H)
            if c == "c":
                mat(q + "conv.in_proj.weight", 3 * H, H)
                normal(q + "conv.conv.weight", H, 1, 3, std=0.6)
                mat(q + "conv.out_proj.weight", H, H)
            else:
                mat(q + "self_attn.q_proj.weight", p["heads"] * HEAD, H)
                mat(q + "self_attn.k_proj.weight", p["kv_heads"] * HEAD, H)
                mat(q + "self_attn.v_proj.weight", p["kv_heads"] * HEAD, H)
                mat(q + "self_attn.out_proj.weight", H, p["heads"] * HEAD)
                vec(q + "self_attn.q_layernorm.weight", HEAD, low=1.5, high=2.0)
                vec(q + "self_attn.k_layernorm.weight", HEAD, low=1.5, high=2.0)
            mat(q + "feed_forward.w1.weight", F, H)
            mat(q + "feed_forward.w3.weight", F, H)
            mat(q + "feed_forward.w2.weight", H, F)
    elif kind == "delta":
        d = DELTA
        H, n, qk, vv = d["width"], d["streams"], d["kv_heads"] * d["dim"], d["heads"] * d["vdim"]
        mat("embed", SMALL_VOCAB, H, 1.0)
        vec("final.norm", H)
        for hc in ("hc1", "hc2"):
            vec(f"l0.{hc}.in", n, low=0.1, high=0.5)
            vec(f"l0.{hc}.out", n, low=0.5, high=1.5)
            W[f"l0.{hc}.mix"] = 0.8 * torch.eye(n, device="cuda") + 0.05 * torch.randn(n, n, generator=gen, device="cuda")
        vec("l0.norm1", H)
        vec("l0.norm2", H)
        m = "l0.mix."
        mat(m + "q", qk, H)
        mat(m + "k", qk, H)
        mat(m + "v", vv, H)
        normal(m + "q.conv", qk, d["taps"], std=0.5)
        normal(m + "k.conv", qk, d["taps"], std=0.5)
        normal(m + "v.conv", vv, d["taps"], std=0.5)
        mat(m + "b", d["heads"], H)
        vec(m + "A_log", d["heads"], low=-3.0, high=0.0)
        vec(m + "norm", d["vdim"])
        mat(m + "a1", d["inner"], H)
        mat(m + "a2", d["heads"] * d["dim"], d["inner"])
        vec(m + "dt_bias", d["heads"] * d["dim"], low=-4.0, high=-1.0)
        mat(m + "g1", d["inner"], H)
        mat(m + "g2", vv, d["inner"])
        mat(m + "o", H, vv)
        mat("l0.mlp.gate", d["ff"], H)
        mat("l0.mlp.up", d["ff"], H)
        mat("l0.mlp.down", H, d["ff"])
    elif kind == "state_space":
        s = SSM
        H, inner, N = s["width"], s["heads"] * s["vdim"], s["state"]
        mat("embed", SMALL_VOCAB, H, 1.0)
        vec("final.norm", H, low=-0.1, high=0.1)          # stored as the distance from one
        for i in range(2):
            vec(f"l{i}.norm1", H, low=-0.1, high=0.1)
            m = f"l{i}.mix."
            mat(m + "in", 2 * inner + 2 * N + s["heads"], H)
            normal(m + "conv", inner + 2 * N, s["taps"], std=0.5)
            normal(m + "conv.b", inner + 2 * N, std=0.02)
            vec(m + "dt_bias", s["heads"], low=-4.0, high=-1.0)
            vec(m + "A_log", s["heads"], low=-1.0, high=1.5)
            vec(m + "D", s["heads"], low=0.5, high=1.5)
            vec(m + "norm", inner)
            mat(m + "o", H, inner)
    elif kind == "memory":
        z = MEMORY
        H, qk, vv = z["width"], z["heads"] * z["dim"], z["heads"] * z["vdim"]
        mat("embed", SMALL_VOCAB, H, 1.0)
        mat("head", SMALL_VOCAB, H)
        mat("pos", 2048, H, 0.3)
        vec("final.norm", H)
        vec("l0.norm1", H)
        m = "l0.mix."
        for name, n in (("q", qk), ("k", qk), ("v", vv), ("g", vv)):
            mat(m + name, n, H)
        mat(m + "o", H, vv)
        vec(m + "norm", vv)
        mat(m + "i", z["heads"], H)
        mat(m + "f", z["heads"], H)
        vec(m + "i.b", z["heads"], low=-2.0, high=1.0)
        vec(m + "f.b", z["heads"], low=1.0, high=4.0)
        normal("l0.mlp.router", z["experts"], H, std=H ** -0.5)
        for e in [f"e{j}" for j in range(z["experts"])] + ["shared"]:
            mat(f"l0.mlp.{e}.gate", z["ff"], H)
            mat(f"l0.mlp.{e}.up", z["ff"], H)
            mat(f"l0.mlp.{e}.down", H, z["ff"])
    return W


def _write_folder(folder, config, tensors):
    """A model folder: config.json and model.safetensors (length, JSON header, raw little-endian tensors)."""
    header, at = {}, 0
    for name, t in tensors.items():
        n = t.numel() * t.element_size()
        header[name] = {"dtype": "BF16" if t.dtype == torch.bfloat16 else "F32", "shape": list(t.shape), "data_offsets": [at, at + n]}
        at += n
    text = json.dumps(header).encode()
    text += b" " * (-len(text) % 8)
    with open(os.path.join(folder, "model.safetensors"), "wb") as f:
        f.write(struct.pack("<Q", len(text)))
        f.write(text)
        for t in tensors.values():
            f.write(t.contiguous().view(torch.uint8).reshape(-1).cpu().numpy().data)
    with open(os.path.join(folder, "config.json"), "w") as f:
        json.dump(config, f)


# ---- inputs -------------------------------------------------------------------------------------------------------

def _vocab(case):
    config = _config(case)
    return config.get("vocab_size") or config["vocab"]


def _tokens(case, seed, n, stream):
    gen = torch.Generator()
    gen.manual_seed(int(seed) * 1009 + stream)
    return torch.randint(0, _vocab(case), (n,), generator=gen).tolist()


def _lengths(case):
    """A prompt step's tokens over its prompts: one about half as long as the one before."""
    left, out = case["tokens"], []
    for i in range(case["prompts"], 1, -1):
        out.append(max(1, min(left - (i - 1), left * 4 // 7)))
        left -= out[-1]
    return out + [left]


def _contexts(case):
    """Positions the decode rows hold: three lengths, so that rows of one step differ."""
    c = case["context"]
    return [(c, c * 3 // 4 + 1, c * 7 // 8)[i % 3] for i in range(case["rows"])]


def _engine(case, seed, **settings):
    from imparo_b200 import Engine
    kind = case["kind"]
    dtype = "float32" if kind == "blocks_f32" else "bfloat16"
    if kind in ("decode", "prompt", "mixed", "experts_decode"):
        return Engine(config=_config(case), seed=int(seed), dtype=dtype, page_size=16, **settings)
    with tempfile.TemporaryDirectory(prefix="imparo_cases_") as folder:
        _write_folder(folder, _config(case), _weights(case, seed))
        return Engine(folder, dtype=dtype, page_size=16, **settings)


def prepare(case, seed):
    from imparo_b200.engine import StepItem
    kind = case["kind"]
    if kind in ("prompt", "blocks_f32", "delta", "state_space", "memory"):
        lengths = _lengths(case)
        engine = _engine(case, seed, ctx=2048, parallel=len(lengths), max_step_tokens=2048)
        want = (lambda n: [n - 1]) if kind == "prompt" else (lambda n: list(range(n)))
        items = [StepItem(r, _tokens(case, seed, n, r), want(n)) for r, n in enumerate(lengths)]
        return {"engine": engine, "items": items, "prompts": True}
    if kind == "attention":
        n, context = case["tokens"], case["context"]
        engine = _engine(case, seed, ctx=context + n, parallel=1, max_step_tokens=8192)
        engine.add_request(0)
        text = _tokens(case, seed, context + n, 0)
        for at in range(0, context, 8192):
            engine.step([StepItem(0, text[at:min(at + 8192, context)])])
        items = [StepItem(0, text[context:], list(range(n)))]
    else:                                              # decode rows, and with a portion of a prompt beside them
        contexts = _contexts(case)
        engine = _engine(case, seed, ctx=2560, parallel=len(contexts) + 1, max_step_tokens=2048)
        items = []
        for r, c in enumerate(contexts):
            engine.add_request(r)
            text = _tokens(case, seed, c + 1, r)
            engine.step([StepItem(r, text[:c])])
            items.append(StepItem(r, text[c:], [0]))
        if kind == "mixed":
            r, n = len(contexts), case["portion"]
            engine.add_request(r)
            text = _tokens(case, seed, 2 * n, r)
            engine.step([StepItem(r, text[:n])])
            items.append(StepItem(r, text[n:], [n - 1]))
    for it in items:
        engine.cache.reserve(it.request, len(it.tokens))
    return {"engine": engine, "items": items, "prompts": False}


def run(state):
    engine, items = state["engine"], state["items"]
    if not state["prompts"]:
        return engine.step_fn(items, manage_cache=False)
    for it in items:
        engine.add_request(it.request)
    logits = engine.step(items)
    for it in items:
        engine.end_request(it.request)
    return logits


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def _lfm2_layer(p, c):
    """Matrix entries of one layer's mixer and of its feed-forward."""
    H = p["width"]
    mixer = 4 * H * H if c == "c" else (2 * p["heads"] + 2 * p["kv_heads"]) * HEAD * H
    return mixer, 3 * H * p["ff"]


def _causal(n, start=0, window=None):
    """Pairs of query and key of `n` queries from position `start` on."""
    if window is None:
        return n * start + n * (n + 1) // 2
    return sum(min(start + i + 1, window) for i in range(n))


def work(case):
    kind = case["kind"]
    if kind in ("decode", "prompt", "mixed", "blocks_f32", "attention"):
        p = PRESETS[case["model"]]
        H = p["width"]
        layers = {"blocks_f32": "ca", "attention": "a"}.get(kind, p["layers"])
        vocab = SMALL_VOCAB if kind in ("blocks_f32", "attention") else VOCAB
        size = 4 if kind == "blocks_f32" else 2
        # (tokens, positions before them, wanted rows) of every request of the step
        if kind in ("prompt", "blocks_f32"):
            reqs = [(n, 0, 1 if kind == "prompt" else n) for n in _lengths(case)]
        elif kind == "attention":
            reqs = [(case["tokens"], case["context"], case["tokens"])]
        else:
            reqs = [(1, c, 1) for c in _contexts(case)]
            if kind == "mixed":
                reqs.append((case["portion"], case["portion"], 1))
        T, wanted = sum(r[0] for r in reqs), sum(r[2] for r in reqs)
        n_attn = layers.count("a")
        mixers, ffs = (sum(_lfm2_layer(p, c)[i] for c in layers) for i in (0, 1))
        last = ffs // len(layers)
        kv = n_attn * 2 * p["kv_heads"] * HEAD * size
        flops = 2.0 * T * (mixers + ffs - last) + 2.0 * wanted * (last + vocab * H)
        flops += n_attn * 4.0 * p["heads"] * HEAD * sum(_causal(n, s) for n, s, _ in reqs)
        moved = (mixers + ffs + vocab * H) * size + kv * sum(n + s for n, s, _ in reqs) + wanted * vocab * 4
        return {"bytes": moved, "flops": flops}
    if kind == "experts_decode":
        x = EXPERTS
        H, n = x["width"], case["rows"]
        lat = (x["lat_heads"] * (x["lat_dim"] + x["rot"] + x["lat_dim"]) + x["rank"] + x["rot"]) * H + 2 * x["lat_heads"] * x["lat_dim"] * x["rank"]
        att = (2 * x["heads"] + x["kv_heads"]) * x["head"] * H
        expert = 2 * H * x["ff"]
        each = x["layers"] // 2 * (lat + att) + x["layers"] * (x["experts"] * H + expert + 2 * H * x["side"])
        reached = x["experts"] * (1.0 - (1.0 - x["top"] / x["experts"]) ** n)          # on average, for choices that are spread
        cached = sum(x["layers"] // 4 * min(c, x["window"]) * (x["rank"] + x["rot"]) + x["layers"] // 2 * c * x["kv_heads"] * x["head"]
                     for c in _contexts(case))
        flops = 2.0 * n * (each + x["layers"] * x["top"] * expert + 32768 * H)
        flops += sum(x["layers"] // 2 * (4.0 * x["heads"] * x["head"] * c + 2.0 * x["lat_heads"] * (2 * x["rank"] + x["rot"]) * min(c, x["window"]))
                     for c in _contexts(case))
        return {"bytes": 2.0 * (each + x["layers"] * reached * expert + 32768 * H + cached) + n * 32768 * 4, "flops": flops}
    T, reqs = case["tokens"], case["prompts"]
    if kind == "delta":
        d = DELTA
        H, qk, vv = d["width"], d["kv_heads"] * d["dim"], d["heads"] * d["vdim"]
        params = (2 * qk + 2 * vv + d["heads"] + 2 * d["inner"]) * H + d["inner"] * (d["heads"] * d["dim"] + vv) + 3 * H * d["ff"]
        inner, state = 7.0 * d["heads"] * d["dim"] * d["vdim"], d["heads"] * d["dim"] * d["vdim"]
    elif kind == "state_space":
        s = SSM
        H, n = s["width"], s["heads"] * s["vdim"]
        params = 2 * ((2 * n + 2 * s["state"] + s["heads"]) * H + n * H)
        inner, state = 2 * 5.0 * n * s["state"], 2 * n * s["state"]
    else:
        z = MEMORY
        H, qk, vv = z["width"], z["heads"] * z["dim"], z["heads"] * z["vdim"]
        used = (2 * qk + 3 * vv + 2 * z["heads"] + z["experts"]) * H + (z["top"] + 1) * 3 * H * z["ff"]
        params = used + (z["experts"] - z["top"]) * 3 * H * z["ff"]
        inner, state = 5.0 * z["heads"] * z["dim"] * z["vdim"], z["heads"] * z["dim"] * z["vdim"]
        return {"bytes": 2.0 * params + 2.0 * SMALL_VOCAB * H + T * SMALL_VOCAB * 4 + reqs * state * 8,
                "flops": 2.0 * T * (used + SMALL_VOCAB * H) + T * inner}
    return {"bytes": 2.0 * params + 2.0 * SMALL_VOCAB * H + T * SMALL_VOCAB * 4 + reqs * state * 8,
            "flops": 2.0 * T * (params + SMALL_VOCAB * H) + T * inner}


def tolerance(case):
    """Whole bfloat16 models: rounding at every matrix of 8 to 16 layers.  One or two bfloat16 layers: activations are rounded
    between the products.  32-bit: sums of up to 4,608 products."""
    kind = case["kind"]
    if kind in ("decode", "prompt", "mixed", "experts_decode"):
        return {"rel": 0.03, "max": 0.3}
    if kind == "blocks_f32":
        return {"rel": 6e-6, "max": 6e-5}
    return {"rel": 0.01, "max": 0.1}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------

def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _conv(u, taps):
    """u [T, C], taps [C, n], the last column on the current row, zeros before the start."""
    n = taps.shape[1]
    padded = torch.cat([u.new_zeros(n - 1, u.shape[1]), u])
    return sum(taps[:, j] * padded[j:j + u.shape[0]] for j in range(n))


def _silu(z):
    return z * torch.sigmoid(z)


def _rotate(x, positions, theta):
    """x [T, heads, HEAD], half-split pairs; frequencies and angles are 32-bit numbers by the model's definition."""
    half = HEAD // 2
    inv = (theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) * 2.0 / HEAD)).float()
    a = (positions.float()[:, None] * inv[None, :]).double()[:, None, :]
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * a.cos() - v * a.sin(), u * a.sin() + v * a.cos()], -1)


def _attention(q, k, v, start):
    """q [n, heads, HEAD] from position `start` on, k and v [start + n, kv_heads, HEAD]."""
    n, heads = q.shape[:2]
    out = torch.empty_like(q)
    seen = torch.arange(k.shape[0], device=q.device)[None, :] <= torch.arange(start, start + n, device=q.device)[:, None]
    for h in range(heads):
        g = h // (heads // k.shape[1])
        s = (q[:, h] @ k[:, g].T) * HEAD ** -0.5
        out[:, h] = torch.softmax(s.masked_fill(~seen, -math.inf), -1) @ v[:, g]
    return out.reshape(n, -1)


def _exact_lfm2(case, W, tokens, start, layers):
    """Logits of the positions from `start` on (with one attention layer, whose keys come from the embeddings alone)."""
    x = W["model.embed_tokens.weight"][tokens]
    positions = torch.arange(len(tokens), device=x.device)
    for i, c in enumerate(layers):
        p = f"model.layers.{i}."
        h = _rms(x, 1e-5) * W[p + "operator_norm.weight"]
        if c == "c":
            b, g, u = (h @ W[p + "conv.in_proj.weight"].T).chunk(3, -1)
            y = (g * _conv(b * u, W[p + "conv.conv.weight"][:, 0])) @ W[p + "conv.out_proj.weight"].T
        else:
            q, k, v = ((h @ W[p + f"self_attn.{n}_proj.weight"].T).reshape(len(tokens), -1, HEAD) for n in "qkv")
            q = _rotate(_rms(q, 1e-5) * W[p + "self_attn.q_layernorm.weight"], positions, 1000000.0)
            k = _rotate(_rms(k, 1e-5) * W[p + "self_attn.k_layernorm.weight"], positions, 1000000.0)
            x = x[start:]
            y = _attention(q[start:], k, v, start) @ W[p + "self_attn.out_proj.weight"].T
        x = x + y
        h = _rms(x, 1e-5) * W[p + "ffn_norm.weight"]
        x = x + (_silu(h @ W[p + "feed_forward.w1.weight"].T) * (h @ W[p + "feed_forward.w3.weight"].T)) @ W[p + "feed_forward.w2.weight"].T
    return (_rms(x, 1e-5) * W["model.embedding_norm.weight"]) @ W["model.embed_tokens.weight"].T


def _exact_delta(W, tokens):
    d, T = DELTA, len(tokens)
    heads, dim, vdim = d["heads"], d["dim"], d["vdim"]
    X = W["embed"][tokens][None].repeat(d["streams"], 1, 1)

    def mixer(h):
        m = "l0.mix."
        q = _silu(_conv(h @ W[m + "q"].T, W[m + "q.conv"])).reshape(T, -1, dim)
        k = _silu(_conv(h @ W[m + "k"].T, W[m + "k.conv"])).reshape(T, -1, dim)
        v = _silu(_conv(h @ W[m + "v"].T, W[m + "v.conv"])).reshape(T, heads, vdim)
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dim ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        q, k = (t.repeat_interleave(heads // d["kv_heads"], 1) for t in (q, k))
        beta = torch.sigmoid(h @ W[m + "b"].T)
        dt = torch.nn.functional.softplus((h @ W[m + "a1"].T) @ W[m + "a2"].T + W[m + "dt_bias"], threshold=40).reshape(T, heads, dim)
        g = torch.exp(-torch.exp(W[m + "A_log"])[None, :, None] * dt)
        S, o = h.new_zeros(heads, dim, vdim), torch.empty_like(v)
        for t in range(T):
            S = S * g[t][:, :, None]
            u = beta[t][:, None] * (v[t] - (k[t][:, None] @ S)[:, 0])
            S = S + k[t][:, :, None] * u[:, None]
            o[t] = (q[t][:, None] @ S)[:, 0]
        gate = torch.sigmoid((h @ W[m + "g1"].T) @ W[m + "g2"].T)
        return ((_rms(o, 1e-5) * W[m + "norm"]).reshape(T, -1) * gate) @ W[m + "o"].T

    def feed_forward(h):
        return (_silu(h @ W["l0.mlp.gate"].T) * (h @ W["l0.mlp.up"].T)) @ W["l0.mlp.down"].T

    for hc, norm, f in (("l0.hc1.", "l0.norm1", mixer), ("l0.hc2.", "l0.norm2", feed_forward)):
        y = f(_rms(torch.einsum("s,stw->tw", W[hc + "in"], X), 1e-5) * W[norm])
        X = torch.einsum("st,snw->tnw", W[hc + "mix"], X) + W[hc + "out"][:, None, None] * y
    return (_rms(X.sum(0), 1e-5) * W["final.norm"]) @ W["embed"].T


def _exact_state_space(W, tokens):
    s, T = SSM, len(tokens)
    heads, vdim, N = s["heads"], s["vdim"], s["state"]
    inner = heads * vdim
    x = W["embed"][tokens]
    for i in range(2):
        m = f"l{i}.mix."
        proj = x @ W[m + "in"].T
        z, dt = proj[:, :inner], proj[:, 2 * inner + 2 * N:]
        xbc = _silu(_conv(proj[:, inner:2 * inner + 2 * N], W[m + "conv"]) + W[m + "conv.b"])
        u, B, C = xbc[:, :inner].reshape(T, heads, vdim), xbc[:, inner:inner + N], xbc[:, inner + N:]
        dt = torch.nn.functional.softplus(dt + W[m + "dt_bias"], threshold=40)
        keep = torch.exp(-torch.exp(W[m + "A_log"]) * dt)
        S, y = x.new_zeros(heads, N, vdim), torch.empty_like(u)
        for t in range(T):
            S = keep[t][:, None, None] * S + dt[t][:, None, None] * B[t][None, :, None] * u[t][:, None]
            y[t] = C[t] @ S + W[m + "D"][:, None] * u[t]
        y = _rms(y.reshape(T, inner) * _silu(z), 1e-5) * W[m + "norm"]
        x = x + _rms(y @ W[m + "o"].T, 1e-5) * (1.0 + W[f"l{i}.norm1"])
    return (_rms(x, 1e-5) * (1.0 + W["final.norm"])) @ W["embed"].T


def _exact_memory(W, tokens):
    z, T = MEMORY, len(tokens)
    heads, dim, vdim, cap = z["heads"], z["dim"], z["vdim"], z["cap"]
    x = W["embed"][tokens] + W["pos"][:T]
    h = _rms(x, 1e-5) * W["l0.norm1"]
    m = "l0.mix."
    q = (h @ W[m + "q"].T).reshape(T, heads, dim) * dim ** -0.5
    k = (h @ W[m + "k"].T).reshape(T, heads, dim)
    v = (h @ W[m + "v"].T).reshape(T, heads, vdim)
    a = cap * torch.tanh((h @ W[m + "i"].T + W[m + "i.b"]) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ W[m + "f"].T + W[m + "f.b"]) / cap))
    S, n, top, o = h.new_zeros(heads, dim, vdim), h.new_zeros(heads, dim), h.new_zeros(heads), torch.empty_like(v)
    for t in range(T):
        new = torch.maximum(f[t] + top, a[t])
        keep, put = torch.exp(f[t] + top - new), torch.exp(a[t] - new)
        S = keep[:, None, None] * S + put[:, None, None] * k[t][:, :, None] * v[t][:, None]
        n = keep[:, None] * n + put[:, None] * k[t]
        top = new
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        o[t] = (q[t][:, None] @ S)[:, 0] / den[:, None]
    y = (_rms(o, 1e-5).reshape(T, -1) * W[m + "norm"] * torch.sigmoid(h @ W[m + "g"].T)) @ W[m + "o"].T

    def expert(u, e):
        p, c = f"l0.mlp.{e}.", z["limit"]
        gate, up = (u @ W[p + "gate"].T).clamp(max=c), (u @ W[p + "up"].T).clamp(-c, c)
        return (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ W[p + "down"].T

    # (the choice is made on the activations as the bfloat16 path has them: a row that falls between two experts is no error)
    s = torch.softmax(h.to(torch.bfloat16).double() @ W["l0.mlp.router"].T, -1)
    groups = s.reshape(T, z["groups"], -1).amax(-1).topk(z["keep"], -1).indices
    allowed = torch.zeros(T, z["groups"], device=x.device, dtype=torch.bool).scatter(1, groups, True)
    w, ids = s.masked_fill(~allowed.repeat_interleave(z["experts"] // z["groups"], 1), -1.0).topk(z["top"], -1)
    w = w / (w.sum(-1, keepdim=True) + 1e-20) * 2.5
    y = y + expert(h, "shared")
    for e in range(z["experts"]):
        row, place = (ids == e).nonzero(as_tuple=True)
        y[row] += w[row, place][:, None] * expert(h[row], f"e{e}")
    return (_rms(x + y, 1e-5) * W["final.norm"]) @ W["head"].T


def exact(case, seed):
    """The kinds of one or two layers; whole models would take their weights from the engine itself."""
    kind = case["kind"]
    if kind in ("decode", "prompt", "mixed", "experts_decode"):
        return None
    W = {name: t.double() for name, t in _weights(case, seed).items()}
    if kind == "attention":
        text = torch.tensor(_tokens(case, seed, case["context"] + case["tokens"], 0), device="cuda")
        return _exact_lfm2(case, W, text, case["context"], "a")
    out = []
    for r, n in enumerate(_lengths(case)):
        text = torch.tensor(_tokens(case, seed, n, r), device="cuda")
        if kind == "blocks_f32":
            out.append(_exact_lfm2(case, W, text, 0, "ca"))
        else:
            out.append({"delta": _exact_delta, "state_space": _exact_state_space, "memory": _exact_memory}[kind](W, text))
    return torch.cat(out)

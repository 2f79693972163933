"""The workloads by which this engine's speed is judged: what a server does with the model families that the package runs.

A case is a model of one of the benchmark's sizes with random weights, some requests in flight, and one PASS of the step function
(``ModelRunner.step``) over given tokens: an optional first step that brings prompt portions (beside decoded tokens of the other
requests, where there are any), then ``tokens`` decode steps of all requests. The tokens are given, nothing is fed back, so that two
implementations can be compared step by step. Requests' earlier tokens (``context_*``) went through the engine before the pass, as in
serving; a pass starts at the same positions every time, so it can be repeated on the same state.

``exact`` states every family plainly in float64 (dense masks, recurrences token by token, experts one by one).

Fields of a case: model, size, dtype; requests; context_lo/hi: tokens already cached (spread over the requests, geometrically);
prompting: how many requests bring a prompt portion in the first step, of prompt_lo/hi tokens (the others bring one token each);
tokens: decode steps behind it; graphs: the engine's ``cuda_graphs``; sampling: rows of ``top_p`` draw a token from logits in hand
before the first step.
"""
from __future__ import annotations

import hashlib
import json
import math
import os
import shutil
import tempfile
from pathlib import Path

import torch

# ------------------------------------------------------------------------------------------------------------ models
# Layer sizes are those of bench.py (full layer counts for Qwen2, eight layer runs for the others).


def _qwen2(size: str) -> dict:
    W, ff, layers, H = {"0.5b": (896, 4864, 24, 14), "1.5b": (1536, 8960, 28, 12)}[size]
    return {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "vocab_size": 151936, "hidden_size": W, "intermediate_size": ff,
            "num_hidden_layers": layers, "num_attention_heads": H, "num_key_value_heads": 2, "rms_norm_eps": 1e-6, "rope_theta": 1000000.0,
            "tie_word_embeddings": True, "max_position_embeddings": 32768, "use_sliding_window": False, "hidden_act": "silu"}


def _luvutar(size: str) -> dict:
    W, H, G, d, r, qr, kr, win, ff = {"0.5b-like": (896, 14, 2, 64, 32, 384, 256, 1024, 3584),
                                      "3b-like": (2048, 16, 4, 128, 64, 768, 512, 2048, 8192)}[size]
    layers = []
    for i in range(8):
        if i % 2:
            m = {"heads": H, "dim": d, "rot_dim": r, "vdim": d, "q_rank": qr, "kv_rank": kr, "scale": (d + r) ** -0.5,
                 "mask": {"size": win}, "rot": {"base": 10000.0, "dims": r}}
        else:
            m = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "bias_max": 4096, "q_temp": {"coef": 0.1, "every": 1024}}
            if i % 4 == 2:
                m["kv_from"] = i - 2
        layers.append({"type": "latent_attention" if i % 2 else "attention", "mixer": m, "mlp": {"kind": "dense", "ff": ff}})
    return {"architecture": "Luvutar", "vocab": 32768, "width": W, "norm": {"eps": 1e-6}, "streams": 4, "layers": layers}


def _zepalorn(size: str) -> dict:
    W, H, G, d, win, chunk, dh, dd, dv, sh, sv, ns, sg, ff = {
        "0.5b-like": (896, 14, 2, 64, 1024, 2048, 8, 64, 128, 28, 64, 128, 2, 2432),
        "3b-like": (2048, 16, 4, 128, 2048, 4096, 16, 128, 128, 64, 64, 128, 8, 5504)}[size]
    scaling = {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}
    mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    layers = []
    for i in range(8):
        if i % 4 in (0, 3):
            layers.append({"type": "channel_delta", "mixer": {"heads": dh, "kv_heads": dh, "dim": dd, "vdim": dv, "conv": 4}, "mlp": mlp})
        elif i % 4 == 1:
            m = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "mask": {"size": win, "keep_first": 4},
                 "rot": {"base": 1000000.0, "dims": d, "scaling": scaling}}
            layers.append({"type": "attention", "mixer": m, "mlp": mlp})
        else:
            left = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "conv": 4, "softcap": 50.0, "mask": {"size": chunk},
                    "rot": {"base": 10000.0, "dims": d // 2, "scaling": scaling}}
            right = {"heads": sh, "vdim": sv, "state": ns, "groups": sg, "norm_groups": sg, "conv": 4}
            layers.append({"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": mlp})
    return {"architecture": "Zepalorn", "vocab": 32768, "width": W, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}, "layers": layers}


def _mufotar(size: str) -> dict:
    W, dh, dg, dd, dv, H, G, d, ci, ns, rk, E, ident, top, eff, sff, ff = {
        "1b-like": (1024, 8, 4, 128, 128, 8, 2, 128, 2048, 16, 64, 16, 2, 4, 512, 768, 2816),
        "3b-like": (2048, 16, 8, 128, 128, 16, 4, 128, 4096, 16, 128, 32, 2, 4, 768, 2432, 5504)}[size]
    moe = {"kind": "moe", "expert": {"ff": eff}, "router": {"experts": E, "identity": ident, "top": top}, "shared": {"ff": sff}}
    delta = {"heads": dh, "kv_heads": dg, "dim": dd, "vdim": dv, "conv": 4}
    pair = {"left": {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "rot": {"base": 100000.0, "dims": d}},
            "right": {"inner": ci, "state": ns, "dt_rank": rk, "conv": 4}, "left_scale": 1.0, "right_scale": 1.0}
    layers = []
    for i in range(8):
        if i % 4 == 2:
            layers.append({"type": "parallel", "mixer": pair, "mlp": moe, **({"weights_of": 2} if i > 2 else {})})
        else:
            layers.append({"type": "delta", "mixer": delta, "mlp": {"kind": "dense", "ff": ff} if i % 4 == 0 else moe})
    return {"architecture": "Mufotar", "vocab": 32768, "width": W, "norm": {"eps": 1e-6}, "logit_softcap": 30.0, "layers": layers}


def _memilorn(size: str) -> dict:
    W, mh, md, mv, H, G, d, lh, ld, rank, E, top, eff, sff = {
        "1b-like": (1024, 8, 128, 128, 8, 2, 128, 8, 128, 256, 16, 4, 512, 768),
        "3b-like": (2048, 16, 128, 128, 16, 4, 128, 16, 128, 512, 32, 4, 768, 2432)}[size]
    moe = {"kind": "moe", "expert": {"ff": eff, "limit": 7.0}, "router": {"experts": E, "top": top}, "shared": {"ff": sff, "limit": 7.0}}
    memory = {"type": "mlstm", "mixer": {"heads": mh, "dim": md, "vdim": mv, "gate_cap": 15.0}, "mlp": moe}
    attention = {"type": "attention", "mixer": {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "softcap": 30.0,
                                                "rot": {"base": 100000.0, "dims": d}}, "mlp": moe}
    latent = {"type": "latent_attention", "mixer": {"heads": lh, "dim": ld, "vdim": ld, "kv_rank": rank, "scale": ld ** -0.5}, "mlp": moe}
    return {"architecture": "Memilorn", "vocab": 32768, "width": W, "norm": {"eps": 1e-6}, "layers": [attention, memory, memory, latent, memory],
            "loop": {"start": 1, "stop": 4, "times": 2}}


def _sinorax(size: str) -> dict:
    W, H, G, d, win, ff = {"0.5b-like": (896, 14, 2, 64, 1024, 7296), "3b-like": (2048, 16, 4, 128, 1024, 8256)}[size]
    heads = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5}
    mlp = {"kind": "dense", "ff": ff}
    full = {"type": "attention", "mixer": {**heads, "rot": {"dims": d, "base": 1000000.0, "scaling": {"factor": 2.0}}}, "mlp": mlp}
    windowed = {"type": "attention_2", "mixer": {**heads, "mask": {"size": win}}, "mlp": mlp}
    return {"architecture": "Sinorax", "vocab": 32768, "width": W, "norm": {"eps": 1e-6},
            "embedding": {"bigram": {"buckets": 65521, "mul_prev": 8191, "mul_cur": 127}}, "logit_scale": 0.25, "logit_softcap": 30.0,
            "layers": [full] * 4 + [windowed] * 4}


def _putelix(size: str) -> dict:
    W, H, G, d, chunk, lh, ld, lv, ff, E, top, eff, sff = {
        "1b-like": (1024, 8, 2, 128, 2048, 8, 128, 128, 4224, 16, 4, 512, 768),
        "3b-like": (2048, 16, 4, 128, 4096, 16, 128, 128, 8256, 32, 4, 768, 2432)}[size]
    left = {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "softcap": 50.0, "bias_max": 1024, "mask": {"size": chunk}}
    right = {"heads": lh, "dim": ld, "vdim": lv, "decay": [1.0 - 2.0 ** -(1 + 8 * (h + 1) / lh) for h in range(lh)]}
    moe = {"kind": "moe", "expert": {"ff": eff}, "router": {"experts": E, "top": top}, "shared": {"ff": sff}}
    return {"architecture": "Putelix", "vocab": 32768, "width": W, "norm": {"eps": 1e-6}, "max_positions": 8192,
            "layers": [{"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": moe if i % 2 else {"kind": "dense", "ff": ff}}
                       for i in range(8)]}


_MODELS = {"qwen2": _qwen2, "luvutar": _luvutar, "zepalorn": _zepalorn, "mufotar": _mufotar, "memilorn": _memilorn, "sinorax": _sinorax,
           "putelix": _putelix}


def _config(case: dict) -> dict:
    return _MODELS[case["model"]](case["size"])


def _vocab(cfg: dict) -> int:
    return cfg.get("vocab") or cfg["vocab_size"]


def _folder(cfg: dict) -> Path:
    """A model folder with random weights, bfloat16 on disk; written once per machine, the same numbers every time. ``_settle`` takes
    some tensors from the plain draw to what training makes of them."""
    from llm_infrence_engine_b200.weights.random_init import write_random_model

    base = Path(tempfile.gettempdir()) / f"llmie_models_{os.getuid()}"
    to = base / hashlib.sha256(json.dumps(cfg, sort_keys=True).encode()).hexdigest()[:16]
    if not to.is_dir():
        base.mkdir(exist_ok=True)
        work = Path(tempfile.mkdtemp(dir=base))
        write_random_model(cfg, work, seed=0, store_dtype="bfloat16")
        about, data = _open(work, shared=True)
        for name, a in about.items():
            _settle(name, data[a["data_offsets"][0]:a["data_offsets"][1]].view(torch.bfloat16))
        try:
            os.rename(work, to)
        except OSError:   # another process was first
            shutil.rmtree(work, ignore_errors=True)
    return to


def _settle(name: str, t: torch.Tensor) -> None:
    """Without these a deep stack of random weights multiplies its own roundings from layer to layer, and outputs of the same precision
    would lie further apart than outputs of a lower one do in a trained model."""
    if name.endswith(("o_proj.weight", "down_proj.weight")):
        t.mul_(0.02)      # a layer adds a little to the stream (the embedding's rows are as small)
    elif name.endswith((".ls1", ".ls2")):
        t.mul_(0.01)      # likewise: layer scales start small
    elif name.endswith(".mlp.router"):
        t.mul_(4.0)       # a router decides: it seldom hangs on the last bit ...
    elif ".mlp.e" in name and name.endswith(".down"):
        t.mul_(0.03125)   # ... and where it does, the two experts are much alike
    elif name.endswith(".pb"):
        t.fill_(-7.0)     # sigmoid attention starts at minus the logarithm of its window


# ------------------------------------------------------------------------------------------------------------ cases
def _case(name, model, size, requests, context=(0, 0), prompting=0, prompt=(0, 0), tokens=0, dtype="bfloat16", graphs=True, sampling=""):
    return {"name": name, "model": model, "size": size, "dtype": dtype, "requests": requests, "context_lo": context[0], "context_hi": context[1],
            "prompting": prompting, "prompt_lo": prompt[0], "prompt_hi": prompt[1], "tokens": tokens, "graphs": graphs, "sampling": sampling}


def listed() -> list:
    return [
        # one user, one token: the latency of a chat answer
        _case("chat_token", "qwen2", "0.5b", 1, context=(517, 517), tokens=1),
        # the benchmark's headline: eight long conversations
        _case("long_decode", "qwen2", "0.5b", 8, context=(8130, 8188), tokens=2),
        # a busy server with a larger model: 64 ragged conversations, sampled with top-p
        _case("busy_decode", "qwen2", "1.5b", 64, context=(128, 2048), tokens=2, sampling="top_p"),
        # the benchmark's prompt
        _case("prompt_2048", "qwen2", "0.5b", 1, prompting=1, prompt=(2048, 2048)),
        # continuous batching: three prompts arrive while 29 conversations go on
        _case("mixed_batch", "qwen2", "0.5b", 32, context=(130, 2300), prompting=3, prompt=(301, 1100)),
        # the 32-bit path, used for parity: three short prompts and their first tokens, engine defaults
        _case("float32_short", "qwen2", "0.5b", 3, prompting=3, prompt=(33, 190), tokens=2, dtype="float32", graphs=False),
        # the other families: prompts of one to many requests, and the tokens that follow
        _case("luvutar_four", "luvutar", "0.5b-like", 4, prompting=4, prompt=(200, 901), tokens=8),
        _case("zepalorn_prompt", "zepalorn", "3b-like", 1, prompting=1, prompt=(2048, 2048), tokens=8),
        _case("mufotar_eight", "mufotar", "1b-like", 8, prompting=8, prompt=(64, 511), tokens=8),
        _case("memilorn_pair", "memilorn", "1b-like", 2, prompting=2, prompt=(700, 1301), tokens=4),
        _case("sinorax_long", "sinorax", "3b-like", 1, prompting=1, prompt=(4003, 4003), tokens=4),
        _case("putelix_many", "putelix", "1b-like", 16, prompting=16, prompt=(20, 300), tokens=16),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(case: dict) -> float:
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def draw(rng) -> dict:
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.randrange(12)
        if kind < 3:      # decode steps of Qwen2
            lo = _log(rng, 20, 8000)
            c = _case("", "qwen2", rng.choice(["0.5b", "1.5b"]), _log(rng, 1, 64), context=(lo, _log(rng, lo, 8188)), tokens=rng.randint(1, 3),
                      sampling=rng.choice(["", "top_p"]))
            if c["requests"] * c["context_hi"] > 140000:
                continue
        elif kind == 3:   # a prompt or a few
            n, hi = rng.randint(1, 4), _log(rng, 20, 4096)
            c = _case("", "qwen2", rng.choice(["0.5b", "1.5b"]), n, prompting=n, prompt=(_log(rng, 20, hi), hi))
        elif kind == 4:   # prompts arriving among conversations
            n, hi, lo = rng.randint(2, 48), _log(rng, 40, 1500), _log(rng, 20, 2000)
            c = _case("", "qwen2", "0.5b", n, context=(lo, _log(rng, lo, 2500)), prompting=rng.randint(1, min(4, n)), prompt=(_log(rng, 30, hi), hi))
        elif kind == 5:   # 32-bit
            n, hi = rng.randint(1, 6), _log(rng, 17, 300)
            c = _case("", "qwen2", "0.5b", n, prompting=n, prompt=(_log(rng, 16, hi), hi), tokens=rng.randint(0, 3), dtype="float32", graphs=False)
        else:             # the other families
            model = ("luvutar", "zepalorn", "mufotar", "memilorn", "sinorax", "putelix")[kind - 6]
            n, hi = _log(rng, 1, 16), _log(rng, 20, 4096)
            size = rng.choice({"luvutar": ["0.5b-like", "3b-like"], "zepalorn": ["0.5b-like", "3b-like"],
                               "sinorax": ["0.5b-like", "3b-like"]}.get(model, ["1b-like", "3b-like"]))
            c = _case("", model, size, n, prompting=n, prompt=(_log(rng, 17, hi), hi), tokens=rng.randint(0, 16))
            if n * hi > 8192:
                continue
        del c["name"]
        if _cost(c) <= most:
            return c


# ------------------------------------------------------------------------------------------------------------ the requests of a case
def _spread(lo: int, hi: int, n: int) -> list:
    """n lengths from lo to hi, geometric, in a fixed mixed order."""
    if n == 0:
        return []
    v = [hi if n == 1 else int(round(lo * (hi / lo) ** (i / (n - 1)))) if lo else 0 for i in range(n)]
    step = next(s for s in (5, 7, 11, 13, 1) if math.gcd(s, n) == 1)
    return [v[(i * step) % n] for i in range(n)]


def _plan(case: dict):
    """(tokens in the cache, tokens of the first step or 0 without one) per request."""
    n, p = case["requests"], case["prompting"]
    ctx = [0] * p + _spread(case["context_lo"], case["context_hi"], n - p)
    first = _spread(case["prompt_lo"], case["prompt_hi"], p) + [1] * (n - p) if p else [0] * n
    return ctx, first


def _sequences(case: dict, seed: int) -> list:
    """Every request's tokens: those in the cache, those of the first step, one per decode step."""
    g = torch.Generator().manual_seed(int(seed))
    ctx, first = _plan(case)
    vocab = _vocab(_config(case))
    return [torch.randint(0, vocab, (c + f + case["tokens"],), generator=g).tolist() for c, f in zip(ctx, first)]


def _logits_in_hand(case: dict, seed: int) -> torch.Tensor:
    """What a server has when it samples: a row of float32 logits per request (of a model's spread: a few likely tokens, a long tail)."""
    g = torch.Generator("cuda").manual_seed(int(seed))
    return torch.randn(case["requests"], _vocab(_config(case)), generator=g, device="cuda") * 2.5


def prepare(case: dict, seed: int):
    """An engine with the model loaded, its decode graph captured and the requests' earlier tokens run; the tokens to come as lists."""
    from llm_infrence_engine_b200.engine import Engine, StepEntry
    from llm_infrence_engine_b200.sampling import SamplingParams

    ctx, first = _plan(case)
    seqs = _sequences(case, seed)
    n, page = case["requests"], 16
    longest = max(len(s) for s in seqs) + 1
    pages = sum(-(-(len(s) + 1) // page) for s in seqs) + 1
    eng = Engine(str(_folder(_config(case))), dtype=case["dtype"], block_size=page, num_blocks=pages, max_seqs=n, max_len=longest,
                 max_num_batched_tokens=8192, cuda_graphs=case["graphs"])
    if case["tokens"] and case["graphs"]:
        eng.warmup([n])
    for i, s in enumerate(seqs):
        eng.cache.admit(i)
        eng.cache.reserve(i, 0, len(s))
        for at in range(0, ctx[i], 2048):
            eng.runner.step([StepEntry(i, s[at:min(at + 2048, ctx[i])], at)])
    state = {"case": case, "engine": eng, "ctx": ctx, "first": first, "seqs": seqs, "entry": StepEntry}
    if case["sampling"]:
        state["logits"] = _logits_in_hand(case, seed)
        state["params"] = [SamplingParams(temperature=0.8, top_p=0.95, seed=seed + i) for i in range(n)]
    return state


def run(state):
    """The tokens drawn from the logits in hand (if the case samples), then the float32 logits of every step [requests, vocab]."""
    case, eng, Entry = state["case"], state["engine"], state["entry"]
    step, out = eng.runner.step, {}
    if case["sampling"]:
        out["tokens"] = eng.sampler.sample_device(state["logits"], state["params"], state["ctx"])
    at, seqs, logits = list(state["ctx"]), state["seqs"], []
    if case["prompting"]:
        logits.append(step([Entry(i, s[a:a + f], a, (f - 1,)) for i, (s, a, f) in enumerate(zip(seqs, at, state["first"]))]))
        at = [a + f for a, f in zip(at, state["first"])]
    for t in range(case["tokens"]):
        got = step([Entry(i, s[a:a + 1], a, (0,)) for i, (s, a) in enumerate(zip(seqs, at))])
        logits.append(got if t + 1 == case["tokens"] else got.clone())   # a captured step's logits are overwritten by the next
        at = [a + 1 for a in at]
    out["logits"] = logits
    return out


# ------------------------------------------------------------------------------------------------------------ work, tolerance
def work(case: dict) -> dict:
    """Weights once per step (of the experts, those that a step's tokens can choose), the cached keys that a token sees once per step,
    states in and out, logits out; operations of the products and of the attention's visible pairs."""
    cfg, n, size = _config(case), case["requests"], 4 if case["dtype"] == "float32" else 2
    vocab = _vocab(cfg)
    ctx, first = _plan(case)
    steps = ([list(zip(ctx, first))] if case["prompting"] else []) + [[(c + f + t, 1) for c, f in zip(ctx, first)] for t in range(case["tokens"])]
    layers, width = _layer_sizes(cfg)
    flops = nbytes = 0.0
    for batch in steps:
        tok = sum(f for _, f in batch)
        nbytes += size * vocab * width + 4.0 * n * vocab
        flops += 2.0 * n * vocab * width
        seen_weights = set()
        for L in layers:
            flops += 2.0 * tok * (L["matrix"] + L["expert"] * L["top"]) + tok * L["state_flops"]
            if L["id"] not in seen_weights:
                seen_weights.add(L["id"])
                nbytes += size * (L["matrix"] + L["expert"] * min(L["experts"], tok * L["top"]))
            nbytes += 8.0 * n * L["state"]
            for c, f in batch:
                seen = min(c + f, L["window"]) if L["window"] else c + f
                nbytes += size * seen * L["row"]
                pairs = sum(min(c + 1 + i, L["window"] or 1 << 30) for i in range(f))
                flops += L["pair_flops"] * pairs
    if case["sampling"]:
        nbytes += 4.0 * n * vocab
    return {"bytes": nbytes, "flops": flops}


def _layer_sizes(cfg: dict):
    """Per layer run: matrix weights, experts (weights of one, how many, chosen), cache row entries per token, window, operations per visible
    pair, state entries and their operations per token."""
    out = []
    if "hidden_size" in cfg:
        W, H, G = cfg["hidden_size"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
        d = W // H
        for i in range(cfg["num_hidden_layers"]):
            out.append(dict(id=i, matrix=W * d * (2 * H + 2 * G) + 3 * W * cfg["intermediate_size"], expert=0, experts=0, top=0, row=2 * G * d,
                            window=0, pair_flops=4 * H * d, state=0, state_flops=0))
        return out, W
    W = cfg["width"]
    order = list(range(len(cfg["layers"])))
    if cfg.get("loop"):
        lp = cfg["loop"]
        order = order[:lp["stop"]] + order[lp["start"]:lp["stop"]] * (lp["times"] - 1) + order[lp["stop"]:]
    for i in order:
        layer = cfg["layers"][i]
        L = dict(id=layer.get("weights_of", i), matrix=0, expert=0, experts=0, top=0, row=0, window=0, pair_flops=0, state=0, state_flops=0)
        m = layer["mixer"]
        for part in ([m["left"], m["right"]] if layer["type"] == "parallel" else [m]):
            if "inner" in part:             # selective scan
                c, s = part["inner"], part["state"]
                L["matrix"] += W * 3 * c + c * (2 * part["dt_rank"] + 2 * s)
                L["state"] += c * s
                L["state_flops"] += 6 * c * s
            elif "groups" in part:          # state-space mixer
                inner = part["heads"] * part["vdim"]
                L["matrix"] += W * (3 * inner + 2 * part["groups"] * part["state"])
                L["state"] += inner * part["state"]
                L["state_flops"] += 5 * inner * part["state"]
            elif layer["type"] in ("channel_delta", "delta", "mlstm") or "decay" in part:
                H, D, V = part["heads"], part["dim"], part.get("vdim", part["dim"])
                G = part.get("kv_heads", H)
                L["matrix"] += W * (2 * G * D + 3 * H * V)
                L["state"] += H * D * V
                L["state_flops"] += 8 * H * D * V
            elif "kv_rank" in part:         # latent attention: cached are the latent and the rotated part
                H, D, V, r = part["heads"], part["dim"], part.get("vdim", part["dim"]), part.get("rot_dim", 0)
                qr, kr = part.get("q_rank", 0), part["kv_rank"]
                L["matrix"] += (W * qr + qr * H * (D + r) if qr else W * H * D) + W * (kr + r) + kr * H * (D + V) + W * H * V * (2 if qr else 1)
                L["row"] += kr + r
                L["window"] = (part.get("mask") or {}).get("size", 0)
                L["pair_flops"] += 2 * H * (D + r + V)
            else:
                H, G, D, V = part["heads"], part["kv_heads"], part["dim"], part["vdim"]
                L["matrix"] += W * (H * D + H * V) + (0 if "kv_from" in part else W * G * (D + V))
                L["row"] += G * (D + V)
                L["window"] = (part.get("mask") or {}).get("size", 0)
                L["pair_flops"] += 2 * H * (D + V)
        mlp = layer["mlp"]
        if mlp["kind"] == "dense":
            L["matrix"] += W * mlp["ff"] * (2 if cfg["architecture"] in ("Luvutar", "Sinorax", "Putelix") else 3)
        else:
            L["matrix"] += W * mlp["router"]["experts"] + 3 * W * mlp["shared"]["ff"]
            L["expert"], L["experts"], L["top"] = 3 * W * mlp["expert"]["ff"], mlp["router"]["experts"], mlp["router"]["top"]
        out.append(L)
    return out, W


def tolerance(case: dict) -> dict:
    """Relative error of a step's logits, about four times what the engine's lie off the float64 ones: 2e-6 to 3e-6 in float32; in bfloat16
    0.003 to 0.017 by family, so two of its kind differ by up to 0.025. Draws from given logits are the same but for ties."""
    return {"rel": 1e-5} if case["dtype"] == "float32" else {"rel": 0.03, "differ": 0.01}


# ------------------------------------------------------------------------------------------------------------ the same in float64
def exact(case: dict, seed: int):
    W = _Weights(_folder(_config(case)))
    cfg = _config(case)
    ctx, first = _plan(case)
    rows = []
    for c, f, s in zip(ctx, first, _sequences(case, seed)):
        wanted = ([c + f - 1] if case["prompting"] else []) + [c + f + t for t in range(case["tokens"])]
        rows.append(_logits(cfg, W, torch.tensor(s, device="cuda"), wanted))
    out = {"logits": list(torch.stack(rows, dim=1))}
    if case["sampling"]:
        out["tokens"] = None
    return out


def _open(folder: Path, shared: bool = False):
    """(what a folder's file says of its tensors by name, their bytes)"""
    file = folder / "model.safetensors"
    raw = torch.from_file(str(file), shared=shared, size=os.path.getsize(file), dtype=torch.uint8)
    head = int.from_bytes(bytes(raw[:8].tolist()), "little")
    about = json.loads(bytes(raw[8:8 + head].tolist()))
    about.pop("__metadata__", None)
    return about, raw[8 + head:]


class _Weights(dict):
    """A folder's tensors by name, float64 on the device, read when first asked for."""

    def __init__(self, folder: Path):
        self.about, self.data = _open(folder)

    def __contains__(self, name):
        return name in self.about

    def __missing__(self, name):
        a, (lo, hi) = self.about[name], self.about[name]["data_offsets"]
        kind = {"BF16": torch.bfloat16, "F32": torch.float32}[a["dtype"]]
        self[name] = self.data[lo:hi].clone().view(kind).view(a["shape"]).cuda().double()
        return self[name]


def _logits(cfg, W, ids, wanted):
    kind = cfg.get("architecture")
    fn = {None: _qwen2_stream, "Luvutar": _luvutar_stream, "Zepalorn": _zepalorn_stream, "Mufotar": _mufotar_stream, "Memilorn": _memilorn_stream,
          "Sinorax": _sinorax_stream, "Putelix": _putelix_stream}[kind]
    x = fn(cfg, W, ids)[torch.tensor(wanted, device=ids.device)]
    if kind is None:
        return _rms(x, cfg["rms_norm_eps"]) * W["model.norm.weight"] @ W["model.embed_tokens.weight"].T
    eps = cfg["norm"]["eps"]
    if kind == "Luvutar":
        return _rms(x, eps) * (1 + W["final.norm"]) @ W["head"].T
    if kind == "Sinorax":
        return _cap(_dyt(x, W, "final.norm") @ W["head"].T * cfg["logit_scale"], cfg["logit_softcap"])
    if kind == "Putelix":
        return _rms(x, eps) * W["final.norm"] @ W["embed"].T
    return _cap(_ln(x, W["final.norm"], eps, W["final.norm.b"] if kind == "Mufotar" else 0.0) @ W["embed"].T, cfg.get("logit_softcap"))


# small pieces
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _ln(x, w, eps, b=0.0):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w + b


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu_tanh(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _softplus(x):
    return torch.where(x > 30, x, torch.log1p(torch.exp(x.clamp(max=30))))


def _cap(x, cap):
    return cap * torch.tanh(x / cap) if cap else x


def _dyt(x, W, name):
    return torch.tanh(W[name + ".alpha"] * x) * W[name] + W[name + ".b"]


def _conv(u, w, b=0.0):
    taps, T = w.shape[1], u.shape[0]
    padded = torch.cat([u.new_zeros(taps - 1, u.shape[1]), u])
    return sum(padded[j:j + T] * w[:, j] for j in range(taps)) + b


def _turn(x, freqs, neighbours=False, mult=1.0, back=False):
    """x [T, heads, D]: pairs of the first 2 * len(freqs) entries turn by position * frequency; neighbours: pairs (2i, 2i + 1), else halves."""
    T, half = x.shape[0], len(freqs)
    a = torch.arange(T, device=x.device, dtype=x.dtype)[:, None] * torch.tensor(freqs, device=x.device, dtype=x.dtype)
    c, s = (torch.cos(a) * mult)[:, None], (torch.sin(-a if back else a) * mult)[:, None]
    at = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if neighbours else (slice(0, half), slice(half, 2 * half))
    u, v, out = x[..., at[0]], x[..., at[1]], x.clone()
    out[..., at[0]], out[..., at[1]] = u * c - v * s, v * c + u * s
    return out


def _freqs(base, dims, factor=1.0):
    return [base ** (-2.0 * i / dims) / factor for i in range(dims // 2)]


def _attend(q, k, v, scale, scores=None, seen=None, weigh=None):
    """q [T, H, D], k [T, G, D], v [T, G, V] -> [T, H, V]. ``scores(s, i, j)``: what happens to the scaled scores [H, rows, T]; ``seen(i, j)``:
    which of the keys not later are seen; ``weigh(s)``: masked scores (-inf) to weights, softmax if not given."""
    T, per = q.shape[0], q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(per, 1).permute(1, 2, 0), v.repeat_interleave(per, 1).transpose(0, 1)
    j, out = torch.arange(T, device=q.device)[None, :], []
    for at in range(0, T, 1024):
        i = torch.arange(at, min(at + 1024, T), device=q.device)[:, None]
        s = torch.matmul(q[at:at + 1024].transpose(0, 1), k) * scale
        if scores:
            s = scores(s, i, j)
        ok = (j <= i) if seen is None else (j <= i) & seen(i, j)
        s = s.masked_fill_(~ok, -math.inf)
        out.append(torch.matmul((weigh or (lambda z: torch.softmax(z, -1)))(s), v).transpose(0, 1))
    return torch.cat(out)


def _with_sink(sink):
    def weigh(s):
        top = torch.maximum(s.max(-1, keepdim=True).values, sink[:, None, None])
        e = torch.exp(s - top)
        return e / (e.sum(-1, keepdim=True) + torch.exp(sink[:, None, None] - top))
    return weigh


def _far_bias(rel, T, far):
    """[heads, T]: the bias of a distance."""
    rows = rel.shape[0]
    half = rows // 2
    b = [n if n < half else min(rows - 1, half + int(math.floor(math.log(n / half) / math.log(far / half) * (rows - half)))) for n in range(T)]
    return rel[torch.tensor(b, device=rel.device)].T


def _moe(h, W, p, idx, weights, unit, on_input=False):
    """sum of the chosen experts' results, weighted (or of their results on the weighted input)."""
    out = torch.zeros_like(h)
    for e in idx.unique().tolist():
        t, place = torch.nonzero(idx == e, as_tuple=True)
        w = weights[t, place][:, None]
        out.index_add_(0, t, unit(w * h[t], f"{p}.e{e}") if on_input else w * unit(h[t], f"{p}.e{e}"))
    return out


# one function per family: tokens to the residual stream behind the last layer
def _qwen2_stream(cfg, W, ids):
    H, G, eps, T = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["rms_norm_eps"], len(ids)
    D = cfg["hidden_size"] // H
    f = _freqs(cfg["rope_theta"], D)
    x = W["model.embed_tokens.weight"][ids]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}"
        h = _rms(x, eps) * W[p + ".input_layernorm.weight"]
        q, k, v = ((h @ W[f"{p}.self_attn.{n}_proj.weight"].T + W[f"{p}.self_attn.{n}_proj.bias"]).view(T, -1, D) for n in "qkv")
        x = x + _attend(_turn(q, f), _turn(k, f), v, D ** -0.5).reshape(T, -1) @ W[p + ".self_attn.o_proj.weight"].T
        h = _rms(x, eps) * W[p + ".post_attention_layernorm.weight"]
        x = x + (_silu(h @ W[p + ".mlp.gate_proj.weight"].T) * (h @ W[p + ".mlp.up_proj.weight"].T)) @ W[p + ".mlp.down_proj.weight"].T
    return x


def _luvutar_stream(cfg, W, ids):
    eps, T, S = cfg["norm"]["eps"], len(ids), cfg["streams"]
    xs = W["embed"][ids][None].repeat(S, 1, 1)
    kept = {}

    def attention(h, i, m, p):
        H, D, src = m["heads"], m["dim"], m.get("kv_from", i)
        steps = torch.div(torch.arange(T, device=h.device) + 1, m["q_temp"]["every"], rounding_mode="floor")
        q = (h @ W[p + ".q"].T).view(T, H, D) * (1 + m["q_temp"]["coef"] * torch.log(steps.double() + 1))[:, None, None]
        if src == i:
            kept[i] = tuple((h @ W[f"{p}.{n}"].T).view(T, m["kv_heads"], D) for n in "kv")
        bias = _far_bias(W[p + ".rel"], T, m["bias_max"])
        o = _attend(q, *kept[src], m["scale"], scores=lambda s, a, b: s + bias[:, (a - b).clamp(min=0)])
        return (o * torch.sigmoid(h @ W[p + ".g"].T)[:, :, None]).reshape(T, -1) @ W[p + ".o"].T

    def latent(h, m, p):
        H, D, r, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        f = _freqs(m["rot"]["base"], m["rot"]["dims"])
        q = (_rms(h @ W[p + ".dq"].T, eps) * W[p + ".dq.norm"] @ W[p + ".uq"].T).view(T, H, D + r)
        dkv = h @ W[p + ".dkv"].T
        c = _rms(dkv[:, :rank], eps) * W[p + ".dkv.norm"]
        q = torch.cat([q[..., :D], _turn(q[..., D:], f, True)], -1)
        k = torch.cat([(c @ W[p + ".uk"].T).view(T, H, D), _turn(dkv[:, None, rank:], f, True).expand(T, H, r)], -1)
        o = _attend(q, k, (c @ W[p + ".uv"].T).view(T, H, -1), m["scale"], seen=lambda a, b: a - b < m["mask"]["size"],
                    weigh=_with_sink(W[p + ".sink"]) if p + ".sink" in W else None)
        return o.reshape(T, -1) * torch.sigmoid(h @ W[p + ".g"].T) @ W[p + ".o"].T

    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}"
        for n in (1, 2):
            u = _rms(torch.einsum("s,stw->tw", W[f"{p}.hc{n}.in"], xs), eps) * (1 + W[f"{p}.norm{n}"])
            if n == 2:
                y = _gelu_tanh(u @ W[p + ".mlp.up"].T) @ W[p + ".mlp.down"].T
            else:
                y = latent(u, layer["mixer"], p + ".mix") if "kv_rank" in layer["mixer"] else attention(u, i, layer["mixer"], p + ".mix")
            xs = torch.einsum("sr,stw->rtw", W[f"{p}.hc{n}.mix"], xs) + W[f"{p}.hc{n}.out"][:, None, None] * y
    return xs.sum(0)


def _scaled_freqs(rot):
    dims, base, sc = rot["dims"], rot["base"], rot["scaling"]

    def dim_of(turns):
        return dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))

    lo, hi = max(math.floor(dim_of(sc["fast"])), 0), min(math.ceil(dim_of(sc["slow"])), dims - 1)
    out = []
    for i, f in enumerate(_freqs(base, dims)):
        ramp = min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
        out.append(f / sc["factor"] * ramp + f * (1 - ramp))
    return out, 0.1 * math.log(sc["factor"]) + 1.0


def _delta_rule(q, k, v, beta, decay):
    """q, k [T, H, D], v [T, H, V], beta [T, H], decay [T, H, D or 1]: S <- decay S; S += k (beta (v - S^T k))^T; o = S^T q."""
    S, out = q.new_zeros(q.shape[1], q.shape[2], v.shape[2]), []
    for t in range(len(q)):
        S = decay[t][:, :, None] * S
        u = beta[t][:, None] * (v[t] - (k[t][:, None] @ S)[:, 0])
        S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
        out.append((q[t][:, None] @ S)[:, 0])
    return torch.stack(out)


def _delta_inputs(h, m, W, p):
    T, D = len(h), m["dim"]
    q, k, v = (_silu(_conv(h @ W[f"{p}.{n}"].T, W[f"{p}.{n}.conv"])) for n in "qkv")
    q, k, v = q.view(T, -1, D), k.view(T, -1, D), v.view(T, m["heads"], -1)
    per = m["heads"] // q.shape[1]
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * D ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    return q.repeat_interleave(per, 1), k.repeat_interleave(per, 1), v, torch.sigmoid(h @ W[p + ".b"].T)


def _zepalorn_stream(cfg, W, ids):
    eps, T = cfg["norm"]["eps"], len(ids)
    x = W["embed"][ids] * cfg["embedding"]["scale"]

    def attention(h, m, p, chunked):
        y = [h @ W[f"{p}.{n}"].T for n in "qkv"]
        if chunked:
            y = [_conv(a, W[f"{p}.{n}.conv"]) for a, n in zip(y, "qkv")]
        q, k, v = (a.view(T, -1, m["dim"]) for a in y)
        if chunked:
            q, k = _rms(q, eps) * W[p + ".q.norm"], _rms(k, eps) * W[p + ".k.norm"]
        f, mult = _scaled_freqs(m["rot"])
        q, k = _turn(q, f, chunked, mult), _turn(k, f, chunked, mult)
        size, keep = m["mask"]["size"], m["mask"].get("keep_first", 0)
        seen = (lambda a, b: a // size == b // size) if chunked else (lambda a, b: (a - b < size) | (b < keep))
        return _attend(q, k, v, m["scale"], lambda s, a, b: _cap(s, m.get("softcap")), seen).reshape(T, -1) @ W[p + ".o"].T

    def delta(h, m, p):
        H = m["heads"]
        q, k, v, beta = _delta_inputs(h, m, W, p)
        dt = _softplus((h @ W[p + ".a1"].T) @ W[p + ".a2"].T + W[p + ".dt_bias"]).view(T, H, -1)
        o = _delta_rule(q, k, v, beta, torch.exp(-torch.exp(W[p + ".A_log"])[:, None] * dt))
        gate = torch.sigmoid((h @ W[p + ".g1"].T) @ W[p + ".g2"].T).view(T, H, -1)
        return (_rms(o, eps) * W[p + ".norm"] * gate).reshape(T, -1) @ W[p + ".o"].T

    def state_space(h, m, p):
        H, V, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        inner, y = H * V, []
        z, xbc, dt = (h @ W[p + ".in"].T).split([inner, inner + 2 * G * N, H], -1)
        xbc = _silu(_conv(xbc, W[p + ".conv"], W[p + ".conv.b"]))
        u = xbc[:, :inner].view(T, H, V)
        B, C = (a.view(T, G, N).repeat_interleave(H // G, 1) for a in xbc[:, inner:].split(G * N, -1))
        dt = _softplus(dt + W[p + ".dt_bias"])
        a = torch.exp(-torch.exp(W[p + ".A_log"]) * dt)
        S = h.new_zeros(H, N, V)
        for t in range(T):
            S = torch.baddbmm(a[t][:, None, None] * S, (dt[t][:, None] * B[t])[:, :, None], u[t][:, None])
            y.append((C[t][:, None] @ S)[:, 0] + W[p + ".D"][:, None] * u[t])
        y = torch.stack(y).reshape(T, inner) * _silu(z)
        y = _rms(y.view(T, m["norm_groups"], -1), eps).reshape(T, inner) * W[p + ".norm"]
        return y @ W[p + ".o"].T

    for i, layer in enumerate(cfg["layers"]):
        p, m, limit = f"l{i}", layer["mixer"], layer["mlp"]["limit"]
        h = _ln(x, W[p + ".norm1"], eps)
        if layer["type"] == "channel_delta":
            y = delta(h, m, p + ".mix")
        elif layer["type"] == "attention":
            y = attention(h, m, p + ".mix", False)
        else:
            y = 0.5 * (_rms(attention(h, m["left"], p + ".mix.left", True), eps) * W[p + ".mix.left.out"]
                       + _rms(state_space(h, m["right"], p + ".mix.right"), eps) * W[p + ".mix.right.out"])
        x = x + _ln(y, W[p + ".norm1b"], eps)
        h = _ln(x, W[p + ".norm2"], eps)
        g, u = (h @ W[p + ".mlp.gate"].T).clamp(max=limit), (h @ W[p + ".mlp.up"].T).clamp(-limit, limit)
        x = x + _ln((g * torch.sigmoid(1.702 * g) * (u + 1)) @ W[p + ".mlp.down"].T, W[p + ".norm2b"], eps)
    return x


def _mufotar_stream(cfg, W, ids):
    eps, T = cfg["norm"]["eps"], len(ids)
    x = W["embed"][ids]

    def unit(act):
        return lambda h, p: (act(h @ W[p + ".gate"].T) * (h @ W[p + ".up"].T)) @ W[p + ".down"].T

    def attention(h, m, p):
        q, k, v = ((h @ W[f"{p}.{n}"].T).view(T, -1, m["dim"]) for n in "qkv")
        f = _freqs(m["rot"]["base"], m["rot"]["dims"])
        q, k = _turn(_rms(q, eps) * W[p + ".q.norm"], f), _turn(_rms(k, eps) * W[p + ".k.norm"], f)
        return _attend(q, k, v, m["scale"]).reshape(T, -1) @ W[p + ".o"].T

    def scan(h, m, p):
        inner, N, R = m["inner"], m["state"], m["dt_rank"]
        u, z = (h @ W[p + ".in"].T).split(inner, -1)
        u = _silu(_conv(u, W[p + ".conv"], W[p + ".conv.b"]))
        r, B, C = (u @ W[p + ".x"].T).split([R, N, N], -1)
        dt = _softplus(r @ W[p + ".dt"].T + W[p + ".dt.b"])
        A, S, y = -torch.exp(W[p + ".A_log"]), h.new_zeros(inner, N), []
        for t in range(T):
            S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * B[t]
            y.append(S @ C[t] + W[p + ".D"] * u[t])
        return (torch.stack(y) * _silu(z)) @ W[p + ".o"].T

    def delta(h, m, p):
        q, k, v, beta = _delta_inputs(h, m, W, p)
        g = torch.exp(-torch.exp(W[p + ".A_log"]) * _softplus(h @ W[p + ".a"].T + W[p + ".dt_bias"]))
        o = _rms(_delta_rule(q, k, v, beta, g[:, :, None]), eps) * W[p + ".norm"]
        return o.reshape(T, -1) * _silu(h @ W[p + ".g"].T) @ W[p + ".o"].T

    def experts(h, mlp, p):
        s = torch.softmax(h @ W[p + ".router"].T, -1)
        idx = torch.topk(s + W[p + ".correction"] if p + ".correction" in W else s, mlp["router"]["top"], -1).indices
        w = s.gather(1, idx)
        E, one = mlp["router"]["experts"], unit(_silu)
        out = _moe(h, W, p, idx, w / (w.sum(-1, keepdim=True) + 1e-20), lambda a, name: one(a, name) if int(name.rsplit("e", 1)[1]) < E else a)
        return out + one(h, p + ".shared")

    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{layer.get('weights_of', i)}", layer["mixer"]
        h = _ln(x, W[p + ".norm1"], eps, W[p + ".norm1.b"])
        if layer["type"] == "delta":
            y = delta(h, m, p + ".mix")
        else:
            y = m["left_scale"] * attention(h, m["left"], p + ".mix.left") + m["right_scale"] * scan(h, m["right"], p + ".mix.right")
        x = x + y + (unit(_gelu_tanh)(h, p + ".mlp") if layer["mlp"]["kind"] == "dense" else experts(h, layer["mlp"], p + ".mlp"))
    return x


def _memilorn_stream(cfg, W, ids):
    eps, T = cfg["norm"]["eps"], len(ids)
    first = W["embed"][ids]
    x = first.clone()

    def memory(h, m, p):
        H, D, cap = m["heads"], m["dim"], m["gate_cap"]
        q, k, v = ((h @ W[f"{p}.{n}"].T).view(T, H, -1) for n in "qkv")
        q = q * D ** -0.5
        i_log = _cap(h @ W[p + ".i"].T + W[p + ".i.b"], cap)
        f_log = -_softplus(-_cap(h @ W[p + ".f"].T + W[p + ".f.b"], cap))
        S, n, top, out = h.new_zeros(H, D, v.shape[2]), h.new_zeros(H, D), h.new_zeros(H), []
        for t in range(T):
            new = torch.maximum(f_log[t] + top, i_log[t])
            keep, take = torch.exp(f_log[t] + top - new)[:, None], torch.exp(i_log[t] - new)[:, None] * k[t]
            S = torch.baddbmm(keep[:, :, None] * S, take[:, :, None], v[t][:, None])
            n, top = keep * n + take, new
            out.append((q[t][:, None] @ S)[:, 0] / (torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6)[:, None])
        o = _rms(torch.stack(out), eps).reshape(T, -1) * W[p + ".norm"] * torch.sigmoid(h @ W[p + ".g"].T)
        return o @ W[p + ".o"].T

    def latent(h, m, p):
        H = m["heads"]
        c = _rms(h @ W[p + ".dkv"].T, eps) * W[p + ".dkv.norm"]
        o = _attend((h @ W[p + ".q"].T).view(T, H, -1), (c @ W[p + ".uk"].T).view(T, H, -1), (c @ W[p + ".uv"].T).view(T, H, -1), m["scale"])
        return (o * torch.sigmoid(h @ W[p + ".g"].T)[:, :, None]).reshape(T, -1) @ W[p + ".o"].T

    def talking(h, m, p):
        q, k, v = ((h @ W[f"{p}.{n}"].T).view(T, -1, m["dim"]) for n in "qkv")
        f = _freqs(m["rot"]["base"], m["rot"]["dims"])
        o = _attend(_turn(q, f, True), _turn(k, f, True), v, m["scale"], weigh=_with_sink(W[p + ".sink"]),
                    scores=lambda s, a, b: torch.einsum("hg,gij->hij", W[p + ".talk"], _cap(s, m["softcap"])))
        return (o * torch.sigmoid(h @ W[p + ".g"].T)[:, :, None]).reshape(T, -1) @ W[p + ".o"].T

    def unit(limit):
        def fn(a, p):
            g, u = (a @ W[p + ".gate"].T).clamp(max=limit), (a @ W[p + ".up"].T).clamp(-limit, limit)
            return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ W[p + ".down"].T
        return fn

    order = list(range(len(cfg["layers"])))
    a, b = cfg["loop"]["start"], cfg["loop"]["stop"]
    order = [(i, False) for i in order[:b]] + [(i, i == a) for i in order[a:b]] * (cfg["loop"]["times"] - 1) + [(i, False) for i in order[b:]]
    for i, again in order:
        layer, p = cfg["layers"][i], f"l{i}"
        x = x + first if again else x
        mixer = {"mlstm": memory, "latent_attention": latent, "attention": talking}[layer["type"]]
        x = x + W[p + ".ls1"] * mixer(_ln(x, W[p + ".norm1"], eps), layer["mixer"], p + ".mix")
        h, mlp = _ln(x, W[p + ".norm2"], eps), layer["mlp"]
        s = torch.sigmoid(h @ W[p + ".mlp.router"].T)
        idx = torch.topk(s, mlp["router"]["top"], -1).indices
        y = _moe(h, W, p + ".mlp", idx, s.gather(1, idx), unit(mlp["expert"]["limit"]), on_input=True)
        x = x + W[p + ".ls2"] * (y + unit(mlp["shared"]["limit"])(h, p + ".mlp.shared"))
    return x


def _sinorax_stream(cfg, W, ids):
    T, big = len(ids), cfg["embedding"]["bigram"]
    rows = torch.cat([ids.new_tensor([big["buckets"]]), (ids[:-1] * big["mul_prev"] + ids[1:] * big["mul_cur"]) % big["buckets"]])
    x = W["embed"][ids] + W["bigram"][rows]

    def turned(h, m, p):
        q, k, v = ((h @ W[f"{p}.{n}"].T + W[f"{p}.{n}.b"]).view(T, -1, m["dim"]) for n in "qkv")
        f, plain = _freqs(m["rot"]["base"], m["rot"]["dims"], m["rot"]["scaling"]["factor"]), _freqs(m["rot"]["base"], m["vdim"])
        o = _attend(_turn(q, f), _turn(k, f), _turn(v, plain), m["scale"])
        return _turn(o, plain, back=True).reshape(T, -1) @ W[p + ".o"].T + W[p + ".o.b"]

    def sigmoid(h, m, p):
        q, k, v = ((h @ W[f"{p}.{n}"].T).view(T, -1, m["dim"]) for n in "qkv")
        r1, r2, pb = (W[f"{p}.{n}"][:, None, None] for n in ("r1", "r2", "pb"))
        o = _attend(q, k, v, m["scale"], lambda s, a, b: s - r1 * torch.log(1 + r2 * (a - b).clamp(min=0)) + pb,
                    lambda a, b: a - b < m["mask"]["size"], torch.sigmoid)
        return o.reshape(T, -1) @ W[p + ".o"].T

    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}"
        y = (turned if layer["type"] == "attention" else sigmoid)(_dyt(x, W, p + ".norm1"), layer["mixer"], p + ".mix")
        x = x + _dyt(y, W, p + ".norm1b")
        h = _dyt(x, W, p + ".norm2") @ W[p + ".mlp.up"].T
        x = x + _dyt(0.5 * h * (1 + torch.erf(h / math.sqrt(2))) @ W[p + ".mlp.down"].T, W, p + ".norm2b")
    return x


def _putelix_stream(cfg, W, ids):
    eps, T = cfg["norm"]["eps"], len(ids)
    x = W["embed"][ids] + W["pos"][:T]

    def attention(h, m, p):
        D, size = m["dim"], m["mask"]["size"]
        q, k = (h @ W[f"{p}.{n}"].T + W[f"{p}.{n}.b"] for n in "qk")
        v = k.view(T, -1, D)
        q, k = ((_rms(a, eps) * W[f"{p}.{n}.norm"]).view(T, -1, D) for a, n in ((q, "q"), (k, "k")))
        bias = _far_bias(W[p + ".rel"], T, m["bias_max"])
        o = _attend(q, k, v, m["scale"], lambda s, a, b: _cap(s, m["softcap"]) + bias[:, (a - b).clamp(min=0)], lambda a, b: a // size == b // size)
        return (o * torch.sigmoid(h @ W[p + ".g"].T)[:, :, None]).reshape(T, -1) @ W[p + ".o"].T + W[p + ".o.b"]

    def linear(h, m, p):
        q, k, v = (_silu(h @ W[f"{p}.{n}"].T).view(T, m["heads"], -1) for n in "qkv")
        decay, S, out = torch.tensor(m["decay"], device=h.device, dtype=h.dtype)[:, None, None], h.new_zeros(m["heads"], m["dim"], m["vdim"]), []
        for t in range(T):
            S = torch.baddbmm(decay * S, k[t][:, :, None], v[t][:, None])
            out.append((q[t][:, None] @ S)[:, 0])
        return _rms(torch.stack(out).reshape(T, -1), eps) * W[p + ".norm"] * torch.sigmoid(h @ W[p + ".g"].T) @ W[p + ".o"].T

    def unit(a, p):
        return (_silu(a @ W[p + ".gate"].T) * (a @ W[p + ".up"].T)) @ W[p + ".down"].T

    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}", layer["mixer"], layer["mlp"]
        y = 0.5 * (_rms(attention(x, m["left"], p + ".mix.left"), eps) * W[p + ".mix.left.out"]
                   + _rms(linear(x, m["right"], p + ".mix.right"), eps) * W[p + ".mix.right.out"])
        x = x + _rms(y, eps) * W[p + ".norm1"]
        p += ".mlp"
        if mlp["kind"] == "dense":
            y = (x @ W[p + ".up"].T).clamp(min=0) ** 2 @ W[p + ".down"].T
        else:
            values, idx = torch.topk(x @ W[p + ".router"].T + W[p + ".router.b"], mlp["router"]["top"], -1)
            y = _moe(x, W, p, idx, torch.softmax(values, -1), unit) + unit(x, p + ".shared") * torch.sigmoid(x @ W[p + ".shared.sg"].T)
        x = x + _rms(y, eps) * W[f"l{i}.norm2"]
    return x

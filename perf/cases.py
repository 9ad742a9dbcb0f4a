"""The work that users of this library have it do, as cases to be timed: requests served through `Engine.alloc`,
`Engine.step` and `Engine.free` (a prompt step, then decode steps, as `Engine.generate`, `bin/trace_run` and the C API
drive them), and the choice of tokens through `Engine.sampler`.

A pass is a whole batch of requests: slots are taken, the prompts go in, the given number of tokens is decoded and the
slots are given back.  The tokens that follow the prompts are fixed (as in a replayed trace), so that two
implementations see the same sequences, and all logits asked for are the outcome.  The model (weights, cache of 40,960
tokens, captured graphs) is what a server keeps; its weights are the same for every seed, the tokens are not.

Models: the Llama shapes that the benchmark has (1B, 3B, 8B), and the Fuvipel, Fovirax and Mavinex decoders of its
design comparison (8 layers; recurrent layers, mixtures of experts, windows and latents).  The Pusunex, Bogupel and Goridra
decoders run on the same products, attention and mixtures and are not repeated here.
"""
from __future__ import annotations

import math
import zlib

import torch

from oracle_engine_b200.config.base import get_architecture
from oracle_engine_b200.engine.batch import SequenceStep
from oracle_engine_b200.engine.engine import Engine
from oracle_engine_b200.sampling.params import GenParams

MAX_TOKENS = 40960          # what the cache holds; each sequence's count is rounded up to a page of 64
MAX_SEQ = 8192
SLOTS = 64
VOCAB = {"llama": 128256, "fuvipel": 32000, "fovirax": 32000, "mavinex": 32000}
LLAMA = {"1b": dict(hidden_size=2048, num_hidden_layers=16, num_attention_heads=32, head_dim=64, intermediate_size=8192),
         "3b": dict(hidden_size=3072, num_hidden_layers=28, num_attention_heads=24, head_dim=128, intermediate_size=8192),
         "8b": dict(hidden_size=4096, num_hidden_layers=32, num_attention_heads=32, head_dim=128, intermediate_size=14336,
                    tie_word_embeddings=False)}
LAYERS = 8                  # of the other designs


# ------------------------------------------------------------------------------------------------------- the cases
def listed():
    def llama(name, shape, **kw):
        return dict({"name": name, "kind": "serve", "design": "llama", "shape": shape, "dtype": "bfloat16", "want": "last",
                     "portion": 0}, **kw)

    def design(name, which, **kw):
        return dict({"name": name, "kind": "serve", "design": which, "shape": "2048", "dtype": "bfloat16", "want": "last",
                     "portion": 0}, **kw)

    return [
        # the defaults of the command line (temperature 0.7, top-k 40, top-p 0.9, penalty 1.15): what follows every step
        {"name": "sample-8", "kind": "sample", "rows": 8, "vocab": 128256, "draws": 16, "temperature": 0.7, "top_k": 40,
         "top_p": 0.9, "penalty": 1.15},
        # one user's short question: the latency of a small prompt and of one token after another
        llama("chat-3b", "3b", batch=1, lo=41, hi=41, steps=24),
        # the headline: eight sequences of 512 tokens decoding
        llama("batch8-3b", "3b", batch=8, lo=512, hi=512, steps=48),
        # a full server: 64 sequences of unequal length
        llama("batch64-3b", "3b", batch=64, lo=33, hi=480, steps=16),
        # one prompt of 2,048 tokens, its first token wanted (time to first token)
        llama("prompt-3b", "3b", batch=1, lo=2048, hi=2048, steps=0),
        # documents of up to 4,096 tokens read by the largest model, a few tokens of answer each
        llama("documents-8b", "8b", batch=7, lo=366, hi=4019, steps=4),
        # a prompt that enters in portions beside the decoding rows of other requests
        llama("portions-3b", "3b", batch=5, lo=150, hi=1500, steps=0, portion=192),
        # texts scored: the logits of every position
        llama("score-1b", "1b", batch=3, lo=97, hi=640, steps=0, want="all"),
        # the true 32-bit path
        llama("float32-1b", "1b", batch=3, lo=37, hi=210, steps=8, dtype="float32"),
        # recurrent layers: a page of text read by one user and continued
        design("fuvipel", "fuvipel", batch=1, lo=1111, hi=1111, steps=24),
        # a mixture of experts beside attention with a window longer than most prompts, one user
        design("fovirax", "fovirax", batch=1, lo=1500, hi=1500, steps=24),
        # selective scans, attention over latents and a mixture, a small batch of unequal requests
        design("mavinex", "mavinex", batch=8, lo=50, hi=900, steps=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sample", "decode", "decode", "decode", "prompt", "portion", "score", "float32", "design", "design", "design"])
    if kind == "sample":
        rows = _log(rng, 1, 64)
        return {"kind": "sample", "rows": rows, "vocab": rng.choice([32000, 128256]), "draws": rng.randint(4, max(4, min(32, 500 // rows))),
                "temperature": rng.choice([0.0, 0.7, 1.0]), "top_k": rng.choice([0, 40]), "top_p": rng.choice([0.9, 0.95, 1.0]),
                "penalty": rng.choice([1.0, 1.15])}
    case = {"kind": "serve", "design": "llama", "shape": rng.choice(["1b", "3b", "3b", "8b"]), "dtype": "bfloat16", "want": "last",
            "portion": 0, "batch": _log(rng, 1, 64), "lo": 0, "hi": 0, "steps": rng.randint(8, 32)}
    most = 12000                            # prompt tokens of a batch
    if kind == "design":
        case.update(design=rng.choice(["fuvipel", "fovirax", "mavinex"]), shape=rng.choice(["1024", "2048", "3072"]),
                    batch=_log(rng, 1, 32), dtype=rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32"]))
        most = 4500 if case["dtype"] == "bfloat16" else 700
    elif kind == "prompt":
        case.update(batch=_log(rng, 1, 8), steps=rng.randint(0, 2))
    elif kind == "portion":
        case.update(batch=rng.randint(2, 12), portion=rng.choice([64, 100, 192, 256, 500]), steps=0)
    elif kind == "score":
        case.update(want="all", batch=_log(rng, 1, 6), steps=0, shape=rng.choice(["1b", "3b"]))
        most = 1500
    elif kind == "float32":
        case.update(dtype="float32", shape=rng.choice(["1b", "3b"]), batch=_log(rng, 1, 16))
        most = 900 if case["shape"] == "1b" else 400
    hi = _log(rng, 16, min(4096, most / case["batch"] if case["portion"] == 0 else 3000)) if most / case["batch"] > 16 else 16
    case.update(lo=max(1, int(hi * rng.choice([0.1, 0.5, 1.0]))), hi=hi)
    if case["portion"] and case["hi"] < 2 * case["portion"]:
        case["hi"] = 2 * case["portion"] + rng.randint(1, 500)
    if case["portion"]:
        case["lo"] = max(1, case["hi"] // 10)
    return case


# --------------------------------------------------------------------------------------------- requests of a case
def _requests(case, seed):
    """(prompts, tokens that follow them): lists of ids, one per sequence.  The lengths are the case's own."""
    spread = torch.Generator().manual_seed(12345 + case["batch"] * 7 + case["hi"])
    n = torch.randint(case["lo"], case["hi"] + 1, (case["batch"],), generator=spread).tolist()
    n[-1] = case["hi"]                      # the longest is there
    extra = case["steps"]
    if case["portion"]:
        n[:-1] = [max(1, min(v, case["lo"] * 2)) for v in n[:-1]]
        extra = -(-n[-1] // case["portion"])
    g = torch.Generator().manual_seed(seed * 1000003 + 17)
    vocab = VOCAB[case["design"]]
    return ([torch.randint(0, vocab, (v,), generator=g).tolist() for v in n],
            [torch.randint(0, vocab, (extra,), generator=g).tolist() for _ in n])


# ------------------------------------------------------------------------------------------------------ the models
def _raw_config(design, shape):
    if design == "llama":
        return dict(dict(architectures=["LlamaForCausalLM"], vocab_size=VOCAB["llama"], num_key_value_heads=8, rms_norm_eps=1e-5,
                         rope_theta=500000.0, rope_scaling={"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0,
                                                            "high_freq_factor": 4.0, "original_max_position_embeddings": 8192},
                         max_position_embeddings=131072, tie_word_embeddings=True, bos_token_id=128000, eos_token_id=128001),
                    **LLAMA[shape])
    width = int(shape)
    heads, ff = width // 128, (2 * width // 3 + 63) // 64 * 64
    by_wave = {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}
    base = {"vocab": VOCAB[design], "width": width}
    if design == "fuvipel":
        delta = {"type": "delta", "mlp": {"kind": "dense", "ff": 4 * width},
                 "mixer": {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4}}
        par = {"type": "parallel", "mlp": {"kind": "dense", "ff": 4 * width},
               "mixer": {"left": {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                  "rot": {"dims": 64, "base": 1000000.0}},
                         "right": {"heads": width // 64, "dim": 64, "rank": 64}}}
        return dict(base, architecture="Fuvipel", norm={"eps": 1e-6}, layers=[par if i % 4 == 3 else delta for i in range(LAYERS)])
    att = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
           "rot": {"dims": 128, "base": 500000.0, "scaling": by_wave}}
    moe = {"kind": "moe", "expert": {"ff": ff}, "router": {"experts": 8, "top": 2}}
    if design == "fovirax":
        layer = {"type": "parallel", "mlp": dict(moe, shared={"ff": 2 * ff}),
                 "mixer": {"left": dict(att, softcap=50.0), "left_scale": 0.5, "right_scale": 0.5,
                           "right": {"heads": heads, "dim": 64, "vdim": 128, "rot": {"dims": 64, "base": 10000.0},
                                     "decay": [1.0 - 2.0 ** (-5.0 - 3.0 * i / max(1, heads - 1)) for i in range(heads)]}}}
        return dict(base, architecture="Fovirax", norm={"eps": 1e-6}, residual_mult=1.0, layers=[layer] * LAYERS)
    par = {"type": "parallel", "mlp": moe,
           "mixer": {"left": att, "right": {"inner": 2 * width, "state": 16, "dt_rank": width // 16, "conv": 4}}}
    lat = {"type": "latent_attention", "mlp": moe,
           "mixer": {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 192, "scale": 192 ** -0.5, "mask": {"size": 1024},
                     "rot": {"dims": 64, "base": 10000.0, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
    return dict(base, architecture="Mavinex", norm={"eps": 1e-5}, embedding={"scale": 1.0}, postln_alpha=2.0,
                layers=[lat if i % 2 else par for i in range(LAYERS)])


class _Weights:
    """Random weights by tensor name, the same for the engine and for `exact`: the initialisations that models of these kinds
    are trained from.  Embeddings N(0, 1), matrices N(0, 0.02) and those that add to the residual stream divided by
    sqrt(2 layers), gains near one, step sizes and decays over the ranges that scans are started with.  Routers choose as
    trained ones do, with a margin: every token's embedding leans, for each layer, towards two of its experts."""

    def __init__(self, layers, decls=(), experts=0):
        self.layers, self.experts = layers, experts
        self.decls = {d.name: tuple(d.shape) for d in decls}

    class _Info:
        def __init__(self, shape):
            self.dtype, self.shape = torch.bfloat16, shape

    def names(self):
        return self.decls.keys()

    def info(self, name):
        return self._Info(self.decls[name])

    def read(self, name):
        return self.make(name, self.decls[name])

    def make(self, name, shape):
        g = torch.Generator(device="cuda").manual_seed(zlib.crc32(name.encode()) + 1)
        last = name.removesuffix(".weight").rsplit(".", 1)[-1]
        if last == "A_log":
            if len(shape) == 2:
                return torch.arange(1, shape[1] + 1, device="cuda").log().expand(shape).to(torch.bfloat16).contiguous()
            return (torch.rand(shape, generator=g, device="cuda") * 15 + 1).log().to(torch.bfloat16)
        if last == "dt_bias" or name.endswith("dt.b"):
            dt = torch.exp(torch.rand(shape, generator=g, device="cuda") * math.log(100.0) + math.log(1e-3))
            return torch.log(torch.expm1(dt)).to(torch.bfloat16)
        if ".mu." in name:
            return torch.rand(shape, generator=g, device="cuda").to(torch.bfloat16)
        if last == "w0":
            return (torch.rand(shape, generator=g, device="cuda") * 5 - 6).to(torch.bfloat16)
        t = torch.randn(shape, generator=g, device="cuda", dtype=torch.bfloat16)
        if last == "embed" and self.experts:
            t = t.float()
            for i in range(self.layers):
                two = torch.rand(shape[0], self.experts, generator=g, device="cuda").topk(2).indices
                t += 5.5 * self.make(f"l{i}.mlp.router", (self.experts, shape[1])).float()[two].sum(1)
            return t.to(torch.bfloat16)
        if last in ("embed", "embed_tokens", "sink"):
            return t
        if last.startswith("conv") or last == "b" and "conv" in name:
            return t * (0.5 if len(shape) == 2 else 0.1)
        if last == "u":
            return t * 0.3
        if last in ("D", "out", "ls1", "ls2") or len(shape) == 1 and ("norm" in last and self.plain_gain(name)):
            return 1 + 0.1 * t
        if len(shape) == 1:
            return 0.1 * t
        if last in ("o", "down", "o_proj", "down_proj"):
            return t * (0.02 / math.sqrt(2 * self.layers))
        return t * 0.02

    plain = True            # the norms multiply by the gain itself, not by 1 + gain

    def plain_gain(self, name):
        return self.plain or name.endswith(("q.norm", "k.norm", "dkv.norm"))


def _weights(design, shape, decls=()):
    w = _Weights(LLAMA[shape]["num_hidden_layers"] if design == "llama" else LAYERS, decls, 8 if design in ("fovirax", "mavinex") else 0)
    w.plain = design in ("llama", "fuvipel")
    return w


_MODEL = [None, None]       # the one engine that is kept, as by a server: (what it is, the engine)


def _engine(design, shape, dtype):
    key = (design, shape, dtype)
    if _MODEL[0] != key:
        _MODEL[:] = [None, None]
        torch.cuda.empty_cache()
        raw = _raw_config(design, shape)
        arch = get_architecture(raw.get("architecture") or raw["architectures"][0])
        _MODEL[:] = [key, Engine(arch.config_cls.from_dict(raw), arch, lambda model: _weights(design, shape, model.tensors()),
                                 dtype=dtype, max_tokens=MAX_TOKENS, max_seq_len=MAX_SEQ, n_slots=SLOTS)]
    return _MODEL[1]


# ------------------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    if case["kind"] == "sample":
        # any engine has the sampler; logits with the spread of a trained head's and a few candidates that stand out
        engine = _engine("fuvipel", "1024", "bfloat16")
        g = torch.Generator(device="cuda").manual_seed(seed)
        shape = (case["draws"], case["rows"], case["vocab"])
        logits = torch.randn(shape, generator=g, device="cuda") * 2.5
        logits += torch.where(torch.rand(shape, generator=g, device="cuda") < 2e-4, 6.0, 0.0)
        host = torch.Generator().manual_seed(seed)
        return {"case": case, "engine": engine, "logits": logits, "row": torch.empty_like(logits[0]),
                "seed": seed, "prompts": torch.randint(0, case["vocab"], (case["rows"], 100), generator=host).tolist(),
                "tokens": torch.empty(shape[:2], dtype=torch.int32, device="cuda"),
                "params": GenParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"],
                                    repeat_penalty=case["penalty"])}
    engine = _engine(case["design"], case["shape"], case["dtype"])
    prompts, after = _requests(case, seed)
    vocab, B = VOCAB[case["design"]], case["batch"]
    rows = sum(len(p) for p in prompts) if case["want"] == "all" else B
    state = {"case": case, "engine": engine, "prompts": prompts, "after": after}
    empty = lambda *shape: torch.empty(shape + (vocab,), dtype=torch.float32, device="cuda")       # noqa: E731
    if case["portion"]:
        state.update(first=empty(B - 1), rest=empty(len(after[0]), B - 1), late=empty(1))
    else:
        state.update(first=empty(rows), rest=empty(case["steps"], B))
    return state


def run(state):
    case, engine = state["case"], state["engine"]
    if case["kind"] == "sample":
        return _run_sample(state)
    prompts, after = state["prompts"], state["after"]
    slots = [engine.alloc() for _ in prompts]
    try:
        if case["portion"]:
            return _run_portions(state, slots)
        want_all = case["want"] == "all"
        logits = engine.step([SequenceStep(s, p, list(range(len(p))) if want_all else [len(p) - 1]) for s, p in zip(slots, prompts)])
        state["first"].copy_(logits)
        for i in range(case["steps"]):
            state["rest"][i].copy_(engine.step([SequenceStep(s, [a[i]], [0]) for s, a in zip(slots, after)]))
        return {"first": state["first"], "rest": state["rest"]} if case["steps"] else {"first": state["first"]}
    finally:
        for s in slots:
            engine.free(s)


def _run_portions(state, slots):
    engine, prompts, after, size = state["engine"], state["prompts"], state["after"], state["case"]["portion"]
    state["first"].copy_(engine.step([SequenceStep(s, p, [len(p) - 1]) for s, p in zip(slots[:-1], prompts)]))
    long = prompts[-1]
    for i, lo in enumerate(range(0, len(long), size)):
        piece = long[lo:lo + size]
        done = lo + len(piece) == len(long)
        step = [SequenceStep(s, [a[i]], [0]) for s, a in zip(slots[:-1], after)]
        step.append(SequenceStep(slots[-1], piece, [len(piece) - 1] if done else []))
        logits = engine.step(step)
        state["rest"][i].copy_(logits[:len(slots) - 1])
        if done:
            state["late"].copy_(logits[len(slots) - 1:])
    return {"first": state["first"], "rest": state["rest"], "late": state["late"]}


def _run_sample(state):
    engine, params, rows = state["engine"], state["params"], state["case"]["rows"]
    slots = [engine.alloc() for _ in range(rows)]
    try:
        for i, s in enumerate(slots):
            engine.sampler.start_sequence(s, state["seed"] + i, state["prompts"][i], params)
        row_slot = torch.tensor(slots, dtype=torch.int32, device="cuda")
        for k in range(state["case"]["draws"]):
            state["row"].copy_(state["logits"][k])          # the sampler works in place; a step's logits are fresh each time
            engine.sampler.sample(state["row"], row_slot, params, state["tokens"][k])
        return state["tokens"]
    finally:
        for s in slots:
            engine.free(s)


# ------------------------------------------------------------------------------------------------------------ work
def _counts(case):
    """(weights that every token uses, weights of the mixtures' experts altogether, chosen share of those, cached values per
    token, (query-key and value products per pair, window) per attention layer, values of recurrent state per sequence)."""
    raw = _raw_config(case["design"], case["shape"])
    if case["design"] == "llama":
        D, L, H, hd, F = (raw[k] for k in ("hidden_size", "num_hidden_layers", "num_attention_heads", "head_dim", "intermediate_size"))
        return L * (D * hd * (2 * H + 16) + 3 * D * F), 0, 1.0, L * 16 * hd, [(2 * H * hd, 0)] * L, 0
    D, every, experts, cached, pairs, kept = raw["width"], 0, 0, 0, [], 0
    for lay in raw["layers"]:
        m, f = lay["mixer"], lay["mlp"]
        if f["kind"] == "dense":
            every += 2 * D * f["ff"]
        else:
            experts += f["router"]["experts"] * 3 * D * f["expert"]["ff"]
            every += 3 * D * (f.get("shared") or {"ff": 0})["ff"] + D * f["router"]["experts"]
        if lay["type"] == "delta":
            H, G = m["heads"], m["kv_heads"]
            every += D * 128 * (2 * G + 3 * H)
            kept += H * 128 * 128
            continue
        a = m.get("left", m)
        window = (a.get("mask") or {}).get("size", 0)
        if lay["type"] == "latent_attention":
            H = a["heads"]
            every += D * (H * (128 + 64) + 256 + H * 128 + H) + 192 * H * 256
            cached += 256
            pairs.append((H * (256 + 64), window))
            continue
        H, G = a["heads"], a["kv_heads"]
        every += D * 128 * (2 * H + 2 * G + (H if case["design"] == "mavinex" else 0))
        cached += 2 * G * 128
        pairs.append((2 * H * 128, window))
        r = m["right"]
        if case["design"] == "fuvipel":
            every += 5 * D * D + 2 * D * r["rank"]
            kept += r["heads"] * 64 * 64
        elif case["design"] == "fovirax":
            every += D * r["heads"] * (2 * 64 + 3 * 128)
            kept += r["heads"] * 64 * 128
        else:
            C = r["inner"]
            every += 3 * D * C + C * (2 * r["dt_rank"] + 2 * r["state"])
            kept += C * r["state"]
    return every, experts, 0.25, cached, pairs, kept


def work(case):
    if case["kind"] == "sample":
        n = case["draws"] * case["rows"] * case["vocab"]
        return {"bytes": 4.0 * n, "flops": 10.0 * n}
    every, experts, share, cached, pairs, kept = _counts(case)
    size = 2 if case["dtype"] == "bfloat16" else 4
    vocab, D = VOCAB[case["design"]], int(_raw_config(case["design"], case["shape"]).get("width") or LLAMA[case["shape"]]["hidden_size"])
    prompts, after = _requests(case, 0)
    total = {"bytes": 0.0, "flops": 0.0}

    def step(runs, wanted):                 # runs: (first position, tokens) per sequence
        tokens = sum(n for _, n in runs)
        used = experts * min(1.0, 1.0 - (1.0 - share) ** tokens)
        total["bytes"] += size * (every + used + (vocab * D if wanted else 0) + tokens * (D + cached)) + 4.0 * wanted * vocab
        total["bytes"] += sum(8.0 * kept + size * cached * p for p, _ in runs)
        total["flops"] += 2.0 * tokens * (every + share * experts) + 2.0 * wanted * vocab * D + 6.0 * tokens * kept
        for p, n in runs:
            for width, window in pairs:
                seen = sum(min(q + 1, window or q + 1) for q in range(p, p + n))
                total["flops"] += 2.0 * width * seen

    lens = [len(p) for p in prompts]
    if case["portion"]:
        step([(0, n) for n in lens[:-1]], len(lens) - 1)
        for i, lo in enumerate(range(0, lens[-1], case["portion"])):
            step([(n + i, 1) for n in lens[:-1]] + [(lo, min(case["portion"], lens[-1] - lo))], len(lens) - 1)
        return total
    step([(0, n) for n in lens], sum(lens) if case["want"] == "all" else len(lens))
    for i in range(case["steps"]):
        step([(n + i, 1) for n in lens], len(lens))
    return total


def tolerance(case):
    if case["kind"] == "sample":
        return {"rel": 0.0, "differ": 0.01}     # a draw that falls on the edge between two tokens
    # against 64 bits the logits were off by 0.0022 to 0.0067 (bfloat16) and 6e-7 to 1.5e-6 (float32)
    return {"rel": 1e-5, "max": 2e-4} if case["dtype"] == "float32" else {"rel": 0.02, "max": 0.2}


# --------------------------------------------------------------------------------------------- the models in 64 bits
F64 = torch.float64


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _frequencies(dims, base, sc):
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device="cuda") / dims)
    if not sc:
        return f, 1.0
    if "low" in sc:                          # by wavelength
        s = ((sc["original"] * f / (2 * math.pi)) - sc["low"]) / (sc["high"] - sc["low"])
        s = s.clamp(0, 1)
        return (1 - s) * f / sc["factor"] + s * f, 1.0
    place = lambda t: dims * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(base))       # noqa: E731
    lo, hi = max(math.floor(place(sc["fast"])), 0), min(math.ceil(place(sc["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F64, device="cuda") - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def _turn(x, rot, halves):
    """x [T, heads, n] of one sequence, its first rot.dims dimensions turned by the position."""
    f, m = _frequencies(rot["dims"], rot["base"], rot.get("scaling"))
    ang = torch.arange(x.shape[0], dtype=F64, device="cuda")[:, None] * f
    c, s = m * torch.cos(ang)[:, None], m * torch.sin(ang)[:, None]
    d = rot["dims"]
    a, b = (x[..., :d // 2], x[..., d // 2:d]) if halves else (x[..., 0:d:2], x[..., 1:d:2])
    u, v = a * c - b * s, b * c + a * s
    return torch.cat([torch.cat([u, v], -1) if halves else torch.stack([u, v], -1).flatten(-2), x[..., d:]], -1)


def _attend(q, k, v, scale, window=0, cap=0.0, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv] of one sequence -> [T, H, dv].  sink: a score without a value per head."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(T, device="cuda")
    hidden = i[None, :] > i[:, None]
    if window:
        hidden |= i[:, None] - i[None, :] >= window
    out = torch.empty(T, H, v.shape[2], dtype=F64, device="cuda")
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h] @ k[:, g].T) * scale
        s = (cap * torch.tanh(s / cap) if cap else s).masked_fill(hidden, -math.inf)
        if sink is None:
            p = torch.softmax(s, -1)
        else:
            top = torch.maximum(s.max(-1, keepdim=True).values, sink[h])
            e = torch.exp(s - top)
            p = e / (e.sum(-1, keepdim=True) + torch.exp(sink[h] - top))
        out[:, h] = p @ v[:, g]
    return out


def _conv(x, taps):
    """Causal convolution per channel of one sequence: x [T, C], taps [C, K], the last one the current token's."""
    K = taps.shape[1]
    x = torch.cat([x.new_zeros(K - 1, x.shape[1]), x])
    return sum(x[j:j + x.shape[0] - K + 1] * taps[:, j] for j in range(K))


def _moe(h, w, pre, f, D, bias):
    E, ff, top = f["router"]["experts"], f["expert"]["ff"], f["router"]["top"]
    z = h @ w(pre + "router", E, D).T
    if bias:
        z = z + w(pre + "router.b", E)
    val, idx = torch.topk(z, top)
    wt = torch.zeros_like(z).scatter_(1, idx, torch.softmax(val, -1))

    def expert(x, p, n):
        return (_silu(x @ w(p + "gate", n, D).T) * (x @ w(p + "up", n, D).T)) @ w(p + "down", D, n).T
    out = torch.zeros_like(h)
    for e in range(E):
        rows = torch.nonzero(wt[:, e]).flatten()
        out[rows] += wt[rows, e:e + 1] * expert(h[rows], f"{pre}e{e}.", ff)
    if f.get("shared"):
        out += torch.sigmoid(h @ w(pre + "shared.sg", 1, D).T) * expert(h, pre + "shared.", f["shared"]["ff"])
    return out


def _llama(raw, w, x, each):
    D, H, G, hd, F = (raw[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim", "intermediate_size"))
    sc, eps = raw["rope_scaling"], raw["rms_norm_eps"]
    rot = {"dims": hd, "base": raw["rope_theta"], "scaling": {"factor": sc["factor"], "low": sc["low_freq_factor"],
                                                                "high": sc["high_freq_factor"], "original": sc["original_max_position_embeddings"]}}
    for i in range(raw["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * w(p + "input_layernorm.weight", D)
        q, k, v = ((h @ w(f"{p}self_attn.{n}_proj.weight", c * hd, D).T).view(-1, c, hd) for n, c in (("q", H), ("k", G), ("v", G)))
        o = each(lambda q, k, v: _attend(_turn(q, rot, True), _turn(k, rot, True), v, hd ** -0.5), q, k, v)
        x = x + o.flatten(1) @ w(p + "self_attn.o_proj.weight", D, H * hd).T
        h = _rms(x, eps) * w(p + "post_attention_layernorm.weight", D)
        a = _silu(h @ w(p + "mlp.gate_proj.weight", F, D).T) * (h @ w(p + "mlp.up_proj.weight", F, D).T)
        x = x + a @ w(p + "mlp.down_proj.weight", D, F).T
    return _rms(x, eps) * w("model.norm.weight", D)


def _delta(x, w, p, m, D, eps, each):
    H, G, d = m["heads"], m["kv_heads"], m["dim"]
    q, k, v = (each(lambda y, n=n, c=c: _silu(_conv(y, w(f"{p}{n}.conv", c * d, m["conv"]))), x @ w(p + n, c * d, D).T).view(-1, c, d)
               for n, c in (("q", G), ("k", G), ("v", H)))
    unit = lambda y: y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)              # noqa: E731
    q, k = (unit(y).repeat_interleave(H // G, 1) for y in (q, k))
    beta = torch.sigmoid(x @ w(p + "b", H, D).T)
    decay = torch.exp(-torch.exp(w(p + "A_log", H)) * torch.nn.functional.softplus(x @ w(p + "a", H, D).T + w(p + "dt_bias", H), threshold=50.0))

    def scan(q, k, v, beta, decay):
        S, out = q.new_zeros(H, d, d), torch.empty_like(v)
        for t in range(q.shape[0]):
            S = decay[t][:, None, None] * S
            u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            out[t] = torch.einsum("hkv,hk->hv", S, q[t])
        return out
    o = each(scan, q * d ** -0.5, k, v, beta, decay)
    y = _rms(o, eps) * w(p + "norm", d) * _silu(x @ w(p + "g", H * d, D).T).view(-1, H, d)
    return y.flatten(1) @ w(p + "o", D, H * d).T


def _sink_attention(x, w, p, m, D, eps, each):
    H, G, d = m["heads"], m["kv_heads"], m["dim"]
    q, k = (x @ w(p + "q", H * d, D).T).view(-1, H, d), (x @ w(p + "k", G * d, D).T).view(-1, G, d)
    zero = torch.zeros(H, dtype=F64, device="cuda")
    o = each(lambda q, k: _attend(_rms(_turn(q, m["rot"], False), eps), _rms(_turn(k, m["rot"], False), eps), k, m["scale"], sink=zero), q, k)
    return (o.flatten(1) * torch.sigmoid(x @ w(p + "g", H * d, D).T)) @ w(p + "o", D, H * d).T


def _time_mix(x, w, p, m, D, eps, each):
    H, d = m["heads"], m["dim"]
    prev = each(lambda y: torch.cat([torch.zeros_like(y[:1]), y[:-1]]), x)
    mix = {s: x + (prev - x) * w(p + "mu." + s, D) for s in "rkvgw"}
    r, k, v = ((mix[s] @ w(p + s, D, D).T).view(-1, H, d) for s in "rkv")
    lam = torch.tanh(mix["w"] @ w(p + "w1", m["rank"], D).T) @ w(p + "w2", D, m["rank"]).T + w(p + "w0", D)
    decay, bonus = torch.exp(-torch.exp(lam)).view(-1, H, d), w(p + "u", H, d)

    def scan(r, k, v, decay):
        S, out = r.new_zeros(H, d, d), torch.empty_like(v)
        for t in range(r.shape[0]):
            kv = k[t][:, :, None] * v[t][:, None, :]
            out[t] = torch.einsum("hkv,hk->hv", S + bonus[:, :, None] * kv, r[t])
            S = decay[t][:, :, None] * S + kv
        return out
    y = _rms(each(scan, r, k, v, decay), eps).flatten(1) * w(p + "norm", D) * _silu(mix["g"] @ w(p + "g", D, D).T)
    return y @ w(p + "o", D, D).T


def _fuvipel(raw, w, x, each):
    D, eps = raw["width"], raw["norm"]["eps"]
    for i, lay in enumerate(raw["layers"]):
        p, m = f"l{i}.", lay["mixer"]
        if lay["type"] == "delta":
            y = _delta(x, w, p + "mix.", m, D, eps, each)
        else:
            a = _sink_attention(x, w, p + "mix.left.", m["left"], D, eps, each)
            b = _time_mix(x, w, p + "mix.right.", m["right"], D, eps, each)
            y = 0.5 * (_rms(a, eps) * w(p + "mix.left.out", D) + _rms(b, eps) * w(p + "mix.right.out", D))
        x = x + _rms(y, eps) * w(p + "norm1", D)
        z = torch.relu(x @ w(p + "mlp.up", lay["mlp"]["ff"], D).T)
        x = x + _rms((z * z) @ w(p + "mlp.down", D, lay["mlp"]["ff"]).T, eps) * w(p + "norm2", D)
    return _rms(x, eps) * w("final.norm", D)


def _retention(h, w, p, m, D, eps, each):
    H, d, dv = m["heads"], m["dim"], m["vdim"]
    q, k, v = ((h @ w(p + n, H * c, D).T).view(-1, H, c) for n, c in (("q", d), ("k", d), ("v", dv)))
    decay = torch.tensor(m["decay"], dtype=F64, device="cuda")

    def whole(q, k, v):                      # sum over the past of decay^(t - s) (q_t . k_s) v_s
        q, k = _turn(q, m["rot"], True), _turn(k, m["rot"], True) * d ** -0.5
        i = torch.arange(q.shape[0], dtype=F64, device="cuda")
        gap = i[:, None] - i[None, :]
        out = torch.empty_like(v)
        for hh in range(H):
            s = (q[:, hh] @ k[:, hh].T) * torch.where(gap >= 0, decay[hh] ** gap.clamp(min=0), 0.0)
            out[:, hh] = s @ v[:, hh]
        return out
    y = _rms(each(whole, q, k, v), eps).flatten(1) * _silu(h @ w(p + "g", H * dv, D).T)
    return y @ w(p + "o", D, H * dv).T


def _fovirax(raw, w, x, each):
    D, eps = raw["width"], raw["norm"]["eps"]
    for i, lay in enumerate(raw["layers"]):
        p, m = f"l{i}.", lay["mixer"]
        h, a = _rms(x, eps) * (1 + w(p + "norm1", D)), m["left"]
        H, G, d = a["heads"], a["kv_heads"], a["dim"]
        q, k, v = ((h @ w(f"{p}mix.left.{n}", c * d, D).T).view(-1, c, d) for n, c in (("q", H), ("k", G), ("v", G)))
        o = each(lambda q, k, v: _attend(_turn(q, a["rot"], True), _turn(k, a["rot"], True), v, a["scale"], a["mask"]["size"], a["softcap"]), q, k, v)
        y = m["left_scale"] * (o.flatten(1) @ w(p + "mix.left.o", D, H * d).T)
        y = y + m["right_scale"] * _retention(h, w, p + "mix.right.", m["right"], D, eps, each)
        x = x + w(p + "ls1", D) * y
        x = x + w(p + "ls2", D) * _moe(_rms(x, eps) * (1 + w(p + "norm2", D)), w, p + "mlp.", lay["mlp"], D, False)
    return _rms(x, eps) * (1 + w("final.norm", D))


def _selective(h, w, p, m, D, each):
    C, N, r = m["inner"], m["state"], m["dt_rank"]
    both = h @ w(p + "in", 2 * C, D).T
    u = _silu(each(lambda y: _conv(y, w(p + "conv", C, m["conv"])), both[:, :C]) + w(p + "conv.b", C))
    thin = u @ w(p + "x", r + 2 * N, C).T
    dt = torch.nn.functional.softplus(thin[:, :r] @ w(p + "dt", C, r).T + w(p + "dt.b", C), threshold=50.0)
    A = -torch.exp(w(p + "A_log", C, N))

    def scan(u, dt, b, c):
        S, out = torch.zeros_like(A), torch.empty_like(u)
        for t in range(u.shape[0]):
            S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * b[t]
            out[t] = S @ c[t]
        return out
    y = each(scan, u, dt, thin[:, r:r + N], thin[:, r + N:]) + w(p + "D", C) * u
    return (y * _silu(both[:, C:])) @ w(p + "o", D, C).T


def _mavinex(raw, w, x, each):
    D, eps, alpha = raw["width"], raw["norm"]["eps"], raw["postln_alpha"]
    for i, lay in enumerate(raw["layers"]):
        p, m = f"l{i}.", lay["mixer"]
        if lay["type"] == "parallel":
            a, n = m["left"], p + "mix.left."
            H, G, d = a["heads"], a["kv_heads"], a["dim"]
            q = (_rms(x @ w(n + "q", H * d, D).T, eps) * w(n + "q.norm", H * d)).view(-1, H, d)
            k = (_rms(x @ w(n + "k", G * d, D).T, eps) * w(n + "k.norm", G * d)).view(-1, G, d)
            v = (x @ w(n + "v", G * d, D).T).view(-1, G, d)
            o = each(lambda q, k, v: _attend(_turn(q, a["rot"], False), _turn(k, a["rot"], False), v, a["scale"], a["mask"]["size"]), q, k, v)
            left = (o.flatten(1) * torch.sigmoid(x @ w(n + "g", H * d, D).T)) @ w(n + "o", D, H * d).T
            right = _selective(x, w, p + "mix.right.", m["right"], D, each)
            y = 0.5 * (_rms(left, eps) * w(n + "out", D) + _rms(right, eps) * w(p + "mix.right.out", D))
        else:
            H, d, dv, r, rd, n = m["heads"], m["dim"], m["vdim"], m["kv_rank"], m["rot_dim"], p + "mix."
            q, down = (x @ w(n + "q", H * (d + rd), D).T).view(-1, H, d + rd), x @ w(n + "dkv", r + rd, D).T
            lat = _rms(down[:, :r], eps) * w(n + "dkv.norm", r)
            k, v = (lat @ w(n + "uk", H * d, r).T).view(-1, H, d), (lat @ w(n + "uv", H * dv, r).T).view(-1, H, dv)
            sink = w(n + "sink", H)

            def attend(q, k, kr, v):
                qt = torch.cat([q[..., :d], _turn(q[..., d:], m["rot"], True)], -1)
                kt = torch.cat([k, _turn(kr[:, None], m["rot"], True).expand(-1, H, -1)], -1)
                return _attend(qt, kt, v, m["scale"], m["mask"]["size"], sink=sink)
            o = each(attend, q, k, down[:, r:], v) * torch.sigmoid(x @ w(n + "g", H, D).T)[..., None]
            y = o.flatten(1) @ w(n + "o", D, H * dv).T
        x = _rms(alpha * x + y, eps) * (1 + w(p + "norm1", D))
        x = _rms(alpha * x + _moe(x, w, p + "mlp.", lay["mlp"], D, True), eps) * (1 + w(p + "norm2", D))
    return _rms(x, eps) * (1 + w("final.norm", D))


def exact(case, seed):
    """The same logits from the whole sequences at once, in 64 bits (no value for the sampler's tokens)."""
    if case["kind"] == "sample":
        return None
    design, raw = case["design"], _raw_config(case["design"], case["shape"])
    prompts, after = _requests(case, seed)
    V, D = VOCAB[design], raw.get("width") or raw["hidden_size"]
    source = _weights(design, case["shape"])

    def w(name, *shape):
        return source.make(name, shape).to(F64)
    whole = [p + a for p, a in zip(prompts, after)]
    if case["portion"]:
        whole[-1] = prompts[-1]
    ends = torch.tensor([len(s) for s in whole]).cumsum(0).tolist()
    runs = [(hi - len(s), hi) for s, hi in zip(whole, ends)]

    def each(f, *xs):                        # f on every sequence by itself
        return torch.cat([f(*(x[lo:hi] for x in xs)) for lo, hi in runs])
    ids = torch.tensor([t for s in whole for t in s], device="cuda")
    llama = design == "llama"
    x = {"llama": _llama, "fuvipel": _fuvipel, "fovirax": _fovirax, "mavinex": _mavinex}[design](
        raw, w, source.make("model.embed_tokens.weight" if llama else "embed", (V, D))[ids].to(F64), each)
    tied = raw["tie_word_embeddings"] if llama else design == "fuvipel"
    name = ("model.embed_tokens.weight" if tied else "lm_head.weight") if llama else ("embed" if tied else "head")
    head = w(name, V, D)

    def rows(at):
        return x[torch.tensor(at, device="cuda")] @ head.T
    starts, n = [lo for lo, _ in runs], [len(p) for p in prompts]
    if case["portion"]:
        return {"first": rows([lo + k - 1 for lo, k in zip(starts[:-1], n)]),
                "rest": torch.stack([rows([lo + k + i for lo, k in zip(starts[:-1], n)]) for i in range(len(after[0]))]),
                "late": rows([ends[-1] - 1])}
    first = rows(list(range(ends[-1]))) if case["want"] == "all" else rows([lo + k - 1 for lo, k in zip(starts, n)])
    if not case["steps"]:
        return {"first": first}
    return {"first": first, "rest": torch.stack([rows([lo + k + i for lo, k in zip(starts, n)]) for i in range(case["steps"])])}

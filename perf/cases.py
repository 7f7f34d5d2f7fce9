"""The work that users of this framework have it do, as cases that can be timed and compared.

Four kinds of work, each through the engine's own entry points:

``prefill``   whole prompts in one step (``Engine.step``), logits of every prompt's last token: reading a document, scoring,
              the first token of a chat.
``decode``    requests whose prompts are in the cache continue by one token a step, every step a CUDA graph of model and
              sampler launched one ahead of the tokens (``Engine.decode_launch`` / ``decode_collect``, as the scheduler runs
              them), then one step whose logits come back whole: chat, alone or in a batch.
``mixed``     a prompt arrives in portions beside requests that decode (``Engine.step`` and the device sampler): a server.
``generate``  requests from nothing to their last token: through ``batch_generate`` for the tiny float32 models (all calls
              small: launches and host work), through steps for the designs with recurrent layers, whose state cannot be
              wound back as a cache of keys and values can.

Models: GPT-2 of the sizes this repository is quoted on (tiny, medium, large, XL), and two designs that stand for the
other kinds of layers it runs: Lelatar (state-space and delta-rule recurrences beside attention) and Nufetar (attention with
mixed scores, attention over latent rows, a recurrence with a decay from the data).  Designs with experts are left out: with
random weights one bfloat16 rounding sends a token to another expert or is amplified tenfold (Fisesun's logits in bfloat16
are 4 to 12 % off those in 64 bits, in float32 2e-5), so two correct implementations cannot be told from a wrong one.
Types: bfloat16, and float32 for GPT-2.
Ranges: 1 to 64 requests, prompts of 8 to 1024 tokens, up to 2048 tokens a step, contexts of 16 to 1000 positions.

Tokens are given and not drawn (teacher forcing) except in the float32 generations: two correct bfloat16 implementations
round differently, and one other token would change all that follow.  For the same reason a step's outcome is the
log-probability of its likeliest token, and the logits of the last step.
"""
import math
import random
from collections import OrderedDict

import numpy as np
import torch

from mlx_lm_b200 import batch_generate
from mlx_lm_b200.config import get_architecture
from mlx_lm_b200.engine import Engine, StepEntry
from mlx_lm_b200.engine.scheduler import Request
from mlx_lm_b200.sampling import GREEDY, make_sampler
from mlx_lm_b200.sampling.device import DeviceSampler
from mlx_lm_b200.weights import build_model

PAGE = 16


# ------------------------------------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest calls: two short prompts of a tiny model in float32, greedy; launches and host work are all of it
        dict(name="tiny generate float32", model="gpt2-tiny-a", dtype="float32", work="generate", requests=2, tokens=13,
             steps=16, ragged=True, temp=0.0),
        # one user's chat
        dict(name="medium decode 1", model="gpt2-medium", dtype="bfloat16", work="decode", requests=1, tokens=512,
             steps=16, ragged=False),
        # a few users at once: the repository's headline
        dict(name="medium decode 8", model="gpt2-medium", dtype="bfloat16", work="decode", requests=8, tokens=512,
             steps=16, ragged=False),
        # a full batch, every request at a length of its own
        dict(name="medium decode 64", model="gpt2-medium", dtype="bfloat16", work="decode", requests=64,
             tokens=900, steps=12, ragged=True),
        # reading: two prompts of the full context
        dict(name="medium prefill", model="gpt2-medium", dtype="bfloat16", work="prefill", requests=2,
             tokens=1024, ragged=False),
        # the all-32-bit path: three prompts of odd lengths
        dict(name="medium prefill float32", model="gpt2-medium", dtype="float32", work="prefill", requests=3, tokens=301,
             ragged=True),
        # a server: a prompt in portions of 256 tokens beside 31 requests that decode
        dict(name="large mixed", model="gpt2-large", dtype="bfloat16", work="mixed", requests=31, tokens=700,
             steps=4, portion=256, ragged=True),
        # the largest dense model
        dict(name="xl prefill", model="gpt2-xl", dtype="bfloat16", work="prefill", requests=2, tokens=1024,
             ragged=False),
        # reading with recurrent layers
        dict(name="lelatar prefill", model="lelatar-1024", dtype="bfloat16", work="prefill", requests=2,
             tokens=1024, ragged=False),
        # short questions and their answers with recurrent layers
        dict(name="lelatar generate", model="lelatar-1024", dtype="bfloat16", work="generate", requests=8,
             tokens=100, steps=16, ragged=True),
        # reading prompts of odd lengths with mixed scores, latent rows and a recurrence
        dict(name="nufetar prefill", model="nufetar-1024", dtype="bfloat16", work="prefill", requests=3,
             tokens=731, ragged=True),
        # prompts and their answers, twice as wide
        dict(name="nufetar 2048 generate", model="nufetar-2048", dtype="bfloat16", work="generate", requests=4,
             tokens=400, steps=8, ragged=True),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges; none costs more than XL's two whole prompts."""
    work = rng.choice(("prefill", "prefill", "decode", "generate", "mixed"))
    ragged = rng.random() < 0.7
    if work == "prefill":
        model = rng.choice(("gpt2-medium", "gpt2-large", "lelatar-1024", "lelatar-2048", "nufetar-1024", "nufetar-2048"))
        dtype = "float32" if model == "gpt2-medium" and rng.random() < 0.4 else "bfloat16"
        n = rng.randint(1, 4)
        tokens = _log_int(rng, 8, min(1024, (1024 if dtype == "float32" else 2048) // n))
        return dict(model=model, dtype=dtype, work=work, requests=n, tokens=tokens, ragged=ragged)
    if work == "decode":
        dtype = "float32" if rng.random() < 0.15 else "bfloat16"
        model = "gpt2-medium" if dtype == "float32" else rng.choice(("gpt2-medium", "gpt2-large"))
        return dict(model=model, dtype=dtype, work=work, requests=_log_int(rng, 1, 8 if dtype == "float32" else 64),
                    tokens=_log_int(rng, 16, 1000), steps=rng.randint(4, 12), ragged=ragged)
    if work == "mixed":
        portion = rng.choice((64, 128, 256))
        return dict(model=rng.choice(("gpt2-medium", "gpt2-large")), dtype="bfloat16", work=work, requests=_log_int(rng, 1, 63),
                    tokens=_log_int(rng, 32, 900), steps=rng.randint(1, 4), portion=portion, ragged=ragged)
    model = rng.choice(("gpt2-tiny-a", "gpt2-tiny-b", "lelatar-1024", "nufetar-1024", "lelatar-2048", "nufetar-2048"))
    if model.startswith("gpt2-tiny"):
        return dict(model=model, dtype="float32", work=work, requests=rng.randint(1, 8), tokens=_log_int(rng, 4, 64),
                    steps=rng.randint(8, 24), ragged=ragged, temp=rng.choice((0.0, 0.8)))
    n = _log_int(rng, 1, 32)
    return dict(model=model, dtype="bfloat16", work=work, requests=n, tokens=_log_int(rng, 8, min(1000, 2048 // n)),
                steps=rng.randint(4, 16), ragged=ragged)


def _lengths(case):
    """Prompt lengths (``prefill``, ``generate``) or positions in the cache (``decode``, ``mixed``) of the requests."""
    n, t = case["requests"], case["tokens"]
    if not case["ragged"]:
        return [t] * n
    return [max(1, t - (i * 37 + i * i * 11) % (t // 2 + 1)) for i in range(n)]


# ------------------------------------------------------------------------------------------------ models

def _gpt2(layers, width, heads, vocab=50257, positions=1024, inner=None, eps=1e-5, gains=0.0):
    return dict(model_type="gpt2", n_layer=layers, n_embd=width, n_head=heads, n_inner=inner, vocab_size=vocab,
                n_positions=positions, layer_norm_epsilon=eps, activation_function="gelu_new", ln_gain_std=gains)


def _inner(width):
    return (width * 11 // 4 + 127) // 128 * 128


def _lelatar(width, vocab=32000):
    H = width // 64
    mamba = lambda mlp: {"type": "mamba2", "mlp": mlp, "mixer": {"conv": 4, "groups": 1, "heads": 2 * H, "norm_groups": 1,
                                                                 "state": 128, "vdim": 64}}
    ff = {"ff": _inner(width), "kind": "dense"}
    par = {"type": "parallel", "mlp": ff,
           "mixer": {"left": {"dim": 64, "heads": H, "kv_heads": max(1, H // 4), "vdim": 64, "scale": 0.125,
                              "rot": {"base": 500000.0, "dims": 32}},
                     "right": {"conv": 4, "dim": 64, "heads": H, "kv_heads": max(1, H // 4), "vdim": 64}}}
    return {"architecture": "Lelatar", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "token_side": {"dim": 64},
            "loop": {"start": 0, "stop": 4, "times": 2}, "layers": [mamba(None), par, mamba(ff), par, mamba(None), par]}


def _nufetar(width, vocab=32000):
    H = width // 64
    ff = {"ff": _inner(width), "kind": "dense"}
    rot = {"base": 500000.0, "dims": 32}
    att = {"type": "attention", "mlp": ff,
           "mixer": {"dim": 64, "heads": H, "kv_heads": max(1, H // 4), "vdim": 64, "scale": 0.125, "mask": {"size": 1024},
                     "rot": rot}}
    lat = {"type": "latent_attention", "mlp": ff,
           "mixer": {"dim": 64, "heads": H, "kv_rank": 256, "rot_dim": 32, "vdim": 64, "scale": 0.1, "mask": {"size": 1024},
                     "rot": rot}}
    rec = {"type": "wkv", "mlp": ff, "mixer": {"dim": 64, "heads": H, "decay_rank": 64}}
    return {"architecture": "Nufetar", "vocab": vocab, "width": width, "norm": {"eps": 1e-5},
            "layers": [att, lat, lat, rec, att] * 2}


CONFIGS = {
    "gpt2-tiny-a": lambda: _gpt2(2, 64, 4, vocab=512, positions=128),
    "gpt2-tiny-b": lambda: _gpt2(3, 96, 3, vocab=1000, positions=256, inner=320, eps=1e-6, gains=0.1),
    "gpt2-medium": lambda: _gpt2(24, 1024, 16),
    "gpt2-large": lambda: _gpt2(36, 1280, 20),
    "gpt2-xl": lambda: _gpt2(48, 1600, 25),
    "lelatar-1024": lambda: _lelatar(1024), "lelatar-2048": lambda: _lelatar(2048),
    "nufetar-1024": lambda: _nufetar(1024), "nufetar-2048": lambda: _nufetar(2048),
}


def _description(config):
    arch = get_architecture(config)
    return arch.build(arch.args_class.from_dict(dict(config)))


def _tensors(name):
    """The model's tensors: the design's own rules of random weights, drawn on the GPU in a fixed order, as bfloat16."""
    config = CONFIGS[name]()
    g = torch.Generator(device="cuda").manual_seed(1)
    out = {}
    for s in _description(config).param_specs():
        t = torch.randn(s.shape, generator=g, device="cuda") * s.init.std + s.init.mean
        out[s.name] = t.to(torch.bfloat16)
    return config, out


_models, _engines = OrderedDict(), OrderedDict()


def _engine(case):
    """A program keeps its model and its engine; here the last few of each are kept.  Room for the requests of five states."""
    n = case["requests"] + 1
    span = case["tokens"] + case.get("steps", 0) * max(1, case.get("portion", 1)) + 2
    limit = 1024 if case["model"].startswith("gpt2") else 2048
    pages = 5 * n * (min(span, limit) // PAGE + 2)
    model_key = (case["model"], case["dtype"])
    key = model_key + (5 * n, pages)
    if key not in _engines:
        if model_key not in _models:
            config, tensors = _tensors(case["model"])
            _models[model_key] = build_model(config, tensors, getattr(torch, case["dtype"]), "cuda")
            while len(_models) > 3:
                _models.popitem(last=False)
        _engines[key] = Engine(_models[model_key], page_size=PAGE, n_pages=pages, max_requests=5 * n,
                               max_len=None if case["model"].startswith("gpt2") else 2048)
        while len(_engines) > 3:
            _engines.popitem(last=False)
    return _engines[key]


# ------------------------------------------------------------------------------------------------ preparation

class State:
    """What a program holds between calls: its engine, and requests in the engine's cache that are let go with it."""
    numbers = iter(range(1, 1 << 40))

    def __init__(self, case, seed):
        self.case, self.engine = case, _engine(case)
        self.held = []
        self.sampler = DeviceSampler(self.engine.model.device, seed=seed, engine=self.engine)

    def hold(self, tokens):
        rid = next(State.numbers)
        self.engine.add_request(rid)
        self.held.append(rid)
        return Request(rid, tokens, len(tokens), 1 << 30, GREEDY)

    def __del__(self):
        for rid in self.held:
            self.engine.finish(rid)


def _tokens(case, seed):
    """(the requests' tokens before the timed steps, the tokens they are given in them, the prompt that arrives)."""
    vocab = CONFIGS[case["model"]]()
    vocab = vocab.get("vocab_size") or vocab["vocab"]
    rng = np.random.RandomState((seed * 7919 + 17) % (1 << 32))
    lengths = _lengths(case)
    first = [rng.randint(0, vocab, n).tolist() for n in lengths]
    given = [rng.randint(0, vocab, case.get("steps", 0) + 1).tolist() for _ in lengths]
    arriving = rng.randint(0, vocab, max(1, case.get("steps", 0) * case.get("portion", 0) - 19)).tolist()
    return first, given, arriving


def prepare(case, seed):
    s = State(case, seed)
    s.first, s.given, s.arriving = _tokens(case, seed)
    if case["work"] in ("decode", "mixed"):
        s.requests = [s.hold(t) for t in s.first]
        entries = [StepEntry(r.uid, r.tokens) for r in s.requests]
        at, room = 0, 2048
        for i, e in enumerate(entries + [None]):
            if e is None or room < len(e.tokens):
                s.engine.step(entries[at:i])
                at, room = i, 2048
            if e is not None:
                room -= len(e.tokens)
    if case["work"] == "generate":
        s.options = make_sampler(case.get("temp", 0.0))
    return s


# ------------------------------------------------------------------------------------------------ one pass

def _decode(s, requests):
    """The given tokens but the last through CUDA graphs, each step launched before the one before it is read; the last
    through a step whose logits come back."""
    engine, steps, flying, seen = s.engine, s.case["steps"], None, []
    for k in range(steps):
        ahead = engine.decode_launch([StepEntry(r.uid, g[k:k + 1], [0]) for r, g in zip(requests, s.given)], requests, s.sampler)
        if flying is not None:
            seen.append(engine.decode_collect(flying)[1])
        flying = ahead
    seen.append(engine.decode_collect(flying)[1])
    return engine.step([StepEntry(r.uid, g[steps:], [0]) for r, g in zip(requests, s.given)]), seen


def run(s):
    case, engine = s.case, s.engine
    if case["work"] == "prefill":
        rids = [next(State.numbers) for _ in s.first]
        for rid in rids:
            engine.add_request(rid)
        logits = engine.step([StepEntry(rid, t, [len(t) - 1]) for rid, t in zip(rids, s.first)])
        for rid in rids:
            engine.finish(rid)
        return {"logits": logits}
    if case["work"] == "decode":
        for r, t in zip(s.requests, s.first):
            engine.cache.truncate(r.uid, len(t))
        logits, seen = _decode(s, s.requests)
        return {"logits": logits, "logprobs": np.array(seen, dtype=np.float32)}
    if case["work"] == "mixed":
        for r, t in zip(s.requests, s.first):
            engine.cache.truncate(r.uid, len(t))
        new = Request(next(State.numbers), s.arriving, len(s.arriving), 1 << 30, GREEDY)
        engine.add_request(new.uid)
        seen, portion = [], case["portion"]
        for k in range(case["steps"]):
            entries = [StepEntry(r.uid, g[k:k + 1], [0]) for r, g in zip(s.requests, s.given)]
            last = k + 1 == case["steps"]
            part = s.arriving[k * portion:(k + 1) * portion]
            entries.append(StepEntry(new.uid, part, [len(part) - 1] if last else []))
            logits = engine.step(entries)
            seen.append(s.sampler(logits, s.requests + [s.requests[0]] if last else s.requests)[1][:len(s.requests)])
        engine.finish(new.uid)
        return {"logits": logits, "logprobs": np.array(seen, dtype=np.float32)}
    if case["model"].startswith("gpt2"):
        r = batch_generate(engine.model, None, s.first, max_tokens=case["steps"], return_token_ids=True, return_logprobs=True,
                           engine=engine, seed=5, sampler=s.options, completion_batch_size=8)
        return {"tokens": np.array(r.token_ids), "logprobs": np.array(r.logprobs, dtype=np.float32)}
    requests = [Request(next(State.numbers), t, len(t), 1 << 30, GREEDY) for t in s.first]
    for r in requests:
        engine.add_request(r.uid)
    seen = [s.sampler(engine.step([StepEntry(r.uid, r.tokens, [len(r.tokens) - 1]) for r in requests]), requests)[1]]
    logits, more = _decode(s, requests)
    for r in requests:
        engine.finish(r.uid)
    return {"logits": logits, "logprobs": np.array(seen + more, dtype=np.float32)}


# ------------------------------------------------------------------------------------------------ what a pass needs

def _sizes(name):
    """Per token: matrix elements multiplied and (token, key) flops per key of all layers; elements kept in the cache; per
    request: state elements; elements of all weights but the embeddings, and the head's."""
    c = CONFIGS[name]()
    if name.startswith("gpt2"):
        D, L = c["n_embd"], c["n_layer"]
        lin = L * (4 * D * D + 2 * D * (c["n_inner"] or 4 * D))
        return dict(lin=lin, weights=lin, key=4 * D * L, cache=2 * D * L, state=0, scan=0, head=D * c["vocab_size"])
    D, out = c["width"], dict(lin=0, weights=0, key=0, cache=0, state=0, scan=0, head=c["width"] * c["vocab"])
    loop = c.get("loop")
    for i, layer in enumerate(c["layers"]):
        runs = loop["times"] if loop and loop["start"] <= i < loop["stop"] else 1
        m, kind = layer["mixer"], layer["type"]
        lin = key = cache = state = 0
        if kind == "mamba2":
            inner, state = m["heads"] * m["vdim"], m["heads"] * m["vdim"] * m["state"]
            lin = D * (3 * inner + 2 * m["groups"] * m["state"] + m["heads"])
        elif kind == "parallel":
            l, r = m["left"], m["right"]
            lin = D * (2 * l["heads"] + 2 * l["kv_heads"]) * l["dim"]
            lin += D * (3 * r["heads"] * r["vdim"] + 2 * r["kv_heads"] * r["dim"] + 2 * r["heads"])
            key, cache, state = 4 * l["heads"] * l["dim"], 2 * l["kv_heads"] * l["dim"], r["heads"] * r["dim"] * r["vdim"]
        elif kind == "attention":
            lin, key = D * (2 * m["heads"] + 2 * m["kv_heads"]) * m["dim"], 4 * m["heads"] * m["dim"]
            cache = 2 * m["kv_heads"] * m["dim"]
        elif kind == "latent_attention":
            R, H = m["kv_rank"], m["heads"]
            lin = D * (H * (m["dim"] + m["rot_dim"]) + R + m["rot_dim"] + H * m["vdim"]) + R * H * (m["dim"] + m["vdim"])
            key, cache = 2 * H * (m["dim"] + m["rot_dim"] + m["vdim"]), R + m["rot_dim"]
        elif kind == "wkv":
            lin = D * (5 * m["heads"] * m["dim"] + m["decay_rank"]) + m["decay_rank"] * m["heads"] * m["dim"]
            state = m["heads"] * m["dim"] ** 2
        if layer["mlp"] is not None:
            lin += D * layer["mlp"]["ff"] * (2 if c["architecture"] == "Nufetar" else 3)
        for k, v in (("lin", lin), ("key", key), ("cache", cache), ("state", state), ("scan", 5 * state)):
            out[k] += runs * v
        out["weights"] += lin
    return out


def work(case):
    z, size = _sizes(case["model"]), 2 if case["dtype"] == "bfloat16" else 4
    lengths, steps = _lengths(case), case.get("steps", 0)
    bytes_, flops = 0.0, 0.0

    def step(spans, wanted):
        """``spans``: (positions in the cache before, new tokens) of every request in one step."""
        nonlocal bytes_, flops
        new = sum(n for _, n in spans)
        keys = sum(n * a + n * (n + 1) / 2 for a, n in spans)
        state = 4 * z["state"] * sum(2 if a else 1 for a, n in spans)
        bytes_ += size * (z["weights"] + z["head"]) + size * z["cache"] * (new + sum(a for a, _ in spans)) + state
        bytes_ += 4 * wanted * z["head"] / max(1, _width(case)) + 8 * new
        flops += 2 * z["lin"] * new + z["key"] * keys + z["scan"] * new + 2 * z["head"] * wanted

    if case["work"] in ("prefill", "generate"):
        step([(0, n) for n in lengths], len(lengths))
    if case["work"] in ("decode", "generate"):
        more = steps + 1 if not case["model"].startswith("gpt2-tiny") else steps - 1
        for k in range(more):
            step([(n + k, 1) for n in lengths], len(lengths))
    if case["work"] == "mixed":
        total = max(1, steps * case["portion"] - 19)
        for k in range(steps):
            a = k * case["portion"]
            step([(n + k, 1) for n in lengths] + [(a, min(case["portion"], total - a))], len(lengths))
    return {"bytes": bytes_, "flops": flops}


def _width(case):
    c = CONFIGS[case["model"]]()
    return c.get("n_embd") or c["width"]


def tolerance(case):
    # against 64 bits one pass of float32 is 2e-6 off, one of bfloat16 0.7e-2 (Nufetar) to 1.7e-2 (Lelatar); the largest
    # difference of a logit is some five times the mean one
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    return {"rel": 0.03, "max": 0.3}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
# Whole sequences, one mechanism a function, plain torch; recurrences token by token.

def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _softplus(x):
    return torch.log1p(torch.exp(-x.abs())) + torch.clamp(x, min=0.0)


def _visible(T, window=None, run=None):
    i = torch.arange(T, device="cuda")
    back = i[:, None] - i[None, :]
    ok = back >= 0
    if window:
        ok &= back < window
    if run:
        ok &= (i[:, None] // run) == (i[None, :] // run)
    return ok


def _turn(x, rot, neighbours=False):
    """``x [T, heads, d]``: pairs ``(i, i + dims / 2)`` or ``(2 i, 2 i + 1)`` of the first dims turned by the position."""
    n = rot["dims"]
    freq = [float(rot["base"]) ** (-2.0 * i / n) for i in range(n // 2)]
    a = torch.arange(x.shape[0], dtype=torch.float64, device="cuda")[:, None] * torch.tensor(freq, dtype=torch.float64, device="cuda")
    c, s = torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]
    u, v = (x[..., 0:n:2], x[..., 1:n:2]) if neighbours else (x[..., :n // 2], x[..., n // 2:n])
    u, v = u * c - v * s, v * c + u * s
    turned = torch.stack([u, v], dim=-1).flatten(-2) if neighbours else torch.cat([u, v], dim=-1)
    return torch.cat([turned, x[..., n:]], dim=-1)


def _attend(scores, ok, v):
    """``scores [H, T, T]``, ``v [T, H, dv]`` -> ``[T, H dv]``."""
    p = torch.softmax(scores.masked_fill(~ok, -math.inf), dim=-1)
    return torch.einsum("hij,jhd->ihd", p, v).flatten(1)


def _per_head(x, H):
    """Key/value heads repeated for the query heads that share them."""
    return x.repeat_interleave(H // x.shape[1], dim=1)


def _short_conv(u, w, b=None):
    T, taps = u.shape[0], w.shape[1]
    out = torch.zeros_like(u)
    for j in range(min(taps, T)):
        out[j:] += u[:T - j] * w[:, taps - 1 - j]
    return out if b is None else out + b


def _exact_gpt2(c, w, tokens):
    D, H, T = c["n_embd"], c["n_head"], len(tokens)
    norm = lambda x, p: ((x - x.mean(-1, keepdim=True)) / torch.sqrt(x.var(-1, unbiased=False, keepdim=True) + c["layer_norm_epsilon"])
                         * w[p + ".weight"] + w[p + ".bias"])
    lin = lambda x, p: x @ w[p + ".weight"] + w[p + ".bias"]
    x = w["wte.weight"][tokens] + w["wpe.weight"][:T]
    ok = _visible(T)
    for i in range(c["n_layer"]):
        p = f"h.{i}."
        q, k, v = (t.view(T, H, D // H) for t in lin(norm(x, p + "ln_1"), p + "attn.c_attn").split(D, dim=-1))
        x = x + lin(_attend(torch.einsum("ihd,jhd->hij", q, k) * (D // H) ** -0.5, ok, v), p + "attn.c_proj")
        x = x + lin(_gelu(lin(norm(x, p + "ln_2"), p + "mlp.c_fc")), p + "mlp.c_proj")
    return norm(x, "ln_f"), w["wte.weight"]


def _mamba2(h, w, p, m, eps):
    T, H, V, N, G = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * V
    z, xbc, dt = (h @ w[p + "in"].T).split([inner, inner + 2 * G * N, H], dim=-1)
    xbc = _silu(_short_conv(xbc, w[p + "conv"], w[p + "conv.b"]))
    x, B, C = xbc.split([inner, G * N, G * N], dim=-1)
    x = x.view(T, H, V)
    B, C = _per_head(B.view(T, G, N), H), _per_head(C.view(T, G, N), H)
    dt = _softplus(dt + w[p + "dt_bias"])
    a = torch.exp(-torch.exp(w[p + "A_log"]) * dt)
    S, y = h.new_zeros(H, N, V), h.new_empty(T, H, V)
    Bx = dt[:, :, None] * B
    for t in range(T):
        S = a[t, :, None, None] * S + Bx[t, :, :, None] * x[t, :, None, :]
        y[t] = torch.bmm(C[t, :, None, :], S)[:, 0]
    y = (y + w[p + "D"][:, None] * x).flatten(1) * _silu(z)
    return (_rms(y.view(T, m["norm_groups"], -1), eps).flatten(1) * w[p + "norm"]) @ w[p + "o"].T


def _sinks(h, w, p, m, eps):
    T, H, G, d = h.shape[0], m["heads"], m["kv_heads"], m["dim"]
    q = _turn((_rms(h @ w[p + "q"].T, eps) * w[p + "q.norm"]).view(T, H, d), m["rot"])
    k = _turn((_rms(h @ w[p + "k"].T, eps) * w[p + "k.norm"]).view(T, G, d), m["rot"])
    v = (h @ w[p + "v"].T).view(T, G, m["vdim"])
    s = torch.einsum("ihd,jhd->hij", q, _per_head(k, H)) * m["scale"]
    s = s.masked_fill(~_visible(T), -math.inf)
    s = torch.cat([s, w[p + "sink"][:, None, None].expand(H, T, 1)], dim=-1)      # a column that has no value
    o = torch.einsum("hij,jhd->ihd", torch.softmax(s, dim=-1)[..., :T], _per_head(v, H))
    return o.flatten(1) @ w[p + "o"].T


def _delta(h, w, p, m, eps):
    T, H, G, dk, dv = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    part = lambda n, heads, d: _silu(_short_conv(h @ w[p + n].T, w[p + n + ".conv"])).view(T, heads, d)
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
    q, k = _per_head(unit(part("q", G, dk)) * dk ** -0.5, H), _per_head(unit(part("k", G, dk)), H)
    v = part("v", H, dv)
    beta = torch.sigmoid(h @ w[p + "b"].T)
    decay = torch.exp(-torch.exp(w[p + "A_log"]) * _softplus(h @ w[p + "a"].T + w[p + "dt_bias"]))
    S, o = h.new_zeros(H, dk, dv), h.new_empty(T, H, dv)
    for t in range(T):
        S = decay[t, :, None, None] * S
        u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None, :], S)[:, 0])
        S = S + k[t, :, :, None] * u[:, None, :]
        o[t] = torch.bmm(q[t, :, None, :], S)[:, 0]
    o = (_rms(o, eps) * w[p + "norm"]).flatten(1) * _silu(h @ w[p + "g"].T)
    return o @ w[p + "o"].T


def _gated(h, w, p):
    return (_silu(h @ w[p + ".gate"].T) * (h @ w[p + ".up"].T)) @ w[p + ".down"].T


def _exact_lelatar(c, w, tokens):
    eps, dim = c["norm"]["eps"], c["token_side"]["dim"]
    norm = lambda x, p: _rms(x, eps) * (1.0 + w[p])
    first = x = w["embed"][tokens]
    a, b, times = c["loop"]["start"], c["loop"]["stop"], c["loop"]["times"]
    order = [(i, None) for i in range(a)] + [(i, t) for t in range(times) for i in range(a, b)]
    for i, t in order + [(i, None) for i in range(b, len(c["layers"]))]:
        if t is not None and i == a:
            x = torch.cat([x, first], dim=-1) @ w["loop.in"].T + w["loop.step"][t]
        layer, p = c["layers"][i], f"l{i}."
        h, m = norm(x, p + "norm1"), layer["mixer"]
        if layer["type"] == "mamba2":
            x = x + _mamba2(h, w, p + "mix.", m, eps)
        else:
            left, right = _sinks(h, w, p + "mix.left.", m["left"], eps), _delta(h, w, p + "mix.right.", m["right"], eps)
            x = x + 0.5 * (_rms(left, eps) * w[p + "mix.left.out"] + _rms(right, eps) * w[p + "mix.right.out"])
        if layer["mlp"] is not None:
            x = x + _gated(norm(x, p + "norm2"), w, p + "mlp")
        e = w["side.embed"][tokens][:, i * dim:(i + 1) * dim]
        x = x + _rms((_gelu(x @ w[p + "side.gate"].T) * e) @ w[p + "side.proj"].T, eps) * w[p + "side.norm"]
    return norm(x, "final.norm"), w["head"]


def _talking(h, w, p, m, eps):
    T, H, G, d = h.shape[0], m["heads"], m["kv_heads"], m["dim"]
    part = lambda n, heads: (h @ w[p + n].T + w[p + n + ".b"]).view(T, heads, -1)
    q, k, v = _turn(part("q", H), m["rot"]), _turn(part("k", G), m["rot"]), _rms(part("v", G), eps)
    s = torch.einsum("ihd,jhd->hij", q, _per_head(k, H)) * m["scale"]
    o = _attend(torch.einsum("hg,gij->hij", w[p + "talk"], s), _visible(T, run=m["mask"]["size"]), _per_head(v, H))
    gate = torch.sigmoid(h @ w[p + "g"].T)
    return (o.view(T, H, -1) * gate[:, :, None]).flatten(1) @ w[p + "o"].T + w[p + "o.b"]


def _latent(h, w, p, m, eps):
    T, H, d, r, R = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    q, down = (h @ w[p + "q"].T).view(T, H, d + r), h @ w[p + "dkv"].T
    row = _rms(down[:, :R], eps) * w[p + "dkv.norm"]
    turned = _turn(down[:, None, R:], m["rot"], True).expand(T, H, r)
    k = torch.cat([(row @ w[p + "uk"].T).view(T, H, d), turned], dim=-1)
    q = torch.cat([q[..., :d], _turn(q[..., d:], m["rot"], True)], dim=-1)
    s = torch.einsum("ihd,jhd->hij", q, k) * m["scale"]
    return _attend(s, _visible(T, window=m["mask"]["size"]), (row @ w[p + "uv"].T).view(T, H, -1)) @ w[p + "o"].T


def _wkv(h, w, p, m, eps):
    T, H, d = h.shape[0], m["heads"], m["dim"]
    before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    mix = {s: h + (before - h) * w[p + "mu." + s] for s in "rkvgw"}
    r, k, v = ((mix[s] @ w[p + s].T).view(T, H, d) for s in "rkv")
    decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w[p + "w1"].T) @ w[p + "w2"].T + w[p + "w0"])).view(T, H, d)
    S, o = h.new_zeros(H, d, d), h.new_empty(T, H, d)
    for t in range(T):
        o[t] = torch.bmm(r[t, :, None, :], S)[:, 0]
        S = decay[t, :, :, None] * S + k[t, :, :, None] * v[t, :, None, :]
    o = o + (r * w[p + "u"] * k).sum(-1, keepdim=True) * v
    return (_rms(o, eps).flatten(1) * w[p + "norm"] * _silu(mix["g"] @ w[p + "g"].T)) @ w[p + "o"].T


def _exact_nufetar(c, w, tokens):
    eps, mixers = c["norm"]["eps"], {"attention": _talking, "latent_attention": _latent, "wkv": _wkv}
    x = w["embed"][tokens]
    for i, layer in enumerate(c["layers"]):
        p = f"l{i}."
        x = x + mixers[layer["type"]](_rms(x, eps) * w[p + "norm1"], w, p + "mix.", layer["mixer"], eps)
        z = (_rms(x, eps) * w[p + "norm2"]) @ w[p + "mlp.up"].T
        a, b = _softplus(w[p + "mlp.act"][0]), _softplus(w[p + "mlp.act"][1])
        z = torch.where(z > 0, a * z * z + z / 2, (0.5 + b) * (torch.expm1(torch.clamp(z, max=0.0)) - z) + z / 2)
        x = x + z @ w[p + "mlp.down"].T
    return _rms(x, eps) * w["final.norm"], w["embed"]


def _exact_logits(case, sequences):
    """``sequences``: (tokens, positions whose logits are wanted), one after the other."""
    config, w = _tensors(case["model"])
    w = {k: t.double() for k, t in w.items()}
    forward = globals()["_exact_" + case["model"].split("-")[0]]
    for tokens, wanted in sequences:
        x, head = forward(config, w, torch.tensor(tokens, device="cuda"))
        yield x[wanted] @ head.T


def _likeliest(logits):
    return logits.max(-1).values - torch.logsumexp(logits, -1)


def exact(case, seed):
    with torch.no_grad():
        first, given, arriving = _tokens(case, seed)
        steps = case.get("steps", 0)
        if case["work"] == "prefill":
            return {"logits": torch.cat(list(_exact_logits(case, [(t, [len(t) - 1]) for t in first])))}
        if case["model"].startswith("gpt2-tiny"):
            if case["temp"]:
                return None                                             # which tokens are drawn is the sampler's own
            found, lps = [], []
            for t in first:
                t, lp = list(t), []
                for _ in range(steps):
                    logits = next(_exact_logits(case, [(t, [len(t) - 1])]))
                    lp.append(_likeliest(logits)[0].item())
                    t.append(int(logits.argmax()))
                found.append(t[-steps:])
                lps.append(lp)
            return {"tokens": np.array(found), "logprobs": np.array(lps)}
        if case["work"] == "mixed":
            sequences = [(t + g[:steps], range(len(t), len(t) + steps)) for t, g in zip(first, given)]
            got = list(_exact_logits(case, [(t, list(r)) for t, r in sequences] + [(arriving, [len(arriving) - 1])]))
            logits = torch.cat([g[-1:] for g in got])
            return {"logits": logits, "logprobs": torch.stack([_likeliest(g) for g in got[:-1]], dim=1)}
        before = 1 if case["work"] == "generate" else 0
        sequences = [(t + g, list(range(len(t) - before, len(t) + steps + 1))) for t, g in zip(first, given)]
        got = [(g[-1:], _likeliest(g[:-1])) for g in _exact_logits(case, sequences)]
        return {"logits": torch.cat([g for g, _ in got]), "logprobs": torch.stack([p for _, p in got], dim=1)}


if __name__ == "__main__":
    rng = random.Random(0)
    for c in listed() + [draw(rng) for _ in range(8)]:
        w = work(c)
        print("%-120s %8.1f MB %10.2f GFLOP" % ({k: v for k, v in c.items()}, w["bytes"] / 1e6, w["flops"] / 1e9))

"""Workloads that the framework's performance is measured on: what a user's program has the engine and the stand-alone
operators do, through ``Engine`` and ``ops``, at sizes from single small calls to a long prompt of the largest shape.

Models are random-init ones of the shapes that the benchmark and the tests use, with the numerical habits of trained ones:
the token's own embedding dominates the residual stream, layers add a bounded part, and the classifier is confident about
one successor of every token (so that sampled sequences do not hang on the last bit of a sum).

A case is a dict of plain values:

* ``kind`` "step": one token through ``step_logits`` and ``sample``, as a host-driven loop calls them;
* ``kind`` "decode": ``n`` tokens through the device-resident loop at position ``start``, then the next step's logits;
* ``kind`` "prompt": ``n`` prompt tokens at position ``start`` through ``extend``, with the logits of the last ``want`` ones;
* ``kind`` "generate": a prompt of ``start`` tokens from position 0, then "decode" (for models whose state is recurrent);
* ``kind`` "layer": one decoder layer operator by operator, as a partly ported host calls the reference's wrappers;
* ``kind`` "sample": the stand-alone sampler on logits that lie on the GPU.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from lighterpp_b200 import ops
from lighterpp_b200.engine import Engine
from lighterpp_b200.formats import (LatentMixer, Layer, LayeredConfig, Loop, MambaMixer, ModelConfig, Rotation, SharedKvMixer, Yarn,
                                    tensor_shapes)
from lighterpp_b200.models import ARCHITECTURES
from lighterpp_b200.synth import SHAPES

EMB_STD, SUCCESSOR, CONFIDENCE = 3.0, 7919, 17.0
_MLA = dict(dim=128, rot_dim=64, vdim=128, kv_rank=512)
# width, layers (kolatar: groups of two scan layers and an attention layer, the first group running twice), ff, vocabulary,
# mixer sizes, window
LAYERED = {
    "rutenex-300m": (1024, 24, 2816, 32768, dict(heads=16, dim=64, rot_dim=32, vdim=64, kv_rank=256), 512),
    "rutenex-1b": (2048, 16, 8192, 32768, dict(heads=16, **_MLA), 1024),
    "kolatar-300m": (1024, 8, 2816, 32768, dict(inner=2048, state=16, conv=4, dt_rank=64, heads=16, kv_heads=4, dim=64), 512),
    "kolatar-1b": (2048, 6, 8192, 32768, dict(inner=4096, state=16, conv=4, dt_rank=128, heads=32, kv_heads=8, dim=64), 1024),
}


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # a host program that drives a small FP32 model token by token and samples on logits it has seen: latency of one call
        dict(name="step-stories15m", kind="step", model="stories15m", start=100, n=1, temperature=1.0, penalty=1.0),
        # a chat reply of the headline model: device-resident sampling loop behind a medium context
        dict(name="decode-1b", kind="decode", model="llama-3.2-1b", start=640, n=48, temperature=0.8, penalty=1.1),
        # greedy decoding of the largest model over a long context: weights and cache both count
        dict(name="decode-8b-32k", kind="decode", model="llama-3-8b", start=32768, n=8, temperature=0.0, penalty=1.0),
        # a story prompt of a llama2.c checkpoint: everything in FP32
        dict(name="prompt-stories15m", kind="prompt", model="stories15m", start=0, n=201, want=1),
        # the next turn of a chat: a short, odd number of tokens behind an existing context
        dict(name="turn-tinyllama", kind="prompt", model="tinyllama-1.1b", start=1100, n=47, want=1),
        # a page of text as prompt of the headline model
        dict(name="prompt-1b", kind="prompt", model="llama-3.2-1b", start=0, n=1023, want=1),
        # a document as prompt of the largest model
        dict(name="prompt-8b", kind="prompt", model="llama-3-8b", start=0, n=3000, want=1),
        # the same through latent attention under a window, BF16 weights
        dict(name="prompt-rutenex-1b", kind="prompt", model="rutenex-1b", start=0, n=1023, want=1, dtype="bf16"),
        # decoding of a small latent-attention model: many short kernels
        dict(name="decode-rutenex-300m", kind="decode", model="rutenex-300m", start=700, n=32, temperature=0.0, penalty=1.0, dtype="bf16"),
        # a whole request to a recurrent model: prompt, then sampled tokens
        dict(name="generate-kolatar-1b", kind="generate", model="kolatar-1b", start=517, n=32, temperature=0.8, penalty=1.1, dtype="bf16"),
        # the reference's operators one by one over one layer of the largest shape (FP16 weights and cache)
        dict(name="layer-ops-8b", kind="layer", model="llama-3-8b", start=1500),
        # the stand-alone sampler on a 128 K vocabulary with history
        dict(name="sample-128k", kind="sample", vocab=128256, temperature=0.8, penalty=1.1, history=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "decode", "decode", "prompt", "prompt", "prompt", "prompt", "generate", "layer", "sample"])
    if kind == "sample":
        return dict(kind=kind, vocab=_log_int(rng, 1000, 262144), temperature=rng.choice([0.0, 0.7, 1.0]), penalty=rng.choice([1.0, 1.2]),
                    history=rng.randint(0, 256))
    if kind == "layer":
        return dict(kind=kind, model=rng.choice(["tinyllama-1.1b", "llama-3.2-1b", "llama-3-8b"]), start=_log_int(rng, 1, 3000))
    if kind == "step":
        return dict(kind=kind, model=rng.choice(["stories15m", "tinyllama-1.1b", "llama-3.2-1b"]), start=rng.randint(0, 250), n=1,
                    temperature=rng.choice([0.0, 0.8]), penalty=rng.choice([1.0, 1.1]))
    if kind == "generate":
        return dict(kind=kind, model=rng.choice(["kolatar-300m", "kolatar-1b"]), start=_log_int(rng, 2, 1500), n=_log_int(rng, 4, 40),
                    temperature=rng.choice([0.0, 0.8]), penalty=1.0, dtype="bf16")
    if kind == "decode":
        model = rng.choice(["stories15m", "tinyllama-1.1b", "llama-3.2-1b", "llama-3-8b", "rutenex-300m", "rutenex-1b"])
        top = {"stories15m": 200, "llama-3-8b": 16384}.get(model, 1900)
        c = dict(kind=kind, model=model, start=_log_int(rng, 1, top), n=_log_int(rng, 4, 40), temperature=rng.choice([0.0, 0.8]),
                 penalty=rng.choice([1.0, 1.1]))
        return dict(c, dtype="bf16") if model in LAYERED else c
    model = rng.choice(["stories15m", "tinyllama-1.1b", "llama-3.2-1b", "llama-3-8b", "rutenex-300m", "rutenex-1b", "kolatar-300m", "kolatar-1b"])
    n = _log_int(rng, 2, {"stories15m": 230, "llama-3-8b": 2500}.get(model, 1900))
    start = 0 if model.startswith("kolatar") or rng.random() < 0.5 else _log_int(rng, 1, 20 if model == "stories15m" else 2000)
    c = dict(kind=kind, model=model, start=start, n=n, want=rng.choice([1, 1, min(n, 9)]))
    if model in LAYERED:
        c["dtype"] = "f32" if model.endswith("300m") and n < 300 and rng.random() < 0.3 else "bf16"
    return c


# ------------------------------------------------------------------ models

def _config(case):
    name = case["model"]
    need = case["start"] + case.get("n", 0) + 8
    if name in LAYERED:
        width, layers, ff, vocab, mix, window = LAYERED[name]
        yarn = Yarn(4.0, 4096, 32.0, 1.0)
        if name.startswith("rutenex"):
            m = LatentMixer(scale=(mix["dim"] + mix["rot_dim"]) ** -0.5, window=window, rotation=Rotation(mix["rot_dim"], 1e6, yarn), **mix)
            return LayeredConfig(width, vocab, max(need, 2048), [Layer(m, ff, "gelu_tanh")] * layers, "layer", 1e-6)
        scan = Layer(MambaMixer(mix["inner"], mix["state"], mix["conv"], mix["dt_rank"]))
        dim = mix["dim"]
        attn = Layer(SharedKvMixer(mix["heads"], mix["kv_heads"], dim, dim ** -0.5, Rotation(dim // 2, 1e6, yarn), window, 30.0, True, True), ff)
        return LayeredConfig(width, vocab, max(need, 2048), [scan, scan, attn] * layers, "rms", 1e-5, 1.0, 1.0, Loop(0, 3, 2))
    c = SHAPES[name][0]
    return ModelConfig(**{**c.asdict(), "seq_len": max(need, c.seq_len)})


def _dtype(case):
    return {"f16": torch.float16, "f32": torch.float32, "bf16": torch.bfloat16}[case.get("dtype") or SHAPES[case["model"]][1]]


def _generator(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 16 + stream)
    return g


def _weights(case, seed):
    """(engine tensor, layer, values on the GPU) of the case's model, always in the same order."""
    c, dt, g = _config(case), _dtype(case), _generator(seed, 0)

    def normal(shape, std):
        return (torch.randn(shape, device="cuda", generator=g, dtype=dt) * std)

    D, V = c.dim, c.vocab_size
    emb = normal((V, D), EMB_STD)
    yield "tok_emb", 0, emb
    head = normal((V, D), 0.9 * D ** -0.5)
    # token t names token t + SUCCESSOR: x (unit size after the norm) . head is about CONFIDENCE there
    head += torch.roll(emb, SUCCESSOR, 0) * (CONFIDENCE / (D * EMB_STD))
    yield "w_cls", 0, head
    del emb, head
    if isinstance(c, LayeredConfig):
        depth = (2 * c.n_layers) ** -0.5
        arch = ARCHITECTURES["Rutenex" if c.norm == "layer" else "Kolatar"]
        rows = [(ours, layer, tensor, shape) for ours, layer, tensor, shape in arch.tensors(c) if ours not in ("tok_emb", "w_cls")]
        for ours, layer, tensor, shape in rows:
            if tensor.endswith("dt.b"):
                t = -2.0 + normal(shape, 0.7)
            elif tensor.endswith("A_log"):
                t = torch.log(0.1 + 3.9 * torch.rand(shape, device="cuda", generator=g)).to(dt)
            elif tensor.endswith(".b"):
                t = normal(shape, 0.1)
            elif tensor == "loop.step":
                t = normal(shape, 0.3)
            elif len(shape) == 1:
                t = 1.0 + normal(shape, 0.1)
            else:
                t = normal(shape, shape[1] ** -0.5 * (depth if ours in ("wo", "w2") else 1.0))
            yield ours, layer, t
        return
    depth = (2 * c.n_layers) ** -0.5
    for name, shape in tensor_shapes(c, True).items():
        if name == "tok_emb":
            continue
        for l in range(c.n_layers if len(shape) > 1 else 1):
            s = shape[1:] if len(shape) > 1 else shape
            if name.startswith("rms"):
                yield name, l, 1.0 + 0.1 * torch.randn(s, device="cuda", generator=g)
            else:
                yield name, l, normal(s, 0.02 * (depth if name in ("wo", "w2") else 1.0))


def _tokens(case, seed, n):
    return np.random.default_rng([int(seed), 1]).integers(0, _config(case).vocab_size, n).astype(np.int32)


def _draws(seed, n):
    # away from the last percent at either end, where a confident distribution has no mass to speak of
    return (0.02 + 0.96 * np.random.default_rng([int(seed), 2]).random(n)).astype(np.float32)


def _random_cache(case, seed):
    """Keys and values [kv heads][start][head size] of every layer: a cache that an earlier program has filled."""
    c, g = _config(case), _generator(seed, 1)
    for _ in range(c.n_layers):
        yield [torch.randn((c.n_kv_heads, case["start"], c.head_size), device="cuda", generator=g, dtype=torch.float16) for _ in range(2)]


def _cache_given(case):
    """Contexts beyond a couple of thousand tokens come as a filled cache, shorter ones as tokens."""
    return case["start"] > 4096


# ------------------------------------------------------------------ prepare and run

class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.seed = case, seed
    if case["kind"] == "sample":
        g, V = _generator(seed, 0), case["vocab"]
        s.logits = torch.randn(V, device="cuda", generator=g) * 3.0
        s.logits[torch.randint(0, V, (1,), device="cuda", generator=g)] += 12.0
        s.work = torch.empty_like(s.logits)
        s.history = torch.randint(0, V, (max(case["history"], 1),), device="cuda", generator=g, dtype=torch.int32)
        s.r = float(_draws(seed, 1)[0])
        s.token = torch.zeros(1, device="cuda", dtype=torch.int32)
        return s
    if case["kind"] == "layer":
        return _prepare_layer(s)
    cfg, dt = _config(case), _dtype(case)
    kv = "f32" if dt == torch.float32 else "f16"
    s.engine = Engine(cfg, {torch.float16: "f16", torch.float32: "f32", torch.bfloat16: "bf16"}[dt], kv)
    for name, layer, t in _weights(case, seed):
        s.engine.upload(name, t, layer)
    s.engine.finalize()
    start, n = case["start"], case["n"]
    s.tokens = _tokens(case, seed, start + n + 1)
    s.r = _draws(seed, n)
    if case["kind"] != "generate" and start > 0:
        if _cache_given(case):
            for l, (k, v) in enumerate(_random_cache(case, seed)):
                s.engine.kv_prefill(l, k, v, start)
        else:
            s.engine.prefill(s.tokens[:start], 0)
    s.history = [int(t) for t in s.tokens[:start + 1][-64:]]
    return s


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "sample":
        state.work.copy_(state.logits)
        ops.cuda_sample(state.work, case["vocab"], case["temperature"], case["penalty"], state.history, case["history"], state.r, state.token)
        return {"token": state.token, "logits": state.work}
    if kind == "layer":
        return _run_layer(state)
    e, start, n = state.engine, case["start"], case["n"]
    if kind == "step":
        logits = e.step_logits(int(state.tokens[start]), start)
        return {"logits": logits, "token": e.sample(logits, case["temperature"], case["penalty"], state.history, float(state.r[0]))}
    if kind == "prompt":
        return {"logits": e.extend(state.tokens[start:start + n], start, range(n - case["want"], n))}
    out = {}
    if kind == "generate":
        out["prompt"] = e.extend(state.tokens[:start], 0, [start - 1])
    out["tokens"], _ = e.decode(int(state.tokens[start]), start, n, case["temperature"], case["penalty"], state.history, 64, state.r)
    out["logits"] = e.step_logits(int(out["tokens"][-1]), start + n)
    return out


def _prepare_layer(s):
    c, g = _config(s.case), _generator(s.seed, 0)
    D, F, KV, S = c.dim, c.hidden_dim, c.kv_dim, c.seq_len

    def normal(shape, std, dt=torch.float16):
        return torch.randn(shape, device="cuda", generator=g, dtype=dt) * std

    s.W = {"wq": normal((D, D), 0.02), "wk": normal((KV, D), 0.02), "wv": normal((KV, D), 0.02), "wo": normal((D, D), 0.02),
           "w1": normal((F, D), 0.02), "w3": normal((F, D), 0.02), "w2": normal((D, F), 0.02),
           "n1": 1.0 + normal((D,), 0.1, torch.float32), "n2": 1.0 + normal((D,), 0.1, torch.float32)}
    s.x = normal((D,), 1.0, torch.float32)
    s.kc, s.vc = normal((1, c.n_kv_heads, S, c.head_size), 1.0), normal((1, c.n_kv_heads, S, c.head_size), 1.0)
    new = lambda *shape: torch.zeros(shape, device="cuda")  # noqa: E731
    s.b = dict(xb=new(D), q=new(D), k=new(KV), v=new(KV), att=new(c.n_heads, S), o=new(D), p=new(D), x1=new(D), h1=new(F), h3=new(F),
               hb=new(F), d=new(D), x2=new(D))
    s.cfg = c
    return s


def _run_layer(s):
    c, W, b, pos = s.cfg, s.W, s.b, s.case["start"]
    D, F, KV, S, hs, H, G = c.dim, c.hidden_dim, c.kv_dim, c.seq_len, c.head_size, c.n_heads, c.n_kv_heads
    fp16 = ops.WEIGHT_FP16
    ops.cuda_rmsnorm(b["xb"], s.x, W["n1"], D)
    ops.cuda_gemv(b["q"], b["xb"], W["wq"], D, D, fp16)
    ops.cuda_gemv(b["k"], b["xb"], W["wk"], KV, D, fp16)
    ops.cuda_gemv(b["v"], b["xb"], W["wv"], KV, D, fp16)
    ops.cuda_rope(b["q"], b["k"], pos, D, KV, hs, c.rope_base)
    ops.cuda_scatter_kv(s.kc, s.vc, b["k"], b["v"], 0, pos, G, hs, S)
    ops.cuda_multihead_gemv(b["att"], b["q"], s.kc, 0, pos, H, G, hs, S)
    ops.cuda_scale_multihead(b["att"], hs ** -0.5, H, pos + 1, S)
    ops.cuda_softmax_multihead(b["att"], b["att"], H, pos + 1, S)
    ops.cuda_aggregation_multihead(b["o"], s.vc, b["att"], H, pos + 1, hs, H // G, S)
    ops.cuda_gemv(b["p"], b["o"], W["wo"], D, D, fp16)
    ops.cuda_residual_add(b["x1"], s.x, b["p"], D)
    ops.cuda_rmsnorm(b["xb"], b["x1"], W["n2"], D)
    ops.cuda_gemv(b["h1"], b["xb"], W["w1"], F, D, fp16)
    ops.cuda_gemv(b["h3"], b["xb"], W["w3"], F, D, fp16)
    ops.cuda_swiglu(b["hb"], b["h1"], b["h3"], F)
    ops.cuda_gemv(b["d"], b["hb"], W["w2"], D, F, fp16)
    ops.cuda_residual_add(b["x2"], b["x1"], b["d"], D)
    return {"q": b["q"], "k": b["k"], "v": b["v"], "att": b["att"], "o": b["o"], "hb": b["hb"], "x1": b["x1"], "x2": b["x2"]}


# ------------------------------------------------------------------ what a pass cannot do without

def _sizes(case):
    """Weight elements of one pass over the layers (looped ones counted as often as they run, in "used"), cache elements per
    position, attention multiplications per (token, visible position), windows."""
    c = _config(case)
    if not isinstance(c, LayeredConfig):
        w = c.n_layers * (c.dim * (2 * c.dim + 2 * c.kv_dim) + 3 * c.dim * c.hidden_dim)
        return dict(held=w, used=w, cache=2 * c.n_layers * c.kv_dim, att=2 * c.n_layers * c.dim, window=0)
    held = used = cache = att = window = 0
    for i, y in enumerate(c.layers):
        times = c.loop.times if c.loop and c.loop.start <= i < c.loop.stop else 1
        m, D = y.mixer, c.dim
        if isinstance(m, LatentMixer):
            w = D * (m.heads * (m.dim + m.rot_dim) + m.kv_rank + m.rot_dim + m.heads) + m.heads * (m.dim + m.vdim) * m.kv_rank + D * m.heads * m.vdim
            cache += times * (m.kv_rank + m.rot_dim)
            att += times * m.heads * (m.dim + m.rot_dim + m.vdim)
            window = m.window
        elif isinstance(m, MambaMixer):
            w = D * 3 * m.inner + m.inner * (2 * m.dt_rank + 2 * m.state)
        else:
            w = D * m.dim * (3 * m.heads + m.kv_heads)
            cache += times * m.dim * m.kv_heads
            att += times * m.heads * 2 * m.dim
            window = m.window
        w += 3 * D * y.ff
        held += w
        used += times * w
    return dict(held=held, used=used, cache=cache, att=att, window=window)


def _run_work(case, start, n, passes, logits):
    """n tokens behind `start` others; `passes`: times the weights have to be read, `logits`: rows through the classifier."""
    c, z = _config(case), _sizes(case)
    esz = 4 if _dtype(case) == torch.float32 else 2
    kvsz = 4 if esz == 4 else 2
    span = lambda p: min(p, z["window"]) if z["window"] else p  # noqa: E731
    pairs = sum(span(p + 1) for p in range(start, start + n))
    read = sum(span(p) for p in range(start, start + n)) if passes == n else span(start)
    return {"bytes": passes * z["held"] * esz + (passes if passes == n else 1) * (c.vocab_size * c.dim * esz if logits else 0) + n * c.dim * esz +
            (read + n) * z["cache"] * kvsz + logits * c.vocab_size * 4,
            "flops": 2.0 * n * z["used"] + 2.0 * logits * c.vocab_size * c.dim + 2.0 * pairs * z["att"]}


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": 8.0 * case["vocab"], "flops": 4.0 * case["vocab"]}
    start, n = case["start"], case.get("n", 1)
    if kind == "layer":
        c = _config(case)
        w = c.dim * (2 * c.dim + 2 * c.kv_dim) + 3 * c.dim * c.hidden_dim
        return {"bytes": 2.0 * w + 4.0 * c.kv_dim * (start + 1) + 4.0 * c.n_heads * (start + 1), "flops": 2.0 * w + 4.0 * c.dim * (start + 1)}
    if kind == "prompt":
        return _run_work(case, start, n, 1, case["want"])
    if kind == "step":
        return _run_work(case, start, 1, 1, 1)
    w = _run_work(case, start, n + 1, n + 1, n + 1)
    if kind == "generate":
        p = _run_work(case, 0, start, 1, 1)
        w = {k: w[k] + p[k] for k in w}
    return w


def tolerance(case):
    """About four times the error against 64 bits: rounding of FP16 cache rows, queries and probabilities where there are any
    (4e-6 to 4e-5 with the size of the model), else of 32-bit sums (operators: single-precision angles, 1.5e-5)."""
    if case["kind"] == "sample":
        return {"rel": 1e-5}
    if case["kind"] == "layer":
        return {"rel": 6e-5}
    return {"rel": 2e-6} if _dtype(case) == torch.float32 else {"rel": 1.5e-4}


# ------------------------------------------------------------------ the same in 64 bits

def _norm64(x, w, eps, b=None):
    if b is not None:
        x = x - x.mean(-1, keepdim=True)
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w
    return y + b if b is not None else y


def _turn(x, angles, magnitude=1.0):
    """x [tokens, heads, d]: neighbours 2i, 2i + 1 turn by angles[token, i]."""
    n = 2 * angles.shape[-1]
    c, s = (angles.cos() * magnitude)[:, None], (angles.sin() * magnitude)[:, None]
    u, v = x[..., 0:n:2], x[..., 1:n:2]
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., n:]], -1)


def _attend(q, k, v, scale, window=0, cap=0.0):
    """q [n, H, d] of the last n of m positions, k and v [m, G, .]."""
    n, H, m, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    i, j = torch.arange(m - n, m, device="cuda")[:, None], torch.arange(m, device="cuda")[None]
    hidden = (j > i) | ((i - j >= window) if window else False)
    out = torch.empty((n, H, v.shape[2]), device="cuda", dtype=torch.float64)
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].T * scale
        s = (cap * torch.tanh(s / cap) if cap else s).masked_fill(hidden, -math.inf)
        out[:, h] = torch.softmax(s, 1) @ v[:, h * G // H]
    return out.reshape(n, -1)


def _llama_angles(c, pos):
    """Rotation angles in the single precision that the model format's table has."""
    hs = c.head_size
    f = np.float32(1) / np.power(np.float32(c.rope_base), (2 * np.arange(hs // 2, dtype=np.float32)) / np.float32(hs)).astype(np.float32)
    return torch.from_numpy((pos.astype(np.float32)[:, None] * f[None].astype(np.float32)).astype(np.float64)).cuda()


def _yarn_angles(rot, pos):
    y, f = rot.yarn, []
    border = lambda turns: rot.dims * math.log(y.original / (2 * math.pi * turns)) / (2 * math.log(rot.base))  # noqa: E731
    lo, hi = max(math.floor(border(y.fast)), 0), min(math.ceil(border(y.slow)), rot.dims - 1)
    for i in range(rot.dims // 2):
        a, blend = rot.base ** (-2.0 * i / rot.dims), min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
        f.append(a / y.factor * blend + a * (1 - blend))
    return torch.from_numpy(pos.astype(np.float64)[:, None] * np.array(f)[None]).cuda(), 0.1 * math.log(y.factor) + 1.0


class _Model64:
    """The case's model in 64 bits; keeps what a sequence leaves behind, like the engine."""

    def __init__(self, case, seed):
        self.c, self.case = _config(case), case
        self.W = {(name, layer): t for name, layer, t in _weights(case, seed)}
        self.left, self.length = {}, 0
        if _cache_given(case):
            for l, (k, v) in enumerate(_random_cache(case, seed)):
                self.left[l] = (k.transpose(0, 1), v.transpose(0, 1))
            self.length = case["start"]

    def w(self, name, layer=0):
        return self.W[name, layer].double()

    def grown(self, run, *rows):
        old = self.left.get(run)
        self.left[run] = tuple(torch.cat([a, b.to(a.dtype) if _cache_given(self.case) else b]) for a, b in zip(old, rows)) if old else rows
        return tuple(t.double() for t in self.left[run])

    def extend(self, tokens, want=1):
        c = self.c
        pos = np.arange(self.length, self.length + len(tokens))
        self.length += len(tokens)
        x = self.w("tok_emb")[torch.as_tensor(np.asarray(tokens), device="cuda", dtype=torch.long)]
        if isinstance(c, LayeredConfig):
            x = self.layered(x, pos)
            x = _norm64(x[-want:], self.w("rms_final"), c.norm_eps, self.w("norm_final_b") if c.norm == "layer" else None)
        else:
            for l in range(c.n_layers):
                x = self.llama_layer(x, l, pos)
            x = _norm64(x[-want:], self.w("rms_final"), 1e-5)
        return x @ self.w("w_cls").T

    def llama_layer(self, x, l, pos):
        c, n, hs = self.c, x.shape[0], self.c.head_size
        h, a = _norm64(x, self.w("rms_att", l), 1e-5), _llama_angles(c, pos)
        q = _turn((h @ self.w("wq", l).T).view(n, -1, hs), a)
        k = _turn((h @ self.w("wk", l).T).view(n, -1, hs), a)
        k, v = self.grown(l, k, (h @ self.w("wv", l).T).view(n, -1, hs))
        x = x + _attend(q, k, v, hs ** -0.5) @ self.w("wo", l).T
        h = _norm64(x, self.w("rms_ffn", l), 1e-5)
        return x + (torch.nn.functional.silu(h @ self.w("w1", l).T) * (h @ self.w("w3", l).T)) @ self.w("w2", l).T

    def layered(self, x, pos):
        c, run = self.c, 0
        lo, hi, times = (c.loop.start, c.loop.stop, c.loop.times) if c.loop else (0, 0, 0)
        order = list(range(lo)) + [l for _ in range(times) for l in range(lo, hi)] + list(range(hi, c.n_layers))
        passes = 0
        for run, l in enumerate(order):
            if hi > lo and l == lo:
                x, passes = x + self.w("loop_step")[passes], passes + 1
            y = c.layers[l]
            ln = c.norm == "layer"
            h = _norm64(x, self.w("rms_att", l), c.norm_eps, self.w("norm1_b", l) if ln else None)
            mixer = self.latent if isinstance(y.mixer, LatentMixer) else self.scan if isinstance(y.mixer, MambaMixer) else self.shared
            x = x + mixer(h, l, run, y.mixer, pos)
            if y.ff:
                h = _norm64(x, self.w("rms_ffn", l), c.norm_eps, self.w("norm2_b", l) if ln else None)
                act = torch.nn.functional.silu if y.act == "silu" else lambda z: torch.nn.functional.gelu(z, approximate="tanh")
                x = x + (act(h @ self.w("w1", l).T) * (h @ self.w("w3", l).T)) @ self.w("w2", l).T
        return x

    def latent(self, h, l, run, m, pos):
        n, (a, mag) = h.shape[0], _yarn_angles(m.rotation, pos)
        q = (h @ self.w("lat_q", l).T).view(n, m.heads, -1)
        d = h @ self.w("lat_dkv", l).T
        lat = _norm64(d[:, :m.kv_rank], self.w("lat_norm", l), self.c.norm_eps)
        lat, kr = self.grown(run, lat, _turn(d[:, None, m.kv_rank:], a, mag)[:, 0])
        k = torch.cat([(lat @ self.w("lat_uk", l).T).view(-1, m.heads, m.dim), kr[:, None].expand(-1, m.heads, -1)], -1)
        q = torch.cat([q[..., :m.dim], _turn(q[..., m.dim:], a, mag)], -1)
        o = _attend(q, k, (lat @ self.w("lat_uv", l).T).view(-1, m.heads, m.vdim), m.scale, m.window)
        gate = torch.sigmoid(h @ self.w("lat_g", l).T)
        return (o.view(n, m.heads, -1) * gate[..., None]).reshape(n, -1) @ self.w("wo", l).T

    def shared(self, h, l, run, m, pos):
        n, (a, mag) = h.shape[0], _yarn_angles(m.rotation, pos)
        q = _turn((h @ self.w("wq", l).T + self.w("wq_b", l)).view(n, m.heads, -1), a, mag)
        v = (h @ self.w("wk", l).T + self.w("wk_b", l)).view(n, m.kv_heads, -1)
        k, v = self.grown(run, _turn(v, a, mag), v)
        o = _attend(q, k, v, m.scale, m.window, m.softcap)
        return (o * torch.sigmoid(h @ self.w("wg", l).T)) @ self.w("wo", l).T + self.w("wo_b", l)

    def scan(self, h, l, run, m, pos):
        n = h.shape[0]
        xz = h @ self.w("scan_in", l).T
        old, S = self.left.get(run) or (torch.zeros((m.conv - 1, m.inner), device="cuda", dtype=torch.float64),
                                        torch.zeros((m.inner, m.state), device="cuda", dtype=torch.float64))
        line = torch.cat([old, xz[:, :m.inner]])
        taps = self.w("scan_conv", l)
        x = torch.nn.functional.silu(sum(line[i:i + n] * taps[:, i] for i in range(m.conv)) + self.w("scan_conv_b", l))
        low = x @ self.w("scan_low", l).T
        dt = torch.nn.functional.softplus(low[:, :m.dt_rank] @ self.w("scan_dt", l).T + self.w("scan_dt_b", l))
        A, B, C = -torch.exp(self.w("scan_a_log", l)), low[:, m.dt_rank:m.dt_rank + m.state], low[:, m.dt_rank + m.state:]
        y = torch.empty_like(x)
        for t in range(n):
            S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * x[t])[:, None] * B[t][None]
            y[t] = S @ C[t]
        self.left[run] = (line[n:], S)
        return ((y + self.w("scan_d", l) * x) * torch.nn.functional.silu(xz[:, m.inner:])) @ self.w("wo", l).T


def _sample64(logits, temperature, penalty, history, r):
    """(token, logits after penalty and temperature)"""
    v = logits.clone()
    if penalty > 1:
        for t in history:
            v[t] = v[t] / penalty if v[t] > 0 else v[t] * penalty
    if temperature == 0:
        return int(v.argmax()), v
    v = v / temperature
    return min(int((torch.softmax(v, 0).cumsum(0) <= r).sum()), v.numel() - 1), v


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "sample":
            s = prepare(case, seed)
            history = s.history.tolist()[:case["history"]]
            scaled = _sample64(s.logits.double(), case["temperature"], case["penalty"], history, s.r)[1]
            # like the reference's, the buffer ends up as probabilities; a greedy draw leaves it alone
            return {"token": None, "logits": torch.softmax(scaled, 0) if case["temperature"] else s.logits.double()}
        if kind == "layer":
            return _exact_layer(case, seed)
        m, start, n = _Model64(case, seed), case["start"], case["n"]
        tokens = _tokens(case, seed, start + n + 1)
        if kind == "prompt":
            if start:
                m.extend(tokens[:start])
            return {"logits": m.extend(tokens[start:start + n], case["want"])}
        out = {}
        if m.length < start:
            head = m.extend(tokens[:start])
            if kind == "generate":
                out["prompt"] = head
        logits = m.extend(tokens[start:start + 1])
        if kind == "step":
            return {"logits": logits[0], "token": None}
        history, token = [int(t) for t in tokens[:start + 1][-64:]], 0
        r = _draws(seed, n)
        for i in range(n):
            token, _ = _sample64(logits[0], case["temperature"], case["penalty"], history, float(r[i]))
            history = (history + [token])[-64:]
            logits = m.extend([token])
        out.update(tokens=None, logits=logits[0])
        return out


def _exact_layer(case, seed):
    s = _State()
    s.case, s.seed = case, seed
    s = _prepare_layer(s)
    c, pos, D = s.cfg, case["start"], s.cfg.dim
    W = {k: v.double() for k, v in s.W.items()}
    x, hs = s.x.double(), c.head_size
    h, a = _norm64(x, W["n1"], 1e-5), _llama_angles(c, np.array([pos]))
    q, k = [_turn((W[w] @ h).view(1, -1, hs), a) for w in ("wq", "wk")]
    v = W["wv"] @ h
    keys, values = s.kc[0, :, :pos + 1].double(), s.vc[0, :, :pos + 1].double()
    keys[:, pos], values[:, pos] = k[0].half().double(), v.view(-1, hs).half().double()
    g = c.n_heads // c.n_kv_heads
    att = torch.zeros((c.n_heads, c.seq_len), device="cuda", dtype=torch.float64)
    att[:, :pos + 1] = torch.softmax((q.view(-1, g, hs) @ keys.transpose(1, 2)).reshape(c.n_heads, -1) * hs ** -0.5, 1)
    o = (att[:, :pos + 1].reshape(-1, g, pos + 1) @ values).reshape(-1)
    x1 = x + W["wo"] @ o
    h = _norm64(x1, W["n2"], 1e-5)
    hb = torch.nn.functional.silu(W["w1"] @ h) * (W["w3"] @ h)
    return {"q": q.view(-1), "k": k.view(-1), "v": v, "att": att, "o": o, "hb": hb, "x1": x1, "x2": x1 + W["w2"] @ hb}

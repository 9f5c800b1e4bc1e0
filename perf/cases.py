"""The work that programs give this framework, as cases that can be timed and checked.

Three kinds of programs: callers of the reference's kernel symbols (one matvec on raw quantized blocks),
hosts of the quantized decode engine (prompt and greedy tokens, or one fused step per call), and hosts of
models described layer by layer (Mitotar, Kuzipel: prompts, greedy tokens, replayed traces).  Sizes are
those of the named configurations; where a configuration has many equal layers, a few of them stand for
all, so that a model is made in about a second.

Weights are random and made from the seed.  Two things about them are as in a trained model and unlike
plain noise: the next token is clear (the head points from a token's embedding to another token's row, so
rounding decides no argmax), and so is the router's choice (some channels of the residual keep each token's
own levels, and the router reads those).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mongoose_b200 import configs as mc
from mongoose_b200 import kernels, synthetic
from mongoose_b200.fused_infer import CUDAFusedInference
from mongoose_b200.layered import (MATH, NORM_LAYER, LatentAttention, LayeredInference, ParallelLayer, cache_bytes_per_position, prefill_flops,
                                   slot_shapes, state_bytes, weight_bytes_per_token)

FORMATS = {"q8_0": mc.FMT_Q8_0, "q4_0": mc.FMT_Q4_0, "f16": mc.FMT_F16}
DENSE = {"qwen2.5-0.5b": mc.QWEN25_05B, "tinyllama-1.1b": mc.TINYLLAMA_11B, "qwen2.5-7b-class": mc.QWEN25_7B}
F64 = torch.float64


# ---- the cases ------------------------------------------------------------------------------------

def listed():
    return [
        # the smallest call: one projection of a 0.5B model through the reference's kernel symbol
        {"name": "matvec q8_0 4864x896", "do": "matvec", "format": "q8_0", "rows": 4864, "cols": 896},
        # the largest matrix of a 7B-class layer through the same family of symbols
        {"name": "matvec q4_0 3584x18944", "do": "matvec", "format": "q4_0", "rows": 3584, "cols": 18944},
        # a short chat turn on the 0.5B model, Q8_0 as most files of it are
        {"name": "generate 0.5b q8_0", "do": "generate", "model": "qwen2.5-0.5b", "layers": 24, "format": "q8_0", "head": "q8_0",
         "prompt": 32, "new": 200},
        # the same with 4-bit layers and everything else in fp16
        {"name": "generate 0.5b q4_0", "do": "generate", "model": "qwen2.5-0.5b", "layers": 24, "format": "q4_0", "head": "f16",
         "prompt": 32, "new": 200},
        # a long question with a long answer, 1.1B widths
        {"name": "generate 1.1b-width q8_0", "do": "generate", "model": "tinyllama-1.1b", "layers": 6, "format": "q8_0", "head": "q8_0",
         "prompt": 512, "new": 512},
        # a host that drives the model one fused step per call, hidden state in and logits out, 1.1B widths
        {"name": "step 1.1b-width q8_0", "do": "step", "model": "tinyllama-1.1b", "layers": 4, "format": "q8_0", "head": "q8_0", "context": 301},
        # 7B-class widths, where the weight stream is what counts
        {"name": "generate 7b-width q8_0", "do": "generate", "model": "qwen2.5-7b-class", "layers": 2, "format": "q8_0", "head": "q8_0",
         "prompt": 128, "new": 128},
        # a whole document into a Mitotar model, logits where a caller scores it
        {"name": "prompt mitotar-1.1b", "do": "replay", "model": "mitotar-1.1b", "layers": 6, "math": "bfloat16", "prompt": 2048, "portions": 1,
         "steps": 0},
        # a chat turn on it
        {"name": "generate mitotar-1.1b", "do": "generate", "model": "mitotar-1.1b", "layers": 6, "math": "bfloat16", "prompt": 300, "new": 64},
        # a document of no round length into a Kuzipel model, in two portions
        {"name": "prompt kuzipel-1.1b", "do": "replay", "model": "kuzipel-1.1b", "layers": 6, "math": "bfloat16", "prompt": 1500, "portions": 2,
         "steps": 0},
        # a chat turn on it
        {"name": "generate kuzipel-1.1b", "do": "generate", "model": "kuzipel-1.1b", "layers": 6, "math": "bfloat16", "prompt": 300, "new": 64},
        # a short trace in 32-bit arithmetic, as one replays it to compare two implementations
        {"name": "replay mitotar-0.5b f32", "do": "replay", "model": "mitotar-0.5b", "layers": 4, "math": "float32", "prompt": 333, "portions": 3,
         "steps": 13},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(("matvec", "generate", "generate", "replay", "replay", "step"))
    if do == "matvec":
        return {"do": do, "format": rng.choice(("q8_0", "q4_0")), "rows": _log_uniform(rng, 100, 20000), "cols": 32 * _log_uniform(rng, 8, 600)}
    if do == "generate" and rng.random() < 0.6 or do == "step":
        model = rng.choice(tuple(DENSE))
        fmt = rng.choice(("q8_0", "q8_0", "q4_0", "f16"))
        case = {"do": do, "model": model, "layers": rng.randint(1, 2 if "7b" in model else 5), "format": fmt,
                "head": "q8_0" if fmt == "q8_0" else "f16"}
        if do == "step":
            return {**case, "context": _log_uniform(rng, 2, 380)}
        return {**case, "prompt": _log_uniform(rng, 1, 700), "new": _log_uniform(rng, 2, 250)}
    model = rng.choice(("mitotar-0.5b", "mitotar-1.1b", "mitotar-7b-width-4l", "kuzipel-0.5b", "kuzipel-1.1b", "kuzipel-7b-width-4l"))
    wide = "7b" in model
    case = {"do": do, "model": model, "layers": rng.randint(3, 4) if "kuzipel" in model else rng.randint(1, 2 if wide else 5)}
    if do == "generate":
        return {**case, "math": "bfloat16", "prompt": _log_uniform(rng, 2, 1200), "new": _log_uniform(rng, 2, 80)}
    math_ = "float32" if rng.random() < 0.2 else "bfloat16"
    prompt = _log_uniform(rng, 3, (150 if wide else 400) if math_ == "float32" else 2048)
    return {**case, "math": math_, "prompt": prompt, "portions": rng.randint(1, min(3, prompt)), "steps": rng.choice((0, 0, rng.randint(1, 12)))}


def _config(case):
    if "math" in case:
        c = synthetic.LAYERED[case["model"]]
        n = case["layers"]
        layers = c.layers[:n] if case["model"].startswith("mitotar") else c.layers[:n - 1]      # Kuzipel's first recurrent layer runs twice
        return c.with_(layers=layers, math=MATH[case["math"]])
    c = DENSE[case["model"]]
    length = case["context"] + 1 if case["do"] == "step" else case["prompt"] + case["new"] + 1
    return c.with_(n_layers=case["layers"], layer_fmt=FORMATS[case["format"]], head_fmt=FORMATS[case["head"]], max_seq=max(c.max_seq, length))


# ---- inputs ----------------------------------------------------------------------------------------

def _generator(seed, idx):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + idx) % (1 << 62))


def _randn(seed, idx, *shape):
    return torch.randn(shape, generator=_generator(seed, idx), device="cuda")


def _ids(seed, n, vocab):
    return torch.randint(0, vocab, (n,), generator=_generator(seed, 1 << 30), device="cuda", dtype=torch.int32)


def _quantize(fmt, w):
    """(raw blocks, values): the bytes of GGUF blocks or halves, and a function that gives the values they hold in 64 bits."""
    rows, cols = w.shape
    if fmt == mc.FMT_F16:
        h = w.half()
        return h.view(torch.uint8), lambda: h.to(F64)
    b = w.view(rows, cols // 32, 32)
    amax = b.abs().amax(-1, keepdim=True)
    top = 127.0 if fmt == mc.FMT_Q8_0 else 8.0
    d = (amax / top).half()
    q = torch.round(b * torch.where(amax > 0, top / amax, torch.zeros_like(amax)))
    if fmt == mc.FMT_Q8_0:
        q = q.clamp_(-127, 127).to(torch.int8)
        raw = torch.cat((d.view(torch.uint8), q.view(torch.uint8)), -1)
    else:
        q = q.clamp_(-8, 7).to(torch.int8)
        nib = (q + 8).view(torch.uint8)
        raw = torch.cat((d.view(torch.uint8), nib[..., :16] | (nib[..., 16:] << 4)), -1)
    return raw.reshape(rows, -1), lambda: (d.to(F64) * q.to(F64)).view(rows, cols)


def _dense_weights(cfg, seed):
    """Yield (slot, raw blocks or fp32 vector, values in 64 bits as a function)."""
    biased = cfg.name.startswith("qwen")
    for i in range(cfg.n_layers):
        b = 12 * i
        for s in range(12):
            if s in mc.MATRIX_SLOTS:
                yield (b + s, *_quantize(cfg.layer_fmt, _randn(seed, b + s, *cfg.matrix_shape(s)).mul_(0.02)))
            elif s in (mc.SLOT_NORM1, mc.SLOT_NORM2):
                v = 1.0 + 0.1 * _randn(seed, b + s, cfg.dim)
                yield b + s, v, v.double
            elif biased:
                v = 0.1 * _randn(seed, b + s, cfg.dim if s == mc.SLOT_BQ else cfg.kv_dim)
                yield b + s, v, v.double
    b = 12 * cfg.n_layers
    v = 1.0 + 0.1 * _randn(seed, b, cfg.dim)
    yield b, v, v.double
    yield (b + 1, *_quantize(cfg.head_fmt, _randn(seed, b + 1, cfg.vocab, cfg.dim)))


def _next_tokens(seed, vocab):
    """The token that a layer-described model of these cases gives after each."""
    return torch.randperm(vocab, generator=_generator(seed, (1 << 30) + 1), device="cuda")


def _layered_weights(cfg, seed):
    """Yield (slot, name, layer, bf16 tensor); vectors are flat."""
    moes = [l.moe for l in cfg.layers if getattr(l, "moe", None)]
    kept = max((m.experts for m in moes), default=0)        # channels that keep each token's own levels for the router
    around_zero = {"at.bias", "mem.i_bias"} | ({"norm1", "norm2", "final_norm"} if cfg.norm != NORM_LAYER else set())
    neutral = {"mem.f_bias": 3.0, "wkv.w0": -2.0, **{"wkv.mu_" + t: 0.5 for t in "rkvgw"}}

    def embedding():
        e = _randn(seed, 1 << 20, cfg.vocab, cfg.width)
        if kept:
            e[:, :kept] = torch.argsort(torch.rand(cfg.vocab, kept, generator=_generator(seed, (1 << 20) + 1), device="cuda"), -1).float() - 0.5 * kept
        return e

    for idx, name, layer, rows, cols in slot_shapes(cfg):
        if name == "embed":
            w = embedding()
        elif name == "head":
            w = torch.empty(rows, cols, device="cuda")
            w[_next_tokens(seed, cfg.vocab)] = embedding().mul_(cols ** -0.5)
            w[:, :kept] = 0
        elif name == "loop_in":
            w = _randn(seed, idx, rows, cols).mul_(0.1 * cols ** -0.5)
            w[:kept] = 0
            w[:, :rows] += 0.5 * torch.eye(rows, device="cuda")
            w[:, rows:] += 0.5 * torch.eye(rows, device="cuda")
        elif name == "moe.router":
            w = torch.zeros(rows, cols, device="cuda")
            w[:, :rows] = torch.eye(rows, device="cuda")
        elif name == "at.talk":
            n = cfg.layers[layer].attn.heads
            w = (torch.eye(n, device="cuda") + 0.3 * n ** -0.5 * _randn(seed, idx, n, n)).view(-1)
        elif rows:
            w = _randn(seed, idx, rows, cols).mul_(cols ** -0.5)
        elif name == "moe.bias":
            w = 0.05 * _randn(seed, idx, cols)
        else:
            w = neutral.get(name, 0.0 if name in around_zero else 1.0) + 0.2 * _randn(seed, idx, cols)
            if kept and name in ("norm1", "norm2"):
                w[:kept] = 1.0
            elif kept and name in ("ls1", "ls2"):
                w[:kept] = 0.0
        yield idx, name, layer, w.bfloat16()


def _matvec_inputs(case, seed):
    rows, cols = case["rows"], case["cols"]
    return (*_quantize(FORMATS[case["format"]], _randn(seed, 0, rows, cols).mul_(0.02)), _randn(seed, 1, cols))


def _portions(case):
    """Ends of the prompt's portions."""
    n, p = case["prompt"], case["portions"]
    return [n * (i + 1) // p for i in range(p)]


def prepare(case, seed):
    if case["do"] == "matvec":
        raw, _, x = _matvec_inputs(case, seed)
        return {"case": case, "w": raw, "x": x, "out": torch.empty(case["rows"], device="cuda")}
    cfg = _config(case)
    if "math" in case:
        engine = LayeredInference(cfg)
        for idx, _, _, w in _layered_weights(cfg, seed):
            engine.SetWeightBF16(idx, w.view(torch.int16).cpu().numpy().view(np.uint16))
    else:
        engine = CUDAFusedInference(cfg)
        for idx, w, _ in _dense_weights(cfg, seed):
            if w.dtype == torch.uint8:
                engine.SetWeightRaw(idx, w.cpu().numpy(), cfg.head_fmt if idx > 12 * cfg.n_layers else cfg.layer_fmt)
            else:
                engine.SetWeight(idx, w.cpu().numpy())
    engine.BuildFusedDispatch()
    state = {"case": case, "engine": engine}
    if case["do"] == "step":
        n = case["context"]
        engine.Forward(_ids(seed, n, cfg.vocab).cpu().numpy(), 0)
        state["hidden"] = _randn(seed, 1 << 29, cfg.dim).cpu().pin_memory()
        state["logits"] = torch.empty(cfg.vocab, pin_memory=True)
    elif case["do"] == "generate":
        state["tokens"] = _ids(seed, case["prompt"], cfg.vocab).cpu().numpy()
        state["logits"] = np.empty(cfg.vocab, np.float32)
    else:
        state["tokens"] = _ids(seed, case["prompt"] + case["steps"], cfg.vocab).cpu().numpy()
    return state


# ---- one pass --------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    if case["do"] == "matvec":
        f = kernels.KQ8_0Matvec if case["format"] == "q8_0" else kernels.KQ4_0Matvec
        f(state["x"], state["w"], state["out"], case["rows"], case["cols"])
        return state["out"]
    engine = state["engine"]
    if case["do"] == "step":
        engine.PartialStep(state["hidden"], case["context"], 0, engine.cfg.n_layers, None, state["logits"])
        return state["logits"]
    if case["do"] == "generate":            # the answer's tokens, and the logits behind the last one
        n, new = case["prompt"], case["new"]
        tokens = engine.Generate(state["tokens"], new)
        engine.StepToken(int(tokens[-1]), n + new - 1, state["logits"])
        return {"tokens": tokens, "logits": state["logits"]}
    logits, at = [], 0
    for end in _portions(case):             # the logits behind the middle and the last token of every portion
        n = end - at
        logits.append(engine.Forward(state["tokens"][at:end], at, sorted({n // 2, n - 1})))
        at = end
    for i in range(case["steps"]):
        logits.append(engine.Forward(state["tokens"][at + i:at + i + 1], at + i, (0,)))
    return logits


# ---- what a pass cannot do without -----------------------------------------------------------------

def work(case):
    if case["do"] == "matvec":
        rows, cols = case["rows"], case["cols"]
        return {"bytes": rows * mc.fmt_row_bytes(FORMATS[case["format"]], cols) + 4 * (rows + cols), "flops": 2 * rows * cols}
    cfg = _config(case)
    if "math" in case:
        n, m = case["prompt"], case["new"] if case["do"] == "generate" else case["steps"]
        prompts = case.get("portions", 1)
        outs = 2 * prompts + m
        stream, cached = weight_bytes_per_token(cfg), cache_bytes_per_position(cfg)
        # a portion reads every weight (all experts), a step those it chooses, the cache so far and the state (which it writes)
        whole = sum(2 * r * c for _, name, _, r, c in slot_shapes(cfg) if name != "embed")
        return {"bytes": prompts * whole + m * (stream + 2 * state_bytes(cfg)) + cached * (n + m * (n + m / 2)) + outs * 4 * cfg.vocab,
                "flops": prefill_flops(cfg, n + m) + 2.0 * cfg.width * cfg.vocab * outs}
    stream, kv = mc.weight_bytes_per_token(cfg), mc.kv_bytes_per_position(cfg)
    layer = cfg.n_layers * sum(r * c for r, c in map(cfg.matrix_shape, mc.MATRIX_SLOTS))
    head = cfg.vocab * cfg.dim
    if case["do"] == "step":
        return {"bytes": stream + kv * (case["context"] + 1) + 4 * cfg.vocab, "flops": 2 * (layer + head)}
    n, m = case["prompt"], case["new"]
    attend = 2 * cfg.n_layers * cfg.dim * (n + m) ** 2
    return {"bytes": stream * (1 + m) + kv * (n + m * (n + m / 2)) + 4 * cfg.vocab, "flops": 2 * (layer * (n + m) + head * (m + 1)) + attend}


def tolerance(case):
    if case["do"] == "matvec":              # fp32 sums in another order
        return {"rel": 1e-6, "max": 1e-5}
    if "math" not in case:                  # keys and values are rounded to fp16 (1e-4 to 3.4e-4 off 64 bits): a sum's last bit moves some of them
        return {"rel": 1e-3, "max": 1e-2}
    if case["math"] == "float32":           # up to 4e-6 off 64 bits
        return {"rel": 3e-5, "max": 1e-3}
    return {"rel": 0.03, "max": 0.5}        # bf16 inputs of every product: up to 8e-3 off 64 bits


# ---- the same in 64 bits, by plain torch -----------------------------------------------------------

def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _dense_model(cfg, seed):
    """A function of (tokens, last hidden state or None) -> the final hidden states [n, dim], and the head."""
    w = {idx: values for idx, _, values in _dense_weights(cfg, seed)}
    head = w[12 * cfg.n_layers + 1]()
    H, KV, D = cfg.n_heads, cfg.n_kv_heads, cfg.head_dim
    freq = float(cfg.rope_theta) ** (-torch.arange(0, D, 2, device="cuda", dtype=F64) / D)

    def rope(x):
        a = torch.arange(x.shape[0], device="cuda", dtype=F64)[:, None, None] * freq
        u, v = x[..., :D // 2], x[..., D // 2:]
        return torch.cat((u * a.cos() - v * a.sin(), u * a.sin() + v * a.cos()), -1)

    def hidden(tokens, last=None):
        x = head[tokens.long()]
        if last is not None:
            x = torch.cat((x, last[None].double()))
        n = x.shape[0]
        mask = torch.ones(n, n, device="cuda", dtype=torch.bool).tril()
        for i in range(cfg.n_layers):
            g = lambda s: w[12 * i + s]()
            bias = lambda s: w[12 * i + s]() if 12 * i + s in w else 0.0
            y = _rms(x, cfg.eps) * g(mc.SLOT_NORM1)
            q = rope((y @ g(mc.SLOT_WQ).T + bias(mc.SLOT_BQ)).view(n, H, D))
            k = rope((y @ g(mc.SLOT_WK).T + bias(mc.SLOT_BK)).view(n, KV, D)).repeat_interleave(H // KV, 1)
            v = (y @ g(mc.SLOT_WV).T + bias(mc.SLOT_BV)).view(n, KV, D).repeat_interleave(H // KV, 1)
            s = torch.einsum("ihd,jhd->hij", q, k) * D ** -0.5
            o = torch.einsum("hij,jhd->ihd", s.masked_fill_(~mask, -math.inf).softmax(-1), v)
            x = x + o.reshape(n, -1) @ g(mc.SLOT_WO).T
            y = _rms(x, cfg.eps) * g(mc.SLOT_NORM2)
            x = x + (torch.nn.functional.silu(y @ g(mc.SLOT_GATE).T) * (y @ g(mc.SLOT_UP).T)) @ g(mc.SLOT_DOWN).T
        return _rms(x, cfg.eps) * w[12 * cfg.n_layers]()

    return hidden, head


def _gate_attention(a, w, h, eps):
    n, H, KV, D = h.shape[0], a.heads, a.kv_heads, a.dim
    pos = torch.arange(n, device="cuda", dtype=F64)
    temp = 1.0 + a.temp_coef * torch.log(torch.floor((pos + 1) / a.temp_every) + 1)
    q = _rms((h @ w["at.q"].T).view(n, H, D), eps) * w["at.q_norm"] * temp[:, None, None]
    k = (h @ w["at.k"].T).view(n, KV, D).repeat_interleave(H // KV, 1)
    kn = _rms(k, eps) * w["at.k_norm"]
    slope = 2.0 ** (-8.0 * torch.arange(1, H + 1, device="cuda", dtype=F64) / H)
    talk, out = w["at.talk"].view(H, H), []
    for r in range(0, n, 256):
        i = pos[r:r + 256]
        s = torch.einsum("ihd,jhd->hij", q[r:r + 256], kn) * a.scale
        s -= slope[:, None, None] * (i[:, None] - pos)
        s = (s + w["at.bias"][:, None, None]).sigmoid_().masked_fill_(pos > i[:, None], 0.0)
        out.append(torch.einsum("hij,jhd->ihd", torch.einsum("hg,gij->hij", talk, s), k))
    return torch.cat(out).reshape(n, -1) @ w["at.o"].T


def _matrix_memory(a, w, h, eps):
    n, H = h.shape[0], a.heads
    q = (h @ w["mem.q"].T).view(n, H, a.dim) * a.dim ** -0.5
    k = (h @ w["mem.k"].T).view(n, H, a.dim)
    v = (h @ w["mem.v"].T).view(n, H, a.vdim)
    cap = lambda z: a.gate_cap * torch.tanh(z / a.gate_cap)
    ig = cap(h @ w["mem.i"].T + w["mem.i_bias"])
    f = torch.nn.functional.logsigmoid(cap(h @ w["mem.f"].T + w["mem.f_bias"])).cumsum(0)
    later, out = torch.ones(n, n, device="cuda", dtype=torch.bool).triu(1), []
    for x in range(H):
        d = (f[:, x, None] - f[None, :, x] + ig[None, :, x]).masked_fill(later, -math.inf)
        m = torch.maximum(d.amax(-1), f[:, x])
        s = torch.exp(d - m[:, None]) * (q[:, x] @ k[:, x].T)
        out.append(s @ v[:, x] / (torch.maximum(s.sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None])
    y = _rms(torch.stack(out, 1), eps).reshape(n, -1) * w["mem.norm"] * torch.sigmoid(h @ w["mem.g"].T)
    return y @ w["mem.o"].T


def _latent_attention(a, w, h, eps):
    n, H = h.shape[0], a.heads
    half = a.rot_dim // 2
    angle = torch.arange(n, device="cuda", dtype=F64)[:, None] * a.rot_base ** (-torch.arange(half, device="cuda", dtype=F64) / half)

    def turn(x):
        c = angle.view(n, *[1] * (x.dim() - 2), half)
        u, v = x[..., :half], x[..., half:]
        return torch.cat((u * c.cos() - v * c.sin(), v * c.cos() + u * c.sin()), -1)

    q = (_rms(h @ w["la.dq"].T, eps) * w["la.dq_norm"] @ w["la.uq"].T).view(n, H, -1)
    down = h @ w["la.dkv"].T
    c, t = _rms(down[:, :a.kv_rank], eps) * w["la.dkv_norm"], turn(down[:, a.kv_rank:])
    qr = turn(q[..., a.dim:])
    k, v = (c @ w["la.uk"].T).view(n, H, a.dim), (c @ w["la.uv"].T).view(n, H, a.vdim)
    later, out = torch.ones(n, n, device="cuda", dtype=torch.bool).triu(1), []
    for x in range(H):
        s = (q[:, x, :a.dim] @ k[:, x].T + qr[:, x] @ t.T) * a.scale
        out.append(s.masked_fill_(later, -math.inf).softmax(-1) @ v[:, x])
    return torch.stack(out, 1).reshape(n, -1) @ w["la.o"].T


def _recurrence(a, w, h, eps):
    n, H, D = h.shape[0], a.heads, a.dim
    before = torch.cat((torch.zeros_like(h[:1]), h[:-1]))
    mix = {t: h + (before - h) * w["wkv.mu_" + t] for t in "rkvgw"}
    r, k, v = ((mix[t] @ w["wkv." + t].T).view(n, H, D) for t in "rkv")
    d = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w["wkv.w1"].T) @ w["wkv.w2"].T + w["wkv.w0"])).view(n, H, D, 1)
    u, state, out = w["wkv.u"].view(H, D, 1), torch.zeros(H, D, D, device="cuda", dtype=F64), []
    for t in range(n):
        kv = k[t, :, :, None] * v[t, :, None]
        out.append((r[t, :, None] @ torch.addcmul(state, u, kv)).view(H, D))
        state = torch.addcmul(kv, d[t], state)
    y = _rms(torch.stack(out), eps).reshape(n, -1) * w["wkv.norm"] * torch.nn.functional.silu(mix["g"] @ w["wkv.g"].T)
    return y @ w["wkv.o"].T


def _experts(e, w, h):
    z = h @ w["moe.router"].T + w["moe.bias"]
    top, chosen = z.topk(e.top, -1)
    share = torch.zeros_like(z).scatter_(1, chosen, top.softmax(-1))

    def glu(x, gate, up, down):
        return (torch.nn.functional.silu(x @ gate.T) * (x @ up.T)) @ down.T

    gate, up, down = (w["moe." + t].view(e.experts, -1, c) for t, c in (("gate", h.shape[1]), ("up", h.shape[1]), ("down", e.ff)))
    y = torch.zeros_like(h)
    for x in range(e.experts):
        at = share[:, x].nonzero().view(-1)
        y[at] += share[at, x, None] * glu(h[at], gate[x].double(), up[x].double(), down[x].double())
    return y + torch.sigmoid(h @ w["shared.sg"].T) * glu(h, w["shared.gate"], w["shared.up"], w["shared.down"])


def _layered_model(cfg, seed):
    tables = {}
    for _, name, layer, t in _layered_weights(cfg, seed):
        tables.setdefault(layer, {})[name] = t

    class Wide(dict):
        """A layer's tensors in 64 bits, each widened when it is used (the experts one by one)."""
        def __getitem__(self, k):
            t = super().__getitem__(k)
            return t if k in ("moe.gate", "moe.up", "moe.down") else t.double()

    eps, W = cfg.norm_eps, cfg.width
    top = Wide(tables[-1])

    def last_norm(x, w):
        if cfg.norm == NORM_LAYER:
            d = x - x.mean(-1, keepdim=True)
            return _rms(d, eps) * w
        return _rms(x, eps) * (1.0 + w)

    def hidden(tokens, last=None):
        x = dict.__getitem__(top, "embed")[tokens.long()].double()
        n = x.shape[0]
        if isinstance(cfg.layers[0], ParallelLayer):
            c = torch.arange(W, device="cuda")
            a = torch.arange(n, device="cuda", dtype=F64)[:, None] * 10000.0 ** (-(c - c % 2).double() / W)
            x = x + torch.where(c % 2 == 1, a.cos(), a.sin())
        x0, seen = x, set()
        for i in cfg.runs():
            l, w = cfg.layers[i], Wide(tables[i])
            if isinstance(l, ParallelLayer):
                y = 0.5 * (_rms(_gate_attention(l.attn, w, x, eps), eps) * w["at.out"] + _rms(_matrix_memory(l.mem, w, x, eps), eps) * w["mem.out"])
                x = x + last_norm(y, w["norm1"])
                x = x + last_norm(torch.nn.functional.gelu(x @ w["up"].T, approximate="tanh") @ w["down"].T, w["norm2"])
                continue
            if cfg.loop and i == cfg.loop.start:
                x = torch.cat((x, x0), -1) @ top["loop_in"].T
            mixer = _latent_attention if isinstance(l.mixer, LatentAttention) else _recurrence
            x = x + cfg.residual_mult * w["ls1"] * mixer(l.mixer, w, last_norm(x, w["norm1"]), eps)
            x = x + cfg.residual_mult * w["ls2"] * _experts(l.moe, w, last_norm(x, w["norm2"]))
        return last_norm(x, top["final_norm"])

    return hidden, top["head"]


def exact(case, seed):
    if case["do"] == "matvec":
        _, values, x = _matvec_inputs(case, seed)
        return values() @ x.double()
    cfg = _config(case)
    hidden, head = (_layered_model if "math" in case else _dense_model)(cfg, seed)
    if case["do"] == "step":
        last = _randn(seed, 1 << 29, cfg.dim)
        return head @ hidden(_ids(seed, case["context"], cfg.vocab), last)[-1]
    if case["do"] == "replay":
        x = hidden(_ids(seed, case["prompt"] + case["steps"], cfg.vocab))
        out, at = [], 0
        for end in _portions(case):
            n = end - at
            out.append(x[[at + i for i in sorted({n // 2, n - 1})]] @ head.T)
            at = end
        return out + [x[at + i:at + i + 1] @ head.T for i in range(case["steps"])]
    n, new = case["prompt"], case["new"]
    tokens = _ids(seed, n, cfg.vocab).long()
    follow = _next_tokens(seed, cfg.vocab) if "math" in case else None
    for _ in range(new):                    # the answer that the weights are made to give, then as the logits say
        tokens = torch.cat((tokens, follow[tokens[-1:]] if follow is not None else tokens[-1:]))
    for _ in range(4):
        logits = hidden(tokens)[n - 1:] @ head.T
        said = logits.argmax(-1)
        if torch.equal(said[:-1], tokens[n:]):
            return {"tokens": None, "logits": logits[-1]}
        tokens[n:] = said[:-1]
    return None

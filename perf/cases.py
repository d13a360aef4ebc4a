"""The calls a program makes on this framework, as measurable cases: single ternary products, layer forwards of a host loop, and
decoders (ternary blocks, Zitupel and Donodra stacks) that read prompts and generate.

Every case is a dict with a "kind":

  linear  quantize a few float32 rows and multiply them with a packed ternary matrix (device buffers)
  gemm    a token block through an up- and a down-projection (device buffers)
  layer   one transformer block's attention and feed-forward layers called one by one from host code (host buffers)
  decode  one sequence of a ternary decoder: a token from the host, then greedy tokens on the device
  prompt  a prompt through a ternary decoder
  batch   several independent sequences of a ternary decoder, one token each per step
  stack   a request on a layer stack: prompts, then single tokens of every sequence

All weights are seeded random numbers of the shapes and spreads that trained models have; a ternary matrix is made from
N(0, 0.02) float32 masters by the library's own packer.  `exact` recomputes what `run` returns in 64 bits with torch, rounding
to float32 only where the arithmetic of the ternary path is defined that way.
"""
import math
import zlib

import numpy as np
import torch

from loom_b200 import cabi, models

EPS = 1e-5
THETA = 500000.0
ACTS = {"linear": cabi.ACT_LINEAR, "relu2": cabi.ACT_RELU2}

DECODER_2B = dict(layers=30, heads=20, kv_heads=5, head_dim=128, inter=6912, vocab=128256)
STACK_2B = dict(layers=8, width=2560, vocab=128256, rec_heads=10, rec_dim=128, rec_vdim=256, heads=20, kv_heads=5, dim=128, ff=6912, experts=0, top=0)


def listed():
    return [
        # one row through a gate projection of the 2B shape: the smallest call, all latency
        dict(name="linear 1x2560x6912", kind="linear", tokens=1, rows=6912, cols=2560, act="linear", bias=False, residual=False),
        # the 2B feed-forward's projections in an ordinary prompt
        dict(name="gemm 512 2b", kind="gemm", tokens=512, hidden=2560, inter=6912),
        # and the 8B ones in a long, ragged one
        dict(name="gemm 2999 8b", kind="gemm", tokens=2999, hidden=4096, inter=14336),
        # a host program that walks the layers itself: 23 tokens and one more, 2B shape
        dict(name="layer 23 2b", kind="layer", seq=23, heads=20, kv_heads=5, head_dim=128, inter=6912),
        # batch-1 generation at context 1024, the headline workload
        dict(name="decode 2b", kind="decode", prompt=1024, steps=32, **DECODER_2B),
        # time to first token of the same decoder
        dict(name="prompt 1024 2b", kind="prompt", prompt=1024, **DECODER_2B),
        # serving: 16 sequences at context 2048, 8B-shaped blocks
        dict(name="batch 16 8b", kind="batch", batch=16, prompt=2048, steps=8, layers=8, heads=32, kv_heads=8, head_dim=128, inter=14336, vocab=128256),
        # a long prompt on a Zitupel stack
        dict(STACK_2B, name="zitupel prompt 2048", kind="stack", design="zitupel", dtype="bfloat16", batch=1, prompt=2048, steps=0),
        # a chat turn on it: a short prompt, then an answer
        dict(STACK_2B, name="zitupel turn 100+48", kind="stack", design="zitupel", dtype="bfloat16", batch=1, prompt=100, steps=48),
        # eight short requests served together on routed experts
        dict(name="zitupel experts 8x61+24", kind="stack", design="zitupel", dtype="bfloat16", batch=8, prompt=61, steps=24, layers=4, width=4096, vocab=128256,
             rec_heads=16, rec_dim=128, rec_vdim=256, heads=32, kv_heads=8, dim=128, ff=1792, experts=32, top=4),
        # a request with a long document on a Donodra stack
        dict(STACK_2B, name="donodra 3000+24", kind="stack", design="donodra", dtype="bfloat16", batch=1, prompt=3000, steps=24),
        # float32 stacks, as when a checkpoint is checked against its training code
        dict(name="donodra float32 333+8", kind="stack", design="donodra", dtype="float32", batch=2, prompt=333, steps=8, layers=4, width=1024, vocab=32000,
             rec_heads=4, rec_dim=128, rec_vdim=256, heads=8, kv_heads=2, dim=128, ff=2816, experts=0, top=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _decoder(rng, most_layers):
    kv = rng.choice([1, 2, 4, 5, 8])
    heads = kv * rng.choice([1, 2, 4] if kv < 5 else [2, 4])
    hidden = heads * 128
    return dict(layers=rng.randint(2, most_layers), heads=heads, kv_heads=kv, head_dim=128, inter=16 * int(hidden * rng.uniform(2.4, 3.6) / 16), vocab=_log(rng, 4000, 128256))


def draw(rng):
    kind = rng.choice(["linear", "gemm", "layer", "decode", "prompt", "batch", "stack", "stack", "stack"])
    if kind == "linear":
        return dict(kind=kind, tokens=_log(rng, 1, 24), rows=_log(rng, 200, 16000), cols=_log(rng, 200, 16000), act=rng.choice(sorted(ACTS)),
                    bias=rng.random() < 0.5, residual=rng.random() < 0.5)
    if kind == "gemm":
        hidden = 128 * rng.randint(4, 32)
        return dict(kind=kind, tokens=_log(rng, 32, 3000), hidden=hidden, inter=int(hidden * rng.uniform(2.4, 3.5)))
    if kind == "layer":
        d = _decoder(rng, 2)
        return dict(kind=kind, seq=_log(rng, 1, 60), heads=d["heads"], kv_heads=d["kv_heads"], head_dim=128, inter=d["inter"])
    if kind == "decode":
        return dict(kind=kind, prompt=_log(rng, 40, 1800), steps=rng.randint(4, 32), **_decoder(rng, 24))
    if kind == "prompt":
        return dict(kind=kind, prompt=_log(rng, 33, 2000), **_decoder(rng, 20))
    if kind == "batch":
        return dict(kind=kind, batch=rng.randint(2, 20), prompt=_log(rng, 40, 2000), steps=rng.randint(2, 8), **_decoder(rng, 8))
    design = rng.choice(["zitupel", "donodra"])
    kv = rng.choice([1, 2, 4])
    rec_heads = rng.randint(2, 10)
    dtype = "bfloat16" if rng.random() < 0.8 else "float32"
    batch = 1 if dtype == "float32" else rng.choice([1, 1, 2, 5, 8])
    return dict(kind=kind, design=design, dtype=dtype, batch=batch,
                prompt=_log(rng, 30, 2400 if batch == 1 else 200), steps=rng.randint(0, 24), layers=rng.randint(4, 8), width=256 * rng.randint(2, 10),
                vocab=_log(rng, 4000, 64000), rec_heads=rec_heads, rec_dim=rng.choice([64, 128]), rec_vdim=rng.choice([64, 128, 256]), heads=kv * rng.choice([1, 2, 4]),
                kv_heads=kv, dim=rng.choice([64, 128]), ff=16 * rng.randint(200, 430), experts=0, top=0)


# ---- inputs ---------------------------------------------------------------------------------------------------------


def _generator(seed, what):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1000003 + zlib.crc32(what.encode())) & 0x7FFFFFFFFFFF)
    return g


def _randn(seed, what, *shape):
    return torch.randn(*shape, device="cuda", generator=_generator(seed, what), dtype=torch.float32)


def _tokens(seed, what, n, vocab):
    return torch.randint(0, vocab, (n,), device="cuda", generator=_generator(seed, what)).cpu().numpy().astype(np.int32)


def _master(seed, what, rows, cols):
    return _randn(seed, what, rows * cols) * 0.02


def _pack(ctx, seed, what, rows, cols):
    m = _master(seed, what, rows, cols)
    torch.cuda.synchronize()  # the library works on a stream of its own
    return ctx.pack_ternary_f32(m, rows, cols)


def _block_shapes(c):
    hidden, kvd = c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"]
    return ((hidden, hidden), (kvd, hidden), (kvd, hidden), (hidden, hidden), (c["inter"], hidden), (c["inter"], hidden), (hidden, c["inter"]))


def _gains(seed, what, n):
    return 1.0 + 0.1 * _randn(seed, what, n)


class _StackWeights:
    """Seeded tensors under a checkpoint's interface, made on the device as they are asked for."""

    def __init__(self, c, seed):
        self.c, self.seed = c, seed
        self.dtype = cabi.DTYPES[c["dtype"]]

    def shape(self, name):
        return {"a1": (16, self.c["width"]), "rel": (32, self.c["heads"])}[name.rsplit(".", 1)[-1]]

    def tensor(self, name, shape):
        """float32 values; matrices of a bf16 stack hold bf16 numbers."""
        last, t = name.rsplit(".", 1)[-1], _randn(self.seed, name, *shape)
        if last.startswith("norm"):
            return 1.0 + 0.1 * t
        if last in ("conv", "canon1"):
            return 0.5 * t
        if last in ("A_log", "b", "dt_bias", "rel"):
            middle = {"A_log": -2.0, "b": 0.0 if name.endswith("i.b") else 3.0}
            return middle.get(last, 0.0) + 0.5 * t
        t = self.routed(last, t) * shape[-1] ** -0.5
        return t if self.dtype == cabi.DTYPE_F32 or last == "a2" else t.to(torch.bfloat16).float()

    def routed(self, last, t):
        """Routers are sure of their choice, as trained ones mostly are: embeddings lie around one of `experts` directions, each with
        `top` experts of its own, and a router's rows point along the directions that their expert serves."""
        E, W = self.c["experts"], self.c["width"]
        if not E or last not in ("embed", "router"):
            return t
        directions = _randn(self.seed, "directions", E, W).sign()
        if last == "embed":
            return 0.5 * t + directions.repeat(len(t) // E + 1, 1)[:len(t)]
        serves = torch.zeros(E, E, device="cuda")
        for k in range(self.c["top"]):
            at = torch.arange(E, device="cuda")
            serves[(5 * at + 7 * k) % E, at] = 0.15
        return serves @ directions

    def raw(self, name, shape):
        t = self.tensor(name, shape)
        t = t if self.dtype == cabi.DTYPE_F32 else t.to(torch.bfloat16)
        torch.cuda.synchronize()  # the library copies on a stream of its own
        return t, self.dtype

    def f32(self, name, shape):
        return self.tensor(name, shape).cpu().numpy()

    def scalar(self, name):
        return 1.0


def _stack_config(c):
    """Every fourth Zitupel layer is latent attention, every second of those reading the latents of the one before; Donodra
    alternates attention with its two recurrent mixers."""
    layers, last, W = [], None, c["width"]
    rec = dict(heads=c["rec_heads"], dim=c["rec_dim"], vdim=c["rec_vdim"])
    mlp = {"kind": "dense", "ff": c["ff"]}
    if c["experts"]:
        mlp = {"kind": "moe", "expert": {"ff": c["ff"], "limit": 7.0}, "router": {"experts": c["experts"], "top": c["top"]}}
    for i in range(c["layers"]):
        if c["design"] == "zitupel":
            if i % 4 == 3:
                m = dict(heads=c["heads"], dim=c["dim"], vdim=c["dim"], kv_rank=4 * c["dim"], scale=c["dim"] ** -0.5)
                if last is not None:
                    m["kv_from"], last = last, None
                else:
                    last = i
                layers.append({"type": "latent_attention", "mixer": m, "mlp": mlp})
            else:
                layers.append({"type": "gla", "mixer": dict(rec, tau=16.0), "mlp": mlp})
        elif i % 2 == 0:
            m = dict(heads=c["heads"], kv_heads=c["kv_heads"], dim=c["dim"], vdim=c["dim"], scale=c["dim"] ** -0.5, bias_max=128, mask={"size": 8192})
            layers.append({"type": "attention", "mixer": m, "mlp": mlp})
        elif i % 4 == 1:
            layers.append({"type": "delta", "mixer": dict(rec, kv_heads=c["rec_heads"], conv=4), "mlp": mlp})
        else:
            layers.append({"type": "mlstm", "mixer": dict(rec, gate_cap=15.0), "mlp": mlp})
    common = {"layers": layers, "norm": {"eps": EPS}, "vocab": c["vocab"], "width": W}
    if c["design"] == "zitupel":
        return dict(common, architecture="Zitupel", canon={"taps": 4}, residual_mult=0.7)
    return dict(common, architecture="Donodra", postln_alpha=2.0)


def prepare(case, seed):
    c, kind = case, case["kind"]
    ctx = cabi.Context(0)
    s = dict(case=c, ctx=ctx)
    if kind == "linear":
        M, R, K = c["tokens"], c["rows"], c["cols"]
        s.update(w=_pack(ctx, seed, "w", R, K), x=_randn(seed, "x", M, K), q=torch.empty(M, K, dtype=torch.int8, device="cuda"),
                 amax=torch.empty(M, device="cuda"), out=torch.empty(M, R, device="cuda"), bias=_randn(seed, "bias", R) if c["bias"] else None,
                 residual=_randn(seed, "residual", M, R) if c["residual"] else None)
    elif kind == "gemm":
        M, H, I = c["tokens"], c["hidden"], c["inter"]
        s.update(up=_pack(ctx, seed, "up", I, H), down=_pack(ctx, seed, "down", H, I), x=_randn(seed, "x", M, H), y=_randn(seed, "y", M, I),
                 out_up=torch.empty(M, I, device="cuda"), out_down=torch.empty(M, H, device="cuda"), residual=_randn(seed, "residual", M, H))
    elif kind == "layer":
        H = c["heads"] * c["head_dim"]
        w = [_pack(ctx, seed, "w%d" % i, r, k) for i, (r, k) in enumerate(_block_shapes(c))]
        inner = _gains(seed, "inner", c["inter"]).cpu().numpy()
        s.update(w=w, inner=inner, x=_randn(seed, "x", c["seq"] + 1, H).cpu().numpy(),
                 mha=cabi.MHA(ctx, H, c["heads"], c["kv_heads"], c["head_dim"], 256, THETA, EPS, *w[:4]))
    elif kind in ("decode", "prompt", "batch"):
        B, L, H, V = c.get("batch", 1), c["layers"], c["heads"] * c["head_dim"], c["vocab"]
        dec = cabi.Decoder(ctx, L, H, c["heads"], c["kv_heads"], c["head_dim"], c["inter"], V, EPS, THETA, cabi.ACT_SILU, 4096)
        if B > 1:
            dec.set_batch(B)
        for b in range(L):
            dec.set_block(b, [_pack(ctx, seed, "b%d.w%d" % (b, i), r, k) for i, (r, k) in enumerate(_block_shapes(c))],
                          _gains(seed, "b%d.g1" % b, H).cpu().numpy(), _gains(seed, "b%d.g2" % b, H).cpu().numpy())
        emb = _randn(seed, "emb", V, H) * 0.02
        dec.set_embeddings(emb, _gains(seed, "final", H).cpu().numpy())
        torch.cuda.synchronize()
        prompts = [_tokens(seed, "prompt%d" % i, c["prompt"], V) for i in range(B)]
        s.update(dec=dec, emb=emb, prompts=prompts, next=_tokens(seed, "next", B * c.get("steps", 1), V).reshape(-1, B))
        for i in range(B if kind != "prompt" else 0):
            if B > 1:
                dec.select(i)
            dec.forward(prompts[i], want_logits=False)
    else:
        dec = models.build(ctx, _stack_config(c), _StackWeights(c, seed), models.LoadOptions(cabi.DTYPES[c["dtype"]], c["prompt"] + c["steps"], c["batch"]))
        s.update(dec=dec, prompts=[_tokens(seed, "prompt%d" % i, c["prompt"], c["vocab"]) for i in range(c["batch"])],
                 next=_tokens(seed, "next", c["batch"] * c["steps"], c["vocab"]).reshape(c["steps"], c["batch"]))
    ctx.sync()
    torch.cuda.synchronize()
    return s


# ---- one pass -------------------------------------------------------------------------------------------------------


def run(s):
    c, kind, ctx = s["case"], s["case"]["kind"], s["ctx"]
    if kind == "linear":
        ctx.quantize_activation(c["tokens"], c["cols"], s["x"], s["q"], s["amax"])
        ctx.ternary_linear(s["w"], c["tokens"], s["q"], s["amax"], s["out"], bias=s["bias"], residual=s["residual"], act=ACTS[c["act"]])
        return {"q": s["q"], "amax": s["amax"], "out": s["out"]}
    if kind == "gemm":
        ctx.ternary_gemm(s["up"], c["tokens"], s["x"], out=s["out_up"])
        ctx.ternary_gemm(s["down"], c["tokens"], s["y"], out=s["out_down"], residual=s["residual"])
        return {"up": s["out_up"], "down": s["out_down"]}
    if kind == "layer":
        mha, w, x = s["mha"], s["w"], s["x"]
        mha.reset()
        a_pre, a = mha.forward(x[:-1])
        b_pre, b = mha.forward(x[-1:])
        f_pre, f = cabi.swiglu_forward(ctx, w[4], w[5], w[6], a, inner_w=s["inner"])
        g_pre, g = cabi.swiglu_forward(ctx, w[4], w[5], w[6], b, inner_w=s["inner"])
        return {"attention": [a_pre, a, b_pre, b], "feed_forward": [f_pre, f, g_pre, g]}
    dec = s["dec"]
    if kind == "prompt":
        return {"logits": dec.forward(s["prompts"][0])}
    if kind == "decode":
        dec.set_kv_offset(c["prompt"])
        logits = dec.forward(s["next"][0])
        dec.continue_greedy(c["steps"] - 1)
        return {"logits": logits, "tokens": dec.generated_tokens(c["steps"] - 1), "hidden": dec.last_hidden()}
    if kind == "batch":
        for i in range(c["batch"]):
            dec.select(i)
            dec.set_kv_offset(c["prompt"])
        return {"logits": [dec.step_batch(t) for t in s["next"]]}
    first = []
    for i, p in enumerate(s["prompts"]):
        dec.select(i)
        dec.reset()
        first.append(dec.extend(p, [len(p) - 1])[0])
    if c["batch"] == 1:
        return {"first": first, "logits": [dec.extend(t, [0]) for t in s["next"]]}
    return {"first": first, "logits": [dec.step_batch(t) for t in s["next"]]}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------


def _ternary(rows, cols):
    return rows * (-(-cols // 16)) * 4


def _stack_work(c):
    """(parameters every token goes through, parameters of one expert's three matrices, floats of recurrent state, bytes of cache per
    position, flops of a token's recurrences, flops of a token per position of context), summed over the layers."""
    W, params, expert, state, cache, rec, ctx = c["width"], 0, 0, 0, 0, 0, 0
    size = 4 if c["dtype"] == "float32" else 2
    latents = 0
    for layer in _stack_config(c)["layers"]:
        m = layer["mixer"]
        h, d, v = m["heads"], m["dim"], m["vdim"]
        if layer["type"] == "latent_attention":
            params += W * h * d + (W * m["kv_rank"] if "kv_from" not in m else 0) + (h * d + h * v) * m["kv_rank"] + W * h * v
            latents += "kv_from" not in m
            cache += m["kv_rank"] * size
            ctx += 2 * h * (d + v)
        elif layer["type"] == "attention":
            params += W * (h * d + m["kv_heads"] * (d + v) + h) + W * h * v
            cache += m["kv_heads"] * (d + v) * size
            ctx += 2 * h * (d + v)
        else:
            params += W * (2 * h * d + 2 * h * v + 16) + W * h * v
            state += h * d * v
            rec += 6 * h * d * v
        if c["experts"]:
            params += W * c["experts"]
            expert += 3 * W * c["ff"]
        else:
            params += (2 if c["design"] == "zitupel" else 3) * W * c["ff"]
    return params, expert, state, cache, rec, ctx


def work(case):
    c, kind = case, case["kind"]
    if kind == "linear":
        M, R, K = c["tokens"], c["rows"], c["cols"]
        return {"bytes": _ternary(R, K) + M * K * 5 + M * R * 4 * (1 + c["residual"]) + 4 * R * c["bias"], "flops": 2 * M * R * K}
    if kind == "gemm":
        M, H, I = c["tokens"], c["hidden"], c["inter"]
        return {"bytes": _ternary(I, H) + _ternary(H, I) + 4 * M * (2 * I + 3 * H), "flops": 4 * M * H * I}
    if kind == "stack":
        size, B, P, S, V, W = 4 if c["dtype"] == "float32" else 2, c["batch"], c["prompt"], c["steps"], c["vocab"], c["width"]
        params, expert, state, cache, rec, ctx = _stack_work(c)
        head = V * W
        met = min(c["experts"], P * c["top"]), min(c["experts"], B * c["top"])  # experts that some token goes through
        prompt = size * (params + expert * met[0] + head) + P * cache + 4 * state + 4 * V
        step = size * (params + expert * met[1] + head) + B * ((P + S // 2) * cache + 8 * state + 4 * V)
        token = 2 * (params + expert * c["top"]) + rec
        return {"bytes": B * prompt + S * step, "flops": B * (P * token + ctx * P * P // 2 + 2 * head) + S * B * (token + 2 * head + ctx * P)}
    shapes = _block_shapes(c)
    H, kvd = c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"]
    params, packed = sum(r * k for r, k in shapes), sum(_ternary(r, k) for r, k in shapes)
    if kind == "layer":
        n = c["seq"] + 1
        return {"bytes": 2 * packed + 4 * n * (4 * H + c["inter"]), "flops": 2 * n * params + 2 * H * n * n}
    L, V, P = c["layers"], c["vocab"], c["prompt"]
    if kind == "prompt":
        return {"bytes": L * (packed + 8 * P * kvd) + 4 * V * (H + 1), "flops": L * P * (2 * params + 2 * P * H) + 2 * V * H}
    B, S = c.get("batch", 1), c["steps"]
    return {"bytes": S * (L * (packed + B * 8 * P * kvd) + 4 * V * (H + B)), "flops": S * B * (L * (2 * params + 4 * P * H) + 2 * V * H)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("linear", "gemm"):
        return "exact"  # integers, and float64 arithmetic with a fixed order
    if kind in ("layer", "decode", "prompt", "batch"):
        return {"rel": 1e-5, "max": 1e-4}  # the order of float64 sums
    # measured against `exact`: 1.6e-6 in float32 and up to 1.5e-2 in bf16, through eight layers of rounded activations
    return {"rel": 1e-5, "max": 4e-4} if case["dtype"] == "float32" else {"rel": 0.03, "max": 0.9}


# ---- 64-bit recomputation ---------------------------------------------------------------------------------------------


def _codes(seed, what, rows, cols):
    """(weights -1, 0, 1 as float32 so that products of integers stay exact, scale) of a matrix that _pack makes."""
    m = _master(seed, what, rows, cols).view(rows, cols)
    scale = m.double().abs().sum().div(m.numel()).float()
    r = m / scale
    return torch.where(r.abs() >= 0.5, r.sign(), torch.zeros_like(r)), scale.double()


def _quantize(x):
    """Rows of float64 -> codes (float32 integers), absmax (float64 of a float32)."""
    amax = x.abs().amax(1).float().clamp_min(1e-5).double()
    r = x * (torch.full_like(amax, 127.0) / amax)[:, None]  # (torch divides by or into a plain number with its reciprocal)
    return (r.sign() * (r.abs() + 0.5).floor()).clamp(-128, 127).float(), amax


def _product(w, q, amax):
    codes, scale = w
    return (q @ codes.T).double() * (scale * amax / torch.full_like(amax, 127.0))[:, None]


def _block_norm(x, gain):
    rms = (x.double().square().mean(1, keepdim=True) + EPS).sqrt()
    return (x.double() / rms * gain.double()).float()


def _rope(x, pos, heads, hd):
    """float64 rows [n, heads * hd], halves rotated against each other."""
    div = torch.tensor([math.pow(THETA, 2 * d / hd) for d in range(hd // 2)], dtype=torch.float64, device=x.device)
    a = pos.double()[:, None, None] / div
    v = x.view(len(pos), heads, hd)
    v0, v1 = v[..., :hd // 2], v[..., hd // 2:]
    return torch.cat([v0 * a.cos() - v1 * a.sin(), v0 * a.sin() + v1 * a.cos()], -1)


def _attention(c, w, x, cache):
    """float32 rows through the attention layer, appended to `cache` (a dict); (normalised attention rows, output) as float64."""
    q, amax = _quantize(x.double())
    n, hd, heads, kvh = len(x), c["head_dim"], c["heads"], c["kv_heads"]
    pos = torch.arange(n, device=x.device) + cache.get("n", 0)
    Q = _rope(_product(w[0], q, amax), pos, heads, hd)
    K = _rope(_product(w[1], q, amax).float().double(), pos, kvh, hd).float()
    V = _product(w[2], q, amax).float().view(n, kvh, hd)
    if "k" in cache:
        K, V = torch.cat([cache["k"], K]), torch.cat([cache["v"], V])
    cache.update(k=K, v=V, n=len(K))
    per = heads // kvh
    out = torch.empty(n, heads, hd, dtype=torch.float64, device=x.device)
    mask = torch.arange(len(K), device=x.device)[None] > pos[:, None]
    for g in range(kvh):
        sc = torch.einsum("nhd,kd->hnk", Q[:, g * per:(g + 1) * per], K[:, g].double()) / math.sqrt(hd)
        out[:, g * per:(g + 1) * per] = (sc.masked_fill_(mask, -math.inf).softmax(-1) @ V[:, g].double()).transpose(0, 1)
    a = out.view(n, heads * hd)
    a = a / (a.square().mean(1, keepdim=True) + EPS).sqrt()
    return a, _product(w[3], *_quantize(a))


def _feed_forward(w, x, inner=None):
    q, amax = _quantize(x.double())
    g, u = _product(w[4], q, amax), _product(w[5], q, amax)
    p = (g * torch.sigmoid(g) * u).float().double()
    p = p / (p.square().mean(1, keepdim=True) + EPS).sqrt()
    p = (p if inner is None else p * inner.double()).float()
    return p, _product(w[6], *_quantize(p.double()))


class _ExactDecoder:
    def __init__(self, c, seed):
        self.c, H = c, c["heads"] * c["head_dim"]
        self.w = [[_codes(seed, "b%d.w%d" % (b, i), r, k) for i, (r, k) in enumerate(_block_shapes(c))] for b in range(c["layers"])]
        self.g = [(_gains(seed, "b%d.g1" % b, H), _gains(seed, "b%d.g2" % b, H)) for b in range(c["layers"])]
        self.emb, self.final = _randn(seed, "emb", c["vocab"], H) * 0.02, _gains(seed, "final", H)

    def forward(self, tokens, caches):
        """Appends tokens; the final-normalised rows (float32)."""
        x = self.emb[torch.as_tensor(tokens, dtype=torch.long, device="cuda")]
        for w, (g1, g2), cache in zip(self.w, self.g, caches):
            x = _attention(self.c, w, _block_norm(x, g1), cache)[1].float() + x
            x = _feed_forward(w, _block_norm(x, g2))[1].float() + x
        return _block_norm(x, self.final)

    def logits(self, rows):
        return torch.cat([rows.double() @ e.double().T for e in self.emb.split(16384)], 1)


def _conv(x, w):
    """Depthwise over time; the last column of w belongs to the current row."""
    taps = w.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(padded[j:j + len(x)] * w[:, j] for j in range(taps))


def _rms(x, gain):
    return x / (x.square().mean(-1, keepdim=True) + EPS).sqrt() * gain


def _unit(x):
    return x / (x.square().sum(-1, keepdim=True) + 1e-6).sqrt()


def _causal(q, k, v, scale, rel=None, far=0, chunk=1 << 30, sink=False):
    """q [n, heads, d], k and v [n, kv_heads, d]."""
    n, heads = q.shape[:2]
    per, at = heads // k.shape[1], torch.arange(n, device=q.device)
    hidden = (at[None] > at[:, None]) | (at[None] // chunk != at[:, None] // chunk)
    if rel is not None:
        near, buckets = rel.shape[0] // 2, rel.shape[0]
        row = [i if i < near else min(buckets - 1, near + math.floor(math.log(i / near) / math.log(far / near) * (buckets - near))) for i in range(n)]
        bias = rel[torch.tensor(row, device=q.device)]  # [distance, heads]
    out = torch.empty(n, heads, v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(heads):
        s = q[:, h] @ k[:, h // per].T * scale
        if rel is not None:
            s = s + bias[:, h][(at[:, None] - at[None]).clamp_min(0)]
        s = s.masked_fill(hidden, -math.inf)
        if sink:
            s = torch.cat([s, s.new_zeros(n, 1)], 1)
        out[:, h] = s.softmax(1)[:, :n] @ v[:, h // per]
    return out


def _exact_mixer(layer, h, t, p, latents, i):
    """The mixer of layer i (in front of its output projection) on rows h [n, width]; t(name, shape) gives a tensor."""
    m, n, W = layer["mixer"], h.shape[0], h.shape[1]
    H, d, v = m["heads"], m["dim"], m["vdim"]

    def project(name, heads, size):
        return (h @ t(p + name, (heads * size, W)).T).view(n, heads, size)

    if layer["type"] == "latent_attention":
        r, src = m["kv_rank"], m.get("kv_from", i)
        if src == i:
            latents[i] = _rms(h @ t(p + "dkv", (r, W)).T, t(p + "dkv.norm", (r,)))
        k = (latents[src] @ t(p + "uk", (H * d, r)).T).view(n, H, d)
        u = (latents[src] @ t(p + "uv", (H * v, r)).T).view(n, H, v)
        return _causal(project("q", H, d), k, u, m["scale"]).reshape(n, H * v)
    if layer["type"] == "attention":
        g = m["kv_heads"]
        o = _causal(_rms(project("q", H, d), 1.0), _rms(project("k", g, d), 1.0), project("v", g, v), m["scale"], t(p + "rel", (32, H)), m["bias_max"],
                    m["mask"]["size"], True)
        return (o * torch.sigmoid(h @ t(p + "g", (H, W)).T)[:, :, None]).reshape(n, H * v)
    q, k, u, gate = project("q", H, d), project("k", H, d), project("v", H, v), h @ t(p + "g", (H * v, W)).T
    S, out = h.new_zeros(H, d, v), h.new_empty(n, H, v)
    if layer["type"] == "gla":
        z = (h @ t(p + "a1", (16, W)).T) @ t(p + "a2", (H * d, 16)).T + t(p + "a2.b", (H * d,))
        alpha = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).view(n, H, d, 1)
        for j in range(n):
            S = torch.baddbmm(alpha[j] * S, k[j, :, :, None], u[j, :, None])
            out[j] = torch.bmm(q[j, :, None], S)[:, 0] / math.sqrt(d)
        return (_rms(out, t(p + "norm", (v,))).reshape(n, H * v)) * torch.nn.functional.silu(gate)
    if layer["type"] == "delta":
        q, k, u = (torch.nn.functional.silu(_conv(a.reshape(n, -1), t(p + x + ".conv", (a.shape[1] * a.shape[2], m["conv"])))).view(a.shape)
                   for a, x in ((q, "q"), (k, "k"), (u, "v")))
        q, k = _unit(q) / math.sqrt(d), _unit(k)
        beta = torch.sigmoid(h @ t(p + "b", (H, W)).T)
        decay = torch.exp(-torch.exp(t(p + "A_log", (H,))) * torch.nn.functional.softplus(h @ t(p + "a", (H, W)).T + t(p + "dt_bias", (H,))))
        for j in range(n):
            S = S * decay[j, :, None, None]
            e = beta[j, :, None, None] * (u[j, :, None] - torch.bmm(k[j, :, None], S))
            S = torch.baddbmm(S, k[j, :, :, None], e)
            out[j] = torch.bmm(q[j, :, None], S)[:, 0]
        return _rms(out, t(p + "norm", (v,))).reshape(n, H * v) * torch.nn.functional.silu(gate)
    cap = m["gate_cap"]
    put = cap * torch.tanh((h @ t(p + "i", (H, W)).T + t(p + "i.b", (H,))) / cap)
    keep = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ t(p + "f", (H, W)).T + t(p + "f.b", (H,))) / cap))
    q = q / math.sqrt(d)
    z, top = h.new_zeros(H, d), h.new_zeros(H)
    for j in range(n):
        new = torch.maximum(keep[j] + top, put[j])
        a, b = torch.exp(keep[j] + top - new), torch.exp(put[j] - new)
        S = torch.baddbmm(S * a[:, None, None], (b[:, None] * k[j])[:, :, None], u[j, :, None])
        z, top = a[:, None] * z + b[:, None] * k[j], new
        out[j] = torch.bmm(q[j, :, None], S)[:, 0] / (torch.maximum((z * q[j]).sum(1).abs(), torch.exp(-new)) + 1e-6)[:, None]
    return _rms(out, 1.0).reshape(n, H * v) * t(p + "norm", (H * v,)) * torch.sigmoid(gate)


def _exact_ffn(c, h, t, p):
    W, ff = c["width"], c["ff"]
    if not c["experts"]:
        up = h @ t(p + "up", (ff, W)).T
        a = torch.nn.functional.gelu(up) if c["design"] == "zitupel" else torch.nn.functional.silu(h @ t(p + "gate", (ff, W)).T) * up
        return a @ t(p + "down", (W, ff)).T
    score, index = torch.sort(torch.sigmoid(h @ t(p + "router", (c["experts"], W)).T), dim=1, descending=True, stable=True)
    out = torch.zeros_like(h)
    for e in range(c["experts"]):
        rows, place = torch.where(index[:, :c["top"]] == e)
        if len(rows):
            x, q = h[rows] * score[rows, place][:, None], "%se%d." % (p, e)
            g, u = (x @ t(q + "gate", (ff, W)).T).clamp_max(7.0), (x @ t(q + "up", (ff, W)).T).clamp(-7.0, 7.0)
            out[rows] += (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ t(q + "down", (W, ff)).T
    return out


def _exact_stack(c, seed):
    weights, W, V, P, S, B = _StackWeights(c, seed), c["width"], c["vocab"], c["prompt"], c["steps"], c["batch"]
    cfg = _stack_config(c)
    prompts = [_tokens(seed, "prompt%d" % i, P, V) for i in range(B)]
    after = _tokens(seed, "next", B * S, V).reshape(S, B)
    rows = [torch.as_tensor(np.concatenate([prompts[i], after[:, i]]), dtype=torch.long, device="cuda") for i in range(B)]

    def t(name, shape):
        return weights.tensor(name, shape).double()

    table = weights.tensor("embed", (V, W))
    first, zit = cfg["layers"], c["design"] == "zitupel"
    xs = [table[r].double() for r in rows]
    if zit:
        xs = [_rms(x, 1.0) for x in xs]
    latents = [{} for _ in range(B)]
    for i, layer in enumerate(first):
        p = "l%d." % i
        o = t(p + "mix.o", (W, layer["mixer"]["heads"] * layer["mixer"]["vdim"]))
        for b in range(B):
            x = xs[b]
            if zit:
                h = _rms(x, 1.0)
                h = h + _conv(h, t(p + "canon1", (W, 4)))
                x = x + 0.7 * (_exact_mixer(layer, h, t, p + "mix.", latents[b], i) @ o.T)
                x = x + 0.7 * _exact_ffn(c, _rms(x, 1.0), t, p + "mlp.")
            else:
                x = _rms(2.0 * x + _exact_mixer(layer, x, t, p + "mix.", latents[b], i) @ o.T, t(p + "norm1", (W,)))
                x = _rms(2.0 * x + _exact_ffn(c, x, t, p + "mlp."), t(p + "norm2", (W,)))
            xs[b] = x
    head = weights.tensor("head", (V, W)) if zit else table
    gain = 1.0 if zit else t("final.norm", (W,))
    logits = [torch.cat([_rms(x[P - 1:], gain) @ part.double().T for part in head.split(16384)], 1) for x in xs]
    every = [torch.stack([logits[b][1 + j] for b in range(B)]) for j in range(S)]
    return {"first": [a[0] for a in logits], "logits": every}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "linear":
        M, R, K = c["tokens"], c["rows"], c["cols"]
        q, amax = _quantize(_randn(seed, "x", M, K).double())
        y = _product(_codes(seed, "w", R, K), q, amax)
        y = (y + _randn(seed, "bias", R).double() if c["bias"] else y).float()
        y = y.clamp_min(0).square() if c["act"] == "relu2" else y
        y = (y.double() + _randn(seed, "residual", M, R).double()) if c["residual"] else y.double()
        return {"q": q.to(torch.int8), "amax": amax, "out": y}
    if kind == "gemm":
        M, H, I = c["tokens"], c["hidden"], c["inter"]
        up = _product(_codes(seed, "up", I, H), *_quantize(_randn(seed, "x", M, H).double()))
        down = _product(_codes(seed, "down", H, I), *_quantize(_randn(seed, "y", M, I).double()))
        return {"up": up, "down": down.float().double() + _randn(seed, "residual", M, H).double()}
    if kind == "layer":
        H = c["heads"] * c["head_dim"]
        w = [_codes(seed, "w%d" % i, r, k) for i, (r, k) in enumerate(_block_shapes(c))]
        x, inner, cache = _randn(seed, "x", c["seq"] + 1, H), _gains(seed, "inner", c["inter"]), {}
        rows = [_attention(c, w, x[:-1], cache), _attention(c, w, x[-1:], cache)]
        ffn = [_feed_forward(w, a[1].float(), inner) for a in rows]
        return {"attention": [y for pair in rows for y in pair], "feed_forward": [y for pair in ffn for y in pair]}
    if kind == "stack":
        return _exact_stack(c, seed)
    dec, B, V = _ExactDecoder(c, seed), c.get("batch", 1), c["vocab"]
    prompts = [_tokens(seed, "prompt%d" % i, c["prompt"], V) for i in range(B)]
    if kind == "prompt":
        return {"logits": dec.logits(dec.forward(prompts[0], [{} for _ in dec.w])[-1:])[0]}
    after = _tokens(seed, "next", B * c["steps"], V).reshape(-1, B)
    if kind == "batch":
        rows = [dec.forward(np.concatenate([prompts[i], after[:, i]]), [{} for _ in dec.w])[c["prompt"]:] for i in range(B)]
        return {"logits": [dec.logits(torch.stack([r[j] for r in rows])) for j in range(c["steps"])]}
    caches = [{} for _ in dec.w]
    dec.forward(prompts[0], caches)
    hidden = dec.forward(after[0], caches)
    first = logits = dec.logits(hidden)[0]
    tokens = []
    for _ in range(c["steps"] - 1):
        tokens.append(int(logits.float().argmax()))
        hidden = dec.forward(tokens[-1:], caches)
        logits = dec.logits(hidden)[0]
    return {"logits": first, "tokens": np.array(tokens, np.int32), "hidden": hidden[0].double()}

"""What this library is used for, as cases that can be timed: single projections, a decode layer, expert banks and
batched products, each through recipe_dev_b200.Context as a host program calls it.

Weights are GGUF blocks of N(0, 0.02) values, activations N(0, 1) times a spread of channel magnitudes (what a
normalised hidden state looks like). Everything is made on the GPU from the seed alone. `exact` computes the same
results in 64 bits from the blocks' own definition, without the library; int8 activations are part of that definition
(codes and steps are fixed by fp32 arithmetic), so it rounds them the same way and sums in 64 bits.
"""
import math

import torch

import recipe_dev_b200 as rq

TYPES = {"Q4_K": rq.Q4_K, "Q6_K": rq.Q6_K, "Q8_0": rq.Q8_0, "Q4_0": rq.Q4_0, "Q4_1": rq.Q4_1, "Q5_0": rq.Q5_0, "Q5_K": rq.Q5_K}
BLOCK = {"Q4_K": (256, 144), "Q6_K": (256, 210), "Q8_0": (32, 34), "Q4_0": (32, 18), "Q4_1": (32, 20), "Q5_0": (32, 22), "Q5_K": (256, 176)}
ACT = {"float": rq.ACT_FLOAT, "int8": rq.ACT_INT8}
DEV = "cuda:0"


def listed():
    return [
        # One projection of a decode step, called by itself: the smallest call a program makes.
        dict(name="projection_q8_0", kind="matvec", type="Q8_0", rows=4096, cols=4096, tokens=1, act="int8", step=32),
        # A decode step's layer (8B-shaped: hidden 4096, 1024 key/value rows, ffn 14336), recorded once and replayed, under
        # int8 activations (the default profile of the stored K-quants) and under fp32 activations (`.fp(32)`).
        dict(name="layer_int8", kind="layer", type="Q4_K", down="Q6_K", hidden=4096, kv=1024, ffn=14336, act="int8", step=32),
        dict(name="layer_float", kind="layer", type="Q4_K", down="Q6_K", hidden=4096, kv=1024, ffn=14336, act="float", step=32),
        # The vocabulary projection, for one sequence and for four decoded together.
        dict(name="head_one", kind="matvec", type="Q6_K", rows=262144, cols=2560, tokens=1, act="int8", step=32),
        dict(name="head_four", kind="matvec", type="Q6_K", rows=262144, cols=2560, tokens=4, act="int8", step=32),
        # A mixture-of-experts block (256 experts, eight a token) for one sequence and for sixteen.
        dict(name="experts_one", kind="experts", type="Q4_K", experts=256, top=8, hidden=2048, ffn=512, tokens=1, scoring=0),
        dict(name="experts_sixteen", kind="experts", type="Q4_K", experts=256, top=8, hidden=2048, ffn=512, tokens=16, scoring=0),
        # Batched products: a small batch of sequences, a short prompt, long prompts (one of a ragged length, over the Q8_0
        # re-encode that `.int(8)` makes of a lone Q6_K tensor).
        dict(name="batch_16", kind="matmul", type="Q4_K", rows=14336, cols=4096, tokens=16, act="float", step=32),
        dict(name="prompt_64_int8", kind="matmul", type="Q6_K", rows=4096, cols=14336, tokens=64, act="int8", step=32),
        dict(name="prompt_512", kind="matmul", type="Q4_K", rows=14336, cols=4096, tokens=512, act="float", step=32),
        dict(name="prompt_509_int8", kind="matmul", type="Q8_0", rows=4096, cols=14336, tokens=509, act="int8", step=32),
        # A projection of a file stored in one of the other formats, fp32 activations.
        dict(name="projection_q5_k", kind="matvec", type="Q5_K", rows=14336, cols=4096, tokens=1, act="float", step=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, kind, lo, hi):
    """Inputs per row: whole 256-value units, for the 32-value formats sometimes any whole number of blocks."""
    unit = 32 if BLOCK[kind][0] == 32 and rng.random() < 0.25 else 256
    return max(1, _log(rng, lo, hi) // unit) * unit


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "matvec", "matmul", "matmul", "matmul", "experts", "experts", "layer"])
    step = rng.choice([32, 32, 32, 256])
    if kind == "matvec":
        t = rng.choice(["Q4_K", "Q6_K", "Q8_0", "Q4_0", "Q4_K", "Q6_K", "Q8_0", "Q4_0", "Q4_1", "Q5_0", "Q5_K"])
        act = "float" if t in ("Q4_1", "Q5_0", "Q5_K") else rng.choice(["float", "int8", "int8"])
        cols = _width(rng, t, 512, 14336)
        tokens = rng.choice([1, 1, 1, 2, 3, 4, 8])
        rows = _log(rng, 512, min(262144, 240_000_000 // (cols * tokens)))
        return dict(kind=kind, type=t, rows=rows, cols=cols, tokens=tokens, act=act, step=step)
    if kind == "matmul":
        t = rng.choice(["Q4_K", "Q4_K", "Q6_K", "Q6_K", "Q8_0", "Q4_0"])
        cols = _width(rng, t, 1024, 14336)
        return dict(kind=kind, type=t, rows=_log(rng, 512, 58_720_256 // cols), cols=cols, tokens=_log(rng, 8, 509), act=rng.choice(["float", "int8"]), step=step)
    if kind == "experts":
        hidden, ffn = 256 * rng.randint(4, 10), 256 * rng.randint(1, 4)
        experts = min(_log(rng, 16, 256), 280_000_000 // (hidden * ffn))
        return dict(kind=kind, type=rng.choice(["Q4_K", "Q4_K", "Q6_K", "Q8_0"]), experts=experts, top=rng.choice([2, 4, 6, 8]), hidden=hidden, ffn=ffn,
                    tokens=_log(rng, 1, 32), scoring=rng.choice([0, 1]))
    t, down = rng.choice([("Q4_K", "Q6_K"), ("Q4_K", "Q4_K"), ("Q8_0", "Q8_0"), ("Q4_0", "Q4_0")])
    hidden = 256 * rng.randint(8, 16)
    return dict(kind=kind, type=t, down=down, hidden=hidden, kv=256 * rng.randint(1, 4), ffn=256 * rng.randint(12, 56 if t == "Q4_K" else 28), act=rng.choice(["int8", "int8", "float"]),
                step=step)


# ---- inputs --------------------------------------------------------------------------------------------


def _gen(seed, stream):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 64 + stream)


def _activations(gen, tokens, cols):
    x = torch.randn((tokens, cols), generator=gen, device=DEV)
    return x * torch.exp(0.5 * torch.randn((1, cols), generator=gen, device=DEV))


def _half(v):
    """fp16 values as their two bytes, and as 64-bit numbers."""
    h = v.to(torch.float16)
    return h.unsqueeze(-1).view(torch.uint8), h.double()


def _six_bit(sc, mn):
    """The twelve bytes that hold eight six-bit scales and minimums ([n, 8] each, int32)."""
    lo_s, hi_s, lo_m, hi_m = sc[:, :4], sc[:, 4:], mn[:, :4], mn[:, 4:]
    return torch.cat([lo_s | ((hi_s >> 4) << 6), lo_m | ((hi_m >> 4) << 6), (hi_s & 15) | ((hi_m & 15) << 4)], dim=1).to(torch.uint8)


def _encode(kind, w, values):
    """GGUF blocks of fp32 values w [n]: uint8 [blocks, bytes], and (values) what they stand for, in 64 bits."""
    per, _ = BLOCK[kind]
    b = w.reshape(-1, per)
    n = b.shape[0]
    u8 = torch.uint8
    if kind in ("Q8_0", "Q4_0", "Q5_0"):
        bits = {"Q8_0": 8, "Q4_0": 4, "Q5_0": 5}[kind]
        half = 1 << (bits - 1)
        big = b.gather(1, b.abs().argmax(1, keepdim=True))
        raw, d = _half(big[:, 0] / (127.0 if bits == 8 else -float(half)))
        q = torch.round(b / torch.where(d == 0, 1.0, d).float()[:, None]).clamp(-half + (bits == 8), half - 1).to(torch.int32)
        v = (q.double() * d[:, None]) if values else None
        if kind == "Q8_0":
            return torch.cat([raw, q.to(torch.int8).view(u8)], 1), v
        q = q + half
        nib = ((q[:, :16] & 15) | ((q[:, 16:] & 15) << 4)).to(u8)
        if kind == "Q4_0":
            return torch.cat([raw, nib], 1), v
        fifth = ((q >> 4).reshape(n, 4, 8) << torch.arange(8, device=DEV)).sum(2).to(u8)
        return torch.cat([raw, fifth, nib], 1), v
    if kind == "Q4_1":
        lo, hi = b.amin(1), b.amax(1)
        rd, d = _half((hi - lo) / 15.0)
        rm, m = _half(lo)
        q = torch.round((b - m.float()[:, None]) / d.float().clamp_min(1e-7)[:, None]).clamp(0, 15).to(torch.int32)
        return torch.cat([rd, rm, (q[:, :16] | (q[:, 16:] << 4)).to(u8)], 1), (q.double() * d[:, None] + m[:, None]) if values else None
    if kind in ("Q4_K", "Q5_K"):
        top = 15 if kind == "Q4_K" else 31
        s = b.reshape(n, 8, 32)
        mn = (-s.amin(2)).clamp_min(0)
        step = (s.amax(2) + mn) / top
        rd, d = _half(step.amax(1) / 63.0)
        rm, dm = _half(mn.amax(1) / 63.0)
        sc = torch.round(step / d.float().clamp_min(1e-7)[:, None]).clamp(0, 63).to(torch.int32)
        mi = torch.round(mn / dm.float().clamp_min(1e-7)[:, None]).clamp(0, 63).to(torch.int32)
        a, off = d[:, None] * sc, dm[:, None] * mi
        q = torch.round((s + off.float()[..., None]) / a.float().clamp_min(1e-9)[..., None]).clamp(0, top).to(torch.int32)
        v = (a[..., None] * q - off[..., None]) if values else None
        p = q.reshape(n, 4, 2, 32)
        nib = ((p[:, :, 0] & 15) | ((p[:, :, 1] & 15) << 4)).reshape(n, 128).to(u8)
        parts = [rd, rm, _six_bit(sc, mi)]
        if kind == "Q5_K":
            parts.append(((q >> 4) << torch.arange(8, device=DEV)[None, :, None]).sum(1).to(u8))
        return torch.cat(parts + [nib], 1), v
    # Q6_K
    s = b.reshape(n, 16, 16)
    big = s.gather(2, s.abs().argmax(2, keepdim=True))[..., 0] / -32.0
    rd, d = _half(big.abs().amax(1) / 127.0)
    sc = torch.round(big / d.float().clamp_min(1e-7)[:, None]).clamp(-127, 127).to(torch.int32)
    a = d[:, None] * sc
    q = torch.round(s / torch.where(a == 0, 1.0, a).float()[..., None]).clamp(-32, 31).to(torch.int32)
    v = (a[..., None] * q) if values else None
    q = (q + 32).reshape(n, 2, 4, 32)  # chunk, group of 32, value
    ql = torch.stack([(q[:, :, 0] & 15) | ((q[:, :, 2] & 15) << 4), (q[:, :, 1] & 15) | ((q[:, :, 3] & 15) << 4)], 2).reshape(n, 128).to(u8)
    qh = ((q >> 4) << torch.tensor([0, 2, 4, 6], device=DEV)[None, None, :, None]).sum(2).reshape(n, 64).to(u8)
    return torch.cat([ql, qh, sc.to(torch.int8).view(u8), rd], 1), v


def _rows(kind, gen, rows, cols, values=False):
    """The blocks of a [rows, cols] weight, some rows at a time, with their values in 64 bits on request."""
    chunk = max(1, (1 << 24) // cols)
    for at in range(0, rows, chunk):
        n = min(chunk, rows - at)
        blocks, v = _encode(kind, 0.02 * torch.randn(n * cols, generator=gen, device=DEV), values)
        yield blocks, v.reshape(n, cols) if values else None


def _blocks(kind, gen, rows, cols):
    per, size = BLOCK[kind]
    out = torch.empty((rows * (cols // per), size), dtype=torch.uint8, device=DEV)
    at = 0
    for blocks, _ in _rows(kind, gen, rows, cols):
        out[at : at + blocks.shape[0]] = blocks
        at += blocks.shape[0]
    return out


def _weight(ctx, kind, gen, rows, cols):
    w = ctx.weight_from_device(TYPES[kind], _blocks(kind, gen, rows, cols), rows, cols)
    torch.cuda.synchronize()  # the blocks are read on the stream: they may go once the planes are written
    return w


def _scores(case, seed):
    return torch.randn((case["experts"], case["tokens"]), generator=_gen(seed, 1), device=DEV) * 1.5


# ---- the cases -----------------------------------------------------------------------------------------


def prepare(case, seed):
    """Resident weights, the activations, an output buffer; for a layer, the recorded sequence."""
    kind = case["kind"]
    ctx = rq.Context(0)
    s = dict(case=case, ctx=ctx)
    if kind in ("matvec", "matmul"):
        s["w"] = _weight(ctx, case["type"], _gen(seed, 2), case["rows"], case["cols"])
        s["x"] = _activations(_gen(seed, 0), case["tokens"], case["cols"])
        s["y"] = torch.empty((case["tokens"], case["rows"]), device=DEV)
        ctx.reserve(case["rows"], case["cols"], case["tokens"])
    elif kind == "experts":
        e, h, f = case["experts"], case["hidden"], case["ffn"]
        gate, up, down = (_blocks(case["type"], _gen(seed, 2 + i), e * r, c).cpu().numpy() for i, (r, c) in enumerate(((f, h), (f, h), (h, f))))
        s["bank"] = ctx.moe_prepare(TYPES[case["type"]], gate, up, down, e, h, f)
        s["scores"] = _scores(case, seed)
        s["x"] = _activations(_gen(seed, 0), case["tokens"], h).T  # [hidden, tokens], a token's values contiguous
        s["y"] = torch.empty((case["tokens"], h), device=DEV).T
        s["weights"] = torch.empty_like(s["scores"])
    else:
        h, kv, f = case["hidden"], case["kv"], case["ffn"]
        t, act, step = case["type"], ACT[case["act"]], case["step"]
        names = (("q", t, h, h), ("k", t, kv, h), ("v", t, kv, h), ("o", t, h, h), ("gate", t, f, h), ("up", t, f, h), ("down", case["down"], h, f))
        w = s["w"] = {n: _weight(ctx, wt, _gen(seed, 2 + i), r, c) for i, (n, wt, r, c) in enumerate(names)}
        gen = _gen(seed, 0)
        s["x"] = _activations(gen, 1, h)[0]
        s["gains"] = 1.0 + 0.1 * torch.randn((2, h), generator=gen, device=DEV)
        b = s["planes"] = {n: torch.empty(r, device=DEV) for n, r in (("n1", h), ("q", h), ("k", kv), ("v", kv), ("o", h), ("h", h), ("n2", h), ("g", f), ("d", h), ("out", h))}
        ctx.reserve(f, f, 1)
        torch.cuda.synchronize()
        stream = ctx.sequence_begin()
        ctx.rmsnorm(s["x"], s["gains"][0], y=b["n1"], stream=stream)
        ctx.matvec_multi([w["q"], w["k"], w["v"]], b["n1"], [b["q"], b["k"], b["v"]], act_mode=act, step=step, stream=stream)
        ctx.matvec(w["o"], b["q"], y=b["o"], act_mode=act, step=step, stream=stream)
        ctx.add(s["x"], b["o"], y=b["h"], stream=stream)
        ctx.rmsnorm(b["h"], s["gains"][1], y=b["n2"], stream=stream)
        ctx.matvec_glu(w["gate"], w["up"], b["n2"], y=b["g"], act_mode=act, step=step, stream=stream)
        ctx.matvec(w["down"], b["g"], y=b["d"], act_mode=act, step=step, stream=stream)
        ctx.add(b["h"], b["d"], y=b["out"], stream=stream)
        s["sequence"] = ctx.sequence_end()
    torch.cuda.synchronize()
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "matvec":
        return ctx.matvec(s["w"], s["x"], y=s["y"], act_mode=ACT[case["act"]], step=case["step"])
    if kind == "matmul":
        return ctx.matmul(s["w"], s["x"], y=s["y"], act_mode=ACT[case["act"]], step=case["step"])
    if kind == "experts":
        y, weights = ctx.moe_route_forward(s["bank"], s["scores"], s["x"], case["top"], scoring=case["scoring"], weights=s["weights"], y=s["y"])
        return {"y": y, "weights": weights}
    s["sequence"].run()
    return {n: s["planes"][n] for n in ("q", "k", "v", "o", "g", "d", "out")}


def _stored(kind, rows, cols):
    per, size = BLOCK[kind]
    return rows * (cols // per) * size


def work(case):
    kind = case["kind"]
    if kind in ("matvec", "matmul"):
        r, c, t = case["rows"], case["cols"], case["tokens"]
        return dict(bytes=_stored(case["type"], r, c) + 4 * t * (r + c), flops=2 * r * c * t)
    if kind == "experts":
        e, k, h, f, t = case["experts"], case["top"], case["hidden"], case["ffn"], case["tokens"]
        touched = e * (1.0 - (1.0 - k / e) ** t)  # experts at least one token is routed to, on average
        one = 2 * _stored(case["type"], f, h) + _stored(case["type"], h, f)
        return dict(bytes=touched * one + 4 * t * (2 * h + 2 * e), flops=6 * h * f * k * t)
    h, kv, f = case["hidden"], case["kv"], case["ffn"]
    t = case["type"]
    stored = _stored(t, 2 * h + 2 * kv + 2 * f, h) + _stored(case["down"], h, f)
    return dict(bytes=stored + 4 * (4 * h + 2 * kv + f + 3 * h), flops=2 * (h * (2 * h + 2 * kv + 3 * f)))


def tolerance(case):
    """fp32 sums over one product; behind a layer's later products an int8 code may round the other way."""
    if case["kind"] == "layer":
        return {"rel": 2e-3, "max": 2e-2} if case["act"] == "int8" else {"rel": 2.5e-6, "max": 2.5e-5}
    return {"rel": 2e-6, "max": 2e-5}


# ---- the same in 64 bits -------------------------------------------------------------------------------


def _rounded(x, act, step):
    """What the dot multiplies: x itself, or its int8 codes times their steps (fp32 arithmetic, groups of `step` inputs)."""
    if act == "float":
        return x.double()
    t, cols = x.shape
    parts = [_rounded_groups(x[:, : cols // step * step], step)]
    if cols % step:
        parts.append(_rounded_groups(x[:, cols // step * step :], cols % step))
    return torch.cat(parts, 1)


def _rounded_groups(x, step):
    if x.shape[1] == 0:
        return x.double()
    g = x.float().reshape(x.shape[0], -1, step)
    best = g.gather(2, g.abs().argmax(2, keepdim=True))
    inverse = torch.where(best == 0, 0.0, torch.full_like(best, -127.0) / best)  # a number over a tensor would be a reciprocal and a product
    d = torch.where(best == 0, 0.0, 1.0 / inverse)
    return (torch.round(g * inverse).clamp(-128, 127).double() * d.double()).reshape(x.shape)


def _product(kind, gen, rows, cols, x):
    return torch.cat([x @ v.T for _, v in _rows(kind, gen, rows, cols, True)], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("matvec", "matmul"):
        x = _rounded(_activations(_gen(seed, 0), case["tokens"], case["cols"]), case["act"], case["step"])
        return _product(case["type"], _gen(seed, 2), case["rows"], case["cols"], x)
    silu = torch.nn.functional.silu
    if kind == "experts":
        e, k, h, f, t = case["experts"], case["top"], case["hidden"], case["ffn"], case["tokens"]
        scores = _scores(case, seed).double()
        p = torch.softmax(scores, 0) if case["scoring"] == 0 else torch.sigmoid(scores)
        kept, at = p.topk(k, 0)
        weights = torch.zeros_like(p).scatter(0, at, kept / kept.sum(0, keepdim=True))
        x = _activations(_gen(seed, 0), t, h).double()
        chosen = sorted(set(at.flatten().tolist()))
        bank = []
        for i, (r, c) in enumerate(((f, h), (f, h), (h, f))):  # each table is drawn as one weight: keep the chosen experts' rows
            per, first, got = r, 0, {}
            for _, v in _rows(case["type"], _gen(seed, 2 + i), e * r, c, True):
                n = v.shape[0]
                for ex in chosen:
                    lo, hi = max(first, ex * per), min(first + n, (ex + 1) * per)
                    if lo < hi:
                        got.setdefault(ex, []).append(v[lo - first : hi - first].clone())
                first += n
            bank.append({ex: torch.cat(got[ex], 0) for ex in chosen})
        y = torch.zeros((t, h), dtype=torch.float64, device=DEV)
        for ex in chosen:
            hid = silu(x @ bank[0][ex].T) * (x @ bank[1][ex].T)
            y += weights[ex][:, None] * (hid @ bank[2][ex].T)
        return {"y": y.T, "weights": weights}
    h, kv, f, t, act, step = case["hidden"], case["kv"], case["ffn"], case["type"], case["act"], case["step"]
    gen = _gen(seed, 0)
    x = _activations(gen, 1, h).double()
    gains = (1.0 + 0.1 * torch.randn((2, h), generator=gen, device=DEV)).double()

    def norm(v, g):
        return v / torch.sqrt((v * v).mean(1, keepdim=True) + 1e-6) * g

    def dot(i, wt, r, c, v):
        return _product(wt, _gen(seed, 2 + i), r, c, _rounded(v, act, step))

    n1 = norm(x, gains[0])
    q, k, v = dot(0, t, h, h, n1), dot(1, t, kv, h, n1), dot(2, t, kv, h, n1)
    o = dot(3, t, h, h, q)
    hidden = x + o
    n2 = norm(hidden, gains[1])
    g = silu(dot(4, t, f, h, n2)) * dot(5, t, f, h, n2)
    d = dot(6, case["down"], h, f, g)
    return {"q": q[0], "k": k[0], "v": v[0], "o": o[0], "g": g[0], "d": d[0], "out": (hidden + d)[0]}

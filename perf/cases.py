"""The framework's work, as timed cases: single factorized linears, a stack of them, both attention
faces, decode steps and prompts of the factorized decoder, decode steps and prompts of the two layered
designs.  ``prepare`` makes what a program holds before the call, ``run`` is one pass through the public
entry points, ``exact`` is the same pass in plain 64-bit torch.
"""

from __future__ import annotations

import functools
import math

import torch

from quantibbler_b200 import virudra, vogizen
from quantibbler_b200.decoder import Decoder, DecoderConfig
from quantibbler_b200.gpu import AttentionShape, GpuContext, LayerGroup, PackedLayer
from quantibbler_b200.layered import LayeredDecoder

VOCAB = 32768
F64 = torch.float64


def listed():
    return [
        # one token through one linear: a host that drives the layers of a model itself
        dict(name="linear_1_token", kind="linear", dout=4096, din=4096, r=1024, tokens=1, serving="float32"),
        # many independent layer applies ready at once (all layers of a step, many requests)
        dict(name="linear_stack", kind="stack", layers=592, dout=4096, din=4096, r=1024),
        # the up projection of a 4096-wide block over a long prompt
        dict(name="linear_prompt", kind="linear", dout=14336, din=4096, r=2560, tokens=2048, serving="bfloat16"),
        # the exact face over a prompt, grouped heads
        dict(name="attention_exact", kind="exact", batch=1, heads=32, kv_heads=8, seq_q=2048, seq_kv=2048, dim=128,
             causal=True),
        # the INT8 face over a long prompt
        dict(name="attention_sage", kind="sage", batch=1, heads=32, kv_heads=8, seq=8192, dim=128, block=64, causal=True),
        # chat, one user: a token at a time; a served batch; and the prompt before both
        dict(name="decode_1", kind="decode", width=4096, layers=8, batch=1, context=2048, serving="bfloat16"),
        dict(name="decode_64", kind="decode", width=4096, layers=8, batch=64, context=2048, serving="bfloat16"),
        dict(name="prompt", kind="prompt", width=4096, layers=8, tokens=2048, serving="bfloat16"),
        # the layered designs, a prompt and a step each; the second prompt is of no round length
        dict(name="vogizen_prompt", kind="vogizen_prompt", width=4096, tokens=2048),
        dict(name="vogizen_decode", kind="vogizen_decode", width=2048, batch=1, context=2048),
        dict(name="virudra_prompt", kind="virudra_prompt", width=2048, tokens=1531),
        dict(name="virudra_decode", kind="virudra_decode", width=4096, batch=64, context=2048),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    """A case of the same kinds: sizes over the ranges that the entry points serve, odd ones among them."""
    kind = rng.choice(["linear", "linear", "stack", "exact", "sage", "decode", "prompt", "vogizen_prompt",
                       "vogizen_decode", "virudra_prompt", "virudra_decode"])
    if kind == "linear":
        serving = rng.choice(["float32", "bfloat16", "bfloat16"])
        return dict(kind=kind, dout=_log(rng, 256, 14336), din=_log(rng, 256, 14336), r=_log(rng, 64, 2560),
                    tokens=_log(rng, 1, 32 if serving == "float32" else 2048), serving=serving)
    if kind == "stack":
        return dict(kind=kind, layers=rng.randint(148, 592), dout=rng.choice([1024, 2048, 4096]),
                    din=rng.choice([1024, 2048, 4096]), r=_log(rng, 200, 1024))
    if kind == "exact":
        heads, group = rng.choice([8, 16, 32]), rng.choice([1, 2, 4, 8])
        seq_kv = _log(rng, 16, 2048)
        causal = rng.random() < 0.7
        seq_q = seq_kv if rng.random() < 0.7 else rng.randint(1, seq_kv)
        return dict(kind=kind, batch=rng.choice([1, 1, 2]), heads=heads, kv_heads=heads // group, seq_q=seq_q,
                    seq_kv=seq_kv, dim=rng.choice([64, 80, 128, 128]), causal=causal)
    if kind == "sage":
        heads, group = rng.choice([8, 16, 32]), rng.choice([1, 2, 4, 8])
        return dict(kind=kind, batch=1, heads=heads, kv_heads=heads // group, seq=_log(rng, 128, 8192),
                    dim=rng.choice([64, 128, 128]), block=rng.choice([32, 64, 64, 64, 128]), causal=rng.random() < 0.7)
    if kind == "decode":
        serving = rng.choice(["float32", "bfloat16", "bfloat16", "bfloat16"])
        return dict(kind=kind, width=rng.choice([2048, 4096]), layers=rng.randint(2, 6),
                    batch=_log(rng, 1, 4 if serving == "float32" else 64), context=_log(rng, 16, 2048), serving=serving)
    if kind == "prompt":
        return dict(kind=kind, width=rng.choice([2048, 4096]), layers=rng.randint(2, 6), tokens=_log(rng, 16, 2048),
                    serving="bfloat16")
    width = rng.choice([1024, 2048, 4096])
    if kind.endswith("prompt"):
        return dict(kind=kind, width=width, tokens=_log(rng, 5, 2048))
    most = 4 if kind == "vogizen_decode" else 64
    return dict(kind=kind, width=width, batch=_log(rng, 1, most), context=_log(rng, 16, 2048))


# ---------------------------------------------------------------------- inputs and weights
@functools.cache
def _context() -> GpuContext:
    return GpuContext.init()


def _stream_context() -> GpuContext:
    """The process's context, launching on torch's current stream."""
    ctx = _context()
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return ctx


def _generator(seed: int):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(gen, *shape):
    return torch.randn(shape, device="cuda", generator=gen)


def _bits(gen, rows: int, n: int):
    """``rows`` random bitplanes of ``n`` signs, pad bits clear."""
    b = torch.randint(0, 256, (rows, (n + 7) // 8), device="cuda", generator=gen, dtype=torch.uint8)
    if n % 8:
        b[:, -1] &= (1 << (n % 8)) - 1
    return b


def _factors(gen, dout: int, din: int, r: int) -> dict:
    """A factorized linear: Bernoulli(0.5) factors, small positive scales."""
    return dict(dout=dout, din=din, r=r, ub=_bits(gen, dout, r), vbt=_bits(gen, r, din),
                s1=_randn(gen, dout).abs() * 0.02 + 1e-3, s2=_randn(gen, din).abs() * 0.02 + 1e-3)


def _host_factors(f: dict) -> dict:
    return dict(dout=f["dout"], din=f["din"], r=f["r"], ub_rows=f["ub"].cpu().numpy(), vb_t_rows=f["vbt"].cpu().numpy(),
                s1=f["s1"].cpu().numpy(), s2=f["s2"].cpu().numpy(), bias=None)


def _packed(ctx, f: dict, serving: str) -> PackedLayer:
    h = _host_factors(f)
    return PackedLayer(ctx, h["ub_rows"], h["vb_t_rows"], f["dout"], f["din"], f["r"], h["s1"], h["s2"], None, serving=serving)


def _signs(bits, n: int):
    at = torch.arange(8, device=bits.device, dtype=torch.uint8)
    return (((bits[:, :, None] >> at) & 1).reshape(bits.shape[0], -1)[:, :n].to(F64) * 2.0) - 1.0


def _linear64(f: dict, x):
    t = (x * f["s2"].to(F64)) @ _signs(f["vbt"], f["din"]).T
    return (t @ _signs(f["ub"], f["r"]).T) * f["s1"].to(F64)


def _ids(gen, n: int) -> list:
    return torch.randint(0, VOCAB, (n,), device="cuda", generator=gen).tolist()


# ---------------------------------------------------------------------- the factorized decoder
RANKS = {"q": 1102, "k": 431, "v": 431, "o": 1102, "gate": 1724, "up": 1724, "down": 1733}


def _llama(case) -> tuple:
    """Config, {linear: (dout, din, rank)}: heads of 128, four query heads per key/value head, ranks of 0.55
    bits per weight."""
    d = case["width"]
    ff, heads = (14336 if d == 4096 else 4 * d), d // 128
    kv = heads // 4 * 128
    prompt = case["kind"] == "prompt"
    cfg = DecoderConfig(n_layers=case["layers"], d_model=d, n_heads=heads, n_kv_heads=heads // 4, head_dim=128, d_ff=ff,
                        vocab=VOCAB, rope_theta=500000.0, serving=case["serving"],
                        max_seq=(case["tokens"] if prompt else case["context"]) + 16,
                        max_batch=1 if prompt else case["batch"])
    shapes = dict(q=(d, d), k=(kv, d), v=(kv, d), o=(d, d), gate=(ff, d), up=(ff, d), down=(d, ff))
    rank = RANKS if d == 4096 else {n: int(0.55 * a * b / (a + b)) - 24 for n, (a, b) in shapes.items()}
    return cfg, {n: (a, b, rank[n]) for n, (a, b) in shapes.items()}


def _llama_weights(case, gen) -> dict:
    cfg, shapes = _llama(case)
    layers = []
    for _ in range(cfg.n_layers):
        layer = {n: _factors(gen, *s) for n, s in shapes.items()}
        layer["input_norm"] = 1.0 + 0.1 * _randn(gen, cfg.d_model)
        layer["post_norm"] = 1.0 + 0.1 * _randn(gen, cfg.d_model)
        layers.append(layer)
    table = lambda: (_randn(gen, VOCAB, cfg.d_model) * 0.02).to(torch.bfloat16)  # noqa: E731
    return dict(layers=layers, final_norm=1.0 + 0.1 * _randn(gen, cfg.d_model), embedding=table(), lm_head=table(),
                vocab_offset=0)


def _llama_cache(case, gen, layer: int):
    """A layer's keys and values of the positions before the step (both are N(0, 1))."""
    cfg, _ = _llama(case)
    shape = (case["batch"], cfg.n_kv_heads, case["context"], 128)
    return [_randn(gen, *shape).to(torch.bfloat16) for _ in range(2)]


def _llama_decoder(ctx, cfg, w: dict) -> Decoder:
    host = dict(w, layers=[{n: (_host_factors(v) if isinstance(v, dict) else v) for n, v in layer.items()}
                           for layer in w["layers"]])
    return Decoder(ctx, cfg, host)


def _rms64(x, w, eps):
    return x / torch.sqrt((x ** 2).mean(-1, keepdim=True) + eps) * w.to(F64)


def _rope64(x, pos, theta):
    """x [tokens, heads, dim], pos [tokens]."""
    half = x.shape[-1] // 2
    inv = theta ** (-2.0 * torch.arange(half, device=x.device, dtype=F64) / x.shape[-1])
    ang = pos.to(F64)[:, None, None] * inv
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1)


def _softmax_attention64(q, k, v, scale, bias=None, mask=None):
    """q [heads, tq, d], k and v [kv heads, tk, d]; head by head, to stay small.  ``bias(head)``; ``mask`` of
    what is seen."""
    group, out = q.shape[0] // k.shape[0], []
    for h in range(q.shape[0]):
        s = (q[h] @ k[h // group].T) * scale
        if bias is not None:
            s = s + bias(h)
        if mask is not None:
            s = s.masked_fill(~mask, -math.inf)
        out.append(torch.softmax(s, -1) @ v[h // group])
    return torch.stack(out)


def _llama64(case, seed):
    gen = _generator(seed)
    cfg, _ = _llama(case)
    w = _llama_weights(case, gen)
    prompt = case["kind"] == "prompt"
    ids = _ids(gen, case["tokens"] if prompt else case["batch"])
    n, kvh = len(ids), cfg.n_kv_heads
    pos = torch.arange(n, device="cuda") if prompt else torch.full((n,), case["context"], device="cuda")
    x = w["embedding"][ids].to(F64)
    keys, values = [], []
    for i, lw in enumerate(w["layers"]):
        h = _rms64(x, lw["input_norm"], cfg.rms_eps)
        q = _rope64(_linear64(lw["q"], h).reshape(n, -1, 128), pos, cfg.rope_theta)
        k = _rope64(_linear64(lw["k"], h).reshape(n, kvh, 128), pos, cfg.rope_theta)
        v = _linear64(lw["v"], h).reshape(n, kvh, 128)
        if prompt:
            seen = pos[:, None] >= pos[None, :]
            att = _softmax_attention64(q.transpose(0, 1), k.transpose(0, 1), v.transpose(0, 1), 128 ** -0.5,
                                       mask=seen).transpose(0, 1)
            keys.append(k.transpose(0, 1)), values.append(v.transpose(0, 1))
        else:
            ck, cv = _llama_cache(case, gen, i)
            att = []
            for b in range(n):
                kk = torch.cat([ck[b].to(F64), k[b][:, None]], 1)
                vv = torch.cat([cv[b].to(F64), v[b][:, None]], 1)
                s = torch.einsum("ghd,gkd->ghk", q[b].reshape(kvh, -1, 128), kk) * 128 ** -0.5
                att.append(torch.einsum("ghk,gkd->ghd", torch.softmax(s, -1), vv).reshape(-1, 128))
            att = torch.stack(att)
            keys.append(k), values.append(v)
        x = x + _linear64(lw["o"], att.reshape(n, -1))
        h = _rms64(x, lw["post_norm"], cfg.rms_eps)
        g, u = _linear64(lw["gate"], h), _linear64(lw["up"], h)
        x = x + _linear64(lw["down"], g * torch.sigmoid(g) * u)
    x = _rms64(x[-1:] if prompt else x, w["final_norm"], cfg.rms_eps)
    return {"logits": x @ w["lm_head"].to(F64).T, "keys": keys, "values": values}


# ---------------------------------------------------------------------- the layered designs
def _layered_config(case) -> tuple:
    """(design, config.json of eight layer runs): heads of 128, the first two layers run twice."""
    d = case["width"]
    heads, ff = d // 128, (14336 if d == 4096 else 4 * d)
    common = {"width": d, "vocab": VOCAB, "norm": {"eps": 1e-5}, "loop": {"start": 0, "stop": 2, "times": 2}}
    if case["kind"].startswith("vogizen"):
        att = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": ff},
               "mixer": {"heads": heads, "dim": 128, "vdim": 128, "kv_rank": 512, "q_rank": 3 * d // 8,
                         "scale": 128 ** -0.5, "mask": {"size": max(2048, d)}}}
        rec = {"type": "delta", "mlp": None,
               "mixer": {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4}}
        return vogizen, dict(common, architecture="Vogizen", embedding={"scale": d ** 0.5},
                             token_side={"dim": d // 16}, layers=[att, rec] * 3)
    mixer = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "bias_max": 1024,
             "q_temp": {"coef": 0.2, "every": 512}}
    dense = {"type": "attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": ff}}
    mixture = {"type": "attention", "mixer": mixer,
               "mlp": {"kind": "moe", "expert": {"ff": ff // 2}, "router": {"experts": 16, "top": 2}}}
    return virudra, dict(common, architecture="Virudra", logit_softcap=30.0, layers=[dense, mixture] * 3)


def _layered_tensors(design, config: dict, gen) -> dict:
    out = {}
    for name, shape in design.shapes(config).items():
        if name.endswith(".table"):   # (a token's experts: neighbours of a random one)
            first = torch.randint(0, 16, (shape[0], 1), device="cuda", generator=gen)
            out[name] = ((first + torch.arange(shape[1], device="cuda")) % 16).to(torch.int32)
            continue
        t = _randn(gen, *[32 if n is None else n for n in shape])
        if name.endswith(("A_log", "dt_bias")):
            t = t * 0.1 - 1.0
        elif len(shape) == 1:
            t = (0.0 if design is virudra else 1.0) + 0.1 * t
        else:
            t = t / shape[-1] ** 0.5
        out[name] = t.to(torch.bfloat16)
    return out


def _layered_runs(config) -> list:
    order, (a, b, times) = list(range(len(config["layers"]))), config["loop"].values()
    return order[:a] + order[a:b] * times + order[b:]


def _virudra_cache(case, config, gen):
    kv = config["layers"][0]["mixer"]["kv_heads"]
    return [_randn(gen, case["batch"], kv, case["context"], 128).to(torch.bfloat16) for _ in range(2)]


def _gelu64(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _silu64(z):
    return z * torch.sigmoid(z)


def _gated64(h, w, name, act):
    return (act(h @ w[name + "gate"].to(F64).T) * (h @ w[name + "up"].to(F64).T)) @ w[name + "down"].to(F64).T


def _buckets(rows: int, bias_max: float, upto: int):
    half = rows // 2
    return torch.tensor([n if n < half else min(rows - 1, half + math.floor(
        math.log(n / half) / math.log(bias_max / half) * (rows - half))) for n in range(upto)], device="cuda")


def _virudra64(case, seed):
    gen = _generator(seed)
    design, config = _layered_config(case)
    w = _layered_tensors(design, config, gen)
    prompt = case["kind"].endswith("prompt")
    ids = _ids(gen, case["tokens"] if prompt else case["batch"])
    n, d = len(ids), case["width"]
    pos = list(range(n)) if prompt else [case["context"]] * n
    temp = torch.tensor([1.0 + 0.2 * math.log(math.floor((p + 1) / 512) + 1) for p in pos], device="cuda", dtype=F64)
    norm = lambda x, name: _rms64(x, 1.0 + w[name].to(F64), 1e-5)  # noqa: E731
    bucket = _buckets(32, 1024, max(pos) + 1)
    x = w["embed"].to(F64)[ids]
    keys, values = [], []
    for i in _layered_runs(config):
        p, m = f"l{i}.", config["layers"][i]["mixer"]
        kvh, heads = m["kv_heads"], m["heads"]
        h = norm(x, p + "norm1")
        q = (h @ w[p + "mix.q"].to(F64).T).reshape(n, heads, 128) * temp[:, None, None]
        k = (h @ w[p + "mix.k"].to(F64).T).reshape(n, kvh, 128)
        v = (h @ w[p + "mix.v"].to(F64).T).reshape(n, kvh, 128)
        rel = w[p + "mix.rel"].to(F64)[bucket]          # [distance, head]
        if prompt:
            at = torch.arange(n, device="cuda")
            back = at[:, None] - at[None, :]
            att = _softmax_attention64(q.transpose(0, 1), k.transpose(0, 1), v.transpose(0, 1), m["scale"],
                                       bias=lambda a: rel[back.clamp(min=0), a], mask=back >= 0).transpose(0, 1)
            keys.append(k.transpose(0, 1)), values.append(v.transpose(0, 1))
        else:
            ck, cv = _virudra_cache(case, config, gen)
            back = rel.flip(0).T.reshape(kvh, -1, case["context"] + 1)
            att = []
            for b in range(n):
                kk, vv = (torch.cat([c[b].to(F64), t[b][:, None]], 1) for c, t in ((ck, k), (cv, v)))
                s = torch.einsum("ghd,gkd->ghk", q[b].reshape(kvh, -1, 128), kk) * m["scale"] + back
                att.append(torch.einsum("ghk,gkd->ghd", torch.softmax(s, -1), vv).reshape(heads, 128))
            att = torch.stack(att)
            keys.append(k), values.append(v)
        x = x + norm(att.reshape(n, -1) @ w[p + "mix.o"].to(F64).T, p + "norm1b")
        h = norm(x, p + "norm2")
        if config["layers"][i]["mlp"]["kind"] == "dense":
            y = _gated64(h, w, p + "mlp.", _gelu64)
        else:
            y, table = torch.zeros(n, d, device="cuda", dtype=F64), w[p + "mlp.table"][ids]
            for e in range(16):
                rows = (table == e).any(1).nonzero()[:, 0]
                if len(rows):
                    y[rows] += _gated64(h[rows], w, f"{p}mlp.e{e}.", _silu64) / 2
        x = x + norm(y, p + "norm2b")
    x = norm(x[-1:] if prompt else x, "final.norm")
    return {"logits": 30.0 * torch.tanh((x @ w["head"].to(F64).T) / 30.0), "keys": keys, "values": values}


def _layer_norm64(x, w, eps=1e-5):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], eps=eps) * w.to(F64)


def _delta64(h, w, p, m):
    n, heads, kv = len(h), m["heads"], m["kv_heads"]

    def branch(name, count):
        x, taps = h @ w[p + name].to(F64).T, w[p + name + ".conv"].to(F64)
        past = torch.cat([x.new_zeros(taps.shape[1] - 1, x.shape[1]), x])
        return _silu64(sum(past[j:j + n] * taps[:, j] for j in range(taps.shape[1]))).reshape(n, count, 128)

    unit = lambda x: x / torch.sqrt((x ** 2).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    spread = lambda x: x.repeat_interleave(heads // kv, 1)  # noqa: E731
    q, k = spread(unit(branch("q", kv)) * 128 ** -0.5), spread(unit(branch("k", kv)))
    v = branch("v", heads)
    beta = torch.sigmoid(h @ w[p + "b"].to(F64).T)
    decay = torch.exp(-torch.exp(w[p + "A_log"].to(F64)) * torch.nn.functional.softplus(
        h @ w[p + "a"].to(F64).T + w[p + "dt_bias"].to(F64), threshold=1e9))
    state = h.new_zeros(heads, 128, 128)      # [value, key]
    out = torch.empty_like(v)
    for t in range(n):
        state = state * decay[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.bmm(state, k[t][:, :, None])[..., 0])
        state = torch.baddbmm(state, u[:, :, None], k[t][:, None, :])
        out[t] = torch.bmm(state, q[t][:, :, None])[..., 0]
    y = _rms64(out, w[p + "norm"], 1e-5) * _silu64(h @ w[p + "g"].to(F64).T).reshape(n, heads, 128)
    return y.reshape(n, -1) @ w[p + "o"].to(F64).T, state


def _latent64(h, w, p, m):
    n, heads = len(h), m["heads"]
    q = (_rms64(h @ w[p + "dq"].to(F64).T, w[p + "dq.norm"], 1e-5) @ w[p + "uq"].to(F64).T).reshape(n, heads, 128)
    c = _rms64(h @ w[p + "dkv"].to(F64).T, w[p + "dkv.norm"], 1e-5)
    k = (c @ w[p + "uk"].to(F64).T).reshape(n, heads, 128)
    v = (c @ w[p + "uv"].to(F64).T).reshape(n, heads, 128)
    at = torch.arange(n, device="cuda")
    back = at[:, None] - at[None, :]
    att = _softmax_attention64(q.transpose(0, 1), k.transpose(0, 1), v.transpose(0, 1), m["scale"],
                               mask=(back >= 0) & (back < m["mask"]["size"])).transpose(0, 1)
    return att.reshape(n, -1) @ w[p + "o"].to(F64).T, c


def _vogizen64(case, seed):
    gen = _generator(seed)
    design, config = _layered_config(case)
    w = _layered_tensors(design, config, gen)
    prompt = case["kind"].endswith("prompt")
    lengths = [case["tokens"]] if prompt else [case["context"] + 1] * case["batch"]
    d, side = case["width"], config["token_side"]["dim"]
    rows = [_ids(gen, n) for n in lengths]
    logits, states, rings = [], [], []
    for ids in rows:
        n = len(ids)
        entry = torch.arange(d, device="cuda")
        angle = torch.arange(n, device="cuda", dtype=F64)[:, None] * 10000.0 ** (-(2.0 * (entry // 2)) / d)
        x = x0 = w["embed"].to(F64)[ids] * d ** 0.5 + torch.where(entry % 2 == 0, angle.sin(), angle.cos())
        mine, ring = [], []
        for at, i in enumerate(_layered_runs(config)):
            p, layer = f"l{i}.", config["layers"][i]
            if at in (0, 2):
                x = torch.cat([x, x0], 1) @ w["loop.in"].to(F64).T
            mixer = _latent64 if layer["type"] == "latent_attention" else _delta64
            y, left = mixer(_layer_norm64(x, w[p + "norm1"]), w, p + "mix.", layer["mixer"])
            (ring if mixer is _latent64 else mine).append(left)
            x = x + y * w[p + "ls1"].to(F64)
            if layer["mlp"] is not None:
                x = x + _gated64(_layer_norm64(x, w[p + "norm2"]), w, p + "mlp.", torch.relu) * w[p + "ls2"].to(F64)
            rows_ = w["side.embed"].to(F64)[ids, i * side:(i + 1) * side]
            y = (_gelu64(x @ w[p + "side.gate"].to(F64).T) * rows_) @ w[p + "side.proj"].to(F64).T
            x = x + _rms64(y, w[p + "side.norm"], 1e-5)
        logits.append(_layer_norm64(x[-1:], w["final.norm"]) @ w["embed"].to(F64).T)
        states.append(mine), rings.append(ring)
    out = {"logits": torch.cat(logits), "states": [torch.stack(s) for s in zip(*states)]}
    if prompt:
        out["latents"] = rings[0]
    return out


# ---------------------------------------------------------------------- the cases
def prepare(case, seed):
    gen, kind = _generator(seed), case["kind"]
    ctx = _stream_context()
    if kind == "linear":
        layer = _packed(ctx, _factors(gen, case["dout"], case["din"], case["r"]), case["serving"])
        # (bfloat16 batches of seven tokens and more take the tensor-core face, as the decoder does)
        call = layer.apply_prefill if case["serving"] == "bfloat16" and case["tokens"] >= 7 else layer.apply_device
        return dict(case=case, layer=layer, call=call, x=_randn(gen, case["tokens"], case["din"]),
                    y=torch.zeros(case["tokens"], case["dout"], device="cuda"))
    if kind == "stack":
        layers = [_packed(ctx, _factors(gen, case["dout"], case["din"], case["r"]), "float32")
                  for _ in range(case["layers"])]
        x = _randn(gen, case["layers"], case["din"])
        y = torch.zeros(case["layers"], case["dout"], device="cuda")
        return dict(case=case, group=LayerGroup(ctx, layers, x.data_ptr(), y.data_ptr()), x=x, y=y)
    if kind in ("exact", "sage"):
        q, k, v, shape = _attention_inputs(case, gen)
        return dict(case=case, ctx=ctx, q=q, k=k, v=v, shape=shape, y=torch.zeros_like(q))
    if kind in ("decode", "prompt"):
        cfg, _ = _llama(case)
        w = _llama_weights(case, gen)
        dec = _llama_decoder(ctx, cfg, w)
        if kind == "prompt":
            n = case["tokens"]
            return dict(case=case, dec=dec, ids=_ids(gen, n), keys=[c[0, :, :n] for c in dec.cache_k],
                        values=[c[0, :, :n] for c in dec.cache_v])
        ids, at = _ids(gen, case["batch"]), case["context"]
        dec.capture()
        for i in range(cfg.n_layers):
            dec.cache_k[i][:, :, :at], dec.cache_v[i][:, :, :at] = _llama_cache(case, gen, i)
        return dict(case=case, dec=dec, ids=ids, at=[at] * len(ids), keys=[c[:, :, at] for c in dec.cache_k],
                    values=[c[:, :, at] for c in dec.cache_v])
    design, config = _layered_config(case)
    tensors = _layered_tensors(design, config, gen)
    prompt = kind.endswith("prompt")
    design.check_tensors(config, tensors)
    dec = LayeredDecoder(ctx, design.parse(config, serving="bfloat16", max_batch=1 if prompt else case["batch"],
                                           max_seq=(case["tokens"] if prompt else case["context"]) + 16), tensors)
    del tensors
    states = [s for _, _, s in dec.runs]
    if kind == "vogizen_decode":
        rows = [_ids(gen, case["context"] + 1) for _ in range(case["batch"])]
        for slot, row in enumerate(rows):
            dec.prefill(row[:-1], seq=slot)
        dec.capture()
        return dict(case=case, dec=dec, ids=[row[-1] for row in rows], at=[case["context"]] * len(rows),
                    states=[s.matrix for s in states[1::2]])
    ids = _ids(gen, case["tokens"] if prompt else case["batch"])
    if kind == "vogizen_prompt":
        return dict(case=case, dec=dec, ids=ids, states=[s.matrix for s in states[1::2]],
                    latents=[s.data[0, :len(ids), :512] for s in states[::2]])
    if kind == "virudra_prompt":
        return dict(case=case, dec=dec, ids=ids, keys=[s.k[0, :, :len(ids), :128] for s in states],
                    values=[s.v[0, :, :len(ids), :128] for s in states])
    dec.capture()
    at = case["context"]
    for s in states:
        s.k[:, :, :at, :128], s.v[:, :, :at, :128] = _virudra_cache(case, config, gen)
    return dict(case=case, dec=dec, ids=ids, at=[at] * len(ids), keys=[s.k[:, :, at, :128] for s in states],
                values=[s.v[:, :, at, :128] for s in states])


def _attention_inputs(case, gen):
    b, h, kv, d = case["batch"], case["heads"], case["kv_heads"], case["dim"]
    sq, sk = (case["seq"],) * 2 if case["kind"] == "sage" else (case["seq_q"], case["seq_kv"])
    q, k, v = _randn(gen, b, h, sq, d), _randn(gen, b, kv, sk, d), _randn(gen, b, kv, sk, d)
    k = k + 2.0 * _randn(gen, 1, kv, 1, d)      # (keys carry an offset per channel)
    return q, k, v, AttentionShape(b, h, kv, sq, sk, d, d)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        state["call"](state["x"].data_ptr(), case["tokens"], state["y"].data_ptr())
        return state["y"]
    if kind == "stack":
        state["group"].apply()
        return state["y"]
    if kind in ("exact", "sage"):
        state["ctx"].attention_dev(state["shape"], state["q"].data_ptr(), state["k"].data_ptr(), state["v"].data_ptr(),
                                   case["causal"], state["y"].data_ptr(), case.get("block"))
        return state["y"]
    dec = state["dec"]
    if kind.endswith("prompt"):
        dec.prefill(state["ids"])
    else:
        dec.start(state["ids"], state["at"])
        dec.decode(1)
    # (the greedy token is the first maximum of these logits)
    out = {"logits": dec.logits}
    out.update({n: state[n] for n in ("keys", "values", "states", "latents") if n in state})
    return out


def exact(case, seed):
    kind, gen = case["kind"], _generator(seed)
    if kind == "linear":
        f = _factors(gen, case["dout"], case["din"], case["r"])
        return _linear64(f, _randn(gen, case["tokens"], case["din"]).to(F64))
    if kind == "stack":
        fs = [_factors(gen, case["dout"], case["din"], case["r"]) for _ in range(case["layers"])]
        x = _randn(gen, case["layers"], case["din"]).to(F64)
        return torch.stack([_linear64(f, row[None])[0] for f, row in zip(fs, x)])
    if kind in ("exact", "sage"):
        q, k, v, shape = _attention_inputs(case, gen)
        seen = None
        if case["causal"]:
            rows = torch.arange(shape.seq_q, device="cuda")[:, None] + (shape.seq_kv - shape.seq_q)
            seen = rows >= torch.arange(shape.seq_kv, device="cuda")[None, :]
        return torch.stack([_softmax_attention64(a.to(F64), b.to(F64), c.to(F64), shape.head_dim ** -0.5, mask=seen)
                            for a, b, c in zip(q, k, v)])
    if kind in ("decode", "prompt"):
        return _llama64(case, seed)
    return _virudra64(case, seed) if kind.startswith("virudra") else _vogizen64(case, seed)


def _params(case) -> tuple:
    """(weights of one token's products, bytes of all weights) of a layered model's eight runs, head included."""
    design, config = _layered_config(case)
    shapes = design.shapes(config)
    weights = bytes_ = 0.0
    n = case.get("tokens", case.get("batch"))
    for i in _layered_runs(config):
        for name, shape in shapes.items():
            if not name.startswith(f"l{i}.") or len(shape) != 2 or name.endswith((".table", ".rel", ".conv")):
                continue
            used = 1.0
            if ".mlp.e" in name:      # two of the sixteen experts per token
                used, some = 2 / 16, 1 - (14 / 16) ** n
                bytes_ += 2 * shape[0] * shape[1] * some
            else:
                bytes_ += 2 * shape[0] * shape[1]
            weights += used * shape[0] * shape[1]
    if "loop.in" in shapes:
        weights, bytes_ = weights + 2 * 2 * case["width"] ** 2, bytes_ + 2 * 2 * 2 * case["width"] ** 2
    return weights, bytes_


def work(case):
    kind = case["kind"]
    if kind in ("linear", "stack"):
        n, m = (case["tokens"], 1) if kind == "linear" else (1, case["layers"])
        a, b, r = case["dout"], case["din"], case["r"]
        return {"bytes": m * (r * (a + b) / 8 + 4 * (a + b) + 4 * n * (a + b)), "flops": 2.0 * m * n * r * (a + b)}
    if kind in ("exact", "sage"):
        b, h, kv, d = case["batch"], case["heads"], case["kv_heads"], case["dim"]
        sq, sk = (case["seq"],) * 2 if kind == "sage" else (case["seq_q"], case["seq_kv"])
        pairs = sq * sk - (sq * (sq - 1) / 2 if case["causal"] else 0)
        return {"bytes": 4.0 * b * d * (2 * h * sq + 2 * kv * sk), "flops": 4.0 * b * h * pairs * d}
    prompt = kind.endswith("prompt")
    n = case["tokens"] if prompt else case["batch"]
    heads = case["width"] // 128
    pairs = n * (n + 1) / 2 if prompt else n * (case["context"] + 1)
    head_rows = 1 if prompt else n
    if kind in ("decode", "prompt"):
        _, shapes = _llama(case)
        weights = case["layers"] * sum(r * (a + b) for a, b, r in shapes.values())
        scales = case["layers"] * sum(4 * (a + b) for a, b, _ in shapes.values())
        bytes_, runs, kv_row = weights / 8 + scales, case["layers"], 2 * 2 * 128 * heads // 4
    else:
        weights, bytes_ = _params(case)
        runs, kv_row = 8, 2 * 2 * 128 * heads // 4
        if kind.startswith("vogizen"):     # (four attention runs of one latent, four matrices of 128 x 128 per head)
            runs, kv_row = 4, 2 * 512
            bytes_ += 2 * 4 * 4 * heads * 128 * 128 * (1 if prompt else n)
    context = n if prompt else n * (case["context"] + 1)
    return {"bytes": bytes_ + 2.0 * VOCAB * case["width"] + runs * kv_row * context + 4.0 * head_rows * VOCAB,
            "flops": 2.0 * n * weights + 4.0 * runs * heads * 128 * pairs + 2.0 * head_rows * VOCAB * case["width"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "exact":
        return {"rel": 1e-5, "max": 1e-3}
    if kind == "sage":            # (the softmax weights' INT8 codes turn on the last bit of exp)
        return {"rel": 1e-3, "max": 0.1}
    if kind == "stack" or case.get("serving") == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    if kind == "linear":          # (three roundings to bfloat16)
        return {"rel": 1e-2, "max": 0.1}
    return {"rel": 0.03, "max": 0.5}     # (bfloat16 all through the layers)

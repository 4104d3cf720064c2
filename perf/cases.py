"""The measured workloads: what a program that serves a quantized transformer has this library do.

A case is a dict of plain values.  ``kind`` names the piece of such a program that one pass runs:

  linear  one ``QuantLinear.forward`` (a stand-alone projection: a classifier, a small draft model, a vocabulary head)
  layer   the four projections of one decoder layer on ``rows`` tokens: qkv, o, gate|up and the down projection on
          silu(gate) * up -- the calls a host makes around its own attention
  mlp     one ``GatedMLP.forward``
  moe     one ``MoELayer.forward`` on ``rows`` tokens
  step    one decode step of a small stack for ``rows`` sequences, from token ids to logits: norms, projections, RoPE and
          cache append, attention over ``n_ctx`` positions, vocabulary head
  host    one ``HostBatch.run``: the projections of ``layers`` decoder layers on page-locked host buffers

Weights are seeded normal draws (sigma 0.02) in the formats' own blocks; activations are unit normal with a per-channel
spread, as they leave a norm layer with trained weights.  Every state owns its weights: with the three states that a
measurement alternates between, all but the smallest case exceed the 126 MB of L2 and stream their weights from memory,
as the many layers of a model do.
"""
import math

import torch

import tattletale_b200 as ttq
from tattletale_b200 import quantize

FORMATS = {"q8_0": ttq.FMT_Q8_0, "q4_k": ttq.FMT_Q4_K, "q6_k": ttq.FMT_Q6_K, "tq3": ttq.FMT_TQ3}
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
EPS = 1e-5
HEAD_DIM = 128

_context = None


def context():
    """One library context per process, as a serving process keeps."""
    global _context
    if _context is None:
        _context = ttq.Context(0)
    return _context


def listed():
    return [
        # a stand-alone projection with a bias for one row of a small model: launches and host work are all there is
        {"name": "small-q8_0-1", "kind": "linear", "fmt": "q8_0", "k": 1024, "n": 1000, "rows": 1, "x": "f16", "y": "f16", "bias": True},
        # one user decoding: one token through the projections of an 8B-class layer
        {"name": "layer-q4_k-1", "kind": "layer", "fmt": "q4_k", "hidden": 4096, "kv": 1024, "ffn": 14336, "rows": 1},
        # a handful of users decoding, or a speculative draft being checked
        {"name": "layer-q4_k-6", "kind": "layer", "fmt": "q4_k", "hidden": 4096, "kv": 1024, "ffn": 14336, "rows": 6},
        # a server's continuous batch
        {"name": "layer-q4_k-23", "kind": "layer", "fmt": "q4_k", "hidden": 4096, "kv": 1024, "ffn": 14336, "rows": 23},
        # a decode batch with a piece of somebody's prompt in it
        {"name": "layer-q4_k-137", "kind": "layer", "fmt": "q4_k", "hidden": 4096, "kv": 1024, "ffn": 14336, "rows": 137},
        # a long prompt
        {"name": "layer-q4_k-2048", "kind": "layer", "fmt": "q4_k", "hidden": 4096, "kv": 1024, "ffn": 14336, "rows": 2048},
        # an ordinary prompt through the MLP of a model kept at higher precision
        {"name": "mlp-q6_k-777", "kind": "mlp", "fmt": "q6_k", "hidden": 4096, "ffn": 14336, "rows": 777},
        # mixture of experts: prompts, and a decode batch that touches most experts with few rows each
        {"name": "moe-q4_k-4096", "kind": "moe", "experts": 128, "top_k": 8, "hidden": 2048, "ffn": 768, "rows": 4096},
        {"name": "moe-q4_k-24", "kind": "moe", "experts": 128, "top_k": 8, "hidden": 2048, "ffn": 768, "rows": 24},
        # a 70B-class layer at three bits per weight serving a small batch
        {"name": "layer-tq3-12", "kind": "layer", "fmt": "tq3", "hidden": 8192, "kv": 1024, "ffn": 28672, "rows": 12},
        # a decode step from tokens to logits
        {"name": "step-q4_k-5", "kind": "step", "layers": 2, "hidden": 4096, "q_heads": 32, "kv_heads": 8, "ffn": 14336, "vocab": 128256,
         "rows": 5, "context": 2048, "n_ctx": 1531},
        # projections whose inputs and results live in host memory
        {"name": "host-q4_k-1", "kind": "host", "fmt": "q4_k", "hidden": 4096, "kv": 1024, "ffn": 14336, "layers": 2, "rows": 1},
    ]


# ---- drawn cases ---------------------------------------------------------------------------------------------------

def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(rng, lo, hi, unit):
    return max(1, _log(rng, lo, hi) // unit) * unit


def _unit(fmt):
    return {"q8_0": 32, "tq3": 128}.get(fmt, 256)


def draw(rng):
    """One more case: any format, from one row to a long prompt, sizes log-uniform, output sizes odd where they may be."""
    kind = rng.choice(["linear", "linear", "layer", "layer", "layer", "mlp", "moe", "step", "host"])
    if kind == "linear":
        fmt = rng.choice(["q8_0", "q4_k", "q6_k", "tq3"])
        n = _log(rng, 256, 24576)
        case = {"kind": kind, "fmt": fmt, "k": _multiple(rng, 512, 12288, _unit(fmt)), "n": max(1, n // 128) * 128 if fmt == "tq3" else n,
                "rows": _log(rng, 1, 2048), "x": rng.choice(["bf16", "f16"]), "y": rng.choice(["bf16", "f16", "f32"]), "bias": rng.random() < 0.5}
    elif kind == "layer":
        fmt = rng.choice(["q8_0", "q4_k", "q4_k", "q6_k", "tq3"])
        hidden = _multiple(rng, 1024, 8192, 256)
        case = {"kind": kind, "fmt": fmt, "hidden": hidden, "kv": max(128, hidden // rng.choice([1, 4, 8]) // 128 * 128),
                "ffn": _multiple(rng, 2 * hidden, 4 * hidden, 256), "rows": _log(rng, 1, 2048)}
    elif kind == "mlp":
        hidden = _multiple(rng, 1024, 8192, 256)
        case = {"kind": kind, "fmt": rng.choice(["q8_0", "q4_k", "q6_k"]), "hidden": hidden, "ffn": _multiple(rng, 2 * hidden, 4 * hidden, 256),
                "rows": _log(rng, 1, 2048)}
    elif kind == "moe":
        experts = rng.choice([8, 16, 60, 64, 128])
        case = {"kind": kind, "experts": experts, "top_k": rng.randint(1, 8), "hidden": _multiple(rng, 1024, 4096, 256),
                "ffn": _multiple(rng, 512, 2048, 256), "rows": _log(rng, 1, 4096)}
    elif kind == "step":
        kv = rng.choice([1, 2, 4, 8])
        q = kv * rng.choice([1, 2, 4, 8])
        while q < 8:
            q *= 2
            kv *= 2
        hidden = 128 * q
        context = _log(rng, 128, 4096)
        case = {"kind": kind, "layers": rng.randint(1, 3), "hidden": hidden, "q_heads": q, "kv_heads": kv, "ffn": _multiple(rng, 2 * hidden, 4 * hidden, 256),
                "vocab": _log(rng, 8192, 131072), "rows": _log(rng, 1, 32), "context": context, "n_ctx": rng.randint(max(1, context // 2), context)}
    else:
        hidden = _multiple(rng, 1024, 4096, 256)
        case = {"kind": kind, "fmt": rng.choice(["q8_0", "q4_k", "q6_k"]), "hidden": hidden, "kv": max(128, hidden // 4 // 128 * 128),
                "ffn": _multiple(rng, 2 * hidden, 4 * hidden, 256), "layers": rng.randint(1, 3), "rows": _log(rng, 1, 8)}
    # no dearer than the dearest listed cases: fewer rows, then fewer experts, then narrower
    while work(case)["flops"] > 8e11 and case["rows"] > 1:
        case["rows"] = case["rows"] * 2 // 3
    while kind == "moe" and case["experts"] * case["hidden"] * case["ffn"] > 128 * 2048 * 1024:
        case["experts"] //= 2
    case["top_k"] = min(case["top_k"], case["experts"]) if kind == "moe" else case.get("top_k", 0)
    if kind != "moe":
        del case["top_k"]
    return case


# ---- states --------------------------------------------------------------------------------------------------------

def _blocks(fmt, n, k, gen):
    """Packed weights of an [n][k] normal matrix, on the device."""
    if fmt == "tq3":
        # every bit string is a valid trellis stream and decodes to unit normal values; 0.02 is the row scale
        tiles = torch.randint(0, 256, (n * k * 3 // 8,), generator=gen, device="cuda", dtype=torch.uint8)
        scale = (0.02 * (1 + 0.1 * torch.randn(n, generator=gen, device="cuda"))).to(torch.float16).view(torch.uint8)
        signs = torch.randint(0, 256, (k // 8,), generator=gen, device="cuda", dtype=torch.uint8)
        return torch.cat((tiles, scale, signs))
    return quantize.quantize(FORMATS[fmt], torch.randn(n, k, generator=gen, device="cuda") * 0.02)


def _linear(fmt, n, k, gen, bias=None):
    return ttq.QuantLinear(context(), FORMATS[fmt], _blocks(fmt, n, k, gen), k, bias=bias, out_features=n)


def _rows(m, k, gen, dtype=torch.bfloat16):
    spread = torch.exp(0.3 * torch.randn(k, generator=gen, device="cuda"))
    return (torch.randn(m, k, generator=gen, device="cuda") * spread).to(dtype)


def _layer_linears(c, gen):
    h, f = c["hidden"], c["ffn"]
    return {"qkv": _linear(c["fmt"], h + 2 * c["kv"], h, gen), "o": _linear(c["fmt"], h, h, gen),
            "gate_up": _linear(c["fmt"], 2 * f, h, gen), "down": _linear(c["fmt"], h, f, gen)}


def _prepare_step(c, gen):
    h, d = c["hidden"], HEAD_DIM
    hq, hkv = c["q_heads"], c["kv_heads"]
    half = torch.arange(0, d, 2, device="cuda", dtype=torch.float64) / d
    ang = (c["n_ctx"] - 1) / (500000.0 ** half)
    layers = []
    for _ in range(c["layers"]):
        layers.append({
            "qkv": _linear("q4_k", (hq + 2 * hkv) * d, h, gen), "o": _linear("q4_k", h, hq * d, gen),
            "gate_up": _linear("q4_k", 2 * c["ffn"], h, gen), "down": _linear("q4_k", h, c["ffn"], gen),
            "attn_norm": (1 + 0.1 * torch.randn(h, generator=gen, device="cuda")).to(torch.bfloat16),
            "mlp_norm": (1 + 0.1 * torch.randn(h, generator=gen, device="cuda")).to(torch.bfloat16),
            "k": torch.randn(c["rows"], hkv, c["context"], d, generator=gen, device="cuda").to(torch.bfloat16),
            "v": torch.randn(c["rows"], hkv, c["context"], d, generator=gen, device="cuda").to(torch.bfloat16)})
    return {"layers": layers, "head": _linear("q6_k", c["vocab"], h, gen),
            "final_norm": (1 + 0.1 * torch.randn(h, generator=gen, device="cuda")).to(torch.bfloat16),
            "emb": torch.randn(c["vocab"], h, generator=gen, device="cuda", dtype=torch.bfloat16),
            "tokens": torch.randint(0, c["vocab"], (c["rows"],), generator=gen, device="cuda"),
            "cos": torch.cat([ang.cos(), ang.cos()]).to(torch.bfloat16), "sin": torch.cat([ang.sin(), ang.sin()]).to(torch.bfloat16)}


def prepare(case, seed):
    c = dict(case)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = c["kind"]
    s = {"case": c}
    if kind == "linear":
        bias = torch.randn(c["n"], generator=gen, device="cuda").to(DTYPES[c["x"]]) if c["bias"] else None
        s["lin"] = _linear(c["fmt"], c["n"], c["k"], gen, bias)
        s["x"] = _rows(c["rows"], c["k"], gen, DTYPES[c["x"]])
        s["y"] = DTYPES[c["y"]]
    elif kind == "layer":
        s.update(_layer_linears(c, gen))
        s["x"], s["att"], s["h"] = (_rows(c["rows"], c["hidden"], gen) for _ in range(3))
    elif kind == "mlp":
        fmt, h, f = c["fmt"], c["hidden"], c["ffn"]
        s["mlp"] = ttq.GatedMLP(context(), FORMATS[fmt], _blocks(fmt, f, h, gen), _blocks(fmt, f, h, gen), _blocks(fmt, h, f, gen), h, f)
        s["x"] = _rows(c["rows"], h, gen)
    elif kind == "moe":
        e, h, f = c["experts"], c["hidden"], c["ffn"]
        gate_up = _blocks("q4_k", e * 2 * f, h, gen).chunk(e)
        down = _blocks("q4_k", e * h, f, gen).chunk(e)
        s["moe"] = ttq.MoELayer(context(), ttq.FMT_Q4_K, list(gate_up), list(down), h, f, c["top_k"], max_tokens=c["rows"])
        s["x"] = _rows(c["rows"], h, gen)
        # a trained router: every token has its own preferences, and some experts are more popular than others
        logits = torch.randn(c["rows"], e, generator=gen, device="cuda") + 0.3 * torch.randn(e, generator=gen, device="cuda")
        weights, ids = torch.softmax(logits, dim=-1).topk(c["top_k"], dim=-1)
        s["ids"], s["weights"] = ids.to(torch.int32), weights / weights.sum(dim=-1, keepdim=True)
    elif kind == "step":
        s.update(_prepare_step(c, gen))
    else:
        items = []
        for _ in range(c["layers"]):
            for lin in _layer_linears(c, gen).values():
                x = _rows(c["rows"], lin.in_features, gen).cpu().pin_memory()
                items.append((lin, x, torch.zeros(c["rows"], lin.out_features, dtype=torch.bfloat16).pin_memory()))
        s["ys"] = [y for _, _, y in items]
        s["batch"] = ttq.HostBatch(context(), items)
    return s


# ---- passes --------------------------------------------------------------------------------------------------------

def _run_step(s):
    c, ctx, d = s["case"], context(), HEAD_DIM
    b, hq, hkv = c["rows"], c["q_heads"], c["kv_heads"]
    h = s["emb"][s["tokens"]]
    # one or two rows: the norm also leaves its rows in the form the next projection reads
    prep = b <= 2 and c["hidden"] <= 8192
    delta = None
    for L in s["layers"]:
        x = ttq.add_rmsnorm(ctx, h, delta, L["attn_norm"], EPS, prepare=prep)
        qkv = L["qkv"].forward_prepared(b, x.dtype) if prep else L["qkv"].forward(x)
        q = ttq.rope_kv_append(ctx, qkv, hq, hkv, d, s["cos"], s["sin"], L["k"], L["v"], c["n_ctx"] - 1)
        att = ttq.decode_attention(ctx, q, L["k"], L["v"], c["n_ctx"])
        o = L["o"].forward(att.view(b, hq * d))
        x = ttq.add_rmsnorm(ctx, h, o, L["mlp_norm"], EPS, prepare=prep)
        gate_up = L["gate_up"].forward_prepared(b, x.dtype) if prep else L["gate_up"].forward(x)
        delta = L["down"].forward_gated(gate_up)
    x = ttq.add_rmsnorm(ctx, h, delta, s["final_norm"], EPS)
    logits = s["head"].forward(x, out_dtype=torch.float32)
    return [logits] + [t for L in s["layers"] for t in (L["k"], L["v"])]


def run(s):
    kind = s["case"]["kind"]
    if kind == "linear":
        return s["lin"].forward(s["x"], out_dtype=s["y"])
    if kind == "layer":
        qkv, o = s["qkv"].forward(s["x"]), s["o"].forward(s["att"])
        gate_up = s["gate_up"].forward(s["h"])
        if s["case"]["fmt"] == "tq3":  # the gated form serves the block formats
            return [qkv, o, s["down"].forward(ttq.silu_and_mul(context(), gate_up))]
        return [qkv, o, s["down"].forward_gated(gate_up)]
    if kind == "mlp":
        return s["mlp"].forward(s["x"])
    if kind == "moe":
        return s["moe"].forward(s["x"], s["ids"], s["weights"])
    if kind == "step":
        return _run_step(s)
    s["batch"].run()
    return s["ys"]


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _packed(fmt, n, k):
    if fmt == "tq3":
        return n * k * 3 // 8 + 2 * n + k // 8
    return ttq.packed_bytes(FORMATS[fmt], n, k)


def _layer_shapes(c):
    h, f = c["hidden"], c["ffn"]
    return [(h + 2 * c["kv"], h), (h, h), (2 * f, h), (h, f)]


def work(case):
    """Packed weights, inputs and results once each; two operations per weight and row."""
    c, m, kind = case, case["rows"], case["kind"]
    size = {"bf16": 2, "f16": 2, "f32": 4}
    if kind == "linear":
        return {"bytes": _packed(c["fmt"], c["n"], c["k"]) + m * (c["k"] * 2 + c["n"] * size[c["y"]]) + (2 * c["n"] if c["bias"] else 0),
                "flops": 2 * m * c["n"] * c["k"]}
    if kind == "layer":
        shapes = _layer_shapes(c)
        return {"bytes": sum(_packed(c["fmt"], n, k) for n, k in shapes) + 2 * m * (3 * c["hidden"] + shapes[0][0] + 2 * c["hidden"]),
                "flops": 2 * m * sum(n * k for n, k in shapes)}
    if kind == "mlp":
        h, f = c["hidden"], c["ffn"]
        return {"bytes": _packed(c["fmt"], 2 * f, h) + _packed(c["fmt"], h, f) + 4 * m * h, "flops": 2 * m * 3 * h * f}
    if kind == "moe":
        h, f, e, k = c["hidden"], c["ffn"], c["experts"], c["top_k"]
        # experts that m tokens with k distinct choices each are expected to reach, if all are equally popular
        reached = e * (1 - (1 - k / e) ** m)
        return {"bytes": int(reached * (_packed("q4_k", 2 * f, h) + _packed("q4_k", h, f))) + m * (4 * h + 8 * k), "flops": 2 * m * k * 3 * h * f}
    if kind == "step":
        h, q, kv, f = c["hidden"], c["q_heads"] * HEAD_DIM, c["kv_heads"] * HEAD_DIM, c["ffn"]
        shapes = [(q + 2 * kv, h), (h, q), (2 * f, h), (h, f)]
        cache = 2 * m * kv * c["n_ctx"] * 2
        weights = c["layers"] * sum(n * k for n, k in shapes) + c["vocab"] * h
        return {"bytes": c["layers"] * (sum(_packed("q4_k", n, k) for n, k in shapes) + cache) + _packed("q6_k", c["vocab"], h)
                + m * (2 * h + 4 * c["vocab"]), "flops": 2 * m * weights + c["layers"] * 4 * m * q * c["n_ctx"]}
    shapes = _layer_shapes(c) * c["layers"]
    return {"bytes": sum(_packed(c["fmt"], n, k) + 2 * m * (n + k) for n, k in shapes), "flops": 2 * m * sum(n * k for n, k in shapes)}


def tolerance(case):
    """About three to four times what the path shows against the same operations in 64 bits with unrounded intermediates (fp16
    operands, 32-bit sums, results and intermediates rounded to the tensors' own type): one projection 3.6e-4 to an f16 or
    f32 result and 1.7e-3 to a bf16 one, a gated MLP 3.5e-3, a step of two layers 7e-3; largest differences 0.002, 0.005,
    0.018 and 0.037."""
    kind = case["kind"]
    if kind == "linear" and case["y"] != "bf16":
        return {"rel": 1.4e-3, "max": 8e-3}
    if kind in ("linear", "host", "moe"):
        return {"rel": 6e-3, "max": 0.02}
    if kind == "step":
        return {"rel": 2.4e-2, "max": 0.15}
    return {"rel": 1.2e-2, "max": 0.06}


# ---- the same results in 64 bits, in plain torch --------------------------------------------------------------------

def _f16_at(b):
    """Little-endian fp16 bytes [..., 2] -> fp64 [...]."""
    return b.contiguous().view(torch.float16).squeeze(-1).double()


def _hadamard(v):
    """Orthonormal Sylvester-Hadamard transform of every run of 128 along the last dimension."""
    shape = v.shape
    h = torch.ones(1, 1, dtype=torch.float64, device=v.device)
    for _ in range(7):
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
    return (v.reshape(-1, 128) @ (h / math.sqrt(128.0))).reshape(shape)


def _dequantize(fmt, blocks, n, k):
    """fp64 [n][k] weights of the packed blocks."""
    if fmt == "tq3":
        tiles = blocks[:n * k * 3 // 8].reshape(n // 16, k // 16, 96).to(torch.int64)
        tiles = torch.nn.functional.pad(tiles, (0, 3))
        bit = 3 * torch.arange(256, device=blocks.device)
        window = tiles[..., bit // 8] | (tiles[..., bit // 8 + 1] << 8) | (tiles[..., bit // 8 + 2] << 16)
        h = (((window >> (bit % 8)) & 0xffff) * 2654435761) & 0xffffffff
        q = (sum((h >> s) & 255 for s in (0, 8, 16, 24)) - 510).double() / 147.8
        q = q.reshape(n // 16, k // 16, 16, 16).transpose(1, 2).reshape(n, k)
        scale = _f16_at(blocks[n * k * 3 // 8:n * k * 3 // 8 + 2 * n].reshape(n, 2))
        signs = blocks[n * k * 3 // 8 + 2 * n:].reshape(-1, 1).to(torch.int64) >> torch.arange(8, device=blocks.device) & 1
        return scale[:, None] * _hadamard(_hadamard(q).t()).t() * (1.0 - 2.0 * signs.reshape(k).double())
    if fmt == "q8_0":
        b = blocks.reshape(n, k // 32, 34)
        return (_f16_at(b[..., :2])[..., None] * b[..., 2:].contiguous().view(torch.int8).double()).reshape(n, k)
    if fmt == "q4_k":
        b = blocks.reshape(n, k // 256, 144)
        s = b[..., 4:16].to(torch.int64)
        sc = torch.cat([s[..., 0:4] & 63, (s[..., 8:12] & 15) | ((s[..., 0:4] >> 6) << 4)], -1).double()
        mn = torch.cat([s[..., 4:8] & 63, (s[..., 8:12] >> 4) | ((s[..., 4:8] >> 6) << 4)], -1).double()
        qs = b[..., 16:].reshape(n, k // 256, 4, 32)
        q = torch.stack([qs & 15, qs >> 4], dim=3).reshape(n, k // 256, 8, 32).double()
        d, dmin = _f16_at(b[..., 0:2])[..., None], _f16_at(b[..., 2:4])[..., None]
        return ((d * sc)[..., None] * q - (dmin * mn)[..., None]).reshape(n, k)
    b = blocks.reshape(n, k // 256, 210)
    ql, qh = b[..., :128].reshape(n, k // 256, 2, 2, 32).to(torch.int64), b[..., 128:192].reshape(n, k // 256, 2, 32).to(torch.int64)
    low = torch.stack([ql[..., 0, :] & 15, ql[..., 1, :] & 15, ql[..., 0, :] >> 4, ql[..., 1, :] >> 4], dim=3)
    high = torch.stack([(qh >> s) & 3 for s in (0, 2, 4, 6)], dim=3)
    q = ((low | (high << 4)) - 32).double().reshape(n, k // 256, 16, 16)
    sc = b[..., 192:208].contiguous().view(torch.int8).double()
    return (_f16_at(b[..., 208:210])[..., None, None] * sc[..., None] * q).reshape(n, k)


def _weights(fmt, n, k, gen):
    return _dequantize(fmt, _blocks(fmt, n, k, gen), n, k)


def _gated(gate_up):
    g, u = gate_up.chunk(2, dim=-1)
    return torch.nn.functional.silu(g) * u


def _exact_moe(c, gen):
    e, h, f = c["experts"], c["hidden"], c["ffn"]
    gate_up, down = _blocks("q4_k", e * 2 * f, h, gen).chunk(e), _blocks("q4_k", e * h, f, gen).chunk(e)
    x = _rows(c["rows"], h, gen).double()
    logits = torch.randn(c["rows"], e, generator=gen, device="cuda") + 0.3 * torch.randn(e, generator=gen, device="cuda")
    weights, ids = torch.softmax(logits, dim=-1).topk(c["top_k"], dim=-1)
    weights = (weights / weights.sum(dim=-1, keepdim=True)).double()
    y = torch.zeros_like(x)
    for i in range(e):
        row, choice = (ids == i).nonzero(as_tuple=True)
        if len(row):
            out = _gated(x[row] @ _dequantize("q4_k", gate_up[i], 2 * f, h).t()) @ _dequantize("q4_k", down[i], h, f).t()
            y.index_add_(0, row, out * weights[row, choice][:, None])
    return y


def _exact_step(c, gen):
    h, d, b, hq, hkv, f = c["hidden"], HEAD_DIM, c["rows"], c["q_heads"], c["kv_heads"], c["ffn"]
    half = torch.arange(0, d, 2, device="cuda", dtype=torch.float64) / d
    ang = (c["n_ctx"] - 1) / (500000.0 ** half)
    cos, sin = (torch.cat([t, t]).to(torch.bfloat16).double() for t in (ang.cos(), ang.sin()))
    layers = []
    for _ in range(c["layers"]):
        layers.append([_weights("q4_k", n, k, gen) for n, k in (((hq + 2 * hkv) * d, h), (h, hq * d), (2 * f, h), (h, f))]
                      + [(1 + 0.1 * torch.randn(h, generator=gen, device="cuda")).to(torch.bfloat16).double() for _ in range(2)]
                      + [torch.randn(b, hkv, c["context"], d, generator=gen, device="cuda").to(torch.bfloat16).double() for _ in range(2)])
    head = _weights("q6_k", c["vocab"], h, gen)
    final = (1 + 0.1 * torch.randn(h, generator=gen, device="cuda")).to(torch.bfloat16).double()
    emb = torch.randn(c["vocab"], h, generator=gen, device="cuda", dtype=torch.bfloat16)
    x = emb[torch.randint(0, c["vocab"], (b,), generator=gen, device="cuda")].double()

    def norm(v, w):
        return v / torch.sqrt((v * v).mean(dim=-1, keepdim=True) + EPS) * w

    def rope(t):
        return t * cos + torch.cat([-t[..., d // 2:], t[..., :d // 2]], dim=-1) * sin

    for qkv, o, gate_up, down, attn_norm, mlp_norm, kc, vc in layers:
        q, k, v = (norm(x, attn_norm) @ qkv.t()).view(b, hq + 2 * hkv, d).split([hq, hkv, hkv], dim=1)
        kc[:, :, c["n_ctx"] - 1], vc[:, :, c["n_ctx"] - 1] = rope(k), v
        q = rope(q).view(b, hkv, hq // hkv, d)
        p = torch.softmax(q @ kc[:, :, :c["n_ctx"]].transpose(2, 3) / math.sqrt(d), dim=-1)
        x = x + (p @ vc[:, :, :c["n_ctx"]]).reshape(b, hq * d) @ o.t()
        x = x + _gated(norm(x, mlp_norm) @ gate_up.t()) @ down.t()
    return [norm(x, final) @ head.t()] + [t for L in layers for t in L[6:]]


def exact(case, seed):
    c, kind = dict(case), case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "linear":
        bias = torch.randn(c["n"], generator=gen, device="cuda").to(DTYPES[c["x"]]).double() if c["bias"] else 0.0
        w = _weights(c["fmt"], c["n"], c["k"], gen)
        return _rows(c["rows"], c["k"], gen, DTYPES[c["x"]]).double() @ w.t() + bias
    if kind == "layer":
        qkv, o, gate_up, down = (_weights(c["fmt"], n, k, gen) for n, k in _layer_shapes(c))
        x, att, h = (_rows(c["rows"], c["hidden"], gen).double() for _ in range(3))
        return [x @ qkv.t(), att @ o.t(), _gated(h @ gate_up.t()) @ down.t()]
    if kind == "mlp":
        gate, up, down = (_weights(c["fmt"], n, k, gen) for n, k in ((c["ffn"], c["hidden"]), (c["ffn"], c["hidden"]), (c["hidden"], c["ffn"])))
        x = _rows(c["rows"], c["hidden"], gen).double()
        return (torch.nn.functional.silu(x @ gate.t()) * (x @ up.t())) @ down.t()
    if kind == "moe":
        return _exact_moe(c, gen)
    if kind == "step":
        return _exact_step(c, gen)
    ys = []
    for _ in range(c["layers"]):
        shapes = _layer_shapes(c)
        ws = [_weights(c["fmt"], n, k, gen) for n, k in shapes]
        ys += [(_rows(c["rows"], k, gen).double() @ w.t()).cpu() for w, (n, k) in zip(ws, shapes)]
    return ys

"""Performance cases of the quantized-matmul path: the calls a decode, verify, prefill, mixture-of-experts or load-time
program makes through the package's public entry points, from the smallest projection to a full prefill block.

A case is a dict of plain values.  `kind` picks the program:
  proj   one projection through QWGemm.encode (one token up to a prefill batch);
  layer  the matmul path of dense transformer layers: norm, QKV, O, norm, gate||up with SwiGLU, down (the attention
         operator itself is not part of this package, so O reads the query columns of the QKV output);
  mlp    the feed-forward half of such a layer;
  head   final norm, LM head with f32 logits, greedy token;
  moe    router logits and the sparse expert block;
  pack   load time: quantize a plane, then decode it again (what a loader that re-packs and checks a plane does).
Weights are N(0, 0.02), activations N(0, 1), router logits N(0, 1): the distributions of the package's own benchmark.
"""
import math

import torch

from qwegn_b200.gemm import CONTAINERS, QWGemm, QWHal, QWWeightView
from qwegn_b200.moe import QWGemmMoE, QWMoEOperator
from qwegn_b200._lib import EPI_NONE, EPI_SILU_PAIR_FWHT

_DT = {"f16": torch.float16, "f32": torch.float32}


def listed():
    return [
        # The smallest call: one token through a small projection (a key/value or a sharded projection of a 2048-wide model).
        {"name": "proj_2048x2048_m1", "kind": "proj", "fmt": "HQ4_G32", "n": 2048, "k": 2048, "m": 1, "y": "f16", "rotated": False},
        # The benchmark's headline: one decode projection, 12288 x 4096, one token.
        {"name": "proj_12288x4096_m1", "kind": "proj", "fmt": "HQ4_G32", "n": 12288, "k": 4096, "m": 1, "y": "f32", "rotated": False},
        # Verifying a full draft of 16 tokens against the 8-bit pack of a 17408 x 5120 projection.
        {"name": "proj_17408x5120_hq8_m16", "kind": "proj", "fmt": "HQ8_G32", "n": 17408, "k": 5120, "m": 16, "y": "f16", "rotated": False},
        # One decode step over layers of a 27B-class dense model (hidden 5120), captured once in a CUDA graph and replayed for
        # every token, as a decode loop runs it.
        {"name": "decode_27b_graph_m1", "kind": "layer", "layers": 4, "hidden": 5120, "q_heads": 40, "kv_heads": 8, "inter": 17408,
         "attn": "HQ4_G32", "mlp": "HQ4_G32", "m": 1, "graph": True},
        # The same without a graph at 70B-class width with mixed containers (8-bit attention, 4-bit feed-forward).
        {"name": "decode_70b_mixed_m1", "kind": "layer", "layers": 2, "hidden": 8192, "q_heads": 64, "kv_heads": 8, "inter": 28672,
         "attn": "HQ8_G32", "mlp": "HQ4_G32", "m": 1, "graph": False},
        # Speculative verify of 5 tokens through the feed-forward half, group-of-64 container.
        {"name": "verify_mlp_g64_m5", "kind": "mlp", "hidden": 5120, "inter": 17408, "fmt": "HQ4_G64", "m": 5},
        # Greedy sampling: LM head over a vocabulary of 248320.
        {"name": "head_248320_m1", "kind": "head", "fmt": "HQ4_G32", "vocab": 248320, "hidden": 5120, "m": 1},
        # A ragged prompt chunk (or a decode batch of that many sequences) through one dense layer.
        {"name": "layer_27b_m333", "kind": "layer", "layers": 1, "hidden": 5120, "q_heads": 40, "kv_heads": 8, "inter": 17408,
         "attn": "HQ4_G32", "mlp": "HQ4_G32", "m": 333, "graph": False},
        # Prefill of 4096 tokens through the feed-forward half: the largest case.
        {"name": "prefill_mlp_27b_m4096", "kind": "mlp", "hidden": 5120, "inter": 17408, "fmt": "HQ4_G32", "m": 4096},
        # Decode of a few sequences through a sparse block of 256 experts, top-8.
        {"name": "moe_e256_t4", "kind": "moe", "fmt": "HQ4_G32", "experts": 256, "top_k": 8, "hidden": 2048, "inter": 512, "t": 4},
        # Prefill of 2048 tokens through the same block.
        {"name": "moe_e256_t2048", "kind": "moe", "fmt": "HQ4_G32", "experts": 256, "top_k": 8, "hidden": 2048, "inter": 512, "t": 2048},
        # Loading: one 17408 x 5120 plane quantized and decoded.
        {"name": "pack_17408x5120", "kind": "pack", "fmt": "HQ4_G32", "n": 17408, "k": 5120},
    ]


_MAX_FLOPS = 2.0e12     # a drawn case stays below the largest listed one
_MAX_WEIGHTS = 8.0e8    # weights of one state


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _mult(rng, lo, hi, q):
    return max(q, _log(rng, lo, hi) // q * q)


def _tokens(rng):
    """Decode, verify and batched sizes about as often as prefill ones."""
    return _log(rng, 1, 16) if rng.random() < 0.5 else _log(rng, 17, 4096)


def _draw_one(rng):
    kind = rng.choice(("proj", "proj", "layer", "mlp", "head", "moe", "moe", "pack"))
    fmt = rng.choice(("HQ4_G32", "HQ4_G32", "HQ8_G32", "HQ4_G64"))
    kq = 256 if fmt == "HQ4_G64" else 128
    if kind == "proj":
        n = _log(rng, 512, 34816)
        if rng.random() < 0.5:
            n = max(128, n // 128 * 128)
        return {"kind": kind, "fmt": fmt, "n": n, "k": _mult(rng, 1024, 28672, kq), "m": _tokens(rng),
                "y": rng.choice(("f16", "f32")), "rotated": rng.random() < 0.5}
    if kind == "layer":
        attn = rng.choice((fmt, "HQ8_G32"))
        kv = rng.choice((2, 4, 8))
        hidden = _mult(rng, 1024, 8192, 256)
        q_heads = max(2, hidden // 256 * 2)
        m = _tokens(rng)
        return {"kind": kind, "layers": rng.choice((1, 2, 4)), "hidden": hidden, "q_heads": q_heads, "kv_heads": kv,
                "inter": _mult(rng, 2 * hidden, 4 * hidden, 256), "attn": attn, "mlp": fmt, "m": m, "graph": m <= 16 and rng.random() < 0.5}
    if kind == "mlp":
        hidden = _mult(rng, 1024, 8192, 256)
        return {"kind": kind, "hidden": hidden, "inter": _mult(rng, 2 * hidden, 4 * hidden, 256), "fmt": fmt, "m": _tokens(rng)}
    if kind == "head":
        return {"kind": kind, "fmt": fmt, "vocab": _log(rng, 32000, 248320), "hidden": _mult(rng, 1024, 8192, 256), "m": _log(rng, 1, 8)}
    if kind == "moe":
        return {"kind": kind, "fmt": fmt, "experts": rng.choice((32, 64, 128, 256)), "top_k": rng.choice((2, 4, 6, 8)),
                "hidden": _mult(rng, 1024, 4096, 256), "inter": _mult(rng, 256, 1536, 256),
                "t": _log(rng, 1, 8) if rng.random() < 0.5 else _log(rng, 9, 2048)}
    return {"kind": kind, "fmt": fmt, "n": _log(rng, 1024, 17408), "k": _mult(rng, 1024, 8192, kq)}


def draw(rng):
    while True:
        c = _draw_one(rng)
        if work(c)["flops"] <= _MAX_FLOPS and _weights(c) <= _MAX_WEIGHTS:
            return c


def _layer_shapes(c):
    """(rows, k, container) of the four projections of one dense layer; heads are 128 wide."""
    qn, kvn = c["q_heads"] * 128, c["kv_heads"] * 128
    return [(qn + 2 * kvn, c["hidden"], c["attn"]), (c["hidden"], qn, c["attn"]), (2 * c["inter"], c["hidden"], c["mlp"]),
            (c["hidden"], c["inter"], c["mlp"])]


def _shapes(c):
    """Every dense plane a case holds."""
    if c["kind"] == "layer":
        return _layer_shapes(c) * c["layers"]
    if c["kind"] == "mlp":
        return [(2 * c["inter"], c["hidden"], c["fmt"]), (c["hidden"], c["inter"], c["fmt"])]
    if c["kind"] == "head":
        return [(c["vocab"], c["hidden"], c["fmt"])]
    if c["kind"] == "moe":
        e = c["experts"]
        return [(e * 2 * c["inter"], c["hidden"], c["fmt"]), (e * c["hidden"], c["inter"], c["fmt"])]
    return [(c["n"], c["k"], c["fmt"])]


def _weights(c):
    return float(sum(n * k for n, k, _ in _shapes(c)))


def _bank_bytes(n, k, fmt):
    return n * CONTAINERS[fmt].row_bytes(k)


def work(c):
    """What one pass cannot do without: packed weights read once, inputs read once, outputs written once."""
    kind = c["kind"]
    banks = sum(_bank_bytes(*s) for s in _shapes(c))
    if kind == "pack":
        nk = c["n"] * c["k"]
        return {"bytes": 4.0 * nk + 2 * banks + 2.0 * nk, "flops": 0.0}
    if kind == "moe":
        t, k, e, h = c["t"], c["top_k"], c["experts"], c["hidden"]
        active = 1.0 - (1.0 - k / e) ** t     # expected share of the experts that some token names
        router = 2.0 * e * h
        return {"bytes": active * banks + router + 2.0 * t * h + 4.0 * t * e + 4.0 * t * h,
                "flops": 2.0 * t * k * 3 * h * c["inter"] + 2.0 * t * e * h}
    m = c["m"]
    flops = 2.0 * m * _weights(c)
    if kind == "proj":
        return {"bytes": banks + 2.0 * m * c["k"] + m * c["n"] * (2.0 if c["y"] == "f16" else 4.0), "flops": flops}
    if kind == "head":
        return {"bytes": banks + 2.0 * m * c["hidden"] + 4.0 * m * c["vocab"] + 4.0 * m, "flops": flops}
    if kind == "layer":
        return {"bytes": banks + 3 * 2.0 * m * c["hidden"], "flops": flops}   # hidden states in; normed rows and residual out
    return {"bytes": banks + 2 * 2.0 * m * c["hidden"], "flops": flops}


def tolerance(c):
    if c["kind"] == "pack":
        return "exact"    # bytes, and f16 values decoded from them
    if c["kind"] == "proj":
        # f16 operands (rotated activations are rounded once to f16), f32 accumulate, f16 or f32 result
        return {"rel": 1e-3}
    if c["kind"] == "moe":
        # f16 rows between the kernels; "max": router logits of another summation order may swap two experts that tie
        return {"rel": 3e-3, "max": 0.5}
    if c["kind"] == "head":
        return {"rel": 1e-3}
    return {"rel": 3e-3}  # a chain of f16 roundings


# ---- states ---------------------------------------------------------------------------------------------------------

_hals = {}


def _hal(static=True):
    """The device context: one per program.  An inference program loads its weights once and says so."""
    if static not in _hals:
        h = QWHal(torch.cuda.current_device())
        h.set_static_weights(static)
        _hals[static] = h
    return _hals[static]


def _randn(gen, *shape, scale=1.0, dtype=torch.float16):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32).mul_(scale).to(dtype)


def _view(gen, n, k, fmt):
    """A packed plane of N(0, 0.02) weights, made a few hundred million weights at a time."""
    hal, cont = _hal(), CONTAINERS[fmt]
    rb = cont.row_bytes(k)
    bank = torch.empty(n * rb, dtype=torch.uint8, device="cuda")
    step = max(1, 200_000_000 // k)
    for r in range(0, n, step):
        e = min(n, r + step)
        QWGemm.quantize(hal, _randn(gen, e - r, k, scale=0.02, dtype=torch.float32), cont, out=bank[r * rb: e * rb])
    return QWWeightView(bank, n, k, cont)


def _workspace(views, m):
    """One workspace for all calls of the program: (view, epilogue, x is rotated) -> the largest need."""
    need = max(QWGemm.workspaceBytes(_hal(), v, m, epi, rot) for v, epi, rot in views)
    return torch.empty(max(need, 256), dtype=torch.uint8, device="cuda")


def _gamma(gen, hidden):
    return _randn(gen, hidden, scale=0.05)


def prepare(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = {"case": c, "hal": _hal(c["kind"] != "pack")}
    f16 = dict(dtype=torch.float16, device="cuda")
    kind = c["kind"]
    if kind == "proj":
        s["w"] = _view(gen, c["n"], c["k"], c["fmt"])
        s["x"] = _randn(gen, c["m"], c["k"])
        s["y"] = torch.empty((c["m"], c["n"]), dtype=_DT[c["y"]], device="cuda")
        s["ws"] = _workspace([(s["w"], EPI_NONE, c["rotated"])], c["m"])
    elif kind in ("layer", "mlp"):
        m, hidden, inter = c["m"], c["hidden"], c["inter"]
        s["layers"] = []
        if kind == "layer":
            shapes = _layer_shapes(c)
            for _ in range(c["layers"]):
                s["layers"].append(dict(zip(("qkv", "o", "gu", "dn"), [_view(gen, *sh) for sh in shapes]),
                                        g1=_gamma(gen, hidden), g2=_gamma(gen, hidden)))
            s["qkv"] = torch.empty((m, shapes[0][0]), **f16)
        else:
            s["layers"].append(dict(zip(("gu", "dn"), [_view(gen, *sh) for sh in _shapes(c)]), g2=_gamma(gen, hidden)))
        s["gf"] = _gamma(gen, hidden)     # the norm that follows the last layer
        s["x"] = _randn(gen, m, hidden)
        s["res"], s["xn"], s["d"] = (torch.empty((m, hidden), **f16) for _ in range(3))
        s["h"] = torch.empty((m, inter), **f16)
        l0 = s["layers"][0]
        uses = [(l0["gu"], EPI_SILU_PAIR_FWHT, True), (l0["dn"], EPI_NONE, True)]
        if kind == "layer":
            uses += [(l0["qkv"], EPI_NONE, True), (l0["o"], EPI_NONE, False)]
        s["ws"] = _workspace(uses, m)
        if c.get("graph"):
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                _layers(s)
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                _layers(s)
    elif kind == "head":
        s["w"] = _view(gen, c["vocab"], c["hidden"], c["fmt"])
        s["x"], s["gamma"] = _randn(gen, c["m"], c["hidden"]), _gamma(gen, c["hidden"])
        s["xn"] = torch.empty_like(s["x"])
        s["logits"] = torch.empty((c["m"], c["vocab"]), dtype=torch.float32, device="cuda")
        s["tokens"] = torch.empty(c["m"], dtype=torch.int32, device="cuda")
        s["ws"] = _workspace([(s["w"], EPI_NONE, True)], c["m"])
    elif kind == "moe":
        t, e, h = c["t"], c["experts"], c["hidden"]
        gu, dn = (_view(gen, *sh) for sh in _shapes(c))
        s["op"] = QWMoEOperator(s["hal"], gu, dn, e, c["inter"], c["top_k"])
        s["router"] = _randn(gen, e, h, scale=h ** -0.5, dtype=torch.bfloat16)
        s["x"] = _randn(gen, t, h)
        s["logits"] = torch.empty((t, e), dtype=torch.float32, device="cuda")
        s["out"] = torch.empty((t, h), dtype=torch.float32, device="cuda")
        s["scratch"] = torch.empty(s["op"].scratchBytes(t), dtype=torch.uint8, device="cuda")
    else:
        n, k, cont = c["n"], c["k"], CONTAINERS[c["fmt"]]
        s["w"] = _randn(gen, n, k, scale=0.02, dtype=torch.float32)
        s["bank"] = torch.empty(n * cont.row_bytes(k), dtype=torch.uint8, device="cuda")
        s["view"] = QWWeightView(s["bank"], n, k, cont)
        s["out"] = torch.empty((n, k), **f16)
    torch.cuda.synchronize()    # the weights are in place before the first pass reads them
    return s


# ---- passes ---------------------------------------------------------------------------------------------------------

def _layers(s):
    """The dense layers over hidden states x: res is the residual stream, d what the last projection adds to it."""
    hal, ws, xn, res, d, h = s["hal"], s["ws"], s["xn"], s["res"], s["d"], s["h"]
    res.copy_(s["x"])
    last = None
    for l in s["layers"]:
        if "qkv" in l:
            if last is None:
                QWGemm.encodeRMSNorm(hal, res, l["g1"], xn)
            else:
                QWGemm.encodeRMSNorm(hal, d, l["g1"], xn, residual=res)
            QWGemm.encode(hal, l["qkv"], xn, s["qkv"], x_is_rotated=True, workspace=ws)
            QWGemm.encode(hal, l["o"], s["qkv"][:, : l["o"].k], d, workspace=ws)
            QWGemm.encodeRMSNorm(hal, d, l["g2"], xn, residual=res)
        else:
            QWGemm.encodeRMSNorm(hal, res, l["g2"], xn)
        QWGemm.encode(hal, l["gu"], xn, h, epi=EPI_SILU_PAIR_FWHT, x_is_rotated=True, workspace=ws)
        QWGemm.encode(hal, l["dn"], h, d, x_is_rotated=True, workspace=ws)
        last = l
    QWGemm.encodeRMSNorm(hal, d, s["gf"], xn, residual=res)
    return xn, res


def run(s):
    c, hal = s["case"], s["hal"]
    kind = c["kind"]
    if kind == "proj":
        QWGemm.encode(hal, s["w"], s["x"], s["y"], x_is_rotated=c["rotated"], workspace=s["ws"])
        return s["y"]
    if kind in ("layer", "mlp"):
        if "graph" in s:
            s["graph"].replay()
            return s["xn"], s["res"]
        return _layers(s)
    if kind == "head":
        QWGemm.encodeRMSNorm(hal, s["x"], s["gamma"], s["xn"])
        QWGemm.encode(hal, s["w"], s["xn"], s["logits"], x_is_rotated=True, workspace=s["ws"])
        QWGemm.encodeArgmax(hal, s["logits"], s["tokens"])
        return s["logits"], s["tokens"]
    if kind == "moe":
        QWGemmMoE.encodeFnRouterGemm(hal, s["router"], s["x"], s["logits"])
        s["op"].encodeResident(s["x"], s["logits"], s["out"], s["scratch"])
        return s["logits"], s["out"]
    QWGemm.quantize(hal, s["w"], CONTAINERS[c["fmt"]], out=s["bank"])
    QWGemm.dequant(hal, s["view"], s["out"])
    return s["bank"], s["out"]

"""The work a program built on this framework has it do, as cases to time: each is one pass through the public entry
points, from the smallest decode call to a prefill, over the formats and options that serving uses.

Kinds of case:
  linear   one projection through dense_reader.linear.linear, a new output a call: a decode row, a few rows, a prefill
  layer    one decoder layer's projections for a decode step of `rows` sequences, into buffers kept from step to step:
           q|k|v as one block list, the output projection with its residual, gate and up with SwiGLU and per-column
           scales, down with a float32 residual and output; `graph`: the step captured once and replayed, as a server does
  head     the LM head that returns token ids (lm_head_topk.DeviceHead with the rescore and the pick on the device)
  moe      a mixture-of-experts layer with its router: one token, or several rows by the union of their experts
  int4     an int4 projection with group scales for one token
  ternary  a ternary projection behind the block Hadamard rotation: one token, or a batch of rows
  pack     the load path: a float32 matrix on the GPU quantised and packed into the stream the kernels read
"""

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "tensix-kernels_b200"))

from common import ttnn_like as ttnn  # noqa: E402
from dense_reader import linear  # noqa: E402
from int4 import w4a16  # noqa: E402
from lm_head_topk import lmhead  # noqa: E402
from moe import moe8  # noqa: E402
from ternary_matmul import t2  # noqa: E402

DTYPES = {"bfp8": ttnn.bfloat8_b, "bfp4": ttnn.bfloat4_b, "bf16": ttnn.bfloat16}
WEIGHT_BYTES = {"bfp8": 1.0625, "bfp4": 0.5625, "bf16": 2.0, "int4": 0.5625}  # a weight, its share of the exponents or scales included
TERNARY_BYTES = 0.25  # 2 bits a trit; the scales apart


def listed():
    return [
        # the smallest call in use: the README's example, one token through a bfloat8_b weight
        {"name": "token_2048x4096", "kind": "linear", "k": 2048, "n": 4096, "rows": 1, "fmt": "bfp8", "scale": False, "epi": "none"},
        # odd sizes: five rows, K past a power of two, N ending inside a panel, per-column scales
        {"name": "odd_rows5", "kind": "linear", "k": 1056, "n": 1072, "rows": 5, "fmt": "bfp4", "scale": True, "epi": "none"},
        # a Llama-3-8B layer's decode step for one sequence, replayed from a CUDA graph: the latency of a chat
        {"name": "layer_m1_graph", "kind": "layer", "hidden": 4096, "kv": 1024, "inter": 14336, "rows": 1, "fmt": "bfp8",
         "fmt_mlp": "bfp4", "graph": True},
        # a small bf16 model's layer for eight sequences, called step by step
        {"name": "layer_m8_bf16", "kind": "layer", "hidden": 2048, "kv": 512, "inter": 5632, "rows": 8, "fmt": "bf16",
         "fmt_mlp": "bf16", "graph": False},
        # the Llama-3-8B layer for a full decode batch of 32 sequences
        {"name": "layer_m32", "kind": "layer", "hidden": 4096, "kv": 1024, "inter": 14336, "rows": 32, "fmt": "bfp8",
         "fmt_mlp": "bfp4", "graph": False},
        # a prompt of 512 tokens through the gate projection
        {"name": "prefill_512", "kind": "linear", "k": 4096, "n": 14336, "rows": 512, "fmt": "bfp8", "scale": False, "epi": "none"},
        # one token's id from a vocabulary of 151936
        {"name": "head_m1", "kind": "head", "vocab": 151936, "dim": 4096, "chunks": 4, "rows": 1, "fmt": "bfp8"},
        # a Qwen3-30B-A3B MoE layer (8 of 128 experts): one token, then a batch of 16
        {"name": "moe_m1", "kind": "moe", "experts": 128, "hidden": 2048, "inter": 768, "k": 8, "rows": 1, "score": "softmax",
         "graph": False},
        {"name": "moe_m16", "kind": "moe", "experts": 128, "hidden": 2048, "inter": 768, "k": 8, "rows": 16, "score": "softmax",
         "graph": False},
        # one token through int4 gate|up weights of that MLP
        {"name": "int4_m1", "kind": "int4", "k": 4096, "n": 28672},
        # one token through a rotated ternary checkpoint's projection
        {"name": "ternary_m1", "kind": "ternary", "k": 4096, "n": 14336, "g": 128, "rows": 1},
        # loading one MLP matrix
        {"name": "pack_bfp4", "kind": "pack", "k": 4096, "n": 14336, "fmt": "bfp4", "col_scale": True},
    ]


def _size(rng, lo, hi, unit):
    """A multiple of `unit` in lo .. hi, even over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // unit * unit, max(-(-lo // unit) * unit, round(v / unit) * unit))


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["layer"] * 4 + ["head", "moe", "moe", "int4", "ternary", "pack"])
    fmt = rng.choice(["bfp8", "bfp4", "bf16"])
    if kind == "linear":
        many = rng.random() < 0.4
        k, n = _size(rng, 512, 8192 if not many else 4096, 32), _size(rng, 512, 14336, 32)
        rows = _size(rng, 33, 512, 1) if many else _size(rng, 1, 32, 1)
        epi = rng.choice(["none", "silu", "swiglu", "residual", "out32"])
        if epi == "swiglu":
            n = n // 64 * 64
        return {"kind": kind, "k": k, "n": n, "rows": rows, "fmt": fmt, "scale": epi in ("none", "silu") and rng.random() < 0.5, "epi": epi}
    if kind == "layer":
        hidden = _size(rng, 1024, 4096, 128)
        return {"kind": kind, "hidden": hidden, "kv": max(128, hidden // rng.choice([1, 4, 8]) // 32 * 32),
                "inter": _size(rng, 2 * hidden, min(14336, 4 * hidden), 64), "rows": _size(rng, 1, 32, 1), "fmt": fmt,
                "fmt_mlp": fmt if rng.random() < 0.5 else "bfp4", "graph": rng.random() < 0.5}
    if kind == "head":
        chunks = rng.choice([4, 8, 16])
        return {"kind": kind, "vocab": chunks * _size(rng, 32000 // chunks, 151936 // chunks, 32), "dim": _size(rng, 1024, 4096, 128),
                "chunks": chunks, "rows": rng.randint(1, 8), "fmt": rng.choice(["bfp8", "bfp4"])}
    if kind == "moe":
        rows = 1 if rng.random() < 0.5 else rng.randint(2, 16)
        return {"kind": kind, "experts": rng.choice([32, 64, 96, 128]), "hidden": _size(rng, 1024, 2048, 64), "inter": _size(rng, 384, 1024, 32),
                "k": rng.choice([2, 4, 6, 8]), "rows": rows, "score": rng.choice(["softmax", "sigmoid"]), "graph": rows == 1 and rng.random() < 0.5}
    if kind == "int4":
        return {"kind": kind, "k": _size(rng, 1024, 4096, 32), "n": _size(rng, 1024, 14336, 32)}
    if kind == "ternary":
        return {"kind": kind, "k": 1024 * rng.randint(1, 4), "n": _size(rng, 1024, 8192, 32), "g": rng.choice([32, 64, 128]),
                "rows": 1 if rng.random() < 0.5 else _size(rng, 2, 128, 1)}
    return {"kind": kind, "k": _size(rng, 1024, 4096, 32), "n": _size(rng, 1024, 14336, 32), "fmt": fmt, "col_scale": rng.random() < 0.5}


# --- inputs -----------------------------------------------------------------------------------------------------------


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def _matrix(g, n, k):
    """A weight [out, in] as initialised models have them, its output channels of different sizes."""
    return _randn(g, n, k) * 0.02 * (0.5 + torch.rand(n, 1, generator=g, device="cuda"))


def _tensor(dev, t, dtype=ttnn.bfloat16):
    return ttnn.from_torch(t.reshape(1, 1, *t.shape), dtype=dtype, layout=ttnn.TILE_LAYOUT, device=dev)


def _acts(dev, g, rows, k):
    """Activations: standard normal with a few outlier channels."""
    x = _randn(g, rows, k)
    x[:, torch.randint(0, k, (4,), generator=g, device="cuda")] *= 8
    return _tensor(dev, x.to(torch.bfloat16))


def _empty(dev, rows, n, dtype=ttnn.bfloat16):
    return ttnn.allocate_tensor_on_device([1, 1, rows, n], dtype, ttnn.TILE_LAYOUT, dev)


def _captured(step):
    """`step` as a CUDA graph (warmed up first), and what it returns."""
    step()
    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    return graph, out


def _prepare_linear(c, dev, g):
    k, n, rows = c["k"], c["n"], c["rows"]
    s = {"x": _acts(dev, g, rows, k), "scale": None, "opts": {}}
    w = _matrix(g, n, k)
    if c["epi"] == "swiglu":  # the rows are the interleaved gate|up matrix's
        s["opts"]["activation"] = "swiglu"
    elif c["epi"] == "silu":
        s["opts"]["activation"] = "silu"
    elif c["epi"] == "out32":
        s["opts"]["out_dtype"] = ttnn.float32
    elif c["epi"] == "residual":
        s["opts"]["residual"] = _tensor(dev, _randn(g, rows, n).to(torch.bfloat16))
    s["w"], scale = linear.native_weight(dev, w, DTYPES[c["fmt"]], col_scale=c["scale"])
    if c["scale"]:
        s["scale"] = scale
    return s


def _prepare_layer(c, dev, g):
    h, kv, inter, rows = c["hidden"], c["kv"], c["inter"], c["rows"]
    weight = lambda n, k, fmt: linear.native_weight(dev, _matrix(g, n, k), DTYPES[fmt])[0]  # noqa: E731
    wq, wk, wv, wo = (weight(n, h, c["fmt"]) for n in (h, kv, kv, h))
    wg, wu, wd = weight(inter, h, c["fmt_mlp"]), weight(inter, h, c["fmt_mlp"]), weight(h, inter, c["fmt"])
    x, attn, stream = _acts(dev, g, rows, h), _acts(dev, g, rows, h), _tensor(dev, _randn(g, rows, h), ttnn.float32)
    qkv_w = [(wq, 0), (wk, h // 32), (wv, (h + kv) // 32)]
    cols = tuple(0.5 + torch.rand(inter, generator=g, device="cuda") for _ in range(2))
    qkv, hid, mid, y = (_empty(dev, rows, h + 2 * kv), _empty(dev, rows, h), _empty(dev, rows, inter), _empty(dev, rows, h, ttnn.float32))

    def step():
        linear.matmul(x, qkv_w, None, out=qkv)
        linear.matmul(attn, wo, None, residual=x, out=hid)
        linear.matmul(hid, wg, None, w_up=wu, glu=True, col_scales=cols, out=mid)
        linear.matmul(mid, wd, None, residual=stream, out32=True, out=y)
        return [qkv.t, hid.t, mid.t, y.t]

    return _steps(c, step)


def _steps(c, step):
    if not c["graph"]:
        return {"step": step}
    graph, out = _captured(step)
    return {"step": step, "graph": graph, "out": out}


def _prepare_head(c, dev, g):
    w = torch.empty(c["vocab"], c["dim"], dtype=torch.bfloat16, device="cuda")
    for i in range(0, c["vocab"], 16384):
        w[i : i + 16384] = _matrix(g, min(16384, c["vocab"] - i), c["dim"]).to(torch.bfloat16)
    head = lmhead.DeviceHead(dev, w, fmt=c["fmt"], chunks=c["chunks"], device_pick=True)
    return {"head": head, "x": _acts(dev, g, c["rows"], c["dim"]), "rows": c["rows"]}


def _prepare_moe(c, dev, g):
    e, h, i, k, rows = c["experts"], c["hidden"], c["inter"], c["k"], c["rows"]
    P = moe8.pack(dev, _randn(g, e, h, 2 * i) * 0.02, _randn(g, e, i, h) * 0.02)
    x, logits = _acts(dev, g, rows, h), _tensor(dev, _randn(g, rows, e), ttnn.float32)
    bias = _tensor(dev, 0.1 * _randn(g, 1, e), ttnn.float32) if c["score"] == "sigmoid" else None
    ids = _tensor(dev, torch.zeros(rows, k, dtype=torch.int16, device="cuda"), ttnn.uint16)
    w = _empty(dev, rows, k)

    def step():
        moe8.route(logits, ids, w, k, kind=c["score"], bias=bias)
        if rows == 1:
            hid = moe8.gate_up(x, P, ids, w, k)
            y = moe8.down(hid, P, ids, k)
        else:
            hid = moe8.gate_up_rows(x, P, ids, w, k, rows)
            y = moe8.down_rows(hid, P, ids, k, rows)
        return [ids.t, w.t, hid.t, y.t]

    return _steps(c, step)


def _prepare_int4(c, dev, g):
    k, n = c["k"], c["n"]
    codes = torch.randint(-7, 8, (n, k), generator=g, device="cuda", dtype=torch.int8)
    scales = 0.002 + 0.004 * torch.rand(n, k // 32, generator=g, device="cuda")
    s = {"w": w4a16.int4_weight(dev, codes), "scale": w4a16.group_scales(dev, scales), "x": _acts(dev, g, 1, k)}
    w4a16.packed(s["w"], s["scale"])
    return s


def _prepare_ternary(c, dev, g):
    k, n, group = c["k"], c["n"], c["g"]
    u = torch.randint(0, 10, (n, k), generator=g, device="cuda")  # zero with probability 0.3, else +-1
    trits = torch.where(u < 3, 0, torch.where(u % 2 == 0, 1, -1)).to(torch.int8)
    scales = 0.01 + 0.02 * torch.rand(n, k // group, generator=g, device="cuda")
    signs = torch.where(torch.rand(k, generator=g, device="cuda") < 0.5, -1.0, 1.0)
    s = {"w": t2.ternary_weight(dev, trits), "scale": t2.group_scales(dev, scales, t2.HADAMARD_SCALE),
         "had": t2.hadamard_signs(dev, signs), "g": group, "x": _acts(dev, g, c["rows"], k)}
    t2.packed(s["w"], s["scale"], group)
    return s


def _prepare_pack(c, dev, g):
    return {"dev": dev, "w": _matrix(g, c["n"], c["k"]), "dtype": DTYPES[c["fmt"]], "col_scale": c["col_scale"]}


_PREPARE = {"linear": _prepare_linear, "layer": _prepare_layer, "head": _prepare_head, "moe": _prepare_moe, "int4": _prepare_int4,
            "ternary": _prepare_ternary, "pack": _prepare_pack}


def prepare(case, seed):
    dev = ttnn.open_device(0)
    g = torch.Generator(device="cuda").manual_seed(seed)
    return {"kind": case["kind"], **_PREPARE[case["kind"]](case, dev, g)}


def run(s):
    kind = s["kind"]
    if kind == "linear":
        return linear.linear(s["x"], s["w"], s["scale"], **s["opts"]).t
    if kind in ("layer", "moe"):
        if "graph" not in s:
            return s["step"]()
        s["graph"].replay()
        return s["out"]
    if kind == "head":
        records = s["head"].logits_topk(s["x"], s["rows"])
        return [records.t, s["head"].picks[s["rows"]].t[:, :, : s["rows"]]]  # (the page has 32 rows; the call writes its own)
    if kind == "int4":
        return w4a16.w4a16_linear(s["x"], s["w"], s["scale"]).t
    if kind == "ternary":
        return t2.linear(s["x"], s["w"], s["scale"], s["g"], hadamard=s["had"]).t
    w, scale = linear.native_weight(s["dev"], s["w"], s["dtype"], col_scale=s["col_scale"])
    return [w.t, w.emax, scale.t]


# --- what a pass cannot do without, and how far two right answers may lie apart ---------------------------------------


def work(c):
    kind = c["kind"]
    if kind == "linear":
        k, n, m = c["k"], c["n"], c["rows"]
        out = {"swiglu": m * n, "out32": 4 * m * n, "residual": 4 * m * n}.get(c["epi"], 2 * m * n)
        return {"bytes": k * n * WEIGHT_BYTES[c["fmt"]] + 2 * m * k + out + (2 * n if c["scale"] else 0), "flops": 2 * m * k * n}
    if kind == "layer":
        h, kv, i, m = c["hidden"], c["kv"], c["inter"], c["rows"]
        weights = (2 * h * h + 2 * h * kv + h * i) * WEIGHT_BYTES[c["fmt"]] + 2 * h * i * WEIGHT_BYTES[c["fmt_mlp"]]
        acts = m * (2 * h + 2 * (h + 2 * kv) + 6 * h + 2 * h + 2 * i + 2 * i + 8 * h) + 8 * i
        return {"bytes": weights + acts, "flops": 2 * m * (2 * h * h + 2 * h * kv + 3 * h * i)}
    if kind == "head":
        v, d, m = c["vocab"], c["dim"], c["rows"]
        records = c["chunks"] * -(-v // c["chunks"] // 2048) * 8 * 8 * m  # eight (key, index) pairs a row and 2048 columns
        return {"bytes": v * d * WEIGHT_BYTES[c["fmt"]] + 2 * m * d + records + 16 * m * 2 * d, "flops": 2 * m * d * (v + 16)}
    if kind == "moe":
        e, h, i, k, m = c["experts"], c["hidden"], c["inter"], c["k"], c["rows"]
        used = e * (1 - (1 - k / e) ** m)  # distinct experts, on average
        hid = 2 * i * (k if m == 1 else 32 * min(e, m * k))  # the result of gate_up as the entry point returns it
        return {"bytes": used * 3 * h * i * WEIGHT_BYTES["bfp4"] + 2 * m * h + hid + 2 * m * k * i + 2 * h * (1 if m == 1 else 32) + 4 * m * e,
                "flops": 6 * m * k * h * i}
    if kind == "int4":
        return {"bytes": c["k"] * c["n"] * WEIGHT_BYTES["int4"] + 2 * (c["k"] + c["n"]), "flops": 2 * c["k"] * c["n"]}
    if kind == "ternary":
        k, n, m = c["k"], c["n"], c["rows"]
        return {"bytes": k * n * (TERNARY_BYTES + 2 / c["g"]) + 2 * m * (k + n) + k / 8, "flops": 2 * m * k * n}
    return {"bytes": c["k"] * c["n"] * (4 + WEIGHT_BYTES[c["fmt"]]) + 2 * c["n"], "flops": 0}


def tolerance(c):
    if c["kind"] == "pack":
        return "exact"
    if c["kind"] == "linear" and c["epi"] == "out32":
        return {"rel": 1e-5, "max": 1e-3}  # float32 sums of exact products, returned as they are
    if c["kind"] == "head":
        return {"rel": 0, "differ": 0.005}  # keys are bf16 logits: one may round the other way, two near ones trade places
    return {"rel": 1e-2, "max": 0.1}  # bf16 results

"""The performance cases of the quantized-linear layer: what a host program has it do, from one small projection to a
long prefill, each through the public entry points of the package.

Five kinds of work make up the range:

``matvec``   a few projections called one after the other (one call each), 1 ... 16 tokens, every bit width and group size
``dense``    the same for layers whose weights are not quantized
``step``     one decode step of a transformer without its attention: embedding lookup, residual + norm, the fused q/k/v
             projections, o, residual + norm, fused gate/up, the activation product, down, the vocabulary head and the
             greedy token; called directly, or captured once and replayed
``head``     the vocabulary head and the greedy selection over its logits
``prefill``  one transformer layer's seven projections (or one projection) over a prompt of 17 ... 8192 tokens

Activations and weights follow the distributions of the benchmark's configurations: uniform codes,
scale = |N(0, 1)| * 0.002 + 1e-4, bias = -2^(bits - 1) * scale, x ~ N(0, 1).
"""
import importlib

import torch

mlxq = importlib.import_module("mlx-runner_b200")

BITS = (2, 3, 4, 5, 6, 8)
TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
EPS = 1e-6


# ---- the cases -------------------------------------------------------------------------------------------------------
def _step(name, hidden, inter, q, kv, layers, bits, group, vocab, head_bits, tokens, captured):
    return {"name": name, "kind": "step", "hidden": hidden, "inter": inter, "q": q, "kv": kv, "layers": layers, "bits": bits,
            "group": group, "vocab": vocab, "head_bits": head_bits, "tokens": tokens, "captured": captured, "scales": "bf16"}


def _prefill(name, hidden, inter, q, kv, bits, group, scales, x, tokens):
    return {"name": name, "kind": "prefill", "hidden": hidden, "inter": inter, "q": q, "kv": kv, "bits": bits, "group": group,
            "scales": scales, "x": x, "tokens": tokens}


def listed():
    return [
        # the smallest call: a k/v projection of a small model in the layer's own fp32 in, fp32 out
        {"name": "matvec-1024x1024-b4", "kind": "matvec", "rows": 1024, "cols": 1024, "layers": 1, "bits": 4, "group": 64,
         "scales": "f16", "x": "f32", "tokens": 1},
        # one shape of the bit width x group sweep with its largest batch (speculative verification, a few streams)
        {"name": "matvec-11008x4096-b3-t8", "kind": "matvec", "rows": 11008, "cols": 4096, "layers": 8, "bits": 3, "group": 64,
         "scales": "f16", "x": "f16", "tokens": 8},
        # an unquantized output head, two streams
        {"name": "dense-32000x4096-t2", "kind": "dense", "rows": 32000, "cols": 4096, "weights": "bf16", "x": "f32", "tokens": 2},
        # a small 8-bit model's decode step, every call made by the host
        _step("step-1024x28-b8-t1-calls", 1024, 3072, 2048, 1024, 28, 8, 64, 32768, 8, 1, False),
        # the decode step of the 36-layer configuration: 4-bit projections, 6-bit vocabulary head, replayed from a graph
        _step("step-4096x36-b4-t1", 4096, 12288, 4096, 1024, 36, 4, 64, 151936, 6, 1, True),
        # ... and with a batch
        _step("step-4096x36-b4-t6", 4096, 12288, 4096, 1024, 36, 4, 64, 151936, 6, 6, True),
        # the vocabulary head of an 8-bit model with a ragged batch of streams
        {"name": "head-151936-b8-t13", "kind": "head", "rows": 151936, "cols": 4096, "bits": 8, "group": 64, "scales": "f16",
         "x": "f16", "tokens": 13},
        # a short prompt, a middling one and a long one through a layer of the 36-layer configuration
        _prefill("prefill-b4-bf16-t77", 4096, 12288, 4096, 1024, 4, 64, "bf16", "bf16", 77),
        _prefill("prefill-b4-f32-t512", 4096, 12288, 4096, 1024, 4, 64, "bf16", "f32", 512),
        _prefill("prefill-b8-bf16-t384", 4096, 12288, 4096, 1024, 8, 64, "bf16", "bf16", 384),
        _prefill("prefill-b4-bf16-t1999", 4096, 12288, 4096, 1024, 4, 64, "bf16", "bf16", 1999),
        # the largest batch of the prefill benchmark, one projection
        {"name": "prefill-14336x4096-b4-t8192", "kind": "prefill", "rows": 14336, "cols": 4096, "bits": 4, "group": 64,
         "scales": "bf16", "x": "bf16", "tokens": 8192},
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = lo * (hi / lo) ** rng.random()
    return max(lo, int(v) // multiple * multiple)


def _any_format(rng):
    return {"bits": rng.choice((4, 4, 4) + BITS), "group": rng.choice((32, 64, 64, 128)), "scales": rng.choice(("f16", "bf16"))}


def draw(rng):
    kind = rng.choice(("matvec", "matvec", "dense", "step", "step", "head", "prefill", "prefill", "prefill"))
    if kind == "matvec":
        rows, cols = _log_int(rng, 512, 28672, 8), _log_int(rng, 512, 14336, 256)
        return {"kind": kind, "rows": rows, "cols": cols, "layers": rng.randint(1, 8), **_any_format(rng),
                "x": rng.choice(("f32", "f16", "bf16")), "tokens": rng.choice((1, 1, 1, 2, 3, 4, 5, 7, 8, 12, 16))}
    if kind == "dense":
        return {"kind": kind, "rows": _log_int(rng, 512, 65536, 8), "cols": _log_int(rng, 512, 8192, 128),
                "weights": rng.choice(("bf16", "f16")), "x": rng.choice(("f32", "bf16")), "tokens": rng.choice((1, 1, 2, 3, 4, 8, 16))}
    if kind == "step":
        hidden = rng.choice((1024, 1536, 2048, 2560, 4096))
        c = _step("", hidden, _log_int(rng, 2 * hidden, 4 * hidden, 256), hidden, rng.choice((512, 1024)), rng.randint(4, 28 if hidden <= 2048 else 14), 0, 0,
                  _log_int(rng, 16384, 151936, 64), rng.choice((4, 6, 8)), rng.choice((1, 1, 1, 2, 3, 4, 6, 8)), rng.random() < 0.7)
        del c["name"]
        c.update(_any_format(rng))
        return c
    if kind == "head":
        return {"kind": kind, "rows": _log_int(rng, 32000, 151936, 8), "cols": rng.choice((1024, 2048, 2560, 4096)),
                "bits": rng.choice((4, 6, 8)), "group": rng.choice((32, 64, 128)), "scales": rng.choice(("f16", "bf16")),
                "x": rng.choice(("f32", "f16", "bf16")), "tokens": rng.randint(1, 16)}
    x = rng.choice(("f32", "bf16", "bf16", "f16"))
    fmt = _any_format(rng)
    top = 512 if x == "f32" or fmt["bits"] != 4 else 4096
    if rng.random() < 0.5:
        return {"kind": kind, "rows": _log_int(rng, 512, 14336, 8), "cols": _log_int(rng, 512, 14336, 256), **fmt, "x": x,
                "tokens": _log_int(rng, 17, top)}
    hidden = rng.choice((1024, 2048, 2560, 4096))
    c = _prefill("", hidden, _log_int(rng, 2 * hidden, 3 * hidden, 256), hidden, rng.choice((512, 1024)), 0, 0, "", x, _log_int(rng, 17, top // 2))
    del c["name"]
    c.update(fmt)
    return c


# ---- inputs ----------------------------------------------------------------------------------------------------------
class _Maker:
    """Seeded layers and activations on the GPU."""

    def __init__(self, seed):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.gen = torch.Generator(device=self.dev)
        self.gen.manual_seed(seed)

    def normal(self, shape, dtype):
        return torch.randn(shape, device=self.dev, generator=self.gen).to(TORCH[dtype])

    def ids(self, n, top):
        return torch.randint(0, top, (n,), dtype=torch.int32, device=self.dev, generator=self.gen)

    def zeros(self, shape, dtype="f32"):
        return torch.zeros(shape, dtype=TORCH[dtype], device=self.dev)

    def linear(self, rows, cols, bits, group, scales):
        w = torch.randint(-(1 << 31), (1 << 31) - 1, (rows, cols * bits // 32), dtype=torch.int32, device=self.dev, generator=self.gen)
        s = (torch.randn((rows, cols // group), device=self.dev, generator=self.gen).abs() * 0.002 + 1e-4).to(TORCH[scales])
        b = (-float(1 << (bits - 1)) * s.float()).to(TORCH[scales])
        lin = mlxq.Linear(w, s, b, None, inDim=cols)
        lin.prepare()
        return lin

    def dense(self, rows, cols, weights):
        w = (torch.randn((rows, cols), device=self.dev, generator=self.gen) * 0.02).to(TORCH[weights])
        return mlxq.Linear(w, None, None, None, inDim=cols)


class _State:
    pass


def _selection(s, m, rows, tokens):
    s.rows, s.blocks = rows, (rows + mlxq.SELECT_BLOCK - 1) // mlxq.SELECT_BLOCK
    s.logits = m.zeros((tokens, rows))
    s.pairs = torch.zeros(2 * tokens * s.blocks, dtype=torch.int32, device=m.dev)
    s.token = torch.zeros(tokens, dtype=torch.int32, device=m.dev)
    s.value = m.zeros(tokens)


def _prepare_step(s, m, c):
    T, H, I, fmt = c["tokens"], c["hidden"], c["inter"], (c["bits"], c["group"], c["scales"])
    s.head = m.linear(c["vocab"], H, c["head_bits"], 64, c["scales"])
    s.layers = []
    for _ in range(c["layers"]):
        qkv = [m.linear(n, H, *fmt) for n in (c["q"], c["kv"], c["kv"])]
        gate_up = [m.linear(I, H, *fmt) for _ in range(2)]
        norms = [1.0 + 0.1 * m.normal((H,), "f32") for _ in range(2)]
        s.layers.append((norms[0], qkv, m.linear(H, c["q"], *fmt), norms[1], gate_up, m.linear(H, I, *fmt)))
    s.norm = 1.0 + 0.1 * m.normal((H,), "f32")
    s.ids = m.ids(T, c["vocab"])
    s.h, s.x, s.r, s.zero = (m.zeros((T, H)) for _ in range(4))
    s.qkv_width = c["q"] + 2 * c["kv"]
    s.qkv, s.gu, s.a = m.zeros((T, s.qkv_width)), m.zeros((T, 2 * I)), m.zeros((T, I))
    s.hidden, s.inter = H, I
    _selection(s, m, c["vocab"], T)
    s.graph = None
    if c["captured"]:
        _decode_step(s)
        torch.cuda.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            _decode_step(s)


def _prepare_prefill(s, m, c):
    T, fmt = c["tokens"], (c["bits"], c["group"], c["scales"])
    s.y_dtype = c["x"]
    if "rows" in c:
        s.one = m.linear(c["rows"], c["cols"], *fmt)
        s.x, s.y = m.normal((T, c["cols"]), c["x"]), m.zeros((T, c["rows"]), c["x"])
        return
    H, I, Q, KV = c["hidden"], c["inter"], c["q"], c["kv"]
    s.one = None
    s.hidden, s.inter, s.q_width = H, I, Q
    s.lin = [m.linear(o, k, *fmt) for o, k in ((Q, H), (KV, H), (KV, H), (H, Q), (I, H), (I, H), (H, I))]
    s.x1, s.x2, s.act = m.normal((T, H), c["x"]), m.normal((T, H), c["x"]), m.normal((T, I), c["x"])
    s.q, s.k, s.v, s.o = m.zeros((T, Q), c["x"]), m.zeros((T, KV), c["x"]), m.zeros((T, KV), c["x"]), m.zeros((T, H), c["x"])
    s.gu, s.down = m.zeros((T, 2 * I), c["x"]), m.zeros((T, H), c["x"])


def prepare(case, seed):
    s, m, c = _State(), _Maker(seed), case
    s.kind, s.tokens = c["kind"], c["tokens"]
    if s.kind == "matvec":
        s.layers = [m.linear(c["rows"], c["cols"], c["bits"], c["group"], c["scales"]) for _ in range(c["layers"])]
        s.x = m.normal((s.tokens, c["cols"]), c["x"])
        s.y = [m.zeros((s.tokens, c["rows"])) for _ in s.layers]
    elif s.kind == "dense":
        s.layers = [m.dense(c["rows"], c["cols"], c["weights"])]
        s.x = m.normal((s.tokens, c["cols"]), c["x"])
        s.y = [m.zeros((s.tokens, c["rows"]))]
    elif s.kind == "head":
        s.head = m.linear(c["rows"], c["cols"], c["bits"], c["group"], c["scales"])
        s.x = m.normal((s.tokens, c["cols"]), c["x"])
        _selection(s, m, c["rows"], s.tokens)
    elif s.kind == "step":
        _prepare_step(s, m, c)
    else:
        _prepare_prefill(s, m, c)
    return s


# ---- one pass --------------------------------------------------------------------------------------------------------
def _head(s, x):
    s.head.encode(None, x, s.head.inDim, s.logits, s.rows, s.tokens)
    mlxq.blockMax(None, s.logits, s.rows, s.tokens, s.rows, s.pairs)
    mlxq.blockArgmax(None, s.pairs, 1, s.tokens, s.blocks, s.token, s.value)


def _decode_step(s):
    T, H, I = s.tokens, s.hidden, s.inter
    s.head.encodeLookup(None, s.ids, s.h, T)
    r = s.zero
    for norm1, qkv, o, norm2, gate_up, down in s.layers:
        mlxq.addRMSNorm(None, s.h, r, s.x, norm1, H, T, H, EPS)
        mlxq.Linear.encodeFusedDecode(None, qkv, s.x, s.qkv, H, s.qkv_width, T)
        o.encode(None, s.qkv, s.qkv_width, s.r, H, T)          # (the query rows stand in for the attention's output)
        mlxq.addRMSNorm(None, s.h, s.r, s.x, norm2, H, T, H, EPS)
        mlxq.Linear.encodeFusedDecode(None, gate_up, s.x, s.gu, H, 2 * I, T)
        mlxq.actMul(None, s.gu, 2 * I, I, T, mlxq.ACT_SILU, s.a)
        down.encode(None, s.a, I, s.r, H, T)
        r = s.r
    mlxq.addRMSNorm(None, s.h, r, s.x, s.norm, H, T, H, EPS)
    _head(s, s.x)


def _run_prefill(s):
    T = s.tokens
    if s.one is not None:
        s.one.encode(None, s.x, s.one.inDim, s.y, s.one.outDim, T)
        return s.y
    H, I, Q = s.hidden, s.inter, s.q_width
    q, k, v, o, gate, up, down = s.lin
    for lin, y in ((q, s.q), (k, s.k), (v, s.v)):
        lin.encode(None, s.x1, H, y, lin.outDim, T)
    o.encode(None, s.q, Q, s.o, H, T)                           # (the queries stand in for the attention's output)
    gate.encode(None, s.x2, H, s.gu, 2 * I, T)
    up.encode(None, s.x2, H, s.gu[:, I:], 2 * I, T)
    if s.y_dtype == "f32":
        mlxq.actMul(None, s.gu, 2 * I, I, T, mlxq.ACT_SILU, s.act)
    down.encode(None, s.act, I, s.down, H, T)
    return s.q, s.k, s.v, s.o, s.gu, s.down


def run(state):
    s = state
    if s.kind in ("matvec", "dense"):
        for lin, y in zip(s.layers, s.y):
            lin.encode(None, s.x, lin.inDim, y, lin.outDim, s.tokens)
        return s.y
    if s.kind == "head":
        _head(s, s.x)
        return s.logits, s.token, s.value
    if s.kind == "step":
        if s.graph is not None:
            s.graph.replay()
        else:
            _decode_step(s)
        return s.logits, s.token, s.value, s.h
    return _run_prefill(s)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _size(name):
    return 4 if name == "f32" else 2


def _layer_bytes(rows, cols, bits, group):
    return rows * cols * bits // 8 + 2 * 2 * rows * (cols // group)


def work(case):
    c = case
    T = c["tokens"]
    if c["kind"] == "matvec":
        n, O, K = c["layers"], c["rows"], c["cols"]
        return {"bytes": n * (_layer_bytes(O, K, c["bits"], c["group"]) + T * O * 4) + T * K * _size(c["x"]), "flops": 2 * n * T * O * K}
    if c["kind"] == "dense":
        O, K = c["rows"], c["cols"]
        return {"bytes": 2 * O * K + T * (K * _size(c["x"]) + 4 * O), "flops": 2 * T * O * K}
    if c["kind"] == "head":
        O, K = c["rows"], c["cols"]
        return {"bytes": _layer_bytes(O, K, c["bits"], c["group"]) + T * (K * _size(c["x"]) + 4 * O), "flops": 2 * T * O * K}
    if c["kind"] == "prefill" and "rows" in c:
        O, K, e = c["rows"], c["cols"], _size(c["x"])
        return {"bytes": _layer_bytes(O, K, c["bits"], c["group"]) + T * (K + O) * e, "flops": 2 * T * O * K}
    H, I, Q, KV = c["hidden"], c["inter"], c["q"], c["kv"]
    shapes = ((Q, H), (KV, H), (KV, H), (H, Q), (I, H), (I, H), (H, I))
    weights = sum(_layer_bytes(o, k, c["bits"], c["group"]) for o, k in shapes)
    params = sum(o * k for o, k in shapes)
    if c["kind"] == "prefill":
        return {"bytes": weights + T * (2 * H + I + Q + 2 * KV + H + 2 * I + H) * _size(c["x"]), "flops": 2 * T * params}
    head = _layer_bytes(c["vocab"], H, c["head_bits"], 64)
    return {"bytes": c["layers"] * weights + head + 4 * T * (H + c["vocab"]), "flops": 2 * T * (c["layers"] * params + c["vocab"] * H)}


def tolerance(case):
    """Four times the distance of each path's outputs from the same sums in 64 bits ("max": the largest single difference
    over the outputs' root mean square, or over the value itself where that is larger)."""
    if case["kind"] == "step":
        return {"rel": 6e-5, "max": 2e-4}       # fp32 sums through every layer; measured 1.4e-5 / 2.9e-5
    if case["kind"] == "prefill":
        if case["x"] == "bf16":
            return {"rel": 6.6e-3, "max": 1.6e-2}   # the rounding of the outputs; measured 1.66e-3 / 3.9e-3
        if case["x"] == "f16":
            return {"rel": 8e-4, "max": 2e-3}       # measured 2.1e-4 / 4.9e-4
        return {"rel": 2e-5, "max": 1e-4}           # fp32 sums; measured 4.1e-6 / 2.3e-5
    return {"rel": 6e-6, "max": 3e-5}           # fp32 sums; measured 1.4e-6 / 6.8e-6

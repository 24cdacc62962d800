"""The workloads whose speed matters to users of this library, as data plus four functions: ``listed`` / ``draw`` name them,
``prepare`` makes what a program holds before the call, ``run`` is one pass through the public entry points, and ``exact`` gives the
same outputs in 64 bits from plain torch (no code of this library).

Shapes: hidden 4096, intermediate 14336, QKV 6144 is the decoder layer of the library's own benchmark; 8192 x 8192 is its
quantization benchmark and 4096 x 4096 x 4096 its W4A4 benchmark.  The rest is generic.  Weights are N(0, 0.02^2) and come in the way
a checkpoint brings them (nibbles, E4M3 block scales, a decode factor); activations are N(0, 1) with 1 % of the entries ten times
larger, as the activations of a decoder are.
"""
import math

import torch

import nvfp4effma_b200.api as nf
from nvfp4effma_b200.tp import TPLinear

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # One token through one square projection, called from Python: the smallest call there is, bound by latency and launches.
        {"name": "decode_call", "kind": "call", "act": "exact", "image": True, "tokens": 1, "n": 4096, "k": 4096, "dtype": "bf16", "bias": False},
        # Decoding: all linear layers of a few decoder layers as one captured CUDA graph, the way a serving loop replays them;
        # one sequence, and a full small batch (both sides of the line between the two decode kernels).
        {"name": "decode_graph_1", "kind": "stack", "tokens": 1, "layers": 4, "hidden": 4096, "inter": 14336, "qkv": 6144},
        {"name": "decode_graph_8", "kind": "stack", "tokens": 8, "layers": 4, "hidden": 4096, "inter": 14336, "qkv": 6144},
        # A few tokens on a plain checkpoint weight with default options: activations go to INT8 first (W4A8 decode).
        {"name": "decode_w4a8", "kind": "call", "act": "auto", "image": False, "tokens": 4, "n": 14336, "k": 4096, "dtype": "bf16", "bias": False},
        # Prefill of the gate / up projection with SwiGLU: the largest W4A16 GEMM of a layer.
        {"name": "prefill_swiglu", "kind": "glu", "tokens": 2048, "n": 28672, "k": 4096},
        # Prefill with default options and a ragged prompt: W4A8 on the QKV projection, with bias.
        {"name": "prefill_w4a8", "kind": "call", "act": "auto", "image": False, "tokens": 1000, "n": 6144, "k": 4096, "dtype": "bf16", "bias": True},
        # Prefill of a half-precision model: FP16 activations used as they are, a short ragged prompt.
        {"name": "prefill_fp16", "kind": "call", "act": "exact", "image": False, "tokens": 333, "n": 4096, "k": 4096, "dtype": "fp16", "bias": True},
        # W4A4 on operands that are already quantized (swizzled scales): the library's headline GEMM.
        {"name": "w4a4_4096", "kind": "w4a4", "tokens": 4096, "n": 4096, "k": 4096},
        # Training step of one linear layer in NVFP4: both activations quantized in both directions, forward, dgrad and wgrad.
        {"name": "train_linear", "kind": "train", "tokens": 2048, "n": 4096, "k": 4096},
        # Mixture of experts, default options, uneven experts.
        {"name": "moe", "kind": "moe", "experts": 8, "tokens": 1100, "n": 2048, "k": 4096},
        # Quantization of a large matrix with the amax computed by the call, and the way back.
        {"name": "quantize_8192", "kind": "quantize", "rows": 8192, "cols": 8192, "dtype": "bf16", "swizzled": True},
        {"name": "dequantize", "kind": "dequantize", "rows": 4096, "cols": 14336, "dtype": "bf16", "swizzled": False},
    ]


def _log(rng, lo, hi, multiple=1):
    """An integer in [lo, hi], spread over its logarithm, rounded to a multiple."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // multiple * multiple, max(-(-lo // multiple) * multiple, int(round(v / multiple)) * multiple))


def draw(rng):
    kind = rng.choice(["call", "call", "call", "call", "stack", "stack", "glu", "w4a4", "train", "moe", "quantize", "quantize", "dequantize"])
    if kind == "stack":
        hidden = _log(rng, 1024, 4096, 256)
        return {"kind": kind, "tokens": rng.randint(1, 8), "layers": rng.randint(2, 4), "hidden": hidden, "inter": _log(rng, 2 * hidden, 7 * hidden // 2, 256),
                "qkv": hidden + _log(rng, 256, hidden, 128)}
    if kind == "call":
        act = rng.choice(["exact", "auto"])
        dtype = "bf16" if act == "auto" else rng.choice(["bf16", "bf16", "fp16"])
        image = act == "exact" and dtype == "bf16" and rng.random() < 0.6
        tokens = _log(rng, 9, 1200) if rng.random() < 0.6 else rng.randint(1, 8)
        if dtype == "fp16":
            tokens = min(tokens, 400)
        return {"kind": kind, "act": act, "image": image, "tokens": tokens, "n": _log(rng, 512, 8192, rng.choice([1, 8, 64])), "k": _log(rng, 1024, 8192, 64),
                "dtype": dtype, "bias": rng.random() < 0.5}
    if kind == "glu":
        return {"kind": kind, "tokens": _log(rng, 64, 2048), "n": _log(rng, 4096, 28672, 128), "k": _log(rng, 1024, 4096, 64)}
    if kind == "w4a4":
        return {"kind": kind, "tokens": _log(rng, 128, 4096), "n": _log(rng, 1024, 8192, rng.choice([8, 64])), "k": _log(rng, 1024, 8192, 64)}
    if kind == "train":
        return {"kind": kind, "tokens": _log(rng, 256, 2048, 64), "n": _log(rng, 1024, 4096, 64), "k": _log(rng, 1024, 4096, 64)}
    if kind == "moe":
        return {"kind": kind, "experts": rng.choice([4, 8, 16]), "tokens": _log(rng, 500, 1100), "n": _log(rng, 1024, 2048, 16), "k": _log(rng, 1024, 4096, 64)}
    rows, cols = _log(rng, 256, 8192, rng.choice([1, 16])), _log(rng, 1024, 8192, 64)
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])
    return {"kind": kind, "rows": rows if dtype != "fp32" else max(rows // 2, 128), "cols": cols, "dtype": dtype, "swizzled": rng.random() < 0.5}


# ---- inputs -----------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _activations(g, rows, cols, dtype=torch.bfloat16):
    x = torch.randn(rows, cols, generator=g, device=DEV)
    return torch.where(torch.rand(rows, cols, generator=g, device=DEV) < 0.01, x * 10.0, x).to(dtype)


def _e2m1(a):
    """Magnitude codes 0 .. 7 of non-negative values, round to nearest, ties to the even code."""
    return ((a > 0.25).to(torch.uint8) + (a >= 0.75) + (a > 1.25) + (a >= 1.75) + (a > 2.5) + (a >= 3.5) + (a > 5.0)).to(torch.uint8)


def _checkpoint(g, n, k, std=0.02):
    """A weight as a checkpoint holds it: packed nibbles [n, k / 2], E4M3 block scales [n, k / 16], decode factor [1]."""
    w = (torch.randn(n, k, generator=g, device=DEV) * std).to(torch.bfloat16).float().view(n, k // 16, 16)
    glob = (w.abs().max() / (6.0 * 448.0)).reshape(1)
    scales = (w.abs().amax(-1) / (6.0 * glob)).clamp_(max=448.0).to(torch.float8_e4m3fn)
    step = (scales.float() * glob).unsqueeze(-1)
    v = torch.where(step > 0, w / step, torch.zeros_like(w))
    codes = _e2m1(v.abs()) | ((v < 0).to(torch.uint8) << 3)
    codes = codes.view(n, k)
    return codes[:, 0::2] | (codes[:, 1::2] << 4), scales, glob


def _weight(g, n, k):
    return nf.NVFP4Tensor(*_checkpoint(g, n, k))


def _experts(c, g):
    """Row offsets of uneven experts: int32 [experts + 1] on the device."""
    share = torch.rand(c["experts"], generator=g, device=DEV) + 0.25
    cut = (torch.cumsum(share, 0) / share.sum() * c["tokens"]).round()
    return torch.cat([torch.zeros(1, device=DEV), cut]).to(torch.int32)


def _quantize_input(c, g):
    """N(0, 1) with 1 % of the entries x 50."""
    x = torch.randn(c["rows"], c["cols"], generator=g, device=DEV)
    return torch.where(torch.rand(c["rows"], c["cols"], generator=g, device=DEV) < 0.01, x * 50.0, x).to(DTYPES[c["dtype"]])


def _stack_shapes(c):
    return ((c["qkv"], c["hidden"], False), (c["hidden"], c["hidden"], False), (2 * c["inter"], c["hidden"], True), (c["hidden"], c["inter"], False))


def _stack_forward(s):
    return [down(gate_up(o(qkv(s["x"])[:, :s["hidden"]]))) for qkv, o, gate_up, down in s["layers"]]


def prepare(case, seed):
    c, g = case, _gen(seed)
    kind = c["kind"]
    if kind == "call":
        x = _activations(g, c["tokens"], c["k"], DTYPES[c["dtype"]])
        w = _weight(g, c["n"], c["k"])
        bias = torch.randn(c["n"], generator=g, device=DEV).to(x.dtype) if c["bias"] else None
        return {"kind": kind, "x": x, "w": nf.TCWeight(w, "exact") if c["image"] else w, "bias": bias, "act": c["act"]}
    if kind == "glu":
        x = _activations(g, c["tokens"], c["k"])
        return {"kind": kind, "x": x, "layer": TPLinear(_weight(g, c["n"], c["k"]), swiglu=True, replicate=True)}
    if kind == "stack":
        x = _activations(g, c["tokens"], c["hidden"])
        s = {"kind": kind, "x": x, "hidden": c["hidden"],
             "layers": [[TPLinear(_weight(g, n, k), swiglu=glu, replicate=True) for n, k, glu in _stack_shapes(c)] for _ in range(c["layers"])]}
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _stack_forward(s)
        torch.cuda.current_stream().wait_stream(side)
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            s["y"] = _stack_forward(s)
        return s
    if kind == "w4a4":
        x = _activations(g, c["tokens"], c["k"])
        return {"kind": kind, "x": nf.quantize(x, swizzled=True), "w": _weight(g, c["n"], c["k"]).with_scale_layout(True)}
    if kind == "train":
        x, dy = _activations(g, c["tokens"], c["k"]), _activations(g, c["tokens"], c["n"])
        w = (torch.randn(c["n"], c["k"], generator=g, device=DEV) * 0.02).to(torch.bfloat16)
        return {"kind": kind, "x": x, "dy": dy, "w": nf.quantize(w, block="16x16", columnwise=True, swizzled=True)}
    if kind == "moe":
        x = _activations(g, c["tokens"], c["k"])
        return {"kind": kind, "x": x, "w": _weight(g, c["experts"] * c["n"], c["k"]), "seg": _experts(c, g), "experts": c["experts"]}
    if kind == "quantize":
        return {"kind": kind, "x": _quantize_input(c, g), "swizzled": c["swizzled"]}
    if kind == "dequantize":
        w = _weight(g, c["rows"], c["cols"])
        return {"kind": kind, "w": w.with_scale_layout(c["swizzled"]), "dtype": DTYPES[c["dtype"]]}
    raise ValueError(kind)


def run(s):
    kind = s["kind"]
    if kind == "call":
        return nf.linear(s["x"], s["w"], s["bias"], act=s["act"])
    if kind == "glu":
        return s["layer"](s["x"])
    if kind == "stack":
        s["graph"].replay()
        return s["y"]
    if kind == "w4a4":
        return nf.linear(s["x"], s["w"])
    if kind == "train":
        w = s["w"]
        x = nf.quantize(s["x"], columnwise=True, swizzled=True)
        dy = nf.quantize(s["dy"], columnwise=True, swizzled=True)
        y = nf.linear(x, w)
        dx = nf.linear(dy, w.columnwise)
        dw = nf.linear(dy.columnwise, x.columnwise, out_dtype=torch.float32)
        return {"y": y, "dx": dx, "dw": dw}
    if kind == "moe":
        return nf.grouped_linear(s["x"], s["w"], s["seg"], s["experts"])
    if kind == "quantize":
        q = nf.quantize(s["x"], swizzled=s["swizzled"])
        return {"data": q.data, "scales": q.scales.view(torch.uint8), "amax": q.amax}
    return nf.dequantize(s["w"], s["dtype"])


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------------------
FP4 = 0.5625   # bytes of a quantized value: half a byte and a sixteenth of a scale byte


def _size(c):
    return 4 if c["dtype"] == "fp32" else 2


def work(case):
    c = case
    kind = c["kind"]
    if kind == "call":
        t, n, k = c["tokens"], c["n"], c["k"]
        return {"bytes": FP4 * n * k + 2 * t * (n + k), "flops": 2.0 * t * n * k}
    if kind == "glu":
        t, n, k = c["tokens"], c["n"], c["k"]
        return {"bytes": FP4 * n * k + 2 * t * (n // 2 + k), "flops": 2.0 * t * n * k}
    if kind == "stack":
        weights = c["layers"] * sum(n * k for n, k, _ in _stack_shapes(c))
        return {"bytes": FP4 * weights + 2 * c["tokens"] * c["hidden"] * (c["layers"] + 1), "flops": 2.0 * c["tokens"] * weights}
    if kind == "w4a4":
        t, n, k = c["tokens"], c["n"], c["k"]
        return {"bytes": FP4 * k * (n + t) + 2 * t * n, "flops": 2.0 * t * n * k}
    if kind == "train":
        t, n, k = c["tokens"], c["n"], c["k"]
        return {"bytes": 2 * t * (n + k) + 2 * FP4 * n * k + 2 * t * (n + k) + 4 * n * k, "flops": 6.0 * t * n * k}
    if kind == "moe":
        t, n, k = c["tokens"], c["n"], c["k"]
        return {"bytes": FP4 * c["experts"] * n * k + 2 * t * (n + k), "flops": 2.0 * t * n * k}
    return {"bytes": c["rows"] * c["cols"] * (FP4 + _size(c)), "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind in ("quantize", "dequantize"):
        return "exact"          # bytes and correctly rounded products
    if kind == "stack":
        return {"rel": 2e-2}    # four BF16 roundings in a row
    if kind == "glu":
        return {"rel": 7e-3}    # one BF16 rounding of the result: 1.7e-3 off the exact value
    if kind == "call" and case["dtype"] == "fp16":
        return {"rel": 1e-3}    # one FP16 rounding: 2.1e-4 off
    return {"rel": 7e-3}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------------------
_VALUES = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


def _value_of(codes):
    table = torch.tensor(_VALUES + tuple(-v for v in _VALUES), dtype=torch.float64, device=DEV)
    return table[codes.long()]


def _decoded(parts):
    """The checkpoint weight [n, k] in float64."""
    data, scales, glob = parts
    n, half = data.shape
    codes = torch.stack((data & 15, data >> 4), -1).view(n, 2 * half)
    return (_value_of(codes).view(n, half // 8, 16) * scales.double().unsqueeze(-1) * glob.double()).view(n, 2 * half)


def _as_int8(x):
    """Activations after the INT8 step: q * s with s = max |x| of 16 values / 127."""
    v = x.float().view(x.shape[0], -1, 16)
    s = v.abs().amax(-1, keepdim=True) / 127.0
    q = torch.where(s > 0, (v / s).round().clamp_(-127, 127), torch.zeros_like(v))
    return (q.double() * s.double()).view(x.shape)


def _as_nvfp4(x, tile=1):
    """x after NVFP4 quantization in Transformer Engine's arithmetic with the amax of x; tile 16: 16 x 16 tiles share a scale."""
    v = x.float().view(x.shape[0], -1, 16)
    amax = v.abs().max()
    enc = torch.tensor(2688.0, device=DEV) / amax
    dec = torch.ones((), device=DEV) / enc
    bmax = v.abs().amax(-1)
    if tile == 16:
        bmax = bmax.view(-1, 16, bmax.shape[1]).amax(1, keepdim=True).expand(-1, 16, -1).reshape(bmax.shape)
    scale = (bmax * (enc * torch.tensor(1.0 / 6.0, device=DEV))).clamp(max=448.0).to(torch.float8_e4m3fn).float()
    inv = (torch.ones((), device=DEV) / (scale * dec)).clamp(max=torch.finfo(torch.float32).max).unsqueeze(-1)
    q = v * inv
    mag = _value_of(_e2m1(q.abs()))
    out = torch.where(q < 0, -mag, mag) * scale.double().unsqueeze(-1) * (amax.double() / 2688.0)
    return out.view(x.shape)


def _swiglu(y):
    """Rows of gate and up weights alternate in groups of eight: silu(gate) * up."""
    v = y.view(y.shape[0], -1, 2, 8)
    gate, up = v[:, :, 0], v[:, :, 1]
    return (gate * torch.sigmoid(gate) * up).reshape(y.shape[0], -1)


def exact(case, seed):
    c, g = case, _gen(seed)
    kind = c["kind"]
    if kind == "call":
        x = _activations(g, c["tokens"], c["k"], DTYPES[c["dtype"]])
        w = _decoded(_checkpoint(g, c["n"], c["k"]))
        bias = torch.randn(c["n"], generator=g, device=DEV).to(x.dtype) if c["bias"] else None
        int8 = c["act"] == "auto" and c["tokens"] > 2
        y = (_as_int8(x) if int8 else x.double()) @ w.t()
        return y if bias is None else y + bias.double()
    if kind == "glu":
        x = _activations(g, c["tokens"], c["k"])
        return _swiglu(x.double() @ _decoded(_checkpoint(g, c["n"], c["k"])).t())
    if kind == "stack":
        x = _activations(g, c["tokens"], c["hidden"]).double()
        out = []
        for _ in range(c["layers"]):
            y = x
            for i, (n, k, glu) in enumerate(_stack_shapes(c)):
                y = y @ _decoded(_checkpoint(g, n, k)).t()
                y = _swiglu(y) if glu else y[:, :c["hidden"]] if i == 0 else y
            out.append(y)
        return out
    if kind == "w4a4":
        x = _activations(g, c["tokens"], c["k"])
        return _as_nvfp4(x) @ _decoded(_checkpoint(g, c["n"], c["k"])).t()
    if kind == "train":
        x, dy = _activations(g, c["tokens"], c["k"]), _activations(g, c["tokens"], c["n"])
        w = (torch.randn(c["n"], c["k"], generator=g, device=DEV) * 0.02).to(torch.bfloat16)
        xc, dyc = _as_nvfp4(x.t().contiguous()), _as_nvfp4(dy.t().contiguous())     # the transposes, quantized along the tokens
        wq = _as_nvfp4(w, 16)
        return {"y": _as_nvfp4(x) @ wq.t(), "dx": _as_nvfp4(dy) @ wq, "dw": dyc @ xc.t()}
    if kind == "moe":
        x = _as_int8(_activations(g, c["tokens"], c["k"]))
        w = _decoded(_checkpoint(g, c["experts"] * c["n"], c["k"])).view(c["experts"], c["n"], c["k"])
        seg = _experts(c, g).tolist()
        return torch.cat([x[a:b] @ w[e].t() for e, (a, b) in enumerate(zip(seg[:-1], seg[1:]))])
    if kind == "dequantize":
        return _decoded(_checkpoint(g, c["rows"], c["cols"]))
    return None    # quantization: codes, compared byte for byte

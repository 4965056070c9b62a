"""The calls whose speed counts: the quantized-linear operators as a compiled
model makes them (krnl.call entry points of libomcuda on device tensors, weights
registered as the constants they are) and whole encoder runs.

A case is a dict of plain values.  `prepare` makes what a program holds before
the call, `run` is one pass through the public entry points, `work` the bytes
and operations the pass cannot do without (every input read once, every output
written once)."""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "onnx-mlir_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import omcuda  # noqa: E402

# hidden, heads, ffn, layers of the two encoder configurations
ENCODERS = {"base": (768, 12, 3072, 12), "large": (1024, 16, 4096, 24)}

# A registered constant is known by its address until omcudaForgetConstants, so
# its memory is never given back while the process lives: a serving program
# keeps its weights as well.
_constants = []


def listed():
    return [
        # one linear layer on a 128-token request: the smallest tensor-core call
        {"name": "linear_128x768x768", "kind": "linear", "M": 128, "K": 768, "N": 768,
         "w": "i8", "per_column": False},
        # decoding, one row: a pass over the weight
        {"name": "linear_1x4096x14336", "kind": "linear", "M": 1, "K": 4096, "N": 14336,
         "w": "i8", "per_column": False},
        # decoding, 16 sequences at once
        {"name": "linear_16x14336x4096", "kind": "linear", "M": 16, "K": 14336, "N": 4096,
         "w": "i8", "per_column": False},
        # nothing divides anything; unsigned weights with a zero point and
        # per-column scales
        {"name": "linear_777x1001x1537_u8", "kind": "linear", "M": 777, "K": 1001, "N": 1537,
         "w": "u8", "per_column": True},
        # prefill: the square size GEMMs are compared at
        {"name": "linear_4096x4096x4096", "kind": "linear", "M": 4096, "K": 4096, "N": 4096,
         "w": "i8", "per_column": False},
        # statically quantized linear, u8 in and out, per-column weight scales
        {"name": "qlinear_16384x1024x4096", "kind": "qlinear", "M": 16384, "K": 1024, "N": 4096,
         "y": "u8", "per_column": True},
        # attention scores of a quantized model: both operands are activations
        {"name": "matmul_integer_384x128x64x128", "kind": "matmul_integer", "batch": 32,
         "heads": 12, "M": 128, "K": 64, "N": 128},
        # a large activation quantized by itself
        {"name": "dynamic_quantize_64Mi", "kind": "quantize", "n": 64 << 20, "dynamic": True},
        # and the other direction, an odd number of elements
        {"name": "dequantize_8191x3073", "kind": "dequantize", "n": 8191 * 3073, "x": "u8"},
        # one short question to a bert_base-shaped model, numpy in and out
        {"name": "encoder_base_1x61_host", "kind": "encoder", "model": "base", "batch": 1,
         "seq": 61, "host": True},
        # the two encoder configurations at their own sizes, resident activations
        {"name": "encoder_base_32x128", "kind": "encoder", "model": "base", "batch": 32,
         "seq": 128, "host": False},
        {"name": "encoder_large_256x512", "kind": "encoder", "model": "large", "batch": 256,
         "seq": 512, "host": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A matrix dimension: mostly a multiple of 64, as model widths are, else any."""
    v = _log(rng, lo, hi)
    return max(64, v // 64 * 64) if rng.random() < 0.7 else v


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "linear", "qlinear", "matmul_integer",
                       "quantize", "dequantize", "encoder", "encoder", "encoder"])
    if kind == "linear":
        return {"kind": kind, "M": _log(rng, 1, 16384), "K": _width(rng, 256, 14336),
                "N": _width(rng, 256, 14336), "w": rng.choice(["i8", "i8", "u8"]),
                "per_column": rng.random() < 0.3}
    if kind == "qlinear":
        return {"kind": kind, "M": _log(rng, 16, 16384), "K": _width(rng, 256, 4096),
                "N": _width(rng, 256, 4096), "y": rng.choice(["u8", "i8"]),
                "per_column": rng.random() < 0.7}
    if kind == "matmul_integer":
        s, d = _log(rng, 17, 512), rng.choice([32, 64, 128])
        scores = rng.random() < 0.5  # Q K^T, or probabilities times V
        return {"kind": kind, "batch": _log(rng, 1, 32), "heads": rng.choice([8, 12, 16]),
                "M": s, "K": d if scores else s, "N": s if scores else d}
    if kind == "quantize":
        return {"kind": kind, "n": _log(rng, 1000, 128 << 20), "dynamic": rng.random() < 0.7}
    if kind == "dequantize":
        return {"kind": kind, "n": _log(rng, 1000, 128 << 20),
                "x": rng.choice(["u8", "i8", "i32"])}
    model = rng.choice(["base", "large"])
    seq = rng.choice([128, 256, 384, 512, rng.randint(16, 512), rng.randint(16, 512)])
    host = rng.random() < 0.3
    batch = max(1, _log(rng, 16, 4096 if host else 65536) // seq)
    return {"kind": kind, "model": model, "batch": batch, "seq": seq, "host": host}


def _bytes(dtype):
    return 4 if dtype == "i32" else 1


def work(c):
    kind = c["kind"]
    if kind in ("linear", "qlinear"):
        M, K, N = c["M"], c["K"], c["N"]
        io = 4 if kind == "linear" else 1
        return {"bytes": io * M * K + K * N + io * M * N + 4 * N, "flops": 2 * M * K * N}
    if kind == "matmul_integer":
        n, M, K, N = c["batch"] * c["heads"], c["M"], c["K"], c["N"]
        return {"bytes": n * (M * K + K * N + 4 * M * N), "flops": 2 * n * M * K * N}
    if kind == "quantize":
        return {"bytes": 5 * c["n"], "flops": 0}
    if kind == "dequantize":
        return {"bytes": (4 + _bytes(c["x"])) * c["n"], "flops": 0}
    H, heads, F, layers = ENCODERS[c["model"]]
    T = c["batch"] * c["seq"]
    weights = layers * (4 * H * H + 2 * H * F)
    return {"bytes": 8 * T * H + weights,
            "flops": 2 * T * weights + layers * 4 * T * c["seq"] * H}


def tolerance(c):
    if c["kind"] in ("qlinear", "matmul_integer", "quantize"):
        return "exact"
    if c["kind"] in ("linear", "dequantize"):
        return {"rel": 1e-5}  # integer sums, then a few fp32 operations
    # Every linear of an encoder rounds its input to 8 bits: an fp32 softmax or
    # LayerNorm summed in another order moves some values to the next step, and
    # 12 to 24 layers carry that on.
    return {"rel": 1e-2}


# ---- inputs -----------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, shape, std=1.0):
    return torch.empty(shape, device="cuda").normal_(0.0, std, generator=g)


def _int8(g, shape, dtype):
    lo, hi = (-127, 128) if dtype == "i8" else (0, 256)
    return torch.randint(lo, hi, shape, device="cuda", generator=g,
                         dtype=torch.int8 if dtype == "i8" else torch.uint8)


def _scalar(v, dtype):
    return torch.tensor(v, device="cuda", dtype=dtype)


def _t(x):
    return omcuda.Tensor.from_cuda_array(x)


def _constant(x):
    """A weight: registered, so that the library lays it out once."""
    t = _t(x)
    omcuda.lib().omcudaRegisterConstant(t.handle)
    _constants.append((t, x))
    return t


def _empty(shape, dtype):
    return torch.empty(shape, device="cuda", dtype=dtype)


class _Op:
    """A krnl.call: the library function, its tensors (outputs first) and its
    integer attributes, and the buffers of the outputs."""

    def __init__(self, name, tensors, attrs, outputs):
        self.fn = getattr(omcuda.lib(), name)
        self.tensors = tensors
        self.args = [t.handle if t is not None else None for t in tensors] + attrs
        self.outputs = outputs


class _Model:
    """An encoder with its weights and one request."""

    def __init__(self, c, seed):
        H, heads, F, layers = ENCODERS[c["model"]]
        g = _gen(seed)
        self.encoder = omcuda.Encoder(H, heads, F, [_layer(g, H, F) for _ in range(layers)])
        x = _normal(g, (c["batch"], c["seq"], H))
        self.host = c["host"]
        if self.host:
            self.x = x.cpu().numpy()
        else:
            self.y = torch.empty_like(x)
            self.x, self.out = _t(x), _t(self.y)


def _layer(g, H, F):
    """N(0, 0.02) weights quantized per tensor, symmetric; N(0, 0.02) biases."""
    w, sc = {}, []
    for name, shape in (("wq", (H, H)), ("wk", (H, H)), ("wv", (H, H)), ("wo", (H, H)),
                        ("w1", (H, F)), ("w2", (F, H))):
        f = _normal(g, shape, 0.02)
        s = f.abs().max() / 127.0
        w[name] = torch.round(f / s).clamp_(-127, 127).to(torch.int8).cpu().numpy()
        sc.append(float(s))
    w["sc"] = np.array(sc, np.float32)
    for name, n in (("bq", H), ("bk", H), ("bv", H), ("bo", H), ("b1", F), ("b2", H),
                    ("ln1b", H), ("ln2b", H)):
        w[name] = _normal(g, (n,), 0.02).cpu().numpy()
    for name in ("ln1g", "ln2g"):
        w[name] = 1 + _normal(g, (H,), 0.02).cpu().numpy()
    return w


def prepare(c, seed):
    omcuda.init()
    kind = c["kind"]
    if kind == "encoder":
        state = _Model(c, seed)
        torch.cuda.synchronize()
        return state
    g = _gen(seed)
    if kind == "linear":
        M, K, N = c["M"], c["K"], c["N"]
        x, y = _normal(g, (M, K)), _empty((M, N), torch.float32)
        w = _constant(_int8(g, (K, N), c["w"]))
        sc = (torch.rand((N,), device="cuda", generator=g) * 0.009 + 0.001) if c["per_column"] \
            else _scalar(0.0157, torch.float32)
        zp = _t(_scalar(128, torch.uint8)) if c["w"] == "u8" else None
        op = _Op("omcudaDynQuantLinear",
                 [_t(y), _t(x), w, _t(sc), zp, _t(_normal(g, (N,), 0.02))], [0], [y])
    elif kind == "qlinear":
        M, K, N = c["M"], c["K"], c["N"]
        yt = torch.uint8 if c["y"] == "u8" else torch.int8
        a, y = _int8(g, (M, K), "u8"), _empty((M, N), yt)
        n = (N,) if c["per_column"] else ()
        bs = torch.rand(n, device="cuda", generator=g) * 0.009 + 0.001
        op = _Op("omcudaQLinearMatMul",
                 [_t(y), _t(a), _t(_scalar(0.02, torch.float32)), _t(_scalar(128, torch.uint8)),
                  _constant(_int8(g, (K, N), "i8")), _t(bs),
                  _t(torch.zeros(n, device="cuda", dtype=torch.int8)),
                  _t(_scalar(0.5, torch.float32)),
                  _t(_scalar(128 if c["y"] == "u8" else 0, yt))], [], [y])
    elif kind == "matmul_integer":
        lead = (c["batch"], c["heads"])
        a = _int8(g, lead + (c["M"], c["K"]), "u8")
        b = _int8(g, lead + (c["K"], c["N"]), "u8")
        y = _empty(lead + (c["M"], c["N"]), torch.int32)
        op = _Op("omcudaMatMulInteger", [_t(y), _t(a), _t(b), _t(_scalar(131, torch.uint8)),
                                         _t(_scalar(120, torch.uint8))], [], [y])
    elif kind == "quantize":
        x, y = _normal(g, (c["n"],)), _empty((c["n"],), torch.uint8)
        if c["dynamic"]:
            s, z = _empty((), torch.float32), _empty((), torch.uint8)
            op = _Op("omcudaDynamicQuantizeLinear", [_t(y), _t(s), _t(z), _t(x)], [], [y, s, z])
        else:
            op = _Op("omcudaQuantizeLinear", [_t(y), _t(x), _t(_scalar(0.03, torch.float32)),
                                              _t(_scalar(128, torch.uint8))], [], [y])
    elif kind == "dequantize":
        if c["x"] == "i32":
            x = torch.randint(-(1 << 20), 1 << 20, (c["n"],), device="cuda", generator=g,
                              dtype=torch.int32)
            zp = None
        else:
            x = _int8(g, (c["n"],), c["x"])
            zp = _t(_scalar(3, x.dtype))
        y = _empty((c["n"],), torch.float32)
        op = _Op("omcudaDequantizeLinear",
                 [_t(y), _t(x), _t(_scalar(0.02, torch.float32)), zp], [], [y])
    else:
        raise ValueError("unknown kind %r" % kind)
    torch.cuda.synchronize()
    return op


def run(state):
    if isinstance(state, _Op):
        state.fn(*state.args)
        omcuda.check()
        return state.outputs
    if state.host:
        return state.encoder.run(state.x)
    state.encoder.run_into(state.x, state.out)
    return state.y

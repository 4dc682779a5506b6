"""The work that is timed: what a user of the quantization path has it do, through the package's public functions.

A case is a dict of plain values.  ``listed()`` are the fixed ones, ``draw()`` gives others of the same ranges,
``prepare()`` makes what a program holds before the call (inputs, weights laid out once), ``run()`` is one pass.
Shapes are the repository's benchmark configurations, the benchmark shapes of ``saturated_cast`` and generic
layer sizes; values follow ``driss_torch_b200.workloads``.

Kinds of work (``case["kind"]``):

* ``cast``        saturated_cast with a known scale: the static-scale fp8 cast of a tensor of any shape.
* ``operands``    delayed scaling of a training operand: the tensor's amax for the next step's scale, and the fp8
                  casts of x and of its transpose with this step's (known) scale.
* ``tensorwise``  dynamic tensor-wise quantization: amax -> scale -> cast, with the amax and scale returned.
* ``mx_cast``     the MX block-32 cast with row-major scales.
* ``rowwise``     a row-wise scaled fp8 linear layer: activations quantized per row, then sweep_mm with weights
                  that were quantized when they were loaded.  Few tokens: decode; many: prefill.
* ``mx8``         an MXFP8 linear layer: activations cast with scales in the GEMM's layout, then mx_fp8_bf16.
* ``mx4``         the same in MXFP4 (mx_fp4_quantize, mx_fp4_bf16).
* ``mx8_train``   one training step's work of an MXFP8 linear layer: x, w and the output gradient cast in both
                  orientations, then the three products (forward, input gradient, weight gradient).
* ``both``        the tensor-wise and the MX quantization of one large matrix (ShardedQuantizer on one GPU).
"""
import math

import torch

import driss_torch_b200 as dtq

DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
FP8 = {"e4m3": torch.float8_e4m3fn, "e5m2": torch.float8_e5m2}
DEVICE = "cuda"

# The largest drawn products and tensors stay below the largest listed ones.
MAX_LINEAR_FLOPS = 1.1e12
MAX_ELEMENTS = 2 ** 28


def listed():
    return [
        # A single ragged row: nothing but launch and host latency (the smallest of the cast's benchmark shapes).
        {"name": "cast_row", "kind": "cast", "rows": 1, "cols": 3232, "in": "bf16", "out": "e4m3"},
        # The widest of the cast's benchmark shapes, as a gradient (e5m2): a pure stream.
        {"name": "cast_wide", "kind": "cast", "rows": 2048, "cols": 109760, "in": "bf16", "out": "e5m2"},
        # A training operand under delayed scaling; packed sequences give token counts that are no multiple of anything.
        {"name": "operands_ragged", "kind": "operands", "rows": 5003, "cols": 4096, "in": "bf16", "out": "e4m3"},
        # The benchmark's dynamic tensor-wise quantization: an activation matrix with outliers.
        {"name": "tensorwise_square", "kind": "tensorwise", "rows": 8192, "cols": 8192, "in": "bf16", "out": "e4m3"},
        # A small fp32 tensor of odd sizes (fp32 is the only input type the reference's fused op takes), e5m2 out.
        {"name": "tensorwise_odd_fp32", "kind": "tensorwise", "rows": 2047, "cols": 1023, "in": "fp32", "out": "e5m2"},
        # The benchmark's MX cast: blocks over a wide exponent range, with zeros.
        {"name": "mx_cast", "kind": "mx_cast", "rows": 16384, "cols": 8192, "in": "bf16", "out": "e4m3"},
        # Decode of 16 sequences through a row-wise scaled layer: latency, and the weights read once.
        {"name": "rowwise_decode", "kind": "rowwise", "tokens": 16, "k": 4096, "n": 8192, "bias": False},
        # Prefill through the same kind of layer: the benchmark's row-wise activations, then a large product with bias.
        {"name": "rowwise_prefill", "kind": "rowwise", "tokens": 32768, "k": 4096, "n": 4096, "bias": True},
        # Decode of 8 sequences through a large MXFP8 layer.
        {"name": "mx8_decode", "kind": "mx8", "tokens": 8, "k": 8192, "n": 8192},
        # An ordinary ragged prompt through an MXFP4 layer.
        {"name": "mx4_prompt", "kind": "mx4", "tokens": 2000, "k": 4096, "n": 12288},
        # Forward and backward of an MXFP8 layer at the benchmark's GEMM size.
        {"name": "mx8_train", "kind": "mx8_train", "tokens": 8192, "k": 8192, "n": 8192},
        # The benchmark's step: a 4 GiB matrix quantized tensor-wise and in MX blocks.
        {"name": "both_4gib", "kind": "both", "rows": 262144, "cols": 8192, "out": "e4m3"},
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, its logarithm uniform."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _log_multiple(rng, lo, hi, m):
    return max(m, _log(rng, lo, hi) // m * m)


def draw(rng):
    kind = rng.choice(["cast", "operands", "tensorwise", "mx_cast", "rowwise", "rowwise", "mx8", "mx8", "mx4", "mx8_train", "both"])
    if kind in ("cast", "tensorwise"):
        numel = _log(rng, 2048, MAX_ELEMENTS // (2 if kind == "cast" else 1))
        rows = _log(rng, 1, min(16384, numel))
        return {"kind": kind, "rows": rows, "cols": max(1, numel // rows), "in": rng.choice(["bf16", "bf16", "fp32"]),
                "out": rng.choice(["e4m3", "e5m2"])}
    if kind == "operands":
        rows, cols = _log(rng, 32, 16384), _log_multiple(rng, 256, 8192, 8)
        if rng.random() < 0.5:  # padded token counts beside ragged ones
            rows = -(-rows // 16) * 16
        return {"kind": kind, "rows": rows, "cols": cols, "in": rng.choice(["bf16", "bf16", "fp32"]), "out": rng.choice(["e4m3", "e5m2"])}
    if kind == "mx_cast":
        rows, cols = _log(rng, 1, 32768), _log_multiple(rng, 128, 8192, 32)
        return {"kind": kind, "rows": rows, "cols": cols, "in": rng.choice(["bf16", "bf16", "fp32"]), "out": rng.choice(["e4m3", "e4m3", "e5m2"])}
    if kind == "both":
        return {"kind": kind, "rows": _log(rng, 1024, 262144), "cols": _log_multiple(rng, 1024, 8192, 32), "out": rng.choice(["e4m3", "e5m2"])}
    if kind == "mx8_train":
        t, k, n = (_log_multiple(rng, 256, 8192, 32) for _ in range(3))
        return {"kind": kind, "tokens": t, "k": k, "n": n}
    k = _log_multiple(rng, 256, 8192, 16 if kind == "rowwise" else 32)
    n = _log_multiple(rng, 256, 16384, 8)
    # decode batches and prompts in equal shares
    tokens = _log(rng, 1, 128) if rng.random() < 0.5 else _log(rng, 128, 32768)
    tokens = max(1, min(tokens, int(MAX_LINEAR_FLOPS / (2.0 * k * n))))
    case = {"kind": kind, "tokens": tokens, "k": k, "n": n}
    if kind == "rowwise":
        case["bias"] = rng.random() < 0.5
    return case


# ---- inputs -----------------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _normal(g, rows, cols, dtype=torch.bfloat16, outliers=0.0, factor=100.0):
    """N(0,1) with a share of the elements multiplied by ``factor``; in row chunks, so that no full fp32 copy is held."""
    out = torch.empty(rows, cols, dtype=dtype, device=DEVICE)
    step = max(1, (1 << 27) // cols)
    for r in range(0, rows, step):
        x = torch.randn(min(step, rows - r), cols, generator=g, device=DEVICE)
        if outliers:
            x = torch.where(torch.rand(x.shape, generator=g, device=DEVICE) < outliers, x * factor, x)
        out[r:r + step] = x.to(dtype)
    return out


def _lognormal(g, rows, cols, dtype):
    """Random sign times lognormal magnitude (sigma 3), 1 % zeros: MX blocks over a wide exponent range."""
    mag = torch.exp(3.0 * torch.randn(rows, cols, generator=g, device=DEVICE))
    u = torch.rand(rows, cols, generator=g, device=DEVICE)
    mag = torch.where(u < 0.5, -mag, mag)
    return torch.where((u > 0.495) & (u < 0.505), torch.zeros((), device=DEVICE), mag).to(dtype)


def _train_inputs(g, case):
    t, k, n = case["tokens"], case["k"], case["n"]
    return _normal(g, t, k), _normal(g, n, k) * k ** -0.5, _normal(g, t, n)


def _linear_inputs(g, case):
    tokens, k, n = case["tokens"], case["k"], case["n"]
    x = _normal(g, tokens, k, outliers=1e-3)
    w = _normal(g, n, k) * k ** -0.5
    if case["kind"] == "rowwise":
        x *= torch.pow(10.0, torch.rand(tokens, 1, generator=g, device=DEVICE) * 2.0 - 1.0).to(torch.bfloat16)
    return x, w


def _bias(g, case):
    return torch.randn(case["n"], generator=g, device=DEVICE).to(torch.bfloat16) if case["bias"] else None


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind in ("cast", "operands"):
        s["out"] = FP8[case["out"]]
        s["x"] = _normal(g, case["rows"], case["cols"], DTYPES[case["in"]])
        # a scale from earlier steps: near fp8_max / amax, so that a few elements saturate now and then
        s["scale"] = (torch.finfo(s["out"]).max / (4.0 + torch.rand(1, generator=g, device=DEVICE))).to(torch.float32)
    elif kind == "tensorwise":
        s["out"] = FP8[case["out"]]
        s["x"] = _normal(g, case["rows"], case["cols"], DTYPES[case["in"]], outliers=1e-3)
    elif kind == "mx_cast":
        s["out"] = FP8[case["out"]]
        s["x"] = _lognormal(g, case["rows"], case["cols"], DTYPES[case["in"]])
    elif kind == "both":
        s["out"] = FP8[case["out"]]
        s["x"] = _normal(g, case["rows"], case["cols"], outliers=1e-4, factor=1000.0)
        s["quantizer"] = dtq.ShardedQuantizer()
    elif kind == "mx8_train":
        s["x"], s["w"], s["grad"] = _train_inputs(g, case)
    else:
        s["x"], w = _linear_inputs(g, case)
        if kind == "rowwise":
            payload, _, scale = dtq.dynamic_scaled_quant_rowwise(w, torch.float8_e4m3fn)
            s["w"], s["w_scale"] = payload.t(), scale.reciprocal().t()
            s["bias"] = _bias(g, case)
        elif kind == "mx8":
            payload, s["w_scale"] = dtq.mx_fp8_quantize_blocked(w)
            s["w"] = payload.t()
        else:
            payload, s["w_scale"] = dtq.mx_fp4_quantize(w, blocked=True)
            s["w"] = payload.t()
    return s


# ---- one pass ---------------------------------------------------------------------------------------------------

def run(s):
    kind, x = s["kind"], s["x"]
    if kind == "cast":
        return dtq.saturated_cast(x, s["scale"], s["out"])
    if kind == "operands":
        amax = dtq.amax(x)
        payload, payload_t = dtq.saturated_cast_dual(x, s["scale"], s["out"])
        return payload, payload_t, amax
    if kind == "tensorwise":
        return dtq.dynamic_scaled_quant_with_scale(x, s["out"])
    if kind == "mx_cast":
        return dtq.mx_fp8_quantize(x, ScalarType=s["out"])
    if kind == "both":
        return s["quantizer"].tensorwise_and_mx(x, s["out"])
    if kind == "rowwise":
        payload, _, scale = dtq.dynamic_scaled_quant_rowwise(x, torch.float8_e4m3fn)
        return dtq.sweep_mm(payload, s["w"], scale.reciprocal(), s["w_scale"], s["bias"], torch.bfloat16, False, 1, 1, 1, False, 1)
    if kind == "mx8":
        payload, scale = dtq.mx_fp8_quantize_blocked(x)
        return dtq.mx_fp8_bf16(payload, s["w"], scale, s["w_scale"])
    if kind == "mx4":
        payload, scale = dtq.mx_fp4_quantize(x, blocked=True)
        return dtq.mx_fp4_bf16(payload, s["w"], scale, s["w_scale"])
    # training step: y = x w^T, dx = g w, dw = g^T x, every product contracting along its operands' MX blocks
    px, sx, pxt, sxt = dtq.mx_fp8_quantize_dual(x, blocked=True)
    pw, sw, pwt, swt = dtq.mx_fp8_quantize_dual(s["w"], blocked=True)
    y = dtq.mx_fp8_bf16(px, pw.t(), sx, sw)
    pg, sg, pgt, sgt = dtq.mx_fp8_quantize_dual(s["grad"], blocked=True)
    dx = dtq.mx_fp8_bf16(pg, pwt.t(), sg, swt)
    dw = dtq.mx_fp8_bf16(pgt, pxt.t(), sgt, sxt)
    return y, dx, dw


# ---- the same in 64 bits ------------------------------------------------------------------------------------------

def _rowwise64(x):
    """Row-wise e4m3: the payload, and the fp32 factor that undoes its scale, both as fp64."""
    sd = 448.0 / (x.abs().amax(1, keepdim=True).double() + 1e-12)
    payload = (x.double() * sd).float().clamp(-448.0, 448.0).to(torch.float8_e4m3fn).double()
    return payload, sd.float().reciprocal().double()


def _mx64(x, fp4=False):
    """The values that the MX blocks of 32 along the last dimension stand for, as fp64."""
    rows, cols = x.shape
    v = x.reshape(rows, cols // 32, 32)
    mag = (v.contiguous().view(torch.int16).to(torch.int32) & 0x7FFF).amax(2, keepdim=True)
    exponent = (((mag + 0x7F) >> 7) - (2 if fp4 else 8)).clamp_min(0) - 127  # ceil(log2) less the format's largest exponent
    scale = torch.exp2(exponent.double())
    v = v.double() / scale
    if fp4:
        a = v.abs()
        step = torch.where(a < 2.0, 0.5, torch.where(a < 4.0, 1.0, 2.0))  # of e2m1: 0 .5 1 1.5 2 3 4 6
        v = (torch.round(v / step) * step).clamp(-6.0, 6.0)
    else:
        v = v.float().clamp(-448.0, 448.0).to(torch.float8_e4m3fn).double()
    return (v * scale).reshape(rows, cols)


def exact(case, seed):
    """The products of the quantized operands in fp64; the casts are bit patterns and have no such value."""
    kind = case["kind"]
    if kind not in ("rowwise", "mx8", "mx4", "mx8_train"):
        return None
    g = _gen(seed)
    if kind == "mx8_train":
        x, w, grad = _train_inputs(g, case)
        return (_mx64(x) @ _mx64(w).t(), _mx64(grad) @ _mx64(w.t()).t(), _mx64(grad.t()) @ _mx64(x.t()).t())
    x, w = _linear_inputs(g, case)
    if kind != "rowwise":
        return _mx64(x, kind == "mx4") @ _mx64(w, kind == "mx4").t()
    bias = _bias(g, case)
    (px, fx), (pw, fw) = _rowwise64(x), _rowwise64(w)
    y = (px @ pw.t()).mul_(fx).mul_(fw.t())
    return y if bias is None else y.add_(bias.double())


# ---- what a pass cannot do without, and how far two correct ones may differ ---------------------------------------

def work(case):
    """Bytes: inputs read once, outputs written once (what lies between two calls is not counted); flops: the products'."""
    kind = case["kind"]
    if kind in ("cast", "operands", "tensorwise", "mx_cast", "both"):
        elems = case["rows"] * case["cols"]
        size = 4 if case.get("in") == "fp32" else 2
        out = {"cast": 1.0, "operands": 2.0, "tensorwise": 1.0, "mx_cast": 1.0 + 1.0 / 32, "both": 2.0 + 1.0 / 32}[kind]
        return {"bytes": elems * (size + out), "flops": 0.0}
    t, k, n = case["tokens"], case["k"], case["n"]
    if kind == "mx8_train":
        return {"bytes": 2.0 * 2.0 * (t * k + n * k + t * n), "flops": 6.0 * t * k * n}
    w = {"rowwise": 1.0, "mx8": 1.0 + 1.0 / 32, "mx4": 0.5 + 1.0 / 32}[kind]
    return {"bytes": 2.0 * t * k + w * n * k + 2.0 * t * n, "flops": 2.0 * t * k * n}


def tolerance(case):
    if case["kind"] in ("cast", "operands", "tensorwise", "mx_cast", "both"):
        return "exact"  # the casts are defined bit for bit; a maximum does not depend on its order
    # The products accumulate in fp32 and are rounded once to bf16.  Against the same sums in fp64, and against fp32 sums
    # in four parts of K, up to 1e-4 (2-norm) and 0.0078 (one bf16 step) were seen, a few results in ten thousand rounding
    # the other way.
    return {"rel": 4e-4, "max": 0.016}

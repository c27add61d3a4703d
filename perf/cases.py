"""Cases that the library's speed is measured on: single Tile contractions through the kernel C ABI
(``plaidml_b200.kernels.Plan``, device pointers in, device pointers out) and whole EDSL programs through
``Executable.run`` (host buffers in, host buffers out).

A case is a dict of plain values; ``kind`` names the entry point:

  gemm       C = A * B with an optional bias / residual / ReLU epilogue or row maxima (``Plan("gemm")``)
  conv       NHWC convolution with bias and ReLU (``Plan("conv")``)
  depthwise  one filter per channel, a contraction that is no matrix product (``Plan("contract")``)
  weightgrad dW[k, n] += X[m, k] * dY[m, n], the backward direction of a dense layer (``Plan("contract")``)
  softmax    a softmax program over rows of scores, built with the op library (``Executable.run``)
  resnet     ResNet-50 v1.5 inference, bf16 with f32 accumulation (``Executable.run``)
"""

import functools
import math

import numpy as np
import torch

from plaidml_b200 import edsl, kernels, op, programs
from plaidml_b200.core import Buffer, DType, Program, f32_to_bf16_bits
from plaidml_b200.exec import Executable

TORCH = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16, "i8": torch.int8, "i32": torch.int32}
CODE = {"f32": kernels.F32, "bf16": kernels.BF16, "f16": kernels.F16, "i8": kernels.I8, "i32": kernels.I32}
BYTES = {"f32": 4, "bf16": 2, "f16": 2, "i8": 1, "i32": 4}


def gemm(m, n, k, dtype, out, batch=1, b_nk=False, bias=False, residual=False, relu=False, rowmax=False):
    return {"kind": "gemm", "m": m, "n": n, "k": k, "batch": batch, "dtype": dtype, "out": out, "b_nk": b_nk,
            "bias": bias, "residual": residual, "relu": relu, "rowmax": rowmax}


def conv(n, h, w, c, k, r, stride, dtype, out):
    return {"kind": "conv", "n": n, "h": h, "w": w, "c": c, "k": k, "r": r, "stride": stride, "dtype": dtype, "out": out}


def listed():
    return [
        # a classifier head on one image in the reference's own element type: the smallest call, latency counts
        {"name": "gemm_f32_head_1", **gemm(1, 1000, 2048, "f32", "f32", bias=True)},
        # the fp32 Tile GEMM of the benchmark
        {"name": "gemm_f32_1024", **gemm(1024, 1024, 1024, "f32", "f32")},
        # a dense layer on an odd number of rows, weights stored [n][k]
        {"name": "gemm_f32_ragged", **gemm(777, 2050, 515, "f32", "f32", b_nk=True, bias=True, relu=True)},
        # the int8 Tile GEMM of the benchmark
        {"name": "gemm_i8_4096", **gemm(4096, 4096, 4096, "i8", "i32")},
        # a 1x1 convolution at the end of a residual block: few rows, residual and ReLU
        {"name": "gemm_bf16_residual", **gemm(1568, 1000, 512, "bf16", "bf16", bias=True, residual=True, relu=True)},
        # attention scores with the row maxima that a softmax starts from, the batched GEMM of the benchmark
        {"name": "scores_rowmax", **gemm(512, 512, 64, "bf16", "f32", batch=1024, b_nk=True, rowmax=True)},
        # the convolution of the benchmark
        {"name": "conv_bf16_3x3", **conv(128, 56, 56, 64, 64, 3, 1, "bf16", "bf16")},
        # a 3x3 layer of an image network in the reference's own element type
        {"name": "conv_f32_3x3", **conv(8, 28, 28, 128, 128, 3, 1, "f32", "f32")},
        # a depthwise layer of a mobile image network
        {"name": "depthwise_f32", "kind": "depthwise", "n": 32, "h": 56, "w": 56, "c": 128, "r": 3, "stride": 1},
        # the weight gradient of a dense layer over a batch of 4096 rows
        {"name": "weightgrad_f32", "kind": "weightgrad", "m": 4096, "k": 512, "n": 512},
        # a small program of reductions and element-wise steps, end to end
        {"name": "softmax_program", "kind": "softmax", "rows": 512, "n": 1000},
        # a whole network, end to end
        {"name": "resnet50_b16", "kind": "resnet", "batch": 16},
    ]


def _log(rng, lo, hi, multiple=1):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(multiple, (v + multiple // 2) // multiple * multiple)


def draw(rng):
    kind = rng.choice(["f32", "f32", "i8", "bf16", "scores", "conv_bf16", "conv_f32", "depthwise", "weightgrad", "softmax", "resnet"])
    if kind == "f32":
        m, n, k = _log(rng, 1, 2048), _log(rng, 16, 4096), _log(rng, 64, 4096)
        while m * n * k > 1 << 32:
            k = max(64, k // 2)
        return gemm(m, n, k, "f32", "f32", b_nk=rng.random() < 0.5, bias=rng.random() < 0.5, relu=rng.random() < 0.3)
    if kind == "i8":
        m, n, k = _log(rng, 16, 4096), _log(rng, 16, 4096, 16), _log(rng, 128, 4096, 16)
        return gemm(m, n, k, "i8", "i32", b_nk=rng.random() < 0.5)
    if kind == "bf16":
        m, n, k = _log(rng, 16, 16384), _log(rng, 64, 2048, 8), _log(rng, 64, 2048, 8)
        residual = rng.random() < 0.5
        return gemm(m, n, k, rng.choice(["bf16", "bf16", "f16"]), "same", b_nk=rng.random() < 0.3, bias=True,
                    residual=residual, relu=rng.random() < 0.7)
    if kind == "scores":
        s = _log(rng, 100, 512, 4)
        return gemm(s, s, rng.choice([32, 64, 128]), "bf16", "f32", batch=_log(rng, 8, 512), b_nk=True, rowmax=True)
    if kind in ("conv_bf16", "conv_f32"):
        r, hw, stride = rng.choice([1, 3, 3, 5]), rng.choice([7, 14, 27, 28, 55, 56]), rng.choice([1, 1, 2])
        c, k = _log(rng, 32, 512, 8), _log(rng, 32, 512, 8)
        most = 1 << 34 if kind == "conv_bf16" else 1 << 32
        n = _log(rng, 1, 128 if kind == "conv_bf16" else 32)
        while n > 1 and n * hw * hw * c * k * r * r > most * stride * stride:
            n = (n + 1) // 2
        d = "bf16" if kind == "conv_bf16" else "f32"
        return conv(n, hw, hw + rng.choice([0, 1]), c, k, r, stride, d, d)
    if kind == "depthwise":
        hw = rng.choice([7, 14, 28, 56, 57, 112])
        c = _log(rng, 16, 960, rng.choice([1, 4, 8]))
        n = _log(rng, 1, 64)
        while n > 1 and n * hw * hw * c > 32 * 56 * 56 * 128:
            n = (n + 1) // 2
        return {"kind": "depthwise", "n": n, "h": hw, "w": hw, "c": c, "r": rng.choice([3, 3, 5]), "stride": rng.choice([1, 1, 2])}
    if kind == "weightgrad":
        m, k, n = _log(rng, 128, 8192), _log(rng, 32, 1024), _log(rng, 32, 1024)
        while m * k * n > 4096 * 512 * 512:
            m = m // 2
        return {"kind": "weightgrad", "m": m, "k": k, "n": n}
    if kind == "softmax":
        return {"kind": "softmax", "rows": _log(rng, 1, 1024), "n": _log(rng, 10, 2000)}
    return {"kind": "resnet", "batch": _log(rng, 1, 16)}


# ---------------------------------------------------------------------------------------- inputs


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _values(shape, dtype, seed, scale=1.0, uniform=False):
    g = _generator(seed)
    if dtype == "i8":
        return torch.randint(-128, 128, shape, dtype=torch.int8, device="cuda", generator=g)
    if uniform:
        x = torch.rand(shape, dtype=torch.float32, device="cuda", generator=g) * 2 - 1
    else:
        x = torch.randn(shape, dtype=torch.float32, device="cuda", generator=g) * scale
    return x.to(TORCH[dtype])


def _out_type(case):
    return case["dtype"] if case["out"] == "same" else case["out"]


def _gemm_inputs(case, seed):
    m, n, k, b, dt = case["m"], case["n"], case["k"], case["batch"], case["dtype"]
    # fp32: uniform in [-1, 1) like the benchmark; 16 bits: activations of unit variance, weights scaled to keep it
    wide = dt == "f32" or case["rowmax"]
    x = {"a": _values((b, m, k), dt, 10 * seed + 1, uniform=dt == "f32"),
         "b": _values((b, n, k) if case["b_nk"] else (b, k, n), dt, 10 * seed + 2, 1.0 if wide else k ** -0.5, uniform=dt == "f32")}
    x["bias"] = _values((n,), "f32", 10 * seed + 3) if case["bias"] else None
    x["residual"] = _values((b, m, n), _out_type(case), 10 * seed + 4) if case["residual"] else None
    return x


def _conv_geometry(case):
    pad = (case["r"] - 1) // 2
    p = (case["h"] + 2 * pad - case["r"]) // case["stride"] + 1
    q = (case["w"] + 2 * pad - case["r"]) // case["stride"] + 1
    return pad, p, q


def _conv_inputs(case, seed):
    c, k, r = case["c"], case["k"], case["r"]
    return {"x": _values((case["n"], case["h"], case["w"], c), "f32", 10 * seed + 1).abs().to(TORCH[case["dtype"]]),
            "f": _values((r, r, c, k), case["dtype"], 10 * seed + 2, (2.0 / (r * r * c)) ** 0.5),
            "bias": _values((k,), "f32", 10 * seed + 3, 0.1)}


def _depthwise_inputs(case, seed):
    c, r = case["c"], case["r"]
    return {"x": _values((case["n"], case["h"], case["w"], c), "f32", 10 * seed + 1),
            "f": _values((r, r, c), "f32", 10 * seed + 2, 1.0 / r)}


def _weightgrad_inputs(case, seed):
    return {"x": _values((case["m"], case["k"]), "f32", 10 * seed + 1),
            "dy": _values((case["m"], case["n"]), "f32", 10 * seed + 2)}


def _softmax_inputs(case, seed):
    g = np.random.Generator(np.random.PCG64(int(seed)))
    return (g.standard_normal((case["rows"], case["n"]), dtype=np.float32) * np.float32(3.0))


@functools.lru_cache(maxsize=1)
def _resnet_weights():
    return programs.resnet50_weights()


# ---------------------------------------------------------------------------------------- prepare


def _epilogue(case):
    flags = 0
    for name, flag in (("bias", kernels.EPI_BIAS), ("residual", kernels.EPI_RESIDUAL), ("relu", kernels.EPI_RELU),
                       ("rowmax", kernels.EPI_ROWMAX)):
        flags |= flag if case[name] else 0
    return flags


def _prepare_gemm(case, seed):
    m, n, k, b = case["m"], case["n"], case["k"], case["batch"]
    s = _gemm_inputs(case, seed)
    out = _out_type(case)
    d = kernels.GemmDesc()
    d.in_dtype, d.out_dtype = CODE[case["dtype"]], CODE[out]
    d.m, d.n, d.k, d.batch = m, n, k, b
    d.lda, d.ldb, d.ldc = k, k if case["b_nk"] else n, n
    if b > 1:
        d.stride_a, d.stride_b, d.stride_c = m * k, n * k, m * n
    d.b_is_nk = int(case["b_nk"])
    d.epilogue = _epilogue(case)
    d.ldr, d.stride_r = d.ldc, d.stride_c
    s["plan"] = kernels.Plan("gemm", d)
    s["c"] = torch.empty((b, m, n), dtype=TORCH[out], device="cuda")
    s["rowmax"] = torch.empty((b, m), dtype=torch.float32, device="cuda") if case["rowmax"] else None
    return s


def _prepare_conv(case, seed):
    pad, p, q = _conv_geometry(case)
    s = _conv_inputs(case, seed)
    d = kernels.ConvDesc()
    d.in_dtype, d.out_dtype = CODE[case["dtype"]], CODE[case["out"]]
    d.n, d.h, d.w, d.c = case["n"], case["h"], case["w"], case["c"]
    d.r = d.s = case["r"]
    d.k, d.p, d.q = case["k"], p, q
    d.stride_h = d.stride_w = case["stride"]
    d.pad_h = d.pad_w = pad
    d.dil_h = d.dil_w = 1
    d.epilogue = kernels.EPI_BIAS | kernels.EPI_RELU
    s["plan"] = kernels.Plan("conv", d)
    s["plan"].set_filter(s["f"].data_ptr(), CODE[case["dtype"]], torch.cuda.current_stream().cuda_stream)
    s["y"] = torch.empty((case["n"], p, q, case["k"]), dtype=TORCH[case["out"]], device="cuda")
    return s


def _contract(out, sources, ranges):
    d = kernels.ContractDesc()
    d.agg, d.combo = kernels.AGG_SUM, kernels.COMBO_MUL
    d.n_idx, d.n_src = len(ranges), len(sources)
    for i, r in enumerate(ranges):
        d.range[i] = r
    d.out = out
    for i, s in enumerate(sources):
        d.src[i] = s
    return kernels.Plan("contract", d)


def _prepare_depthwise(case, seed):
    pad, p, q = _conv_geometry(case)
    n, h, w, c, r, st = case["n"], case["h"], case["w"], case["c"], case["r"], case["stride"]
    s = _depthwise_inputs(case, seed)
    # O[n, y, x, c] += I[n, st*y + i - pad, st*x + j - pad, c] * F[i, j, c], taps outside the image skipped
    N, Y, X, C, I, J = range(6)
    s["plan"] = _contract(
        kernels.make_access(kernels.F32, [n, p, q, c], [{N: 1}, {Y: 1}, {X: 1}, {C: 1}]),
        [kernels.make_access(kernels.F32, [n, h, w, c], [{N: 1}, {Y: st, I: 1}, {X: st, J: 1}, {C: 1}], offs=[0, -pad, -pad, 0]),
         kernels.make_access(kernels.F32, [r, r, c], [{I: 1}, {J: 1}, {C: 1}])],
        [n, p, q, c, r, r])
    s["y"] = torch.empty((n, p, q, c), dtype=torch.float32, device="cuda")
    return s


def _prepare_weightgrad(case, seed):
    m, k, n = case["m"], case["k"], case["n"]
    s = _weightgrad_inputs(case, seed)
    K, N, M = range(3)
    s["plan"] = _contract(kernels.make_access(kernels.F32, [k, n], [{K: 1}, {N: 1}]),
                          [kernels.make_access(kernels.F32, [m, k], [{M: 1}, {K: 1}]),
                           kernels.make_access(kernels.F32, [m, n], [{M: 1}, {N: 1}])], [k, n, m])
    s["dw"] = torch.empty((k, n), dtype=torch.float32, device="cuda")
    return s


def _prepare_program(program, inputs):
    program.compile("cuda")
    s = {"program": program, "exe": Executable(program, "cuda.0"),
         "in": [Buffer(shape) for shape in program.inputs], "out": [Buffer(shape) for shape in program.outputs]}
    for buf, x in zip(s["in"], inputs):
        buf.copy_from_ndarray(x)
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "gemm":
        s = _prepare_gemm(case, seed)
    elif kind == "conv":
        s = _prepare_conv(case, seed)
    elif kind == "depthwise":
        s = _prepare_depthwise(case, seed)
    elif kind == "weightgrad":
        s = _prepare_weightgrad(case, seed)
    elif kind == "softmax":
        S = edsl.Placeholder(DType.FLOAT32, [case["rows"], case["n"]], name="scores")
        s = _prepare_program(Program("softmax", [S], [op.softmax(S, axis=1)]), [_softmax_inputs(case, seed)])
    else:
        program, _ = programs.resnet50(case["batch"], _resnet_weights())
        g = np.random.Generator(np.random.PCG64(int(seed)))
        s = _prepare_program(program, [f32_to_bf16_bits(g.random((case["batch"], 224, 224, 3), dtype=np.float32))])
    s["kind"] = kind
    return s


# ---------------------------------------------------------------------------------------- run


def _ptr(t):
    return None if t is None else t.data_ptr()


def run(s):
    kind = s["kind"]
    if kind in ("softmax", "resnet"):
        s["exe"].run(s["in"], s["out"])
        return [buf.as_ndarray() for buf in s["out"]]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "gemm":
        s["plan"].gemm(s["a"].data_ptr(), s["b"].data_ptr(), s["c"].data_ptr(), _ptr(s["bias"]), _ptr(s["residual"]),
                       _ptr(s["rowmax"]), stream)
        return [s["c"]] if s["rowmax"] is None else [s["c"], s["rowmax"]]
    if kind == "conv":
        s["plan"].conv(s["x"].data_ptr(), s["y"].data_ptr(), s["bias"].data_ptr(), None, stream)
        return [s["y"]]
    if kind == "depthwise":
        s["plan"].contract([s["x"].data_ptr(), s["f"].data_ptr()], s["y"].data_ptr(), stream=stream)
        return [s["y"]]
    s["plan"].contract([s["x"].data_ptr(), s["dy"].data_ptr()], s["dw"].data_ptr(), stream=stream)
    return [s["dw"]]


# ---------------------------------------------------------------------------------------- work, tolerance, exact


def work(case):
    kind = case["kind"]
    if kind == "gemm":
        m, n, k, b = case["m"], case["n"], case["k"], case["batch"]
        e, o = BYTES[case["dtype"]], BYTES[_out_type(case)]
        nbytes = b * (m * k + n * k) * e + b * m * n * o * (2 if case["residual"] else 1)
        nbytes += (4 * n if case["bias"] else 0) + (4 * b * m if case["rowmax"] else 0)
        return {"bytes": nbytes, "flops": 2 * b * m * n * k}
    if kind in ("conv", "depthwise"):
        _, p, q = _conv_geometry(case)
        n, h, w, c, r = case["n"], case["h"], case["w"], case["c"], case["r"]
        if kind == "depthwise":
            return {"bytes": 4 * (n * h * w * c + n * p * q * c + r * r * c), "flops": 2 * n * p * q * c * r * r}
        k, e = case["k"], BYTES[case["dtype"]]
        # a strided 1x1 layer reads only the pixels it keeps
        read = n * p * q * c if r == 1 else n * h * w * c
        return {"bytes": e * (read + r * r * c * k) + BYTES[case["out"]] * n * p * q * k + 4 * k,
                "flops": 2 * n * p * q * c * k * r * r}
    if kind == "weightgrad":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 4 * (m * k + m * n + k * n), "flops": 2 * m * k * n}
    if kind == "softmax":
        return {"bytes": 8 * case["rows"] * case["n"], "flops": 5 * case["rows"] * case["n"]}
    return {"bytes": case["batch"] * (224 * 224 * 3 * 2 + 4000) + 51e6, "flops": case["batch"] * programs.RESNET50_GFLOP_PER_IMAGE * 1e9}


def tolerance(case):
    kind = case["kind"]
    if kind in ("gemm", "conv"):
        if case["dtype"] == "i8":
            return "exact"
        if case["dtype"] == "f32":
            # products of split operands: the tensor core's accumulator truncates, and the error against 64 bits
            # was measured to grow with the length of the sum (7e-9 per term: 7.2e-6 at 1024, 1.4e-5 at 2048)
            return {"rel": max(1e-5, 3e-8 * (case["k"] if kind == "gemm" else case["r"] ** 2 * case["c"]))}
        return {"rel": 1e-5} if _out_type(case) == "f32" else {"rel": 1e-2 if _out_type(case) == "bf16" else 2e-3}
    # sums of a few thousand 32-bit products, or a handful of them
    if kind in ("weightgrad", "depthwise", "softmax"):
        return {"rel": 1e-5}
    # every layer rounds to bf16: 53 of them
    return {"rel": 2e-2}


def exact(case, seed):
    kind = case["kind"]
    f64 = torch.float64
    if kind == "gemm":
        if case["dtype"] == "i8":
            return None
        x = _gemm_inputs(case, seed)
        y = x["a"].to(f64) @ (x["b"].to(f64).transpose(1, 2) if case["b_nk"] else x["b"].to(f64))
        if case["bias"]:
            y = y + x["bias"].to(f64)
        if case["residual"]:
            y = y + x["residual"].to(f64)
        if case["relu"]:
            y = y.clamp_min(0)
        return [y, y.amax(dim=2)] if case["rowmax"] else [y]
    if kind == "conv":
        x = _conv_inputs(case, seed)
        pad, p, q = _conv_geometry(case)
        st, r = case["stride"], case["r"]
        xp = torch.nn.functional.pad(x["x"].to(f64), (0, 0, pad, pad, pad, pad))
        f = x["f"].to(f64)
        y = x["bias"].to(f64).expand(case["n"], p, q, case["k"]).clone()
        for i in range(r):
            for j in range(r):
                y += xp[:, i:i + st * (p - 1) + 1:st, j:j + st * (q - 1) + 1:st, :] @ f[i, j]
        return [y.clamp_min(0)]
    if kind == "depthwise":
        x = _depthwise_inputs(case, seed)
        pad, p, q = _conv_geometry(case)
        st, r = case["stride"], case["r"]
        xp = torch.nn.functional.pad(x["x"].to(f64), (0, 0, pad, pad, pad, pad))
        y = torch.zeros((case["n"], p, q, case["c"]), dtype=f64, device="cuda")
        for i in range(r):
            for j in range(r):
                y += xp[:, i:i + st * (p - 1) + 1:st, j:j + st * (q - 1) + 1:st, :] * x["f"][i, j].to(f64)
        return [y]
    if kind == "weightgrad":
        x = _weightgrad_inputs(case, seed)
        return [x["x"].to(f64).t() @ x["dy"].to(f64)]
    if kind == "softmax":
        x = _softmax_inputs(case, seed).astype(np.float64)
        e = np.exp(x - x.max(axis=1, keepdims=True))
        return [e / e.sum(axis=1, keepdims=True)]
    return None  # 53 layers that each round to 16 bits

"""The work that programs give this framework, as cases that can be timed.

A case is one pass through the public entry points of hecbench_b200: a mat-vec of a
decode step, the two products of an MLP block, a batched product of a prefill or of
many requests at once, the quantization of activations, or the conversion of
weights.  listed() holds fixed cases, draw() makes further ones over the same ranges.
"""
import math

import torch

import hecbench_b200 as hq

#: bytes of the largest listed case; drawn cases stay below it
LARGEST_BYTES = 370e6

DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32}


def listed():
    return [
        # key / value projection of an 8B model with grouped heads: the smallest
        # layer of a decode step, latency and host time count
        {"name": "gemv nf4 1024x4096", "path": "gemv", "format": "nf4", "outputs": 1024, "inputs": 4096},
        # the run size of the 3-bit mat-vec benchmark, fp32 activations
        {"name": "gemv q3 f32 4096x4096", "path": "gemv", "format": "q3_f32", "outputs": 4096, "inputs": 4096},
        # the same with fp16 activations on the MLP expansion of a 175B model
        {"name": "gemv q3 f16 49152x12288", "path": "gemv", "format": "q3_f16", "outputs": 49152, "inputs": 12288},
        # the uniform 4-bit mat-vec with one scale and zero point per tensor
        {"name": "gemv int4 8192x8192", "path": "gemv", "format": "int4", "outputs": 8192, "inputs": 8192},
        # MLP block of an 8B model at batch 1: RMSNorm, up / gate product and SwiGLU
        # in one call, then the down projection
        {"name": "mlp nf4 4096-14336", "path": "mlp", "format": "nf4", "hidden": 4096, "inner": 14336, "act": "swiglu"},
        # binary-coding mat-vec, a square layer of a 175B model at three bit planes
        {"name": "lutgemm 12288x12288", "path": "lutgemm", "outputs": 12288, "inputs": 12288, "planes": 3, "group": 128, "bias": True},
        # additive-codebook mat-vec, attention projection of a 7B model
        {"name": "aqlm 1x16 4096x4096", "path": "aqlm", "format": "1x16", "outputs": 4096, "inputs": 4096},
        # up / gate product of a 70B model for 64 tokens
        {"name": "qgemm q3 64x8192x28672", "path": "qgemm", "format": "q3", "tokens": 64, "inputs": 8192, "outputs": 28672},
        # its down projection for a batch that fills no tile
        {"name": "qgemm nf4 37x28672x8192", "path": "qgemm", "format": "nf4", "tokens": 37, "inputs": 28672, "outputs": 8192},
        # per-token int8 quantization of a prefill's activations, rows of odd length
        {"name": "int8 4096x5137", "path": "int8", "tokens": 4096, "hidden": 5137, "dtype": "float16", "form": "dynamic"},
        # a tensor packed to MXFP4 and read back
        {"name": "mxfp4 bf16 32Mi", "path": "codec", "format": "mxfp4", "values": 1 << 25, "dtype": "bfloat16"},
        # a layer converted for the binary-coding mat-vec: the largest case
        {"name": "pack bcq 12288x12288", "path": "pack", "format": "bcq", "inputs": 12288, "outputs": 12288, "dtype": "float16", "planes": 3},
    ]


def _size(rng, low, high, step=1):
    """A multiple of step, spread over the logarithm of [low, high]."""
    v = math.exp(rng.uniform(math.log(low), math.log(high)))
    return min(high // step * step, max(-(-low // step) * step, round(v / step) * step))


def draw(rng):
    while True:
        case = _draw(rng)
        if work(case)["bytes"] <= LARGEST_BYTES:
            return case


def _draw(rng):
    path = rng.choice(["gemv", "gemv", "mlp", "lutgemm", "aqlm", "qgemm", "qgemm", "int8", "codec", "pack"])
    if path == "gemv":
        fmt = rng.choice(["nf4", "q3_f32", "q3_f16", "int8", "int4"])
        # the 3-bit rows are a whole number of 16-byte pieces; the others take any count of rows
        return {"path": path, "format": fmt, "outputs": _size(rng, 512, 49152, 4 if fmt.startswith("q3") else 1),
                "inputs": _size(rng, 1024, 16384, 64)}
    if path == "mlp":
        return {"path": path, "format": rng.choice(["nf4", "nf4", "int8", "int4"]), "hidden": _size(rng, 1024, 8192, 64),
                "inner": _size(rng, 2816, 28672, 64), "act": rng.choice(["swiglu", "geglu"])}
    if path == "lutgemm":
        group = rng.choice([64, 128, 128])
        return {"path": path, "outputs": _size(rng, 1024, 12288, 4), "inputs": _size(rng, 1024, 12288, group),
                "planes": rng.choice([2, 3, 3, 4]), "group": group, "bias": rng.random() < 0.75}
    if path == "aqlm":
        return {"path": path, "format": rng.choice(["1x16", "2x8"]), "outputs": _size(rng, 1024, 14336),
                "inputs": _size(rng, 1024, 14336, 64)}
    if path == "qgemm":
        return {"path": path, "format": rng.choice(["q3", "nf4"]), "tokens": rng.randint(2, 128),
                "inputs": _size(rng, 2048, 28672, 128), "outputs": _size(rng, 1024, 28672, 128)}
    if path == "int8":
        return {"path": path, "tokens": _size(rng, 1, 8192), "hidden": _size(rng, 1024, 16384),
                "dtype": rng.choice(["float16", "bfloat16", "float32"]), "form": rng.choice(["static", "dynamic", "dynamic", "dynamic_azp"])}
    if path == "codec":
        fmt = rng.choice(["mxfp4", "nf4"])
        return {"path": path, "format": fmt, "values": _size(rng, 1 << 20, 1 << 26, 64), "dtype": rng.choice(["float16", "bfloat16"])}
    fmt = rng.choice(["bcq", "q3"])
    case = {"path": path, "format": fmt, "inputs": _size(rng, 1024, 12288, 128), "outputs": _size(rng, 1024, 12288, 8),
            "dtype": rng.choice(["float16", "bfloat16", "float32"])}
    return dict(case, planes=rng.choice([2, 3, 4])) if fmt == "bcq" else case


def _floats(g, shape, dtype=torch.float16, std=1.0):
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype).mul_(std)


def _between(g, low, high, shape, dtype=torch.float32):
    return torch.rand(shape, generator=g, device="cuda").mul_(high - low).add_(low).to(dtype)


def _bytes(g, shape):
    """Uniform packed codes: bytes, whatever the format."""
    return torch.randint(0, 256, shape, generator=g, device="cuda", dtype=torch.uint8)


def _words(g, shape):
    return torch.randint(-2**31, 2**31, shape, generator=g, device="cuda", dtype=torch.int64).to(torch.int32)


def _levels(g):
    """16 ascending levels with exact -1, 0 and 1, like a normal-float table."""
    side = torch.cat([_between(g, 0.05, 0.95, 6).neg(), _between(g, 0.05, 0.95, 7),
                      torch.tensor([-1.0, 0.0, 1.0], device="cuda")])
    return side.sort().values


def _rows(g, fmt, outputs, inputs):
    """Weights in a row-major format, with their parameters; products of unit inputs are of order one."""
    if fmt == "nf4":
        absmax = _between(g, 0.5, 2.0, outputs * inputs // 64).div_(math.sqrt(inputs))
        return {"mat": _bytes(g, (outputs, inputs // 2)), "absmax": absmax, "lut16": _levels(g)}
    if fmt == "int8":
        return {"mat": _bytes(g, (outputs, inputs)).view(torch.int8), "scale": 1 / (74 * math.sqrt(inputs)), "zero_point": 1.0}
    return {"mat": _bytes(g, (outputs, inputs // 2)), "scale": 1 / (4.6 * math.sqrt(inputs)), "zero_point": 7.5}


def _multiply(fmt, w, x, outputs, inputs):
    if fmt == "nf4":
        return hq.gemv_nf4(x, w["mat"], w["absmax"], w["lut16"], outputs, inputs, 64, weights_resident=True)
    if fmt == "int8":
        return hq.gemv_int8_quantized(w["mat"], x, w["scale"], w["zero_point"])
    return hq.gemv_int4_quantized(w["mat"], x, w["scale"], w["zero_point"])


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    s = dict(case)
    path, fmt = case["path"], case.get("format")
    n, k = case.get("outputs"), case.get("inputs")
    if path == "gemv" and fmt in ("q3_f32", "q3_f16"):
        scales = _between(g, 0.001, 0.01, n)
        s.update(vec=_floats(g, k, torch.float16 if fmt == "q3_f16" else torch.float32), mat=_words(g, (k * 3 // 32, n)), scales=scales,
                 zeros=scales * torch.randint(0, 8, (n,), generator=g, device="cuda"), out=torch.zeros(n, device="cuda"))
    elif path == "gemv":
        s.update(vec=_floats(g, k), weights=_rows(g, fmt, n, k))
    elif path == "mlp":
        h, m = case["hidden"], case["inner"]
        s.update(x=_floats(g, h, std=2.0), gamma=_between(g, 0.5, 1.5, h, torch.float16), up=_rows(g, fmt, 2 * m, h), down=_rows(g, fmt, h, m))
    elif path == "lutgemm":
        groups = k // case["group"]
        s.update(x=_floats(g, k), out=torch.empty(n, dtype=torch.float16, device="cuda"), weights=hq.nQWeight_fp16(
            _words(g, (k // 32, case["planes"], n)), _between(g, 0.001, 0.05, (groups, case["planes"], n)), k, n, case["planes"], False,
            groups, _floats(g, (groups, n), torch.float32, 0.01) if case["bias"] else None))
    elif path == "aqlm":
        s.update(x=_floats(g, k), out=torch.empty(n, dtype=torch.float16, device="cuda"), scales=_between(g, 0.5, 2.0, n, torch.float16))
        if fmt == "1x16":
            s.update(codes=_bytes(g, (n, k // 4)).view(torch.int16), books=_floats(g, (1, 65536, 8), std=0.02))
        else:
            s.update(codes=_bytes(g, (n, k // 8, 2)), books=_floats(g, (2, 256, 8), std=0.02))
    elif path == "qgemm" and fmt == "q3":
        scales = _between(g, 0.001, 0.01, (k // 128, n))
        zeros = scales * torch.randint(0, 8, (k // 128, n), generator=g, device="cuda")
        s.update(x=_floats(g, (case["tokens"], k)), mat=_words(g, (k * 3 // 32, n)), scales=scales.half(), zeros=zeros.half())
    elif path == "qgemm":
        s.update(x=_floats(g, (case["tokens"], k)), **_rows(g, "nf4", n, k))
    elif path == "int8":
        x = _floats(g, (case["tokens"], case["hidden"]), torch.float32).mul_(_between(g, 0.5, 4.0, (case["tokens"], 1)))
        s.update(x=x.to(DTYPES[case["dtype"]]), out=torch.empty(x.shape, dtype=torch.int8, device="cuda"), scale=4.0 / 32,
                 scales=torch.empty(len(x), device="cuda"), azp=torch.empty(len(x), dtype=torch.int32, device="cuda"))
    elif path == "codec":
        s.update(values=_floats(g, case["values"], DTYPES[case["dtype"]], 0.05), lut16=_levels(g))
    else:
        s.update(values=_floats(g, (k, n), DTYPES[case["dtype"]], 0.05))
    return s


def run(s):
    path, fmt = s["path"], s.get("format")
    if path == "gemv" and fmt in ("q3_f32", "q3_f16"):
        s["out"].zero_()  # the products are added to what is there
        call = hq.vecquant3matmul if fmt == "q3_f32" else hq.vecquant3matmul_faster
        call(s["vec"], s["mat"], s["out"], s["scales"], s["zeros"], s["inputs"] * 3 // 32, s["outputs"])
        return s["out"]
    if path == "gemv":
        return _multiply(fmt, s["weights"], s["vec"], s["outputs"], s["inputs"])
    if path == "mlp":
        h, m, w = s["hidden"], s["inner"], dict(s["up"])
        act = hq.ACT_SWIGLU if s["act"] == "swiglu" else hq.ACT_GEGLU
        inner = hq.gemv_fused(fmt, s["x"], w.pop("mat"), m, gamma=s["gamma"], act=act, weights_resident=True, **w)
        return inner, _multiply(fmt, s["down"], inner, h, m)
    if path == "lutgemm":
        hq.matmul(s["out"], s["x"], s["weights"])
        return s["out"]
    if path == "aqlm" and fmt == "1x16":
        n = s["outputs"]
        hq.code1x16_matvec(s["codes"], s["x"], s["out"], s["books"], n, s["inputs"], [n, n, n, n], 65536, s["scales"])
        return s["out"]
    if path == "aqlm":
        hq.code2x8_matvec(s["codes"], s["x"], s["out"], s["books"], s["outputs"], s["inputs"], s["scales"])
        return s["out"]
    if path == "qgemm" and fmt == "q3":
        return hq.qgemm_q3(s["x"], s["mat"], s["scales"], s["zeros"], s["outputs"], s["inputs"])
    if path == "qgemm":
        return hq.qgemm_nf4(s["x"], s["mat"], s["absmax"], s["lut16"], s["outputs"], s["inputs"])
    if path == "int8":
        if s["form"] == "static":
            hq.static_scaled_int8_quant(s["out"], s["x"], s["hidden"], s["tokens"], s["scale"])
            return s["out"]
        azp = s["azp"] if s["form"] == "dynamic_azp" else None
        hq.dynamic_scaled_int8_quant(s["out"], s["x"], s["hidden"], s["tokens"], s["scales"], azp)
        return s["out"], s["scales"], azp
    if path == "codec" and fmt == "mxfp4":
        codes, scales = hq.mxfp4_quantize(s["values"])
        return codes, scales, hq.mxfp4_dequantize(codes, scales, s["values"].dtype)
    if path == "codec":
        codes, absmax = hq.quantize_nf4(s["values"], s["lut16"])
        return codes, absmax, hq.dequantize_nf4(codes, absmax, s["lut16"], s["values"].numel())
    if fmt == "bcq":
        return hq.quantize_bcq(s["values"], s["planes"])
    return hq.quantize_q3(s["values"])


def _weight_bytes(fmt, outputs, inputs):
    per_value = {"nf4": 0.5 + 4 / 64, "q3_f32": 0.375, "q3_f16": 0.375, "int8": 1.0, "int4": 0.5}[fmt]
    return outputs * inputs * per_value + (8 * outputs if fmt.startswith("q3") else 0)


def work(case):
    path, fmt = case["path"], case.get("format")
    n, k = case.get("outputs", 0), case.get("inputs", 0)
    if path == "gemv":
        wide = {"q3_f32": (4, 4), "q3_f16": (2, 4)}.get(fmt, (2, 2))
        return {"bytes": _weight_bytes(fmt, n, k) + wide[0] * k + wide[1] * n, "flops": 2 * n * k}
    if path == "mlp":
        h, m = case["hidden"], case["inner"]
        return {"bytes": _weight_bytes(fmt, 2 * m, h) + _weight_bytes(fmt, h, m) + 4 * h + 2 * m + 2 * h, "flops": 6 * h * m}
    if path == "lutgemm":
        planes = case["planes"]
        return {"bytes": n * k * planes / 8 + n * k / case["group"] * 2 * (planes + case["bias"]) + 2 * n + 2 * k, "flops": 2 * n * k}
    if path == "aqlm":
        return {"bytes": n * k / 4 + 4 * n + 2 * k + (65536 if fmt == "1x16" else 512) * 16, "flops": 2 * n * k}
    if path == "qgemm":
        weights = n * k * 3 / 8 + 4 * n * k / 128 if fmt == "q3" else _weight_bytes("nf4", n, k)
        return {"bytes": weights + 2 * case["tokens"] * (n + k), "flops": 2 * case["tokens"] * n * k}
    if path == "int8":
        values = case["tokens"] * case["hidden"]
        params = {"static": 0, "dynamic": 4, "dynamic_azp": 8}[case["form"]]
        return {"bytes": values * (DTYPES[case["dtype"]].itemsize + 1) + params * case["tokens"], "flops": values}
    size = DTYPES[case["dtype"]].itemsize
    if path == "codec":
        # values in, packed form out, values out
        return {"bytes": case["values"] * (2 * size + 0.5 + (1 / 32 if fmt == "mxfp4" else 4 / 64)), "flops": 2 * case["values"]}
    if fmt == "bcq":
        planes = case["planes"]
        return {"bytes": n * k * (size + planes / 8 + 2 * (planes + 1) / 128), "flops": 2 * n * k * planes}
    return {"bytes": n * k * (size + 0.375) + 8 * n, "flops": 3 * n * k}


def tolerance(case):
    path, fmt = case["path"], case.get("format")
    if path in ("int8", "codec", "pack"):
        return "exact"
    if fmt == "q3_f32":
        return {"rel": 1e-5}
    # fp16 results of fp32 sums; the mat-vecs form short partial sums in fp16
    if path in ("lutgemm", "aqlm", "qgemm"):
        return {"rel": 1e-3}
    return {"rel": 3e-3} if path == "mlp" else {"rel": 2e-3}

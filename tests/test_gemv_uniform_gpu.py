"""gemv (uniform int8 / int4 weight-only mat-vec, plus the fp16 baseline) on the
GPU through the mirrored launchers: against the fp64 CPU oracle, which restates
the reference's own device-side checks (gemv-cuda/gemv.cu:83-141), and against
the reference's CUDA kernels run beside ours on the same buffers with the
reference launch shapes.  Inputs are drawn like the reference's
(simple_tensor.h:63-87)."""
import ctypes as C

import numpy as np
import pytest

from hecbench_b200 import synth
from conftest import to_dev
import refgpu

pytestmark = pytest.mark.gpu
TOL_F16 = 1e-2


def _run(hq, bits, mat, vec, scale, zp, dev):
    dm, dv = to_dev(mat, dev), to_dev(vec, dev)
    if bits == 16:
        return hq.gemv_fp16(dm, dv)
    if bits == 8:
        return hq.gemv_int8_quantized(dm, dv, scale, zp)
    return hq.gemv_int4_quantized(dm, dv, scale, zp)


@pytest.mark.parametrize("bits", [8, 4, 16])
@pytest.mark.parametrize("rows,n,scale,zp", [
    (512, 512, 0.0625, 0.01),      # the reference driver's defaults (main.cu:31-36)
    (4096, 4096, 0.0625, 0.01),
    (1000, 2048, 0.0123, 3.0),     # rows != n, a zero point that matters
    (37, 32, 1.0, 0.0),            # one chunk per row, fewer rows than warps
    (3, 24576, 0.001, 7.5),        # long rows, fewer rows than a CTA has warps
    (20, 65536, 0.001, 0.5),       # rows that leave room for one CTA per SM only
    (8192, 1056, 0.5, -2.0)])      # a row that is not a whole number of warp steps
def test_gemv_uniform_against_oracle(hq, oracle, dev, bits, rows, n, scale, zp):
    mat, vec = synth.gemv_uniform_case(rows, n, bits, seed=rows + n + bits)
    y = _run(hq, bits, mat, vec, scale, zp, dev)
    ref = oracle.gemv_uniform_f64(mat, vec, bits, scale, zp)
    assert y.shape == (rows,)
    assert oracle.rel_err(y.cpu().numpy().astype(np.float64), ref) < TOL_F16


@pytest.mark.parametrize("bits", [8, 4, 16])
@pytest.mark.parametrize("extra,n", [(-33, 64), (-1, 4096), (0, 1024), (1, 1024), (0, 60032)])
def test_gemv_uniform_around_one_cta_per_sm(hq, oracle, dev, bits, extra, n):
    """32 rows per CTA: one CTA per SM less one, exactly one, one more; rows whose inputs
    alone take more than half an SM's shared memory.  Each call reads the output of the
    one before as part of its input."""
    import torch
    rows = 32 * torch.cuda.get_device_properties(dev).multi_processor_count + extra
    mat, vec = synth.gemv_uniform_case(rows, n, bits, seed=rows + n + bits)
    dm, dv = to_dev(mat, dev), to_dev(vec, dev)
    call = {16: lambda v: hq.gemv_fp16(dm, v), 8: lambda v: hq.gemv_int8_quantized(dm, v, 2 ** -9, 0.5),
            4: lambda v: hq.gemv_int4_quantized(dm, v, 2 ** -9, 0.5)}[bits]
    chain = [dv]
    for _ in range(4):
        y = call(chain[-1])
        chain.append(torch.cat([y[:32] * 2 ** -12, chain[-1][32:]]))
    torch.cuda.synchronize()
    for a, b in zip(chain, chain[1:]):
        ref = oracle.gemv_uniform_f64(mat, a.cpu().numpy(), bits, 2 ** -9, 0.5)
        got = call(a).cpu().numpy().astype(np.float64)
        assert oracle.rel_err(got, ref) < TOL_F16
        assert torch.equal(b[:32], torch.from_numpy(got[:32]).to(torch.float16).to(dev) * 2 ** -12)


def test_gemv_uniform_signed_inputs_and_extreme_codes(hq, oracle, dev):
    """Inputs of both signs (the reference only draws U(0,1)), all-minimum and
    all-maximum codes: the sign-flip / exponent-byte conversion of int8 and the
    nibble table of int4 must be exact at the ends of their ranges."""
    import torch
    n, rows = 2048, 64
    vec = (np.random.default_rng(5).standard_normal(n) * 2).astype(np.float16)
    for bits, lo, hi, dt in ((8, -128, 127, np.int8), (4, 0x00, 0xFF, np.uint8)):
        cols = n if bits == 8 else n // 2
        mat = np.empty((rows, cols), dtype=dt)
        mat[0::2] = lo
        mat[1::2] = hi
        y = _run(hq, bits, mat, vec, 0.25, 1.0, dev)
        ref = oracle.gemv_uniform_f64(mat, vec, bits, 0.25, 1.0)
        assert oracle.rel_err(y.cpu().numpy().astype(np.float64), ref) < TOL_F16
    # overwrite semantics: the result does not depend on what `out` held
    mat, vec = synth.gemv_uniform_case(256, 1024, 8, seed=2)
    out = torch.full((256,), 77.0, dtype=torch.float16, device=dev)
    hq.gemv_int8_quantized(to_dev(mat, dev), to_dev(vec, dev), 0.0625, 0.01, out=out)
    ref = oracle.gemv_uniform_f64(mat, vec, 8, 0.0625, 0.01)
    assert oracle.rel_err(out.cpu().numpy().astype(np.float64), ref) < TOL_F16


def test_gemv_uniform_argument_errors(hq, dev):
    import torch
    lib = hq.load_library()
    m = torch.zeros(64 * 64, dtype=torch.int8, device=dev)
    v = torch.zeros(64, dtype=torch.float16, device=dev)
    o = torch.zeros(64, dtype=torch.float16, device=dev)
    p = lambda t: t.data_ptr()
    assert lib.hq_gemv_int8_f16(None, p(v), p(o), 64, 64, 1.0, 0.0, None) == -2
    assert lib.hq_gemv_int8_f16(p(m), p(v), p(o), 64, 40, 1.0, 0.0, None) == -1      # n % 16
    assert lib.hq_gemv_int4_f16(p(m), p(v), p(o), 64, 48, 1.0, 0.0, None) == -1      # n % 32
    assert lib.hq_gemv_int8_f16(p(m) + 4, p(v), p(o), 4, 64, 1.0, 0.0, None) == -3   # alignment
    assert lib.hq_gemv_int4_f16(p(m), p(v), p(o), 1, 131072, 1.0, 0.0, None) == -7   # too long
    torch.cuda.synchronize()


@pytest.mark.parametrize("bits", [8, 4, 16])
def test_gemv_uniform_against_reference_kernel(hq, oracle, dev, bits):
    """The reference kernels with the reference driver's block shape (32 x 4,
    main.cu:33-34) on a square matrix: both results against the fp64 oracle; ours
    must be inside the tolerance and the two must agree to fp16 rounding."""
    import torch
    ref = refgpu.load()
    if ref is None or not hasattr(ref, "ref_gemv_int8"):
        pytest.skip("reference CUDA build not present")
    size, scale, zp = 2048, 0.0625, 0.01
    mat, vec = synth.gemv_uniform_case(size, size, bits, seed=bits)
    dm, dv = to_dev(mat, dev), to_dev(vec, dev)
    a = torch.empty(size, dtype=torch.float16, device=dev)
    args = (C.c_void_p(dm.data_ptr()), C.c_void_p(dv.data_ptr()), C.c_void_p(a.data_ptr()),
            C.c_uint(size))
    if bits == 8:
        ref.ref_gemv_int8(*args, C.c_float(scale), C.c_float(zp), C.c_uint(32), C.c_uint(4))
    elif bits == 4:
        ref.ref_gemv_int4(*args, C.c_float(scale), C.c_float(zp), C.c_uint(32), C.c_uint(4))
    else:
        ref.ref_gemv_f16(*args, C.c_uint(32), C.c_uint(4))
    b = _run(hq, bits, mat, vec, scale, zp, dev)
    torch.cuda.synchronize()
    y64 = oracle.gemv_uniform_f64(mat, vec, bits, scale, zp)
    ea = oracle.rel_err(a.cpu().numpy().astype(np.float64), y64)
    eb = oracle.rel_err(b.cpu().numpy().astype(np.float64), y64)
    assert ea < TOL_F16 and eb < TOL_F16
    assert oracle.rel_err(b.cpu().numpy().astype(np.float64),
                          a.cpu().numpy().astype(np.float64)) < TOL_F16


# one to a few pairs of rows; both sides of the lines between one and two CTAs per SM, blocks of 16 pairs and
# pairs one by one, and a last round a quarter full (148 SMs: 126, 148, 252 and 296 blocks; 4736 pairs a round)
@pytest.mark.parametrize("rows", [1, 2, 3, 33, 295, 296, 4000, 4031, 4033, 4736, 4739, 8051, 8053, 9473, 11839, 11843])
@pytest.mark.parametrize("bits,n", [(8, 48), (4, 2112)])
def test_every_row_once(hq, dev, rows, bits, n):
    """Each row's product, fp16 of fp32 sums of fp16 partial sums (rows of small integers and inputs of
    small halves: every sum is exact), where nothing but the division of the rows can go wrong."""
    import torch
    g = torch.Generator(device=dev).manual_seed(rows + n)
    x = torch.randint(-1, 2, (n,), generator=g, device=dev).half()
    if bits == 8:
        w = torch.randint(-2, 3, (rows, n), generator=g, device=dev)
        out = hq.gemv_int8_quantized(w.to(torch.int8), x, 1.0, 1.0)
        want = (w.double() - 1.0) @ x.double()
    else:
        b = torch.randint(0, 256, (rows, n // 2), generator=g, device=dev)
        w = torch.stack([b & 15, b >> 4], dim=2).reshape(rows, n)
        out = hq.gemv_int4_quantized(b.to(torch.uint8), x, 1.0, 8.0)
        want = (w.double() - 8.0) @ x.double()
    assert torch.equal(out.double(), want.half().double())


@pytest.mark.parametrize("bits", [16, 8, 4])
@pytest.mark.parametrize("rows,n,dealt", [(1024, 512, 1), (4736, 1024, 0)])
def test_a_kernel_for_each_division(hq, dev, bits, rows, n, dealt):
    """Blocks of pairs and pairs one by one are kernels of their own, plain and fused (as a parameter the
    division costs the 4-bit loops 3 to 7 %); plain 8-bit rows have one kernel, which is faster so."""
    import torch
    from launches import launched
    mat = torch.zeros((rows, n * bits // 8), dtype=torch.uint8, device=dev)
    w = {16: mat.view(torch.float16), 8: mat.view(torch.int8), 4: mat}[bits]
    x = torch.ones(n, dtype=torch.float16, device=dev)
    plain = {16: lambda: hq.gemv_fp16(w, x), 8: lambda: hq.gemv_int8_quantized(w, x, 1.0, 0.0),
             4: lambda: hq.gemv_int4_quantized(w, x, 1.0, 0.0)}[bits]
    fused = lambda: hq.gemv_fused({16: "f16", 8: "int8", 4: "int4"}[bits], x, w, rows // 2, gamma=x, act=hq.ACT_SWIGLU)
    for call, kernel in ((plain, "gemv_uniform_kernel"), (fused, "gemv_fused_kernel")):
        ((name, _),) = launched(call)
        assert f"{kernel}ILi{bits}ELb{0 if (bits, call) == (8, plain) else dealt}E" in name


@pytest.mark.parametrize("bits,rows,n,dealt", [
    (4, 9000, 4096, 0), (4, 8000, 6144, 0), (8, 9000, 2048, 0), (8, 9000, 3072, 1), (4, 7500, 4096, 1),  # two CTAs per SM
    (4, 32000, 2048, 0), (4, 41000, 4096, 0), (4, 41000, 512, 0), (4, 32000, 512, 1), (4, 35000, 2048, 1),  # a last round
    (4, 22016, 4096, 0), (4, 22016, 2048, 1), (8, 41000, 512, 1), (4, 12800, 2048, 1)])
def test_division_by_rule(hq, dev, bits, rows, n, dealt):
    """Rows in blocks where pairs one by one are 2 to 8 % slower (148 SMs), one by one where they gain."""
    import torch
    from launches import launched
    w = torch.zeros((rows, n * bits // 8), dtype=torch.uint8, device=dev).view(torch.int8 if bits == 8 else torch.uint8)
    x = torch.ones(n, dtype=torch.float16, device=dev)
    call = (lambda: hq.gemv_fused("int8", x, w, rows, gamma=x)) if bits == 8 else \
        (lambda: hq.gemv_int4_quantized(w, x, 1.0, 0.0))
    ((name, _),) = launched(call)
    assert f"ILi{bits}ELb{dealt}E" in name


def _small_case(bits, rows, n, dev):
    """Integer weights and inputs whose sums are exact in every order: weights for the kernels, their values less
    the zero point in fp64, inputs."""
    import torch
    g = torch.Generator(device=dev).manual_seed(rows + n)
    x = torch.randint(-1, 2, (n,), generator=g, device=dev).half()
    if bits == 4:
        b = torch.randint(0, 256, (rows, n // 2), generator=g, device=dev).to(torch.uint8)
        return b, torch.stack([b & 15, b >> 4], dim=2).reshape(rows, n).double() - 8.0, x
    w = torch.randint(-2, 3, (rows, n), generator=g, device=dev)
    return (w.half(), w.double(), x) if bits == 16 else (w.to(torch.int8), w.double() - 1.0, x)


ROWS_OVER_LINES = [1, 2, 3, 33, 296, 4000, 4033, 4736, 7999, 8053, 9473, 11839, 11843, 21500, 30783, 32003]


@pytest.mark.parametrize("rows", ROWS_OVER_LINES)
def test_every_f16_row_once(hq, dev, rows):
    """fp16 rows, where nothing but their division can go wrong (every sum is exact)."""
    import torch
    mat, w, x = _small_case(16, rows, 264, dev)
    assert torch.equal(hq.gemv_fp16(mat, x).double(), w @ x.double())


@pytest.mark.parametrize("rows_out", [(r + 1) // 2 for r in ROWS_OVER_LINES])
@pytest.mark.parametrize("bits,n", [(16, 264), (8, 48), (4, 2112)])
def test_every_fused_pair_once(hq, dev, bits, n, rows_out):
    """Value / gate pairs over the same lines.  v and g are exact; the gate is fp32 (2^-20 for its exponential,
    quotient and products), the result rounded to fp16 once, to 2^-25 where it is subnormal."""
    import torch
    mat, w, x = _small_case(bits, 2 * rows_out, n, dev)
    zero = {16: 0.0, 8: 1.0, 4: 8.0}[bits]
    kw = {} if bits == 16 else dict(scale=1.0, zero_point=zero)
    fmt = {16: "f16", 8: "int8", 4: "int4"}[bits]
    y = w @ x.double()
    v, gate = y[0::2], y[1::2]
    want = v * gate / (1 + torch.exp(-gate))
    got = hq.gemv_fused(fmt, x, mat, rows_out, act=hq.ACT_SWIGLU, **kw).double()
    finite = want.abs() < 65504
    assert bool(((got - want).abs() <= want.abs() * (2.0 ** -11 + 2.0 ** -20) + 2.0 ** -25)[finite].all())
    assert bool((got.abs() >= 65504)[~finite].all())
    plain = hq.gemv_fused(fmt, x, mat, 2 * rows_out, **kw)
    assert torch.equal(plain.double(), y.half().double())

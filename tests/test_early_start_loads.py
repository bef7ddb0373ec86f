"""Kernels that start while the launch before them drains (griddepcontrol.wait in
their source) read nothing by loads that may move above the wait: no ld.global.nc in
any spelling, no const __restrict__ parameter."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "hecbench_b200" / "csrc"
MAY_MOVE = re.compile(r"__ldg\(|\bldg_\w+\(|ld\.global\.nc|const[^;,()]*__restrict__")


def _blocks(text):
    """The top-level definitions of a source file, without comments."""
    text = re.sub(r"//[^\n]*", "", text)
    return re.split(r"^}\n", text, flags=re.M)


@pytest.mark.parametrize("name", ["aqlm.cu", "gemv_fused.cu", "gemv_uniform.cu", "lutgemm.cu", "nf4.cu",
                                  "q3_gemv.cu", "qgemm.cu"])
def test_no_load_can_pass_the_wait(name):
    blocks = _blocks((CSRC / name).read_text())
    early = [b for b in blocks if "__global__" in b and "pdl_wait();" in b]
    helpers = [b for b in blocks if "__device__" in b and "__global__" not in b]
    assert early
    for block in early + helpers:
        assert not MAY_MOVE.findall(block)


def _consumer(hq, family, dev):
    """How many fp16 numbers the operand takes, and call(buffer, out) with the output size."""
    import torch
    g = torch.Generator(device=dev).manual_seed(17)

    def codes(*shape):
        return torch.randint(0, 256, shape, generator=g, device=dev, dtype=torch.uint8)

    def halves(*shape, scale=1.0):
        return (torch.rand(shape, generator=g, device=dev) * scale).half()

    kind, operand = family.split()
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    if kind == "lutgemm":
        M, K = 4096, 512
        w = hq.nQWeight_fp16(codes(K // 8, 2, M).view(torch.int32), halves(K // 128, 2, M).float(),
                             K, M, 2, False, K // 128, halves(K // 128, M).float(), device=dev)
        x = halves(K)
        name = {"words": "bWeight", "alpha": "alpha", "bias": "q_bias"}[operand]
        dtype, n = getattr(w, name).dtype, getattr(w, name).numel()

        def call(buf, out):
            setattr(w, name, buf.view(dtype)[:n])
            hq.matmul(out, x, w)
        return n * dtype.itemsize // 2, call, (M,)
    if kind in ("1x16", "2x8"):
        K = 512
        M = 16 * 2 * sms                     # two CTAs per SM: both forms start early
        c = codes(M, K // 8, 2)
        book = halves(1, 65536, 8, scale=.05) if kind == "1x16" else halves(2, 256, 8, scale=.05)
        x, scales = halves(K), halves(M)
        n = {"codes": c.numel() // 2, "codebook": book.numel(), "scales": M}[operand]

        def call(buf, out):
            a = buf if operand == "codes" else c.view(-1).view(torch.float16)
            b = buf.view_as(book) if operand == "codebook" else book
            s = buf if operand == "scales" else scales
            if kind == "1x16":
                hq.code1x16_matvec(a.view(torch.int16), x, out, b, M, K, [M] * 4, 65536, scales=s)
            else:
                hq.code2x8_matvec(a.view(torch.uint8), x, out, b, M, K, scales=s)
        return n, call, (M,)
    if kind in ("q3mv", "nf4mv", "int4mv", "fused"):
        N, K = 2048, 512
        lut, x = torch.linspace(-1, 1, 16, device=dev), halves(K)
        if kind == "q3mv":
            parts = {"words": codes(K * 3 // 8, N).view(torch.int32).view(K * 3 // 32, N),
                     "scales": halves(N, scale=2 ** -5 if operand == "zeros" else 1).float(),
                     "zeros": halves(N, scale=1 if operand == "zeros" else 2 ** -5).float()}
        elif kind == "nf4mv":
            parts = {"codes": codes(N, K // 2), "absmax": halves(N * K // 64).float()}
        elif kind == "int4mv":
            parts = {"codes": codes(N, K // 2)}
        else:
            parts = {"gamma": halves(K), "codes": codes(N, K // 2)}
        operand_t = parts[operand]

        def call(buf, out):
            p = {**parts, operand: buf.view(operand_t.dtype).view(operand_t.shape)}
            if kind == "q3mv":
                mul = torch.zeros(N, device=dev)
                hq.vecquant3matmul_faster(x, p["words"], mul, p["scales"], p["zeros"], K * 3 // 32, N)
                out.copy_(mul * 2 ** -2)
            elif kind == "nf4mv":
                hq.gemv_nf4(x, p["codes"], p["absmax"], lut, N, K, 64, out=out)
            elif kind == "int4mv":
                hq.gemv_int4_quantized(p["codes"], x, 2 ** -4, 7.0, out=out)
            else:
                hq.gemv_fused("int4", x, p["codes"], N, gamma=p["gamma"], scale=2 ** -4, zero_point=7.0,
                              out=out)
        return operand_t.numel() * operand_t.dtype.itemsize // 2, call, (N,)
    Mb, N, K = 20, 1024, 512
    X = halves(Mb, K)
    if kind == "q3":
        words = codes(K * 3 // 8, N).view(torch.int32).view(K * 3 // 32, N)
        scales = halves(K // 128, N)

        def call(buf, out):
            m = buf.view(torch.int32) if operand == "words" else words
            s = buf if operand == "scales" else scales
            hq.qgemm_q3(X, m, s, scales, N, K, 128, out=out)
        return (words.numel() * 2 if operand == "words" else scales.numel()), call, (Mb, N)
    lut = torch.linspace(-1, 1, 16, device=dev)
    mat, absmax = codes(N, K // 2), halves(N * K // 64).float()

    def call(buf, out):
        b = buf.view(torch.uint8) if operand == "codes" else mat
        s = buf.view(torch.float32) if operand == "absmax" else absmax
        hq.qgemm_nf4(X, b, s, lut, N, K, 64, out=out)
    return (mat.numel() // 2 if operand == "codes" else absmax.numel() * 2), call, (Mb, N)


@pytest.mark.gpu
@pytest.mark.parametrize("family", ["lutgemm words", "lutgemm alpha", "lutgemm bias", "1x16 codes",
                                    "1x16 codebook", "1x16 scales", "2x8 codes", "2x8 codebook",
                                    "2x8 scales", "q3 words", "q3 scales", "nf4 codes", "nf4 absmax",
                                    "q3mv words", "q3mv scales", "q3mv zeros", "nf4mv codes", "nf4mv absmax",
                                    "int4mv codes", "fused codes", "fused gamma"])
def test_weights_written_by_the_launch_before(hq, dev, family):
    """An operand is the output of the launch right before, which itself started early:
    the numbers 0.5 to 2, or their bit patterns as codes (as absmax: 1e-4 to 2).  The
    same calls with a synchronisation after each are the oracle.  Sums of split rows
    meet in no fixed order: a result moves by one fp16 step at most, 2^-10 of itself."""
    import torch
    n, call, shape = _consumer(hq, family, dev)
    g = torch.Generator(device=dev).manual_seed(23)
    mat = torch.randint(0, 256, (n, 16), generator=g, device=dev, dtype=torch.uint8)
    steps = 6
    x = [((0.8 if t % 2 else 1.25) * (1 + 0.3 * torch.randn(32, generator=g, device=dev)) / 32).half()
         for t in range(steps)]
    buf = torch.ones(n, dtype=torch.float16, device=dev)
    outs = [torch.empty(shape, dtype=torch.float16, device=dev) for _ in range(steps)]

    def chain(sync=lambda: None):
        for t in range(steps):
            hq.gemv_int4_quantized(mat, x[t], 0.06, -8.0, out=buf)
            sync()
            call(buf, outs[t])
            sync()

    def results():
        torch.cuda.synchronize()
        return torch.stack(outs).float()

    chain(torch.cuda.synchronize)
    want = results()
    assert bool(torch.isfinite(want).all()) and float((want[0] - want[1]).norm() / want[0].norm()) > 0.02

    def check():
        got = results()
        for o in outs:
            o.zero_()
        error, size = (got - want).flatten(1).norm(dim=1), want.flatten(1).norm(dim=1)
        assert float((error / size).max()) < 2 ** -10

    for _ in range(10):
        chain()
        check()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        chain()
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            chain()
        for _ in range(10):
            graph.replay()
            check()

"""The quantizers start while the launch before them drains: they read
nothing by loads that may move above the wait, and see what that launch wrote."""
import pytest

from test_early_start_loads import CSRC, MAY_MOVE, _blocks


@pytest.mark.parametrize("name", ["mxfp4.cu", "vllm_quant.cu", "nf4_quantize.cu", "q3_quantize.cu",
                                  "lutgemm_quantize.cu", "qgemm_stream.cuh"])
def test_no_load_can_pass_the_wait(name):
    blocks = _blocks((CSRC / name).read_text())
    kernels = [b for b in blocks if "__global__" in b]
    assert kernels and all("pdl_wait();" in b for b in kernels)
    for block in blocks:
        assert not MAY_MOVE.findall(block)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["static", "dynamic", "dynamic odd", "dynamic_azp", "element-wise", "mxfp4", "nf4", "q3",
                                  "bcq"])
@pytest.mark.parametrize("rows", [64, 3000])
def test_input_written_by_the_launch_before(hq, dev, form, rows):
    """x is the output of a mat-vec that itself started early, and is overwritten by the next
    one right after the call; bytes as with a synchronisation after every call."""
    import torch
    n = rows * 1024
    g = torch.Generator(device=dev).manual_seed(rows)
    mat = torch.randint(0, 256, (n, 16), generator=g, device=dev, dtype=torch.uint8)
    steps = 5
    lut = torch.linspace(-1, 1, 16, device=dev)
    v = [torch.randn(32, generator=g, device=dev).half() for _ in range(steps)]
    buf = torch.zeros(n, dtype=torch.float16, device=dev)
    hidden = {"dynamic odd": 1023, "element-wise": 1021}.get(form, 1024)
    first = 1 if form == "element-wise" else 0               # not 16-byte aligned

    def call():
        if form == "nf4":
            codes, absmax = hq.quantize_nf4(buf, lut)
            return codes, absmax, hq.dequantize_nf4(codes, absmax, lut, n)
        if form == "q3":
            return hq.quantize_q3(buf.view(rows, 1024)[:rows // 32 * 32])
        if form == "bcq":
            return hq.quantize_bcq(buf.view(1024, rows), 3)
        if form == "mxfp4":
            codes, scales = hq.mxfp4_quantize(buf)
            return codes, scales, hq.mxfp4_dequantize(codes, scales, buf.dtype)
        x = buf[first:first + rows * hidden]
        out = torch.empty(rows * hidden, dtype=torch.int8, device=dev)
        scales, azp = torch.zeros(rows, device=dev), torch.zeros(rows, dtype=torch.int32, device=dev)
        if form == "static":
            hq.static_scaled_int8_quant(out, x, hidden, rows, 0.1)
        else:
            hq.dynamic_scaled_int8_quant(out, x, hidden, rows, scales, azp if form == "dynamic_azp" else None)
        return out, scales, azp

    def chain(sync=lambda: None):
        outs = []
        for t in range(steps):
            hq.gemv_int4_quantized(mat, v[t], 0.05, 7.5, out=buf)
            sync()
            outs.append(call())
            sync()
        return outs

    want = chain(torch.cuda.synchronize)
    torch.cuda.synchronize()
    assert not torch.equal(want[0][0], want[1][0])
    for _ in range(5):
        got = chain()
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert all(torch.equal(x, y) for x, y in zip(a, b))

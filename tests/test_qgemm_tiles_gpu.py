"""Edges of the batched product's tiles: the last half tile of 256 features, the last half
step of 128 inputs, token counts around multiples of 16 and the 64-token line, scale groups of
64, one CTA per few steps and tiles cut between CTAs."""
import pytest

pytestmark = pytest.mark.gpu


def _operands(hq, fmt, K, N, group, dev, g):
    """call(X, **kw) and the dequantised weights [K][N] in fp64."""
    import torch
    if fmt == "nf4":
        lut = torch.sort(torch.rand(16, generator=g, device=dev) * 2 - 1).values
        B = torch.randint(0, 256, (N, K // 2), generator=g, device=dev, dtype=torch.uint8)
        absmax = torch.rand(N * K // group, generator=g, device=dev) + 0.5
        W = hq.dequantize_nf4(B, absmax, lut, N * K, group, 0).view(N, K).t()
        return (lambda X, **kw: hq.qgemm_nf4(X, B, absmax, lut, N, K, group, 0, **kw)), W.double()
    mat = torch.randint(-2**31, 2**31, (K * 3 // 32, N), generator=g, device=dev).to(torch.int32)
    scales = (torch.rand((K // group, N), generator=g, device=dev) * 0.01 + 0.001).half()
    zeros = (scales * torch.randint(0, 8, (K // group, N), generator=g, device=dev)).half()
    codes = hq.vecquant3_dequant(mat, torch.ones(N, device=dev), torch.zeros(N, device=dev), K * 3 // 32, N,
                                 dtype=torch.float32)
    up = lambda p: p.double().repeat_interleave(group, 0)
    W = (codes.double() * up(scales) - up(zeros)).half()     # one rounding, as the fp16 fma
    return (lambda X, **kw: hq.qgemm_q3(X, mat, scales, zeros, N, K, group, **kw)), W.double()


@pytest.mark.parametrize("fmt", ["q3", "nf4"])
@pytest.mark.parametrize("Mb,K,N,group", [
    (1, 64, 128, 64), (16, 128, 128, 64), (17, 192, 384, 64), (64, 320, 256, 64), (65, 448, 640, 64),
    (128, 1088, 128, 64), (2, 4096, 1152, 128), (37, 8192, 4224, 128), (64, 1024, 37888, 128),
    (96, 8256, 2176, 64), (128, 2048, 38016, 128), (33, 28672, 1024, 128),
    # long layers on both sides of the line to the streamed form: half a step and half a tile left over,
    # scale groups of half a step, whole and cut tiles, tokens on both sides of 64
    (1, 8256, 14464, 64), (64, 3648, 28672, 64), (65, 16448, 7296, 64), (128, 1088, 104704, 64),
    (16, 28672, 4096, 128), (100, 1024, 120064, 128)])
def test_edges(hq, dev, fmt, Mb, K, N, group):
    """Within 2^-11 of the result (one fp16 rounding) plus what fp32 sums of K products may
    lose, K * 2^-24 of the sum of their magnitudes; the scratch is left zero, without
    scratch the same bound holds."""
    import torch
    from hecbench_b200 import api
    g = torch.Generator(device=dev).manual_seed(Mb + K + N)
    call, W = _operands(hq, fmt, K, N, group, dev, g)
    X = torch.randn((Mb, K), generator=g, device=dev).half()
    want = X.double() @ W
    bound = want.abs() * 2.0 ** -11 + (X.double().abs() @ W.abs()) * K * 2.0 ** -24 + 2.0 ** -24
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    for split in (True, True, False):
        got = call(X, status=status, split_k=split)
        torch.cuda.synchronize()
        assert int(status.item()) == 0, "a bounded in-kernel wait ran out"
        assert bool(((got.double() - want).abs() <= bound).all())
    assert all(int(torch.count_nonzero(w)) == 0 for w in api._qgemm_ws.values())


@pytest.mark.parametrize("fmt", ["q3", "nf4"])
@pytest.mark.parametrize("Mb,K,N,group", [
    (1, 8256, 14464, 64), (64, 5184, 38016, 64), (65, 16448, 7296, 64), (128, 1088, 104704, 64),
    (64, 28736, 6528, 64), (16, 28672, 8064, 128), (100, 1024, 120064, 128)])
def test_streamed_edges(hq, dev, fmt, Mb, K, N, group):
    """The same bounds where the streamed form runs (one CTA per SM of 148): a half step and a half tile
    left over, 1 to 128 tokens, whole tiles, cut ones in a fixed order and, on narrow layers, in none."""
    import torch
    from launches import launched
    g = torch.Generator(device=dev).manual_seed(Mb + K + N)
    call, _ = _operands(hq, fmt, K, N, group, dev, g)
    X = torch.randn((Mb, K), generator=g, device=dev).half()
    ((name, grid),) = launched(lambda: call(X))
    assert "qgemm_stream_kernel" in name and grid == torch.cuda.get_device_properties(dev).multi_processor_count
    test_edges(hq, dev, fmt, Mb, K, N, group)


@pytest.mark.parametrize("Mb,K,N,shifted_form", [
    (64, 8320, 14464, "stream"), (100, 8320, 14464, "stream"), (37, 8448, 14464, "stream"), (128, 8448, 7296, "parts"),
    (128, 12672, 7296, "stream"), (3, 28800, 8064, "stream"), (65, 28800, 8064, "stream")])
def test_streamed_absmax(hq, dev, Mb, K, N, shifted_form):
    """NF4 in blocks of 64 inputs: absmax rows that begin on 16 bytes and rows of which every other one
    begins in the middle of 16 (K = 128 modulo 256); the same values from an address that the
    copy unit cannot take give the same bits where the order of the sums is fixed (N above 12629) and the
    streamed form runs all the same, else what fp16 results of sums in another order may differ by."""
    import torch
    from launches import launched
    test_edges(hq, dev, "nf4", Mb, K, N, 64)
    g = torch.Generator(device=dev).manual_seed(Mb + K + N)
    lut = torch.sort(torch.rand(16, generator=g, device=dev) * 2 - 1).values
    B = torch.randint(0, 256, (N, K // 2), generator=g, device=dev, dtype=torch.uint8)
    absmax = torch.rand(N * K // 64, generator=g, device=dev) + 0.5
    shifted = torch.cat([absmax[:1], absmax])[1:]
    X = torch.randn((Mb, K), generator=g, device=dev).half()
    assert absmax.data_ptr() % 16 == 0 and shifted.data_ptr() % 16 == 4
    out = []
    wide = int(Mb > 64)
    forms = {"stream": f"qgemm_stream_kernelILi1ELb{wide}ELb0E", "parts": "12qgemm_kernelILi1E"}
    for values, form in ((absmax, f"qgemm_stream_kernelILi1ELb{wide}ELb1E"), (shifted, forms[shifted_form])):
        call = lambda: hq.qgemm_nf4(X, B, values, lut, N, K, 64, 0)
        ((name, _),) = launched(call)
        assert form in name
        out.append(call())
    if shifted_form == "stream" and N > 12629:
        assert torch.equal(*out)
    else:
        assert float((out[0] - out[1]).double().norm() / out[0].double().norm()) < 2.0 ** -11


@pytest.mark.parametrize("fmt,Mb,K,N,group", [
    ("q3", 64, 15744, 12800, 128), ("q3", 16, 9472, 12800, 128), ("q3", 2, 12672, 13952, 128),
    ("q3", 128, 12544, 12928, 128), ("nf4", 64, 9472, 12800, 64), ("nf4", 35, 8960, 13312, 64),
    ("nf4", 2, 9472, 12800, 128)])
def test_streamed_for_ordered_parts(hq, dev, fmt, Mb, K, N, group):
    """Layers that the form with parts would take in three or more ordered parts, 1.15 to 1.4 times slower
    than streamed: the streamed form takes them, with the same bits from every call."""
    import torch
    from launches import launched
    g = torch.Generator(device=dev).manual_seed(Mb + K + N)
    call, _ = _operands(hq, fmt, K, N, group, dev, g)
    X = torch.randn((Mb, K), generator=g, device=dev).half()
    ((name, _),) = launched(lambda: call(X))
    assert "qgemm_stream_kernel" in name
    assert torch.equal(call(X), call(X))


@pytest.mark.parametrize("fmt,Mb,K,N,streamed", [
    ("q3", 8, 1024, 52224, False), ("q3", 37, 1536, 50432, False), ("q3", 128, 2176, 19968, False),
    ("nf4", 64, 1536, 50432, False), ("q3", 100, 1024, 75776, True), ("q3", 128, 4096, 26624, True)])
def test_short_layers_in_parts(hq, dev, fmt, Mb, K, N, streamed):
    """Few steps per tile and cut tiles: 5 to 9 % slower streamed (148 SMs); whole tiles and longer layers are not."""
    import torch
    from launches import launched
    call, _ = _operands(hq, fmt, K, N, 64 if fmt == "nf4" else 128, dev, torch.Generator(device=dev).manual_seed(K))
    X = torch.zeros((Mb, K), dtype=torch.float16, device=dev)
    ((name, _),) = launched(lambda: call(X))
    assert ("qgemm_stream_kernel" in name) == streamed

"""Mat-vecs and batched products back to back, each reading the result of the one
before: the kernels start while the previous launch drains and have to wait for its
results.  The same chain with a synchronisation after every call is the oracle; the
sums of split rows meet in no fixed order, hence 5e-3 of the 2-norm after six calls
(fp16 results, each off by at most 2^-11 of its value and carried through the rest)."""
import pytest

pytestmark = pytest.mark.gpu


def _calls(hq, family, dev):
    """call(x, out) and the shape of x and out."""
    import torch
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    # 2x8 starts early from two CTAs of 16 rows (64 from 64 * SMs rows on: 32 rows) per SM
    # on, where SMs are not evenly full or hold no third CTA
    SIZE = {"aqlm 2x8": 64 * (sms // 2 + 4), "aqlm 2x8 long": 64 * sms}.get(family, 4096)
    g = torch.Generator(device=dev)
    g.manual_seed(11)

    def uniform(low, high, *shape):
        return torch.rand(shape, generator=g, device=dev) * (high - low) + low

    def codes(*shape):
        return torch.randint(0, 256, shape, generator=g, device=dev, dtype=torch.uint8)

    if family == "lutgemm":
        words = torch.randint(-2**31, 2**31, (SIZE // 32, 3, SIZE), generator=g, device=dev).to(torch.int32)
        w = hq.nQWeight_fp16(words, uniform(0.005, 0.015, SIZE // 128, 3, SIZE), SIZE, SIZE, 3, False,
                             SIZE // 128, None)
        return lambda x, out: hq.matmul(out, x, w), (SIZE,)
    if family == "aqlm 1x16":
        c = codes(SIZE, SIZE // 4).view(torch.int16)
        book = (torch.randn((1, 65536, 8), generator=g, device=dev) * 0.016).half()
        return lambda x, out: hq.code1x16_matvec(c, x, out, book, SIZE, SIZE, [SIZE] * 4, 65536), (SIZE,)
    if family.startswith("aqlm 2x8"):
        rows = 32 if family.endswith("long") else 16
        assert SIZE // rows >= 2 * sms and (rows == 32) == (SIZE // 32 >= 2 * sms)
        c = codes(SIZE, SIZE // 8, 2)
        book = (torch.randn((2, 256, 8), generator=g, device=dev) * (0.5 / SIZE) ** 0.5).half()
        return lambda x, out: hq.code2x8_matvec(c, x, out, book, SIZE, SIZE), (SIZE,)
    if family == "qgemm q3":
        words = codes(SIZE * 3 // 8, SIZE).view(torch.int32).view(SIZE * 3 // 32, SIZE)
        scales = uniform(0.8, 1.2, SIZE // 128, SIZE).div(2.3 * SIZE ** 0.5).half()
        zeros = scales * 3.5
        return lambda x, out: hq.qgemm_q3(x, words, scales, zeros, SIZE, SIZE, 128, out=out), (48, SIZE)
    mat = codes(SIZE, SIZE // 2)
    absmax = uniform(0.5, 2.0, SIZE * SIZE // 64) / SIZE ** 0.5
    lut = torch.linspace(-1, 1, 16, device=dev)
    return lambda x, out: hq.qgemm_nf4(x, mat, absmax, lut, SIZE, SIZE, 64, out=out), (48, SIZE)


@pytest.mark.parametrize("replayed", [False, True])
@pytest.mark.parametrize("family", ["lutgemm", "aqlm 1x16", "aqlm 2x8", "aqlm 2x8 long", "qgemm",
                                    "qgemm q3"])
def test_each_launch_waits_for_the_one_before(hq, dev, family, replayed):
    import torch
    call, shape = _calls(hq, family, dev)
    x0 = torch.randn(shape, generator=torch.Generator(device=dev).manual_seed(5), device=dev).half()

    a0, b0 = x0.clone(), torch.zeros_like(x0)

    def chain(sync):
        a, b = a0, b0
        a.copy_(x0)
        for _ in range(6):
            call(a, b)
            if sync:
                torch.cuda.synchronize()
            a, b = b, a
        return a

    want = chain(True).float()
    assert bool(torch.isfinite(want).all()) and float(want.norm()) > 0
    if replayed:
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            chain(False)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=s):
                chain(False)
    for _ in range(20):
        if replayed:
            graph.replay()
            got = a0
        else:
            got = chain(False)
        assert float((got.float() - want).norm() / want.norm()) < 5e-3


@pytest.mark.parametrize("per_cta,ctas_per_sm,extra", [(16, 2, -1), (16, 2, 0), (16, 2, 1), (16, 3, 0),
                                                       (32, 2, 0), (32, 2, 1), (32, 3, 5),
                                                       (32, 240, 0)])
def test_2x8_around_the_early_start(hq, dev, per_cta, ctas_per_sm, extra):
    """Row counts around two and three CTAs per SM, 16 and 32 rows per CTA, and more CTAs
    per SM than it has KiB of shared memory, against the product of the decoded weights in fp64; the kernel rounds sums of 16 products to fp16
    (2^-11 of a sum whose terms are a few times larger), so 1e-2 of the rms."""
    import torch
    m = per_cta * ctas_per_sm * torch.cuda.get_device_properties(dev).multi_processor_count + extra
    k = 192 if ctas_per_sm < 100 else 64
    g = torch.Generator(device=dev).manual_seed(m)
    codes = torch.randint(0, 256, (m, k // 8, 2), generator=g, device=dev, dtype=torch.uint8)
    book = torch.randn((2, 256, 8), generator=g, device=dev).half()
    x = torch.randn(k, generator=g, device=dev).half()
    out = torch.full((m + 8,), 3.0, dtype=torch.float16, device=dev)
    for _ in range(2):
        hq.code2x8_matvec(codes, x, out[:m], book, m, k)
    w = sum(book[i].double()[codes[..., i].long()] for i in range(2)).view(m, k)
    want = w @ x.double()
    assert float((out[:m].double() - want).abs().max() / want.pow(2).mean().sqrt()) < 1e-2
    assert bool((out[m:] == 3).all())

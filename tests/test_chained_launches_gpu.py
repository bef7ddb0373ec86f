"""Mat-vecs and batched products back to back, each reading the result of the one
before: the kernels start while the previous launch drains and have to wait for its
results.  The same chain with a synchronisation after every call is the oracle; the
sums of split rows meet in no fixed order, hence 5e-3 of the 2-norm after six calls
(fp16 results, each off by at most 2^-11 of its value and carried through the rest)."""
import pytest

pytestmark = pytest.mark.gpu
SIZE = 4096


def _calls(hq, family, dev):
    """call(x, out) and the shape of x and out."""
    import torch
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
    if family == "aqlm 2x8":
        c = codes(SIZE, SIZE // 8, 2)
        book = (torch.randn((2, 256, 8), generator=g, device=dev) * 0.011).half()
        return lambda x, out: hq.code2x8_matvec(c, x, out, book, SIZE, SIZE), (SIZE,)
    mat = codes(SIZE, SIZE // 2)
    absmax = uniform(0.5, 2.0, SIZE * SIZE // 64) / SIZE ** 0.5
    lut = torch.linspace(-1, 1, 16, device=dev)
    return lambda x, out: hq.qgemm_nf4(x, mat, absmax, lut, SIZE, SIZE, 64, out=out), (48, SIZE)


@pytest.mark.parametrize("family", ["lutgemm", "aqlm 1x16", "aqlm 2x8", "qgemm"])
def test_each_launch_waits_for_the_one_before(hq, dev, family):
    import torch
    call, shape = _calls(hq, family, dev)
    x0 = torch.randn(shape, generator=torch.Generator(device=dev).manual_seed(5), device=dev).half()

    def chain(sync):
        a, b = x0.clone(), torch.zeros_like(x0)
        for _ in range(6):
            call(a, b)
            if sync:
                torch.cuda.synchronize()
            a, b = b, a
        return a.float()

    want = chain(True)
    assert bool(torch.isfinite(want).all()) and float(want.norm()) > 0
    for _ in range(20):
        assert float((chain(False) - want).norm() / want.norm()) < 5e-3

"""Edges of the NF4 mat-vec's tensor form (absmax blocks of 64): rows around a tile of 16, rows
of one absmax block up to a whole and a broken super-step of 512 inputs, one to sixteen warps
per tile, more tiles than groups of warps, both nibble orders, early and late weights; against
fp64 products of the stored levels."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("N,K", [(1, 64), (15, 128), (16, 512), (17, 576), (33, 1024), (513, 1088), (5000, 2816),
                                 (2369, 4096), (31, 8256), (100, 16384), (7, 33024), (40001, 1024)])
def test_edges(hq, dev, N, K, early):
    """fp16 levels, exact products, fp32 sums of blocks and of their scaled sums: K * 2^-24 of the
    sum of magnitudes, and one rounding of the result to fp16."""
    import torch
    g = torch.Generator(device=dev).manual_seed(N + K)
    x = torch.randn(K, generator=g, device=dev).half()
    B = torch.randint(0, 256, (N, K // 2), generator=g, device=dev, dtype=torch.uint8)
    absmax = (torch.rand(N * K // 64, generator=g, device=dev) + 0.5) / K ** 0.5
    lut = torch.sort(torch.rand(16, generator=g, device=dev) * 2 - 1).values
    for order in (hq.NF4_HIGH_NIBBLE_FIRST, hq.NF4_LOW_NIBBLE_FIRST):
        hi, lo = (B >> 4).long(), (B & 15).long()
        codes = torch.stack([lo, hi] if order == hq.NF4_LOW_NIBBLE_FIRST else [hi, lo], -1).view(N, K)
        terms = lut.half().double()[codes] * x.double() * absmax.double().view(N, K // 64).repeat_interleave(64, 1)
        want = terms.sum(1)
        bound = want.abs() * 2.0 ** -11 + terms.abs().sum(1) * K * 2.0 ** -24 + 2.0 ** -24
        got = hq.gemv_nf4(x, B, absmax, lut, N, K, 64, order, weights_resident=early)
        assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("K", [38144, 38208, 65536])
def test_longest_fused_rows(hq, dev, K):
    """RMSNorm, value / gate pairs and SwiGLU on the longest rows, against fp64 of the scaled inputs
    rounded to fp16.  Those roundings may fall the other way where fp32 and fp64 norms differ: 2^-11 of
    the sum of magnitudes more; both bounds pass through the product with the activation, whose slope is below 1.1."""
    import torch
    g = torch.Generator(device=dev).manual_seed(K)
    rows = 34
    x = torch.randn(K, generator=g, device=dev).half()
    gamma = (torch.rand(K, generator=g, device=dev) + 0.5).half()
    B = torch.randint(0, 256, (rows, K // 2), generator=g, device=dev, dtype=torch.uint8)
    absmax = (torch.rand(rows * K // 64, generator=g, device=dev) + 0.5) / K ** 0.5
    lut = torch.sort(torch.rand(16, generator=g, device=dev) * 2 - 1).values
    codes = torch.stack([(B >> 4).long(), (B & 15).long()], -1).view(rows, K)
    xd = x.double()
    xn = (xd * torch.rsqrt((xd * xd).mean() + 1e-5) * gamma.double()).half().double()
    terms = lut.half().double()[codes] * xn * absmax.double().view(rows, K // 64).repeat_interleave(64, 1)
    sums, off = terms.sum(1), terms.abs().sum(1) * (K * 2.0 ** -24 + 2.0 ** -11)
    value, gate = sums[0::2], sums[1::2]
    want = value * torch.nn.functional.silu(gate)
    bound = want.abs() * 2.0 ** -10 + off[0::2] * gate.abs() + off[1::2] * 1.1 * value.abs() + 1.1 * off[0::2] * off[1::2]
    got = hq.gemv_fused("nf4", x, B, rows // 2, gamma=gamma, eps=1e-5, act=hq.ACT_SWIGLU, absmax=absmax, lut16=lut,
                        blocksize=64)
    assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("level", [0, 3, 15])
@pytest.mark.parametrize("N,K", [(33, 1024), (40, 576), (100, 2816), (70, 4096)])
def test_infinite_level(hq, dev, N, K, level):
    """A level that no fp16 number holds: rows without its code keep their value, the others become
    infinite with the sign of the product, or NaN where two signs meet, as the sum of the products has it."""
    import torch
    from launches import launched
    g = torch.Generator(device=dev).manual_seed(N + K + level)
    x = torch.randn(K, generator=g, device=dev).half()
    codes = torch.randint(0, 15, (N, K), generator=g, device=dev)
    codes += codes >= level                                            # every code but `level`
    once = torch.arange(0, N, 3, device=dev)                           # one such code in every third row,
    codes[once, torch.randint(0, K, (len(once),), generator=g, device=dev)] = level
    codes[0, [1, 40]] = level                                          # and two of one block in the first
    x[1], x[40] = 1.0, -1.0
    B = (codes[:, 0::2] << 4 | codes[:, 1::2]).to(torch.uint8)
    absmax = (torch.rand(N * K // 64, generator=g, device=dev) + 0.5) / K ** 0.5
    lut = torch.linspace(-1, 1, 16, device=dev)
    lut[level] = 1e30 if level else -float("inf")
    terms = lut.half().double()[codes] * x.double() * absmax.double().view(N, K // 64).repeat_interleave(64, 1)
    want = terms.sum(1)
    got = []
    ((name, _),) = launched(lambda: got.append(hq.gemv_nf4(x, B, absmax, lut, N, K, 64)))
    assert "nf4_gemv_mma_kernel" in name
    got = got[0].double()
    finite = want.isfinite()
    assert bool(want[0].isnan()) and bool(want.isinf().any()) and bool(finite.any())
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[want.isinf()], want[want.isinf()])
    bound = want.abs() * 2.0 ** -11 + terms.abs().sum(1) * K * 2.0 ** -24 + 2.0 ** -24
    assert bool(((got - want).abs() <= bound)[finite].all())

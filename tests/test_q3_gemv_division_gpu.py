"""The 3-bit mat-vec's division into blocks of columns and steps along K: ranges that begin inside a
block, a last block, a last quad of groups and a last slice of K that are not full, 8, 16 and 20
warps side by side or in turn; inputs of every exponent, and an infinity."""
import pytest

pytestmark = pytest.mark.gpu

# warps of a CTA, those of them side by side (at 148 SMs), columns, inputs: ranges of one step, of several and into the next block;
# more than 16384 inputs are two slices of K
FORMS = [(8, 8, 4, 32), (8, 8, 260, 160), (8, 8, 512, 1024), (8, 8, 5116, 4288), (8, 8, 4100, 4160),
         (16, 16, 1612, 13632), (16, 16, 804, 26144), (16, 8, 1548, 15136), (16, 8, 3308, 16448),
         (16, 4, 572, 14016), (16, 4, 1544, 16800),
         (20, 20, 3200, 3040), (20, 20, 8804, 1280), (20, 20, 11008, 4096), (20, 20, 516, 16416), (20, 20, 1028, 33024),
         (20, 10, 944, 10752), (20, 10, 820, 11424), (20, 10, 264, 24736), (20, 5, 684, 13344), (20, 5, 2312, 19008)]


def _layer(hq, dev, N, K):
    import torch
    g = torch.Generator(device=dev).manual_seed(N * 7 + K)
    mat = torch.randint(-2**31, 2**31, (K * 3 // 32, N), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
    scales = torch.rand(N, generator=g, device=dev) * 0.01 + 0.001
    zeros = scales * torch.randint(0, 8, (N,), generator=g, device=dev)
    codes = hq.vecquant3_dequant(mat, torch.ones(N, device=dev), torch.zeros(N, device=dev), K * 3 // 32, N)
    return g, mat, scales, zeros, codes.double()


@pytest.mark.parametrize("half", [True, False])
@pytest.mark.parametrize("warps,beside,N,K", FORMS)
def test_divisions(hq, dev, warps, beside, N, K, half):
    """Products are exact, so what differs from fp64 is the order of fp32 sums: K * 2^-24 of the sum of
    the products' magnitudes at most, whatever the inputs' exponents (here 2^-8 to 2^8).  Inputs of one sign too: a piece
    of theirs that went missing would be 2^-9 of them (the third of fp32 inputs 2^-17, seen with the fewest inputs)."""
    import torch
    from launches import launched
    g, mat, scales, zeros, codes = _layer(hq, dev, N, K)
    x = torch.randn(K, generator=g, device=dev) * torch.exp2(torch.randint(-8, 9, (K,), generator=g, device=dev).float())
    call = hq.vecquant3matmul_faster if half else hq.vecquant3matmul
    s, z = (scales.half().double(), zeros.half().double()) if half else (scales.double(), zeros.double())
    start = torch.randn(N, generator=g, device=dev)
    for x in (x, x.abs()):
        x = x.half() if half else x
        out = start.clone()
        call(x, mat, out, scales, zeros, K * 3 // 32, N)
        want = start.double() + s * (x.double() @ codes) - z * x.double().sum()
        size = s * (x.double().abs() @ codes) + z * x.double().abs().sum()
        assert bool(((out.double() - want).abs() <= size * K * 2.0 ** -24 + want.abs() * 2.0 ** -22 + 2.0 ** -22).all())
    ((name, _),) = launched(lambda: call(x, mat, out, scales, zeros, K * 3 // 32, N))
    if torch.cuda.get_device_properties(dev).multi_processor_count == 148:
        assert f"q3_gemv_kernelILb{int(half)}ELi{warps}ELi{beside}EE" in name, name


@pytest.mark.parametrize("exponent,K", [(-123, 2048), (-110, 2048), (-60, 2048), (-1, 2048), (0, 2048), (60, 2048), (110, 2048),
                                        (-123, 32), (0, 32), (118, 32)])
def test_fp32_inputs_of_any_exponent(hq, dev, exponent, K):
    """Inputs are split exactly and scaled by their largest exponent: the bound above holds for tiny and huge
    ones, also beside ones of another size (every 256 inputs 2^-20 of the others, single ones 2^-12).  The sums are
    held as 2^-8 of their value: below 2^-118 an addition may lose 2^-142, a quantum of fp32 times 2^8.  (Large scales
    with small inputs: an atomic addition takes what is below 2^-126 for zero.)"""
    import torch
    N = 516
    g, mat, scales, zeros, codes = _layer(hq, dev, N, K)
    scales, zeros = (v * 2.0 ** (16 if exponent < 0 else 0) for v in (scales, zeros))
    x = torch.randn(K, generator=g, device=dev).abs() * 2.0 ** exponent
    x[256:512] *= 2.0 ** -20
    x[5::37] *= 2.0 ** -12
    for x in (x, x * torch.randint(0, 2, (K,), generator=g, device=dev).mul(2).sub(1)):
        out = torch.zeros(N, device=dev)
        hq.vecquant3matmul(x, mat, out, scales, zeros, K * 3 // 32, N)
        want = scales.double() * (x.double() @ codes) - zeros.double() * x.double().sum()
        size = scales.double() * (x.double().abs() @ codes) + zeros.double() * x.double().abs().sum()
        bound = size * K * 2.0 ** -24 + scales.double() * (K // 16 + 8) * 2.0 ** -142 + (K // 128 + 1) * 2.0 ** -126
        assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("half", [True, False])
def test_an_infinite_input(hq, dev, half):
    """An infinity times a code above zero is one, with the sign of the input (zeros below zero: what the
    sum of inputs adds has that sign too); times zero it is no number."""
    import torch
    N, K = 132, 96
    g, mat, scales, zeros, codes = _layer(hq, dev, N, K)
    x = torch.randn(K, generator=g, device=dev)
    x[37] = float("-inf")
    x = x.half() if half else x
    out = torch.zeros(N, device=dev)
    (hq.vecquant3matmul_faster if half else hq.vecquant3matmul)(x, mat, out, scales, -scales, K * 3 // 32, N)
    above = codes[37] > 0
    assert bool((out[above] == float("-inf")).all()) and bool(out[~above].isnan().all())

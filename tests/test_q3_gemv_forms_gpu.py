"""The 3-bit mat-vec on layers of one column block to many, with short and long rows and ragged last blocks; fp16
and fp32 inputs, added to what the sums hold."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(4, 32), (132, 96), (1024, 4096), (16388, 2048), (8196, 8192), (28676, 4096),
                                 (36868, 12288), (49152, 12288)])
def test_forms(hq, dev, N, K):
    """Against fp64 sums of the codes and inputs, scale and zero of the fp16 form rounded to fp16
    as its rule has it.  Products are exact in both forms, sums in fp32: K * 2^-24 of the sum of their magnitudes."""
    import torch
    g = torch.Generator(device=dev).manual_seed(N + K)
    mat = torch.randint(-2**31, 2**31, (K * 3 // 32, N), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
    scales = torch.rand(N, generator=g, device=dev) * 0.01 + 0.001
    zeros = scales * torch.randint(0, 8, (N,), generator=g, device=dev)
    start = torch.randn(N, generator=g, device=dev)
    codes = hq.vecquant3_dequant(mat, torch.ones(N, device=dev), torch.zeros(N, device=dev), K * 3 // 32, N)
    for half in (True, False):
        x = torch.randn(K, generator=g, device=dev)
        x = x.half() if half else x
        s, z = (scales.half().double(), zeros.half().double()) if half else (scales.double(), zeros.double())
        want = start.double() + s * (x.double() @ codes.double()) - z * x.double().sum()
        size = s * (x.double().abs() @ codes.double()) + z * x.double().abs().sum()
        out = start.clone()
        (hq.vecquant3matmul_faster if half else hq.vecquant3matmul)(x, mat, out, scales, zeros, K * 3 // 32, N)
        bound = size * K * 2.0 ** -24 + want.abs() * 2.0 ** -22 + 2.0 ** -22
        assert bool(((out.double() - want).abs() <= bound).all())

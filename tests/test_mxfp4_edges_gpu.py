"""MXFP4 at the edges of its kernels: ragged group counts, buffers aligned to 16 and 4
bytes only, infinities, every scale byte in the unpacker."""
import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu
GRID = np.array([0, .5, 1, 1.5, 2, 3, 4, 6], dtype=np.float64)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("groups,shift", [(1, 0), (255, 8), (257, 8), (4096, 0)])
def test_pack_alignment_and_specials(hq, oracle, dev, dtype, groups, shift):
    bf16 = dtype == torch.bfloat16
    rng = np.random.default_rng(groups)
    bits = rng.integers(0, 65536, groups * 32).astype(np.uint16)      
    nan = (bits & 0x7fff) > (0x7f80 if bf16 else 0x7c00)
    bits[nan] &= 0xbfff
    bits.reshape(-1, 32)[1::2] &= 0xbfff                              # and groups of finite values
    base = torch.zeros(groups * 32 + 16, dtype=torch.int16, device=dev)
    a = base[shift:shift + groups * 32]
    a.copy_(to_dev(bits.view(np.int16), dev))
    a = a.view(dtype)
    cbase = torch.zeros(groups * 16 + 16, dtype=torch.uint8, device=dev)
    codes, scales = hq.mxfp4_quantize(a, codes=cbase[shift // 2:shift // 2 + groups * 16])
    oc, osc = oracle.mxfp4_quantize(bits, bf16)
    assert np.array_equal(codes.cpu().numpy(), oc)
    assert np.array_equal(scales.cpu().numpy(), osc)
    ybase = torch.zeros(groups * 32 + 16, dtype=dtype, device=dev)
    y = ybase[shift:shift + groups * 32]
    hq.mxfp4(y, a, groups * 32)
    back = hq.mxfp4_dequantize(codes, scales, dtype, out=torch.empty_like(ybase)[shift:shift + groups * 32])
    assert torch.equal(back.view(torch.int16), y.view(torch.int16))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_unpack_every_code_and_scale(hq, dev, dtype):
    """All 16 codes under the 255 finite scale bytes: value * 2^k rounded once to the type."""
    codes = np.tile(np.arange(256, dtype=np.uint8), (255, 1)).reshape(-1)     # 16 groups per scale
    scales = np.repeat(np.arange(255, dtype=np.uint8), 16)
    out = hq.mxfp4_dequantize(to_dev(codes, dev), to_dev(scales, dev), dtype)
    n = np.stack([codes & 15, codes >> 4], 1).reshape(-1)
    val = GRID[n & 7] * np.where(n & 8, -1.0, 1.0) * np.repeat(2.0 ** (scales.astype(np.float64) - 127), 32)
    want = torch.from_numpy(val).to(dtype)        # fp64 -> fp32 is exact here
    assert torch.equal(out.cpu().view(torch.int16), want.view(torch.int16))

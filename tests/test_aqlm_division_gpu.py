"""Division of the additive-codebook mat-vecs' rows over CTAs and warps: dealt one by one or in blocks,
both sides of the lines between them (148 SMs, two rows per warp up to 9471 rows, four beyond)."""
import numpy as np
import pytest

from hecbench_b200 import synth
from conftest import to_dev

pytestmark = pytest.mark.gpu

ROWS = [1, 2, 3, 295, 297, 1025, 2241, 2257, 2368, 2369, 4097, 4495, 4513, 4737, 6145, 8193, 9473, 14337, 18945]


@pytest.mark.parametrize("m", ROWS)
@pytest.mark.parametrize("k", [64, 2112])
def test_1x16_rows(hq, oracle, dev, m, k):
    """The bits of the restated reference arithmetic, in a buffer whose end stays untouched."""
    import torch
    codes, x, cb, scales = synth.aqlm_1x16_case(m, k, 1, seed=m + k)
    h = lambda a: to_dev(a.view(np.uint16), dev).view(torch.float16)
    out = torch.full((m + 64,), 7.0, dtype=torch.float16, device=dev)
    sizes = [m, m, m, 1 << 30]
    hq.code1x16_matvec(to_dev(codes, dev), h(x), out[:m], h(cb), m, k, sizes, 65536, h(scales))
    want = oracle.aqlm_1x16_ref(codes, x, cb, m, k, sizes, 65536, scales)
    got = out.cpu().numpy()
    assert np.array_equal(got[:m].view(np.uint16), want.view(np.uint16)) and (got[m:] == 7.0).all()


@pytest.mark.parametrize("m", ROWS)
def test_2x8_rows(hq, oracle, dev, m):
    """Each row within what short fp16 sums lose: 2^-9 of the 2-norm over rows (16 products of half
    precision, 2^-11 each, and the result's rounding)."""
    import torch
    k = 576
    codes, x, cbs, scales = synth.aqlm_2x8_case(m, k, seed=m + k)
    h = lambda a: to_dev(a.view(np.uint16), dev).view(torch.float16)
    out = torch.full((m + 64,), 7.0, dtype=torch.float16, device=dev)
    hq.code2x8_matvec(to_dev(codes, dev), h(x), out[:m], h(cbs), m, k, h(scales))
    want = oracle.aqlm_2x8_f64(codes, x, cbs, m, k, scales)
    got = out.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got[:m] - want) <= 2.0 ** -9 * np.linalg.norm(want) and (got[m:] == 7.0).all()


@pytest.mark.parametrize("m,k,dealt", [
    (4737, 8192, 0), (9473, 5056, 0), (5504, 6144, 0), (9728, 11008, 0), (11008, 5056, 1), (6144, 14336, 1),
    (4737, 4992, 1), (9473, 4096, 1),
    # nearly even blocks stay
    (2240, 4096, 0), (6656, 4096, 0), (13312, 4096, 0), (12288, 4096, 1), (13400, 8192, 1)])
def test_2x8_deals_what_fits(hq, dev, m, k, dealt):
    """More CTAs than an SM holds (two beyond 4992 inputs) only for long rows and more than a tenth of a
    last round: each stages the codebooks again, up to 1.6 times the time (148 SMs).  Blocks that are
    nearly even stay."""
    import torch
    from launches import launched
    codes = torch.zeros((m, k // 8, 2), dtype=torch.uint8, device=dev)
    x, cbs = (torch.ones(s, dtype=torch.float16, device=dev) for s in (k, (2, 256, 8)))
    out, scales = (torch.ones(m, dtype=torch.float16, device=dev) for _ in range(2))
    ((name, grid),) = launched(lambda: hq.code2x8_matvec(codes, x, out, cbs, m, k, scales))
    rows = 32 if m // 32 >= 296 else 16
    assert f"aqlm_2x8_kernelILb{dealt}E" in name and grid == (444 if dealt else -(-m // rows))
    assert bool((out == 2 * k).all())

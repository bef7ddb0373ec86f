"""One and two planes of the LUT-GEMM mat-vec on both sides of the line between register form and rings."""
import numpy as np
import pytest

from hecbench_b200 import synth
from conftest import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,gs,line", [(1, 64, 2.65), (1, 128, 3.6), (2, 64, 2.65), (2, 128, 2.65)])
@pytest.mark.parametrize("ring", [False, True])
def test_rings_from_their_line_on(hq, oracle, dev, nb, gs, line, ring):
    """Column steps of a warp, M tiles / (512 SMs), just below the line and just behind it.  Against fp64: one
    fp16 rounding, 2^-11, and fp32 sums whose loss is far below it: 1e-3 of the 2-norm."""
    import torch
    from launches import launched
    K = 4096
    M = int(line * 512 * torch.cuda.get_device_properties(dev).multi_processor_count / (K // 128)) // 4 * 4 + 4 * ring
    x, bW, alpha, qb = synth.lutgemm_case(M, K, nb, gs, seed=M + nb, bias=True)
    w = hq.nQWeight_fp16()
    w.parsing(bW, alpha.astype(np.float32), K, M, nb, False, K // gs, qb.astype(np.float32), device=dev)
    out = torch.empty(M, dtype=torch.float16, device=dev)
    dx = to_dev(x.view(np.uint16), dev).view(torch.float16)
    ((name, _),) = launched(lambda: hq.matmul(out, dx, w))
    assert ("lutgemm_ring_kernel" in name) == ring, name
    ref = oracle.lutgemm_gemv_f64(x, bW, alpha, qb, M, K, nb, gs)
    assert np.linalg.norm(out.cpu().numpy().astype(np.float64) - ref) <= 1e-3 * np.linalg.norm(ref)
    assert torch.count_nonzero(w.workspace()) == 0

"""Edges of the LUT-GEMM mat-vec's units: column counts around a warp's 32 and a range's 256, K
tiles past the end of K, alpha groups below a tile, four planes in one launch, more column
ranges than completion counters, and several units per CTA with ragged last ranges and tiles."""
import numpy as np
import pytest

from hecbench_b200 import synth
from conftest import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,nb,gs,bias", [
    (4, 32, 1, 32, True), (36, 160, 4, 32, True), (252, 192, 4, 64, True), (260, 320, 2, 64, False),
    (1028, 96, 3, 32, True), (4096, 12288, 4, 128, True), (12292, 4096, 2, 64, True),
    (2052, 1344, 4, 192, True), (40960, 256, 3, 128, False)])
def test_edges(hq, oracle, dev, M, K, nb, gs, bias):
    """Against fp64: one fp16 rounding, 2^-11, and fp32 sums whose loss is far below it: 1e-3
    of the 2-norm.  Repeated, the scratch is left zero."""
    import torch
    x, bW, alpha, qb = synth.lutgemm_case(M, K, nb, gs, seed=M + K + nb, bias=bias)
    w = hq.nQWeight_fp16()
    w.parsing(bW, alpha.astype(np.float32), K, M, nb, False, K // gs,
              None if qb is None else qb.astype(np.float32), device=dev)
    dx = to_dev(x.view(np.uint16), dev).view(torch.float16)
    ref = oracle.lutgemm_gemv_f64(x, bW, alpha, qb, M, K, nb, gs)
    for _ in range(3):
        out = torch.full((M,), 7.0, dtype=torch.float16, device=dev)
        hq.matmul(out, dx, w)
        got = out.cpu().numpy().astype(np.float64)
        assert np.linalg.norm(got - ref) <= 1e-3 * np.linalg.norm(ref)
    assert torch.count_nonzero(w.workspace()) == 0


@pytest.mark.parametrize("M,K,nb,gs,bias", [
    (6148, 9632, 3, 32, True), (6148, 9664, 4, 64, True), (3076, 20544, 4, 64, False), (8196, 9664, 3, 64, False)])
def test_several_units_per_cta(hq, oracle, dev, M, K, nb, gs, bias):
    """228 to 322 units on the CTAs of the ring form, one per SM of 148: a last column range of four columns
    more than whole warps, one to two rows of four in the last tile."""
    import torch
    from launches import launched
    x, bW, alpha, qb = synth.lutgemm_case(M, K, nb, gs, seed=M + K + nb, bias=bias)
    w = hq.nQWeight_fp16()
    w.parsing(bW, alpha.astype(np.float32), K, M, nb, False, K // gs,
              None if qb is None else qb.astype(np.float32), device=dev)
    out = torch.empty(M, dtype=torch.float16, device=dev)
    dx = to_dev(x.view(np.uint16), dev).view(torch.float16)
    ((name, grid),) = launched(lambda: hq.matmul(out, dx, w))
    assert f"lutgemm_ring_kernelILi{nb}E" in name
    assert grid == torch.cuda.get_device_properties(dev).multi_processor_count
    test_edges(hq, oracle, dev, M, K, nb, gs, bias)


@pytest.mark.parametrize("M,K,nb,gs,bias", [
    (6148, 9664, 1, 64, True), (6148, 9664, 2, 64, False), (8196, 9728, 1, 128, True), (8196, 9728, 2, 128, True),
    (4100, 4096, 3, 128, False), (4100, 4096, 7, 64, True)])
def test_fewer_planes_in_rings(hq, oracle, dev, M, K, nb, gs, bias):
    """One to three planes where the ring form takes them, alone or after four: lanes of a column of their
    own, a last column range that ends inside a warp, two rows of four in the last tile."""
    import torch
    from launches import launched
    x, bW, alpha, qb = synth.lutgemm_case(M, K, nb, gs, seed=M + K + nb, bias=bias)
    w = hq.nQWeight_fp16()
    w.parsing(bW, alpha.astype(np.float32), K, M, nb, False, K // gs,
              None if qb is None else qb.astype(np.float32), device=dev)
    out = torch.empty(M, dtype=torch.float16, device=dev)
    dx = to_dev(x.view(np.uint16), dev).view(torch.float16)
    names = [name for name, _ in launched(lambda: hq.matmul(out, dx, w))]
    planes = [4] * (nb // 4) + [nb % 4]
    assert len(names) == len(planes) and all(f"lutgemm_ring_kernelILi{n}E" in k for n, k in zip(planes, names))
    test_edges(hq, oracle, dev, M, K, nb, gs, bias)

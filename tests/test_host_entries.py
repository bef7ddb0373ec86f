"""The native launch path (csrc/host/host.cpp): argument checks without a GPU, and
the same checks with CUDA tensors of the wrong type, layout or count."""
import pytest
import torch


def test_entries_reject_bad_arguments_without_gpu(hq):
    from hecbench_b200 import _lib, _host
    host = hq.load_library().host
    assert set(_host.symbols) <= set(_lib.SIGNATURES)
    t = torch.zeros(64)
    with pytest.raises(TypeError, match="takes 7 positional"):
        host.hq_q3_gemv_f32(t, t)
    with pytest.raises(TypeError, match="expected a torch.Tensor"):
        host.hq_q3_gemv_f32(1, t, t, t, t, 3, 4)
    with pytest.raises(TypeError, match="no CPU path"):
        host.hq_q3_gemv_f32(t, t, t, t, t, 3, 4)
    with pytest.raises(TypeError):
        host.empty(t, torch.float16, 4)
    with pytest.raises(KeyError):
        _host.Entry("hq_version", 1, None)


@pytest.mark.gpu
def test_entries_reject_bad_cuda_tensors(hq, dev):
    x, mat = torch.ones(64, device=dev), torch.zeros(6, 8, dtype=torch.int32, device=dev)
    par, y = torch.ones(8, device=dev), torch.zeros(8, device=dev)
    with pytest.raises(TypeError, match="vec: expected dtype torch.float32, got torch.float16"):
        hq.vecquant3matmul(x.half(), mat, y, par, par, 6, 8)
    with pytest.raises(TypeError, match="mat: must be contiguous"):
        hq.vecquant3matmul(x, mat.t(), y, par, par, 6, 8)
    with pytest.raises(hq.HqError, match="hq_q3_gemv_f32 failed: bad shape"):
        hq.vecquant3matmul(x, mat, y, par, par, 5, 8)
    with pytest.raises(ValueError):
        hq.code1x16_matvec(torch.zeros(4, 8, dtype=torch.int16, device=dev), x.half(), y.half(),
                           x.half(), 4, 64, [4, 4], 65536)
    # another stream than the default one: the launch goes where torch's does
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        hq.vecquant3matmul(x, mat, y, par, par, 6, 8)
    s.synchronize()
    assert torch.equal(y, torch.full_like(y, -64.0))  # codes 0: sum of (0 - zero) * 1

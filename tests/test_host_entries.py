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
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        hq.vecquant3matmul(x, mat, y, par, par, 6, 8)
    s.synchronize()
    assert torch.equal(y, torch.full_like(y, -64.0))  # codes 0: sum of (0 - zero) * 1


def test_codebook_limits_must_reach_a_codebook(hq):
    """Fewer than three limits: the missing ones count as 0, which moves every row to a
    later codebook."""
    a, x, y = torch.zeros(4, 8, dtype=torch.int16), torch.zeros(64).half(), torch.zeros(4).half()
    one, four = torch.zeros(1, 65536, 8).half(), torch.zeros(4, 65536, 8).half()
    for sizes in ([4], [4, 4], [], (4.0, 4)):
        with pytest.raises(ValueError, match="beyond the last codebook"):
            hq.code1x16_matvec(a, x, y, one, 4, 64, sizes, 65536)
        with pytest.raises(TypeError, match="no CPU path"):
            hq.code1x16_matvec(a, x, y, four, 4, 64, sizes, 65536)


@pytest.mark.gpu
def test_codebook_limits_in_other_forms(hq, dev):
    """What int() takes, and up to four of them."""
    g = torch.Generator(device=dev).manual_seed(1)
    m, k = 48, 64
    a = torch.randint(0, 1 << 15, (m, k // 8), generator=g, device=dev).to(torch.int16)
    book = torch.randn((3, 65536, 8), generator=g, device=dev).half()
    x = torch.randn(k, generator=g, device=dev).half()

    def run(sizes):
        y = torch.empty(m, dtype=torch.float16, device=dev)
        hq.code1x16_matvec(a, x, y, book, m, k, sizes, 65536)
        return y

    want = run([16, 32, m, m])
    assert not torch.equal(want, run([m, m, m, m]))
    for sizes in ([16, 32, m], (16.0, 32.9, float(m)), torch.tensor([16, 32, m, m]),
                  (v for v in (16, 32, m, 0))):
        assert torch.equal(run(sizes), want)
    assert torch.equal(run([m]), run([m, 0, 0, 0]))
    with pytest.raises(ValueError, match="at most four"):
        run([m] * 5)


def test_extension_is_rebuilt_for_another_torch(monkeypatch, tmp_path):
    import os
    import subprocess
    from types import SimpleNamespace
    from hecbench_b200 import build
    ext, version = tmp_path / "_host.so", tmp_path / "torch" / "version.py"
    version.parent.mkdir()
    for f in (ext, version):
        f.write_text("")
    t = (build.CSRC / "host" / "host.cpp").stat().st_mtime
    os.utime(ext, (t + 10, t + 10))
    runs = []
    monkeypatch.setattr(build, "HOST_EXT", ext)
    monkeypatch.setattr(torch, "__file__", str(version.parent / "__init__.py"))
    monkeypatch.setattr(subprocess, "run",
                        lambda cmd, **kw: runs.append(cmd) or SimpleNamespace(returncode=0))
    for when, expected in ((t, 0), (t + 20, 1)):
        os.utime(version, (when, when))
        build.build_host()
        assert len(runs) == expected

"""Batched dequant-GEMM on the tensor cores (tcgen05 / tensor memory), 3-bit
and NF4 weights, against the oracle: bit-exact fp16 dequantised weights
(oracle rule) times X in fp64.
No reference implementation exists for this path (parity unpinned); tolerance
1e-2 on |y - ref| / max(|ref|, rms(ref)) for the fp16 output."""
import numpy as np
import pytest

from hecbench_b200 import synth
from conftest import to_dev

pytestmark = pytest.mark.gpu
TOL_F16 = 1e-2


def _run(hq, oracle, dev, Mb, K, N, group, seed):
    import torch
    X, codes, scales, zeros = synth.qgemm_q3_case(Mb, K, N, group, seed)
    mat = synth.q3_pack(codes)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    Y = hq.qgemm_q3(to_dev(X, dev), to_dev(mat, dev), to_dev(scales, dev), to_dev(zeros, dev), N, K,
                    group, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0, "a bounded in-kernel wait ran out"
    W16 = oracle.q3g_dequant_f16(mat, scales, zeros, K, N, group)
    ref = oracle.gemm_f16_f64(X, W16)
    return oracle.rel_err(Y.cpu().numpy().astype(np.float64), ref)


@pytest.mark.parametrize("Mb,K,N,group", [(64, 256, 128, 128), (16, 128, 256, 128),
                                          (64, 1024, 512, 128), (128, 512, 256, 64),
                                          (37, 256, 128, 128), (1, 128, 128, 64)])
def test_qgemm_q3_small(hq, oracle, dev, Mb, K, N, group):
    assert _run(hq, oracle, dev, Mb, K, N, group, seed=Mb + K + N) < TOL_F16


def _run_nf4(hq, oracle, dev, Mb, K, N, blocksize, low_first, seed):
    import torch
    X, B, absmax, lut16 = synth.qgemm_nf4_case(Mb, K, N, blocksize, seed)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    Y = hq.qgemm_nf4(to_dev(X, dev), to_dev(B, dev), to_dev(absmax, dev), to_dev(lut16, dev), N, K,
                     blocksize, low_first, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0, "a bounded in-kernel wait ran out"
    W16 = oracle.nf4_dequant_f16(B, absmax, lut16, N * K, blocksize, low_first).reshape(N, K)
    ref = oracle.gemm_f16_nk_f64(X, W16)
    return oracle.rel_err(Y.cpu().numpy().astype(np.float64), ref)


@pytest.mark.parametrize("Mb,K,N,blocksize,low_first", [
    (64, 256, 128, 64, 0), (16, 128, 256, 64, 1), (64, 1024, 512, 64, 0), (128, 512, 256, 128, 0),
    (37, 768, 128, 256, 1), (1, 128, 128, 64, 0), (64, 4096, 1024, 64, 0), (32, 576, 384, 192, 0)])
def test_qgemm_nf4_small(hq, oracle, dev, Mb, K, N, blocksize, low_first):
    assert _run_nf4(hq, oracle, dev, Mb, K, N, blocksize, low_first, seed=Mb + K + N) < TOL_F16


def test_qgemm_nf4_matches_dequant_then_gemm(hq, dev):
    """Llama-2-7B MLP shape (11008 x 4096): the fused kernel against the library's
    own NF4 dequantisation followed by a dense fp32 product in torch (checker only)."""
    import torch
    Mb, K, N = 64, 4096, 11008
    X, B, absmax, lut16 = synth.qgemm_nf4_case(Mb, K, N, 64, 5)
    dX, dB, dA, dL = (to_dev(a, dev) for a in (X, B, absmax, lut16))
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    Y = hq.qgemm_nf4(dX, dB, dA, dL, N, K, 64, 0, status=status)
    W = hq.dequantize_nf4(dB, dA, dL, N * K, 64, 0).view(N, K)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    ref = dX.float() @ W.float().t()
    err = (Y.float() - ref).abs() / torch.maximum(ref.abs(), ref.pow(2).mean().sqrt())
    assert float(err.max()) < TOL_F16


@pytest.mark.parametrize("Mb,K,N", [(64, 8192, 20480), (33, 8192, 24576), (100, 4096, 12288)])
def test_qgemm_parts_of_k(hq, dev, Mb, K, N):
    """Shapes where the number of parts K is cut into leaves the one that fills the GPU
    once (three parts in two waves; one part beyond 64 tokens), twice on one workspace,
    against the library's own dequantisation and a dense fp32 product in torch."""
    import torch
    X, B, absmax, lut16 = synth.qgemm_nf4_case(Mb, K, N, 64, 7)
    dX, dB, dA, dL = (to_dev(a, dev) for a in (X, B, absmax, lut16))
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    Y = [hq.qgemm_nf4(dX, dB, dA, dL, N, K, 64, 0, status=status) for _ in range(2)]
    W = hq.dequantize_nf4(dB, dA, dL, N * K, 64, 0).view(N, K)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    ref = dX.float() @ W.float().t()
    for y in Y:
        err = (y.float() - ref).abs() / torch.maximum(ref.abs(), ref.pow(2).mean().sqrt())
        assert float(err.max()) < TOL_F16


@pytest.mark.parametrize("fmt", ["q3", "nf4"])
@pytest.mark.parametrize("Mb,K,N", [(64, 8192, 20480), (5, 8192, 24576), (100, 8192, 20480),
                                    (33, 28672, 28672), (128, 28672, 12800)])
def test_qgemm_parts_of_k_repeat(hq, dev, fmt, Mb, K, N):
    """Wide layers (more than two thirds of a tile per SM) in two to five parts of K: the same
    bits from every call, also beside another stream's product and on fresh scratch, and
    the dense fp32 product of the dequantised weights."""
    import torch
    g = torch.Generator(device=dev).manual_seed(K + N)
    X = torch.randn((Mb, K), generator=g, device=dev).half()
    if fmt == "nf4":
        lut = torch.linspace(-1, 1, 16, device=dev)
        B = torch.randint(0, 256, (N, K // 2), generator=g, device=dev, dtype=torch.uint8)
        absmax = torch.rand(N * K // 64, generator=g, device=dev) + 0.5
        W = hq.dequantize_nf4(B, absmax, lut, N * K, 64, 0).view(N, K)
        ref = X.float() @ W.float().t()
        call = lambda: hq.qgemm_nf4(X, B, absmax, lut, N, K, 64, 0, status=status)
    else:
        mat = torch.randint(-2**31, 2**31, (K * 3 // 32, N), generator=g, device=dev).to(torch.int32)
        scales = (torch.rand((K // 128, N), generator=g, device=dev) * 0.01).half()
        zeros = scales * 3.5
        one, zero = torch.ones(N, device=dev), torch.zeros(N, device=dev)
        W = hq.vecquant3_dequant(mat, one, zero, K * 3 // 32, N, dtype=torch.float16)
        W = torch.addcmul(-zeros.float().repeat_interleave(128, 0), W.float(),
                          scales.float().repeat_interleave(128, 0)).half()
        ref = X.float() @ W.float()
        call = lambda: hq.qgemm_q3(X, mat, scales, zeros, N, K, 128, status=status)
    del W
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    first = call()
    err = (first.float() - ref).abs() / torch.maximum(ref.abs(), ref.pow(2).mean().sqrt())
    assert float(err.max()) < TOL_F16
    outs = [call() for _ in range(6)]
    torch.cuda.synchronize()
    for s in (torch.cuda.Stream(), torch.cuda.Stream()):
        with torch.cuda.stream(s):
            outs += [call() for _ in range(3)]
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for y in outs:
        assert torch.equal(y, first)


@pytest.mark.parametrize("fmt,Mb,K,N", [("q3", 64, 8960, 14976), ("q3", 2, 8960, 14976), ("nf4", 64, 8960, 15104)])
def test_qgemm_ordered_parts_of_two_ctas(hq, dev, fmt, Mb, K, N):
    """The few wide layers that stay in more than two parts with one tile per CTA, where the parts add in
    the order of K: the same bits from every call as well."""
    import torch
    from launches import launched
    from test_qgemm_tiles_gpu import _operands
    call, _ = _operands(hq, fmt, K, N, 128, dev, torch.Generator(device=dev).manual_seed(K))
    X = torch.zeros((Mb, K), dtype=torch.float16, device=dev)
    ((name, grid),) = launched(lambda: call(X))
    assert "12qgemm_kernel" in name and grid > 2 * (N // 128)
    test_qgemm_parts_of_k_repeat(hq, dev, fmt, Mb, K, N)


LLAMA3_70B_MLP = [(8192, 28672), (28672, 8192)]  # (K, N): up/gate and down projections


def _feature_subset(N, tiles=4, width=128):
    """`tiles` whole 128-feature tiles spread over [0, N): first, last and evenly between."""
    starts = np.unique(np.linspace(0, N - width, tiles).astype(np.int64) // width * width)
    return np.concatenate([np.arange(s0, s0 + width) for s0 in starts])


@pytest.mark.parametrize("K,N", LLAMA3_70B_MLP)
def test_qgemm_q3_llama3_70b_mlp(hq, oracle, dev, K, N):
    """Batch 64 at the full Llama-3-70B MLP shapes (the second one takes the K-split
    path): 512 output features against the CPU oracle (bit-exact fp16 dequantised
    weights times X in fp64), then every output against a dense fp32 product of
    the dequantised weights computed by torch on the same GPU."""
    import torch
    Mb, group = 64, 128
    X, codes, scales, zeros = synth.qgemm_q3_case(Mb, K, N, group, seed=K % 97)
    mat = synth.q3_pack(codes)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    dX, dS, dZ = to_dev(X, dev), to_dev(scales, dev), to_dev(zeros, dev)
    Y = hq.qgemm_q3(dX, to_dev(mat, dev), dS, dZ, N, K, group, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0, "a bounded in-kernel wait ran out"
    cols = _feature_subset(N)
    W16 = oracle.q3g_dequant_f16(np.ascontiguousarray(mat[:, cols]),
                                 np.ascontiguousarray(scales[:, cols]),
                                 np.ascontiguousarray(zeros[:, cols]), K, cols.size, group)
    ref = oracle.gemm_f16_f64(X, W16)
    got = Y[:, torch.from_numpy(cols).to(dev)].cpu().numpy().astype(np.float64)
    assert oracle.rel_err(got, ref) < TOL_F16
    assert oracle.rel_err_above_floor(got, ref) < TOL_F16
    s = dS.float().repeat_interleave(group, dim=0)
    z = dZ.float().repeat_interleave(group, dim=0)
    W = torch.addcmul(-z, torch.from_numpy(codes).to(dev).float(), s).half().float()
    del s, z
    full = dX.float() @ W
    err = (Y.float() - full).abs() / torch.maximum(full.abs(), full.pow(2).mean().sqrt())
    assert float(err.max()) < TOL_F16


@pytest.mark.parametrize("K,N", LLAMA3_70B_MLP)
def test_qgemm_nf4_llama3_70b_mlp(hq, oracle, dev, K, N):
    """The NF4 operand at the same two shapes: 512 output features against the CPU
    oracle, every output against the library's own bit-exact dequantisation
    followed by a dense fp32 product in torch."""
    import torch
    Mb, bs = 64, 64
    X, B, absmax, lut16 = synth.qgemm_nf4_case(Mb, K, N, bs, seed=K % 89)
    dX, dB, dA, dL = (to_dev(a, dev) for a in (X, B, absmax, lut16))
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    Y = hq.qgemm_nf4(dX, dB, dA, dL, N, K, bs, 0, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0, "a bounded in-kernel wait ran out"
    rows = _feature_subset(N)
    Brows = np.ascontiguousarray(B.reshape(N, K // 2)[rows]).reshape(-1)
    Arows = np.ascontiguousarray(absmax.reshape(N, K // bs)[rows]).reshape(-1)
    W16 = oracle.nf4_dequant_f16(Brows, Arows, lut16, rows.size * K, bs, 0).reshape(rows.size, K)
    ref = oracle.gemm_f16_nk_f64(X, W16)
    got = Y[:, torch.from_numpy(rows).to(dev)].cpu().numpy().astype(np.float64)
    assert oracle.rel_err(got, ref) < TOL_F16
    assert oracle.rel_err_above_floor(got, ref) < TOL_F16
    W = hq.dequantize_nf4(dB, dA, dL, N * K, bs, 0).view(N, K)
    full = dX.float() @ W.float().t()
    err = (Y.float() - full).abs() / torch.maximum(full.abs(), full.pow(2).mean().sqrt())
    assert float(err.max()) < TOL_F16

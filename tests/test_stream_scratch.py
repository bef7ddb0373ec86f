"""Scratch of calls whose partial sums meet in device memory: one per stream, and
none kept from a stream capture."""
from types import SimpleNamespace

import pytest
import torch


@pytest.fixture()
def place(monkeypatch):
    """The fake library's device and stream, on the CPU."""
    from hecbench_b200 import api
    state = SimpleNamespace(where=(0, 1), capturing=False)
    fake = SimpleNamespace(host=SimpleNamespace(place=lambda t: state.where,
                                                capturing=lambda t: state.capturing),
                           hq_lutgemm_workspace_bytes=lambda m: 4 * m,
                           hq_qgemm_workspace_bytes=lambda m, n: 4 * m * n)
    monkeypatch.setattr(api, "load_library", lambda: fake)
    return state


def _weight():
    from hecbench_b200 import api
    return api.nQWeight_fp16(torch.zeros(1 * 1 * 8, dtype=torch.int32), torch.zeros(8), 32, 8, 1,
                             device="cpu")


def test_lutgemm_scratch_per_stream(place):
    w = _weight()
    first = w.workspace()
    assert w.workspace() is first
    place.where = (0, 2)
    other = w.workspace()
    assert other.data_ptr() != first.data_ptr() and not other.any()
    place.where = (0, 1)
    assert w.workspace() is first


def test_lutgemm_scratch_of_a_capture_is_not_kept(place):
    w = _weight()
    place.capturing = True
    a, b = w.workspace(), w.workspace()
    assert a.data_ptr() != b.data_ptr()
    place.capturing = False
    c = w.workspace()
    assert c is not a and c is not b
    place.capturing = True
    assert w.workspace() is c                    # cleared by an eager call on this stream


def test_qgemm_scratch_of_a_capture_is_not_kept(place, monkeypatch):
    from hecbench_b200 import api
    monkeypatch.setattr(api, "_qgemm_ws", {})
    lib, X = api.load_library(), torch.zeros(2, 64)
    place.capturing = True
    a, n = api._qgemm_workspace(lib, X, 2, 128)
    assert n == 4 * 2 * 128
    place.capturing = False
    b, _ = api._qgemm_workspace(lib, X, 2, 128)
    assert b is not a and api._qgemm_workspace(lib, X, 2, 128)[0] is b


@pytest.mark.gpu
def test_one_layer_on_two_streams(hq, dev):
    """Two streams multiply by the same layer at the same time; sums meet in no fixed
    order, which moves an fp16 result by one step at most."""
    M = K = 4096
    g = torch.Generator(device=dev).manual_seed(3)
    words = torch.randint(-2**31, 2**31, (K // 32, 3, M), generator=g, device=dev).to(torch.int32)
    w = hq.nQWeight_fp16(words, torch.rand((K // 128, 3, M), generator=g, device=dev), K, M, 3, False,
                         K // 128, None, device=dev)
    x = torch.randn((2, K), generator=g, device=dev).half()
    want = torch.empty((2, M), dtype=torch.float16, device=dev)
    for i in range(2):
        hq.matmul(want[i], x[i], w)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [[torch.zeros(M, dtype=torch.float16, device=dev) for _ in range(40)] for _ in streams]
    torch.cuda.synchronize()
    for t in range(40):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                hq.matmul(outs[i][t], x[i], w)
    torch.cuda.synchronize()
    for i in range(2):
        for o in outs[i]:
            assert float((o.float() - want[i].float()).norm() / want[i].float().norm()) < 2 ** -10


@pytest.mark.gpu
def test_graph_before_its_stream_has_scratch(hq, dev):
    """A graph captured on a stream that never multiplied by the layer, then an eager
    call there before the graph has run: neither finds the other's scratch."""
    M, K = 1024, 1024
    g = torch.Generator(device=dev).manual_seed(4)
    words = torch.randint(-2**31, 2**31, (K // 32, 3, M), generator=g, device=dev).to(torch.int32)
    w = hq.nQWeight_fp16(words, torch.rand((K // 128, 3, M), generator=g, device=dev), K, M, 3, False,
                         K // 128, None, device=dev)
    x = torch.randn(K, generator=g, device=dev).half()
    want, eager, replayed = (torch.zeros(M, dtype=torch.float16, device=dev) for _ in range(3))
    hq.matmul(want, x, w)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            hq.matmul(replayed, x, w)
        hq.matmul(eager, x, w)
        graph.replay()
        graph.replay()
    torch.cuda.synchronize()
    for o in (eager, replayed):
        assert float((o.float() - want.float()).norm() / want.float().norm()) < 2 ** -10


@pytest.mark.gpu
def test_qgemm_graph_before_its_stream_has_scratch(hq, dev):
    """As above for the batched product with K split over several CTAs."""
    Mb, K, N = 16, 4096, 640
    g = torch.Generator(device=dev).manual_seed(6)
    X = torch.randn((Mb, K), generator=g, device=dev).half()
    B = torch.randint(0, 256, (N, K // 2), generator=g, device=dev, dtype=torch.uint8)
    absmax = torch.rand(N * K // 64, generator=g, device=dev)
    args = (X, B, absmax, torch.linspace(-1, 1, 16, device=dev), N, K, 64)
    want = hq.qgemm_nf4(*args)
    eager, replayed = torch.zeros_like(want), torch.zeros_like(want)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            hq.qgemm_nf4(*args, out=replayed)
        hq.qgemm_nf4(*args, out=eager)
        graph.replay()
        graph.replay()
    torch.cuda.synchronize()
    for o in (eager, replayed):
        assert float((o.float() - want.float()).norm() / want.float().norm()) < 2 ** -10

"""Which of the library's kernels a call launches, read from a stream capture of it (nothing runs then)."""


def launched(call):
    """[(mangled name, grid blocks)] of the kernels of call(), in no fixed order; a fill of fresh
    scratch is not among them."""
    import torch
    from cuda.bindings import driver

    def done(result):
        assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
        return result[1:]

    call()  # first use: attributes set, scratch in place
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    (_, count) = done(driver.cuGraphGetNodes(raw))
    (nodes, _) = done(driver.cuGraphGetNodes(raw, count))
    found = []
    for node in nodes:
        if done(driver.cuGraphNodeGetType(node))[0] != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        (p,) = done(driver.cuGraphKernelNodeGetParams(node))
        (name,) = done(driver.cuFuncGetName(p.func) if int(p.func) else driver.cuKernelGetName(p.kern))
        if name.startswith(b"_ZN2hq"):
            found.append((name.decode(), p.gridDimX * p.gridDimY * p.gridDimZ))
    return found

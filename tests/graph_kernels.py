"""Which kernels a call queues, by the sizes of their blocks: the call is captured and not run."""


def block_sizes(eng, call):
    """Threads a block of every kernel that call() queues on the engine's stream, which this replaces by one of its own."""
    import torch
    from cuda.bindings import driver
    stream = torch.cuda.Stream()
    eng.set_stream(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        call()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    _, _, n = driver.cuGraphGetNodes(raw)
    _, nodes, n = driver.cuGraphGetNodes(raw, n)
    out = []
    for node in nodes[:n]:
        err, kind = driver.cuGraphNodeGetType(node)
        assert err == driver.CUresult.CUDA_SUCCESS
        if kind == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            err, p = driver.cuGraphKernelNodeGetParams(node)
            assert err == driver.CUresult.CUDA_SUCCESS
            out.append(p.blockDimX)
    return out

"""Which of the library's kernels a call launches: the call is captured into a
CUDA graph and the graph's kernel nodes are named.  The call runs once before,
so that scratch memory and kernel attributes exist."""


def kernel_names(call):
    import torch
    from cuda.bindings import driver

    def ok(result):
        assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
        return result[1:] if len(result) > 2 else result[1]

    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    count = ok(driver.cuGraphGetNodes(raw))[1]
    names = []
    for node in ok(driver.cuGraphGetNodes(raw, count))[0]:
        if ok(driver.cuGraphNodeGetType(node)) != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        params = ok(driver.cuGraphKernelNodeGetParams(node))
        if int(params.func):
            names.append(ok(driver.cuFuncGetName(params.func)).decode())
        else:
            names.append(ok(driver.cuKernelGetName(params.kern)).decode())
    return names

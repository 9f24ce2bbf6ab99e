"""The kernels that a call launches, with their grids and blocks, read from a capture of it."""


def launches(be, call):
    from cuda.bindings import driver as cu

    def ok(result):
        assert result[0] == cu.CUresult.CUDA_SUCCESS, result
        return result[1] if len(result) == 2 else result[1:]

    ok(cu.cuStreamBeginCapture(be.stream(), cu.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED))
    try:
        call()
    finally:
        graph = ok(cu.cuStreamEndCapture(be.stream()))
    count = ok(cu.cuGraphGetNodes(graph))[1]
    nodes = ok(cu.cuGraphGetNodes(graph, count))[0]
    got = []
    for node in nodes:
        if ok(cu.cuGraphNodeGetType(node)) == cu.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            p = ok(cu.cuGraphKernelNodeGetParams(node))
            got.append(([p.gridDimX, p.gridDimY, p.gridDimZ], p.blockDimX * p.blockDimY * p.blockDimZ))
    cu.cuGraphDestroy(graph)
    return got

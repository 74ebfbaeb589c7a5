"""The kernel launches that a call enqueues, from a captured CUDA graph."""


def kernels_of(torch, call):
    """Runs `call` (which must not allocate from torch) once, then captures it; returns its kernel launches as dicts
    (name, grid, block, shared bytes, registers, blocks resident per SM)."""
    from cuda.bindings import driver

    def ok(r):
        assert r[0] == driver.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]

    call()
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        ok(driver.cuStreamBeginCapture(s.cuda_stream, driver.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL))
        try:
            call()
        finally:
            graph = ok(driver.cuStreamEndCapture(s.cuda_stream))
    out = []
    _, n = ok(driver.cuGraphGetNodes(graph))
    for node in ok(driver.cuGraphGetNodes(graph, n))[0]:
        if ok(driver.cuGraphNodeGetType(node)) != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        p = ok(driver.cuGraphKernelNodeGetParams(node))
        block = p.blockDimX * p.blockDimY * p.blockDimZ
        func = p.func if int(p.func) else ok(driver.cuKernelGetFunction(p.kern))
        name = ok(driver.cuFuncGetName(func))
        out.append(dict(name=name.decode() if isinstance(name, bytes) else name,
                        grid=(p.gridDimX, p.gridDimY, p.gridDimZ), block=block, smem=p.sharedMemBytes,
                        regs=ok(driver.cuFuncGetAttribute(driver.CUfunction_attribute.CU_FUNC_ATTRIBUTE_NUM_REGS,
                                                          func)),
                        per_sm=ok(driver.cuOccupancyMaxActiveBlocksPerMultiprocessor(func, block,
                                                                                     p.sharedMemBytes))))
    driver.cuGraphDestroy(graph)
    return out

"""Which kernels a call launches, from a graph that captured it (test infrastructure)."""
from __future__ import annotations

import torch


def launches(call):
    """(name, CTAs, bytes of dynamic shared memory) of every kernel of a call, in the order of the graph's nodes."""
    from cuda.bindings import driver

    def ok(result):
        assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
        return result[1:]

    call()   # what the first call on new parameters copies and loads stays out
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    count = ok(driver.cuGraphGetNodes(raw))[1]
    found = []
    for node in ok(driver.cuGraphGetNodes(raw, count))[0]:
        if ok(driver.cuGraphNodeGetType(node))[0] != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        p = ok(driver.cuGraphKernelNodeGetParams(node))[0]
        name = ok(driver.cuFuncGetName(p.func))[0] if int(p.func) else ok(driver.cuKernelGetName(p.kern))[0]
        found.append((name.decode(), p.gridDimX * p.gridDimY * p.gridDimZ, p.sharedMemBytes))
    return found

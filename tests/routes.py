"""Which kernels a call launches, and how: the call is captured into a CUDA graph, and the graph's kernel nodes are read."""
import ctypes as C
import re

import torch


def kernels(call, stream=None, full=False):
    """``call()`` captured: the launched kernels in order as (name, grid size, launched beside its predecessor) and the number of other nodes.
    "Beside": the only edge into the node is a programmatic one (programmatic stream serialization). full: mangled names, which tell a template's instances apart."""
    from cuda.bindings import driver as cu

    def ok(r):
        assert int(r[0]) == 0, r[0]
        return r[1:] if len(r) > 2 else (r[1] if len(r) == 2 else None)

    stream = stream or torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):                                         # first-use set-up (the stream's workspace) outside the capture
        call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        call()
    raw = cu.CUgraph(graph.raw_cuda_graph())
    n = int(ok(cu.cuGraphGetNodes(raw, 0))[1])
    nodes = ok(cu.cuGraphGetNodes(raw, n))[0]
    # the edges and their types (eight bytes each: source port, target port, type), straight from the driver
    lib, count = C.CDLL("libcuda.so.1"), C.c_size_t(0)
    assert lib.cuGraphGetEdges_v2(C.c_void_p(int(raw)), None, None, None, C.byref(count)) == 0
    m = count.value
    sources, targets, data = (C.c_void_p * max(m, 1))(), (C.c_void_p * max(m, 1))(), (C.c_ubyte * (8 * max(m, 1)))()
    if m:
        assert lib.cuGraphGetEdges_v2(C.c_void_p(int(raw)), sources, targets, data, C.byref(count)) == 0
    into = {}
    for i in range(m):
        into.setdefault(targets[i], []).append(data[8 * i + 2])
    found, others = [], 0
    for node in nodes:
        if ok(cu.cuGraphNodeGetType(node)) != cu.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            others += 1
            continue
        p = ok(cu.cuGraphKernelNodeGetParams(node))
        name = ok(cu.cuKernelGetName(p.kern) if int(p.kern) else cu.cuFuncGetName(p.func)).decode()
        short = re.search(r"\d+([a-z_]+_kernel)", name)
        edges = into.get(int(node), [])
        beside = bool(edges) and all(kind == 1 for kind in edges)
        found.append((short.group(1) if short and not full else name, p.gridDimX * p.gridDimY * p.gridDimZ, beside))
    return found, others


def names(call):
    return [k for k, _, _ in kernels(call)[0]]

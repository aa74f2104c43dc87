"""What a call launches, from the graph that it is captured into: the kernels' names, and how each depends on the one before."""
import ctypes as C

import torch

EDGE_PLAIN, EDGE_PROGRAMMATIC = 0, 1                      # CUgraphDependencyType


class _KernelParams(C.Structure):                         # CUDA_KERNEL_NODE_PARAMS
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("shared", C.c_uint), ("params", C.c_void_p),
                ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


class _EdgeData(C.Structure):                             # CUgraphEdgeData
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]


def captured(call):
    """(kernel names in the order of their launches, types of the edges between nodes) of what `call` enqueues on the current stream."""
    cu = C.CDLL("libcuda.so.1")

    def ok(status, what):
        assert status == 0, f"{what}: {status}"
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw, n = C.c_void_p(graph.raw_cuda_graph()), C.c_size_t(0)
    ok(cu.cuGraphGetNodes(raw, None, C.byref(n)), "cuGraphGetNodes")
    nodes = (C.c_void_p * n.value)()
    ok(cu.cuGraphGetNodes(raw, nodes, C.byref(n)), "cuGraphGetNodes")
    names = []
    for node in nodes:
        kind = C.c_int()
        ok(cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)), "cuGraphNodeGetType")
        if kind.value != 0:                               # CU_GRAPH_NODE_TYPE_KERNEL
            continue
        p, name = _KernelParams(), C.c_char_p()
        ok(cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)), "cuGraphKernelNodeGetParams")
        if p.func:
            ok(cu.cuFuncGetName(C.byref(name), C.c_void_p(p.func)), "cuFuncGetName")
        else:
            ok(cu.cuKernelGetName(C.byref(name), C.c_void_p(p.kern)), "cuKernelGetName")
        names.append(name.value.decode())
    m = C.c_size_t(0)
    ok(cu.cuGraphGetEdges_v2(raw, None, None, None, C.byref(m)), "cuGraphGetEdges")
    edges = (_EdgeData * max(m.value, 1))()
    if m.value:
        a, b = (C.c_void_p * m.value)(), (C.c_void_p * m.value)()
        ok(cu.cuGraphGetEdges_v2(raw, a, b, edges, C.byref(m)), "cuGraphGetEdges")
    return names, [e.type for e in edges[:m.value]]

"""What a call launches: the kernels of its captured graph with their grids, read back from the driver."""
import ctypes as C

import torch


class _Params(C.Structure):  # CUDA_KERNEL_NODE_PARAMS
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("smem", C.c_uint), ("args", C.c_void_p), ("extra", C.c_void_p),
                ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def launches(call):
    """[(kernel's mangled name, grid), ..] of call(stream); it has run once outside a graph before"""
    cu = C.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, rc
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call(torch.cuda.current_stream().cuda_stream)
    raw, n = C.c_void_p(graph.raw_cuda_graph()), C.c_size_t()
    ok(cu.cuGraphGetNodes(raw, None, C.byref(n)))
    nodes, found = (C.c_void_p * n.value)(), []
    ok(cu.cuGraphGetNodes(raw, nodes, C.byref(n)))
    for node in nodes:
        kind, p, name = C.c_int(), _Params(), C.c_char_p()
        ok(cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)))
        if kind.value != 0:  # CU_GRAPH_NODE_TYPE_KERNEL
            continue
        ok(cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)))
        ok(cu.cuKernelGetName(C.byref(name), C.c_void_p(p.kern)) if p.kern else cu.cuFuncGetName(C.byref(name), C.c_void_p(p.func)))
        found.append((name.value.decode(), tuple(p.grid)))
    return found

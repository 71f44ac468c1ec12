"""Kernels of a CUDA graph, read through the driver: what a call would launch, without running it."""
import ctypes as C


class KernelNode(C.Structure):
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("shared", C.c_uint), ("params", C.c_void_p), ("extra", C.c_void_p),
                ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def graph_kernels(graph):
    cu, n = C.CDLL("libcuda.so.1"), C.c_size_t(0)
    assert cu.cuGraphGetNodes(graph, None, C.byref(n)) == 0
    nodes, kernels, kind = (C.c_void_p * n.value)(), [], C.c_int(-1)
    assert n.value == 0 or cu.cuGraphGetNodes(graph, nodes, C.byref(n)) == 0
    for node in nodes:
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        if kind.value == 0:
            kernels.append(KernelNode())
            assert cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(kernels[-1])) == 0
    return kernels

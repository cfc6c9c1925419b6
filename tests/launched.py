"""Which kernels a call launches: tests of a route check that it was taken."""

import ctypes

import torch


class _KernelNodeParams(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("shared_bytes", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def _demangled(name: bytes) -> str:
    demangle = ctypes.CDLL("libstdc++.so.6").__cxa_demangle
    demangle.restype, demangle.argtypes = ctypes.c_void_p, [ctypes.c_char_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    text = demangle(name, None, None, None)
    return ctypes.string_at(text).decode() if text else name.decode()


def graph_of(fn):
    """fn captured on a stream of its own after a call outside of the capture: the graph and what fn returned in it."""
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        res = fn()
    return graph, res


def kernels(fn):
    """What fn() returns, and the names of the kernels it launches, read from the nodes of a captured graph.  (A profile
    would do, but now and then, and then again and again, the profiler hands back one without a single record.)"""
    res = fn()
    graph, _ = graph_of(fn)
    cuda = ctypes.CDLL("libcuda.so.1")
    handle, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cuda.cuGraphGetNodes(handle, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert cuda.cuGraphGetNodes(handle, nodes, ctypes.byref(n)) == 0
    names = []
    for node in nodes:
        kind, params, name = ctypes.c_int(-1), _KernelNodeParams(), ctypes.c_char_p()
        assert cuda.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value != 0:  # not a kernel
            continue
        assert cuda.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(params)) == 0
        if params.kern:
            assert cuda.cuKernelGetName(ctypes.byref(name), ctypes.c_void_p(params.kern)) == 0
        else:
            assert cuda.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(params.func)) == 0
        names.append(_demangled(name.value))
    graph.reset()
    torch.cuda.synchronize()
    return res, names

"""Which kernels a call launches: read from a CUDA graph that it is captured into."""
import ctypes

import torch


class _KernelNode(ctypes.Structure):               # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", ctypes.c_void_p), ("shape", ctypes.c_uint * 7), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def kernels(call):
    """Mangled names of the kernels that `call()` launches on the current stream, template arguments included (`ILi4ELb0EE`)."""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        call()                                     # (attributes are set and workspaces made by first calls)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        call()
    cu = ctypes.CDLL("libcuda.so.1")
    handle, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cu.cuGraphGetNodes(handle, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(handle, nodes, ctypes.byref(n)) == 0
    names = []
    for node in nodes:
        kind, p, name = ctypes.c_int(-1), _KernelNode(), ctypes.c_char_p()
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value == 0:                        # CU_GRAPH_NODE_TYPE_KERNEL
            assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(p)) == 0
            get, what = (cu.cuFuncGetName, p.func) if p.func else (cu.cuKernelGetName, p.kern)
            assert get(ctypes.byref(name), ctypes.c_void_p(what)) == 0
            names.append(name.value.decode())
    return names

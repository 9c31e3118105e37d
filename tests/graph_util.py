"""What calls launch, read from a graph that they are captured into: no profiler, whose records depend on its clocks."""
import contextlib
import ctypes

import torch

KERNEL, MEMCPY = 0, 1  # CUgraphNodeType


class _KernelParams(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3), ("shared", ctypes.c_uint),
                ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p), ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


@contextlib.contextmanager
def _captured(calls):
    cu = ctypes.CDLL("libcuda.so.1")
    side = torch.cuda.Stream()
    stream, graph = ctypes.c_void_p(side.cuda_stream), ctypes.c_void_p()
    torch.cuda.synchronize()
    assert cu.cuStreamBeginCapture_v2(stream, 2) == 0  # CU_STREAM_CAPTURE_MODE_RELAXED
    with torch.cuda.stream(side):
        for call in calls:
            call()
    assert cu.cuStreamEndCapture(stream, ctypes.byref(graph)) == 0
    try:
        yield cu, graph
    finally:
        cu.cuGraphDestroy(graph)


def nodes(*calls):
    """(type, kernel's name, its grid) of each node that the calls are captured as."""
    with _captured(calls) as (cu, graph):
        n, out = ctypes.c_size_t(16), []
        found = (ctypes.c_void_p * 16)()
        assert cu.cuGraphGetNodes(graph, found, ctypes.byref(n)) == 0
        for node in list(found)[:n.value]:
            kind, p, name = ctypes.c_int(), _KernelParams(), ctypes.c_char_p()
            assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
            if kind.value != KERNEL:
                out.append((kind.value, "", None))
                continue
            assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(p)) == 0
            get, which = (cu.cuFuncGetName, p.func) if p.func else (cu.cuKernelGetName, p.kern)
            assert get(ctypes.byref(name), ctypes.c_void_p(which)) == 0
            out.append((KERNEL, name.value.decode(), tuple(p.grid)))
        return out


def edge_types(*calls):
    """What connects the nodes of these calls: 0 a full dependency, 1 one that lets the second kernel come up early."""
    with _captured(calls) as (cu, graph):
        n = ctypes.c_size_t(16)
        ends, data = [(ctypes.c_void_p * 16)() for _ in range(2)], (ctypes.c_ubyte * 8 * 16)()  # CUgraphEdgeData: its third byte is the type
        assert cu.cuGraphGetEdges_v2(graph, ends[0], ends[1], data, ctypes.byref(n)) == 0
        return [data[i][2] for i in range(n.value)]

"""Captures a call into a CUDA graph through the driver API and lists the kernels it launched: what a call launches is then
read from the driver instead of from the library's own claims."""
import ctypes as C


class _KernelParams(C.Structure):
    """CUDA_KERNEL_NODE_PARAMS_v2"""
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("shared", C.c_uint),
                ("params", C.c_void_p), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def _ok(rc, what):
    assert rc == 0, f"{what}: driver error {rc}"


def captured_kernels(call):
    """[(name, grid)] of the kernels that `call(stream)` launches on `stream`; it is run once before, uncaptured (set-up)."""
    import torch
    cu = C.CDLL("libcuda.so.1")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    call(stream.cuda_stream)
    stream.synchronize()
    graph = C.c_void_p()
    _ok(cu.cuStreamBeginCapture_v2(C.c_void_p(stream.cuda_stream), 1), "begin capture")       # 1: thread-local mode
    try:
        call(stream.cuda_stream)
    finally:
        rc = cu.cuStreamEndCapture(C.c_void_p(stream.cuda_stream), C.byref(graph))
    _ok(rc, "end capture")
    n = C.c_size_t()
    _ok(cu.cuGraphGetNodes(graph, None, C.byref(n)), "node count")
    nodes = (C.c_void_p * n.value)()
    _ok(cu.cuGraphGetNodes(graph, nodes, C.byref(n)), "nodes")
    found = []
    for node in nodes:
        kind = C.c_int()
        _ok(cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)), "node type")
        if kind.value != 0:                                                                   # 0: kernel
            continue
        p, name = _KernelParams(), C.c_char_p()
        _ok(cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)), "node parameters")
        if p.kern:
            _ok(cu.cuKernelGetName(C.byref(name), C.c_void_p(p.kern)), "kernel name")
        else:
            _ok(cu.cuFuncGetName(C.byref(name), C.c_void_p(p.func)), "function name")
        found.append((name.value.decode(), tuple(p.grid)))
    _ok(cu.cuGraphDestroy(graph), "destroy")
    return found

"""What a call launches, read from a capture of it (nothing runs)."""
import ctypes


class _KernelParams(ctypes.Structure):
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("smem", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


NODE_KERNEL, NODE_MEM_ALLOC = 0, 10


def captured(torch, call):
    """call(stream) captured: ([(kernel name, CTAs, threads per CTA)], memory nodes)."""
    cu = ctypes.CDLL("libcuda.so.1")

    def check(rc):
        assert rc == 0, rc

    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    handle, graph = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p()
    check(cu.cuStreamBeginCapture_v2(handle, 1))  # thread-local
    try:
        call(stream)
    finally:
        rc = cu.cuStreamEndCapture(handle, ctypes.byref(graph))
    check(rc)
    count = ctypes.c_size_t()
    check(cu.cuGraphGetNodes(graph, None, ctypes.byref(count)))
    nodes = (ctypes.c_void_p * max(1, count.value))()
    check(cu.cuGraphGetNodes(graph, nodes, ctypes.byref(count)))
    kernels, allocs = [], 0
    for node in nodes[:count.value]:
        kind = ctypes.c_int()
        check(cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)))
        allocs += kind.value == NODE_MEM_ALLOC
        if kind.value != NODE_KERNEL:
            continue
        p, name = _KernelParams(), ctypes.c_char_p()
        check(cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(p)))
        if p.func:
            check(cu.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(p.func)))
        else:
            check(cu.cuKernelGetName(ctypes.byref(name), ctypes.c_void_p(p.kern)))
        kernels.append((name.value.decode(), p.grid[0], p.block[0]))
    check(cu.cuGraphDestroy(graph))
    return kernels, allocs

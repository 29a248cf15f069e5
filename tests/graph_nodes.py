"""What a call launches, read off the nodes of a captured graph."""
import ctypes as C
from collections import namedtuple

import torch

Kernel = namedtuple("Kernel", "name grid block ctas_per_sm")


class _Params(C.Structure):
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("shared", C.c_uint), ("params", C.c_void_p),
                ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def kernels(fn):
    """Name, CTAs, threads a CTA and CTAs that fit an SM, of every kernel that fn launches."""
    cu = C.CDLL("libcuda.so.1")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g, stream=stream):
            fn()
        n, raw = C.c_size_t(0), C.c_void_p(g.raw_cuda_graph())
        assert cu.cuGraphGetNodes(raw, None, C.byref(n)) == 0
        nodes = (C.c_void_p * n.value)()
        assert cu.cuGraphGetNodes(raw, nodes, C.byref(n)) == 0
        out = []
        for node in nodes:
            p, name, per_sm = _Params(), C.c_char_p(), C.c_int(0)
            if cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)) != 0:
                continue
            func = C.c_void_p(p.func)
            if not p.func:
                assert cu.cuKernelGetFunction(C.byref(func), C.c_void_p(p.kern)) == 0
            assert cu.cuFuncGetName(C.byref(name), func) == 0
            assert cu.cuOccupancyMaxActiveBlocksPerMultiprocessor(C.byref(per_sm), func, C.c_int(p.block[0]), C.c_size_t(p.shared)) == 0
            out.append(Kernel(name.value.decode(), p.grid[0], p.block[0], per_sm.value))
    torch.cuda.synchronize()
    return out

"""Kernel launches read from a captured CUDA graph (driver API)."""
import ctypes as C
import re

KERNEL, MEMSET, PROGRAMMATIC = 0, 2, 1


class NodeParams(C.Structure):  # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", C.c_void_p), ("dims", C.c_uint * 7), ("params", C.c_void_p), ("extra", C.c_void_p),
                ("kern", C.c_void_p), ("ctx", C.c_void_p)]


class Edge(C.Structure):  # CUgraphEdgeData
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]


def captured(fn):
    """Captures fn(stream); returns {node: (kind, name, [(dependency, edge type)], (grid, block))}."""
    import torch
    cu = C.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, f"driver call failed: {rc}"

    st = torch.cuda.Stream()
    graph = C.c_void_p()
    ok(cu.cuStreamBeginCapture_v2(C.c_void_p(st.cuda_stream), 1))
    fn(st)
    ok(cu.cuStreamEndCapture(C.c_void_p(st.cuda_stream), C.byref(graph)))
    n = C.c_size_t()
    ok(cu.cuGraphGetNodes(graph, None, C.byref(n)))
    nodes = (C.c_void_p * n.value)()
    ok(cu.cuGraphGetNodes(graph, nodes, C.byref(n)))
    out = {}
    for v in nodes:
        kind, name, dims = C.c_int(), "", None
        ok(cu.cuGraphNodeGetType(C.c_void_p(v), C.byref(kind)))
        if kind.value == KERNEL:
            prm, s = NodeParams(), C.c_char_p()
            ok(cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(v), C.byref(prm)))
            if prm.func:
                ok(cu.cuFuncGetName(C.byref(s), C.c_void_p(prm.func)))
            else:
                ok(cu.cuKernelGetName(C.byref(s), C.c_void_p(prm.kern)))
            name, dims = s.value.decode(), (prm.dims[0], prm.dims[3])
        m = C.c_size_t(64)
        deps, edges = (C.c_void_p * 64)(), (Edge * 64)()
        ok(cu.cuGraphNodeGetDependencies_v2(C.c_void_p(v), deps, edges, C.byref(m)))
        out[v] = (kind.value, name, [(deps[i], edges[i].type) for i in range(m.value)], dims)
    ok(cu.cuGraphDestroy(graph))
    return out


def row_launches(fn):
    """(template arguments, grid, block) of the row kernels fn(stream) launches, in order."""
    out = []
    for kind, name, _, dims in captured(fn).values():
        if "k_bluestein_rows" in name:
            out.append((tuple(int(x) for x in re.findall(r"L[ib](\d+)E", name)), *dims))
    return out


def kernel_names(fn):
    return [name for _, name, _, _ in captured(fn).values() if name]

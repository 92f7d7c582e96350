"""What a batch's kernels wait for, read from a captured graph.

Row kernels read the sums pass 1 wrote, so each needs an edge from every
pass-1 kernel of its batch; classes of rows run beside one another, so none
may lean on another class's wait.  A programmatic edge is a wait only in
kernels that execute griddepcontrol.wait before their first read, which the
row kernels do.
"""
import ctypes as C

import numpy as np
import pytest

import cuspfft_gb300 as gb
from cuspfft_gb300 import synthetic

pytestmark = pytest.mark.gpu

KERNEL, MEMSET, PROGRAMMATIC = 0, 2, 1


class NodeParams(C.Structure):  # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", C.c_void_p), ("dims", C.c_uint * 7), ("params", C.c_void_p), ("extra", C.c_void_p),
                ("kern", C.c_void_p), ("ctx", C.c_void_p)]


class Edge(C.Structure):  # CUgraphEdgeData
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]


def captured(fn):
    """Captures fn(stream); returns {node: (kind, name, [(dependency, edge type)])}."""
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
        kind, name = C.c_int(), ""
        ok(cu.cuGraphNodeGetType(C.c_void_p(v), C.byref(kind)))
        if kind.value == KERNEL:
            prm, s = NodeParams(), C.c_char_p()
            ok(cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(v), C.byref(prm)))
            if prm.func:
                ok(cu.cuFuncGetName(C.byref(s), C.c_void_p(prm.func)))
            else:
                ok(cu.cuKernelGetName(C.byref(s), C.c_void_p(prm.kern)))
            name = s.value.decode()
        m = C.c_size_t(64)
        deps, edges = (C.c_void_p * 64)(), (Edge * 64)()
        ok(cu.cuGraphNodeGetDependencies_v2(C.c_void_p(v), deps, edges, C.byref(m)))
        out[v] = (kind.value, name, [(deps[i], edges[i].type) for i in range(m.value)])
    ok(cu.cuGraphDestroy(graph))
    return out


SHAPES = {
    "fp32": [(900, 2048), (1500, 257), (700, 1024), (300, 3500), (401, 4603), (3000, 31)],
    "both": [(900, 2048), (1500, 257), (6001, 133), (4100, 51), (401, 4603), (9001, 3000)],
    "one": [(500, 500), (500, 500)],
}


@pytest.mark.parametrize("shapes", list(SHAPES))
def test_batch_rows_depend_on_pass_1_themselves(cuda, shapes):
    mats = [synthetic.uniform_matrix(r, c, 8 * max(r, c), seed=c) for r, c in SHAPES[shapes]]
    with gb.Batch(mats, length_policy=gb.GBSP_LEN_7SMOOTH) as b:
        outs = b.empty_outputs()
        b.set_outputs(outs)
        g = captured(lambda st: b.execute(stream=st))
    pass1 = {v for v, (_, name, _) in g.items() if "k_twiddle" in name}
    rows = {v for v, (_, name, _) in g.items() if "k_bluestein_rows_batch" in name}
    assert len(pass1) == (2 if shapes == "both" else 1) and len(rows) >= (1 if shapes == "one" else 2)
    assert len(g) == len(pass1) + len(rows) + 1  # and the queues' memset
    for v in pass1:
        assert [(g[d][0], t) for d, t in g[v][2]] == [(MEMSET, 0)]
    for v in rows:
        assert {d for d, _ in g[v][2]} == pass1
    # the first class alone may start early, and only where one kernel is ahead of it
    early = [v for v in rows if any(t == PROGRAMMATIC for _, t in g[v][2])]
    assert len(early) <= (0 if shapes == "both" else 1)


def test_batch_classes_replay_to_the_same_bits(cuda):
    import torch
    mats = [synthetic.uniform_matrix(r, c, 8 * max(r, c), seed=c) for r, c in
            SHAPES["both"] + SHAPES["fp32"] + [(2001, 16706)]]
    with gb.Batch(mats, length_policy=gb.GBSP_LEN_7SMOOTH) as b:
        outs = b.empty_outputs()
        b.set_outputs(outs)
        b.execute()
        torch.cuda.synchronize()
        want = [o.clone() for o in outs]
        for launch in (b.execute, b.graph_launch, b.graph_launch):
            for o in outs:
                o.fill_(complex(np.nan, np.nan))
            launch()
            torch.cuda.synchronize()
            assert b.error_flags() == 0
            assert all(torch.equal(o, w) for o, w in zip(outs, want))
        for coo, o in zip(mats, outs):
            with gb.Plan(coo, length_policy=gb.GBSP_LEN_7SMOOTH) as p:
                one = p.empty_output()
                p.execute(one)
                torch.cuda.synchronize()
                assert torch.equal(one, o)

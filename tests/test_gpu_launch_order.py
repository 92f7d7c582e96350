"""What kernels wait for, read from captured graphs.

Row kernels read the sums pass 1 wrote, so each needs an edge from every
pass-1 kernel of its batch; classes of rows run beside one another, so none
may lean on another class's wait.  A programmatic edge is a wait only in
kernels that execute griddepcontrol.wait before their first read, which the
row kernels do.
"""
import numpy as np
import pytest

import cuspfft_gb300 as gb
from cuspfft_gb300 import synthetic
from graph_nodes import MEMSET, PROGRAMMATIC, captured

pytestmark = pytest.mark.gpu

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
    pass1 = {v for v, (_, name, _, _) in g.items() if "k_twiddle" in name}
    rows = {v for v, (_, name, _, _) in g.items() if "k_bluestein_rows_batch" in name}
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


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


# rows, columns: a small launch, one CTA an SM, rows that fill whole rounds; and
# rows that would crowd on some SMs, a long launch, clusters
@pytest.mark.parametrize("n,cols,kw,early", [
    (151, 257, {}, True), (100, 8219, {}, True), (1000, 8219, {}, True), ("2", 5003, {}, True), ("4", 5003, {}, True),
    (151, 1201, {}, True), (151, 3163, {}, True), (1001, 5003, {}, False), (1001, 601, {}, False), (76, 11003, {}, False),
    (4000, 16706, {}, False),
    (151, 40421, dict(channel_mode=1), False)])
def test_rows_start_early_only_where_they_spread(cuda, n, cols, kw, early):
    n = n if isinstance(n, int) else int(n) * sms()
    coo = synthetic.uniform_matrix(2 * (n - 1), cols, 3 * cols, seed=cols)
    with gb.Plan(coo, length_policy=gb.GBSP_LEN_7SMOOTH, **kw) as p:
        assert p.info["half_rows"] == n
        out = p.empty_output()
        g = captured(lambda st: p.execute(out, stream=st))
    [deps] = [d for _, name, d, _ in g.values() if "k_bluestein_rows" in name]
    assert len(deps) == 1 and "k_twiddle" in g[deps[0][0]][1]
    assert (deps[0][1] == PROGRAMMATIC) == early


def test_execute_is_captured_after_any_node(cuda):
    # pass 1 carries the attribute of an early start: after a copy, a memset, a join of two streams, a batch
    import torch
    coo = synthetic.uniform_matrix(301, 257, 4000, seed=1)
    mats = [synthetic.uniform_matrix(r, c, 8 * max(r, c), seed=c) for r, c in SHAPES["both"]]
    with gb.Plan(coo) as p, gb.Batch(mats) as b:
        want, out, aux = p.empty_output(), p.empty_output(), torch.zeros(1 << 20, device="cuda")
        bout = b.empty_outputs()
        b.set_outputs(bout)
        p.execute(want)
        torch.cuda.synchronize()
        side = torch.cuda.Stream()

        def memset(st):
            aux.zero_()

        def copy(st):
            aux[: 1 << 19].copy_(aux[1 << 19:])

        def join(st):
            side.wait_stream(st)
            with torch.cuda.stream(side):
                aux.add_(1.0)
            aux.new_ones(8)
            st.wait_stream(side)

        def batch(st):
            b.execute(stream=st)

        for before in (memset, copy, join, batch):
            graph = torch.cuda.CUDAGraph()
            out.fill_(complex(np.nan, np.nan))
            torch.cuda.synchronize()
            with torch.cuda.graph(graph):
                before(torch.cuda.current_stream())
                p.execute(out)
                p.execute(out)
            for _ in range(2):
                out.fill_(complex(np.nan, np.nan))
                graph.replay()
                torch.cuda.synchronize()
                assert torch.equal(out, want), before.__name__
        assert p.error_flags() == 0 and b.error_flags() == 0

"""Which block, grid and instance a row launch gets, read from a captured graph.

Short rows run 32, 64 or 128 threads each where that gives every SM 320
threads, and wider blocks where there are fewer rows; the rows are those of the
launch, not of the plan.
"""
import numpy as np
import pytest

import cuspfft_gb300 as gb
from cuspfft_gb300 import synthetic
from graph_nodes import row_launches
from oracle import fp64

pytestmark = pytest.mark.gpu


def sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("full,last", [(16, 16), (16, 9), (16, 5), (16, 1), (8, 7), (8, 3), (4, 1)])
def test_a_short_tile_gets_a_wider_block(cuda, full, last):
    import torch
    n = sms()
    tile, tail = full * n, last * n + 3
    rows, cols = 2 * (tile + tail - 1), 257  # tiles of `tile` and `tail` Bluestein rows
    coo = synthetic.uniform_matrix(rows, cols, 4 * rows, seed=rows)
    with gb.Plan(coo, length_policy=gb.GBSP_LEN_7SMOOTH, u_tile=tile) as p:
        assert p.info["channel_len"] == 525 and p.info["rows_threads"] == 256
        out = p.empty_output()
        got = row_launches(lambda st: p.execute(out, stream=st))
        tails = [tail] if tail <= tile else [tile, tail - tile]
        assert len(got) == 1 + len(tails)
        for (_, grid, block), rows_here in zip(got, [tile] + tails):
            per_sm = rows_here // n
            assert block == next(b for b in (32, 64, 128, 256) if per_sm * b >= 320 or b == 256)
            assert grid <= rows_here
        p.execute(out)
        torch.cuda.synchronize()
        assert p.error_flags() == 0
        us = np.unique(np.r_[0, 1, 2, tile - 1, tile, tile + tail - 1, rows - 1, np.arange(5, rows, rows // 31)])
        res = out[torch.from_numpy(us).cuda()].cpu().numpy()[:, :cols // 2 + 1]
    # rel-L2 bar of the FP32 transform at this length, as in test_gpu_row_layout.py
    assert fp64.rel_l2(res, fp64.spectrum_rows_fp64(rows, cols, coo.row_idx, coo.col_idx, us)) <= 1e-6


def test_no_more_blocks_than_rows(cuda):
    for cols, kw in ((12001, {}), (16706, {}), (16706, dict(channel_mode=1)), (40421, {}), (4603, {})):
        coo = synthetic.uniform_matrix(41, cols, 400, seed=cols)
        with gb.Plan(coo, length_policy=gb.GBSP_LEN_7SMOOTH, **kw) as p:
            out = p.empty_output()
            [(_, grid, _)] = row_launches(lambda st: p.execute(out, stream=st))
            assert grid <= 21 * (p.info["channels"] if kw else 1)

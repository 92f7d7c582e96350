"""Which block, grid and instance a row launch gets, read from a captured graph.

Short rows run 32, 64 or 128 threads each where there are rows enough for
every SM, and wider blocks where there are fewer; the rows are those of the
launch, not of the plan.  Long rows run 352 threads where that divides their
stages better, two channels that hold the row an instance of their own, and rows
whose last radix is a power of two a padded buffer.

Spectra are held to rel-L2 1e-6 against FP64, the bar of test_gpu_row_layout.py
for an FP32 FFT and its inverse of up to five stages; the two or more channels of
a long row and their sum add one product and one sum each, 1.2e-7.
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


# rows an SM of the first tile (all alike) and the second (one SM has another
# row), and their blocks: 525 points (257 columns) and 135 (65)
@pytest.mark.parametrize("cols,full,last,blocks", [
    (257, 18, 16, (32, 64)), (257, 18, 4, (32, 64)), (257, 16, 3, (64, 128)), (257, 16, 1, (64, 256)),
    (257, 8, 7, (64, 64)), (257, 4, 2, (128, 128)), (257, 2, 1, (256, 256)), (65, 18, 16, (32, 64)),
    (65, 18, 0, (32, 256))])
def test_a_short_tile_gets_a_wider_block(cuda, cols, full, last, blocks):
    import torch
    n = sms()
    tile, tail = full * n, last * n + 3
    rows = 2 * (tile + tail - 1)  # tiles of `tile` and `tail` Bluestein rows
    coo = synthetic.uniform_matrix(rows, cols, 4 * rows, seed=rows)
    with gb.Plan(coo, length_policy=gb.GBSP_LEN_7SMOOTH, u_tile=tile) as p:
        assert p.info["channel_len"] == {257: 525, 65: 135}[cols] and p.info["rows_threads"] == 256
        out = p.empty_output()
        got = row_launches(lambda st: p.execute(out, stream=st))
        assert [block for _, _, block in got] == list(blocks)
        assert got[0][1] <= tile and got[1][1] <= tail
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


SINGLE, SEQ, DIRECT, SEQ2 = 0, 2, 4, 5


# rows, columns, options; compiled block bound, kind of row, padded; block (None:
# as planned, rows of several channels)
@pytest.mark.parametrize("rows,cols,kw,instance,block", [
    (401, 8193, dict(length_policy=2), (512, SEQ2, 1), None),
    (401, 9001, dict(length_policy=2), (512, SEQ2, 1), None),
    (701, 11003, dict(length_policy=2), (512, SEQ2, 1), None),
    (401, 16382, dict(length_policy=2), (512, SEQ2, 1), None),
    (401, 16383, dict(length_policy=2), (512, SEQ2, 1), None),
    (401, 16706, dict(length_policy=7), (512, SEQ2, 0), None),
    (401, 16706, dict(length_policy=2), (512, SEQ, 1), None),
    (401, 40421, dict(length_policy=2), (512, SEQ, 1), None),
    (401, 40421, dict(length_policy=7), (512, SEQ, 0), None),
    (401, 8219, dict(length_policy=7), (384, SINGLE, 0), 352),
    (401, 7499, dict(length_policy=7), (512, SINGLE, 0), 512),
    (12001, 2048, dict(length_policy=3), (512, DIRECT, 1), 64),
    (12001, 2401, dict(length_policy=7), (1024, DIRECT, 0), 64),
    (12001, 1000, dict(length_policy=2), (512, SINGLE, 1), 64),
    (20001, 257, dict(length_policy=7), (512, SINGLE, 0), 32),
    (20001, 65, dict(length_policy=7), (1024, SINGLE, 0), 32)])
def test_instances(cuda, rows, cols, kw, instance, block):
    import torch
    coo = synthetic.uniform_matrix(rows, cols, 4 * max(rows, cols), seed=cols)
    with gb.Plan(coo, **kw) as p:
        out = p.empty_output()
        [(args, _, threads)] = row_launches(lambda st: p.execute(out, stream=st))
        assert (args, threads) == (instance, block or p.info["rows_threads"])
        out.fill_(complex(7.0, 7.0))
        p.execute(out)
        torch.cuda.synchronize()
        assert p.error_flags() == 0
        us = np.unique(np.r_[0, 1, rows // 2, rows // 2 + 1, rows - 1, np.arange(5, rows, rows // 12)])
        got = out[torch.from_numpy(us).cuda()].cpu().numpy()
    fc = cols // 2 + 1
    assert np.all(got[:, fc:] == 0)
    assert fp64.rel_l2(got[:, :fc], fp64.spectrum_rows_fp64(rows, cols, coo.row_idx, coo.col_idx, us)) <= 1e-6

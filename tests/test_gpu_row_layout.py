"""Row kernels by block width and with padded row buffers, against FP64.

Short rows run in blocks of 32, 64 or 128 threads when there are enough of
them (edges at 700, 3000 and 7000 points), on the 64- or 128-register kernels;
long ones planned for 512 threads in 352 where that divides their stages
better; rows whose last radix is a power of two use a padded row buffer.  The rel-L2
bar is 1e-6: an FP32 FFT of up to five stages and its inverse round each value
about 30 times at 6e-8, 3.3e-7 when independent, three times that at worst here.
"""
import numpy as np
import pytest

import cuspfft_gb300 as gb
from cuspfft_gb300 import synthetic
from oracle import fp64

pytestmark = pytest.mark.gpu


def check(coo, **kw):
    import torch
    with gb.Plan(coo, **kw) as p:
        out = p.empty_output()
        out.fill_(complex(7.0, 7.0))
        p.execute(out)
        torch.cuda.synchronize()
        assert p.error_flags() == 0
        info = p.info
        r = coo.rows
        us = np.unique(np.r_[0, 1, 2, r // 2, r // 2 + 1, r - 2, r - 1, np.arange(5, r, max(1, r // 40))] % r)
        got = out[torch.from_numpy(us).cuda()].cpu().numpy()
    fc = coo.cols // 2 + 1
    ref = fp64.spectrum_rows_fp64(coo.rows, coo.cols, coo.row_idx, coo.col_idx, us)
    assert np.all(got[:, fc:] == 0)
    err = fp64.rel_l2(got[:, :fc], ref)
    assert err <= 1e-6, f"rel-L2 {err:.2e}"
    return info


# cols: Bluestein (prime) and direct lengths around the block edges
@pytest.mark.parametrize("cols", [2, 3, 7, 97, 343, 347, 351, 700, 701, 1499, 1501, 3000, 3001, 3499, 3511, 7000])
@pytest.mark.parametrize("rows", [311, 2500, 12000])
def test_block_widths(cuda, rows, cols):
    coo = synthetic.uniform_matrix(rows, cols, 3 * max(rows, cols), seed=cols)
    check(coo, length_policy=gb.GBSP_LEN_7SMOOTH)


# long rows: three and four stages that 352 threads divide better than 512
# (7813, 8231, 9407, 10805), and some that stay
@pytest.mark.parametrize("cols", [7499, 7813, 7874, 8231, 8959, 9407, 10805, 11003])
@pytest.mark.parametrize("rows", [303, 1201])
def test_long_row_blocks(cuda, rows, cols):
    coo = synthetic.uniform_matrix(rows, cols, 3 * cols, seed=cols)
    check(coo, length_policy=gb.GBSP_LEN_7SMOOTH)


# padded buffers: spans below 16, last radices 4 to 32, units 16 and 32
@pytest.mark.parametrize("cols,radix", [
    (64, [16, 4]), (64, [4, 4, 4]), (64, [8, 8]), (128, [4, 4, 8]), (256, [2, 8, 16]), (512, [16, 32]),
    (512, [32, 16]), (512, [8, 8, 8]), (1024, [4, 4, 4, 4, 4]), (1024, [32, 32]), (2048, [16, 16, 8]),
    (2048, [32, 16, 4]), (2048, [8, 4, 4, 4, 4]), (4096, [16, 16, 16]), (16384, [32, 32, 16]), (16384, [16, 16, 8, 8]),
    (384, [24, 16]), (1152, [9, 8, 16]), (9216, [24, 24, 16]), (6144, [12, 16, 32]), (240, [15, 16]),
    (480, [15, 32]), (640, [5, 8, 16])])
@pytest.mark.parametrize("bluestein", [0, 1])
def test_padded_buffers(cuda, cols, radix, bluestein):
    policy = gb.GBSP_LEN_7SMOOTH
    if bluestein:
        # a column count whose convolution has this length
        n = (cols + 1) // 2
        while n > 1 and gb.next_smooth(2 * n - 1, policy) > cols:
            n -= 1
        if gb.next_smooth(2 * n - 1, policy) != cols:
            pytest.skip("no convolution of this length")
        cols = n
    coo = synthetic.uniform_matrix(3001, cols, 12000, seed=cols)
    info = check(coo, length_policy=policy, radix=radix, force_bluestein=bluestein)
    assert [r for r in info["radix"] if r] == radix


def test_batch_keeps_the_single_plan_bits(cuda):
    import torch
    mats = [synthetic.uniform_matrix(r, c, 4 * r, seed=c) for r, c in
            ((900, 2048), (1500, 257), (700, 1024), (2000, 64), (300, 3500), (401, 4603), (100, 8192), (3000, 31))]
    with gb.Batch(mats, length_policy=gb.GBSP_LEN_7SMOOTH) as b:
        outs = b.empty_outputs()
        b.set_outputs(outs)
        b.execute()
        torch.cuda.synchronize()
        assert b.error_flags() == 0
        for coo, o, info in zip(mats, outs, b.infos):
            with gb.Plan(coo, length_policy=gb.GBSP_LEN_7SMOOTH, radix=info["radix"],
                         rows_threads=info["rows_threads"]) as p:
                one = p.empty_output()
                p.execute(one)
                torch.cuda.synchronize()
                assert torch.equal(one, o)

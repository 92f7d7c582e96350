"""Column sums of the tensor-core pass 1 (k_twiddle_mma) against FP64.

A sum is sum_r W^{(i-64) r} W^{(u0+64+128 d) r} over the column's nonzeros.
Both factors are correctly rounded FP32 table entries, each component off by at
most 2^-25, so a factor by at most sqrt(2) * 2^-25 = 4.3e-8 and a product by
8.5e-8; products and sums are exact to below 2^-25 per nonzero (3.0e-8), and
the result is rounded once per component (6.0e-8 of it).  So an entry is off by
at most 1.15e-7 * degree + 6.0e-8 * |sum|.  The two-level table makes each
factor a product of two entries, rounded (8.5e-8 + 8.5e-8 a factor, 3.4e-7 +
3.0e-8 a nonzero).  Where nothing cancels that is far above the typical error
(rel-L2 4e-8), so the sums of random columns are held to rel-L2 1e-7 as well
(2e-7 with the two-level table), below the FP32 kernel's.

The sizes sit at the edges of the kernel's blocks: 128 rows per block d; 8, 16
or 32 blocks per item with 16, 8 or 4 columns per window; eight nonzeros per
K-step, 32 per chunk.
"""
import numpy as np
import pytest

import cuspfft_gb300 as gb

pytestmark = pytest.mark.gpu

PER_NZ = {0: 1.15e-7, 1: 1.15e-7, 2: 3.7e-7}  # by table layout: full, half, two-level
REL = {0: 1e-7, 1: 1e-7, 2: 2e-7}


def matrix(rows, degrees, seed):
    """One column per degree (capped at rows), rows drawn without repetition."""
    g = np.random.default_rng(seed)
    r = [np.sort(g.choice(rows, min(d, rows), replace=False)) for d in degrees]
    c = [np.full(x.size, j) for j, x in enumerate(r)]
    r, c = np.concatenate(r), np.concatenate(c)
    order = np.lexsort((c, r))
    return gb.COOMatrix(rows, len(degrees), r[order].astype(np.int32), c[order].astype(np.int32))


def want(coo, us):
    out = np.zeros((len(us), coo.cols), np.complex128)
    for c in range(coo.cols):
        r = coo.row_idx[coo.col_idx == c].astype(np.int64)
        out[:, c] = np.exp(-2j * np.pi * (np.outer(us, r) % coo.rows) / coo.rows).sum(1)
    return out


def check(coo, u0, n, pitch, table=0, **kw):
    import torch
    with gb.Plan(coo, row_table_mode=table, **kw) as p:
        s = torch.full((n, pitch), complex(5.0, 5.0), dtype=torch.complex64, device="cuda")
        p.column_sums(u0, n, s)
        torch.cuda.synchronize()
        assert p.error_flags() == 0
        got = s.cpu().numpy()
    sc = (coo.cols + 1) // 2 * 2
    us = np.arange(u0, u0 + n, dtype=np.int64)
    if n > 600:
        us = us[np.unique(np.r_[0:40, n // 2:n // 2 + 40, n - 40:n])]
    ref = want(coo, us)
    dif = np.abs(got[us - u0, :coo.cols] - ref)
    assert np.all(got[:, coo.cols:sc] == 0)
    if sc % 4 or pitch % 4:
        assert np.all(got[:, sc:] == 5 + 5j)  # nothing past the columns
    lay = max(table - 1, 0 if coo.rows <= 9001 else 1 if coo.rows <= 18000 else 2)
    deg = np.bincount(coo.col_idx, minlength=coo.cols)
    assert np.all(dif <= PER_NZ[lay] * deg + 6.0e-8 * np.abs(ref))
    sparse = 8 * deg <= coo.rows
    if sparse.any() and deg[sparse].sum() > 0:
        rel = np.linalg.norm(dif[:, sparse]) / np.linalg.norm(ref[:, sparse])
        assert rel <= REL[lay], f"rel-L2 {rel:.2e}"


DEGREES = [0, 1, 7, 8, 9, 0, 0, 0, 0, 24, 31, 32, 33, 64, 65, 3, 100, 2]


@pytest.mark.parametrize("rows,u0,n", [(4095, 0, 2048), (4095, 5, 2049), (4999, 0, 4096), (4999, 3, 4097),
                                       (4999, 1, 4110), (8191, 0, 4223), (8191, 0, 4224), (8191, 7, 4225),
                                       (8191, 0, 5120), (8191, 0, 5121), (8191, 0, 6144), (8191, 0, 6145),
                                       (9001, 0, 9001)])
@pytest.mark.parametrize("table", [0, 1, 2, 3])
def test_column_sums(cuda, rows, u0, n, table):
    coo = matrix(rows, DEGREES, rows + u0)
    check(coo, u0, n, 32, table)


@pytest.mark.parametrize("cols", [1, 2, 3, 4, 5, 6, 7, 9, 15, 16, 17, 33])
@pytest.mark.parametrize("extra", [0, 2, 3])
@pytest.mark.parametrize("rows", [4400, 9000, 11000])
def test_window_edges_and_pitches(cuda, cols, extra, rows):
    # odd column counts, partial windows, pitches that rule out wide stores
    coo = matrix(rows, [5 + 9 * j for j in range(cols)], cols)
    check(coo, 0, rows // 2 + 1, (cols + 1) // 2 * 2 + extra)


@pytest.mark.parametrize("rows,index_bytes", [(15013, 2), (40421, 2), (40421, 4), (65536, 2), (70001, 4), (131071, 4)])
def test_tall(cuda, rows, index_bytes):
    # the half table, the two-level table, 64-bit phases
    coo = matrix(rows, [40, 0, 1, 300, 17], rows)
    check(coo, 0, rows // 2 + 1, 6, index_bytes=index_bytes)


def test_heavy_columns(cuda):
    # coherent sums (u = 0 gives the degree) up to the exact range of the first accumulator
    coo = matrix(5003, [1024, 1000, 1, 0, 700, 37], 3)
    check(coo, 0, 2502, 8)


def test_columns_past_the_exact_range_take_the_fp32_kernel(cuda):
    import torch
    coo = matrix(5003, [1025, 3000, 1, 0, 700, 37], 3)
    outs = []
    for kw in ({}, {"kahan_min_degree": 64}):
        with gb.Plan(coo, **kw) as p:
            out = p.empty_output()
            p.execute(out)
            torch.cuda.synchronize()
            outs.append(out.cpu().numpy())
    assert np.array_equal(outs[0], outs[1])
    small = matrix(700, [40] * 50, 4)
    with gb.Batch([small, coo]) as b, gb.Plan(small) as ps, gb.Plan(coo) as pc:
        got = b.empty_outputs()
        b.set_outputs(got)
        b.execute()
        for p, g in zip((ps, pc), got):
            one = p.empty_output()
            p.execute(one)
            torch.cuda.synchronize()
            assert torch.equal(one, g)


def test_explicit_kahan_degree_keeps_fp32_sums(cuda):
    # 64 is the default degree: naming it selects the FP32 kernel, whose sums differ in their last bits
    import torch
    coo = matrix(5003, [40 + j for j in range(64)], 5)
    outs = []
    for kw in ({}, {"kahan_min_degree": 64}):
        for shape in (0, 1, 3, 6):
            with gb.Plan(coo, pass1_shape=shape, **kw) as p:
                s = torch.zeros((2502, 64), dtype=torch.complex64, device="cuda")
                p.column_sums(0, 2502, s)
                outs.append(s.cpu().numpy())
    ref = want(coo, np.arange(2502))
    e = [np.linalg.norm(o - ref) / np.linalg.norm(ref) for o in outs]
    assert all(np.array_equal(o, outs[0]) for o in outs[1:4])  # the tensor-core sums do not depend on the shape
    assert e[0] < 1e-7 and all(x <= 2.5e-7 for x in e[4:]) and not np.array_equal(outs[0], outs[4])


def test_small_tiles_of_a_large_plan_take_the_fp32_kernel(cuda):
    # 2048 rows is the smallest tile for the tensor cores; a tile below it agrees to FP32 rounding
    import torch
    coo = matrix(9001, DEGREES, 7)
    with gb.Plan(coo) as p, gb.Plan(coo, kahan_min_degree=64) as q:
        s = [torch.zeros((n, 32), dtype=torch.complex64, device="cuda") for n in (2048, 2047, 2047)]
        p.column_sums(0, 2048, s[0])
        p.column_sums(0, 2047, s[1])
        q.column_sums(0, 2047, s[2])
        torch.cuda.synchronize()
        assert torch.equal(s[1], s[2])
        assert not torch.equal(s[0][:2047], s[1])
        assert torch.linalg.norm(s[0][:2047] - s[1]) <= 3e-7 * torch.linalg.norm(s[1])


def test_tiles_at_multiples_of_128_rows_keep_the_bits(cuda):
    import torch
    coo = matrix(12001, DEGREES, 8)
    with gb.Plan(coo) as p:
        whole = torch.zeros((6001, 32), dtype=torch.complex64, device="cuda")
        p.column_sums(0, 6001, whole)
        for u0, n in ((128, 2048), (1280, 4300), (3200, 2801)):
            part = torch.zeros((n, 32), dtype=torch.complex64, device="cuda")
            p.column_sums(u0, n, part)
            torch.cuda.synchronize()
            assert torch.equal(part[:, :18], whole[u0:u0 + n, :18])


def test_batch_mixes_both_kernels(cuda):
    import torch
    mats = [matrix(r, [d] * c, r) for r, c, d in ((500, 70, 9), (6001, 133, 20), (4100, 51, 3), (9999, 40, 33),
                                                  (70001, 9, 50))]
    with gb.Batch(mats) as b:
        got = b.empty_outputs()
        b.set_outputs(got)
        b.execute()
        b.graph_launch()
        torch.cuda.synchronize()
        assert b.error_flags() == 0
        for coo, g in zip(mats, got):
            with gb.Plan(coo, index_bytes=4, row_table_mode=3) as p:
                one = p.empty_output()
                p.execute(one)
                torch.cuda.synchronize()
                assert torch.equal(one, g)

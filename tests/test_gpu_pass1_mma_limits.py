"""The tensor-core pass 1 at the ends of its range.

Degree limit.  At u = 0 all of a column's terms are 1, a product of W^{-64 r}
and W^{64 r}, each a rounded table entry split into h (step 2^-7), m and l.
The worst columns are the rows whose h is longest: the h*h sum then runs ahead
of the true one, past 1024 at 1024 nonzeros, and the second accumulator holds a
like amount of the other sign.  Against the sum of the rounded entries'
products, in FP64: the first accumulator loses at most two steps of 2^-14 past
1024 (1.2e-7 of the sum), the second half a step of its size per MMA, five in
each of 128 K-steps, 8.4e-5 in all while it grows to 7 (8e-8), and the result
is rounded once (6e-8): 2.6e-7, held to 3e-7.

Windows.  With few items a window takes fewer columns than it holds.  A sum does
not depend on its window, so the sums of a narrow matrix are, bit for bit, those
of the same columns among many.

Two-level table.  From some 18000 rows on, and where a half table does not fit
beside the operands, a factor is a product of two table entries: errors of
4.3e-8 / sqrt(2) each and the product's 3e-8, four entries and two products a
term, 5.7e-8 in all when independent; held to 8e-8, and to no more than the FP32
kernel's on the same sums.

Routes.  Which kernel a matrix gets, read from a captured graph, on both sides of
each line: rows x nonzeros per column, one column far longer than the others.
"""
import numpy as np
import pytest

import cuspfft_gb300 as gb
from graph_nodes import kernel_names

pytestmark = pytest.mark.gpu


def sums(coo, us, **kw):
    import torch
    n = coo.rows // 2 + 1
    with gb.Plan(coo, **kw) as p:
        s = torch.empty((n, (coo.cols + 1) // 2 * 2), dtype=torch.complex64, device="cuda")
        p.column_sums(0, n, s)
        torch.cuda.synchronize()
        assert p.error_flags() == 0
        return s[torch.as_tensor(us, device="cuda"), :coo.cols].cpu().numpy().astype(np.complex128)


@pytest.mark.parametrize("rows", [5003, 8219, 9001, 12007])
def test_longest_factors_at_the_degree_limit(cuda, rows):
    r = np.arange(rows, dtype=np.int64)
    w = np.exp(-2j * np.pi * (64 * r % rows) / rows).astype(np.complex64).astype(np.complex128)
    h = np.round(w.real * 128) ** 2 + np.round(w.imag * 128) ** 2
    order = np.argsort(-h, kind="stable")
    degrees = [1008, 1012, 1013, 1016, 1020, 1024]
    cols = [np.sort(order[:d]) for d in degrees]
    key = np.unique(np.concatenate([c * len(degrees) + j for j, c in enumerate(cols)]))
    coo = gb.COOMatrix(rows, len(degrees), (key // len(degrees)).astype(np.int32),
                       (key % len(degrees)).astype(np.int32))
    want = np.array([np.sum(np.abs(w[c]) ** 2) for c in cols])
    got = sums(coo, [0])[0]
    assert np.all(np.abs(got - want) <= 3e-7 * want)


def matrix(rows, degrees, seed):
    g = np.random.default_rng(seed)
    r = [g.choice(rows, d, replace=False) for d in degrees]
    key = np.sort(np.concatenate([x.astype(np.int64) * len(degrees) + j for j, x in enumerate(r)]))
    return gb.COOMatrix(rows, len(degrees), (key // len(degrees)).astype(np.int32),
                        (key % len(degrees)).astype(np.int32))


# blocks of 32, 16 and fewer d; one and two columns a window and the widest
@pytest.mark.parametrize("rows", [4097, 4300, 5003, 9001, 12001, 16500])
@pytest.mark.parametrize("cols", [1, 2, 3, 17, 40, 77, 151, 152, 153, 300])
@pytest.mark.parametrize("degree", [20, 40])
def test_sums_do_not_depend_on_the_window(cuda, rows, cols, degree):
    g = np.random.default_rng(cols)
    deg = g.integers(max(1, degree - 9), degree + 10, 700)
    deg[5::7] = 0
    deg[0] = 60
    wide = matrix(rows, deg, rows)
    keep = wide.col_idx < cols
    narrow = gb.COOMatrix(rows, cols, wide.row_idx[keep].copy(), wide.col_idx[keep].copy())
    us = np.unique(np.r_[0:300, rows // 4:rows // 4 + 300, rows // 2 - 200:rows // 2 + 1])
    assert np.array_equal(sums(narrow, us), sums(wide, us)[:, :cols])


@pytest.mark.parametrize("rows,degrees,mma", [
    (4097, [4] * 300, False), (4097, [5] * 300, True),        # 10000 rows x nonzeros a column
    (4097, [4] * 2048, False), (4097, [5] * 2048, True),
    (8001, [2] * 2048, False), (8001, [3] * 2048, True),
    (4094, [60] * 300, True), (4093, [60] * 300, False),      # 2048 rows
    (5003, [10] * 1999 + [250], True), (5003, [10] * 1999 + [1000], False),   # one long column
    (5003, [1024] * 4, True), (5003, [1024] * 3 + [1025], False)])
def test_routes(cuda, rows, degrees, mma):
    import torch
    coo = matrix(rows, degrees, rows)
    n = rows // 2 + 1
    with gb.Plan(coo) as p:
        s = torch.empty((n, (coo.cols + 1) // 2 * 2), dtype=torch.complex64, device="cuda")
        [name] = kernel_names(lambda st: p.column_sums(0, n, s, stream=st))
    assert ("k_twiddle_mma" in name) == mma


@pytest.mark.parametrize("rows", [18503, 20001, 30011, 39001, 70001])
@pytest.mark.parametrize("table", [0, 2, 3])
def test_two_level_sums_against_fp32(cuda, rows, table):
    if table == 2 and rows > 39001:
        pytest.skip("no half table of that many rows")
    g = np.random.default_rng(rows)
    coo = matrix(rows, g.integers(2, 300, 48), rows)
    us = np.unique(np.r_[0:40, rows // 4:rows // 4 + 40, rows // 2 - 40:rows // 2 + 1])
    ref = np.zeros((us.size, coo.cols), np.complex128)
    for c in range(coo.cols):
        r = coo.row_idx[coo.col_idx == c].astype(np.int64)
        ref[:, c] = np.exp(-2j * np.pi * (np.outer(us, r) % rows) / rows).sum(1)
    err = [np.linalg.norm(sums(coo, us, row_table_mode=table, **kw) - ref) / np.linalg.norm(ref)
           for kw in ({}, dict(kahan_min_degree=64))]
    assert err[0] <= 8e-8 and err[0] <= err[1]

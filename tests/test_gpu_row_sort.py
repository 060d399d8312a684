"""Rows of the device transpose in column order: a warp sorts a row of up to 32
entries, a block a longer one.  Every length around that edge, empty rows, and
row counts around a block's eight warps; whole numbers and copied values, so
the arrays are exactly numpy's."""
from __future__ import annotations

import numpy as np
import pytest

from mcpdlp import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 7, 8, 9, 300])
@pytest.mark.parametrize("longest", [1, 31, 32, 33, 70])
def test_rows_come_out_sorted(gpu_ctx, m, longest):
    import torch
    r = np.random.default_rng(100 * m + longest)
    n = 257
    length = r.integers(0, longest + 1, size=m)
    length[-1] = longest
    rows = np.repeat(np.arange(m), length)
    cols = np.concatenate([np.sort(r.choice(n, size=k, replace=False)) for k in length])
    val = r.normal(size=len(rows))
    order = np.lexsort((rows, cols))  # column-major
    start = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))])
    dev = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, dtype=t)).cuda()  # noqa: E731
    cs, ri, v = dev(start, np.int32), dev(rows[order], np.int32), dev(val[order], np.float64)
    rs = torch.zeros(m + 1, dtype=torch.int32, device="cuda")
    ci = torch.zeros(len(rows), dtype=torch.int32, device="cuda")
    rv = torch.zeros(len(rows), dtype=torch.float64, device="cuda")
    _lib.check(_lib.engine().mc_csc_to_csr(gpu_ctx.handle, m, n, len(rows), cs.data_ptr(), ri.data_ptr(), v.data_ptr(),
                                           rs.data_ptr(), ci.data_ptr(), rv.data_ptr()))
    np.testing.assert_array_equal(rs.cpu().numpy(), np.concatenate([[0], np.cumsum(length)]))
    np.testing.assert_array_equal(ci.cpu().numpy(), cols)
    np.testing.assert_array_equal(rv.cpu().numpy(), val)


@pytest.mark.parametrize("per_row", [1, 8, 9])  # up to 8 entries a row on average: a thread per row; above: a warp
def test_many_short_rows_come_out_sorted(gpu_ctx, per_row):
    import torch
    m, n = 148 * 2048 + 5, 400
    r = np.random.default_rng(per_row)
    length = r.integers(0, 2 * per_row + 1, size=m)
    length[[0, 7, 300, m - 1]] = [31, 32, 33, 70]
    assert abs(length.mean() - per_row) < 0.1
    while length.sum() > per_row * m:  # the mean exactly, or less
        length[np.flatnonzero(length[:-1] > 0)[8:8 + int(length.sum()) - per_row * m]] -= 1
    rows = np.repeat(np.arange(m), length)
    first = r.integers(0, n, size=m)  # a row's columns: a run that wraps round, so distinct
    cols = (np.repeat(first, length) + 5 * (np.arange(len(rows)) - np.repeat(np.cumsum(length) - length, length))) % n
    val = r.normal(size=len(rows))
    by_col, by_row = np.lexsort((rows, cols)), np.lexsort((cols, rows))
    start = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))])
    dev = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, dtype=t)).cuda()  # noqa: E731
    cs, ri, v = dev(start, np.int32), dev(rows[by_col], np.int32), dev(val[by_col], np.float64)
    rs = torch.zeros(m + 1, dtype=torch.int32, device="cuda")
    ci = torch.zeros(len(rows), dtype=torch.int32, device="cuda")
    rv = torch.zeros(len(rows), dtype=torch.float64, device="cuda")
    _lib.check(_lib.engine().mc_csc_to_csr(gpu_ctx.handle, m, n, len(rows), cs.data_ptr(), ri.data_ptr(), v.data_ptr(),
                                           rs.data_ptr(), ci.data_ptr(), rv.data_ptr()))
    np.testing.assert_array_equal(rs.cpu().numpy(), np.concatenate([[0], np.cumsum(length)]))
    np.testing.assert_array_equal(ci.cpu().numpy(), cols[by_row])
    np.testing.assert_array_equal(rv.cpu().numpy(), val[by_row])

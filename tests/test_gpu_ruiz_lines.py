"""Lines of every length up to a few windows of their lanes, their last one to
three entries taken together: bit for bit the oracle's matrix and scales, for one
LP and for many short rows."""
from __future__ import annotations

import numpy as np
import pytest

import mcpdlp
from test_gpu_ruiz import scaled

pytestmark = pytest.mark.gpu


def lines(m, n, longest, seed):
    """Row i has i mod (longest + 1) entries."""
    r = np.random.default_rng(seed)
    length = np.arange(m) % (longest + 1)
    rows = np.repeat(np.arange(m), length)
    at = np.arange(len(rows)) - np.repeat(np.cumsum(length) - length, length)
    cols = (np.repeat(r.integers(0, n, m), length) + at) % n  # a run that wraps round
    order = np.lexsort((rows, cols))
    val = 10.0 ** r.uniform(-3, 3, len(rows)) * r.choice([-1.0, 1.0], len(rows))
    start = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))])
    return mcpdlp.Model(m, n, start, rows[order], val[order], r.normal(size=n), np.zeros(n), np.ones(n), np.zeros(m),
                        np.ones(m))


@pytest.mark.parametrize("m,n,longest", [(40, 30, 9), (300, 90, 25), (400, 300, 70), (200, 500, 300), (200_000, 70_000, 3)])
def test_line_lengths(gpu_ctx, oracle, m, n, longest):
    lp = lines(m, n, longest, m)
    exp = oracle.equilibrate(lp, 10)
    v, rv, order, row_scale, col_scale, it = scaled(gpu_ctx, lp, 10)
    assert it == exp["iterations"]
    assert np.array_equal(v, exp["value"]) and np.array_equal(rv, exp["value"][order])
    assert np.array_equal(row_scale, exp["row_scale"]) and np.array_equal(col_scale, exp["col_scale"])

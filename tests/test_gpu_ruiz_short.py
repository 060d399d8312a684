"""Equilibration of matrices whose lines are short on average, by one thread a
line: even and odd lengths, empty lines, one line much longer than the mean, and
several such LPs in a batch; bit for bit the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import mcpdlp
from mcpdlp import PdlpOptions
from test_gpu_ruiz import scaled

pytestmark = pytest.mark.gpu


def short_lines(m, n, nnz, long_row, long_col, seed):
    r = np.random.default_rng(seed)
    rows = np.concatenate([r.integers(0, m, nnz), np.full(long_row, m // 2), r.integers(0, m, long_col)])
    cols = np.concatenate([r.integers(0, n, nnz), r.integers(0, n, long_row), np.full(long_col, n // 3)])
    key = np.unique(cols.astype(np.int64) * m + rows)
    cols, rows = key // m, (key % m).astype(np.int32)
    val = 10.0 ** r.uniform(-3, 3, len(key)) * r.choice([-1.0, 1.0], len(key))
    start = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))])
    return mcpdlp.Model(m, n, start, rows, val, r.normal(size=n), np.zeros(n), np.ones(n), np.zeros(m), np.ones(m))


@pytest.mark.parametrize("m,n,nnz,long_row,long_col", [(1, 3, 2, 0, 0), (257, 255, 900, 0, 0), (700, 600, 1500, 301, 0),
                                                      (600, 700, 1500, 0, 402), (300_000, 280_000, 1_900_000, 5001, 3000)])
@pytest.mark.parametrize("passes", [1, 10])
def test_short_lines(gpu_ctx, oracle, m, n, nnz, long_row, long_col, passes):
    lp = short_lines(m, n, nnz, long_row, long_col, m)
    assert lp.nnz < 8 * min(m, n)
    exp = oracle.equilibrate(lp, passes)
    v, rv, order, row_scale, col_scale, it = scaled(gpu_ctx, lp, passes)
    assert it == exp["iterations"]
    assert np.array_equal(v, exp["value"]) and np.array_equal(rv, exp["value"][order])
    assert np.array_equal(row_scale, exp["row_scale"]) and np.array_equal(col_scale, exp["col_scale"])


def test_batch_of_short_lines(gpu_ctx, oracle):
    lps = [short_lines(90 + 41 * q, 70 + 53 * q, 300 + 150 * q, 20 * q, 10 * q, q) for q in range(6)]
    o = PdlpOptions(max_iterations=40, ruiz_iterations=25)
    for lp, r in zip(lps, gpu_ctx.solve_batch(lps, o)):
        assert r.extra["ruiz_iterations_executed"] == oracle.equilibrate(lp, 25)["iterations"]

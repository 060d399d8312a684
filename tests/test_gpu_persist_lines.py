"""Which solves the persistent loop's form of one block per SM takes, by the shape
of their lines, and that its iterates are those of the streaming kernels (the
same solve with shared_device) on both sides of each edge."""
from __future__ import annotations

import numpy as np
import pytest

import mcpdlp
from mcpdlp import PdlpOptions, Precision, generators

pytestmark = pytest.mark.gpu


def takes_the_loop(gpu_ctx, model, precision) -> bool:
    # no step-size rule and no restart: nothing depends on a reduction's order
    kw = dict(max_iterations=97, precision=Precision[precision], adaptive_step_size=False, initial_primal_weight=1.0,
              restart_strategy=mcpdlp.RestartStrategy.none)
    res = []
    for shared in (False, True):
        o = PdlpOptions(shared_device=shared, **kw)
        o.set_tolerance(1e-14)
        res.append(gpu_ctx.solve(model, o))
    alone, streaming = res
    assert streaming.extra["launches_by_kind"]["dual"] > 0
    np.testing.assert_allclose(alone.primal, streaming.primal, rtol=1e-11, atol=0)
    np.testing.assert_allclose(alone.dual, streaming.dual, rtol=1e-11, atol=0)
    return alone.extra["launches_by_kind"]["dual"] == 0


# one entry a column: the dual is copied by each block while that is at most 6 (FP32
# with most lanes: 8) loads per entry; above, such an FP32 model takes the streaming kernels
# (6108 x 148 blocks is the last multiple up to 8 x 113000)
@pytest.mark.parametrize("m,n,fp64,fp32", [(2000, 113000, True, True), (6105, 113000, True, True), (6107, 113000, True, True),
                                           (6108, 113000, True, True), (6109, 113000, True, False),
                                           (3000, 70000, True, True)])
def test_one_entry_a_column(gpu_ctx, m, n, fp64, fp32):
    model = generators.random_lp(70, m, n, 1)
    assert takes_the_loop(gpu_ctx, model, "fp64") == fp64
    assert takes_the_loop(gpu_ctx, model, "fp32_refine") == fp32


def with_long_lines(m, n, k, row=0, col=0):
    """k entries a column at random rows but the first, which has `row` entries;
    the first column has `col` in all."""
    r = np.random.default_rng(m + n + row + col)
    entries = {(int(i), j): r.normal() for j in range(n) for i in 1 + r.choice(m - 1, size=k, replace=False)}
    for j in range(1, 1 + min(row, n - 1)):
        entries[(0, j)] = r.normal()
    more = [i for i in range(1, m) if (i, 0) not in entries][:max(0, col - k)]
    for i in more:
        entries[(i, 0)] = r.normal()
    i, j = np.array(list(entries)).T
    order = np.lexsort((i, j))
    i, j, v = i[order], j[order], np.array(list(entries.values()))[order]
    x = np.where(r.random(n) < 0.3, 0.0, r.uniform(0.1, 5.0, n))
    b = np.bincount(i, weights=v * x[j], minlength=m)
    return mcpdlp.Model(m, n, np.concatenate([[0], np.cumsum(np.bincount(j, minlength=n))]), i, v, r.normal(size=n),
                        np.zeros(n), np.full(n, 10.0), b, b)


# steps are of four entries per lane; lanes from the mean: 4 a row and 1 a column, 32 a row where it has 200
@pytest.mark.parametrize("shape,row,col,loop", [
    ((4000, 12000, 6), 128, 0, True), ((4000, 12000, 6), 129, 0, False),     # 8 steps
    ((4000, 12000, 6), 0, 16, True), ((4000, 12000, 6), 0, 17, False),       # 4 steps
    ((1000, 6000, 4), 256, 0, True), ((1000, 6000, 4), 257, 0, False),       # few nonzeros: 16 steps
    ((600, 20000, 6), 3072, 0, True), ((600, 20000, 6), 3073, 0, False),     # the dual copied: 24 steps
    ((600, 20000, 6), 0, 500, True),                                         # and columns of any length
    ((1000, 12000, 8), 11999, 0, True)])                                     # and few lines: 192 steps
@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
def test_longest_lines(gpu_ctx, shape, row, col, loop, precision):
    model = with_long_lines(*shape, row=row, col=col)
    if row:
        assert np.bincount(model.row_index).max() == row
    if col:
        assert np.diff(model.col_start).max() == col
    assert takes_the_loop(gpu_ctx, model, precision) == loop

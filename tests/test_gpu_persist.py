"""The persistent kernel of small and medium LPs (csrc/persist.cuh).

Sizes at the edges of its forms -- one block, a full cluster, the grid form
with and without the staged dual, the last sizes before the streaming kernels
-- against two other implementations: the CPU oracle in FP64, and the batched
engine's streaming kernels with the same lanes per line, whose iterates it
must reproduce (FP64 and FP32) up to the rounding of the reductions that feed
the step size and the primal weight.
"""
from __future__ import annotations

import numpy as np
import pytest

import mcpdlp
from mcpdlp import PdlpOptions, Precision, generators

pytestmark = pytest.mark.gpu


def rel(a, b) -> float:
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / max(1e-300, np.linalg.norm(np.asarray(b))))


def lanes(mean: float) -> int:
    g = 1
    while g < 32 and 8.0 * g <= mean:
        g *= 2
    return g


def uneven(seed: int, m: int, n: int) -> mcpdlp.Model:
    """Rows and columns of very different lengths, empty ones, free and boxed
    columns, ranged, one-sided and free rows."""
    r = np.random.default_rng(seed)
    entries = {}
    for j in range(n):
        for i in r.choice(m, size=int(r.integers(0, min(m, 5))), replace=False):
            entries[(int(i), j)] = float(r.normal())
    for j in range(0, n, 2):  # one long row
        entries[(m // 2, j)] = float(r.normal()) + 0.1
    for i in range(0, m, 3):  # one long column
        entries[(i, n // 2)] = float(r.normal()) + 0.1
    rows, cols = zip(*entries)
    act = r.normal(size=m)
    lo, hi = act - r.random(m), act + r.random(m)
    lo[::5] = -np.inf
    hi[1::5] = np.inf
    lo[2::5] = hi[2::5]
    lo[3::10], hi[3::10] = -np.inf, np.inf
    vl, vu = np.zeros(n), np.full(n, np.inf)
    vl[::4], vu[1::4] = -np.inf, 3.0
    return mcpdlp.from_triplets(m, n, list(rows), list(cols), list(entries.values()), objective=r.normal(size=n),
                                var_lower=vl, var_upper=vu, row_lower=lo, row_upper=hi)


def dense_rows(seed: int, m: int, n: int, count: int) -> mcpdlp.Model:
    """The first `count` rows full: one block's share of the matrix is larger
    than its shared memory."""
    r = np.random.default_rng(seed)
    k = 6
    col, row = [], []
    for j in range(n):
        row.append(np.concatenate([np.arange(count), np.sort(count + r.choice(m - count, size=k, replace=False))]))
        col.append(np.full(count + k, j))
    row, col = np.concatenate(row), np.concatenate(col)
    val = r.normal(size=len(row))
    x = np.where(r.random(n) < 0.3, 0.0, r.uniform(0.1, 5.0, n))
    b = np.bincount(row, weights=val * x[col], minlength=m)
    return mcpdlp.Model(m, n, np.arange(n + 1) * (count + k), row, val, r.normal(size=n), np.zeros(n), np.full(n, 10.0),
                        b, b)


CASES = {
    # cluster of one block: fewest lines; 512 lanes exactly; the next size takes two blocks
    "one_line": lambda: uneven(1, 1, 1),
    "one_block": lambda: generators.random_lp(1, 61, 149, 4),
    "block_edge": lambda: generators.random_lp(2, 200, 512, 6),
    "two_blocks": lambda: generators.random_lp(3, 200, 513, 6),
    "uneven": lambda: uneven(4, 131, 377),
    # largest FP64 and FP32 clusters, and the sizes one further (grid form)
    "cluster_last64": lambda: generators.random_lp(5, 1096, 3000, 6),
    "cluster_next64": lambda: generators.random_lp(6, 1097, 3000, 6),
    "cluster_last32": lambda: generators.random_lp(7, 1600, 4800, 6),
    "cluster_next32": lambda: generators.random_lp(8, 1601, 4800, 6),
    # grid form: staged dual, blocks without rows, a slice beyond shared memory, most lanes per block
    "grid_stage": lambda: generators.transport(9, 60, 200),
    "grid_few_rows": lambda: generators.random_lp(10, 40, 9000, 3),
    "grid_unfit": lambda: dense_rows(15, 3000, 12000, 20),
    "grid_wide": lambda: generators.random_lp(12, 20000, 56832, 8),
    # streaming kernels: one column more than the grid form takes; too many lanes; rows of one lane
    "too_wide": lambda: generators.random_lp(13, 20000, 56833, 8),
    "grid_dense": lambda: generators.random_lp(11, 3000, 12000, 90),
    "short_rows": lambda: generators.random_lp(14, 9000, 8000, 6),
}
STREAMING = {"too_wide", "grid_dense", "short_rows"}


@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_persistent_matches_streaming_kernels_and_oracle(gpu_ctx, oracle, name, precision):
    m = CASES[name]()
    # two whole restart periods and 17 iterations of a third
    o = PdlpOptions(max_iterations=97, precision=Precision[precision])
    o.set_tolerance(1e-14)
    res = gpu_ctx.solve(m, o)
    if name in STREAMING:
        assert res.extra["launches_by_kind"]["dual"] >= 80
    else:  # the whole loop: one launch for the whole periods, one for the rest
        assert res.extra["launches_by_kind"]["primal"] == 2
        assert res.extra["launches_by_kind"]["dual"] == 0
    nnz = max(m.nnz, 1)
    o.lanes_per_column, o.lanes_per_row = lanes(nnz / m.num_cols), lanes(nnz / m.num_rows)
    ref = gpu_ctx.solve_batch([m], o)[0]
    assert res.iterations == ref.iterations == 97
    # same operations in the same order; what differs is the grouping of FP64
    # reductions (1e-16 relative) amplified by at most the iteration count
    assert rel(res.primal, ref.primal) <= 1e-11
    assert rel(res.dual, ref.dual) <= 1e-11
    from mcpdlp import _abi
    oo = _abi.default_options_struct()
    oo.primal_tolerance = oo.dual_tolerance = oo.gap_tolerance = 1e-14
    oo.max_iterations = 97
    cpu = oracle.solve(m, oo)
    # FP64: rounding of 97 iterations; FP32 corrections: 2^-24 per operation,
    # 97 iterations of a few tens of terms
    tol = 1e-9 if precision == "fp64" else 1e-4
    assert rel(res.primal, cpu.primal) <= tol
    assert rel(res.dual, cpu.dual) <= tol


def test_step_size_and_restart_options(gpu_ctx, oracle):
    """The loop's options in both forms of the kernel: fixed step size, no
    restarts, restarts at every check, fixed weight, short periods."""
    from mcpdlp import RestartStrategy, _abi
    for model in (generators.random_lp(21, 100, 300, 5), generators.random_lp(22, 2000, 7000, 8)):
        for kw in (dict(adaptive_step_size=False), dict(restart_strategy=RestartStrategy.none),
                   dict(restart_strategy=RestartStrategy.fixed, adaptive_primal_weight=False),
                   dict(restart_every=7)):
            o = PdlpOptions(max_iterations=123, **kw)
            o.set_tolerance(1e-14)
            res = gpu_ctx.solve(model, o)
            oo = _abi.default_options_struct()
            oo.primal_tolerance = oo.dual_tolerance = oo.gap_tolerance = 1e-14
            oo.max_iterations = 123
            for k, v in kw.items():
                setattr(oo, k, int(v))
            cpu = oracle.solve(model, oo)
            assert res.iterations == cpu.iterations
            assert rel(res.primal, cpu.primal) <= 1e-9, kw
            assert rel(res.dual, cpu.dual) <= 1e-9, kw


@pytest.mark.parametrize("m,n", [(40, 90), (1500, 9000)])  # cluster and grid form
@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
def test_unscaled_rows_of_any_magnitude(gpu_ctx, m, n, precision):
    """Without equilibration a row's step size may be any number: the division
    by it must be the streaming kernels' one where its reciprocal leaves the
    safe range."""
    model = generators.random_lp(31, m, n, 5)
    top = 20 if precision == "fp32_refine" else 60
    scale = 10.0 ** np.linspace(-top, top, m)[np.random.default_rng(3).permutation(m)]
    model.value = model.value * scale[model.row_index]
    model.row_lower, model.row_upper = model.row_lower * scale, model.row_upper * scale + scale
    # no step-size rule and no restart check: nothing depends on a reduction's order
    o = PdlpOptions(max_iterations=37, precision=Precision[precision], ruiz_scaling=False, adaptive_step_size=False,
                    initial_primal_weight=1.0)
    o.set_tolerance(1e-14)
    res = gpu_ctx.solve(model, o)
    o.lanes_per_column, o.lanes_per_row = lanes(model.nnz / n), lanes(model.nnz / m)
    ref = gpu_ctx.solve_batch([model], o)[0]
    for a, b in ((res.primal, ref.primal), (res.dual, ref.dual)):
        ok = np.isfinite(b)
        np.testing.assert_array_equal(np.isfinite(a), ok)
        np.testing.assert_allclose(np.asarray(a)[ok], np.asarray(b)[ok], rtol=1e-11, atol=0)


@pytest.mark.parametrize("m,n", [(40, 90), (1500, 9000)])  # cluster and grid form
def test_equality_row_whose_step_size_is_zero(gpu_ctx, m, n):
    """Entries whose sum overflows make the row's norm infinite and its step size
    0: the quotient 0 / 0 is not a number in any form, an equality row's included."""
    model = generators.random_lp(33, m, n, 5)
    model.value[model.row_index == 3] = 1.7e308
    assert np.count_nonzero(model.row_index == 3) > 1 and model.row_lower[3] == model.row_upper[3]
    o = PdlpOptions(max_iterations=80, ruiz_scaling=False, adaptive_step_size=False, initial_primal_weight=1.0)
    o.set_tolerance(1e-14)
    res = gpu_ctx.solve(model, o)
    assert res.extra["launches_by_kind"]["dual"] == 0
    ref = gpu_ctx.solve_batch([model], o)[0]
    assert ref.status == res.status == mcpdlp.PdlpStatus.numerical_failure
    assert ref.iterations == res.iterations
    assert np.isnan(ref.dual[3]) and np.isnan(res.dual[3])


@pytest.mark.parametrize("m,n", [(40, 90), (2000, 9000)])  # cluster and grid form
@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
def test_long_restart_periods_take_several_launches(gpu_ctx, m, n, precision):
    """No launch runs more than 1280 iterations: a restart period of 3001 takes
    three, and so does the rest of 2697; the iterates are the streaming kernels'."""
    model = generators.random_lp(34, m, n, 5)
    # no step-size rule and no restart: nothing depends on a reduction's order
    o = PdlpOptions(max_iterations=2 * 3001 + 2697, restart_every=3001, precision=Precision[precision],
                    adaptive_step_size=False, restart_strategy=mcpdlp.RestartStrategy.none, initial_primal_weight=1.0)
    o.set_tolerance(1e-15)
    res = gpu_ctx.solve(model, o)
    assert res.extra["launches_by_kind"]["primal"] == 9
    o.lanes_per_column, o.lanes_per_row = lanes(model.nnz / n), lanes(model.nnz / m)
    ref = gpu_ctx.solve_batch([model], o)[0]
    assert res.iterations == ref.iterations == 8699
    assert rel(res.primal, ref.primal) <= 1e-11
    assert rel(res.dual, ref.dual) <= 1e-11
    # driven period by period: the same launches, the same result
    s = gpu_ctx.begin(model, o)
    while not s.iterate(1)[1]:
        pass
    step = s.finish()
    np.testing.assert_array_equal(step.primal, res.primal)
    np.testing.assert_array_equal(step.dual, res.dual)


def test_long_restart_periods_keep_the_step_size_rule(gpu_ctx):
    """The rule runs on every tenth iteration wherever a launch begins: a period of
    2563 split in three against the same iterations in periods that are not, with
    no restarts (a check that restarts nothing changes no iterate)."""
    model = generators.random_lp(35, 300, 900, 5)
    out = []
    for every in (2563, 1281):
        o = PdlpOptions(max_iterations=2562, restart_every=every, restart_strategy=mcpdlp.RestartStrategy.none)
        o.set_tolerance(1e-300)
        out.append(gpu_ctx.solve(model, o))
    one_launch = PdlpOptions(max_iterations=2562, restart_every=183, restart_strategy=mcpdlp.RestartStrategy.none)
    one_launch.set_tolerance(1e-300)
    expect = gpu_ctx.solve(model, one_launch)
    for r in out:
        np.testing.assert_array_equal(r.primal, expect.primal)
        np.testing.assert_array_equal(r.dual, expect.dual)

"""The persistent loop's form of one block per SM on models whose lines are of
every kind: empty rows and columns (which wait for nobody), long and short ones,
free and boxed columns, ranged, one-sided, free and equality rows -- with the
dual gathered from the other blocks, and with a copy of it in every block."""
from __future__ import annotations

import numpy as np
import pytest

import mcpdlp
from mcpdlp import PdlpOptions, Precision, _abi

pytestmark = pytest.mark.gpu


def rel(a, b) -> float:
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / max(1e-300, np.linalg.norm(np.asarray(b))))


def uneven(seed, m, n, most, row=0, col=0):
    """Columns of 0 to `most` entries at rows that are not a multiple of 7 (those
    stay empty), one row of `row` entries and one column of `col`."""
    r = np.random.default_rng(seed)
    full = np.flatnonzero(np.arange(m) % 7)
    pairs = [(int(i), j) for j in range(n) for i in r.choice(full, size=int(r.integers(0, most + 1)), replace=False)]
    pairs += [(1, j) for j in r.choice(n, size=row, replace=False).tolist()]
    pairs += [(int(i), n // 2) for i in r.choice(full, size=col, replace=False)]
    i, j = np.array(sorted(set(pairs), key=lambda p: (p[1], p[0]))).T
    v = r.normal(size=len(i))
    x = r.uniform(0.0, 2.0, n)
    act = np.bincount(i, weights=v * x[j], minlength=m)
    lo, hi = act - r.random(m), act + r.random(m)
    lo[::5] = -np.inf
    hi[1::5] = np.inf
    lo[2::5] = hi[2::5] = act[2::5]
    lo[3::10], hi[3::10] = -np.inf, np.inf
    vl, vu = np.zeros(n), np.full(n, np.inf)
    vl[::4], vu[1::4] = -np.inf, 3.0
    return mcpdlp.Model(m, n, np.concatenate([[0], np.cumsum(np.bincount(j, minlength=n))]), i, v, r.normal(size=n), vl, vu,
                        lo, hi)


CASES = {
    "gathered": lambda: uneven(1, 2500, 9000, 8),
    "gathered_long_row": lambda: uneven(2, 2500, 5000, 12, row=100),  # 14 of at most 16 steps
    "copied": lambda: uneven(3, 150, 9000, 8),
    "copied_long_lines": lambda: uneven(4, 250, 9000, 9, row=4000, col=200),
}


@pytest.mark.parametrize("adaptive", [True, False])
@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_uneven_lines(gpu_ctx, oracle, name, precision, adaptive):
    m = CASES[name]()
    assert np.any(np.diff(m.col_start) == 0) and np.any(np.bincount(m.row_index, minlength=m.num_rows) == 0)
    staged = m.num_rows * 148 <= 2 * m.nnz
    assert staged == name.startswith("copied")
    o = PdlpOptions(max_iterations=97, precision=Precision[precision], adaptive_step_size=adaptive)
    o.set_tolerance(1e-14)
    res = gpu_ctx.solve(m, o)
    assert res.extra["launches_by_kind"]["dual"] == 0
    o.shared_device = True
    ref = gpu_ctx.solve(m, o)
    assert ref.extra["launches_by_kind"]["dual"] > 0
    assert res.iterations == ref.iterations == 97
    # same operations in the same order; what differs is the grouping of FP64
    # reductions (1e-16 relative) amplified by at most the iteration count
    assert rel(res.primal, ref.primal) <= 1e-11
    assert rel(res.dual, ref.dual) <= 1e-11
    oo = _abi.default_options_struct()
    oo.primal_tolerance = oo.dual_tolerance = oo.gap_tolerance = 1e-14
    oo.max_iterations = 97
    oo.adaptive_step_size = int(adaptive)
    cpu = oracle.solve(m, oo)
    # FP64: rounding of 97 iterations; FP32 corrections: 2^-24 per operation,
    # 97 iterations of a few tens of terms
    tol = 1e-9 if precision == "fp64" else 1e-4
    assert rel(res.primal, cpu.primal) <= tol
    assert rel(res.dual, cpu.dual) <= tol

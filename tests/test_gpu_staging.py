"""Batched and variant solves move their many small arrays through two pinned
buffers in turn: arrays around the size that is copied directly, runs that
fill a buffer, wrap round both several times and are broken by empty LPs."""
from __future__ import annotations

import numpy as np
import pytest

import mcpdlp
from mcpdlp import PdlpOptions, generators

pytestmark = pytest.mark.gpu


def close(a, b):
    # FP64 solves of 120 iterations: rounding of reductions in another grouping
    return np.linalg.norm(a - b) <= 1e-9 * max(1e-300, np.linalg.norm(b))


def test_batch_of_small_and_large_arrays(gpu_ctx):
    # 16384 columns: objective and bounds of exactly 128 KiB, one column more, far more, and tiny ones between
    sizes = [(4, 9, 3), (5000, 16384, 2), (7, 20, 3), (5000, 16385, 2), (9000, 30011, 4)] + [(30 + i, 90 + i, 4) for i in range(60)]
    models = [generators.random_lp(50 + i, *s) for i, s in enumerate(sizes)]
    empty = mcpdlp.from_triplets(0, 3, [], [], [], objective=[1.0, 2.0, 3.0], var_lower=[0.0] * 3, var_upper=[1.0] * 3,
                                 row_lower=[], row_upper=[])
    models.insert(2, empty)
    o = PdlpOptions(max_iterations=120)
    o.set_tolerance(1e-13)
    starts = [None if i % 2 else np.full(m.num_cols, 0.25) for i, m in enumerate(models)]
    duals = [None if i % 3 else np.full(m.num_rows, -0.5) for i, m in enumerate(models)]
    for x0, y0 in ((None, None), (starts, duals)):
        res = gpu_ctx.solve_batch(models, o, initial_primal=x0, initial_dual=y0)
        for i, (m, r) in enumerate(zip(models, res)):
            if m is empty:
                assert r.message == "trivial"
                continue
            s = PdlpOptions(max_iterations=120)
            s.set_tolerance(1e-13)
            if x0 is not None:
                s.initial_primal, s.initial_dual = x0[i], y0[i]
            solo = gpu_ctx.solve(m, s)
            assert close(r.primal, solo.primal) and close(r.dual, solo.dual), m.name


@pytest.mark.parametrize("count", [1, 3, 90])
def test_variants_wrap_round_the_buffers(gpu_ctx, count):
    base = generators.random_lp(77, 1000, 3000, 6)  # 24 KB of bounds: 21 variants to a buffer
    r = np.random.default_rng(5)
    lo = [base.var_lower + 0.1 * (r.random(3000) < 0.01) for _ in range(count)]
    hi = [None if i == 1 else base.var_upper - r.random(3000) for i in range(count)]
    o = PdlpOptions(max_iterations=120)
    o.set_tolerance(1e-13)
    res = gpu_ctx.solve_variants(base, lo, hi, o)
    for i in sorted({0, count // 2, count - 1, min(1, count - 1)}):
        v = base.copy()
        v.var_lower = lo[i]
        v.var_upper = base.var_upper if hi[i] is None else hi[i]
        solo = gpu_ctx.solve(v, o)
        assert close(res[i].primal, solo.primal) and close(res[i].dual, solo.dual)


def test_invalid_member_is_found_in_its_own_numbering(gpu_ctx):
    for at, what in ((0, "row_index"), (2, "row_index"), (1, "value"), (2, "order")):
        models = [generators.random_lp(90 + i, 50 + i, 150, 4) for i in range(3)]
        bad = models[at]
        if what == "row_index":
            bad.row_index[-1] = bad.num_rows  # in range of the packed rows, not of the LP's own
        elif what == "value":
            bad.value[7] = 0.0
        else:
            bad.row_index[[0, 1]] = bad.row_index[[1, 0]]
        with pytest.raises(ValueError, match="invalid CSC matrix in the batch"):
            gpu_ctx.solve_batch(models, PdlpOptions())


def test_call_after_one_that_failed_between_its_uploads(gpu_ctx):
    class NoColumns(mcpdlp.Model):
        def to_struct(self):
            s = super().to_struct()
            s.col_start = None
            return s

    good = [generators.random_lp(60 + i, 70 + 9 * i, 200, 4) for i in range(3)]
    m = good[1]
    broken = NoColumns(m.num_rows, m.num_cols, m.col_start, m.row_index, m.value, m.objective, m.var_lower,
                       m.var_upper, m.row_lower, m.row_upper)
    o = PdlpOptions(max_iterations=120)
    o.set_tolerance(1e-13)
    expect = gpu_ctx.solve_batch(good, o)
    with pytest.raises(Exception):
        gpu_ctx.solve_batch([good[0], broken, good[2]], o)
    for r, e in zip(gpu_ctx.solve_batch(good, o), expect):
        np.testing.assert_array_equal(r.primal, e.primal)
        np.testing.assert_array_equal(r.dual, e.dual)

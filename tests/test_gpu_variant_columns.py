"""Variants of an LP with long columns, whose indices the primal step asks for
ahead of the gathers: against solo solves, on both sides of the rule."""
from __future__ import annotations

import numpy as np
import pytest

import mcpdlp
from mcpdlp import PdlpOptions, RestartStrategy, generators

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("longest", [64, 65, 72, 300])  # above 64 a column's indices are asked for ahead
@pytest.mark.parametrize("count", [1, 33, 130])
def test_long_columns(gpu_ctx, count, longest):
    base = generators.random_lp(81, 400, 1200, 5)
    r = np.random.default_rng(longest)
    col = {7: np.sort(r.choice(400, size=longest, replace=False)), 900: np.sort(r.choice(400, size=longest - 3, replace=False))}
    parts = [col.get(j, base.row_index[base.col_start[j]:base.col_start[j + 1]]) for j in range(1200)]
    rows = np.concatenate(parts)
    val = r.normal(size=len(rows))
    b = np.bincount(rows, weights=val * np.repeat(base.info["x_star"], [len(q) for q in parts]), minlength=400)
    lp = mcpdlp.Model(400, 1200, np.concatenate([[0], np.cumsum([len(q) for q in parts])]), rows, val, base.objective,
                      base.var_lower, base.var_upper, b, b)
    lo = [lp.var_lower + 0.05 * (r.random(1200) < 0.02) for _ in range(count)]
    o = PdlpOptions(max_iterations=120, adaptive_step_size=False, adaptive_primal_weight=False,
                    restart_strategy=RestartStrategy.none)
    o.set_tolerance(1e-13)
    res = gpu_ctx.solve_variants(lp, lo, [None] * count, o)
    for q in sorted({0, count // 2, count - 1}):
        v = lp.copy()
        v.var_lower = lo[q]
        solo = gpu_ctx.solve(v, o)
        for a, e in ((res[q].primal, solo.primal), (res[q].dual, solo.dual)):
            # the solo engine sums in another order: 120 iterations of rounding, far below 1e-9
            assert np.linalg.norm(a - e) <= 1e-9 * np.linalg.norm(e)

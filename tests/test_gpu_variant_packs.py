"""The iterations of variant solves without a step-size probe run in packs of
variants or, for few variants, with the rows' sums split over lanes.  Neither
changes the order of any sum: with the step size, weight and restarts fixed, a
variant's iterates are the same bits whatever the number of variants."""
from __future__ import annotations

import numpy as np
import pytest

import mcpdlp
from mcpdlp import PdlpOptions, PdlpStatus, Precision, RestartStrategy

pytestmark = pytest.mark.gpu


def ragged(m, n):
    """Feasible at a point of [0.2, 0.8]^n.  Row i has i mod 41 entries (every tail, empty rows, several windows);
    columns of 0 to about 60 entries."""
    r = np.random.default_rng(m + n)
    rows, cols = [], []
    for i in range(m):
        c = (n * r.random(4 * 41) ** 2).astype(int)
        c = np.unique(c)
        c = r.permutation(c)[: i % 41]
        rows += [i] * len(c)
        cols += c.tolist()
    vals = r.uniform(0.5, 1.5, len(rows)) * r.choice([-1.0, 1.0], len(rows))
    x0 = r.uniform(0.2, 0.8, n)
    ax = np.zeros(m)
    np.add.at(ax, rows, vals * x0[cols])
    return mcpdlp.from_triplets(m, n, rows, cols, vals, objective=r.uniform(-1, 1, n), var_lower=np.zeros(n),
                                var_upper=np.ones(n), row_lower=ax - 0.1, row_upper=np.where(np.arange(m) % 3, ax + 0.1, np.inf))


@pytest.mark.parametrize("precision", [Precision.fp64, Precision.fp32_refine])
@pytest.mark.parametrize("m,n", [(1200, 2500), (37, 90)])
def test_same_bits_for_any_number_of_variants(gpu_ctx, precision, m, n):
    base = ragged(m, n)
    r = np.random.default_rng(9)
    lo = [np.where(r.random(n) < 0.05, r.uniform(0, 0.2, n), 0.0) for _ in range(300)]
    hi = [np.where(r.random(n) < 0.05, r.uniform(0.8, 1, n), 1.0) for _ in range(300)]
    hi[7] = hi[7].copy()
    hi[7][3] = -1.0  # crossed bounds: finished before the first iteration
    # 57: the last iterations end inside a period
    o = PdlpOptions(max_iterations=57, precision=precision, adaptive_step_size=False, adaptive_primal_weight=False,
                    restart_strategy=RestartStrategy.none)
    o.set_tolerance(1e-14)
    alone = {}
    for count in (1, 2, 9, 33, 96, 128, 300):  # at 1200 rows up to 32 variants are split, more go in packs
        res = gpu_ctx.solve_variants(base, lo[:count], hi[:count], o)
        for b, x in enumerate(res):
            if b == 7:
                assert x.status == PdlpStatus.infeasible_or_unbounded and x.extra["certificate"] == "crossed_bounds"
                continue
            assert x.iterations == 57
            first = alone.setdefault(b, x)
            assert np.array_equal(x.primal, first.primal) and np.array_equal(x.dual, first.dual), (count, b)
    if precision == Precision.fp64:
        # the solo engine sums in another order: 57 iterations of rounding, far below 1e-9
        for b in (0, 8, 31, 299):
            v = base.copy()
            v.var_lower, v.var_upper = lo[b], hi[b]
            s = gpu_ctx.solve(v, o)
            for p, q in ((alone[b].primal, s.primal), (alone[b].dual, s.dual)):
                assert np.linalg.norm(p - q) <= 1e-9 * np.linalg.norm(q)

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

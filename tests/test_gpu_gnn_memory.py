"""The learned start's workspace: an allocation that fails while it grows leaves
the network without one, not with freed buffers of the old size."""
from __future__ import annotations

import numpy as np
import pytest

import mcpdlp
from mcpdlp import _lib, generators
from mcpdlp.learn import Target, WarmStartNet

pytestmark = pytest.mark.gpu


def target(seed, m, n):
    lp = generators.random_lp(seed, m, n, 4)
    r = np.random.default_rng(seed)
    return Target(lp, r.uniform(0, 2, n), r.normal(0, 0.5, m), 0.4)


@pytest.mark.parametrize("call", ["predict", "loss_and_grad"])
def test_failed_growth_leaves_no_stale_workspace(call):
    small, large = target(1, 30, 70), target(2, 300, 900)
    run = {"predict": lambda net, t: net.predict(t.model), "loss_and_grad": lambda net, t: net.loss_and_grad(t)}[call]
    net, lib = WarmStartNet(0, 3, 5), _lib.engine()
    expect_small, expect_large = run(net, small), run(WarmStartNet(0, 3, 5), large)
    try:
        for _ in range(2):
            lib.mc_test_inject_alloc_failures(1)  # growth to `large` fails at its first buffer
            with pytest.raises(mcpdlp.EngineError, match="out_of_memory"):
                run(net, large)
            lib.mc_test_inject_alloc_failures(1)  # so the small instance has to allocate too: nothing is left over
            with pytest.raises(mcpdlp.EngineError, match="out_of_memory"):
                run(net, small)
            lib.mc_test_inject_alloc_failures(0)
            for a, e in zip(run(net, small), expect_small):
                np.testing.assert_array_equal(a, e)
        for a, e in zip(run(net, large), expect_large):
            np.testing.assert_array_equal(a, e)
    finally:
        lib.mc_test_inject_alloc_failures(0)
        net.close()

"""The learned start's workspaces: an allocation that fails while one grows leaves
the network without it, not with freed buffers of the old size; a prediction
holds none of the gradient's."""
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


def test_prediction_allocates_no_gradient_scratch():
    """A prediction holds its activations only: four pairs of hidden states and
    of gathered ones.  The gradient's buffers come with the first gradient."""
    import torch
    t = target(3, 60_000, 300_000)
    WarmStartNet(0, 3, 5).predict(t.model)  # the pool of instance buffers has its size
    net = WarmStartNet(0, 3, 5)
    before = torch.cuda.mem_get_info()[0]
    x, y, w = net.predict(t.model)
    used = before - torch.cuda.mem_get_info()[0]
    nodes = 360_000
    forward = 4 * 2 * nodes * 64 * 4 + nodes * 4
    assert used <= forward + (64 << 20)  # and each buffer's rounding to 2 MiB pages
    net.loss_and_grad(t)
    assert before - torch.cuda.mem_get_info()[0] > used
    for a, b in zip(net.predict(t.model), (x, y, w)):
        np.testing.assert_array_equal(a, b)
    net.close()


def test_gradient_after_its_own_growth_failed():
    small, large = target(1, 30, 70), target(2, 300, 900)
    net, lib = WarmStartNet(0, 3, 5), _lib.engine()
    try:
        expect = net.loss_and_grad(small)
        net.predict(large.model)  # the activations have grown, the gradient's buffers have not
        lib.mc_test_inject_alloc_failures(1)
        with pytest.raises(mcpdlp.EngineError, match="out_of_memory"):
            net.loss_and_grad(large)
        lib.mc_test_inject_alloc_failures(0)
        for a, e in zip(net.loss_and_grad(small), expect):
            np.testing.assert_array_equal(a, e)
    finally:
        lib.mc_test_inject_alloc_failures(0)
        net.close()

"""Contexts used from several host threads at once: every solve's result is that
of the context alone, bit for bit, whatever else runs on the device."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import mcpdlp
from mcpdlp import PdlpOptions, Precision, generators

pytestmark = pytest.mark.gpu

# a cluster, one block per SM (two kinds fit side by side, or not), the streaming kernels
SHAPES = [(300, 900, 5), (4001, 12007, 9), (10000, 30000, 8), (30000, 90000, 6)]


def opts(**kw):
    o = PdlpOptions(max_iterations=317, **kw)
    o.set_tolerance(1e-14)
    return o


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
@pytest.mark.parametrize("shapes", [SHAPES, SHAPES[1:2] * 3, SHAPES[2:3] * 2], ids=["all", "side_by_side", "in_turn"])
def test_solves_from_several_threads(shapes, precision, shared):
    models = [generators.random_lp(40 + q, *s) for q, s in enumerate(shapes)]
    ctxs = [mcpdlp.Context(0) for _ in shapes]
    o = opts(precision=Precision[precision], shared_device=shared)
    expect = [c.solve(m, o) for c, m in zip(ctxs, models)]
    failed = []

    def work(q):
        try:
            for _ in range(4):
                r = ctxs[q].solve(models[q], o)
                np.testing.assert_array_equal(r.primal, expect[q].primal)
                np.testing.assert_array_equal(r.dual, expect[q].dual)
        except BaseException as e:  # noqa: BLE001 -- reported by the main thread
            failed.append((q, e))

    threads = [threading.Thread(target=work, args=(q,)) for q in range(len(ctxs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in ctxs:
        c.close()
    assert not failed


def test_shared_device_takes_kernels_that_overlap(gpu_ctx):
    """Only where the form for a solve alone would take every SM; the same iterates."""
    for shape, changes in zip(SHAPES, (False, True, True, False)):
        m = generators.random_lp(50, *shape)
        kw = dict(adaptive_step_size=False, initial_primal_weight=1.0,
                  restart_strategy=mcpdlp.RestartStrategy.none)  # nothing depends on a reduction's order
        alone, shared = (gpu_ctx.solve(m, opts(shared_device=s, **kw)) for s in (False, True))
        assert (alone.extra["launches_by_kind"]["dual"] != shared.extra["launches_by_kind"]["dual"]) == changes
        np.testing.assert_allclose(shared.primal, alone.primal, rtol=1e-11, atol=0)
        np.testing.assert_allclose(shared.dual, alone.dual, rtol=1e-11, atol=0)

"""Waits inside the cooperative kernels that run out: with a limit of one poll an
ordinary wait on healthy inputs gives up, the kernel returns, the call ends with
an error, and the next call on the same context is right."""
from __future__ import annotations

import ctypes as C
import time
from contextlib import contextmanager

import numpy as np
import pytest

import mcpdlp
from mcpdlp import PdlpOptions, Precision, _abi, _lib, generators

pytestmark = pytest.mark.gpu

TIMED_OUT = "cuda.*timed out"

# one per form of the loop: a cluster, one block per SM (with and without the
# staged dual), the streaming kernels
MODELS = {
    "cluster": lambda: generators.random_lp(1, 500, 1500, 6),
    "grid": lambda: generators.random_lp(2, 4000, 12000, 9),
    "grid_staged": lambda: generators.transport(3, 60, 200),
    "streaming": lambda: generators.random_lp(4, 30000, 90000, 6),
}


@contextmanager
def limits(ctx, barrier=0, entry=0, per_nonzero=0):
    lib = _lib.engine()
    _lib.check(lib.mc_test_set_wait_limits(ctx.handle, barrier, entry, per_nonzero))
    try:
        yield
    finally:
        _lib.check(lib.mc_test_set_wait_limits(ctx.handle, 0, 0, 2))


def opts(iterations=97, **kw):
    o = PdlpOptions(max_iterations=iterations, **kw)
    o.set_tolerance(1e-14)
    return o


def same(a, b):
    np.testing.assert_array_equal(a.primal, b.primal)
    np.testing.assert_array_equal(a.dual, b.dual)


@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_barrier_between_ruiz_passes(gpu_ctx, name, precision):
    m, o = MODELS[name](), opts(precision=Precision[precision])
    expect = gpu_ctx.solve(m, o)
    with limits(gpu_ctx, barrier=1, entry=100):
        with pytest.raises(mcpdlp.EngineError, match=TIMED_OUT):
            gpu_ctx.solve(m, o)
    same(gpu_ctx.solve(m, o), expect)


def test_barrier_between_ruiz_passes_of_batches_and_variants(gpu_ctx):
    models = [generators.random_lp(s, 300 * s, 900 * s, 5) for s in (1, 2, 3)]
    o, base = opts(), MODELS["cluster"]()
    lo, hi = [None, base.var_lower + 0.01], [None, None]
    expect, expect_v = gpu_ctx.solve_batch(models, o), gpu_ctx.solve_variants(base, lo, hi, o)
    with limits(gpu_ctx, barrier=1):
        with pytest.raises(mcpdlp.EngineError, match=TIMED_OUT):
            gpu_ctx.solve_batch(models, o)
        with pytest.raises(mcpdlp.EngineError, match=TIMED_OUT):
            gpu_ctx.solve_variants(base, lo, hi, o)
    for a, b in zip(gpu_ctx.solve_batch(models, o), expect):
        same(a, b)
    for a, b in zip(gpu_ctx.solve_variants(base, lo, hi, o), expect_v):
        same(a, b)


def test_barrier_of_the_equilibration_calls(gpu_ctx):
    import torch
    m, lib = generators.random_lp(5, 900, 5000, 9, family="precision"), _lib.engine()

    def call(canonical):
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        cs, ri, v = dev(m.col_start), dev(m.row_index), dev(m.value)
        rs = torch.zeros(m.num_rows + 1, dtype=torch.int32, device="cuda")
        ci = torch.zeros(m.nnz, dtype=torch.int32, device="cuda")
        rv = torch.zeros(m.nnz, dtype=torch.float64, device="cuda")
        row = torch.zeros(2, m.num_rows, dtype=torch.float64, device="cuda")
        col = torch.zeros(2, m.num_cols, dtype=torch.float64, device="cuda")
        it, conv = C.c_int64(-1), C.c_int32(-1)
        if canonical:
            rhs, obj = dev(np.ones(m.num_rows)), dev(m.objective)
            rc = lib.mc_ruiz_equilibrate_canonical(
                gpu_ctx.handle, m.num_rows, m.num_cols, m.nnz, cs.data_ptr(), ri.data_ptr(), v.data_ptr(), rhs.data_ptr(),
                obj.data_ptr(), 10, 1e-3, 1e-4, 1e4, row[0].data_ptr(), col[0].data_ptr(), row[1].data_ptr(),
                col[1].data_ptr(), C.addressof(it), C.addressof(conv))
        else:
            _lib.check(lib.mc_csc_to_csr(gpu_ctx.handle, m.num_rows, m.num_cols, m.nnz, cs.data_ptr(), ri.data_ptr(),
                                         v.data_ptr(), rs.data_ptr(), ci.data_ptr(), rv.data_ptr()))
            rc = lib.mc_ruiz_equilibrate(gpu_ctx.handle, m.num_rows, m.num_cols, m.nnz, cs.data_ptr(), ri.data_ptr(),
                                         v.data_ptr(), rs.data_ptr(), ci.data_ptr(), rv.data_ptr(), None, None, None, None,
                                         None, 10, row[0].data_ptr(), col[0].data_ptr(), C.addressof(it))
        torch.cuda.synchronize()
        return rc, row.cpu().numpy(), col.cpu().numpy(), it.value

    for canonical in (False, True):
        expect = call(canonical)
        assert expect[0] == _abi.MC_OK
        with limits(gpu_ctx, barrier=1):
            assert call(canonical)[0] == _abi.MC_ERR_CUDA
            assert "timed out" in _lib.last_error()
        again = call(canonical)
        assert again[0] == _abi.MC_OK and again[3] == expect[3]
        np.testing.assert_array_equal(again[1], expect[1])
        np.testing.assert_array_equal(again[2], expect[2])


@pytest.mark.parametrize("iterations", [97, 17])  # whole restart periods; one partial launch only
@pytest.mark.parametrize("name", ["grid", "grid_staged"])
def test_barrier_at_the_start_of_the_loop(gpu_ctx, name, iterations):
    m, o = MODELS[name](), opts(iterations, ruiz_scaling=False)
    expect = gpu_ctx.solve(m, o)
    with limits(gpu_ctx, barrier=1, entry=100):
        with pytest.raises(mcpdlp.EngineError, match=TIMED_OUT):
            gpu_ctx.solve(m, o)
    same(gpu_ctx.solve(m, o), expect)


@pytest.mark.parametrize("polls", [1, 10])
@pytest.mark.parametrize("iterations", [97, 40, 17, 0])
@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
@pytest.mark.parametrize("name", ["grid", "grid_staged"])
def test_entry_of_another_block(gpu_ctx, name, precision, iterations, polls):
    """The gathers of every block run out, in iterations, checks or reductions."""
    m, o = MODELS[name](), opts(iterations, precision=Precision[precision])
    expect = gpu_ctx.solve(m, o)
    with limits(gpu_ctx, entry=polls):
        with pytest.raises(mcpdlp.EngineError, match=TIMED_OUT):
            gpu_ctx.solve(m, o)
    same(gpu_ctx.solve(m, o), expect)


@pytest.mark.parametrize("block", [0, 1, 77])  # block 0 adds up the partials of all
@pytest.mark.parametrize("iterations", [97, 40, 17, 0])
@pytest.mark.parametrize("name", ["grid", "grid_staged"])
def test_one_block_of_many(gpu_ctx, name, iterations, block):
    """One block's waits run out, all others' are served: the next reduction (in the
    first iteration, or the check without any) tells every block, so that none goes
    on with a result made of stale entries nor waits (for seconds, with the limits
    as they are) for the one that left."""
    m, o = MODELS[name](), opts(iterations)
    expect = gpu_ctx.solve(m, o)
    lib = _lib.engine()
    _lib.check(lib.mc_test_fail_block(gpu_ctx.handle, block))
    try:
        began = time.monotonic()
        with pytest.raises(mcpdlp.EngineError, match=TIMED_OUT):
            gpu_ctx.solve(m, o)
        assert time.monotonic() - began < 1.0
    finally:
        _lib.check(lib.mc_test_fail_block(gpu_ctx.handle, -1))
    same(gpu_ctx.solve(m, o), expect)


@pytest.mark.parametrize("block", [0, 1, 77])
@pytest.mark.parametrize("iterations", [97, 17])
@pytest.mark.parametrize("name", ["grid", "grid_staged"])
def test_one_block_runs_ahead_of_the_others(gpu_ctx, name, iterations, block):
    """Without the step-size rule's reductions the block overwrites entries that
    others have not read: their waits run out in turn, and the call fails."""
    m, o = MODELS[name](), opts(iterations, adaptive_step_size=False)
    expect = gpu_ctx.solve(m, o)
    lib = _lib.engine()
    _lib.check(lib.mc_test_fail_block(gpu_ctx.handle, block))
    try:
        with limits(gpu_ctx, entry=20_000, per_nonzero=2):
            with pytest.raises(mcpdlp.EngineError, match=TIMED_OUT):
                gpu_ctx.solve(m, o)
    finally:
        _lib.check(lib.mc_test_fail_block(gpu_ctx.handle, -1))
    same(gpu_ctx.solve(m, o), expect)


def test_limit_of_the_ruiz_barrier_grows_with_the_matrix(gpu_ctx):
    """One row with an entry in every column among short rows, which get one lane
    each: the blocks of the short ones wait for its lane, longer the longer it is."""
    m, n = 25_000, 100_000
    r = np.random.default_rng(8)
    rows = np.empty((n, 2), np.int32)
    rows[:, 0], rows[:, 1] = 0, r.integers(1, m, n)  # 8 entries a row or fewer on average
    some = r.random(n) < 0.9
    start = np.concatenate([[0], np.cumsum(1 + some)])
    keep = np.stack([np.ones(n, bool), some], 1)
    index = rows[keep]
    lp = mcpdlp.Model(m, n, start, index, r.uniform(0.5, 1.5, len(index)), r.normal(size=n), np.zeros(n), np.ones(n),
                      np.full(m, -np.inf), np.full(m, 50.0))
    assert lp.nnz < 8 * m
    o = opts(2, ruiz_iterations=2)
    expect = gpu_ctx.solve(lp, o)
    with limits(gpu_ctx, barrier=2000):  # 2 ms: not enough for 100,000 entries by one lane
        with pytest.raises(mcpdlp.EngineError, match=TIMED_OUT):
            gpu_ctx.solve(lp, o)
    with limits(gpu_ctx, barrier=2000, per_nonzero=2):
        same(gpu_ctx.solve(lp, o), expect)

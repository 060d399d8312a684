"""Ruiz equilibration in one cooperative launch (k_ruiz): every number of lanes
per line on either side, one block and many, line lengths around a lane's
windows, pass counts from none to the limit -- bit for bit the oracle's scaled
matrix, scales and pass count; and per LP in a batch."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import mcpdlp
from mcpdlp import PdlpOptions, _lib, generators

pytestmark = pytest.mark.gpu


def scaled(gpu_ctx, m, passes):
    import torch
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    cs, ri, v = dev(m.col_start), dev(m.row_index), dev(m.value)
    rs = torch.zeros(m.num_rows + 1, dtype=torch.int32, device="cuda")
    ci = torch.zeros(m.nnz + 1, dtype=torch.int32, device="cuda")
    rv = torch.zeros(m.nnz + 1, dtype=torch.float64, device="cuda")
    lib = _lib.engine()
    _lib.check(lib.mc_csc_to_csr(gpu_ctx.handle, m.num_rows, m.num_cols, m.nnz, cs.data_ptr(), ri.data_ptr(),
                                 v.data_ptr(), rs.data_ptr(), ci.data_ptr(), rv.data_ptr()))
    row_scale = torch.zeros(m.num_rows, dtype=torch.float64, device="cuda")
    col_scale = torch.zeros(m.num_cols, dtype=torch.float64, device="cuda")
    it = C.c_int64(-1)
    _lib.check(lib.mc_ruiz_equilibrate(gpu_ctx.handle, m.num_rows, m.num_cols, m.nnz, cs.data_ptr(), ri.data_ptr(),
                                       v.data_ptr(), rs.data_ptr(), ci.data_ptr(), rv.data_ptr(), None, None, None, None,
                                       None, passes, row_scale.data_ptr(), col_scale.data_ptr(), C.addressof(it)))
    order = np.lexsort((np.repeat(np.arange(m.num_cols), np.diff(m.col_start)), m.row_index))
    return (v.cpu().numpy(), rv.cpu().numpy()[:m.nnz], order, row_scale.cpu().numpy(), col_scale.cpu().numpy(), it.value)


@pytest.mark.parametrize("shape", [(1, 1, 1), (40, 300, 1), (300, 257, 3), (900, 5000, 9), (600, 4000, 17),
                                   (5000, 300, 40), (700, 2000, 130), (20000, 70000, 5)])
@pytest.mark.parametrize("passes", [0, 1, 10, 40])
def test_ruiz_lanes(gpu_ctx, oracle, shape, passes):
    m = generators.random_lp(shape[0], *shape, family="precision")
    exp = oracle.equilibrate(m, passes)
    v, rv, order, row_scale, col_scale, it = scaled(gpu_ctx, m, passes)
    assert it == exp["iterations"]
    assert np.array_equal(v, exp["value"])
    assert np.array_equal(rv, exp["value"][order])
    assert np.array_equal(row_scale, exp["row_scale"])
    assert np.array_equal(col_scale, exp["col_scale"])


def test_ruiz_of_a_batch_is_per_lp(gpu_ctx, oracle):
    """LPs that converge after different numbers of passes, one of them at
    once (every entry 1), next to one that never does."""
    ones = generators.transport(3, 12, 17)
    models = [generators.random_lp(s, 20 * s, 60 * s, 2 + s, family="precision") for s in (1, 2, 5, 9)] + [ones]
    o = PdlpOptions(max_iterations=40, ruiz_iterations=25)
    for m, r in zip(models, gpu_ctx.solve_batch(models, o)):
        assert r.extra["ruiz_iterations_executed"] == oracle.equilibrate(m, 25)["iterations"]
        solo = gpu_ctx.solve(m, o)
        assert np.allclose(r.primal, solo.primal, rtol=1e-11, atol=1e-12 * np.abs(solo.primal).max())


@pytest.mark.parametrize("passes", [63, 64, 65, 128, 129, 200])
def test_passes_without_convergence_take_several_launches(gpu_ctx, passes):
    """A tolerance that is never met: every pass runs, at most 64 to a launch.
    Plain numpy does the same operations, each rounded correctly: same bits."""
    import torch
    m = generators.random_lp(7, 300, 900, 5, family="precision")
    col, row = np.repeat(np.arange(m.num_cols), np.diff(m.col_start)), m.row_index
    v, rscale, cscale = m.value.copy(), np.ones(m.num_rows), np.ones(m.num_cols)
    for _ in range(passes):
        delta = []
        for index, count, scale in ((row, m.num_rows, rscale), (col, m.num_cols, cscale)):
            top = np.zeros(count)
            np.maximum.at(top, index, np.abs(v))
            top[top == 0] = 1.0
            delta.append(1.0 / np.sqrt(top))
            scale *= delta[-1]
        v *= delta[0][row] * delta[1][col]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    cs, ri, val, rhs, obj = dev(m.col_start), dev(row), dev(m.value), dev(np.ones(m.num_rows)), dev(m.objective)
    r, c = (torch.zeros(2, k, dtype=torch.float64, device="cuda") for k in (m.num_rows, m.num_cols))
    it, conv = C.c_int64(-1), C.c_int32(-1)
    _lib.check(_lib.engine().mc_ruiz_equilibrate_canonical(
        gpu_ctx.handle, m.num_rows, m.num_cols, m.nnz, cs.data_ptr(), ri.data_ptr(), val.data_ptr(), rhs.data_ptr(),
        obj.data_ptr(), passes, 0.0, 1e-300, 1e300, r[0].data_ptr(), c[0].data_ptr(), r[1].data_ptr(), c[1].data_ptr(),
        C.addressof(it), C.addressof(conv)))
    assert it.value == passes and conv.value == 0
    np.testing.assert_array_equal(val.cpu().numpy(), v)
    np.testing.assert_array_equal(r[0].cpu().numpy(), rscale)
    np.testing.assert_array_equal(c[0].cpu().numpy(), cscale)


def test_converged_equilibration_ignores_a_large_limit(gpu_ctx, oracle):
    m = generators.random_lp(8, 300, 900, 5, family="precision")
    v, _, _, row_scale, col_scale, it = scaled(gpu_ctx, m, 2**62)
    exp = oracle.equilibrate(m, 1000)
    assert it == exp["iterations"] < 64
    assert np.array_equal(v, exp["value"]) and np.array_equal(row_scale, exp["row_scale"])
    assert np.array_equal(col_scale, exp["col_scale"])


def test_solve_with_more_passes_than_a_launch_runs(gpu_ctx):
    """launches counted: passes that converge in the first launch need one"""
    m = generators.random_lp(9, 300, 900, 5)
    a, b = (gpu_ctx.solve(m, PdlpOptions(max_iterations=40, ruiz_iterations=k)) for k in (60, 600))
    assert a.extra["ruiz_iterations_executed"] == b.extra["ruiz_iterations_executed"]
    assert a.extra["launches_by_kind"]["setup"] == b.extra["launches_by_kind"]["setup"]
    np.testing.assert_array_equal(a.primal, b.primal)

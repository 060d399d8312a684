"""Malformed members of a batch whose matrix has no entries to look at: column
pointers that run past the matrix, entries without columns or without rows.
Nothing may follow them; the call is refused and the context stays usable."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import mcpdlp
from mcpdlp import PdlpOptions, _abi, _lib, generators

pytestmark = pytest.mark.gpu


class Given(mcpdlp.Model):
    """A model whose struct says what `info` says."""

    def to_struct(self):
        s = super().to_struct()
        for k, v in self.info["struct"].items():
            setattr(s, k, v)
        return s


def member(rows, cols, col_start, nnz, memory="host"):
    m = Given(rows, cols, np.array(col_start), np.zeros(max(nnz, 1)), np.ones(max(nnz, 1)), np.ones(cols), np.zeros(cols),
              np.ones(cols), np.zeros(rows), np.ones(rows))
    given = {"nnz": nnz}
    if memory == "device":
        import torch
        keep = {}
        for name in ("col_start", "row_index", "value", "objective", "var_lower", "var_upper", "row_lower", "row_upper"):
            keep[name] = torch.from_numpy(getattr(m, name)).cuda()
            given[name] = keep[name].data_ptr()
        given["memory"] = 1
        m.info["keep"] = keep
    m.info["struct"] = given
    return m


# rows, columns, column pointers, entries
BAD = {
    "pointer_past_the_end": (3, 2, [0, 1000000, 0], 0),
    "negative_pointer": (3, 2, [0, -5, 0], 0),
    "no_rows_pointer_past_the_end": (0, 2, [0, 1000000, 0], 0),
    "first_pointer": (3, 2, [4, 4, 4], 0),
    "last_pointer": (3, 2, [0, 0, 7], 0),
    "entries_without_columns": (3, 0, [0], 4),
    "entries_without_rows": (0, 2, [0, 1, 2], 2),
}


@pytest.mark.parametrize("memory", ["host", "device"])
@pytest.mark.parametrize("name", sorted(BAD))
def test_member_without_entries_is_validated(gpu_ctx, name, memory):
    good = [generators.random_lp(90 + i, 50 + i, 150, 4) for i in range(2)]
    o = PdlpOptions(max_iterations=40)
    expect = gpu_ctx.solve_batch(good, o)
    for at in range(3):
        models = good[:at] + [member(*BAD[name], memory=memory)] + good[at:]
        with pytest.raises(ValueError, match="invalid CSC matrix in the batch|CSC terminal pointer mismatch"):
            gpu_ctx.solve_batch(models, o)
    for r, e in zip(gpu_ctx.solve_batch(good, o), expect):
        np.testing.assert_array_equal(r.primal, e.primal)


@pytest.mark.parametrize("memory", ["host", "device"])
def test_members_without_entries_solve(gpu_ctx, memory):
    """Columns without entries, and an LP without rows: accepted as before."""
    models = [member(3, 2, [0, 0, 0], 0, memory), generators.random_lp(97, 50, 150, 4), member(0, 2, [0, 0, 0], 0, memory)]
    lps = (_abi.McLp * 3)(*[m.to_struct() for m in models])
    out, o = (_abi.McPdlpResult * 3)(), PdlpOptions(max_iterations=40).to_struct()
    _lib.check(_lib.engine().mc_pdlp_ctx_solve_batch(gpu_ctx.handle, C.addressof(lps), 3, C.addressof(o), None, None,
                                                     C.addressof(out)))
    assert out[0].iterations > 0 and out[1].iterations == 40
    assert out[2].message == b"trivial"

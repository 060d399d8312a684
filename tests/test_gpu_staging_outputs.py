"""Results of batches and variants in any memory that the driver can write: the
caller's arrays may be pageable, pinned or on the device whatever memory the LP
is in, some may be missing, and pieces around the buffers' size go another way."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from mcpdlp import PdlpOptions, _abi, _lib, generators

pytestmark = pytest.mark.gpu


def outputs(sizes, kinds):
    """An array (or None) per size of the kind whose turn it is, its pointers, and a reader."""
    import torch
    arrays = []
    for q, size in enumerate(sizes):
        kind = kinds[q % len(kinds)]
        if kind is None:
            arrays.append(None)
        elif kind == "pageable":
            arrays.append(torch.full((size,), np.nan, dtype=torch.float64))
        elif kind == "pinned":
            arrays.append(torch.full((size,), np.nan, dtype=torch.float64).pin_memory())
        else:
            arrays.append(torch.full((size,), np.nan, dtype=torch.float64, device="cuda"))
    torch.cuda.synchronize()
    return arrays, (C.c_void_p * len(sizes))(*[None if a is None else a.data_ptr() for a in arrays])


KINDS = [["device"], ["pinned"], ["pageable", "device", "pinned"], [None, "pageable", "pageable", None, None, "device"]]


def check(arrays, expect):
    for a, e in zip(arrays, expect):
        if a is not None:
            np.testing.assert_array_equal(a.cpu().numpy(), e)


def opts():
    o = PdlpOptions(max_iterations=40, lanes_per_column=1, lanes_per_row=2)
    o.set_tolerance(1e-14)
    return o


@pytest.mark.parametrize("kinds", KINDS, ids=str)
def test_batch_outputs(gpu_ctx, kinds):
    # 65536 columns are a buffer of 512 KiB exactly, 131072 the largest that goes through both
    sizes = [(20, 70), (3000, 65536), (3000, 65537), (3000, 131072), (3000, 131073), (40, 150), (5000, 20000), (5000, 30000)] + [(30 + i, 90 + i) for i in range(25)]
    models = [generators.random_lp(i, m, n, 3) for i, (m, n) in enumerate(sizes)]
    expect = gpu_ctx.solve_batch(models, opts())
    lps = (_abi.McLp * len(models))(*[m.to_struct() for m in models])
    x, xp = outputs([n for _, n in sizes], kinds)
    y, yp = outputs([m for m, _ in sizes], kinds[::-1])
    o, res = opts().to_struct(), (_abi.McPdlpResult * len(models))()
    _lib.check(_lib.engine().mc_pdlp_ctx_solve_batch(gpu_ctx.handle, C.addressof(lps), len(models), C.addressof(o),
                                                     C.addressof(xp), C.addressof(yp), C.addressof(res)))
    check(x, [r.primal for r in expect])
    check(y, [r.dual for r in expect])


@pytest.mark.parametrize("n", [300, 65536, 65537, 131072, 131073])
@pytest.mark.parametrize("kinds", KINDS, ids=str)
def test_variant_outputs(gpu_ctx, kinds, n):
    base, count = generators.random_lp(3, 100, n, 3), 40 if n == 300 else 7
    lo = [base.var_lower + 0.01 * (q % 3) for q in range(count)]
    expect = gpu_ctx.solve_variants(base, lo, [None] * count, opts())
    lp, o, res = base.to_struct(), opts().to_struct(), (_abi.McPdlpResult * count)()
    x, xp = outputs([n] * count, kinds)
    y, yp = outputs([100] * count, kinds[::-1])
    los = (C.c_void_p * count)(*[a.ctypes.data for a in lo])
    _lib.check(_lib.engine().mc_pdlp_ctx_solve_variants(gpu_ctx.handle, C.addressof(lp), count, C.addressof(los), None,
                                                        C.addressof(o), None, None, C.addressof(xp), C.addressof(yp),
                                                        C.addressof(res)))
    check(x, [r.primal for r in expect])
    check(y, [r.dual for r in expect])

"""The tiled kernels of the learned warm start at the edges of their tiles
(32- and 64-row tiles, the last partial tile, windows of 32 block partials and
of 4 entries of a line), against the FP64 oracle.  Tolerance: FP32 sums of up
to 10^4 terms through three rounds, as in the small cases."""
from __future__ import annotations

import numpy as np
import pytest

import gnn_oracle as G
from mcpdlp import generators
from mcpdlp.learn import Target, WarmStartNet

pytestmark = pytest.mark.gpu


# rows and columns around the tiles; 9473 columns are the first in 64-row tiles
# (148 of them and one row); 1024, 1025 and 9473 columns give 16, 17 and 149 block partials
@pytest.mark.parametrize("m,n,k", [(3, 7, 2), (31, 32, 3), (33, 63, 4), (64, 65, 5), (129, 1024, 4), (500, 1025, 6),
                                   (97, 9472, 3), (100, 9473, 2)])
def test_loss_and_gradient_at_tile_edges(m, n, k):
    lp = generators.random_lp(m + n, m, n, k)
    r = np.random.default_rng(n)
    t = Target(lp, r.uniform(0, 2, n), r.normal(0, 0.5, m), 0.4)
    net = WarmStartNet(0, 3, 5)
    loss, grad = net.loss_and_grad(t)
    again, grad2 = net.loss_and_grad(t)
    assert loss == again and np.array_equal(grad, grad2)
    loss_c, grad_c, _ = G.loss_and_grad(net.params.astype(np.float64), lp, t.x, t.y, t.log_omega)
    assert abs(loss - loss_c) <= 1e-4 * abs(loss_c) + 1e-7
    assert np.linalg.norm(grad - grad_c) <= 1e-4 * np.linalg.norm(grad_c)
    net.close()

"""The training kernels at row counts around their tiles (64 rows a tile, 32 a column block, parts of at
least 128 rows), against the float64 oracle.

Tolerance: sums of f32 products in any order are off by at most k * 2^-24 of the sum of their
magnitudes, k <= 2048 terms; with gradients of mixed sign that is 2^-24 * sqrt(2048) of the
root-mean-square scale for random rounding.  relative 1e-3, absolute 1e-5 of the largest
gradient, as for the oracle comparison of the whole batch, is 10 times that."""
from __future__ import annotations

import numpy as np
import pytest

from edge_matching_puzzle_b200 import native
from oracle import mlp_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 31, 33, 63, 65, 127, 129, 1025, 2049])
def test_loss_gradient_at_tile_edges(rows):
    m = native.Mlp(seed=6)
    rng = np.random.default_rng(rows)
    x = (rng.random((rows, 512)) < 0.05).astype(np.float32)
    y = (rng.random(rows) < 0.3).astype(np.float32)
    w = rng.uniform(0.5, 2.0, rows).astype(np.float32)
    loss, g = m.loss_grad(x, y, w)
    want_loss, want_g = mlp_oracle.loss_grad(m.params(), x, y, w)
    assert abs(loss - want_loss) <= 1e-5 * (1 + abs(want_loss))
    np.testing.assert_allclose(g, want_g, rtol=1e-3, atol=1e-5 * np.max(np.abs(want_g)))

"""The surrogate's output-layer gradients (chains over the rows in tiles of 128
rows and 16 columns) and its output value with and without staged rows (256
units), at row counts around a tile's, against the numpy oracle in FP64.

Bound: sums of up to 2 n products of values behind three layers of `hidden`
products, as in the tile tests: (2 n + 3 hidden) 2^-24 of the largest entry.
The output bias's gradient is zero but for the rounding of 2 n additions."""

import numpy as np
import pytest

from oracle import mlp as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inputs,hidden,pairs", [
    (3, 32, 1), (7, 64, 63), (5, 96, 64), (14, 224, 65), (14, 256, 192), (9, 288, 130),
    (5, 320, 70), (14, 384, 260), (40, 1024, 33),
])
def test_gradient_chains(rng, inputs, hidden, pairs):
    from aspartik_gb300.surrogate import Surrogate

    s = Surrogate(inputs, hidden, seed=4)
    p = s.get_params().astype(np.float64)
    xn = rng.normal(size=(pairs, inputs)).astype(np.float32)
    xo = rng.normal(size=(pairs, inputs)).astype(np.float32)
    d = rng.normal(size=pairs).astype(np.float32)
    loss, g = s.loss_grad(xn, xo, d)
    want_loss, want = M.loss_grad(p, xn.astype(np.float64), xo.astype(np.float64),
                                  d.astype(np.float64), inputs, hidden)
    tol = (2 * pairs + 3 * hidden) * 2.0 ** -24
    assert loss == pytest.approx(want_loss, rel=tol)
    assert np.abs(g - want).max() <= tol * np.abs(want).max()

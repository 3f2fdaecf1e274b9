"""The training step's tiled kernels at the edges of their tiles and splits,
against the numpy oracle in FP64: rows below, at and above a 32-row tile and
a gradient split, input counts that are and are not whole float4 vectors, and
hidden widths below a 64-column tile.

Bound: a gradient entry is a sum of up to 2 n products of FP32 values that
passed three layers of at most 256 products each; relative to the largest
gradient entry its rounding error stays below (2 n + 3 * 256) 2^-24, the
accumulated bound of the sums involved."""

import numpy as np
import pytest

from oracle import mlp as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inputs,hidden,pairs", [
    (1, 32, 1), (14, 32, 8), (16, 64, 9), (13, 96, 16), (32, 128, 63), (14, 256, 64),
    (14, 256, 65), (31, 160, 512), (8, 64, 1030),
])
def test_loss_and_gradient(rng, inputs, hidden, pairs):
    from aspartik_gb300.surrogate import Surrogate

    s = Surrogate(inputs, hidden, seed=9)
    p = s.get_params().astype(np.float64)
    for _ in range(2):  # the second pass finds the workspaces of the first
        xn = rng.normal(size=(pairs, inputs)).astype(np.float32)
        xo = rng.normal(size=(pairs, inputs)).astype(np.float32)
        d = rng.normal(size=pairs).astype(np.float32)
        loss, g = s.loss_grad(xn, xo, d)
        want_loss, want = M.loss_grad(p, xn.astype(np.float64), xo.astype(np.float64),
                                      d.astype(np.float64), inputs, hidden)
        tol = (2 * pairs + 3 * 256) * 2.0 ** -24
        assert loss == pytest.approx(want_loss, rel=tol)
        assert np.abs(g - want).max() <= tol * np.abs(want).max()
        np.testing.assert_allclose(s.forward(xn), M.forward(p, xn, inputs, hidden), rtol=2e-4,
                                   atol=2e-5)

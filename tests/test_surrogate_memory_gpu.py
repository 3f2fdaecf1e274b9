"""The surrogate's workspaces: the partial tiles of split weight gradients (68 MB
for 1,024 units and 16 parts) are there only for gradients whose rows are split,
and what a net computes does not depend on what its workspaces were made for
first."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_small_passes_take_little_memory(rng):
    torch = pytest.importorskip("torch")
    from aspartik_gb300.surrogate import Surrogate

    torch.cuda.init()
    x = rng.normal(size=(32, 14)).astype(np.float32)
    d = rng.normal(size=32).astype(np.float32)
    Surrogate(14, 1024, seed=1).loss_grad(x, -x, d)  # the kernels are loaded
    s = Surrogate(14, 1024, seed=1)
    before = torch.cuda.mem_get_info()[0]
    s.forward(x)
    s.loss_grad(x, -x, d)
    # 64 rows x 9 buffers of 1,024 floats and the rest: below 4 MB
    assert before - torch.cuda.mem_get_info()[0] <= 16 << 20


@pytest.mark.parametrize("hidden,pairs", [(64, 64), (64, 65), (256, 600), (1024, 1100)])
def test_any_order_of_sizes(rng, hidden, pairs):
    """Rows around and above a split (128), after a forward pass of more rows,
    a smaller gradient and a larger one: the same bits as a fresh net's."""
    from aspartik_gb300.surrogate import Surrogate

    x = rng.normal(size=(3000, 14)).astype(np.float32)
    d = rng.normal(size=3000).astype(np.float32)

    def grad(s, n):
        return s.loss_grad(x[:n], -x[:n], d[:n])

    loss, want = grad(Surrogate(14, hidden, seed=3), pairs)
    s = Surrogate(14, hidden, seed=3)
    first = s.forward(x)
    for n in (5, pairs, 1400, pairs, 64):
        got = grad(s, n)
        if n == pairs:
            assert got[0] == loss and np.array_equal(got[1], want)
    assert np.array_equal(s.forward(x), first)

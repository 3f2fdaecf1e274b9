"""Which walk a 20-state FP32 list takes (three launches: tcgen05, two: register
walk): long lists of many independent entries over few columns, and few entries
over very many, are tcgen05's; ladders, paths and what a switch has decided are
not.  Both walks' values agree to the form's bar (1e-6)."""

import numpy as np
import pytest

from aspartik_gb300 import sim
from aspartik_gb300.schedule import Topology
from tests.test_phase_words_gpu import ladder

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taxa,sites,K,shape,tree,path", [
    (1200, 40, 1, "yule", 3, 2), (1200, 2000, 2, "yule", 3, 2), (700, 40, 1, "yule", 2, 2),
    (1200, 40, 3, "yule", 2, 2), (1200, 40, 1, "ladder", 2, 2), (3, 300000, 1, "yule", 3, 3),
    (3, 40000, 4, "yule", 2, 2), (10, 300000, 1, "yule", 3, 2), (12, 300000, 1, "yule", 2, 2),
])
def test_launches_and_values(taxa, sites, K, shape, tree, path, monkeypatch):
    from aspartik_gb300.calculator import Calculator

    rng = np.random.default_rng(taxa + K)
    if shape == "yule":
        t = sim.yule_tree(taxa, rng, root_height=1.0)
        top = Topology(t.parents, t.heights)
    else:
        top = Topology(*ladder(taxa, taxa - 2))
    leaves = np.repeat(rng.integers(0, 20, size=(1, sites), dtype=np.uint8), taxa, axis=0)
    other = rng.random(leaves.shape, dtype=np.float32) < 0.2
    leaves[other] = rng.integers(0, 20, size=other.sum(), dtype=np.uint8)
    pi = np.maximum(rng.dirichlet([1.0] * 20), 1e-4)
    rates = rng.lognormal(0.0, 1.0, size=190)
    values = []
    # the deepest tip's path (of the ladder: the shortest)
    lists = (top.full(), max((top.path(v) for v in range(min(taxa, 40))), key=lambda q: len(q[0]))
             if shape == "yule" else top.path(taxa - 1))
    for switch in (None, "0", "1"):
        if switch:
            monkeypatch.setenv("B3G_TC20", switch)
        g = Calculator.GB300(0, "f32").make20(leaves, sites, num_categories=K)
        g.set_weights(np.ones(sites, np.uint32))
        g.set_reversible(rates, pi / pi.sum())
        if K > 1:
            g.set_gamma(1.0)
        for one, launches in zip(lists, (tree, path)):
            g.propose_lengths(*one)
            values.append(g.log_likelihood())
            assert g.last_launches() == (launches if not switch else 3 if switch == "1" else 2)
            g.accept()
        g.close()
    assert np.isfinite(values).all()
    for k in (0, 1):
        for other in (values[2 + k], values[4 + k]):
            assert abs(values[k] - other) <= 1e-6 * abs(other)

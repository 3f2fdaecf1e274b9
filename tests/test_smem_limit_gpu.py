"""Whole trees whose depth-first FP32 walk takes exactly the default 48 KB of dynamic
shared memory, and a row of tips less and more: pure ladders of single tips (one
group, one slot) of 1 category.  64 patterns a block: 512 + 3,072 + 1,280 bytes
and 64 a tip row, so 691 taxa; 128 patterns: 1,024 + 3,072 + 2,560 and 128, 331."""

import numpy as np
import pytest

from aspartik_gb300.schedule import Topology
from oracle import oracle as O
from tests.test_phase_words_gpu import ladder

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,taxa", [(64, 690), (64, 691), (64, 692), (128, 330), (128, 331),
                                       (128, 332)])
def test_exactly_the_default_limit(tile, taxa, monkeypatch):
    from aspartik_gb300.calculator import Calculator

    monkeypatch.setenv("B3G_TREE", "2")
    monkeypatch.setenv("B3G_TREE_TILE", str(tile))
    rng = np.random.default_rng(taxa)
    parents, heights = ladder(taxa, taxa - 2)
    leaves = np.repeat(rng.choice(np.array([1, 2, 4, 8], np.uint8), size=(1, 70)), taxa, axis=0)
    other = rng.random(leaves.shape) < 0.1
    leaves[other] = rng.choice(np.array([1, 2, 4, 8], np.uint8), size=other.sum())
    rates, pi = rng.gamma(2.0, 1.0, size=6), rng.dirichlet([5.0] * 4)
    g = Calculator.GB300(0, "f32").make4(leaves, 70)
    g.set_weights(np.ones(70, np.uint32))
    g.set_reversible(rates, pi)
    g.propose_lengths(*Topology(parents, heights).full())
    got = g.log_likelihood()
    g.close()
    want = O.DnaLikelihood(leaves, np.ones(70, np.uint32), O.DatedTree(parents, heights),
                           O.gtr(rates, pi)).cache
    assert abs(got - want) <= 1e-6 * abs(want)

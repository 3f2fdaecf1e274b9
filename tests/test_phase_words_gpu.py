"""Ladders of single tips above a balanced subtree: their phases outnumber what
a block's shared memory holds for the groups that the list would get (16 in the
four-state FP64 form with one category, four in the 20-state FP32 form), so
they are walked by fewer.  Bars of the forms: 1e-10 (FP64), 1e-6 (FP32)."""

import numpy as np
import pytest

from aspartik_gb300.schedule import Topology
from oracle import generic as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ROOT = 0xFFFFFFFF


def ladder(taxa, tips):
    """Parents and heights: `tips` single tips above a balanced subtree."""
    n = 2 * taxa - 1
    parents, heights = np.full(n, ROOT, np.uint32), np.zeros(n)
    level, new, t = list(range(taxa - tips)), taxa, 0.0
    while len(level) > 1:
        t += 0.02
        up = []
        for a, b in zip(level[::2], level[1::2]):
            parents[a] = parents[b] = new
            heights[new] = t
            up.append(new)
            new += 1
        level = up + (level[-1:] if len(level) % 2 else [])
    top = level[0]
    for k in range(taxa - tips, taxa):
        t += 0.004
        parents[top] = parents[k] = new
        heights[new] = t
        top = new
        new += 1
    return parents, heights


@pytest.mark.parametrize("S,form,K,taxa,tips", [
    (4, "f64", 1, 4200, 190), (4, "f64", 1, 4200, 214), (4, "f64", 1, 1700, 250),
    (20, "f32", 4, 2400, 500), (20, "f32", 4, 2400, 560),
])
def test_ladder(S, form, K, taxa, tips):
    from aspartik_gb300.calculator import Calculator

    rng = np.random.default_rng(taxa + tips)
    parents, heights = ladder(taxa, tips)
    codes = np.repeat(rng.integers(0, S, size=(1, 40)), taxa, axis=0)
    other = rng.random(codes.shape) < 0.1
    codes[other] = rng.integers(0, S, size=other.sum())
    pi = np.maximum(rng.dirichlet([5.0] * S), 1e-3)
    pi /= pi.sum()
    rates = rng.gamma(2.0, 1.0, size=S * (S - 1) // 2)
    model = O.gtr(rates, pi) if S == 4 else O.reversible(rates, pi)
    internals, children, lengths = Topology(parents, heights).full()
    lengths = np.asarray(lengths).reshape(-1, 2)
    cats = O.gamma_categories(0.7, K) if K > 1 else np.ones(1)
    per = np.array([G.prune(codes, internals, np.asarray(children).reshape(-1, 2),
                            np.array([[model.transition(d * r) for d in pair]
                                      for pair in lengths]), model.pi) for r in cats])
    want = float((np.logaddexp.reduce(per, axis=0) - np.log(K)).sum())
    make = Calculator.GB300(0, form)
    g = (make.make4(np.array([1, 2, 4, 8], np.uint8)[codes], 40, num_categories=K) if S == 4
         else make.make20(codes.astype(np.uint8), 40, num_categories=K))
    g.set_weights(np.ones(40, np.uint32))
    g.set_reversible(rates, pi)
    if K > 1:
        g.set_gamma(0.7)
    for _ in range(2):
        g.propose_lengths(internals, children, lengths, 1.0)
        assert abs(g.log_likelihood() - want) <= {"f64": 1e-10, "f32": 1e-6}[form] * abs(want)
        g.accept()
    g.close()

"""Batches under B3G_DIRECT=0: the list of every member is laid out for the
kernel that walks it, whatever its length (below, at and above the 48 entries
of the short-list kernel) and category count (that kernel takes 1, 2 and 4).
Sums against calculators of their own, to 1e-12 (the same terms in another
order), through paths and whole trees in turn."""

import numpy as np
import pytest

from oracle import oracle as O
from tests.cases import dna_case
from tests.test_gpu_parity import lists_and_lengths, make_gpu
from tests.test_oracle import random_move

pytestmark = pytest.mark.gpu

SHAPES = [(30, 300, 4), (49, 400, 1), (50, 500, 2), (20, 200, 3), (120, 700, 4), (90, 150, 1),
          (2, 20, 4)]


@pytest.mark.parametrize("tree_walk", ["0", "1", "2"])
def test_lists_of_every_length(tree_walk, monkeypatch):
    from aspartik_gb300.calculator import Batch

    monkeypatch.setenv("B3G_TREE", tree_walk)
    alone, members, trees = [], [], []
    for taxa, sites, K in SHAPES:
        c = dna_case(taxa, sites, seed=taxa, model="gtr", root_height=1.0, alpha=0.6,
                     num_categories=K)
        for out, direct in ((alone, "1"), (members, "0")):
            monkeypatch.setenv("B3G_DIRECT", direct)
            g = make_gpu(c.leaves, c.weights, K, "f32")
            g.set_reversible(c.rates, c.pi)
            if K > 1:
                g.set_gamma(0.6)
            out.append(g)
        tree = O.DatedTree(c.tree.parents, c.tree.heights)
        tree.mark_all_edges_updated()
        trees.append(tree)
    batch = Batch(members)
    rng = np.random.default_rng(5)
    for step in range(6):
        want = []
        for g, m, t in zip(alone, members, trees):
            lists = lists_and_lengths(t)
            g.propose_lengths(*lists, 1.0)
            want.append(g.log_likelihood())
            m.stage_lengths(*lists, 1.0)
        batch.run()
        np.testing.assert_allclose(batch.log_likelihoods(), want, rtol=1e-12)
        for g, m, t in zip(alone, members, trees):
            for one in (g, m, t):
                one.accept()
            if step % 3 == 2:
                t.mark_all_edges_updated()
            else:
                random_move(t, rng)
    batch.close()
    for g in members + alone:
        g.close()

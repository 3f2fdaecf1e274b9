"""A batch member's log-likelihood does not depend on what the other members
staged in that step: the same bits alone and in company, in every kernel of a
batch (run walk, depth-first walk, short lists)."""

import numpy as np
import pytest

from oracle import oracle as O
from tests.cases import dna_case
from tests.test_gpu_parity import lists_and_lengths, make_gpu
from tests.test_oracle import random_move

pytestmark = pytest.mark.gpu

SHAPES = [(200, 900, 4, 128), (90, 1500, 1, 64), (120, 700, 3, 32), (60, 5000, 4, 64),
          (150, 400, 8, 16)]


@pytest.mark.parametrize("tree_walk", ["0", "1"])
def test_same_bits_in_any_company(tree_walk, monkeypatch):
    from aspartik_gb300.calculator import Batch

    members, lists = [], []
    monkeypatch.setenv("B3G_TREE", tree_walk)
    for taxa, sites, K, tile in SHAPES:
        if tree_walk == "0":
            monkeypatch.setenv("B3G_RUNS_TILE", str(tile))
        c = dna_case(taxa, sites, seed=taxa, model="gtr", root_height=1.0, alpha=0.6,
                     num_categories=K)
        g = make_gpu(c.leaves, c.weights, K, "f32")
        g.set_reversible(c.rates, c.pi)
        if K > 1:
            g.set_gamma(0.6)
        tree = O.DatedTree(c.tree.parents, c.tree.heights)
        tree.mark_all_edges_updated()
        full = lists_and_lengths(tree)
        tree.accept()
        random_move(tree, np.random.default_rng(taxa))
        members.append(g)
        lists.append((full, lists_and_lengths(tree)))
    batch = Batch(members)
    M = len(members)

    def step(kinds):  # 0: whole tree, 1: a path, None: nothing staged
        for g, both, kind in zip(members, lists, kinds):
            if kind is not None:
                g.stage_lengths(*both[kind], 1.0)
        batch.run()
        out = batch.log_likelihoods()
        for g, kind in zip(members, kinds):
            if kind is not None:
                g.reject()
        return out

    for g in members:  # state for the paths
        g.stage_lengths(*lists[members.index(g)][0], 1.0)
    batch.run()
    batch.log_likelihoods()
    for g in members:
        g.accept()
    for kind in (0, 1):
        alone = [step([kind if k == m else None for k in range(M)])[m] for m in range(M)]
        assert np.isfinite(alone).all()
        together = step([kind] * M)
        mixed = step([kind if k % 2 == 0 else 1 - kind for k in range(M)])
        for m in range(M):
            assert together[m] == alone[m], (kind, m)
            if m % 2 == 0:
                assert mixed[m] == alone[m], (kind, m)
    batch.close()

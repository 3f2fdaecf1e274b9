"""Batches of one tiny alignment each, around the default limit of 48 KB of shared
memory that the batched run walk passes with its static part: every size is
taken, and gives the value of a calculator of its own."""

import pytest

from oracle import oracle as O
from tests.cases import dna_case
from tests.test_gpu_parity import lists_and_lengths, make_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taxa", [2, 3, 5, 7, 9, 12, 16, 20])
@pytest.mark.parametrize("K", [1, 3, 4])
def test_tiny_members(taxa, K):
    from aspartik_gb300.calculator import Batch

    c = dna_case(taxa, 28, seed=taxa, model="gtr", root_height=1.0, alpha=0.6, num_categories=K)
    tree = O.DatedTree(c.tree.parents, c.tree.heights)
    tree.mark_all_edges_updated()
    lists = lists_and_lengths(tree)
    g, m = (make_gpu(c.leaves, c.weights, K, "f32") for _ in range(2))
    for one in (g, m):
        one.set_reversible(c.rates, c.pi)
        if K > 1:
            one.set_gamma(0.6)
    g.propose_lengths(*lists, 1.0)
    batch = Batch([m])
    m.stage_lengths(*lists, 1.0)
    batch.run()
    assert batch.log_likelihoods()[0] == pytest.approx(g.log_likelihood(), rel=1e-12)
    batch.close()
    g.close()
    m.close()

"""B3G_TC20=0 keeps the tcgen05 walk off through the autotuner, which has then
nothing to try: 0 (register walk), two launches an evaluation, and the value of
an untuned calculator."""

import pytest

from oracle import oracle as O
from tests.cases import protein_case
from tests.test_gpu_parity import lists_and_lengths

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taxa,sites,K", [(2, 40, 1), (20, 3000, 8), (64, 900, 4)])
def test_autotune_leaves_the_register_walk(taxa, sites, K, monkeypatch):
    from aspartik_gb300.calculator import Calculator

    monkeypatch.setenv("B3G_TC20", "0")
    c = protein_case(taxa, sites, seed=taxa, num_categories=K)
    g = Calculator.GB300(0, "f32").make20(c.leaves, c.leaves.shape[1], num_categories=K)
    g.set_weights(c.weights)
    g.set_reversible(c.rates, c.pi)
    if K > 1:
        g.set_gamma(1.0)
    tree = O.DatedTree(c.tree.parents, c.tree.heights)
    tree.mark_all_edges_updated()
    full = lists_and_lengths(tree)
    g.propose_lengths(*full, 1.0)
    before = g.log_likelihood()
    g.accept()
    assert g.autotune(*full, 1.0) == 0
    assert g.timing_totals()[2] == 0  # nothing to try, so no trial was timed
    g.propose_lengths(*full, 1.0)
    assert g.log_likelihood() == before and g.last_launches() == 2
    g.close()

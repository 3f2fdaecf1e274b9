"""20-state FP32 transition tables in one block and in four (lists of up to 76
tables): whole trees around that size against the generic oracle at the FP32
form's bar of the protein tests (1e-6)."""

import numpy as np
import pytest

from oracle import generic as G
from oracle import oracle as O
from tests.cases import protein_case
from tests.test_gpu_parity import lists_and_lengths

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taxa,K", [(2, 1), (10, 4), (11, 4), (39, 1), (40, 1), (6, 8)])
def test_short_and_long_lists(taxa, K):
    from aspartik_gb300.calculator import Calculator

    c = protein_case(taxa, 70, seed=taxa, num_categories=K, gaps=0.05)
    tree = O.DatedTree(c.tree.parents, c.tree.heights)
    tree.mark_all_edges_updated()
    g = Calculator.GB300(0, "f32").make20(c.leaves, c.leaves.shape[1], num_categories=K)
    g.set_weights(c.weights)
    g.set_reversible(c.rates, c.pi)
    if K > 1:
        g.set_gamma(1.0)
    g.propose_lengths(*lists_and_lengths(tree), 1.0)
    got = g.log_likelihood()
    g.close()
    want = G.log_likelihood(c.leaves, c.weights, c.tree.parents, c.tree.heights,
                            O.reversible(c.rates, c.pi),
                            O.gamma_categories(1.0, K) if K > 1 else np.ones(1))
    assert abs(got - want) <= 1e-6 * abs(want)

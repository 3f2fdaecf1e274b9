"""The four-state FP64 walk in its forms: a thread a column walking the whole
list, and 2 to 16 groups a block walking it run by run; integer products
(soft64.cuh) wherever values are positive normal numbers, FP64 instructions
elsewhere.  Every form against the restated GammaLikelihood at 1e-10 (the FP64
bar of the other parity tests), and the forms against each other bit for bit
per pattern (each entry's arithmetic is the same)."""

import numpy as np
import pytest

from oracle import oracle as O
from tests.cases import dna_case
from tests.test_gpu_parity import full, lists_and_lengths, make_gpu
from tests.test_oracle import random_move

pytestmark = pytest.mark.gpu


def sequence(c, K, alpha, groups, monkeypatch, squeeze):
    if groups:
        monkeypatch.setenv("B3G_F64_GROUPS", str(groups))
    else:
        monkeypatch.delenv("B3G_F64_GROUPS", raising=False)
    g = make_gpu(c.leaves, c.weights, K, "f64")
    g.set_reversible(c.rates, c.pi)
    if K > 1:
        g.set_gamma(alpha)
    heights = c.tree.heights.copy()
    if squeeze:  # zero-length internal branches: identity matrices
        L = c.leaves.shape[0]
        for v, kids in enumerate(c.tree.children()[2::3]):
            top = max(kids)
            if top >= L and heights[top] >= heights[min(kids)]:
                heights[L + 2 + 3 * v] = heights[top]
    tree = O.DatedTree(c.tree.parents, heights)
    tree.mark_all_edges_updated()
    rng = np.random.default_rng(11)
    out = []
    for step in range(4):
        g.propose_lengths(*lists_and_lengths(tree), 1.0)
        lnl = g.log_likelihood()
        out.append((lnl, g.site_log_likelihoods()))
        g.accept()
        tree.accept()
        if not squeeze:
            random_move(tree, rng)
        else:
            tree.mark_all_edges_updated()
    g.close()
    return out


@pytest.mark.parametrize("taxa,sites,K,alpha,squeeze", [
    (2, 1, 1, None, False), (5, 33, 1, None, False), (40, 127, 4, 0.5, False),
    (61, 400, 2, 0.7, True), (33, 300, 3, 0.3, False), (24, 129, 16, 0.5, False),
    (150, 500, 1, None, True),
])
def test_forms_agree(taxa, sites, K, alpha, squeeze, monkeypatch):
    c = dna_case(taxa, sites, seed=taxa, model="gtr", root_height=1.5, alpha=alpha,
                 num_categories=K)
    ref = sequence(c, K, alpha, 1, monkeypatch, squeeze)
    for groups in (None, 2, 4, 8, 16):
        got = sequence(c, K, alpha, groups, monkeypatch, squeeze)
        for (l0, s0), (l1, s1) in zip(ref, got):
            assert np.array_equal(s0, s1)
            assert np.isfinite(l0) and abs(l1 - l0) <= 1e-13 * abs(l0)
    if not squeeze:
        want = O.GammaLikelihood(c.leaves, c.weights,
                                 O.DatedTree(c.tree.parents, c.tree.heights),
                                 O.gtr(c.rates, c.pi), K, alpha if K > 1 else 1.0).cache
        assert abs(ref[0][0] - want) <= 1e-10 * abs(want)


@pytest.mark.parametrize("taxa,sites,K", [(2, 1, 1), (7, 65, 4), (40, 200, 8), (90, 130, 2)])
def test_protein_groups_agree(taxa, sites, K, monkeypatch):
    """20 states, FP64: 1, 2 and 4 groups a block give the same bits per
    pattern, and the generic oracle's likelihood to 1e-10."""
    from oracle import generic as G
    from tests.cases import protein_case
    from aspartik_gb300.calculator import Calculator

    c = protein_case(taxa, sites, seed=taxa, num_categories=K, gaps=0.05)
    tree = O.DatedTree(c.tree.parents, c.tree.heights)
    tree.mark_all_edges_updated()
    lists = lists_and_lengths(tree)
    got = []
    for groups in ("", "1", "2", "4"):
        if groups:
            monkeypatch.setenv("B3G_F64_GROUPS", groups)
        else:
            monkeypatch.delenv("B3G_F64_GROUPS", raising=False)
        g = Calculator.GB300(0, "f64").make20(c.leaves, c.leaves.shape[1], num_categories=K)
        g.set_weights(c.weights)
        g.set_reversible(c.rates, c.pi)
        if K > 1:
            g.set_gamma(1.0)
        for _ in range(2):
            g.propose_lengths(*lists, 1.0)
            got.append((g.log_likelihood(), g.site_log_likelihoods()))
            g.accept()
        g.close()
    want = G.log_likelihood(c.leaves, c.weights, c.tree.parents, c.tree.heights,
                            O.reversible(c.rates, c.pi),
                            O.gamma_categories(1.0, K) if K > 1 else np.ones(1))
    for lnl, sites_ in got:
        assert np.array_equal(sites_, got[0][1])
        assert abs(lnl - want) <= 1e-10 * abs(want)


@pytest.mark.parametrize("taxa,sites,K", [(2, 1, 1), (7, 65, 4), (48, 200, 8), (200, 40, 2)])
def test_protein_fp32_groups_agree(taxa, sites, K, monkeypatch):
    """20 states, FP32 register-MMA walk: one to four warps a block (disjoint
    subtrees, then the entries above them) give the same bits per pattern over
    whole trees, a dirty path and a list that repeats, and the generic
    oracle's likelihood to the FP32 bar (1e-6)."""
    from oracle import generic as G
    from tests.cases import protein_case
    from aspartik_gb300.calculator import Calculator

    c = protein_case(taxa, sites, seed=taxa, num_categories=K, gaps=0.05)
    got = []
    for groups in ("", "1", "2", "3", "4"):
        if groups:
            monkeypatch.setenv("B3G_S20_GROUPS", groups)
        else:
            monkeypatch.delenv("B3G_S20_GROUPS", raising=False)
        tree = O.DatedTree(c.tree.parents, c.tree.heights)
        g = Calculator.GB300(0, "f32").make20(c.leaves, c.leaves.shape[1], num_categories=K)
        g.set_weights(c.weights)
        g.set_reversible(c.rates, c.pi)
        if K > 1:
            g.set_gamma(1.0)
        rng = np.random.default_rng(3)
        tree.mark_all_edges_updated()
        mine = []
        for _ in range(3):
            lists = lists_and_lengths(tree)
            for _ in range(2):
                g.propose_lengths(*lists, 1.0)
                mine.append((g.log_likelihood(), g.site_log_likelihoods()))
            g.accept()
            tree.accept()
            random_move(tree, rng)
        g.close()
        got.append(mine)
    want = G.log_likelihood(c.leaves, c.weights, c.tree.parents, c.tree.heights,
                            O.reversible(c.rates, c.pi),
                            O.gamma_categories(1.0, K) if K > 1 else np.ones(1))
    assert abs(got[0][0][0] - want) <= 1e-6 * abs(want)
    for mine in got[1:]:
        for (l0, s0), (l1, s1) in zip(got[0], mine):
            assert np.array_equal(s0, s1)
            assert l0 == l1

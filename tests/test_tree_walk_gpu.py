"""The four-state FP32 depth-first walk in its forms (64 and 128 patterns a
block, 1 to 16 groups, tip codes and slots in shared memory or not, lists with
and without clean children) against the run walk: every entry's arithmetic is
the same, so the site values and category values agree bit for bit, and the
sums, FP64 in another order, to 1e-13 (a few hundred terms' roundings)."""

import numpy as np
import pytest

from oracle import oracle as O
from tests.cases import dna_case
from tests.test_gpu_parity import lists_and_lengths, make_gpu
from tests.test_oracle import random_move

pytestmark = pytest.mark.gpu


def sequence(c, K, alpha, form, monkeypatch):
    for name in ("B3G_TREE", "B3G_TREE_TILE", "B3G_TREE_GROUPS"):
        monkeypatch.delenv(name, raising=False)
    monkeypatch.setenv("B3G_DIRECT", "0")  # short lists too
    monkeypatch.setenv("B3G_TREE", "2" if form else "0")
    if form:
        monkeypatch.setenv("B3G_TREE_TILE", str(form[0]))
        if form[1]:
            monkeypatch.setenv("B3G_TREE_GROUPS", str(form[1]))
    g = make_gpu(c.leaves, c.weights, K, "f32")
    g.set_reversible(c.rates, c.pi)
    if K > 1:
        g.set_gamma(alpha)
    tree = O.DatedTree(c.tree.parents, c.tree.heights.copy())
    tree.mark_all_edges_updated()
    rng = np.random.default_rng(11)
    mats = np.random.default_rng(12)
    out = []
    for step in range(6):  # the whole tree, then paths above random moves
        internals, children, lengths = lists_and_lengths(tree)
        if step % 3 == 2:  # given matrices, and the category values
            m = mats.random((len(internals), 2, K, 4, 4)) + 8 * np.eye(4)
            g.propose(internals, children, m / m.sum(-1, keepdims=True), c.pi)
            out.append((g.log_likelihood(), g.site_log_likelihoods(), g.likelihoods()))
        else:
            g.propose_lengths(internals, children, lengths, 1.0)
            out.append((g.log_likelihood(), g.site_log_likelihoods(), 0))
        if step == 3:  # a rejected proposal leaves the state behind it
            g.reject()
            tree.reject()
        else:
            g.accept()
            tree.accept()
        random_move(tree, rng)
    g.close()
    return out


@pytest.mark.parametrize("taxa,sites,K,alpha", [
    (2, 1, 1, None), (3, 127, 4, 0.5), (9, 129, 2, 0.4), (40, 700, 4, 0.5), (61, 400, 1, None),
    (33, 300, 3, 0.3), (24, 129, 16, 0.5), (150, 500, 8, 0.6), (700, 90, 4, 0.5),
    (1200, 40, 16, 0.5),
])
def test_forms_agree(taxa, sites, K, alpha, monkeypatch):
    c = dna_case(taxa, sites, seed=taxa, model="gtr", root_height=1.5, alpha=alpha,
                 num_categories=K)
    ref = sequence(c, K, alpha, None, monkeypatch)
    for form in ((64, 0), (64, 1), (64, 2), (64, 4), (64, 16), (128, 0), (128, 1), (128, 3),
                 (128, 8)):
        got = sequence(c, K, alpha, form, monkeypatch)
        for (l0, s0, c0), (l1, s1, c1) in zip(ref, got):
            assert np.array_equal(s0, s1)
            assert np.array_equal(c0, c1)
            assert np.isfinite(l0) and abs(l1 - l0) <= 1e-13 * abs(l0)


def test_batched_lists(monkeypatch):
    """Whole trees and paths of members of several sizes in one batch, walked
    depth first there, against calculators of their own on the run walk: sums
    of the same bits per pattern, to 1e-13."""
    from aspartik_gb300.calculator import Batch
    shapes = [(60, 300, 4, 0.5), (53, 129, 1, None), (80, 700, 5, 0.6), (150, 64, 16, 0.5),
              (260, 500, 3, 0.4), (9, 200, 2, 0.5), (700, 40, 4, 0.7)]
    cases = [dna_case(t, s, seed=t, model="gtr", root_height=1.5, alpha=a, num_categories=K)
             for t, s, K, a in shapes]

    def make(batched):
        monkeypatch.setenv("B3G_TREE", "1" if batched else "0")
        out = []
        for c, (_, _, K, a) in zip(cases, shapes):
            g = make_gpu(c.leaves, c.weights, K, "f32")
            g.set_reversible(c.rates, c.pi)
            if K > 1:
                g.set_gamma(a)
            out.append(g)
        return out

    alone, members = make(False), make(True)
    batch = Batch(members)
    trees = [O.DatedTree(c.tree.parents, c.tree.heights.copy()) for c in cases]
    for t in trees:
        t.mark_all_edges_updated()
    rng = np.random.default_rng(3)
    for step in range(4):
        want = []
        for g, m, t in zip(alone, members, trees):
            lists = lists_and_lengths(t)
            g.propose_lengths(*lists, 1.0)
            want.append(g.log_likelihood())
            m.stage_lengths(*lists, 1.0)
        batch.run()
        got = batch.log_likelihoods()
        for lnl, l in zip(want, got):
            assert abs(l - lnl) <= 1e-13 * abs(lnl)
        for g, m, t in zip(alone, members, trees):
            g.accept()
            m.accept()
            t.accept()
            if step == 1:
                t.mark_all_edges_updated()
            else:
                random_move(t, rng)


def test_impossible_patterns(monkeypatch):
    """Patterns of likelihood zero (identity matrices under different bases)
    give -inf."""
    c = dna_case(12, 200, seed=3, model="gtr", root_height=1.5)
    res = []
    for form in (None, (64, 2), (128, 1)):
        monkeypatch.setenv("B3G_TREE", "2" if form else "0")
        if form:
            monkeypatch.setenv("B3G_TREE_TILE", str(form[0]))
            monkeypatch.setenv("B3G_TREE_GROUPS", str(form[1]))
        g = make_gpu(c.leaves, c.weights, 1, "f32")
        tree = O.DatedTree(c.tree.parents, c.tree.heights.copy())
        tree.mark_all_edges_updated()
        internals, children, _ = lists_and_lengths(tree)
        g.propose(internals, children, np.tile(np.eye(4), (len(internals), 2, 1, 1, 1)), c.pi)
        res.append((g.log_likelihood(), g.site_log_likelihoods()))
        g.close()
    assert res[0][0] == -np.inf and np.isinf(res[0][1]).any()
    for lnl, sites in res[1:]:
        assert lnl == -np.inf and np.array_equal(sites, res[0][1])

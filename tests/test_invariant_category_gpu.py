"""A category of rate zero (invariant sites) in the four-state FP32 walks.  A
variable pattern's value is zero there, and its rescale count stays at zero
while the other categories' counts fall with the tree: the difference of the
exponents passes 128, 384, ... (where a float factor 2^e would be an infinity).
Log-likelihoods against the FP64 oracle at the FP32 form's bar (1e-6), every
pattern finite."""

import numpy as np
import pytest

from oracle import generic as G
from oracle import oracle as O
from tests.cases import dna_case
from tests.test_gpu_parity import lists_and_lengths, make_gpu

pytestmark = pytest.mark.gpu

RATES = {2: [0.0, 2.0], 3: [0.0, 0.7, 2.3], 4: [0.0, 0.4, 0.9, 2.7]}


def exponent_gaps(c, internals, children, lengths, model, rates):
    """Zero categories' exponents above the largest of the positive ones, per
    pattern, with every node's largest entry normalised to [1, 2)."""
    codes = np.log2(c.leaves.astype(float)).astype(int)  # unambiguous bases
    L, P = codes.shape
    counts, dots = [], []
    for r in rates:
        part, cnt = {}, {}
        for v, kids, pair in zip(internals, children, lengths):
            y, n = np.ones((P, 4)), np.zeros(P, dtype=np.int64)
            for ch, d in zip(kids, pair):
                m = model.transition(d * r)
                if ch < L:
                    y = y * m[:, codes[ch]].T
                else:
                    y = y * (part[ch] @ m.T)
                    n = n + cnt[ch]
            top = y.max(axis=1)
            e = np.where(top > 0, np.frexp(top)[1] - 1, 0)
            part[int(v)], cnt[int(v)] = y * np.exp2(-e.astype(float))[:, None], n + e
        counts.append(cnt[int(internals[-1])])
        dots.append(part[int(internals[-1])] @ model.pi)
    counts, dots = np.array(counts), np.array(dots)
    top = np.where(dots > 0, counts, np.iinfo(np.int64).min).max(axis=0)
    return (counts - top)[dots == 0]


@pytest.mark.parametrize("taxa,sites,C", [(128, 3000, 4), (256, 4000, 4), (200, 1500, 2),
                                          (256, 3000, 3)])
def test_every_walk(taxa, sites, C, monkeypatch):
    from aspartik_gb300.calculator import Batch

    c = dna_case(taxa, sites, seed=taxa, model="gtr", root_height=1.0, alpha=0.5,
                 num_categories=4)
    model = O.gtr(c.rates, c.pi)
    tree = O.DatedTree(c.tree.parents, c.tree.heights)
    tree.mark_all_edges_updated()
    full = lists_and_lengths(tree)
    tree.accept()
    gaps = exponent_gaps(c, *full, model, RATES[C])
    assert (gaps == 128).any() and (C < 4 or taxa < 256 or (gaps == 384).any())

    def oracle():
        return G.log_likelihood(np.log2(c.leaves.astype(float)).astype(int), c.weights,
                                tree.parents, tree.heights, model, RATES[C])

    want = [oracle()]
    v = int(c.tree.parents[0])  # a path from a node next to the tips
    tree.set_height(v, 0.5 * (max(tree.heights[int(k)] for k in tree.children_of(v)) +
                              tree.heights[int(tree.parent_of(v))]))
    path = lists_and_lengths(tree)
    assert len(path[0]) <= 48  # the short-list kernel's (C of 2 and 4)
    want.append(oracle())
    for name, value in (("", ""), ("B3G_TREE", "0"), ("B3G_TREE", "2"),
                        ("B3G_TREE_TILE", "128"), ("B3G_DIRECT", "0")):
        if name:
            monkeypatch.setenv(name, value)
        g = make_gpu(c.leaves, c.weights, C, "f32")
        if name:
            monkeypatch.delenv(name)
        g.set_reversible(c.rates, c.pi)
        g.set_category_rates(RATES[C])
        for lists, lnl in zip((full, path), want):
            g.propose_lengths(*lists, 1.0)
            assert abs(g.log_likelihood() - lnl) <= 1e-6 * abs(lnl), (name, value)
            assert np.isfinite(g.site_log_likelihoods()).all()
            g.accept()
        if name == "B3G_DIRECT":  # a batch takes the short list by its own rule
            g.close()
            continue
        batch = Batch([g])
        for lists, lnl in zip((full, path), want):
            g.stage_lengths(*lists, 1.0)
            batch.run()
            assert abs(batch.log_likelihoods()[0] - lnl) <= 1e-6 * abs(lnl), (name, value)
            g.accept()
        batch.close()
        g.close()

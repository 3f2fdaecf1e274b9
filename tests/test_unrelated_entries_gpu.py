"""Lists that are not one tree: entries whose parents are not listed, the root
last.  Every walk, form and group count against the oracle's pruning of the
same state: the root's value, and what the other entries left behind (read
through the rest of the path above them).  Bars of the forms: 1e-10 (FP64),
1e-6 (FP32)."""

import numpy as np
import pytest

from oracle import generic as G
from oracle import oracle as O
from tests.cases import dna_case, protein_case
from tests.test_gpu_parity import lists_and_lengths

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-10, "f32": 1e-6}


def make(c, S, K, form):
    from aspartik_gb300.calculator import Calculator

    make = Calculator.GB300(0, form)
    g = (make.make20 if S == 20 else make.make4)(c.leaves, c.leaves.shape[1], num_categories=K)
    g.set_weights(c.weights)
    g.set_reversible(c.rates, c.pi)
    if K > 1:
        g.set_gamma(0.7)
    return g


def problem(S, K, taxa, sites):
    if S == 4:
        c = dna_case(taxa, sites, seed=taxa, model="gtr", root_height=1.0, alpha=0.7,
                     num_categories=4)
        codes, model = np.log2(c.leaves.astype(float)).astype(int), O.gtr(c.rates, c.pi)
    else:
        c = protein_case(taxa, sites, seed=taxa, num_categories=4)
        codes, model = c.leaves, O.reversible(c.rates, c.pi)
    tree = O.DatedTree(c.tree.parents, c.tree.heights)
    tree.mark_all_edges_updated()
    internals, children, lengths = lists_and_lengths(tree)
    cats = O.gamma_categories(0.7, K) if K > 1 else np.ones(1)

    def lnl(lengths):
        mats = [np.array([[model.transition(d * r) for d in pair] for pair in lengths])
                for r in cats]
        per = np.array([G.prune(codes, internals, children, m, model.pi) for m in mats])
        site = np.logaddexp.reduce(per, axis=0) - np.log(len(cats))
        return float(site @ c.weights.astype(float))

    return c, internals, children, lengths, lnl


@pytest.mark.parametrize("S,form,K,taxa,sites,switches", [
    (20, "f64", 4, 24, 70, [("B3G_F64_GROUPS", v) for v in ("1", "2", "4")]),
    (20, "f64", 1, 12, 200, [("B3G_F64_GROUPS", "2")]),
    (20, "f32", 4, 24, 70, [("B3G_S20_GROUPS", "1"), ("B3G_S20_GROUPS", "4"), ("B3G_TC20", "1")]),
    (4, "f64", 4, 24, 300, [("B3G_F64_GROUPS", v) for v in ("1", "2", "4")]),
    (4, "f64", 1, 40, 90, [("B3G_F64_GROUPS", "16")]),
    (4, "f32", 4, 24, 300, [("B3G_DIRECT", "0"), ("B3G_TREE", "2"), ("B3G_TREE", "0")]),
    (4, "f32", 3, 40, 300, [("B3G_TREE", "2"), ("B3G_TREE", "0")]),
])
def test_root_of_unrelated_entries(S, form, K, taxa, sites, switches, monkeypatch):
    c, internals, children, lengths, lnl = problem(S, K, taxa, sites)
    n, L = len(internals), taxa
    at = {int(v): k for k, v in enumerate(internals)}
    parent = {int(ch): int(v) for v, kids in zip(internals, children) for ch in kids}
    root = int(internals[-1])
    # entries at least two levels below the root, none above another
    below = [k for k in range(n - 1) if parent[int(internals[k])] != root]
    unrelated = [k for k in below
                 if not any(int(ch) >= L and at[int(ch)] in below[:3] for ch in children[k])][:3]
    for extra in (unrelated[:1], unrelated):
        picked = sorted(extra) + [n - 1]
        new = lengths.copy()
        new[picked] *= 1.3
        first = lengths.copy()
        first[n - 1] = new[n - 1]  # the root's edges only: the others are not on its path
        want = (lnl(first), lnl(new))
        rest = sorted({at[p] for k in extra for p in ancestors(int(internals[k]), parent)})
        for name, value in [("", "")] + switches:
            if name:
                monkeypatch.setenv(name, value)
            g = make(c, S, K, form)
            if name:
                monkeypatch.delenv(name)
            g.propose_lengths(internals, children, lengths, 1.0)
            g.log_likelihood()
            g.accept()
            g.propose_lengths(internals[picked], children[picked], new[picked], 1.0)
            assert abs(g.log_likelihood() - want[0]) <= TOL[form] * abs(want[0]), (name, value)
            g.accept()
            g.propose_lengths(internals[rest], children[rest], new[rest], 1.0)
            assert abs(g.log_likelihood() - want[1]) <= TOL[form] * abs(want[1]), (name, value)
            g.close()


def ancestors(v, parent):
    while v in parent:
        v = parent[v]
        yield v

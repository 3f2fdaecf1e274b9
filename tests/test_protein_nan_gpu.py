"""Transition matrices that overflow (a large negative edge length without the
shortcuts) give NaN for the patterns they reach, in every 20-state walk: on a
tip's edge (the tip row enters the parent's partial), on an internal edge (the
table enters a product), and as a partial of an earlier evaluation.  The other
category, of rate zero, stays finite, so that a lost NaN would be a plausible
likelihood."""

import numpy as np
import pytest

from tests.cases import protein_case
from tests.test_gpu_parity import lists_and_lengths
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# (-300: beyond FP32 only)
@pytest.mark.parametrize("form,switch,length", [
    ("f32", None, -1e5), ("f32", None, -300.0), ("f32", "B3G_TC20", -1e5),
    ("f32", "B3G_TC20", -300.0), ("f64", None, -1e5),
])
@pytest.mark.parametrize("kind", ["tip", "internal"])
def test_overflow_stays_nan(form, switch, length, kind, monkeypatch):
    from aspartik_gb300.calculator import Calculator

    if switch:
        monkeypatch.setenv(switch, "1")
    c = protein_case(14, 60, seed=14)
    leaves = np.repeat(c.leaves[:1], c.leaves.shape[0], axis=0)  # constant patterns
    tree = O.DatedTree(c.tree.parents, c.tree.heights)
    tree.mark_all_edges_updated()
    internals, children, lengths = lists_and_lengths(tree)
    n, L = len(internals), leaves.shape[0]
    parent = {int(ch): k for k, kids in enumerate(children) for ch in kids}
    # an edge whose lower end is a tip or not, at least two entries below the root
    at = next((k, j) for k in range(n - 1) for j in range(2)
              if (children[k][j] < L) == (kind == "tip") and
              parent[int(internals[k])] != n - 1)
    bad = lengths.copy()
    bad[at] = length
    g = Calculator.GB300(0, form).make20(leaves, leaves.shape[1], num_categories=2)
    g.set_reversible(c.rates, c.pi, shortcuts=False)
    g.set_category_rates([0.0, 1.0])
    g.propose_lengths(internals, children, lengths, 1.0)
    assert np.isfinite(g.log_likelihood())
    g.accept()
    g.propose_lengths(internals, children, bad, 1.0)
    assert np.isnan(g.log_likelihood())
    assert np.isnan(g.site_log_likelihoods()).all()
    g.accept()
    root = [n - 1]  # from the clean partials of that evaluation
    g.propose_lengths(internals[root], children[root], lengths[root], 1.0)
    assert np.isnan(g.log_likelihood())
    g.close()

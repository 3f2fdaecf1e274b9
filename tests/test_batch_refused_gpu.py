"""A batch whose members' lists do not fit the batched walks' shared memory is
refused with an error, and leaves the calculator and its thread as they were."""

import numpy as np
import pytest

from aspartik_gb300.schedule import Topology
from tests.cases import dna_case
from tests.test_phase_words_gpu import ladder

pytestmark = pytest.mark.gpu


def test_thread_goes_on_after_a_refused_batch():
    from aspartik_gb300._native import B3GError
    from aspartik_gb300.calculator import Batch, Calculator

    taxa = 16000  # a list of 256 KB and more
    parents, heights = ladder(taxa, 100)
    full = Topology(parents, heights).full()
    leaves = np.random.default_rng(1).choice(np.array([1, 2, 4, 8], np.uint8), size=(taxa, 3))
    big = Calculator.GB300(0, "f32").make4(leaves, 3, num_categories=4)
    c = dna_case(20, 100, seed=1)
    big.set_reversible(np.ones(6), c.pi)
    big.set_gamma(0.5)
    big.propose_lengths(*full)
    want = big.log_likelihood()
    big.accept()
    with pytest.raises(B3GError):
        Batch([big])
    big.propose_lengths(*full)
    assert big.log_likelihood() == want
    big.accept()
    small = Calculator.GB300(0, "f32").make4(c.leaves, c.leaves.shape[1])
    small.set_reversible(np.ones(6), c.pi)
    batch = Batch([small])
    lists = Topology(c.tree.parents, c.tree.heights).full()
    small.stage_lengths(*lists)
    batch.run()
    assert np.isfinite(batch.log_likelihoods()[0])
    batch.close()
    big.close()
    small.close()

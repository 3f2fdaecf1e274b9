"""20-state calculators driven from two host threads at once, one on lists that
take much shared memory a block and one on lists that take little (the FP64
walk with four groups and with one; the tcgen05 walk with a long and a short
list): every launch finds the shared memory it asks for, and every value is the
one that the calculator gives alone."""

import threading

import numpy as np
import pytest

from tests.cases import protein_case
from tests.test_gpu_parity import lists_and_lengths
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,jobs_of", [
    ("f64", ((24, "B3G_F64_GROUPS", "4"), (2, "B3G_F64_GROUPS", "1"))),
    ("f32", ((200, "B3G_TC20", "1"), (2, "B3G_TC20", "1"))),
])
def test_two_threads_lists_of_different_sizes(form, jobs_of, monkeypatch):
    from aspartik_gb300.calculator import Calculator

    jobs = []
    for taxa, name, value in jobs_of:
        monkeypatch.setenv(name, value)
        c = protein_case(taxa, 20, seed=taxa, num_categories=1)
        tree = O.DatedTree(c.tree.parents, c.tree.heights)
        tree.mark_all_edges_updated()
        lists = lists_and_lengths(tree)
        g = Calculator.GB300(0, form).make20(c.leaves, c.leaves.shape[1])
        g.set_weights(c.weights)
        g.set_reversible(c.rates, c.pi)
        g.propose_lengths(*lists, 1.0)
        jobs.append((g, lists, g.log_likelihood()))
        g.accept()
    errors, start = [], threading.Barrier(2)

    def drive(g, lists, want, stop, done):
        start.wait()
        try:
            while not stop.is_set():
                g.propose_lengths(*lists, 1.0)
                assert g.log_likelihood() == want
                g.reject()
                done[0] += 1
                if done[0] == 10000:
                    break
        except Exception as e:  # noqa: BLE001
            errors.append(e)
        stop.set()

    stop, counts = threading.Event(), [[0], [0]]
    threads = [threading.Thread(target=drive, args=(*j, stop, d)) for j, d in zip(jobs, counts)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g, _, _ in jobs:
        g.close()
    assert not errors, errors[0]
    assert np.min(counts) > 0

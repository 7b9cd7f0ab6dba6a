"""Serving on frequency nodes: runs over a bounded number of pairs, which requests
share and join between."""
import numpy as np
import pytest

import kestrel_b200 as kb
from kestrel_b200 import synth

pytestmark = pytest.mark.gpu

PANEL, SITES = 1024, 1500


@pytest.fixture(scope="module")
def est():
    with kb.Estimator() as e:
        e.panel_load(synth.make_cohort(PANEL, SITES, 61, missing=0.02).codes)
        yield e


def queries(n, seed):
    return synth.make_cohort(n, SITES, seed, missing=0.02).codes


def equal(a, b):
    return np.array_equal(a.view(np.uint8), b.view(np.uint8))


def test_a_small_request_is_not_held_up_by_large_ones(est):
    """Both workers have a request of 1.5 million pairs when one of 2,048 arrives: it
    joins a run and is answered while both of them still run.  (Several tries, since
    this thread may be stopped for longer than the large ones take; where a request
    waits for a worker, one of them has ended in every try.)"""
    small, large = queries(2, 62), queries(1500, 63)
    alone = est.wait(est.submit(small))
    for _ in range(5):
        big = [est.submit(large), est.submit(large)]
        rid = est.submit(small)
        rows = est.wait(rid)
        running = [not est.poll(b) for b in big]
        assert equal(rows, alone)
        first, second = (est.wait(b) for b in big)
        assert equal(first, second)
        if all(running):
            return
    raise AssertionError("the small request waited for a large one")


@pytest.mark.parametrize("n", [127, 128, 129, 257])
def test_rows_do_not_depend_on_the_runs(est, n):
    """Requests around one and two runs (131,072 pairs), alone and sharing runs."""
    q = queries(n, 70)
    want = np.concatenate([est.wait(est.submit(q[i:i + 40])) for i in range(0, n, 40)])
    alone = est.wait(est.submit(q))
    assert np.array_equal(alone["x"], np.repeat(np.arange(n), PANEL))
    ids = [est.submit(q), est.submit(q[:5]), est.submit(q[:90])]
    shared = [est.wait(i) for i in ids]
    want["x"] = alone["x"]
    assert equal(alone, want)
    for rows, k in zip(shared, (n, 5, 90)):
        assert equal(rows, alone[:k * PANEL])

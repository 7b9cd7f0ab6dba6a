"""kg_relatedness_batch on the buffers that an earlier call left: cohorts of other
sizes, orders and numbers, one that moves between frequency nodes and site
lists, and one that is refused, give the rows of a fresh context bit for bit."""
import numpy as np
import pytest

import kestrel_b200 as kb
from kestrel_b200 import synth

pytestmark = pytest.mark.gpu


def test_rows_on_kept_buffers():
    a, b, c = (synth.make_cohort(n, m, 40 + n, missing=0.03).codes for n, m in ((40, 3000), (9, 700), (17, 5001)))
    rare = np.zeros((30, 900), np.uint8)                      # REF frequencies of 1 in 4e7: on site lists
    rare[:, :] = a[:30, :900]
    af = np.full((900, 2), 0.5)
    af[0] = (1.0 - 2.5e-8, 2.5e-8)
    bad = np.full((4, 50), 7, np.uint8)
    calls = [[(a, None, None), (b, None, None)],
             [(c, None, 12), (a, None, 33), (b, None, None)],
             [(b, None, None), (rare, af, None)],
             [(rare, af, None), (c, None, None), (a, None, None)]]

    def run(est, call):
        return est.relatedness_batch(call, maf=0.0)

    fresh = []
    for call in calls:
        with kb.Estimator() as est:
            fresh.append(run(est, call))
    with kb.Estimator() as est:
        for k in (0, 1, 2, 3, 1, 0):
            for got, want in zip(run(est, calls[k]), fresh[k]):
                assert np.array_equal(got.view(np.uint8), want.view(np.uint8))
            with pytest.raises(kb.KestrelError):
                run(est, [(bad, None, None), (b, None, None)])

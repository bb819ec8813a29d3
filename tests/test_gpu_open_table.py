"""Open sigma calls one after another on one context: the hash table that a call leaves behind
(emptied as it is read out), kept over other numbers of roots, thresholds, body limits and states
of fewer and of more sectors, on either planner.  Every call gives the rows that the oracle gives;
the values are sums of up to a few hundred double products, so 1e-12 of the largest."""
import numpy as np
import pytest

import oracle
from fermicg_gb300.gpu import GpuSigma
from random_operators import random_operators, random_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device_plan", [True, False])
@pytest.mark.parametrize("norb,dims", [((3, 2, 3, 4), (3, 5)), ((1, 2), (2, 3))])
def test_calls_in_a_row(norb, dims, device_plan):
    ops, terms = random_operators(norb, dims, seed=11)
    ref = oracle.Oracle(ops, terms)
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    g.set_planner(device_plan)
    for n, calls in [(4, [(1, 0.0, 4)]), (60, [(3, 0.0, 4), (1, 0.5, 4), (2, 0.0, 2), (5, 0.0, 1), (3, 0.0, 4)]),
                     (9, [(16, 0.0, 3), (1, 1e30, 4), (1, 0.0, 4)])]:
        f, c = random_rows(ops, n, seed=n)
        g.state_set(f, c, plan=False)
        for R, thresh, nbody in calls:
            x = np.random.default_rng(R).standard_normal((len(f), R))
            of, oc, ov = g.sigma_open(x, thresh, nbody)
            rf, rc, rv = ref.sigma_open(f, c, x, thresh, nbody)
            key = lambda a, b: [tuple(r) for r in np.concatenate([a.reshape(len(a), 2 * len(norb)), b], axis=1).tolist()]
            got, want = dict(zip(key(of, oc), ov)), dict(zip(key(rf, rc), rv))
            assert len(got) == len(of)
            assert got.keys() == want.keys()
            if want:
                scale = np.abs(rv).max()
                assert max(np.abs(got[k] - want[k]).max() for k in want) <= 1e-12 * scale
    g.close()

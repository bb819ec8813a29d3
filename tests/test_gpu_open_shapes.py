"""Open sigma over the shapes its expand kernel distinguishes: index lengths of 1 to 4, 5 and 6
(register sums of each size) and above (shared-memory sums), pair counts around multiples of a
warp, and tiles that fit no shared-memory slice.  Row sets and values against the oracle; the
values are sums of up to a few hundred double products, so 1e-12 of the largest."""
import numpy as np
import pytest

import oracle
from fermicg_gb300.gpu import GpuSigma
from random_operators import random_operators, random_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,dims,n,R,thresh", [
    ((2, 3, 1, 2), (3, 4), 40, 2, 1e-3),       # D = 3, pairs below a warp
    ((3, 3, 3, 3), (4, 8), 30, 1, 0.0),        # exactly one warp of pairs; threshold 0 keeps all
    ((4, 4, 4, 4), (5, 7, 11), 25, 4, 0.3),    # D = 4, ragged pairs, sparse candidates
    ((6, 5, 4, 6), (3, 5), 20, 3, 2.0),        # D = 6, unequal lengths
    ((7, 8, 7, 9), (4, 6), 10, 2, 1.0),        # shared-memory sums
    ((9, 9, 9, 9), (20, 3), 4, 2, 0.5),       # tiles over a slice: per element
    ((2, 2, 2), (16, 17, 3), 30, 16, 0.1),     # 16 roots, 272 pairs, no four-cluster terms
])
def test_open_sigma_shapes(norb, dims, n, R, thresh):
    ops, terms = random_operators(norb, dims, seed=sum(norb))
    f, c = random_rows(ops, n, seed=3)
    x = np.random.default_rng(5).standard_normal((len(f), R))
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    g.state_set(f, c, plan=False)
    of, oc, ov = g.sigma_open(x, thresh)
    rf, rc, rv = oracle.Oracle(ops, terms).sigma_open(f, c, x, thresh)
    key = lambda a, b: [tuple(r) for r in np.concatenate([a.reshape(len(a), -1), b], axis=1).tolist()]
    got, want = dict(zip(key(of, oc), ov)), dict(zip(key(rf, rc), rv))
    assert len(got) == len(of) and len(want) > 0
    assert got.keys() == want.keys()
    scale = np.abs(rv).max()
    assert max(np.abs(got[k] - want[k]).max() for k in want) <= 1e-12 * scale
    g.close()

"""Open sigma over the lengths of a transfer's term list that its plan distinguishes (up to 8 by a
thread, longer ones by a warp in steps of 32), with terms left out of the middle of a list by the body
limit and by missing TDM blocks, from one row to more pairs of sectors and transfers than one round
of the plan's scan.  Row sets and values against the
oracle; the values are sums of up to a few hundred double products, so 1e-12 of the largest."""
import itertools

import numpy as np
import pytest

import oracle
from fermicg_gb300.gpu import GpuSigma
from fermicg_gb300.local_fci import OP_ID
from fermicg_gb300.pack import PackedOps, PackedTerms
from random_operators import random_operators, random_rows

pytestmark = pytest.mark.gpu

BODIES = [b for n in (2, 3, 4) for b in itertools.product(("Aa", "Bb"), repeat=n)] + [("A", "a"), ("Aa", "A", "a")]


@pytest.fixture(scope="module")
def problem():
    return random_operators((2, 2, 2, 2), (3, 2, 4), seed=6, bodies=BODIES)


@pytest.mark.parametrize("n", [1, 80])
@pytest.mark.parametrize("length", [1, 7, 8, 9, 31, 32, 33, 64, 75])
def test_lists(problem, length, n):
    ops, terms = problem
    zero = [i for i, t in enumerate(terms.transfers) if not t.any()][0]
    at = np.flatnonzero(terms.table[:, 1] == zero)
    at = np.random.default_rng(length).permutation(at)[:length]
    keep = np.sort(np.concatenate([np.flatnonzero(terms.table[:, 1] != zero), at]))
    terms = PackedTerms(terms.table[keep], terms.ints, terms.transfers)
    drop = (ops.table[:, 1] == OP_ID["Bb"]) & (ops.table[:, 2] == 2)  # of sector (2, 1)
    ops = PackedOps(ops.table[~drop], ops.data, ops.n_clusters, ops.cluster_norb)
    f, c = random_rows(ops, n, seed=3)
    _check(ops, terms, f, c, ((0.0, 4), (0.2, 3), (0.0, 2)))


@pytest.mark.parametrize("clusters,n,pairs", [(4, 300, (1024, 8192)), (5, 900, (8192, 1 << 20))])
def test_pairs(clusters, n, pairs):
    """Pairs of ket sector and transfer for several rounds of the small scan, and for the tiled scans."""
    bodies = list(itertools.permutations(("A", "a", "B", "b"))) + [("A", "a"), ("a", "A"), ("B", "b"), ("b", "B")]
    ops, terms = random_operators((2,) * clusters, (2, 1, 3), seed=8, bodies=bodies)
    f, c = random_rows(ops, n, seed=4)
    assert pairs[0] < len(np.unique(f.reshape(len(f), -1), axis=0)) * len(terms.transfers) + 1 <= pairs[1]
    _check(ops, terms, f, c, ((1.5, 4),))


def _check(ops, terms, f, c, calls):
    x = np.random.default_rng(5).standard_normal((len(f), 2))
    ref = oracle.Oracle(ops, terms)
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    g.state_set(f, c, plan=False)
    for thresh, nbody in calls:
        of, oc, ov = g.sigma_open(x, thresh, nbody)
        rf, rc, rv = ref.sigma_open(f, c, x, thresh, nbody)
        key = lambda a, b: [tuple(r) for r in np.concatenate([a.reshape(len(a), -1), b], axis=1).tolist()]
        got, want = dict(zip(key(of, oc), ov)), dict(zip(key(rf, rc), rv))
        assert len(got) == len(of)
        assert got.keys() == want.keys()
        if want:
            assert max(np.abs(got[k] - want[k]).max() for k in want) <= 1e-12 * np.abs(rv).max()
    g.close()

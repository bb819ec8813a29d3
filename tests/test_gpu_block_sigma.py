"""Closed sigma over the work items that run as block jobs (three or four active clusters), at the
edges of the blocks: groups of one to several hundred rows (partial and several blocks of 32 bras and
128 kets), index lengths with and without the unrolled contractions and over the limit of a block
job, lists of one term, of two of one shape and of unlike shapes, and every root count the kernel
distinguishes.  Against the oracle, through the device planner (block jobs) and the host planner
(lane jobs only).  FP64: sums of up to about 1e3 products of up to 5 factors, 1e-12 of the largest
value; FP32: the same sums at 6e-8, 2e-5."""
import numpy as np
import pytest

import oracle
from fermicg_gb300.gpu import GpuSigma
from helpers import rel_err
from random_operators import BODIES, random_operators, random_rows

pytestmark = pytest.mark.gpu

# merged terms (Aa A a with Bb A a; A a with AAa a), two terms of one shape (AAa Bb a, AAa Aa a)
TWO = [("Aa", "A", "a"), ("Bb", "A", "a"), ("AAa", "Bb", "a"), ("AAa", "Aa", "a"), ("A", "a", "B", "b"), ("A", "a"),
       ("AAa", "a")]
MIXED = [("A", "a", "Bb"), ("AAa", "a", "Aa"), ("A", "a", "Aa"), ("B", "A", "a", "b")]


@pytest.mark.parametrize("norb,dims,n,R,bodies", [
    ((4, 4, 4, 4), (4, 6), 12000, 4, TWO),
    ((4, 4, 4, 4), (9, 2), 12000, 1, MIXED),
    ((4, 4, 4), (17, 20), 8000, 2, BODIES[:5]),     # three clusters: a group is a sector, 600 rows
    ((3, 3, 3, 3), (5, 6), 18000, 3, BODIES),
    ((2, 5, 4, 3), (5, 7), 18000, 5, TWO),
    ((6, 5, 6, 5), (5, 3), 9000, 2, BODIES),
    ((4, 4, 4, 4), (1, 18), 14000, 7, MIXED),       # clusters of one state
    ((7, 7, 7, 7), (5, 4), 6500, 16, BODIES),       # four-cluster columns of 49: lane jobs
])
def test_block_jobs_match_the_oracle(norb, dims, n, R, bodies):
    ops, terms = random_operators(norb, dims, seed=11 + sum(norb), bodies=bodies)
    f, c = random_rows(ops, n, seed=5)
    x = np.random.default_rng(7).standard_normal((len(f), R))
    ref = oracle.Oracle(ops, terms).sigma_closed(f, c, x)
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    g.state_set(f, c)
    assert g.stats()["flops_executed"] // 2 >= 1 << 26  # large enough for block jobs
    assert rel_err(g.sigma_closed(x, "fp64"), ref) < 1e-12
    assert g.stats()["kernel_launches"] == 4  # pack, block jobs, lane jobs, unpack
    assert rel_err(g.sigma_closed(x, "fp32"), ref) < 2e-5
    for cand in range(4):
        g.set_tuning(cand)
        assert rel_err(g.sigma_closed(x, "fp64"), ref) < 1e-12
    g.set_planner(False)
    assert rel_err(g.sigma_closed(x, "fp64"), ref) < 1e-12
    g.close()


def test_planners_agree_on_block_items():
    """The lane jobs of block items come last in both planners' plans, and a plan made again on the
    same context drops the first one's block jobs."""
    ops, terms = random_operators((4, 4, 4, 4), (4, 6), 3, TWO)
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    for n in (21000, 60, 5000):  # with block jobs; with the shortest lane jobs; between
        f, c = random_rows(ops, n, seed=n)
        x = np.random.default_rng(n).standard_normal((len(f), 2))
        g.set_planner(False)
        g.state_set(f, c)
        host = g.plan_arrays()
        g.set_planner(True)
        dev = g.plan_arrays()
        assert all(np.array_equal(host[k], dev[k]) for k in ("perm", "ts", "jobs", "chunk_lo", "chunk_val"))
        assert rel_err(g.sigma_closed(x, "fp64"), oracle.Oracle(ops, terms).sigma_closed(f, c, x)) < 1e-12
    g.close()

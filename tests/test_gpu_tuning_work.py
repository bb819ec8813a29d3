"""What the tuner remembers for a shape is of the lane jobs that it timed: a plan that leaves work items
to block jobs (double, device planner) takes no choice from one that runs them as lane jobs, and a plan
without lane jobs to time leaves none."""
import numpy as np
import pytest

import oracle
from fermicg_gb300.gpu import GpuSigma
from helpers import rel_err
from random_operators import random_operators, random_rows

pytestmark = pytest.mark.gpu

TWO = [("Aa", "A", "a"), ("Bb", "A", "a"), ("AAa", "Bb", "a"), ("A", "a", "B", "b"), ("A", "a")]


def _tuned(ops, terms, f, c, x, device):
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    g.set_planner(device)
    g.state_set(f, c)
    out = g.sigma_closed(x, "fp64")
    s, t = g.stats(), g.tuning()
    g.close()
    return out, s, t


def test_choice_is_kept_by_the_lane_jobs_timed():
    ops, terms = random_operators((4, 4, 4, 4), (4, 6), seed=31, bodies=TWO)
    f, c = random_rows(ops, 15011, seed=6)
    x = np.random.default_rng(1).standard_normal((len(f), 2))
    _, s, _ = _tuned(ops, terms, f, c, x, False)
    assert s["tune_cache_hits"] == 0 and s["flops_executed"] // 2 >= 1 << 26
    _, s, t = _tuned(ops, terms, f, c, x, True)  # the same shape, fewer lane jobs
    assert s["tune_cache_hits"] == 0
    assert all(ms > 0 for ms in t["candidate_ms"]["fp64"])
    _, s, _ = _tuned(ops, terms, f, c, x, True)
    assert s["tune_cache_hits"] == 1
    _, s, _ = _tuned(ops, terms, f, c, x, False)
    assert s["tune_cache_hits"] == 1


def test_no_lane_jobs_to_time():
    """One three-body term over all three clusters: a work item is a pair of sectors, hundreds of rows each,
    and all run as block jobs."""
    ops, terms = random_operators((4, 4, 4), (32,), seed=3, bodies=[("Aa", "A", "a")])
    keep = terms.table[:, 0] == 3
    terms.table = terms.table[keep]
    f, c = random_rows(ops, 16000, seed=2)
    x = np.random.default_rng(1).standard_normal((len(f), 1))
    ref = oracle.Oracle(ops, terms).sigma_closed(f, c, x)
    for _ in range(2):
        out, s, t = _tuned(ops, terms, f, c, x, True)
        assert rel_err(out, ref) < 1e-12
        assert s["flops_executed"] // 2 >= 1 << 26 and s["kernel_launches"] == 3  # pack, block jobs, unpack: no lane jobs
        assert s["tune_cache_hits"] == 0 and t["fp64"] == 0
        assert not any(t["candidate_ms"]["fp64"])

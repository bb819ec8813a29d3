"""What the device planner counts while it joins (work items, triples, flops, lane and block jobs)
against the host planner: from one CTA's matches to more than one round of the counting kernel's grid
(152 x 8 CTAs of 256), and with sets of merged terms of which only some have their TDM block."""
import numpy as np
import pytest

import oracle
from fermicg_gb300.gpu import GpuSigma
from fermicg_gb300.local_fci import OP_ID
from fermicg_gb300.pack import PackedOps
from helpers import config1_subspace, packed, rel_err
from random_operators import random_operators, random_rows
from fermicg_gb300 import pack

pytestmark = pytest.mark.gpu

COUNTS = ("n_work_items", "n_triples", "flops_reference", "flops_executed")


def _counts(g, f, c):
    out = []
    for on_device in (False, True):
        g.set_planner(on_device)
        g.state_set(f, c)
        arrays = g.plan_arrays()
        s = g.stats()
        assert s["join_on_device"] == int(on_device)
        out.append([s[k] for k in COUNTS] + [len(arrays["jobs"]), arrays["items"]])
    assert out[0] == out[1]
    return out[1]


@pytest.mark.parametrize("n", [1, 40, 900, 30000])
def test_counts_over_the_grid(n):
    prob, st = config1_subspace(30000, 4)
    ops, terms = packed(prob)
    f, c, _, _ = pack.pack_state(st)
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    items = _counts(g, f[:n], c[:n])[-1]
    if n == 30000:
        assert items > 152 * 8 * 256
    g.close()


@pytest.mark.parametrize("gone", [("A",), ("AAa",), ("Aa",), ("Bb",), ("A", "Aa")])
def test_sets_with_missing_blocks(gone):
    bodies = [("Aa", "A", "a"), ("Bb", "A", "a"), ("A", "a"), ("AAa", "a"), ("A", "AAa"), ("Aa", "Aa")]
    ops, terms = random_operators((4, 4, 4), (4, 6), 9, bodies)
    # the blocks of these operators between two sectors of every cluster go, one kind at a time
    ids = [OP_ID[o] for o in gone]
    drop = np.isin(ops.table[:, 1], ids) & ((ops.table[:, 2] + ops.table[:, 3]) == 2)
    assert 0 < drop.sum() < np.isin(ops.table[:, 1], ids).sum()
    ops = PackedOps(ops.table[~drop], ops.data, ops.n_clusters, ops.cluster_norb)
    f, c = random_rows(ops, 700, seed=3)
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    _counts(g, f, c)
    x = np.random.default_rng(2).standard_normal((len(f), 2))
    ref = oracle.Oracle(ops, terms).sigma_closed(f, c, x)
    assert rel_err(g.sigma_closed(x, "fp64"), ref) < 1e-12
    g.close()

"""The ways a BST product runs its groups, each reached and counted (fcg_bst_paths), against the
oracle's build_sigma!: warps, CTA chunks with the bra core in shared memory and without, operators cut
into column ranges, cores of more than four modes, global workspaces, and the double groups that join
the latter; and the flop counts of fcg_stats restated from the triples and the ranks.  FP64 sums of up
to 2e4 products of unit variance (a rounding of 1.1e-16 each: 3e-14 of the largest value expected),
1e-12; FP32 2e-5."""
import itertools

import numpy as np
import pytest

from fermicg_gb300 import workloads
from fermicg_gb300.bst import PackedBST
from helpers import packed, rel_err
from oracle import bst as obst

pytestmark = pytest.mark.gpu


def _problem(n, norb=4):
    e = norb // 2
    return workloads.build_problem(norb * n, [norb] * n, [(e, e)] * n, 4 * n, 5, max_roots=1000, delta_elec=1, cmf=False)


def _vector(prob, ranks, sectors, R, seed=3):
    """One block per sector, every local state in range, cluster q of rank ranks[q] or what the sector allows."""
    rng, vec = np.random.default_rng(seed), {}
    for i, fs in enumerate(workloads.single_transfer_sectors(prob)[:sectors]):
        M = [b.basis[f].shape[1] for b, f in zip(prob.bases, fs)]
        rk = [min(r, m) for r, m in zip(ranks(i) if callable(ranks) else ranks, M)]
        factors = [np.linalg.qr(rng.standard_normal((m, r)))[0] for m, r in zip(M, rk)]
        vec[(tuple(fs), tuple((0, m) for m in M))] = {"core": [rng.standard_normal(rk) for _ in range(R)], "factors": factors}
    return vec


def _gpu(prob, pb, nbody):
    from fermicg_gb300.gpu import GpuSigma
    g = GpuSigma(0)
    po, pt = packed(prob)
    g.set_ops(po)
    g.set_terms(pt)
    g.bst_set(pb, nbody=nbody)
    return g


def _counts(pb, g):
    """(fma with every mode before the operator, fma by the cheapest sides) of every group per root, and
    its number of terms."""
    N, groups = pb.N, {}
    table = g.term_clusters
    for b, k, t, _ in g.bst_triples():
        mask = sum(1 << c for c in table[t])
        groups[(b, k, mask)] = groups.get((b, k, mask), 0) + 1
    out = []
    for (b, k, mask), nt in groups.items():
        B, K = pb.blocks[b, 5:5 + N], pb.blocks[k, 5:5 + N]
        act = [c for c in range(N) if mask >> c & 1]
        sp = [c for c in range(N) if not mask >> c & 1]
        m, kk = int(np.prod(B[act])), int(np.prod(K[act]))
        n = int(np.prod(B[sp]))
        modes = [] if b == k else [c for c in sp if B[c] > 1 or K[c] > 1]  # orthonormal factors

        def cost(post):
            size, total = int(np.prod(K)), 0
            for side in (0, 1):
                if side:
                    total += size * m
                    size = size // kk * m
                for c in modes:
                    if (c in post) == bool(side):
                        size = size // int(K[c])
                        total += size * int(B[c]) * int(K[c])
                        size *= int(B[c])
            return total

        best = first = cost(())
        if modes and len(modes) <= 4 and not (m >= 64 and kk >= 16) and m * kk * n <= 1 << 20:
            best = min(cost(p) for i in range(len(modes) + 1) for p in itertools.combinations(modes, i))
        out.append((first, best, nt))
    return out


CASES = {
    # clusters, orbitals of each, ranks, sectors, roots, nbody, (precision, tensor cores) -> paths
    "warps": (4, 2, (2, 1, 2, 2), 5, 1, 4, {("fp64", True): dict(warp=True, chunk=False)}),
    "six modes": (6, 2, (2, 3, 2, 3, 2, 2), 3, 1, 4, {("fp64", True): dict(chunk=True), ("fp32", True): dict(warp=True)}),
    "six larger modes": (6, 2, (4, 4, 3, 3, 3, 4), 2, 1, 4, {("fp64", True): dict(chunk=True), ("fp32", False): dict(chunk=True)}),
    "column ranges": (3, 4, (22, 23, 9), 3, 2, 2, {("fp64", True): dict(split=True, atomic_chunks=False, **{"global": False}),
                                                   ("fp32", False): dict(split=True, atomic_chunks=False)}),
    "bra core apart": (3, 4, (19, 19, 19), 2, 1, 2, {("fp64", True): dict(split=True, atomic_chunks=True, **{"global": False}),
                                                     ("fp32", False): dict(split=True, atomic_chunks=False)}),
    "largest chunks": (4, 4, (10, 11, 10, 11), 2, 2, 2, {("fp64", True): dict(atomic_chunks=True, **{"global": False}),
                                                         ("fp32", False): dict(atomic_chunks=True)}),
    "global": (4, 4, (12, 12, 12, 12), 2, 1, 2, {("fp64", True): {"chunk": False, "global": True},
                                                 ("fp32", False): {"split": True, "atomic_chunks": True, "global": False},
                                                 ("fp32", True): {"tensor": True}}),
}


@pytest.mark.parametrize("case", CASES)
def test_paths(case):
    n, norb, ranks, sectors, R, nbody, runs = CASES[case]
    prob = _problem(n, norb)
    vec = _vector(prob, ranks, sectors, R)
    pb = PackedBST(vec, n, R)
    g = _gpu(prob, pb, nbody)
    g.term_clusters = [list(t[2:2 + t[0]]) for t in packed(prob)[1].table]
    x = pb.cores_of(vec)
    want = pb.cores_of(obst.build_sigma(obst.zero_like(vec, R), vec, prob.ops, prob.ham, n, R, nbody=nbody))
    costs = _counts(pb, g)
    st = g.stats()
    assert len(costs) == st["bst_groups"]
    assert st["bst_flops_reference"] == 2 * sum(f * nt for f, _, nt in costs)
    assert st["bst_flops_executed"] == 2 * sum(f for f, _, _ in costs)
    for (precision, tensor_cores), expect in runs.items():
        g.bst_tensor_cores(tensor_cores)
        assert rel_err(g.bst_sigma(x, precision), want) < (1e-12 if precision == "fp64" else 2e-5)
        paths = g.bst_paths()
        for k, v in expect.items():
            assert (paths[k] > 0) == v, (precision, paths)
        assert paths["warp"] + paths["chunk"] + paths["global"] + paths["tensor"] == len(costs)
        done = g.stats()["bst_flops_executed"] // 2
        if paths["chunk"] == 0:
            assert done == sum(f for f, _, _ in costs)
        elif paths["chunk"] == len(costs):
            assert done == sum(b for _, b, _ in costs)
        else:
            assert sum(b for _, b, _ in costs) <= done <= sum(f for f, _, _ in costs)
    g.close()


@pytest.mark.parametrize("sectors,joined", [(3, False), (13, True)])
def test_double_groups_beside_many_large_ones(sectors, joined):
    """Double groups of 72 to 224 KB run in chunks, and from global workspaces where more than that take
    at least 152 groups."""
    prob = _problem(4)
    vec = _vector(prob, lambda i: (9, 9, 9, 9) if i == 1 else (12, 12, 12, 12), sectors, 1)
    pb = PackedBST(vec, 4, 1)
    g = _gpu(prob, pb, 2)
    x = pb.cores_of(vec)
    want = pb.cores_of(obst.build_sigma(obst.zero_like(vec, 1), vec, prob.ops, prob.ham, 4, 1, nbody=2))
    assert rel_err(g.bst_sigma(x, "fp64"), want) < 1e-12
    paths = g.bst_paths()
    assert (paths["global"] >= 152) == joined
    assert (paths["chunk"] == 0) == joined
    g.close()

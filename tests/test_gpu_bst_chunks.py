"""The CTA chunks of the BST sigma at the edges of their paths: rank-1 modes, ranks that are and are
not multiples of four, overlaps longer than the register mode products, operators small enough for
the coefficient tables and long enough for streamed columns, operator products cut into column
ranges, modes before and after the operator, and every root in its own chunk.  Against the oracle's
build_sigma!: FP64 sums of up to about 1e4 products, 1e-12 of the largest value; FP32 2e-5."""
import pytest

from fermicg_gb300 import workloads
from fermicg_gb300.bst import PackedBST, synthetic_bst
from helpers import packed, rel_err
from oracle import bst as obst

pytestmark = pytest.mark.gpu


def _problem(n):
    return workloads.build_problem(4 * n, [4] * n, [(2, 2)] * n, 8 * n, 5, max_roots=1000, delta_elec=1, cmf=False)


@pytest.mark.parametrize("clusters,sectors,max_q,ranks,R", [
    (3, 3, 3, (5, 8), 1),
    (3, 2, 3, (1, 9), 3),       # rank-1 modes, ranks across the multiples of four
    (3, 2, 2, (17, 20), 2),     # overlaps and operators over 16
    (2, 3, 2, (30, 35), 2),     # 1225 x 1225 operators: streamed, in column ranges
    (4, 2, 3, (3, 6), 2),       # four-cluster operators, up to two spectators
])
def test_chunks_match_the_oracle(clusters, sectors, max_q, ranks, R):
    from fermicg_gb300.gpu import GpuSigma
    prob = _problem(clusters)
    secs = workloads.single_transfer_sectors(prob)[:sectors]
    vec = synthetic_bst(prob, secs, max_q=max_q, rank_range=ranks, R=R, seed=7)
    pb = PackedBST(vec, clusters, R)
    po, pt = packed(prob)
    g = GpuSigma(0)
    g.set_ops(po)
    g.set_terms(pt)
    g.bst_set(pb)
    x = pb.cores_of(vec)
    want = pb.cores_of(obst.build_sigma(obst.zero_like(vec, R), vec, prob.ops, prob.ham, clusters, R))
    assert rel_err(g.bst_sigma(x, "fp64"), want) < 1e-12
    for tensor_cores in (True, False):
        g.bst_tensor_cores(tensor_cores)
        assert rel_err(g.bst_sigma(x, "fp32"), want) < 2e-5
    g.close()

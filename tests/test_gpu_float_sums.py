"""The single-precision products add their row sums in float64: the rms error against the double build
stays at what rounding the inputs and one job's or chunk's own sums give, on vectors whose rows take a
hundred and more sums (float additions of those: 1e-7 and more).

Each rounding to float is uniform within half a unit, u = 2^-24 / sqrt(3) relative at most, and of random
sign, so k of them on every product give sqrt(k) u of the sum.  From stored blocks: the element, the
coefficient, and a lane job's additions (up to 4 kets: sqrt(4 / 2) u) make k = 4.  Direct: the dressed
operator, up to three density matrices, the coefficient and the job's additions, k = 7.  Tucker: operator,
core, two overlaps and the sums, k = 5."""
import numpy as np
import pytest

from fermicg_gb300 import pack, workloads
from fermicg_gb300.bst import PackedBST, synthetic_bst
from fermicg_gb300.gpu import GpuSigma, sigma_closed_grouped
from helpers import packed

pytestmark = pytest.mark.gpu

U = 2.0 ** -24 / 3 ** 0.5


def _rms(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.fixture(scope="module", params=[2000, 4000])  # below and above the lane jobs whose rows are summed in runs
def closed(request):
    p = workloads.config0_problem()
    f, c, _, _ = pack.pack_state(workloads.energy_ordered_space(p, request.param, R=1))
    g = GpuSigma(0)
    g.set_ops(pack.pack_ops(p.ops, p.bases))
    g.set_terms(pack.pack_terms(p.ham))
    yield g, f, c
    g.close()


@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("stored", [False, True])
@pytest.mark.parametrize("R", [1, 2, 3, 4, 6, 8, 12])
def test_closed(closed, R, stored, grouped):
    import torch

    g, f, c = closed
    g.state_set(f, c)
    if stored:
        g.cache_hamiltonian()
    assert (len(g.plan_arrays()["jobs"]) >= 1 << 18) == (len(f) == 4000)
    x = np.asfortranarray(np.random.default_rng(R).standard_normal((len(f), R)))
    want = g.sigma_closed(x, "fp64")
    if grouped:
        d = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
        o = torch.zeros_like(d)
        torch.cuda.synchronize()
        sigma_closed_grouped([g], [d.data_ptr()], [o.data_ptr()], [R], "fp32")
        got = o.cpu().numpy().T
    else:
        got = g.sigma_closed(x, "fp32")
    assert _rms(got, want) < U * (4 if stored else 7) ** 0.5


@pytest.mark.parametrize("R", [1, 2, 3, 4, 6])
def test_infinite_coefficient(closed, R):
    """A row's one infinite product leaves its sum infinite, beside finite ones, in either precision."""
    g, f, c = closed
    g.state_set(f, c)
    g.cache_hamiltonian()
    x = np.asfortranarray(np.random.default_rng(R).standard_normal((len(f), R)))
    x[len(f) // 3] = np.inf
    want, got = g.sigma_closed(x, "fp64"), g.sigma_closed(x, "fp32")
    assert np.isinf(want).any() and np.isfinite(want).any()
    assert np.array_equal(np.isinf(got), np.isinf(want)) and np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.sign(got[np.isinf(want)]), np.sign(want[np.isinf(want)]))


@pytest.mark.parametrize("sectors,max_q,ranks", [(40, 1, (2, 4)), (24, 2, (2, 2)), (1, 4, (4, 6))])
def test_tucker(sectors, max_q, ranks):
    prob = workloads.config2_problem(0)
    vec = synthetic_bst(prob, workloads.single_transfer_sectors(prob)[:sectors], max_q=max_q, rank_range=ranks, R=1, seed=0)
    pb = PackedBST(vec, 8, 1)
    g = GpuSigma(0)
    po, pt = packed(prob)
    g.set_ops(po)
    g.set_terms(pt)
    g.bst_set(pb)
    x = np.random.default_rng(1).standard_normal((1, pb.core_total))
    assert _rms(g.bst_sigma(x, "fp32"), g.bst_sigma(x, "fp64")) < U * 5 ** 0.5
    assert (g.bst_paths()["chunk"] > 0) == (max_q == 4)
    g.close()

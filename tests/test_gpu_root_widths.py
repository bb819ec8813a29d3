"""Closed sigma over the numbers of roots that its kernels are compiled for: exact widths, the widths
of 8, 12 and 16 that serve several numbers, and rows read and added in whole vectors (a multiple of
16 bytes) or by element; direct, from stored blocks, and grouped (one width for all problems).  Every
column against the one-root sigma of that column by the same route: the same products, their sums in
another order, so up to 300 roundings of the largest sum of magnitudes (about 36 Eh on the diagonal
times a coefficient of at most 0.2, and less off it: 10)."""
import numpy as np
import pytest

from fermicg_gb300 import pack, workloads
from fermicg_gb300.gpu import GpuSigma, sigma_closed_grouped

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problem():
    p = workloads.config0_problem()
    f, c, _, _ = pack.pack_state(workloads.energy_ordered_space(p, 700, R=1))
    return pack.pack_ops(p.ops, p.bases), pack.pack_terms(p.ham), f, c


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("fp32", 2e-4)])
@pytest.mark.parametrize("R", [1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 13, 16])
def test_columns(problem, R, precision, tol):
    import torch

    ops, terms, f, c = problem
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    g.state_set(f, c)
    x = np.asfortranarray(np.random.default_rng(R).standard_normal((len(f), R)) / np.sqrt(len(f)))
    want = np.stack([g.sigma_closed(x[:, j:j + 1], "fp64")[:, 0] for j in range(R)], axis=1)
    got = g.sigma_closed(x, precision)
    assert np.abs(got - want).max() <= tol
    other = GpuSigma(0)
    other.set_ops(ops)
    other.set_terms(terms)
    other.state_set(f[:300], c[:300])
    xs = [x, np.asfortranarray(x[:300, :1])]
    small = other.sigma_closed(xs[1], "fp64")
    for stored in (False, True):
        if stored:
            g.cache_hamiltonian()
            assert np.abs(g.sigma_closed(x, precision) - want).max() <= tol
            other.cache_hamiltonian()
        d = [torch.from_numpy(np.ascontiguousarray(v.T)).cuda() for v in xs]
        o = [torch.zeros_like(v) for v in d]
        torch.cuda.synchronize()
        sigma_closed_grouped([g, other], [v.data_ptr() for v in d], [v.data_ptr() for v in o], [R, 1], precision)
        assert np.abs(o[0].cpu().numpy().T - want).max() <= tol
        assert np.abs(o[1].cpu().numpy().T - small).max() <= tol
    g.close()
    other.close()

"""Davidson steps over the sizes their kernels distinguish: a Ritz or projection step in one kernel
with its Gram product (up to 256 rows per row block, staging in 48 KB) or apart, several column
groups of 32, small matrices in the kernel's arguments (up to 128 values) or staged.  A solve stops
when its residual norms are below tol; for a symmetric H and unit vectors each Ritz value then lies
within tol of an eigenvalue (Weyl), and the residual norms of H X - X E, formed here from a sigma of
the returned vectors, agree with tol to the rounding of H X (1e-13 of |H| ~ 200 per element)."""
import numpy as np
import pytest

from fermicg_gb300 import pack, workloads
from fermicg_gb300.gpu import GpuSigma

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problems():
    out = {}
    for name, build in (("12o", workloads.config0_problem), ("24o", workloads.config1_problem)):
        p = build()
        out[name] = (p, pack.pack_ops(p.ops, p.bases), pack.pack_terms(p.ham))
    return out


@pytest.mark.parametrize("system,n,R,max_ss,tol", [
    ("12o", 60, 1, 12, 1e-8),      # one row block
    ("12o", 65, 3, 40, 1e-8),      # two row blocks; more than 32 columns; arguments, then staged
    ("12o", 400, 16, 12, 1e-6),    # staging above 48 KB: separate kernels
    ("12o", 2000, 2, 12, 1e-7),
    ("24o", 8193, 1, 12, 1e-4),    # 128 row blocks of 65 rows
    ("24o", 33000, 1, 12, 1e-3),   # more than 256 rows per row block: separate kernels
])
def test_solutions(problems, system, n, R, max_ss, tol):
    p, ops, terms = problems[system]
    f, c, _, _ = pack.pack_state(workloads.energy_ordered_space(p, n, R=1))
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    g.state_set(f, c)
    m = len(f)
    hd = g.diagonal()
    v0 = np.zeros((m, R))
    for j, i in enumerate(np.argsort(hd, kind="stable")[:R]):
        v0[i, j] = 1.0
    e, x, res, its = g.davidson(v0, max_iter=200, max_ss_vecs=max_ss, tol=tol, precision="fp64")
    assert res.max() < tol
    assert np.abs(x.T @ x - np.eye(R)).max() <= 1e-10
    hx = g.sigma_closed(x, "fp64")
    assert np.linalg.norm(hx - x * e, axis=0).max() <= tol + 2e-11 * np.sqrt(m)
    if m <= 500:
        h = g.sigma_closed(np.eye(m)[:, :16], "fp64")
        h = np.concatenate([h] + [g.sigma_closed(np.eye(m)[:, k:k + 16], "fp64") for k in range(16, m, 16)], axis=1)
        w = np.linalg.eigvalsh(0.5 * (h + h.T))
        assert max(np.abs(w - y).min() for y in e) <= tol
        assert abs(e[0] - w[0]) <= tol
    g.close()

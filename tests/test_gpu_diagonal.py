"""The diagonal of H over the numbers of lanes that share a row (2 to 32, by the number of rows), with
rows left over in the last warp of each, against the oracle.  Sums of about 2e3 terms of magnitude up
to 40 Eh, in another order than the oracle's: 1e-12 of the value."""
import numpy as np
import pytest

import oracle
from fermicg_gb300 import pack
from fermicg_gb300.gpu import GpuSigma
from helpers import config1_subspace, packed

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problem():
    prob, st = config1_subspace(30000, 4)
    ops, terms = packed(prob)
    f, c, _, _ = pack.pack_state(st)
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    yield g, f, c, oracle.Oracle(ops, terms).diagonal_H(f, c)
    g.close()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 2829, 5659, 11315, 22629, 29999])
def test_diagonal(problem, n):
    g, f, c, want = problem
    g.state_set(f[:n], c[:n], plan=False)
    np.testing.assert_allclose(g.diagonal(), want[:n], rtol=1e-12, atol=1e-12)

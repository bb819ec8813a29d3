"""An operator set that fcg_set_ops refuses leaves the context's last one in place: its state, products
and the term sets made from it afterwards."""
import numpy as np
import pytest

from fermicg_gb300.gpu import FcgError, GpuSigma
from fermicg_gb300.pack import PackedOps
from random_operators import random_operators, random_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("column,value", [(0, 3), (1, 99), (2, 9), (5, -1), (6, 0), (7, 300), (9, 1 << 40)])
def test_a_refused_set_changes_nothing(column, value):
    ops, terms = random_operators((2, 3, 2), (3, 4), seed=5)
    f, c = random_rows(ops, 60, seed=1)
    x = np.random.default_rng(0).standard_normal((len(f), 2))
    g = GpuSigma(0)
    g.set_ops(ops)
    g.set_terms(terms)
    g.state_set(f, c)
    want, rows = g.sigma_closed(x, "fp64"), g.sigma_open(x, 0.5)
    bad, at = ops.table.copy(), len(ops.table) // 2
    bad[at, column] = value
    other, _ = random_operators((4, 4), (2,), seed=6)
    for table, data, n, norb in ((bad, ops.data, 3, ops.cluster_norb), (other.table, other.data, 2, [4, 16])):
        with pytest.raises(FcgError):
            g.set_ops(PackedOps(table, data, n, np.array(norb, dtype=np.int32)))
    assert np.array_equal(g.sigma_closed(x, "fp64"), want)
    g.set_terms(terms)
    g.state_set(f, c)
    assert np.allclose(g.sigma_closed(x, "fp64"), want, rtol=0, atol=1e-12 * np.abs(want).max())
    assert len(g.sigma_open(x, 0.5)[0]) == len(rows[0])
    g.close()

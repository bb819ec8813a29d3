"""Random cluster operators and clustered terms of chosen index lengths and local dimensions, in
the packed form of the C ABI: shapes that a molecule small enough for a test does not reach."""
import itertools

import numpy as np

from fermicg_gb300 import pack
from fermicg_gb300.local_fci import OP_H, OP_ID, op_delta

SECTORS = [(1, 1), (0, 1), (2, 1), (1, 0), (1, 2)]
# one string of operators per number of active clusters and transfer
BODIES = [("A", "a"), ("Aa", "Aa"), ("Aa", "A", "a"), ("A", "Bb", "a"), ("B", "b", "Aa"), ("A", "a", "B", "b"),
          ("A", "B", "b", "a")]


def random_operators(norb, dims, seed, bodies=BODIES):
    """norb orbitals and dims[s % len(dims)] local states in sector s of each cluster; every TDM
    block between the sectors above, and one random term per entry of `bodies` and per choice of
    clusters.  Returns (PackedOps, PackedTerms)."""
    rng = np.random.default_rng(seed)
    N = len(norb)
    secs = [[s for s in SECTORS if max(s) <= norb[c]] for c in range(N)]
    dim = [{s: dims[(i + c) % len(dims)] for i, s in enumerate(secs[c])} for c in range(N)]
    rows, data, off = [], [], 0
    for c in range(N):
        for name in ["H"] + sorted({o for b in bodies for o in b}):
            da, db = (0, 0) if name == "H" else op_delta(name)
            nidx = 1 if name == "H" else norb[c] ** len(name)
            for fk in secs[c]:
                fb = (fk[0] + da, fk[1] + db)
                if fb not in dim[c]:
                    continue
                n = nidx * dim[c][fb] * dim[c][fk]
                rows.append([c, OP_H if name == "H" else OP_ID[name], *fb, *fk, nidx, dim[c][fb], dim[c][fk], off])
                data.append(rng.standard_normal(n) / np.sqrt(nidx))
                off += n
    ops = pack.PackedOps(np.array(rows, dtype=np.int64), np.concatenate(data), N, np.array(norb, dtype=np.int32))
    trans, terms, ints, off = {}, [], [], 0
    entries = [((c,), ("H",)) for c in range(N)]
    for b in bodies:
        entries += [(cl, b) for cl in itertools.combinations(range(N), len(b))]
    for cl, names in entries:
        delta = [(0, 0) if o == "H" else op_delta(o) for o in names]
        tr = [(0, 0)] * N
        for c, d in zip(cl, delta):
            tr[c] = d
        tid = trans.setdefault(tuple(tr), len(trans))
        shape = [1 if o == "H" else norb[c] ** len(o) for c, o in zip(cl, names)]
        r = np.zeros(pack.TRM_COLS, dtype=np.int64)
        r[0], r[1] = len(cl), tid
        r[2:10] = -1
        r[22:26] = 1
        for i, (c, o) in enumerate(zip(cl, names)):
            r[2 + i], r[6 + i] = c, OP_H if o == "H" else OP_ID[o]
            r[10 + i], r[14 + i] = delta[i]
            r[18 + i] = 0 if o == "H" else len(o) % 2
            r[22 + i] = shape[i]
        r[26], r[27] = off & 0xFFFFFFFF, off >> 32
        if len(cl) > 1:
            v = rng.standard_normal(int(np.prod(shape)))
            ints.append(v)
            off += v.size
        terms.append(r)
    terms.sort(key=lambda r: r[1])  # transfers in order, as the clustered operator is walked
    tr = np.array(list(trans), dtype=np.int16).reshape(-1, N, 2)
    return ops, pack.PackedTerms(np.array(terms, dtype=np.int64).astype(np.int32), np.concatenate(ints), tr)


def random_rows(ops, n, seed, total=None):
    """n distinct configurations, rows of a sector together: (fock, cfg).  total: (alpha, beta)
    electrons (default one of each spin per cluster)."""
    rng = np.random.default_rng(seed)
    N = ops.n_clusters
    total = total or (N, N)
    dim = {tuple(r[[0, 2, 3]]): int(r[7]) for r in ops.table if r[1] == OP_H}
    by = [[s for s in SECTORS if (c, *s) in dim] for c in range(N)]
    foc = [f for f in itertools.product(*by) if sum(x[0] for x in f) == total[0] and sum(x[1] for x in f) == total[1]]
    seen = {}
    for _ in range(50 * n):
        f = foc[rng.integers(len(foc))]
        c = tuple(int(rng.integers(dim[(q, *f[q])])) for q in range(N))
        seen.setdefault(f, {})[c] = None
        if sum(len(x) for x in seen.values()) >= n:
            break
    rows = [(f, c) for f, cs in seen.items() for c in cs]
    return (np.array([f for f, _ in rows], dtype=np.int16), np.array([c for _, c in rows], dtype=np.int16))

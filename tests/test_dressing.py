"""The dressing tables of a term set (csrc/plan.cpp op_cells, build_dress) against a plain
restatement: which terms share a W, the TDM blocks that each W sums, their order, and where every W
lies.  Whole numbers, compared exactly."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from fermicg_gb300.local_fci import OP_ID
from random_operators import BODIES, random_operators

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SETS = [("Aa", "A", "a"), ("Bb", "A", "a"), ("A", "a"), ("AAa", "a"), ("A", "AAa"), ("Aa", "Aa"), ("Aa", "Bb"),
        ("AAa", "Bb", "a"), ("AAa", "Aa", "a"), ("A", "a", "B", "b")]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("ds") / "libds.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(ROOT, "tests", "dressing_shim.cpp"),
                    os.path.join(ROOT, "fermicg_gb300", "csrc", "plan.cpp"), "-o", str(out)], check=True)
    L = ctypes.CDLL(str(out))
    L.ds_build.restype = ctypes.c_int64
    return L


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def build(lib, norb, table, trm, merge):
    s2 = (max(norb) + 1) ** 2
    n, cap = len(trm), 1 + len(trm) * len(table)
    norb, table = np.asarray(norb, dtype=np.int32), np.ascontiguousarray(table, dtype=np.int64)
    trm = np.ascontiguousarray(trm, dtype=np.int32)
    rep, w_index, w_mb = np.zeros(n, np.int32), np.zeros((n, s2), np.int64), np.zeros((n, s2), np.int32)
    jobs, src, n_src = np.zeros((cap, 6), np.int64), np.zeros((cap, 4), np.int64), ctypes.c_int64(0)
    nj = lib.ds_build(len(norb), _p(norb), ctypes.c_int64(len(table)), _p(table), n, _p(trm), int(merge),
                      ctypes.c_int64(cap), _p(rep), _p(w_index), _p(w_mb), _p(jobs), _p(src), ctypes.byref(n_src))
    assert nj >= 0
    return rep, w_index, w_mb, jobs[:nj], src[:n_src.value]


def plain(norb, table, trm, merge):
    s = max(norb) + 1
    blocks = {tuple(int(x) for x in r[:6]): (int(r[6]), int(r[7]), int(r[8]), int(r[9])) for r in table}
    pos = [max(range(r[0]), key=lambda o: (r[22 + o], -o)) if r[0] > 1 else 0 for r in trm]

    def cells(t):
        r, p = trm[t], pos[t]
        out = {}
        for (c, op, a, b, ka, kb), v in blocks.items():
            if c == r[2 + p] and op == r[6 + p] and a - ka == r[10 + p] and b - kb == r[14 + p]:
                out[a * s + b] = v
        return out

    have = [cells(t) for t in range(len(trm))]
    rep, sets, by = list(range(len(trm))), {}, {}
    for t, r in enumerate(trm):
        sets[t] = [t]
        if not merge or r[0] == 1:
            continue
        key = (r[1], r[0], pos[t]) + tuple((r[2 + o], r[10 + o], r[14 + o], r[18 + o]) +
                                           ((r[6 + o], r[22 + o]) if o != pos[t] else ()) for o in range(r[0]))
        t0 = by.get(key)
        if t0 is None:
            by[key] = t
        elif all(have[m][k][1:3] == have[t][k][1:3] for m in sets[t0] for k in have[m] if k in have[t]):
            rep[t] = t0
            sets[t0].append(t)
    w_index, w_mb = np.full((len(trm), s * s), -1, np.int64), np.zeros((len(trm), s * s), np.int32)
    jobs, src, n_w = [], [], 0
    for t0 in range(len(trm)):
        if rep[t0] != t0:
            continue
        rest = int(np.prod([trm[t0][22 + o] for o in range(trm[t0][0]) if o != pos[t0]])) if trm[t0][0] > 1 else 1
        for cell in sorted(set().union(*[have[t] for t in sets[t0]])):
            first = len(src)
            for t in sets[t0]:
                if cell in have[t]:
                    nidx, mb, mk, off = have[t][cell]
                    r = trm[t]
                    src.append((off, t, 1 if r[0] == 1 else nidx, int(np.prod(r[22:22 + pos[t]]))))
            n_w = (n_w + 7) // 8 * 8
            jobs.append((n_w, mb, mk, first, len(src) - first, int(trm[t0][0] == 1)))
            w_index[t0, cell], w_mb[t0, cell] = n_w, mb
            n_w += rest * mb * mk
    return rep, w_index, w_mb, jobs, src


@pytest.mark.parametrize("merge", [False, True])
@pytest.mark.parametrize("case", ["plain", "bodies", "missing", "shuffled", "repeated", "unequal", "no_blocks"])
def test_tables(lib, case, merge):
    norb = (2, 3, 4) if case != "bodies" else (3, 3, 2, 3)
    ops, terms = random_operators(norb, (3, 5, 2), seed=4, bodies=BODIES if case == "bodies" else SETS)
    table, rng = ops.table.copy(), np.random.default_rng(1)
    if case == "missing":
        table = table[rng.random(len(table)) < 0.6]
    elif case == "shuffled":
        table = table[rng.permutation(len(table))]
    elif case == "repeated":  # a block given twice: the later row counts
        again = table[::3].copy()
        again[:, 9] += 1000
        table = np.concatenate([table, again])
    elif case == "unequal":  # operators whose blocks differ in local dimensions share no W
        table[np.isin(table[:, 1], [OP_ID["Bb"], OP_ID["AAa"]]) & (table[:, 0] != 1), 7] += 1
    elif case == "no_blocks":
        table = table[:0]
    got, want = build(lib, norb, table, terms.table, merge), plain(norb, table, terms.table, merge)
    assert list(got[0]) == want[0]
    if merge and case in ("plain", "bodies", "shuffled", "repeated"):
        assert (got[0] != np.arange(len(got[0]))).any() or case == "bodies"
    assert np.array_equal(got[1], want[1])
    assert np.array_equal(got[2], want[2])
    assert [tuple(x) for x in got[3]] == want[3]
    assert [tuple(x) for x in got[4]] == want[4]

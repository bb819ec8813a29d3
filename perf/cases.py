"""The calls a user of this framework spends GPU time in, over the sizes they are used at.

Three molecules of the framework's own configurations: "12o" (12 orbitals, 4 clusters x 3, every
local state), "24o" (24 orbitals, 6 clusters x 4, 16 local states per sector), "32o" (32
orbitals, 8 clusters x 4, 16 local states per sector).  A molecule's operators and integrals are
built once per process (a program builds them once and runs many vectors on them); the
variational space and the coefficients come from the seed.

Kinds of case:
  sigma   closed sigma H c, matrix elements built on the fly (one matrix-vector product)
  stored  closed sigma from stored Hamiltonian blocks (what a Davidson solve repeats)
  solve   new variational space: state set, stored blocks, Davidson to convergence
  open    first-order-space sigma of a vector (the selection step of a macro-iteration)
  bst     block-sparse Tucker sigma with its operator cache on the device
  bst_set new Tucker factors: operator cache build, then one sigma
"""
import itertools
import itertools
import math

import numpy as np
import torch

from fermicg_gb300 import pack, workloads
from fermicg_gb300.bst import PackedBST
from fermicg_gb300.gpu import GpuSigma

OP_H = 22  # id of the local Hamiltonian in a packed operator table


def listed():
    return [
        # a small active space, one root: latency and launches count
        {"name": "sigma 12o 2e3 R1 fp64", "kind": "sigma", "system": "12o", "n": 2000, "roots": 1, "precision": "fp64"},
        # an ordinary solve's product, ragged size, odd root count, mixed precision
        {"name": "sigma 24o 1e4 R3 fp32", "kind": "sigma", "system": "24o", "n": 10007, "roots": 3, "precision": "fp32"},
        # the benchmark's headline size, mixed precision and double
        {"name": "sigma 24o 1e5 R4 fp32", "kind": "sigma", "system": "24o", "n": 100000, "roots": 4, "precision": "fp32"},
        {"name": "sigma 24o 1e5 R4 fp64", "kind": "sigma", "system": "24o", "n": 100000, "roots": 4, "precision": "fp64"},
        # many clusters, small groups
        {"name": "sigma 32o 2e4 R2 fp64", "kind": "sigma", "system": "32o", "n": 20011, "roots": 2, "precision": "fp64"},
        # the product a Davidson solve repeats once its blocks are stored
        {"name": "stored 24o 5e4 R4 fp32", "kind": "stored", "system": "24o", "n": 50021, "roots": 4, "precision": "fp32"},
        # one macro-iteration's variational solve, everything that a new space costs included
        {"name": "solve 12o 2e3 R1 fp64", "kind": "solve", "system": "12o", "n": 2000, "roots": 1, "precision": "fp64"},
        # the selection step: a small space at a tight threshold, and a large one
        {"name": "open 12o 300 R2 1e-6", "kind": "open", "system": "12o", "n": 300, "roots": 2, "thresh": 1e-6},
        {"name": "open 24o 3e3 R4 1e-3", "kind": "open", "system": "24o", "n": 3001, "roots": 4, "thresh": 1e-3},
        # Tucker vectors: small cores in double, the benchmark's large cores in single
        {"name": "bst 32o s7 q2 R1 fp64", "kind": "bst", "system": "32o", "sectors": 7, "max_q": 2, "rank_lo": 2,
         "rank_hi": 8, "roots": 1, "precision": "fp64"},
        {"name": "bst 32o s5 q4 R2 fp32", "kind": "bst", "system": "32o", "sectors": 5, "max_q": 4, "rank_lo": 4,
         "rank_hi": 12, "roots": 2, "precision": "fp32"},
        # new Tucker factors (each macro-iteration of a Tucker solve): operator cache and one product
        {"name": "bst_set 32o s3 q3 R1 fp64", "kind": "bst_set", "system": "32o", "sectors": 3, "max_q": 3,
         "rank_lo": 3, "rank_hi": 8, "roots": 1, "precision": "fp64"},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sigma", "sigma", "sigma", "stored", "solve", "open", "open", "bst", "bst", "bst_set"])
    if kind in ("sigma", "stored"):
        system = rng.choice(["12o", "24o", "24o", "32o"])
        hi = {"12o": 8000, "24o": 100000, "32o": 50000}[system]
        return {"kind": kind, "system": system, "n": _spread(rng, 500, hi), "roots": rng.randint(1, 6),
                "precision": rng.choice(["fp32", "fp64"])}
    if kind == "solve":
        return {"kind": kind, "system": "12o", "n": _spread(rng, 500, 3000), "roots": 1, "precision": "fp64"}
    if kind == "open":
        system = rng.choice(["12o", "24o"])
        n = _spread(rng, 50, 500) if system == "12o" else _spread(rng, 50, 3000)
        lo = 1e-6 if system == "12o" else (1e-4 if n < 300 else 1e-3)
        return {"kind": kind, "system": system, "n": n, "roots": rng.randint(1, 4),
                "thresh": lo * 10 ** rng.uniform(0.0, 0.7)}
    lo = rng.randint(2, 4)
    if kind == "bst_set":
        q = rng.randint(2, 3)
        return {"kind": kind, "system": "32o", "sectors": rng.randint(1, 3 if q == 3 else 9), "max_q": q, "rank_lo": lo,
                "rank_hi": lo + rng.randint(1, 4), "roots": rng.randint(1, 2), "precision": rng.choice(["fp32", "fp64"])}
    q = rng.randint(2, 4)
    precision = rng.choice(["fp32", "fp64"])
    sectors = rng.randint(1, {2: 24, 3: 9, 4: 5 if precision == "fp32" else 2}[q])
    return {"kind": kind, "system": "32o", "sectors": sectors, "max_q": q, "rank_lo": lo,
            "rank_hi": lo + rng.randint(1, 8 if q < 4 else 6), "roots": rng.randint(1, 2), "precision": precision}


# ---- inputs -------------------------------------------------------------------------------

_molecules = {}
_spaces = {}


class _Molecule:
    def __init__(self, system):
        build = {"12o": workloads.config0_problem, "24o": workloads.config1_problem, "32o": workloads.config2_problem}
        self.prob = build[system]()
        self.ops = pack.pack_ops(self.prob.ops, self.prob.bases)
        self.terms = pack.pack_terms(self.prob.ham)
        self.N = len(self.prob.clusters)


def _molecule(system):
    if system not in _molecules:
        _molecules[system] = _Molecule(system)
    return _molecules[system]


def _superset(system, n):
    """Rows (fock, cfg, summed local energy) of the lowest 5/4 n configurations."""
    want = n + n // 4 + 8
    have = _spaces.get(system)
    if have is None or have[3] < want:
        m = _molecule(system)
        f, c, _, _ = pack.pack_state(workloads.energy_ordered_space(m.prob, want, R=1, seed=0))
        e = np.zeros(len(f))
        for k, b in enumerate(m.prob.bases):
            top = 1 + max(len(x) for x in b.energies.values())
            table = np.zeros((16, 16, top))
            for (na, nb), x in b.energies.items():
                table[na, nb, :len(x)] = x
            e += table[f[:, k, 0], f[:, k, 1], c[:, k]]
        _spaces[system] = have = (f, c, e, want)
    f, c, e, _ = have
    if len(f) > want:  # the lowest `want` of them, in the same row order
        low = np.sort(np.argsort(e, kind="stable")[:want])
        f, c, e = f[low], c[low], e[low]
    return f, c, e


def _space(case, seed):
    """A selected space: n of the lowest 5/4 n configurations, chosen by the seed, and R columns
    of normalised coefficients that fall off with the energy, as a converged vector's do.  For
    the first-order space the seed chooses the coefficients' signs and the rest is the molecule's:
    the thresholds, and so the number of rows that come back, depend on the magnitudes."""
    f, c, e = _superset(case["system"], case["n"])
    n = min(case["n"], len(f))
    rng = np.random.default_rng(0 if case["kind"] == "open" else seed)
    drop = 1 + rng.permutation(len(f) - 1)[:len(f) - n]  # the reference configuration stays
    keep = np.ones(len(f), dtype=bool)
    keep[drop] = False
    f, c, e = np.ascontiguousarray(f[keep]), np.ascontiguousarray(c[keep]), e[keep]
    v = rng.standard_normal((n, case["roots"])) * np.exp(-2.0 * (e - e.min()) / max(np.ptp(e), 1e-12))[:, None]
    if case["kind"] == "open":
        v = v * np.random.default_rng(seed).choice([-1.0, 1.0], size=v.shape)
    return f, c, e, v / np.linalg.norm(v, axis=0, keepdims=True)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _columns(v):
    """Column-major (n, R) on the device: an (R, n) tensor."""
    return torch.from_numpy(np.ascontiguousarray(v.T)).to(_device())


def _tucker(case, seed):
    """A Tucker vector: every configuration of ranges with at most max_q clusters excited (local
    states 1.., the others in their lowest state) of the first charge-transfer sectors.  Ranks
    are the molecule's, orthonormal factors and cores the seed's."""
    m = _molecule(case["system"])
    shapes, rng = np.random.default_rng(0), np.random.default_rng(seed)
    vec = {}
    for fs in workloads.single_transfer_sectors(m.prob)[:case["sectors"]]:
        states = [m.prob.bases[q].basis[fs[q]].shape[1] for q in range(m.N)]
        can = [q for q in range(m.N) if states[q] > 1]
        for nq in range(case["max_q"] + 1):
            for excited in itertools.combinations(can, nq):
                ranges = tuple((1, states[q]) if q in excited else (0, 1) for q in range(m.N))
                factors = []
                for lo, hi in ranges:
                    rank = 1 if hi - lo == 1 else min(hi - lo, int(shapes.integers(case["rank_lo"], case["rank_hi"] + 1)))
                    factors.append(np.linalg.qr(rng.standard_normal((hi - lo, rank)))[0])
                core = rng.standard_normal([case["roots"]] + [x.shape[1] for x in factors])
                vec[(tuple(fs), ranges)] = {"core": list(core), "factors": factors}
    return m, vec, PackedBST(vec, m.N, case["roots"])


def prepare(case, seed):
    s = {"case": case}
    kind = case["kind"]
    if kind in ("bst", "bst_set"):
        m, vec, pb = _tucker(case, seed)
        g = GpuSigma(0)
        g.set_ops(m.ops)
        g.set_terms(m.terms)
        if kind == "bst":
            g.bst_set(pb)
        s.update(g=g, pb=pb, c=torch.from_numpy(pb.cores_of(vec)).to(_device()))
    else:
        m = _molecule(case["system"])
        f, c, _, v = _space(case, seed)
        g = GpuSigma(0)
        g.set_ops(m.ops)
        g.set_terms(m.terms)
        s.update(g=g, f=f, cfg=c, v=v)
        if kind in ("sigma", "stored"):
            g.state_set(f, c)
            if kind == "stored":
                g.cache_hamiltonian()
            s["c"] = _columns(v)
        elif kind == "solve":
            s["guess"] = workloads.davidson_guess(len(f), case["roots"], seed=seed, lowest=[int(np.argmin(_space(case, seed)[2]))])
        else:
            g.state_set(f, c, plan=False)
            s["strides"] = torch.tensor([1 << (4 * j) for j in range(2 * m.N)], dtype=torch.int64, device=_device())
            s["radix"] = torch.tensor([1 << (4 * j) for j in range(m.N)], dtype=torch.int64, device=_device())
    if "c" in s:
        s["out"] = torch.empty_like(s["c"])
    return s


def run(s):
    case, g = s["case"], s["g"]
    kind = case["kind"]
    if kind in ("sigma", "stored"):
        g.sigma_closed_device(s["c"].data_ptr(), s["out"].data_ptr(), case["roots"], case["precision"])
    elif kind == "solve":
        g.state_set(s["f"], s["cfg"])
        g.cache_hamiltonian()
        e, x, _, _ = g.davidson(s["guess"], max_iter=200, tol=1e-9, precision=case["precision"])
        return {"energies": e, "vectors": x}
    elif kind == "open":
        return _ordered(s, *g.sigma_open(s["v"], case["thresh"]))
    else:
        if kind == "bst_set":
            g.bst_set(s["pb"])
        g.bst_sigma_device(s["c"].data_ptr(), s["out"].data_ptr(), case["roots"], case["precision"])
    # the single-precision build writes its float values widened; as floats they are what it computed
    return s["out"].float() if case["precision"] == "fp32" else s["out"]


def _ordered(s, f, c, v):
    """The first-order space in a fixed order (sector, then configuration) on the device, where
    the program that goes on with it has it: the library returns its rows in any order."""
    dev = s["strides"].device
    f, c, v = torch.from_numpy(f).to(dev), torch.from_numpy(c).to(dev), torch.from_numpy(v.T).to(dev)
    sec = (f.reshape(f.shape[0], -1).long() * s["strides"]).sum(1)
    at = torch.argsort((c.long() * s["radix"]).sum(1))  # local states fit 4 bits
    at = at[torch.argsort(sec[at], stable=True)]
    return {"fock": f[at], "cfg": c[at], "coef": v[:, at]}


# ---- what a pass cannot do without ---------------------------------------------------------

def _lists(m):
    """Terms by (transfer, active clusters)."""
    t = m.terms.table
    by = {}
    for i in range(t.shape[0]):
        act = tuple(int(x) for x in t[i, 2:2 + t[i, 0]])
        by.setdefault((int(t[i, 1]), act), []).append(i)
    return by


def _sectors(m, f):
    """Row sectors: distinct Fock rows and the sector of each row."""
    packed = np.zeros(len(f), dtype=np.int64)
    for j in range(2 * m.N):
        packed |= f.reshape(len(f), -1)[:, j].astype(np.int64) << (4 * j) if j < 15 else \
            (f.reshape(len(f), -1)[:, j].astype(np.uint64) << np.uint64(4 * j)).astype(np.int64)
    _, first, sec = np.unique(packed, return_index=True, return_inverse=True)
    return f[first].reshape(len(first), 2 * m.N), sec.reshape(-1)


def _pairs(m, f, c, expand):
    """Coupled pairs of every (transfer, active clusters) list: yields (terms, sector table, sectors,
    bra rows, ket rows), or (terms, pair count) with expand=False.  A ket couples when it equals the
    bra on every other cluster and its sector plus the transfer is the bra's."""
    dev = _device()
    secs, sec = _sectors(m, f)
    index = {tuple(x): i for i, x in enumerate(secs.tolist())}
    cfg = torch.from_numpy(c.astype(np.int64)).to(dev)
    row_sec = torch.from_numpy(sec.astype(np.int64)).to(dev)
    n = len(f)
    by = {}
    for (tr, act), terms in _lists(m).items():
        by.setdefault(tr, []).append((act, terms))
    spec = {}
    for tr, lists in by.items():
        delta = m.terms.transfers[tr].reshape(-1).astype(np.int64)
        of = np.array([index.get(tuple(x), -1) for x in (secs.astype(np.int64) - delta).tolist()], dtype=np.int64)
        if (of < 0).all():
            continue
        ket_of = torch.from_numpy(of).to(dev)[row_sec]  # ket sector that couples to each bra row
        for act, terms in lists:
            if act not in spec:
                k = torch.zeros(n, dtype=torch.int64, device=dev)
                for q in range(m.N):
                    if q not in act:
                        k = k * 32 + cfg[:, q]
                full = row_sec * (1 << 35) + k
                spec[act] = (k, *torch.sort(full))
            k, ks, order = spec[act]
            want = torch.where(ket_of >= 0, ket_of * (1 << 35) + k, torch.full_like(k, -1))
            lo, hi = torch.searchsorted(ks, want), torch.searchsorted(ks, want, right=True)
            cnt = hi - lo
            if not expand:
                yield terms, cnt.sum()
                continue
            total = int(cnt.sum())
            if total == 0:
                continue
            b = torch.repeat_interleave(torch.arange(n, device=dev), cnt)
            at = torch.arange(total, device=dev) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt)
            yield terms, secs, row_sec, b, order[lo[b] + at]


def _open_counts(m, f):
    """(ket row, term, bra tuple) contributions of the open sigma."""
    t, blk = m.terms.table, _blocks(m)[0]
    secs, sec = _sectors(m, f)
    rows = np.bincount(sec, minlength=len(secs))
    total = 0
    for i in range(t.shape[0]):
        fb = secs + m.terms.transfers[t[i, 1]].reshape(-1)
        ok = ((fb >= 0) & (fb < blk.shape[2])).all(axis=1)
        cnt = rows * ok
        g = np.where(ok[:, None], fb, 0)
        for q in range(m.N):  # every cluster has a basis there
            cnt = cnt * (blk[q, OP_H, g[:, 2 * q], g[:, 2 * q + 1], g[:, 2 * q], g[:, 2 * q + 1]] >= 0)
        for o in range(t[i, 0]):
            q, op = t[i, 2 + o], t[i, 6 + o]
            b = blk[q, op, g[:, 2 * q], g[:, 2 * q + 1], secs[:, 2 * q], secs[:, 2 * q + 1]]
            cnt = cnt * np.where(b >= 0, m.ops.table[b, 7], 0)
        total += int(cnt.sum())
    return total


_works = {}


def work(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _works:
        _works[key] = _work(case)
    return _works[key]


def _work(case):
    """Inputs read once and outputs written once; one multiply-add per coupled (bra, ket, term)
    and per (bra, ket, root) for a product, per contribution of a first-order space, and per
    element of the operators and the smaller of the two cores for a Tucker product."""
    kind = case["kind"]
    m = _molecule(case["system"])
    tables = 8.0 * (m.ops.data.size + m.terms.ints.size)
    if kind in ("bst", "bst_set"):
        _, _, pb = _tucker(case, 0)
        by, ops, flops = _tucker_groups(m, pb), 0.0, 0.0
        for (b, k, act) in by:
            rb, rk = pb.blocks[b, 5:5 + m.N], pb.blocks[k, 5:5 + m.N]
            size = float(np.prod([rb[q] * rk[q] for q in act]))
            ops += size
            flops += 2.0 * case["roots"] * size * float(np.prod([min(rb[q], rk[q]) for q in range(m.N) if q not in act]))
        size = 4 if case["precision"] == "fp32" else 8
        nbytes = 16.0 * case["roots"] * pb.core_total + size * ops + (tables + 8.0 * pb.factors.size if kind == "bst_set" else 0.0)
        return {"bytes": nbytes, "flops": flops + (2.0 * ops if kind == "bst_set" else 0.0)}
    f, c, _, _ = _space(case, 0)
    n, R = len(f), case["roots"]
    if kind == "open":
        return {"bytes": tables + n * (8.0 * R + 6.0 * m.N), "flops": 2.0 * _open_counts(m, f)}
    pairs = triples = 0.0
    for terms, cnt in _pairs(m, f, c, False):
        cnt = float(cnt)
        pairs += cnt
        triples += cnt * len(terms)
    vectors = 16.0 * n * R
    if kind == "stored":
        size = 4 if case["precision"] == "fp32" else 8
        return {"bytes": vectors + size * pairs / 2, "flops": 2.0 * pairs * R}  # H is symmetric
    flops = 2.0 * (triples + pairs * R)
    if kind == "solve":  # the elements once, then a product for each of some forty iterations
        return {"bytes": tables + 6.0 * m.N * n + vectors, "flops": 2.0 * (triples + 40 * pairs * R)}
    return {"bytes": vectors + tables + 6.0 * m.N * n, "flops": flops}


# ---- the same results in 64 bits, by plain numpy and torch --------------------------------

def _blocks(m):
    if not hasattr(m, "blk"):
        t = m.ops.table
        top = int(t[:, 2:6].max()) + 1
        blk = np.full((m.N, 24, top, top, top, top), -1, dtype=np.int64)
        for i, r in enumerate(t.tolist()):
            blk[tuple(r[:6])] = i
        dev = _device()
        m.blk = (blk, torch.from_numpy(m.ops.data).to(dev), torch.from_numpy(t).to(dev))
    return m.blk


def _column(m, q, op, fb, fk, I, J):
    """<I| op |J> of cluster q for every orbital index: (pairs, indices), 0 where no block exists.
    fb, fk: (pairs,) sector numbers of the cluster, alpha * top + beta."""
    blk, data, table = _blocks(m)
    top = blk.shape[2]
    flat = torch.from_numpy(blk[q, op].reshape(top * top, top * top)).to(data.device)
    b = flat[fb, fk]
    nidx = int(m.ops.table[(m.ops.table[:, 0] == q) & (m.ops.table[:, 1] == op), 6].max(initial=1))
    r = table[b.clamp(min=0)]
    at = r[:, 9] + nidx * (I + r[:, 7] * J)
    g = data[(at[:, None] + torch.arange(nidx, device=data.device)).clamp(max=data.numel() - 1)]
    return g * (b >= 0)[:, None]


def _elements(m, terms, secs, sb, sk, cb, ck):
    """Sum over a list's terms of <bra| term |ket> for each pair."""
    t, top = m.terms.table, _blocks(m)[0].shape[2]
    dev = cb.device
    sec = torch.from_numpy(secs.astype(np.int64)).to(dev)
    fb, fk = sec[sb], sec[sk]
    out = torch.zeros(len(cb), dtype=torch.float64, device=dev)
    ne = fk[:, 0::2] + fk[:, 1::2]
    for i in terms:
        r = t[i]
        nb = int(r[0])
        g = []
        for o in range(nb):
            q, op = int(r[2 + o]), int(r[6 + o])
            g.append(_column(m, q, op, fb[:, 2 * q] * top + fb[:, 2 * q + 1], fk[:, 2 * q] * top + fk[:, 2 * q + 1],
                             cb[:, q], ck[:, q]))
        if nb == 1:
            out += g[0][:, 0]
            continue
        dims = [int(x) for x in r[22:22 + nb]]
        off = (int(r[26]) & 0xFFFFFFFF) | (int(r[27]) << 32)
        v = torch.from_numpy(m.terms.ints[off:off + int(np.prod(dims))]).to(dev).reshape(-1, dims[0])
        x = g[0] @ v.T  # (pairs, d1 * d2 * d3), the second index fastest
        for o in range(1, nb):
            x = (x.reshape(len(x), -1, dims[o]) * g[o][:, None, :]).sum(2)
        odd = torch.zeros(len(cb), dtype=torch.int64, device=dev)
        for o in range(nb):
            if r[18 + o]:
                odd += ne[:, :int(r[2 + o])].sum(1)
        out += x[:, 0] * (1 - 2 * (odd % 2)).double()
    return out


def _apply(m, f, c, v, dense=False):
    """H v (or the dense H) on the space, pair by pair."""
    dev = _device()
    n = len(f)
    cfg = torch.from_numpy(c.astype(np.int64)).to(dev)
    x = torch.from_numpy(np.ascontiguousarray(v)).to(dev)
    out = torch.zeros((n * n,) if dense else (n, v.shape[1]), dtype=torch.float64, device=dev)
    for terms, secs, row_sec, b, k in _pairs(m, f, c, True):
        for p in range(0, len(b), 1 << 21):
            bb, kk = b[p:p + (1 << 21)], k[p:p + (1 << 21)]
            h = _elements(m, terms, secs, row_sec[bb], row_sec[kk], cfg[bb], cfg[kk])
            if dense:
                out.index_add_(0, bb * n + kk, h)
            else:
                out.index_add_(0, bb, h[:, None] * x[kk])
    return out.reshape(n, n) if dense else out


def _tucker_groups(m, pb):
    """Terms by (bra block, ket block, active clusters) of a Tucker vector."""
    N = m.N
    start, length = pb.blocks[:, 5 + N:5 + 2 * N], pb.blocks[:, 5 + 2 * N:5 + 3 * N]
    fock = [tuple(x for p in key[0] for x in p) for key in pb.keys]
    by_fock = {}
    for i, x in enumerate(fock):
        by_fock.setdefault(x, []).append(i)
    blk, t, out, tables = _blocks(m)[0], m.terms.table, {}, {}
    per_tr = {}
    for (tr, act), terms in _lists(m).items():
        per_tr.setdefault(tr, []).append((act, terms))
    for fb, bras in by_fock.items():
        for tr, lists in per_tr.items():
            fk = tuple(int(a - d) for a, d in zip(fb, m.terms.transfers[tr].reshape(-1)))
            if fk not in by_fock:
                continue
            for act, terms in lists:
                ok = [i for i in terms if all(
                    blk[q, o, fb[2 * q], fb[2 * q + 1], fk[2 * q], fk[2 * q + 1]] >= 0
                    for q, o in zip(act, t[i, 6:10].tolist()))]
                if not ok:
                    continue
                if (fk, act) not in tables:
                    d = {}
                    for k in by_fock[fk]:
                        d.setdefault(tuple((start[k, q], length[k, q]) for q in range(N) if q not in act), []).append(k)
                    tables[(fk, act)] = d
                for b in bras:
                    for k in tables[(fk, act)].get(tuple((start[b, q], length[b, q]) for q in range(N) if q not in act), []):
                        out[(b, k, act)] = ok
    return out


def _tucker_sigma(m, vec, pb, R):
    """build_sigma! block by block; None where that would take long."""
    N, t, blk = m.N, m.terms.table, _blocks(m)[0]
    groups = _tucker_groups(m, pb)
    ranks = pb.blocks[:, 5:5 + N]
    size = sum(float(np.prod([ranks[b, q] * ranks[k, q] for q in act])) * len(terms) for (b, k, act), terms in groups.items())
    if size > 1e9 or len(groups) > 50000:
        return None
    out = {key: np.zeros((R,) + vec[key]["core"][0].shape) for key in pb.keys}
    cores = [np.stack([np.asarray(x) for x in vec[key]["core"]]) for key in pb.keys]
    gammas = {}

    def gamma(q, op, b, k):
        if (q, op, b, k) not in gammas:
            fb, fk = pb.keys[b][0][q], pb.keys[k][0][q]
            r = m.ops.table[blk[q, op, fb[0], fb[1], fk[0], fk[1]]]
            g = m.ops.data[r[9]:r[9] + r[6] * r[7] * r[8]].reshape((r[6], r[7], r[8]), order="F")
            (b0, b1), (k0, k1) = pb.keys[b][1][q], pb.keys[k][1][q]
            ub, uk = vec[pb.keys[b]]["factors"][q], vec[pb.keys[k]]["factors"][q]
            gammas[(q, op, b, k)] = np.einsum("pij,ia,jc->pac", g[:, b0:b1, k0:k1], ub, uk, optimize=True)
        return gammas[(q, op, b, k)]

    for (b, k, act), terms in groups.items():
        fk = pb.keys[k][0]
        ne = [a + c for a, c in fk]
        op = 0.0
        for i in terms:
            r = t[i]
            nb = int(r[0])
            gs = [gamma(int(r[2 + o]), int(r[6 + o]), b, k) for o in range(nb)]
            if nb == 1:
                x = gs[0][0]
            else:
                dims = [int(y) for y in r[22:22 + nb]]
                off = (int(r[26]) & 0xFFFFFFFF) | (int(r[27]) << 32)
                x = m.terms.ints[off:off + int(np.prod(dims))].reshape(dims, order="F")
                for o in range(nb):  # (p.., pairs so far) -> the next cluster's (bra, ket) pair last
                    x = np.tensordot(x, gs[o], axes=([0], [0]))
                if sum(sum(ne[:int(r[2 + o])]) for o in range(nb) if r[18 + o]) % 2:
                    x = -x
            op = op + x
        x = cores[k]
        for q in range(N):
            if q not in act:
                s = vec[pb.keys[b]]["factors"][q].T @ vec[pb.keys[k]]["factors"][q]
                x = np.moveaxis(np.tensordot(x, s, axes=([q + 1], [1])), -1, q + 1)
        n = len(act)
        y = np.tensordot(op, x, axes=([2 * a + 1 for a in range(n)], [q + 1 for q in act]))  # (bra actives, R, spectators)
        order = [n] + [0] * N
        rest = n + 1
        for q in range(N):
            if q in act:
                order[q + 1] = act.index(q)
            else:
                order[q + 1] = rest
                rest += 1
        out[pb.keys[b]] += np.transpose(y, order)
    res = np.zeros((R, pb.core_total))
    for i, key in enumerate(pb.keys):
        o, n = int(pb.blocks[i, 0]), int(pb.blocks[i, 1])
        for r in range(R):
            res[r, o:o + n] = out[key][r].reshape(-1, order="F")
    return res


def _open_exact(m, f, c, v, thresh):
    """First-order space: every (ket row, term, bra tuple) above its threshold, summed by target."""
    dev = _device()
    blk, data, table = _blocks(m)
    t, N = m.terms.table, m.N
    top = blk.shape[2]
    secs, sec = _sectors(m, f)
    fk_all = torch.from_numpy(secs.astype(np.int64)).to(dev)[torch.from_numpy(sec.astype(np.int64)).to(dev)]
    cfg = torch.from_numpy(c.astype(np.int64)).to(dev)
    x_all = torch.from_numpy(np.ascontiguousarray(v)).to(dev)
    cut = thresh / x_all.abs().max(1).values
    radix = torch.tensor([1 << (4 * j) for j in range(N)], dtype=torch.int64, device=dev)
    strides = torch.tensor([1 << (4 * j) for j in range(2 * N)], dtype=torch.int64, device=dev)
    flat = torch.from_numpy(blk.reshape(N, 24, top * top, top * top)).to(dev)
    most = [int(m.ops.table[m.ops.table[:, 0] == q, 7].max()) for q in range(N)]
    acc_key, acc_val, kept = [], [], 0
    for i in range(t.shape[0]):
        r = t[i]
        nb = int(r[0])
        act = [int(q) for q in r[2:2 + nb]]
        fb_all = fk_all + torch.from_numpy(m.terms.transfers[r[1]].reshape(-1).astype(np.int64)).to(dev)
        ok = ((fb_all >= 0) & (fb_all < top)).all(1)
        fbc = fb_all.clamp(0, top - 1)
        nb_id = fbc[:, 0::2] * top + fbc[:, 1::2]
        for q in range(N):
            ok &= flat[q, OP_H, nb_id[:, q], nb_id[:, q]] >= 0
        for o, q in enumerate(act):
            ok &= flat[q, int(r[6 + o]), nb_id[:, q], fk_all[:, 2 * q] * top + fk_all[:, 2 * q + 1]] >= 0
        rows = torch.nonzero(ok)[:, 0]
        per = max(1, (1 << 26) // int(np.prod([most[q] for q in act])))
        for p in range(0, len(rows), per):
            rr = rows[p:p + per]
            fk, ids = fk_all[rr], nb_id[rr]
            cols = []
            for o, q in enumerate(act):  # (rows, bra states, orbital index), 0 past the sector's states
                b = flat[q, int(r[6 + o]), ids[:, q], fk[:, 2 * q] * top + fk[:, 2 * q + 1]]
                tb = table[b]
                nidx = int(r[22 + o]) if nb > 1 else 1
                I = torch.arange(most[q], device=dev)
                at = tb[:, 9, None] + nidx * (I[None, :] + (tb[:, 7] * cfg[rr, q])[:, None])
                g = data[(at[:, :, None] + torch.arange(nidx, device=dev)).clamp(max=data.numel() - 1)]
                cols.append(g * (I[None, :] < tb[:, 7, None])[:, :, None])
            if nb == 1:
                x = cols[0][:, :, 0]
            else:
                dims = [int(y) for y in r[22:22 + nb]]
                off = (int(r[26]) & 0xFFFFFFFF) | (int(r[27]) << 32)
                x = torch.from_numpy(m.terms.ints[off:off + int(np.prod(dims))]).to(dev).reshape(-1, dims[0])
                x = torch.matmul(cols[0], x.T)  # (rows, b0, d1 * d2 * d3)
                for o in range(1, nb):
                    x = x.reshape(len(rr), x.shape[1], -1, dims[o])  # (rows, bras so far, rest, d)
                    x = torch.einsum("nbrd,ncd->nbcr", x, cols[o]).reshape(len(rr), x.shape[1] * cols[o].shape[1], -1)
                x = x[:, :, 0]
            hit = torch.nonzero(x.abs() > cut[rr, None])
            if len(hit) == 0:
                continue
            row = rr[hit[:, 0]]
            ne = fk_all[row][:, 0::2] + fk_all[row][:, 1::2]
            odd = sum((ne[:, :act[o]].sum(1) for o in range(nb) if r[18 + o]), torch.zeros_like(row))
            val = x[hit[:, 0], hit[:, 1]] * (1 - 2 * (odd % 2)).double()
            tuple_, new = hit[:, 1], cfg[row].clone()
            for o in range(nb - 1, -1, -1):
                new[:, act[o]] = tuple_ % most[act[o]]
                tuple_ = tuple_ // most[act[o]]
            acc_key.append(torch.stack([(fb_all[row] * strides).sum(1), (new * radix).sum(1)], 1))
            acc_val.append(val[:, None] * x_all[row])
            kept += len(row)
            if kept > 1 << 26:
                return None
    key = torch.cat(acc_key)
    val = torch.cat(acc_val)
    at = torch.argsort(key[:, 1])
    at = at[torch.argsort(key[at, 0], stable=True)]
    key = key[at]
    new = torch.ones(len(key), dtype=torch.bool, device=dev)
    new[1:] = (key[1:] != key[:-1]).any(1)
    where = torch.cumsum(new.long(), 0) - 1
    out = torch.zeros((int(where[-1]) + 1, v.shape[1]), dtype=torch.float64, device=dev)
    out.index_add_(0, where, val[at])
    return out.T


def exact(case, seed):
    kind = case["kind"]
    if kind in ("bst", "bst_set"):
        m, vec, pb = _tucker(case, seed)
        return _tucker_sigma(m, vec, pb, case["roots"])
    m = _molecule(case["system"])
    f, c, e, v = _space(case, seed)
    if kind in ("sigma", "stored"):
        return _apply(m, f, c, v).T.contiguous()
    if kind == "solve":
        h = _apply(m, f, c, v, dense=True)
        w, x = torch.linalg.eigh(0.5 * (h + h.T))
        x = x[:, :case["roots"]]
        guess = workloads.davidson_guess(len(f), case["roots"], seed=seed, lowest=[int(np.argmin(e))])
        sign = torch.sign((x * torch.from_numpy(guess).to(x.device)).sum(0))
        return {"energies": w[:case["roots"]].cpu().numpy(), "vectors": np.ascontiguousarray((x * sign).cpu().numpy())}
    return {"fock": None, "cfg": None, "coef": _open_exact(m, f, c, v, case["thresh"])}

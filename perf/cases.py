"""What this framework's speed is measured on: the calls a shell-model user's program makes, over the sizes it makes them at.

A case names a valence space (``sd`` or ``fp``), neutron and proton numbers, twice the M projection, and what is done with the
problem: a product ``Y = H X`` with a stored or an on-the-fly Hamiltonian (device buffers, or host buffers as a host eigensolver
passes them), the build of a stored Hamiltonian, a Davidson solve with the spins of its states, or a batch of small problems.
Interactions are rotationally invariant: isospin-coupled two-body matrix elements from a seeded Gaussian (1 MeV), single-particle
energies uniform below zero, plus the ``lambda J-J+`` term; vectors are seeded Gaussians.  ``exact`` evaluates the same operator
term by term on the bit patterns in 64 bits with plain torch.
"""
from __future__ import annotations

import functools
import itertools
import math

import numpy as np
import torch

import cosmo_gb300 as cg

# (l, 2j) of each orbit, and the lower end of the single-particle energies (MeV)
SPACES = {"sd": (((2, 5), (0, 1), (2, 3)), -4.0), "fp": (((3, 7), (1, 3), (3, 5), (1, 1)), -8.0)}
PRECISIONS = {"fp64": cg.CG_PREC_FP64, "fp32": cg.CG_PREC_FP32, "refine": cg.CG_PREC_REFINE}
LAMBDA = 0.5  # weight of J-J+


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # stored products, the inner call of every solve: a small nucleus, where the launch counts; a mid-shell sd nucleus in single
        # precision and in the double precision that a reference-style Davidson of block 4 uses; the largest matrix that is stored
        {"name": "product sd 3+4 fp32", "kind": "product", "space": "sd", "nv": 3, "zv": 4, "twom": 1, "precision": "fp32", "m": 8},
        {"name": "product sd 6+6 fp32", "kind": "product", "space": "sd", "nv": 6, "zv": 6, "twom": 0, "precision": "fp32", "m": 8},
        {"name": "product sd 6+6 fp64", "kind": "product", "space": "sd", "nv": 6, "zv": 6, "twom": 0, "precision": "fp64", "m": 4},
        {"name": "product fp 4+4 fp32", "kind": "product", "space": "fp", "nv": 4, "zv": 4, "twom": 0, "precision": "fp32", "m": 8},
        # a host eigensolver behind the MatrixBase seam: column-major host vectors in and out, the accurate product of a mixed matrix
        {"name": "host product sd 5+6", "kind": "host", "space": "sd", "nv": 5, "zv": 6, "twom": 1, "precision": "refine", "m": 4},
        # nothing stored: the product of problems whose matrix would not fit, or is not worth its build; an ordinary size in both
        # precisions, and a large one
        {"name": "on-the-fly fp 3+3 fp32", "kind": "otf", "space": "fp", "nv": 3, "zv": 3, "twom": 0, "precision": "fp32", "m": 8},
        {"name": "on-the-fly fp 3+4 fp64", "kind": "otf", "space": "fp", "nv": 3, "zv": 4, "twom": 1, "precision": "fp64", "m": 4},
        {"name": "on-the-fly fp 4+4 fp32", "kind": "otf", "space": "fp", "nv": 4, "zv": 4, "twom": 0, "precision": "fp32", "m": 8},
        # a new matrix and its first product, as a parameter fit or a chain of nuclei does for each interaction
        {"name": "build fp 3+4 fp32", "kind": "build", "space": "fp", "nv": 3, "zv": 4, "twom": 1, "precision": "fp32", "m": 8},
        # lowest states and their spins: an ordinary nucleus, and the largest stored one
        {"name": "solve sd 4+4", "kind": "solve", "space": "sd", "nv": 4, "zv": 4, "twom": 0, "nstates": 10},
        {"name": "solve fp 4+4", "kind": "solve", "space": "fp", "nv": 4, "zv": 4, "twom": 0, "nstates": 10},
        # many small nuclei at once (built and solved together)
        {"name": "batch of 24 sd", "kind": "batch", "space": "sd", "mix": 2024, "count": 24, "nmax": 30000, "nstates": 5},
    ]


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while (case := _draw(rng)) in known:
        pass
    return case


def _draw(rng):
    kind = rng.choices(("product", "otf", "solve", "host", "build", "batch"), (6, 6, 3, 2, 2, 1))[0]
    if kind == "batch":
        return {"kind": "batch", "space": "sd", "mix": rng.randrange(1 << 20), "count": rng.randint(4, 24),
                "nmax": int(10 ** rng.uniform(2.5, 4.4)), "nstates": rng.randint(2, 5)}
    precision = rng.choice(("fp32", "fp32", "fp64")) if kind in ("product", "otf", "build") else "refine"
    lo, hi = {"product": (60, 2.0e6), "otf": (60, 2.0e6), "host": (60, 1.0e5), "build": (400, 4.5e5), "solve": (400, 2.0e6)}[kind]
    if precision == "fp64":
        hi = min(hi, 2.0e5 if kind == "product" else 4.5e5)
    want = math.log(lo) + rng.random() * (math.log(hi) - math.log(lo))
    near = sorted((c for c in _sectors() if lo <= c[4] <= hi), key=lambda c: abs(math.log(c[4]) - want))
    space, nv, zv, twom, _ = rng.choice(near[:12])
    case = {"kind": kind, "space": space, "nv": nv, "zv": zv, "twom": twom}
    if kind == "solve":
        return case | {"nstates": rng.randint(4, 10)}
    return case | {"precision": precision, "m": rng.choice((1, 2, 3, 4, 5, 6, 7, 8, 8, 8, 10, 16))}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"kind": kind, "problems": [_problem(case["space"], nv, zv, twom, seed + 1000 * k)
                                           for k, (nv, zv, twom) in enumerate(_batch_systems(case))], "nstates": case["nstates"]}
    p = _problem(case["space"], case["nv"], case["zv"], case["twom"], seed)
    b = cg.ManyBodyStates(p)
    st = {"kind": kind, "problem": p, "basis": b}
    if kind == "solve":
        st["h"] = cg.Hamiltonian(p, b, cg.CG_PREC_FP32)
        st["h"].autotune(8)
        st["nstates"] = case["nstates"]
        return st
    prec, m = PRECISIONS[case["precision"]], case["m"]
    store = cg.CG_PREC_FP64 if case["precision"] == "fp64" else cg.CG_PREC_FP32
    st |= {"store": store, "precision": prec, "m": m}
    if kind != "build":
        st["h"] = cg.Hamiltonian(p, b, store, virtual=kind == "otf")
    if kind == "host":
        st["x"] = np.asfortranarray(_vectors(b.n, m, seed))
        return st
    # device operands: rows of m vectors padded to whole 32-byte sectors, as the library's own solver lays them out
    st["ld"] = ld = (m + 7) // 8 * 8 if store == cg.CG_PREC_FP32 else (m + 3) // 4 * 4
    x = torch.zeros(b.n, ld, dtype=torch.float32 if store == cg.CG_PREC_FP32 else torch.float64)
    x[:, :m] = torch.from_numpy(_vectors(b.n, m, seed)).to(x.dtype)
    st["x"], st["y"] = x.cuda(), torch.zeros_like(x, device="cuda")
    return st


def run(st):
    kind = st["kind"]
    if kind in ("product", "otf", "build"):
        if kind == "build":
            st["h"] = cg.Hamiltonian(st["problem"], st["basis"], st["store"])
        h, x, y = st["h"], st["x"], st["y"]
        h.spmm_device(x.data_ptr(), st["ld"], y.data_ptr(), st["ld"], st["m"], st["precision"])
        if kind == "build":
            return {"y": y, "diagonal": h.diagonal(), "entries": int(h.info.nnz_full)}
        return y
    if kind == "host":
        return st["h"].times_matrix(st["x"], st["precision"])
    if kind == "solve":
        r = cg.davidson_diagonalization(st["h"], st["nstates"], precision=cg.CG_PREC_FP32, tol_resid=1e-5, block=min(8, st["nstates"]),
                                        lim=96, keep=32, algorithm=1, precond=1, switch_resid=3e-5, refine_lim=32, refine_keep=16)
        jj, _ = cg.jt_expectations(st["basis"], r.vecs)
        twoj = np.array([cg.jj_spin(v, int(st["problem"].info.twom)) for v in jj])
        return {"eig": r.eig, "twoj": twoj, "converged": int((r.resid <= 1e-5).sum())}
    eig, _, nconv, _ = cg.Batch(st["problems"]).solve(st["nstates"])
    return {"eig": eig, "converged": nconv}


def work(case):
    """Vectors in and out and the operator's terms; two operations for each nonzero element of H and vector.  A solve cannot do without
    about ten products of its block of vectors, a batch without as many of each problem's, a build without writing its elements."""
    if case["kind"] == "batch":
        both = [_work_of(case["space"], *s, 8, 4) for s in _batch_systems(case)]
        return {"bytes": 10 * sum(w[0] for w in both), "flops": 10 * sum(w[1] for w in both)}
    m = case.get("m", 8)
    size = 4 if case.get("precision") == "fp32" or case["kind"] == "solve" else 8
    nbytes, flops, nnz = _work_of(case["space"], case["nv"], case["zv"], case["twom"], m, size)
    times = 10 if case["kind"] == "solve" else 1
    stored = 12 * nnz if case["kind"] == "build" else 0
    return {"bytes": times * nbytes + stored, "flops": times * flops}


def exact(case, seed):
    kind, dev = case["kind"], "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "batch":
        systems = _batch_systems(case)
        if sum(_dimension(case["space"], *s) for s in systems) > 150000:
            return None
        eig = np.full((case["count"], case["nstates"]), np.nan)
        for k, (nv, zv, twom) in enumerate(systems):
            e = _lowest(_Plain(case["space"], nv, zv, twom, seed + 1000 * k, dev), case["nstates"])
            eig[k, :len(e)] = e
        return {"eig": eig, "converged": None}
    n = _dimension(case["space"], case["nv"], case["zv"], case["twom"])
    if kind == "solve":
        if n > 60000:
            return None
        op = _Plain(case["space"], case["nv"], case["zv"], case["twom"], seed, dev)
        return {"eig": _lowest(op, case["nstates"]), "twoj": None, "converged": None}
    m = case["m"]
    if n * m > 4e7:
        return None
    op = _Plain(case["space"], case["nv"], case["zv"], case["twom"], seed, dev)
    x = torch.from_numpy(_vectors(n, m, seed)).to(dev)
    if kind != "host" and case["precision"] == "fp32":
        x = x.float().double()
    y, diag = op.apply(x)
    if kind == "host":
        return y.cpu().numpy()
    ld = (m + 7) // 8 * 8 if case["precision"] != "fp64" else (m + 3) // 4 * 4
    y = torch.nn.functional.pad(y, (0, ld - m))
    return {"y": y, "diagonal": diag, "entries": None} if kind == "build" else y


# ------------------------------------------------------------------------------------------------ inputs
def _vectors(n, m, seed):
    return np.random.default_rng(seed).standard_normal((n, m))


def _batch_systems(case):
    """A ~ U{2..12} nucleons, Z ~ U, the lowest or next M: the mix of nuclei that a survey of a shell has, up to nmax states."""
    rng, out = np.random.default_rng(case["mix"]), []
    while len(out) < case["count"]:
        a = int(rng.integers(2, 13))
        z = int(rng.integers(0, a + 1))
        twom = 2 * int(rng.integers(0, 2)) + (a & 1)
        if 1 <= _dimension(case["space"], a - z, z, twom) <= case["nmax"]:
            out.append((a - z, z, twom))
    return out


@functools.lru_cache(None)
def _states(space):
    """(orbit, l, 2j, 2m) of the m-states of one species."""
    return [(o, l, j2, m2) for o, (l, j2) in enumerate(SPACES[space][0]) for m2 in range(-j2, j2 + 1, 2)]


def _f(n):
    return math.factorial(n)


@functools.lru_cache(None)
def _cg(j1, m1, j2, m2, j, m):
    """Clebsch-Gordan coefficient, arguments doubled (Racah's closed form)."""
    if m1 + m2 != m or not abs(j1 - j2) <= j <= j1 + j2 or abs(m) > j:
        return 0.0
    a, b, c = (j1 + j2 - j) // 2, (j1 - m1) // 2, (j2 + m2) // 2
    d, e = (j - j2 + m1) // 2, (j - j1 - m2) // 2
    s = sum((-1) ** k / (_f(k) * _f(a - k) * _f(b - k) * _f(c - k) * _f(d + k) * _f(e + k))
            for k in range(max(0, -d, -e), min(a, b, c) + 1))
    return s * math.sqrt((j + 1) * _f(a) * _f((j + j1 - j2) // 2) * _f((j - j1 + j2) // 2) / _f((j1 + j2 + j) // 2 + 1)
                         * _f((j1 + m1) // 2) * _f(b) * _f(c) * _f((j2 - m2) // 2) * _f((j + m) // 2) * _f((j - m) // 2))


@functools.lru_cache(None)
def _coupling(space):
    """m-scheme pairs, the coupled states (a <= b, J, T, M, Tz) and the real matrix between them, and J+ of one particle."""
    one = _states(space)
    sps = [s + (t,) for t in (1, -1) for s in one]  # neutrons, then protons
    ns = len(sps)
    pairs = list(itertools.combinations(range(ns), 2))
    orbits = SPACES[space][0]
    coupled, rows = {}, []
    for r, (x, y) in enumerate(pairs):
        (ox, _, jx, mx, tx), (oy, _, jy, my, ty) = sps[x], sps[y]
        a, b = min(ox, oy), max(ox, oy)
        for J2 in range(abs(jx - jy), jx + jy + 1, 2):
            for T2 in (0, 2):
                v = 0.0
                if (ox, oy) == (a, b):
                    v += _cg(jx, mx, jy, my, J2, mx + my) * _cg(1, tx, 1, ty, T2, tx + ty)
                if (oy, ox) == (a, b):
                    v -= _cg(jy, my, jx, mx, J2, mx + my) * _cg(1, ty, 1, tx, T2, tx + ty)
                if a == b:
                    v /= math.sqrt(2)
                if abs(v) > 1e-12:
                    c = coupled.setdefault((a, b, J2, T2, mx + my, tx + ty), len(coupled))
                    rows.append((r, c, v))
    U = np.zeros((len(pairs), len(coupled)))
    for r, c, v in rows:
        U[r, c] = v
    P = np.zeros((ns, ns))  # P[f, i] = <f| J+ |i>
    for i, (o, _, j2, m2, t) in enumerate(sps):
        for f, (o2, _, _, n2, t2) in enumerate(sps):
            if o2 == o and t2 == t and n2 == m2 + 2:
                P[f, i] = math.sqrt((j2 - m2) * (j2 + m2 + 2)) / 2
    keys = list(coupled)
    labels = {}  # (orbit pair parity, J, T) channels and the position of each orbit pair in them
    chan = np.array([labels.setdefault(((orbits[a][0] + orbits[b][0]) & 1, J, T), len(labels)) for a, b, J, T, _, _ in keys])
    norb = len(orbits)
    ab = np.array([a * norb + b for a, b, *_ in keys])
    mt = np.array([m * 100 + t for *_, m, t in keys])
    return sps, pairs, U, chan, ab, mt, len(labels), norb, P


@functools.lru_cache(4)
def _terms(space, seed):
    """s.p. table and forward-ordered one- and two-body terms of a seeded interaction plus LAMBDA J-J+."""
    sps, pairs, U, chan, ab, mt, nchan, norb, P = _coupling(space)
    rng = np.random.default_rng(seed)
    spe = rng.uniform(SPACES[space][1], 0.0, norb)
    g = rng.standard_normal((nchan, norb * norb, norb * norb))
    g = np.triu(g) + np.triu(g, 1).transpose(0, 2, 1)
    Vc = np.where((chan[:, None] == chan[None]) & (mt[:, None] == mt[None]), g[chan[:, None], ab[:, None], ab[None]], 0.0)
    V = U @ Vc @ U.T
    i, j = np.array(pairs).T
    A, B, C, D = P[np.ix_(i, i)], P[np.ix_(j, j)], P[np.ix_(i, j)], P[np.ix_(j, i)]
    V += LAMBDA * (A * B.T - C * C.T - D * D.T + B * A.T)
    V = (V + V.T) / 2
    e = np.diag([spe[s[0]] for s in sps]) + LAMBDA * (P.T @ P)
    table = np.array([(o, 0, l, j2, m2, 1, t, l & 1) for o, l, j2, m2, t in sps], dtype=np.int32)
    r, c = np.nonzero(np.triu(np.abs(V) > 1e-13))
    p = np.array(pairs, dtype=np.int32)
    k1 = np.argwhere(np.triu(e) != 0)
    return table, k1.astype(np.int32), e[k1[:, 0], k1[:, 1]], np.hstack([p[r], p[c]]), V[r, c]


def _parity(space, a):
    return (SPACES[space][0][0][0] * a) & 1


def _problem(space, nv, zv, twom, seed):
    table, k1, v1, k2, v2 = _terms(space, seed)
    return cg.Problem.from_terms(table, len(table) // 2, nv, zv, twom, _parity(space, nv + zv), k1, v1, k2, v2)


# ------------------------------------------------------------------------------------------------ counting
@functools.lru_cache(None)
def _species(space, k):
    """Occupations (configurations x m-states) of k particles in lexicographic order, and their 2M."""
    one = _states(space)
    conf = np.array(list(itertools.combinations(range(len(one)), k)), dtype=np.int64).reshape(math.comb(len(one), k), k)
    occ = np.zeros((len(conf), len(one)), dtype=np.int64)
    np.put_along_axis(occ, conf, 1, axis=1)
    return occ, occ @ np.array([s[3] for s in one])


def _dimension(space, nv, zv, twom):
    n, p = (np.bincount(_species(space, k)[1] + 200, minlength=401) for k in (nv, zv))
    return int(sum(n[i] * p[400 + twom - i] for i in np.flatnonzero(n) if 0 <= 400 + twom - i <= 400))


@functools.lru_cache(None)
def _moves(space, k):
    """{2M: (configurations, {change of 2m: one-particle moves}, two-particle moves that keep 2M)}."""
    occ, M = _species(space, k)
    m2 = np.array([s[3] for s in _states(space)])
    ms = np.arange(m2.min(), m2.max() + 1, 2)
    in_m = (m2[:, None] == ms[None]).astype(np.int64)
    full, hole = occ @ in_m, (1 - occ) @ in_m
    one = np.stack([(full[:, max(0, -d):len(ms) - max(0, d)] * hole[:, max(0, d):len(ms) + min(0, d)]).sum(1)
                    for d in range(-len(ms) + 1, len(ms))], 1)

    def by_sum(c):
        out = np.zeros((len(c), 2 * len(ms) - 1), dtype=np.int64)
        for i in range(len(ms)):
            out[:, 2 * i] += c[:, i] * (c[:, i] - 1) // 2
            for j in range(i):
                out[:, i + j] += c[:, i] * c[:, j]
        return out

    two = (by_sum(full) * by_sum(hole)).sum(1)
    return {int(m): (int((M == m).sum()), one[M == m].sum(0), int(two[M == m].sum())) for m in np.unique(M)}


@functools.lru_cache(None)
def _elements(space, nv, zv, twom):
    """Pairs of determinants that differ by at most two particle moves and the same M."""
    n, p, total = _moves(space, nv), _moves(space, zv), 0
    for m, (cn, on, tn) in n.items():
        if twom - m in p:
            cp, op, tp = p[twom - m]
            mid = len(on) // 2
            total += cn * cp + tn * cp + cn * tp + cn * int(op[mid]) + int(on[mid]) * cp + int((on * op[::-1]).sum())
    return total


def _work_of(space, nv, zv, twom, m, size):
    n, nnz = _dimension(space, nv, zv, twom), _elements(space, nv, zv, twom)
    return 2 * n * m * size + 80000, 2 * nnz * m, nnz


@functools.lru_cache(None)
def _sectors():
    """(space, nv, zv, 2M, dimension) of every M sector that a draw may take."""
    out = []
    for space, most in (("sd", 12), ("fp", 8)):
        norb = len(_states(space))
        for nv, zv in itertools.product(range(min(most, norb - 1) + 1), repeat=2):
            if nv + zv < 2 or max(math.comb(norb, nv), math.comb(norb, zv)) > 20000:
                continue
            for twom in range((nv + zv) & 1, 5, 2):
                n = _dimension(space, nv, zv, twom)
                if 60 <= n <= 2.0e6:
                    out.append((space, nv, zv, twom, n))
    return out


# ------------------------------------------------------------------------------------------------ plain evaluation in 64 bits
class _Plain:
    """The operator on the determinants' bit patterns, one term at a time."""

    def __init__(self, space, nv, zv, twom, seed, dev):
        self.table, self.k1, self.v1, self.k2, self.v2 = _terms(space, seed)
        self.no = no = len(self.table) // 2
        (on, mn), (op, mp) = _species(space, nv), _species(space, zv)
        bits = np.int64(1) << np.arange(no, dtype=np.int64)
        nmask, pmask = on @ bits, op @ bits
        rank, classes = np.zeros(1 << no, np.int64), {}
        for m in np.unique(mp):
            classes[int(m)] = pmask[mp == m]
            rank[classes[int(m)]] = np.arange(len(classes[int(m)]))
        start, masks, at = np.full(1 << no, -1, np.int64), [], 0
        for nu, m in zip(nmask, mn):
            c = classes.get(twom - int(m))
            if c is not None:
                start[nu] = at
                at += len(c)
                masks.append(nu | (c << no))
        parity = np.zeros(1 << no, np.int64)
        for b in range(no):
            parity ^= (np.arange(1 << no) >> b) & 1
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        self.mask, self.start, self.rank, self.par = put(np.concatenate(masks)), put(start), put(rank), put(parity)
        self.n = at

    def elements(self):
        """(rows of the bra, rows of the ket, values) of each forward term."""
        low = (1 << self.no) - 1
        for keys, vals, k in ((self.k1, self.v1, 1), (self.k2, self.v2, 2)):
            before, src = None, None
            for q, v in zip(keys.tolist(), vals.tolist()):
                ann, cre = sum(1 << b for b in q[:k]), sum(1 << b for b in q[k:])
                if ann != before:
                    before, has = ann, torch.nonzero((self.mask & ann) == ann).flatten()
                    rest = self.mask[has] & ~ann
                free = torch.nonzero((rest & cre) == 0).flatten()
                src, core = has[free], rest[free]
                to = core | cre
                dst = self.start[to & low] + self.rank[to >> self.no]
                f = 0
                for b in q:
                    f ^= (1 << b) - 1
                s = core & f
                sign = 1.0 - 2.0 * (self.par[s & low] ^ self.par[s >> self.no]).double()
                yield src, dst, sign * v, ann == cre

    def apply(self, x):
        y, diag = torch.zeros_like(x), torch.zeros(self.n, dtype=x.dtype, device=x.device)
        for src, dst, v, same in self.elements():
            if same:
                diag.index_add_(0, src, v)
            else:
                y.index_add_(0, dst, v[:, None] * x[src])
                y.index_add_(0, src, v[:, None] * x[dst])
        return y + diag[:, None] * x, diag

    def matrix(self):
        rows, cols, vals = [], [], []
        for src, dst, v, same in self.elements():
            rows += [dst] if same else [dst, src]
            cols += [src] if same else [src, dst]
            vals += [v] if same else [v, v]
        ij = torch.stack([torch.cat(rows), torch.cat(cols)])
        return torch.sparse_coo_tensor(ij, torch.cat(vals), (self.n, self.n)).coalesce().to_sparse_csr()


def _lowest(op, k):
    """The k lowest eigenvalues: dense, or Lanczos with full reorthogonalisation until they stand still."""
    A = op.matrix()
    if op.n <= 1500:
        return np.linalg.eigvalsh(A.to_dense().cpu().numpy())[:k]
    g = torch.Generator().manual_seed(1)
    q = torch.randn(op.n, generator=g, dtype=torch.float64).to(op.mask.device)
    Q = torch.zeros(min(op.n, 800), op.n, dtype=torch.float64, device=q.device)
    Q[0] = q / q.norm()
    alpha, beta, old = [], [], None
    for i in range(Q.shape[0]):
        w = A @ Q[i]
        alpha.append(float(Q[i] @ w))
        for _ in range(2):
            w -= Q[:i + 1].T @ (Q[:i + 1] @ w)
        if i % 40 == 39 or i + 1 == Q.shape[0]:
            e = np.linalg.eigvalsh(np.diag(alpha) + np.diag(beta, 1) + np.diag(beta, -1))[:k]
            if old is not None and np.abs(e - old).max() < 1e-11 or i + 1 == Q.shape[0]:
                return e
            old = e
        beta.append(float(w.norm()))
        Q[i + 1] = w / beta[-1]

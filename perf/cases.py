"""Workloads of the Fock-build engine: what a program that uses the framework
has it do, over the sizes, basis sets, spin cases and precisions it serves.

  fock   one Fock build on a job that the program keeps for its whole SCF (the
         density in, G or J/Ka/Kb out), from host arrays or device buffers
  eri    the unique two-electron integrals of a small molecule (ERI_GPU)
  scf    a whole self-consistent field from atoms and a basis-set name
  scan   a batch of points of a bond-length scan, warm-started in chains

Every case is a molecule of hartree_fock_cpp_gb300.workloads with its atoms
moved by 0.02 bohr (the seed's), so that another seed is another molecule of
the same size.  Fock builds get the density of the bare-nucleus Hamiltonian
with a smeared Fermi level, which is what the first cycle of an SCF sees.

`exact` evaluates the same McMurchie-Davidson integrals in 64 bits with torch
tensor operations from the basis-set tables alone.
"""
import csv
import functools
import math
import os

import numpy as np
import torch

import hartree_fock_cpp_gb300 as H
from hartree_fock_cpp_gb300 import workloads as W

DEVICE = "cuda"
THRESHOLD = 1e-8
SCF = dict(epsilon=1e-7, energy_threshold=1e-8, max_it=200)
EXACT_FOCK_K, EXACT_ERI_K, EXACT_SCF_K = 300, 60, 130


def listed():
    return [
        # the smallest call: one build of a 7-function molecule, all latency and launches
        dict(name="fock_water_sto3g", do="fock", mol="water", n=1, basis="STO-3G", spin="rhf", precision="fp64", tau=0.0,
             host=True),
        # a small molecule in a large basis: f functions, open-shell J/Ka/Kb, host arrays
        dict(name="fock_water_ccpvtz_uhf", do="fock", mol="water", n=1, basis="cc-pVTZ", spin="uhf", precision="fp64",
             tau=0.0, host=True),
        # the headline workload's build: benzene / cc-pVDZ, 23 of these make a solve
        dict(name="fock_benzene_ccpvdz", do="fock", mol="benzene", n=6, basis="cc-pVDZ", spin="rhf", precision="fp64",
             tau=0.0, host=False),
        # the mixed-precision workload's molecule, in FP64 and in mixed precision at the cut its autotuner picks
        dict(name="fock_decane_631gs", do="fock", mol="alkane", n=10, basis="6-31G*", spin="rhf", precision="fp64",
             tau=0.0, host=False),
        dict(name="fock_decane_631gs_mixed", do="fock", mol="alkane", n=10, basis="6-31G*", spin="rhf",
             precision="mixed", tau=0.1, host=False),
        # the scan workload's molecule: long contractions of third-row atoms, f functions
        dict(name="fock_nacl_ccpvtz", do="fock", mol="nacl", n=1, basis="cc-pVTZ", spin="rhf", precision="fp64", tau=0.0,
             host=False),
        # a served request of ordinary size: an open-shell doublet, mixed precision
        dict(name="fock_tree7_ccpvdz_uhf_mixed", do="fock", mol="tree", n=7, basis="cc-pVDZ", spin="uhf",
             precision="mixed", tau=0.03, host=False),
        # a large served request
        dict(name="fock_tree16_631gs_mixed", do="fock", mol="tree", n=16, basis="6-31G*", spin="rhf", precision="mixed",
             tau=0.03, host=False),
        # the integrals themselves, in the reference's packed order
        dict(name="eri_water_631gs", do="eri", mol="water", n=1, basis="6-31G*"),
        # whole solves: the headline one, and a small open-shell request
        dict(name="scf_benzene_ccpvdz", do="scf", mol="benzene", n=6, basis="cc-pVDZ", spin="rhf", precision="fp64",
             tau=0.0),
        dict(name="scf_tree2_631gs_uhf", do="scf", mol="tree", n=2, basis="6-31G*", spin="uhf", precision="fp64", tau=0.0),
        # a piece of a bond-length scan on the batched engine
        dict(name="scan_water_ccpvtz", do="scan", mol="water_scan", n=8, chain=4, basis="cc-pVTZ"),
    ]


def draw(rng):
    # Fock builds are nearly all of what the framework does
    kind = rng.choice(["fock"] * 7 + ["eri", "scf", "scan"])
    if kind == "eri":
        return dict(do="eri", mol=rng.choice(["water", "tree"]), n=1, basis=rng.choice(["STO-3G", "6-31G", "6-31G*"]),
                    shift=round(rng.uniform(0.0, 0.3), 3))
    if kind == "scan":
        n = rng.randint(2, 8)
        return dict(do="scan", mol="water_scan", n=n, chain=rng.randint(1, n), basis=rng.choice(["6-31G*", "cc-pVDZ",
                    "cc-pVTZ"]), shift=round(rng.uniform(0.0, 0.3), 3))
    if kind == "scf":
        precision = rng.choice(["fp64", "mixed"])
        return dict(do="scf", mol="alkane", n=rng.randint(2, 4), basis=rng.choice(["STO-3G", "6-31G*", "cc-pVDZ"]),
                    spin="rhf", precision=precision, tau=0.03 if precision == "mixed" else 0.0,
                    shift=round(rng.uniform(0.0, 0.3), 3))
    mol = rng.choice(["water", "benzene", "alkane", "alkane", "nacl", "tree", "tree", "tree"])
    basis = rng.choice(["STO-3G", "6-31G*", "6-31G*", "cc-pVDZ", "cc-pVDZ", "cc-pVTZ"])
    if mol == "benzene" and basis == "cc-pVTZ":
        basis = "cc-pVDZ"
    most = {"STO-3G": 24, "6-31G*": 14, "cc-pVDZ": 8, "cc-pVTZ": 3}[basis]
    least = 2 if mol == "alkane" else 1
    n = int(round(math.exp(rng.uniform(math.log(least), math.log(most))))) if mol in ("alkane", "tree") else 1
    precision = rng.choice(["fp64", "fp64", "mixed"])
    return dict(do="fock", mol=mol, n=n, basis=basis, spin=rng.choice(["rhf", "rhf", "uhf"]), precision=precision,
                tau=round(10 ** rng.uniform(-3.0, -1.0), 5) if precision == "mixed" else 0.0, host=rng.random() < 0.5,
                shift=round(rng.uniform(0.0, 0.3), 3))


def _molecules(case, seed):
    """The case's molecule (a list of them for a scan), its atoms moved by the
    seed; `shift` stretches a drawn case's molecule by up to 3%."""
    name, n = case["mol"], case["n"]
    if name == "water":
        mols = [W.water()]
    elif name == "benzene":
        mols = [W.benzene()]
    elif name == "alkane":
        mols = [W.n_decane(noise=0.0, n_carbon=n)]
    elif name == "nacl":
        mols = [W.nacl_scan(64)[24]]
    elif name == "water_scan":
        mols = W.water_scan(64)[8:8 + 4 * n:4]
    else:
        # another tree of the same heavy-atom count is another workload: the
        # count fixes the tree, the seed moves its atoms
        grow = np.random.default_rng(1000 + n)
        mols = [None]
        while mols[0] is None:
            mols = [W.random_molecule(grow, n)]
        if case.get("spin") == "uhf":
            last = max(i for i, a in enumerate(mols[0]) if a[0] == "H")
            del mols[0][last]
    rng = np.random.default_rng(seed)
    scale = 1.0 + 0.1 * case.get("shift", 0.0)
    moved = rng.normal(0.0, 0.02, size=(len(mols[0]), 3))
    return [[(s, tuple(float(scale * x + d) for x, d in zip(p, moved[k]))) for k, (s, p) in enumerate(m)] for m in mols]


def _spin(case, mol):
    ne = W.n_electrons(mol)
    return ((ne + 1) // 2, ne // 2) if case.get("spin") == "uhf" and ne % 2 else (
        (ne // 2 + 1, ne // 2 - 1) if case.get("spin") == "uhf" else (ne // 2, ne - ne // 2))


def _precision(case):
    return H.HFX_PREC_MIXED if case.get("precision") == "mixed" else H.HFX_PREC_FP64


def _densities(case, mol):
    """Densities of the bare-nucleus Hamiltonian, occupations smeared over 0.5 Eh."""
    S, T, V = (x.cpu().numpy() for x in _Integrals(mol, case["basis"]).one_electron())
    s, U = np.linalg.eigh(S)
    X = U / np.sqrt(s)
    e, C = np.linalg.eigh(X.T @ (T + V) @ X)
    out = []
    for n in _spin(case, mol):
        lo, hi = e[0] - 50.0, e[-1] + 50.0
        for _ in range(200):
            mu = 0.5 * (lo + hi)
            f = 0.5 * (1.0 - np.tanh((e - mu) / 1.0))
            lo, hi = (mu, hi) if f.sum() < n else (lo, mu)
        B = (X @ C) * np.sqrt(f)
        out.append(B @ B.T)
    return out


def prepare(case, seed):
    mols = _molecules(case, seed)
    st = dict(case=case, mols=mols)
    if case["do"] == "eri":
        st["basis"] = H.basis_construction(mols[0], case["basis"])
    if case["do"] != "fock":
        return st
    Pa, Pb = _densities(case, mols[0])
    st["job"] = H.FockBuilder(config=mols[0], basis_set=case["basis"], screening_threshold=THRESHOLD,
                              precision=_precision(case), fp32_threshold=case["tau"])
    dens = [Pa + Pb] if case["spin"] == "rhf" else [Pa, Pb]
    st["in"] = dens if case["host"] else [torch.from_numpy(d).to(DEVICE) for d in dens]
    if not case["host"]:
        st["out"] = [torch.empty_like(st["in"][0]) for _ in range(1 if case["spin"] == "rhf" else 3)]
    return st


def run(st):
    case = st["case"]
    if case["do"] == "fock":
        if case["host"]:
            return st["job"].repulsion_matrix(*st["in"]) if case["spin"] == "rhf" else list(
                st["job"].coulomb_exchange(*st["in"]))
        ptrs = [t.data_ptr() for t in st["in"] + st["out"]]
        (st["job"].repulsion_matrix_device if case["spin"] == "rhf" else st["job"].coulomb_exchange_device)(*ptrs)
        return st["out"]
    if case["do"] == "eri":
        return H.ERI_GPU(st["basis"], THRESHOLD)
    if case["do"] == "scan":
        res, _ = H.batch_scf([(m, case["basis"]) for m in st["mols"]], warm_chain=case["chain"], **SCF)
        return np.array([r["E_tot"] for r in res])
    mol = st["mols"][0]
    kw = dict(precision=_precision(case), fp32_threshold=case["tau"], **SCF)
    if case["spin"] == "uhf":
        r = H.uhf_diis(mol, case["basis"], spin_occ=_spin(case, mol), **kw)
        return [np.array(r["E_tot"]), r["Pa"], r["Pb"], r["Ea"], r["Eb"]]
    r = H.rhf_diis(mol, case["basis"], **kw)
    return [np.array(r["E_tot"]), r["density"], r["mo_energy"]]


def work(case):
    """Flops: the primitive quartets (distinct exponents only) of the shell
    quartets that pass the Schwarz test, each its Boys function, Hermite
    recursion and transforms, and six multiply-adds per unique integral; for a
    whole solve, 12 builds.  Bytes: the matrices in and out."""
    mols = _molecules(case, 0)
    ints = _Integrals(mols[0], case["basis"])
    flops = ints.build_flops(THRESHOLD)
    K = ints.K
    if case["do"] == "eri":
        P = K * (K + 1) // 2
        return dict(bytes=8 * P * (P + 1) // 2, flops=flops)
    if case["do"] == "scan":
        return dict(bytes=8 * len(mols), flops=12 * len(mols) * flops)
    if case["do"] == "scf":
        return dict(bytes=8 * K * K, flops=12 * flops)
    return dict(bytes=8 * K * K * (2 if case["spin"] == "rhf" else 5), flops=flops)


def exact(case, seed):
    mols = _molecules(case, seed)
    if case["do"] == "scan":
        if _Integrals(mols[0], case["basis"]).K > 70:
            return None
        return torch.stack([_scf(m, case)[0] for m in mols])
    ints = _Integrals(mols[0], case["basis"])
    if ints.K > {"fock": EXACT_FOCK_K, "eri": EXACT_ERI_K, "scf": EXACT_SCF_K}[case["do"]]:
        return None
    if case["do"] == "scf":
        got = _scf(mols[0], case)
        if got is None:
            return None
        E, P, e = got
        return [E, P[0], e[0]] if case["spin"] == "rhf" else [E, P[0], P[1], e[0], e[1]]
    M = ints.two_electron(THRESHOLD)
    if case["do"] == "eri":
        i, j = torch.tril_indices(ints.K, ints.K, device=DEVICE)
        row = ints.index[i, j]
        p, q = torch.tril_indices(len(row), len(row), device=DEVICE)
        return M[row[p], row[q]]
    P = [torch.from_numpy(d).to(DEVICE) for d in _densities(case, mols[0])]
    if case["spin"] == "rhf":
        J, K = ints.coulomb(M, P[0] + P[1]), ints.exchange(M, P[0] + P[1])
        G = J - 0.5 * K
        return G if case["host"] else [G]
    return [ints.coulomb(M, P[0] + P[1]), ints.exchange(M, P[0]), ints.exchange(M, P[1])]


# ---- the integrals in 64 bits, as plain tensor operations --------------------


def _nherm(L):
    return (L + 1) * (L + 2) * (L + 3) // 6


@functools.lru_cache(maxsize=None)
def _hermite_list(L):
    return [(t, u, s - t - u) for s in range(L + 1) for t in range(s + 1) for u in range(s - t + 1)]


@functools.lru_cache(maxsize=None)
def _hermite_place(L):
    return {h: i for i, h in enumerate(_hermite_list(L))}


@functools.lru_cache(maxsize=None)
def _hermite_steps(L):
    """For every Hermite index above 0: the axis, the two indices it follows from and the second's factor."""
    place, axis, one, two, fac = _hermite_place(L), [], [], [], []
    for h in _hermite_list(L)[1:]:
        d = 0 if h[0] else 1 if h[1] else 2
        low = [h[k] - (k == d) for k in range(3)]
        lower = [low[k] - (k == d) for k in range(3)]
        axis.append(d)
        one.append(place[tuple(low)])
        two.append(place[tuple(lower)] if low[d] else 0)
        fac.append(float(low[d]))
    as_long = lambda v: torch.tensor(v, dtype=torch.long, device=DEVICE)  # noqa: E731
    return as_long(axis), as_long(one), as_long(two), torch.tensor(fac, dtype=torch.float64, device=DEVICE)


def _boys(L, T):
    """F_0..F_L(T): the ascending series and downward recursion below T = 40, the
    error function (1 there) and upward recursion above."""
    F = torch.empty((L + 1,) + T.shape, dtype=T.dtype, device=T.device)
    e = torch.exp(-T)
    low = torch.clamp(T, max=40.0)
    term = torch.full_like(T, 1.0 / (2 * L + 1))
    total = term.clone()
    for i in range(1, 160):
        term = term * (low * (2.0 / (2 * L + 2 * i + 1)))
        total += term
    F[L] = torch.exp(-low) * total
    for m in range(L - 1, -1, -1):
        F[m] = (2.0 * T * F[m + 1] + e) / (2 * m + 1)
    far = T > 40.0
    if bool(far.any()):
        Tf, ef = T[far], e[far]
        v = 0.5 * torch.sqrt(math.pi / Tf)
        for m in range(L + 1):
            F[m][far] = v
            v = ((2 * m + 1) * v - ef) / (2.0 * Tf)
    return F


def _hermite_coulomb(L, a, X, Y, Z):
    """R_tuv of exponent a at (X, Y, Z), first index the Hermite one."""
    F = _boys(L, a * (X * X + Y * Y + Z * Z))
    axis, one, two, fac = _hermite_steps(L)
    D = torch.stack([X, Y, Z])
    shape = (-1,) + (1,) * X.dim()
    R = ((-2.0 * a) ** L * F[L])[None]
    for m in range(L - 1, -1, -1):
        n = _nherm(L - m) - 1
        up = D[axis[:n]] * R[one[:n]] + fac[:n].reshape(shape) * R[two[:n]]
        R = torch.cat([((-2.0 * a) ** m * F[m])[None], up])
    return R


def _double_factorial(n):
    return 1 if n <= 0 else n * _double_factorial(n - 2)


def _components(L):
    return [(a, b, L - a - b) for a in range(L + 1) for b in range(L - a + 1)]


@functools.lru_cache(maxsize=None)
def _element(basis, el):
    shells = {}
    with open(os.path.join(H.BASIS_PATH, basis, el + ".csv")) as f:
        for r in csv.DictReader(f):
            L, prims = shells.setdefault(int(r["shell_id"]), ("SPDF".index(r["L"].strip()), []))
            prims.append((float(r["exponent"]), float(r["coefficient"])))
    return [shells[k] for k in sorted(shells)]


class _Group:
    """Shell pairs of one (L, primitive count) combination: p and P are
    [pair, prim], E is [pair, prim, component pair, Hermite index]."""


class _Integrals:
    def __init__(self, mol, basis):
        self.mol, self.shells, self.K = mol, [], 0
        for sym, xyz in mol:
            for L, prims in _element(basis, sym):
                self.shells.append((L, np.array(xyz), np.array(prims), self.K))
                self.K += len(_components(L))
        kinds = {}
        for s, sh in enumerate(self.shells):
            kinds.setdefault((sh[0], len(sh[2])), []).append(s)
        order = sorted(kinds, reverse=True)
        self.groups, self.n2 = [], 0
        rows, cols, weights = [], [], []
        for x, ka in enumerate(order):
            for kb in order[x:]:
                pairs = [(a, b) for a in kinds[ka] for b in kinds[kb] if ka != kb or a >= b]
                g = self._group(ka, kb, pairs)
                g.at = self.n2
                self.n2 += g.n * g.nab
                self.groups.append(g)
                for a, b in pairs:
                    for i in range(len(_components(ka[0]))):
                        for j in range(len(_components(kb[0]))):
                            rows.append(self.shells[a][3] + i)
                            cols.append(self.shells[b][3] + j)
                            weights.append(1.0 if a == b else 2.0)
        as_cuda = lambda v, t: torch.tensor(v, dtype=t, device=DEVICE)  # noqa: E731
        self.rows, self.cols = as_cuda(rows, torch.long), as_cuda(cols, torch.long)
        self.weights = as_cuda(weights, torch.float64)
        self.index = torch.zeros((self.K, self.K), dtype=torch.long, device=DEVICE)
        every = torch.arange(self.n2, device=DEVICE)
        self.index[self.cols, self.rows] = every
        self.index[self.rows, self.cols] = every

    def _group(self, ka, kb, pairs):
        la, lb = ka[0], kb[0]
        g = _Group()
        g.la, g.lb, g.n, g.q, g.L = la, lb, len(pairs), ka[1] * kb[1], la + lb
        ca, cb = _components(la), _components(lb)
        g.nab, g.nh, g.pairs = len(ca) * len(cb), _nherm(la + lb), pairs
        t = lambda v: torch.tensor(np.array(v), dtype=torch.float64, device=DEVICE)  # noqa: E731
        A, B = t([self.shells[a][1] for a, _ in pairs]), t([self.shells[b][1] for _, b in pairs])
        pa, pb = t([self.shells[a][2] for a, _ in pairs]), t([self.shells[b][2] for _, b in pairs])
        n = g.n
        al = pa[:, :, None, 0].expand(n, ka[1], kb[1]).reshape(n, -1)
        be = pb[:, None, :, 0].expand(n, ka[1], kb[1]).reshape(n, -1)
        w = (pa[:, :, None, 1] * pb[:, None, :, 1]).reshape(n, -1)
        g.al, g.be, g.w, g.A, g.B = al, be, w, A, B
        g.p = al + be
        g.P = (al[..., None] * A[:, None] + be[..., None] * B[:, None]) / g.p[..., None]
        E1 = [self._hermite_1d(la, lb, al, be, A[:, None, d], B[:, None, d], g.P[..., d]) for d in range(3)]
        g.E1 = E1
        norm = lambda x, c: (2.0 * x / math.pi) ** 0.75 * torch.sqrt((4.0 * x) ** sum(c) / (  # noqa: E731
            _double_factorial(2 * c[0] - 1) * _double_factorial(2 * c[1] - 1) * _double_factorial(2 * c[2] - 1)))
        g.norms = [(norm(al, a), norm(be, b), a, b) for a in ca for b in cb]
        g.E = torch.zeros((n, g.q, g.nab, g.nh), dtype=torch.float64, device=DEVICE)
        for k, (na, nb, a, b) in enumerate(g.norms):
            for h, (tt, u, v) in enumerate(_hermite_list(g.L)):
                if tt <= a[0] + b[0] and u <= a[1] + b[1] and v <= a[2] + b[2]:
                    g.E[:, :, k, h] = w * na * nb * E1[0][a[0], b[0]][tt] * E1[1][a[1], b[1]][u] * E1[2][a[2], b[2]][v]
        return g

    @staticmethod
    def _hermite_1d(la, lb, al, be, A, B, P):
        p = al + be
        E = {(0, 0): [torch.exp(-al * be / p * (A - B) ** 2)]}

        def step(src, d):
            get = lambda t: src[t] if 0 <= t < len(src) else 0.0  # noqa: E731
            return [get(t - 1) / (2.0 * p) + d * get(t) + (t + 1) * get(t + 1) for t in range(len(src) + 1)]

        for i in range(la + 1):
            if i:
                E[i, 0] = step(E[i - 1, 0], P - A)
            for j in range(1, lb + 1):
                E[i, j] = step(E[i, j - 1], P - B)
        return E

    def _to_matrix(self, parts):
        M = torch.zeros((self.K, self.K), dtype=torch.float64, device=DEVICE)
        v = torch.cat([x.reshape(-1) for x in parts])
        M[self.cols, self.rows] = v
        M[self.rows, self.cols] = v
        return M

    def one_electron(self):
        S, T, V = [], [], []
        xyz = torch.tensor([p for _, p in self.mol], dtype=torch.float64, device=DEVICE)
        Z = torch.tensor([float(W._z(s)) for s, _ in self.mol], dtype=torch.float64, device=DEVICE)
        for g in self.groups:
            root = (math.pi / g.p) ** 1.5
            S.append((g.E[..., 0] * root[..., None]).sum(1))
            E2 = [self._hermite_1d(g.la, g.lb + 2, g.al, g.be, g.A[:, None, d], g.B[:, None, d], g.P[..., d])
                  for d in range(3)]
            kin = []
            for na, nb, a, b in g.norms:
                o = lambda d, k: E2[d][a[d], k][0] if k >= 0 else 0.0  # noqa: E731, B023
                t1 = lambda d: (-2.0 * g.be * g.be * o(d, b[d] + 2) + g.be * (2 * b[d] + 1) * o(d, b[d])  # noqa: E731
                                - 0.5 * b[d] * (b[d] - 1) * o(d, b[d] - 2))  # noqa: B023
                s1 = [o(d, b[d]) for d in range(3)]
                kin.append((g.w * na * nb * root * (t1(0) * s1[1] * s1[2] + s1[0] * t1(1) * s1[2]
                                                    + s1[0] * s1[1] * t1(2))).sum(1))
            T.append(torch.stack(kin, -1))
            pot = torch.zeros((g.n, g.nab), dtype=torch.float64, device=DEVICE)
            Ew = g.E * (2.0 * math.pi / g.p)[..., None, None]
            step = max(1, int(2e9 // (8 * g.n * g.q * 3 * g.nh)))
            for c in range(0, len(Z), step):
                D = g.P[None] - xyz[c:c + step, None, None]
                R = _hermite_coulomb(g.L, g.p[None].expand(D.shape[:-1]), D[..., 0], D[..., 1], D[..., 2])
                pot -= torch.einsum("nqah,hnq->na", Ew, torch.einsum("hcnq,c->hnq", R, Z[c:c + step]))
            V.append(pot)
        return [self._to_matrix(x) for x in (S, T, V)]

    def _sums(self, L1, L2):
        place, at = _hermite_place(L1 + L2), []
        for a in _hermite_list(L1):
            at.append([place[a[0] + b[0], a[1] + b[1], a[2] + b[2]] for b in _hermite_list(L2)])
        sign = [(-1.0) ** sum(b) for b in _hermite_list(L2)]
        return torch.tensor(at, device=DEVICE), torch.tensor(sign, dtype=torch.float64, device=DEVICE)

    def two_electron(self, thr):
        """(ij|kl) over all function pairs (rows x cols), 0 where the Schwarz product is below thr."""
        M = torch.empty((self.n2, self.n2), dtype=torch.float64, device=DEVICE)
        for x, b in enumerate(self.groups):
            for k in self.groups[x:]:
                at, sign = self._sums(b.L, k.L)
                HL = _nherm(b.L + k.L)
                each = 8 * b.q * (k.n * k.q * (3 * HL + k.nh) + k.n * k.nab * 2 * b.nh) + 8 * k.n * k.nab * b.nab
                step = max(1, int(3e9 // each))
                Ek = (k.E * sign).permute(0, 2, 3, 1).reshape(k.n, k.nab, k.nh * k.q)   # [k, cd, (h q)]
                for s in range(0, b.n, step):
                    P, p, E = b.P[s:s + step], b.p[s:s + step], b.E[s:s + step]
                    n = P.shape[0]
                    Pf, pf = P.reshape(-1, 3), p.reshape(-1)
                    D = k.P.reshape(-1, 1, 3)
                    X = Pf[None] - D                                                     # [(k q), (b q), 3]
                    pp, qq = pf[None], k.p.reshape(-1, 1)
                    R = _hermite_coulomb(b.L + k.L, pp * qq / (pp + qq), X[..., 0], X[..., 1], X[..., 2])
                    R = R * (2.0 * math.pi ** 2.5 / (pp * qq * torch.sqrt(pp + qq)))
                    R = R.reshape(HL, k.n, k.q, n * b.q)
                    Wt = torch.empty((n, b.q, b.nh, k.n * k.nab), dtype=torch.float64, device=DEVICE)
                    for h in range(b.nh):
                        r = R[at[h]].permute(1, 0, 2, 3).reshape(k.n, k.nh * k.q, n * b.q)
                        w = torch.bmm(Ek, r)                                             # [k, cd, (b q)]
                        Wt[:, :, h] = w.reshape(k.n * k.nab, n, b.q).permute(1, 2, 0)
                    out = torch.bmm(E.permute(0, 2, 1, 3).reshape(n, b.nab, b.q * b.nh),
                                    Wt.reshape(n, b.q * b.nh, k.n * k.nab))
                    r0 = b.at + s * b.nab
                    M[r0:r0 + n * b.nab, k.at:k.at + k.n * k.nab] = out.reshape(n * b.nab, -1)
                    del R, Wt, X
        for x, b in enumerate(self.groups):
            lo, hi = b.at, b.at + b.n * b.nab
            M[hi:, lo:hi] = M[lo:hi, hi:].T
        Q = torch.sqrt(torch.clamp(torch.diagonal(M), min=0.0))
        for s in range(0, self.n2, 2048):
            M[s:s + 2048] *= (Q[s:s + 2048, None] * Q[None] >= thr)
        return M

    def coulomb(self, M, D):
        J = torch.zeros((self.K, self.K), dtype=torch.float64, device=DEVICE)
        v = M @ (self.weights * D[self.rows, self.cols])
        J[self.cols, self.rows] = v
        J[self.rows, self.cols] = v
        return J

    def exchange(self, M, D):
        out = torch.empty((self.K, self.K), dtype=torch.float64, device=DEVICE)
        flat = self.index.reshape(-1)
        for i in range(self.K):
            T = M[self.index[i]][:, flat].reshape(self.K, self.K, self.K)                # (i k | j l) at [k, j, l]
            out[i] = torch.einsum("kjl,kl->j", T, D)
        return out

    def bounds(self):
        """Largest Schwarz bound of each shell pair, group by group."""
        out = []
        for g in self.groups:
            at, sign = self._sums(g.L, g.L)
            step = max(1, int(1e9 // (8 * g.q * g.q * (3 * _nherm(2 * g.L) + g.nh * g.nh + g.nab * g.nh))))
            got = []
            for s in range(0, g.n, step):
                P, p, E = g.P[s:s + step], g.p[s:s + step], g.E[s:s + step]
                X = P[:, :, None] - P[:, None]
                pp, qq = p[:, :, None], p[:, None]
                R = _hermite_coulomb(2 * g.L, pp * qq / (pp + qq), X[..., 0], X[..., 1], X[..., 2])
                R = R * (2.0 * math.pi ** 2.5 / (pp * qq * torch.sqrt(pp + qq)))
                inner = torch.einsum("hknqr,nrak->nqah", R[at], E * sign)
                got.append(torch.einsum("nqah,nqah->na", inner, E).clamp(min=0).sqrt().amax(1))
            out.append(torch.cat(got))
        return out

    def build_flops(self, thr):
        distinct = {}
        for s, (L, xyz, prims, _) in enumerate(self.shells):
            distinct.setdefault((L, tuple(xyz)), set()).update(prims[:, 0])
        shells_of = {}
        for L, xyz, _, _ in self.shells:
            shells_of[L, tuple(xyz)] = shells_of.get((L, tuple(xyz)), 0) + 1
        share = [len(distinct[L, tuple(xyz)]) / shells_of[L, tuple(xyz)] for L, xyz, _, _ in self.shells]
        prims = [torch.tensor([share[a] * share[b] for a, b in g.pairs], device=DEVICE) for g in self.groups]
        Q = self.bounds()
        total = 0.0
        for x, b in enumerate(self.groups):
            for y in range(x, len(self.groups)):
                k = self.groups[y]
                keep = (Q[x][:, None] * Q[y][None] >= thr)
                one = 0.5 if x == y else 1.0
                L = b.L + k.L
                per = (32 + 3 * L + 3 * math.comb(L + 4, 4) + 2 * b.nh * k.nh * k.nab)
                total += one * float((keep * (prims[x][:, None] * prims[y][None])).sum()) * per
                total += one * float(keep.sum()) * 12 * b.nab * k.nab
        return total


def _scf(mol, case):
    """Energy, densities and orbital energies of the converged solution, from the
    zero density with damped first cycles and DIIS."""
    ints = _Integrals(mol, case["basis"])
    S, T, V = ints.one_electron()
    M = ints.two_electron(THRESHOLD)
    h = T + V
    s, U = torch.linalg.eigh(S)
    X = U @ torch.diag(s.rsqrt()) @ U.T
    rhf = case.get("spin", "rhf") == "rhf"
    occ = _spin(case, mol)[:1 if rhf else 2]
    P = [torch.zeros_like(S) for _ in occ]
    past, E_nuc = [], 0.0
    for i, (a, x) in enumerate(mol):
        for b, y in mol[:i]:
            E_nuc += W._z(a) * W._z(b) / math.dist(x, y)
    for cycle in range(100):
        Pt = 2.0 * P[0] if rhf else P[0] + P[1]
        J = ints.coulomb(M, Pt)
        F = [h + J - ints.exchange(M, D) for D in P]
        E = 0.5 * sum(((h + f) * D).sum() for f, D in zip(F, P)) * (2.0 if rhf else 1.0) + E_nuc
        err = [f @ D @ S - S @ D @ f for f, D in zip(F, P)]
        past = (past + [(F, torch.cat([X @ e @ X for e in err]).reshape(-1))])[-8:]
        if cycle > 3 and float(past[-1][1].abs().max()) < 1e-10:
            break
        if cycle > 2:
            n = len(past)
            B = torch.full((n + 1, n + 1), -1.0, dtype=torch.float64)
            B[n, n] = 0.0
            for i in range(n):
                for j in range(n):
                    B[i, j] = float(past[i][1] @ past[j][1])
            B[:n, :n] /= B[:n, :n].abs().max()
            rhs = torch.zeros(n + 1, dtype=torch.float64)
            rhs[n] = -1.0
            c = torch.linalg.lstsq(B, rhs, driver="gelsd").solution
            F = [sum(float(c[i]) * past[i][0][k] for i in range(n)) for k in range(len(occ))]
        e, new = [], []
        for f, n in zip(F, occ):
            w, C = torch.linalg.eigh(X @ f @ X)
            C = X @ C[:, :n]
            e.append(w)
            new.append(C @ C.T)
        P = [0.7 * a + 0.3 * b for a, b in zip(new, P)] if 0 < cycle < 3 else new
    else:
        return None
    return E, [2.0 * P[0]] if rhf else P, e

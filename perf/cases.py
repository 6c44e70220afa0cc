"""Workloads of the Fock-build and purification path, through the public API.

Kinds of case:
  fock   one Fock build of a prepared engine from a device-resident density
         (PFock.compute_dev), or from a host one (PFock.compute_fock)
  purify one density purification on host matrices (Purif.purify)
  setup  engine and one-electron matrices of a new molecule
  scf    a whole SCF solve of a prepared solver
  batch  many small molecules iterated together, their set-up included

Molecules are the generated families of gtfock_b200.molecules in the bundled
basis sets; densities are seeded matrices with a damped off-diagonal.
`exact` evaluates the same quantities with a dense McMurchie-Davidson code in
64 bits, for the molecules small enough for that.
"""
import math
import os
import tempfile

import numpy as np
import torch

import gtfock_b200 as gb
from gtfock_b200 import molecules as mol

BOHR = 0.529177210903
CHARGE = {"H": 1, "C": 6, "N": 7, "O": 8}


def listed():
    return [
        # the smallest call: one water molecule in a minimal basis, where launches count
        _fock("water1_sto3g", "water", 1, "sto-3g"),
        # a small molecule with d shells: every class pair is launched on little work
        _fock("ethane_ccpvdz", "alkane", 2, "cc-pvdz"),
        # the reference-style call with host matrices on a small molecule
        _fock("butane_ccpvdz_host", "alkane", 4, "cc-pvdz", host=True),
        # an ordinary molecule: the alkane of the CPU-runnable configuration
        _fock("c12h26_ccpvdz", "alkane", 12, "cc-pvdz"),
        # a middle-sized water cluster of the served stream, an odd number of molecules
        _fock("water23_631g", "water", 23, "6-31g"),
        # the large water cluster, FP64 and in the served form (FP32 below a bound of 1e-4)
        _fock("water64_631g", "water", 64, "6-31g"),
        _fock("water64_631g_mixed", "water", 64, "6-31g", cutoff=1e-4),
        # the headline molecule, FP64 and with FP32 quartets below a bound of 1e-6
        _fock("c54h18_ccpvdz", "flake", 2, "cc-pvdz"),
        _fock("c54h18_ccpvdz_mixed", "flake", 2, "cc-pvdz", cutoff=1e-6),
        # purification of the headline molecule's Fock matrix, host matrices as in the C API
        {"name": "purify_c54h18", "kind": "purify", "family": "flake", "n": 2, "basis": "cc-pvdz"},
        # what every new molecule pays before its first build
        {"name": "setup_c12h26", "kind": "setup", "family": "alkane", "n": 12, "basis": "cc-pvdz"},
        # small molecules iterated together, as requests of a server
        {"name": "batch16", "kind": "batch", "count": 16, "iters": 20},
    ]


def _fock(name, family, n, basis, cutoff=0.0, host=False):
    return {"name": name, "kind": "fock", "family": family, "n": n, "basis": basis, "cutoff": cutoff, "host": host}


def draw(rng):
    kind = rng.choice(["fock"] * 6 + ["purify", "setup", "scf", "batch"])
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(2, 16), "iters": rng.randint(18, 20)}
    family = rng.choice(["water", "water", "alkane", "alkane", "flake"])
    if family == "water":
        n, basis = int(64 ** rng.random() + 0.5), rng.choice(["sto-3g", "6-31g"])
    elif family == "alkane":
        n, basis = int(20 ** rng.random() + 0.5), rng.choice(["sto-3g", "6-31g", "cc-pvdz", "cc-pvdz"])
    else:
        n, basis = rng.randint(0, 1), rng.choice(["6-31g", "cc-pvdz"])
    if kind == "scf":
        return {"kind": "scf", "family": "alkane", "n": rng.randint(1, 6), "basis": "cc-pvdz", "iters": rng.randint(18, 20)}
    if kind != "fock":
        return {"kind": kind, "family": family, "n": n, "basis": basis}
    return {"kind": "fock", "family": family, "n": n, "basis": basis, "cutoff": rng.choice([0.0, 0.0, 1e-6, 1e-4]),
            "host": rng.random() < 0.25}


def _atoms(family, n, jitter=0.0, rng=None):
    atoms = (mol.water_cluster(n, 100 + n) if family == "water" else
             mol.alkane(n) if family == "alkane" else mol.graphene_flake(n))
    if jitter:
        atoms = [(s,) + tuple(float(v) for v in np.array(x) + jitter * rng.uniform(-1.0, 1.0, 3)) for s, *x in atoms]
    return atoms


def _xyz(atoms):
    with tempfile.NamedTemporaryFile("w", suffix=".xyz", delete=False) as f:
        path = f.name
    return mol.write_xyz(atoms, path)


def _basis(atoms, name):
    path = _xyz(atoms)
    basis = gb.BasisSet(mol.basis_file(name), path)
    os.unlink(path)
    return basis


def _density(n, seed):
    """Symmetric matrix of a density's size: diagonal 0.3, neighbours correlated."""
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((n, n)) * 0.05
    i = np.arange(n)
    a *= np.exp(-np.abs(i[:, None] - i[None, :]) / 20.0)
    return 0.5 * (a + a.T) + np.eye(n) * 0.3


def _fock_like(n, nocc, seed):
    """Symmetric matrix with an occupied spectrum, a gap and a virtual one, and
    an overlap matrix S with its inverse square root X."""
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    e = np.concatenate([-np.exp(rng.uniform(math.log(0.3), math.log(11.0), nocc)), rng.uniform(0.15, 4.0, n - nocc)])
    f = (q * e) @ q.T
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    s = np.exp(rng.uniform(math.log(0.01), math.log(4.0), n))
    S, X = (q * s) @ q.T, (q / np.sqrt(s)) @ q.T
    return 0.5 * (f + f.T), 0.5 * (S + S.T), 0.5 * (X + X.T)


def _batch_jobs(case, seed):
    """Molecules of a served stream: waters and alkanes in the small basis sets."""
    rng = np.random.default_rng(seed)
    jobs = []
    for i in range(case["count"]):
        family, n = ("water", 1 + i % 2) if i % 2 else ("alkane", 1 + i % 5)
        jobs.append((_atoms(family, n, 0.03, rng), "sto-3g" if i % 3 else "6-31g"))
    return jobs


class _DeviceMatrix:
    """The engine's F as torch sees it; the engine lives as long as the view."""

    def __init__(self, ptr, n, engine):
        self.engine = engine
        self.__cuda_array_interface__ = {"shape": (n, n), "typestr": "<f8", "data": (int(ptr), False), "version": 3,
                                         "strides": None}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return {"kind": kind, "iters": case["iters"],
                "jobs": [(mol.basis_file(name), _xyz(atoms)) for atoms, name in _batch_jobs(case, seed)]}
    if kind == "setup":
        return {"kind": kind, "basis": _basis(_setup_atoms(case, seed), case["basis"])}
    if kind == "scf":
        path = _xyz(_setup_atoms(case, seed))
        solver = gb.SCFSolver(mol.basis_file(case["basis"]), path)
        os.unlink(path)
        solver.set_options(etol=0.0)
        return {"kind": kind, "solver": solver, "iters": case["iters"]}
    basis = _basis(_atoms(case["family"], case["n"]), case["basis"])
    if kind == "purify":
        F, S, X = _fock_like(basis.nbf, basis.nocc, seed)
        purif = gb.Purif(basis)
        purif.set_sx(S, X)
        return {"kind": kind, "purif": purif, "F": F, "basis": basis}
    pf = gb.PFock(basis, tolscr=1e-10)
    if case["cutoff"]:
        pf.set_precision(1, case["cutoff"])
    D = _density(basis.nbf, seed)
    if case["host"]:
        return {"kind": "host", "pf": pf, "D": D, "basis": basis}
    D = torch.from_numpy(D).cuda()
    torch.cuda.synchronize()
    return {"kind": kind, "pf": pf, "D": D, "basis": basis}


def _setup_atoms(case, seed):
    return _atoms(case["family"], case["n"], 0.02, np.random.default_rng(seed))


def run(state):
    kind = state["kind"]
    if kind == "fock":
        ptr = state["pf"].compute_dev(state["D"].data_ptr())
        return torch.as_tensor(_DeviceMatrix(ptr, state["basis"].nbf, (state["pf"], state["basis"])), device="cuda")
    if kind == "host":
        return state["pf"].compute_fock(state["D"])
    if kind == "purify":
        return state["purif"].purify(state["F"])[0]
    if kind == "setup":
        pf = gb.PFock(state["basis"], tolscr=1e-10)
        S, X, H = pf.one_electron()
        pf.close()
        return {"S": S, "X": X, "H": H}
    if kind == "scf":
        energies, _ = state["solver"].solve(state["iters"])
        return {"energies": energies, "D": state["solver"].density()}
    batch = gb.Batch(len(state["jobs"]))
    slots = [batch.add(gbs, xyz, max_iters=state["iters"], etol=0.0) for gbs, xyz in state["jobs"]]
    batch.run()
    out = [batch.result(s)[0] for s in slots]
    batch.close()
    return out


def work(case):
    """Bytes: the matrices in and out.  FLOPs: the Rys-quadrature count of the
    quartets and primitive quartets that pass screening (for whole solves,
    times the iterations), and 2 n^3 per product of a purification."""
    if case["kind"] == "batch":
        f, b = 0.0, 0.0
        for atoms, name in _batch_jobs(case, 0):
            f1, n = _build_flops(atoms, name)
            f += case["iters"] * (f1 + 80.0 * n ** 3)
            b += 8.0 * case["iters"]
        return {"bytes": b, "flops": f}
    atoms = _atoms(case["family"], case["n"])
    if case["kind"] == "purify":
        n = _nbf(atoms, case["basis"])
        return {"bytes": 16.0 * n * n, "flops": 20 * 4.0 * n ** 3}
    if case["kind"] == "setup":
        n = _nbf(atoms, case["basis"])
        return {"bytes": 24.0 * n * n, "flops": 12.0 * n ** 3 + 400.0 * n * n * len(atoms)}
    f, n = _build_flops(atoms, case["basis"])
    if case["kind"] == "scf":
        return {"bytes": 8.0 * n * n, "flops": case["iters"] * (f + 100.0 * n ** 3)}
    return {"bytes": 16.0 * n * n, "flops": f}


def _build_flops(atoms, name):
    basis = _basis(atoms, name)
    pf = gb.PFock(basis, tolscr=1e-10)
    f = sum(x for x, _ in pf.class_work_screened())
    pf.close()
    return float(f), basis.nbf


def _nbf(atoms, name):
    shells, pure = _shells(atoms, name)
    return sum(5 if pure and s[0] == 2 else (s[0] + 1) * (s[0] + 2) // 2 for s in shells)


# -- the same quantities in 64 bits ------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "scf"):
        return None
    if kind == "purify":
        atoms = _atoms(case["family"], case["n"])
        n, nocc = _nbf(atoms, case["basis"]), sum(CHARGE[a[0]] for a in atoms) // 2
        F, _, X = _fock_like(n, nocc, seed)
        v = X @ np.linalg.eigh(F)[1][:, :nocc]
        return v @ v.T
    if kind == "setup":
        S, H = _one_electron(*_shells(_setup_atoms(case, seed), case["basis"]), _setup_atoms(case, seed))
        return {"S": S, "X": None, "H": H}
    atoms = _atoms(case["family"], case["n"])
    n = _nbf(atoms, case["basis"])
    if n > 120:
        return None
    shells, pure = _shells(atoms, case["basis"])
    F = _fock_matrix(shells, pure, _density(n, seed))
    return F.cpu().numpy() if case["host"] else F


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _shells(atoms, name):
    """[(L, exponents, coefficients, centre in bohr)], and whether d is spherical."""
    table, element = {}, None
    with open(mol.basis_file(name)) as f:
        lines = [x.split() for x in f if x.strip() and x.strip() != "****"]
    pure, k = lines[0][0] == "spherical", 1
    while k < len(lines):
        t = lines[k]
        if t[0] in CHARGE:
            element = table.setdefault(t[0], [])
            k += 1
            continue
        rows = np.array([[float(v.replace("D", "e")) for v in r] for r in lines[k + 1:k + 1 + int(t[1])]])
        for col, letter in enumerate(t[0].upper()):
            element.append(("SPD".index(letter), rows[:, 0], rows[:, 1 + col]))
        k += 1 + int(t[1])
    out = []
    for s, *x in atoms:
        for L, a, c in table[s]:
            odd = [1.0, 1.0, 3.0][L]
            c = c * (2 * a / np.pi) ** 0.75 * (4 * a) ** (L / 2) / math.sqrt(odd)
            p = a[:, None] + a[None, :]
            c = c / math.sqrt((c[:, None] * c[None, :] * odd / (2 * p) ** L * (np.pi / p) ** 1.5).sum())
            out.append((L, a, c, np.array(x) / BOHR))
    return out, pure


def _carts(L):
    return [(x, y, L - x - y) for x in range(L, -1, -1) for y in range(L - x, -1, -1)]


def _herms(L):
    return [(t, u, v) for t in range(L + 1) for u in range(L + 1 - t) for v in range(L + 1 - t - u)]


def _hermite(p, PA, PB, mu_r2, imax, jmax):
    """e[i][j][t]: expansion of x_A^i x_B^j exp(...) in Hermite Gaussians."""
    e = [[None] * (jmax + 1) for _ in range(imax + 1)]
    zero = torch.zeros_like(p)

    def up(src, d):
        g = lambda t: src[t] if 0 <= t < len(src) else zero
        return [g(t - 1) / (2 * p) + d * g(t) + (t + 1) * g(t + 1) for t in range(len(src) + 1)]
    for i in range(imax + 1):
        e[i][0] = [torch.exp(-mu_r2)] if i == 0 else up(e[i - 1][0], PA)
        for j in range(jmax):
            e[i][j + 1] = up(e[i][j], PB)
    return e


class _Pairs:
    """Primitive pairs of all shell pairs (i, j) of angular momenta (la, lb), i >= j where la == lb."""

    def __init__(self, shells, la, lb):
        self.la, self.lb, self.L = la, lb, la + lb
        sa = [k for k, s in enumerate(shells) if s[0] == la]
        sb = [k for k, s in enumerate(shells) if s[0] == lb]
        self.pairs = [(i, j) for i in sa for j in sb if la != lb or i >= j]
        cols = [[], [], [], [], []]
        for n, (i, j) in enumerate(self.pairs):
            a, b = np.meshgrid(shells[i][1], shells[j][1], indexing="ij")
            cols[0].append(a.ravel())
            cols[1].append(b.ravel())
            cols[2].append(np.outer(shells[i][2], shells[j][2]).ravel())
            cols[3].append(np.tile(np.concatenate([shells[i][3], shells[j][3]]), (a.size, 1)))
            cols[4].append(np.full(a.size, n))
        a, b, c, x, n = (torch.from_numpy(np.concatenate(v)).to(_dev()) for v in cols)
        self.b, self.c, self.seg = b, c, n
        self.p = a + b
        A, B = x[:, :3], x[:, 3:]
        self.P = (a[:, None] * A + b[:, None] * B) / self.p[:, None]
        self.e = [_hermite(self.p, self.P[:, d] - A[:, d], self.P[:, d] - B[:, d], a * b / self.p * (A - B)[:, d] ** 2,
                           la, lb + 2) for d in range(3)]
        self.comps = [(x, y) for x in _carts(la) for y in _carts(lb)]

    def hermite(self):
        """[components, Hermite functions, primitive pairs], the contraction coefficients included."""
        out = torch.zeros(len(self.comps), len(_herms(self.L)), len(self.p), dtype=torch.float64, device=_dev())
        for k, (x, y) in enumerate(self.comps):
            e = [self.e[d][x[d]][y[d]] for d in range(3)]
            for h, t in enumerate(_herms(self.L)):
                if all(t[d] < len(e[d]) for d in range(3)):
                    out[k, h] = self.c * e[0][t[0]] * e[1][t[1]] * e[2][t[2]]
        return out


def _boys(m, T):
    """F_0 .. F_m of T."""
    small = T < 0.5
    Ts, Tl = torch.where(small, T, torch.zeros_like(T)), torch.where(small, torch.ones_like(T), T)
    term, s = torch.ones_like(T), torch.zeros_like(T)
    for k in range(18):
        s = s + term / (2 * m + 2 * k + 1)
        term = term * -Ts / (k + 1)
    a = torch.full_like(T, m + 0.5)
    f = [torch.where(small, s, math.gamma(m + 0.5) * torch.special.gammainc(a, Tl) / (2 * Tl ** (m + 0.5)))]
    ex = torch.exp(-T)
    for k in range(m - 1, -1, -1):
        f.append((2 * T * f[-1] + ex) / (2 * k + 1))
    return f[::-1]


def _hermite_coulomb(L, alpha, r):
    """{(t, u, v): R_tuv} up to t + u + v = L for exponents alpha and distances r[3]."""
    f = _boys(L, alpha * (r[0] ** 2 + r[1] ** 2 + r[2] ** 2))
    level = {(0, 0, 0): f[L] * (-2 * alpha) ** L}
    for n in range(L - 1, -1, -1):
        up, level = level, {(0, 0, 0): f[n] * (-2 * alpha) ** n}
        for t in sorted(_herms(L - n), key=sum)[1:]:
            d = next(k for k in range(3) if t[k])
            lower = tuple(v - (k == d) for k, v in enumerate(t))
            level[t] = r[d] * up[lower]
            if lower[d]:
                level[t] = level[t] + lower[d] * up[tuple(v - (k == d) for k, v in enumerate(lower))]
    return level


def _transform(shells, pure):
    """Rows: functions of the basis; columns: Cartesian functions."""
    q = math.sqrt(3.0)
    d = np.array([[0, q, 0, 0, 0, 0], [0, 0, 0, 0, q, 0], [-.5, 0, 0, -.5, 0, 1], [0, 0, q, 0, 0, 0],
                  [q / 2, 0, 0, -q / 2, 0, 0]])
    blocks = [d if pure and s[0] == 2 else np.eye(len(_carts(s[0]))) for s in shells]
    T = np.zeros((sum(b.shape[0] for b in blocks), sum(b.shape[1] for b in blocks)))
    i = j = 0
    for b in blocks:
        T[i:i + b.shape[0], j:j + b.shape[1]] = b
        i, j = i + b.shape[0], j + b.shape[1]
    return torch.from_numpy(T).to(_dev())


def _starts(shells):
    return np.concatenate([[0], np.cumsum([len(_carts(s[0])) for s in shells])])


def _classes(shells):
    ls = sorted({s[0] for s in shells})
    return [_Pairs(shells, la, lb) for la in ls for lb in ls if la >= lb]


def _function_pairs(pairs, start):
    """Cartesian function indices [components, shell pairs] of both functions."""
    first = np.array([[start[i], start[j]] for i, j in pairs.pairs]).T
    ca = np.array([_carts(pairs.la).index(x) for x, _ in pairs.comps])
    cb = np.array([_carts(pairs.lb).index(y) for _, y in pairs.comps])
    return [torch.from_numpy(c[:, None] + f[None, :]).to(_dev()) for c, f in zip((ca, cb), first)]


def _one_electron(shells, pure, atoms):
    start = _starts(shells)
    S = torch.zeros(start[-1], start[-1], dtype=torch.float64, device=_dev())
    H = torch.zeros_like(S)
    for X in _classes(shells):
        i, j = _function_pairs(X, start)
        s = torch.zeros(len(X.comps), len(X.pairs), dtype=torch.float64, device=_dev())
        h = torch.zeros_like(s)
        w = X.c * (np.pi / X.p) ** 1.5
        for k, (x, y) in enumerate(X.comps):
            o = [X.e[d][x[d]][y[d]][0] for d in range(3)]
            t = [X.b * (2 * y[d] + 1) * o[d] - 2 * X.b ** 2 * X.e[d][x[d]][y[d] + 2][0]
                 - (0.5 * y[d] * (y[d] - 1) * X.e[d][x[d]][y[d] - 2][0] if y[d] > 1 else 0.0) for d in range(3)]
            s[k].index_add_(0, X.seg, w * o[0] * o[1] * o[2])
            h[k].index_add_(0, X.seg, w * (t[0] * o[1] * o[2] + o[0] * t[1] * o[2] + o[0] * o[1] * t[2]))
        E = X.hermite()
        for name, *x in atoms:
            R = _hermite_coulomb(X.L, X.p, [X.P[:, d] - x[d] / BOHR for d in range(3)])
            v = -2 * np.pi * CHARGE[name] / X.p * sum(E[:, k] * R[t] for k, t in enumerate(_herms(X.L)))
            h.index_add_(1, X.seg, v)
        for M, m in ((S, s), (H, h)):
            M[i, j] = m
            M[j, i] = m
    T = _transform(shells, pure)
    return (T @ S @ T.T).cpu().numpy(), (T @ H @ T.T).cpu().numpy()


def _repulsion(X, Y):
    """(ab|cd) as [components of ab, pairs ab, components of cd, pairs cd]."""
    out = torch.zeros(len(X.comps), len(X.pairs), len(Y.comps), len(Y.pairs), dtype=torch.float64, device=_dev())
    EX, EY = X.hermite(), Y.hermite()
    L, step = X.L + Y.L, max(1, int(2e7 / (len(Y.p) * (len(X.comps) + len(_herms(X.L + Y.L))))))
    for lo in range(0, len(X.p), step):
        i = slice(lo, lo + step)
        p, q = X.p[i, None], Y.p[None, :]
        R = _hermite_coulomb(L, p * q / (p + q), [X.P[i, d, None] - Y.P[None, :, d] for d in range(3)])
        pref = 2 * np.pi ** 2.5 / (p * q * torch.sqrt(p + q))
        for k, t in enumerate(_herms(Y.L)):
            z = sum(EX[:, h, i, None] * R[tuple(a + b for a, b in zip(t, s))] for h, s in enumerate(_herms(X.L)))
            z = torch.zeros(len(X.comps), len(X.pairs), len(Y.p), dtype=torch.float64,
                            device=_dev()).index_add_(1, X.seg[i], z * pref)
            z = z * (-1) ** sum(t)
            for c in range(len(Y.comps)):
                if bool((EY[c, k] != 0).any()):
                    out[:, :, c].index_add_(2, Y.seg, z * EY[c, k])
    return out


def _fock_matrix(shells, pure, D):
    """F = 2 J[D] - K[D] from the full table of repulsion integrals."""
    start, classes = _starts(shells), _classes(shells)
    n = int(start[-1])
    eri = torch.zeros(n, n, n, n, dtype=torch.float64, device=_dev())
    for x, X in enumerate(classes):
        i, j = (v.reshape(-1)[:, None] for v in _function_pairs(X, start))
        for Y in classes[:x + 1]:
            k, l = (v.reshape(-1)[None, :] for v in _function_pairs(Y, start))
            g = _repulsion(X, Y).reshape(i.shape[0], k.shape[1])
            for a, b in ((i, j), (j, i)):
                for c, d in ((k, l), (l, k)):
                    eri[a, b, c, d] = g
                    eri[c, d, a, b] = g
    T = _transform(shells, pure)
    Dc = T.T @ torch.from_numpy(D).to(_dev()) @ T
    J = (eri.reshape(n * n, n * n) @ Dc.reshape(-1)).reshape(n, n)
    K = torch.einsum("acbd,cd->ab", eri, Dc)
    return T @ (2 * J - K) @ T.T

"""Sizes where the kernels change their way of working.

* light classes (Boys functions and recurrences) and lane-split quartets:
  every pair of elements and basis sets, so that 1 to 64 primitive pairs meet
  1 to 64, at short and long distances (small T, the polynomial, the large-T
  form), against the oracle: FP64 within 1e-10 Ha, all quartets in FP32 within
  1e-6 of the largest element of F[|D|], which bounds the sum of the terms
  whatever their signs (the FP32 integrals are off by 1.5e-7 to 4e-7 of their
  quartet's largest on the mean, tests/host/eri_accuracy.cpp);
* a shell of 16 primitives, the most a basis may have: 256 primitive pairs;
* builds of two engines at once, each over several streams;
* one-launch purification of small jobs next to the tiled one of larger ones,
  and the symmetric product at sizes around its 32-wide tiles.
"""
import threading

import numpy as np
import pytest

import gtfock_b200 as gb
from gtfock_b200 import molecules as mol
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

F_TOL = 1e-10
PAIRS = [("C", "C", 1.2), ("C", "H", 1.1), ("N", "O", 1.15), ("O", "H", 3.0), ("O", "C", 9.0)]


def _density(n, seed=3):
    a = np.random.default_rng(seed).standard_normal((n, n)) * 0.1
    return a + a.T


def _engine(gbs, atoms, tmp_path):
    xyz = mol.write_xyz(atoms, str(tmp_path / "m.xyz"))
    b = gb.BasisSet(gbs, xyz)
    return b, gb.PFock(b, tolscr=1e-10), po.Basis(gbs, xyz)


@pytest.mark.parametrize("basis", ["sto-3g", "6-31g", "cc-pvdz"])
@pytest.mark.parametrize("pair", PAIRS, ids=["%s%s%g" % p for p in PAIRS])
def test_diatomics_against_oracle(pair, basis, tmp_path):
    s, t, r = pair
    b, pf, ob = _engine(mol.basis_file(basis), [(s, 0.0, 0.0, 0.0), (t, 0.3 * r, -0.4 * r, 0.866 * r)], tmp_path)
    D = _density(b.nbf)
    ref, usq, _ = po.fock_build(ob, 1e-10, D)
    assert pf.counts()["usq"] == usq
    assert np.abs(pf.compute_fock(D) - ref).max() < F_TOL
    scale = np.abs(pf.compute_fock(np.abs(D))).max()
    pf.set_precision(1, 1e9)
    assert np.abs(pf.compute_fock(D) - ref).max() < min(2e-3, 1e-6 * scale)


def test_many_primitives(tmp_path):
    gbs = tmp_path / "h16.gbs"
    rows = "".join("%20.8f %20.8f\n" % (0.05 * 2.2 ** k, 1.0 / (1.0 + k)) for k in range(16))
    gbs.write_text("spherical\n\nH     0\nS  16   1.00\n%sP   1   1.00\n  0.7  1.0\n****\n" % rows)
    b, pf, ob = _engine(str(gbs), [("H", 0.0, 0.0, 0.0), ("H", 0.0, 0.0, 0.9)], tmp_path)
    D = _density(b.nbf)
    ref, usq, _ = po.fock_build(ob, 1e-10, D)
    assert pf.counts()["usq"] == usq
    assert np.abs(pf.compute_fock(D) - ref).max() < F_TOL


def test_two_engines_at_once(tmp_path):
    mols = [(mol.alkane(3), "cc-pvdz"), (mol.water_cluster(4, 2), "6-31g")]
    eng, ref = [], []
    for k, (atoms, name) in enumerate(mols):
        b = gb.BasisSet(mol.basis_file(name), mol.write_xyz(atoms, str(tmp_path / ("m%d.xyz" % k))))
        pf = gb.PFock(b, tolscr=1e-10)
        D = _density(b.nbf, k)
        eng.append((pf, D, b))
        ref.append(pf.compute_fock(D))
    got = [[], []]

    def work(k):
        for _ in range(20):
            got[k].append(eng[k][0].compute_fock(eng[k][1]))

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (0, 1):
        assert len(got[k]) == 20
        assert max(np.abs(F - ref[k]).max() for F in got[k]) < 1e-11


def test_batch_purification_around_the_size_limit(tmp_path):
    """Alkanes / STO-3G of 9, 93, 100 and 107 functions in one batch: every
    job's density is the projector a purification must leave, D S D = D with
    trace nocc.  The loop stops at ||P - P^2|| < 1e-11 and X, the inverse
    square root of S, has a norm below 10: 1e-9 on D S D, and 1e-8 on the
    trace of about 50."""
    mols = [mol.alkane(n) for n in (1, 13, 14, 15)]
    gbs = mol.basis_file("sto-3g")
    jobs = [mol.write_xyz(m, str(tmp_path / ("a%d.xyz" % k))) for k, m in enumerate(mols)]
    batch = gb.Batch(len(jobs))
    slots = [batch.add(gbs, xyz, max_iters=4, etol=0.0) for xyz in jobs]
    batch.run()
    for slot, xyz, n in zip(slots, jobs, (9, 93, 100, 107)):
        b = gb.BasisSet(gbs, xyz)
        assert b.nbf == n
        S, _, _ = gb.PFock(b, tolscr=1e-10).one_electron()
        D = batch.density(slot, n)
        assert np.abs(D @ S @ D - D).max() < 1e-9
        assert abs(np.sum(D * S) - b.nocc) < 1e-8
        assert batch.job_stats(slot)[2] > 0
    assert batch.info()["purification_steps"] > 0


@pytest.mark.parametrize("kind,n,basis", [("water", 1, "sto-3g"), ("alkane", 1, "cc-pvdz"), ("water", 9, "sto-3g"),
                                          ("alkane", 9, "sto-3g"), ("water", 5, "6-31g"), ("alkane", 4, "cc-pvdz")])
def test_purification_against_eigenvectors(kind, n, basis, tmp_path):
    """7, 34, 63, 65, 65 and 110 functions: around and between multiples of the tile."""
    atoms = mol.alkane(n) if kind == "alkane" else mol.water_cluster(n, 1)
    b = gb.BasisSet(mol.basis_file(basis), mol.write_xyz(atoms, str(tmp_path / "m.xyz")))
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.standard_normal((b.nbf, b.nbf)))
    e = np.concatenate([-rng.uniform(0.3, 11.0, b.nocc), rng.uniform(0.15, 4.0, b.nbf - b.nocc)])
    F = (q * e) @ q.T
    F = 0.5 * (F + F.T)
    p = gb.Purif(b)
    p.set_sx(np.eye(b.nbf), np.eye(b.nbf))
    D, _ = p.purify(F)
    ref = q[:, :b.nocc] @ q[:, :b.nocc].T
    # ||D - D^2|| < 1e-11 and a gap of 0.45: D is within ~1e-11 of the projector
    assert np.abs(D - ref).max() < 1e-9
    assert np.abs(D - D.T).max() < 1e-13


def _purify_plain(F, nocc):
    """The purification loop (pscf/purif.c:301-476) for any square matrix, X = 1."""
    n = len(F)
    off = np.abs(F).sum(0) - np.abs(np.diag(F))
    hmin, hmax, mu = (np.diag(F) - off).min(), (np.diag(F) + off).max(), np.trace(F) / n
    lam = min(nocc / (hmax - mu), (n - nocc) / (mu - hmin))
    D = -lam / n * F + np.eye(n) * (lam * mu / n + nocc / n)
    best, stall = 0.0, 0
    for _ in range(100):
        D2 = D @ D.T
        D3 = D @ D2
        e, c = np.linalg.norm(D - D2), np.trace(D2 - D3) / np.trace(D - D2)
        D = ((1 - 2 * c) * D + (1 + c) * D2 - D3) / (1 - c) if c < 0.5 else ((1 + c) * D2 - D3) / c
        best, stall = (e, 0) if best == 0.0 or e < 0.99 * best else (best, stall + 1)
        if e < 1e-11 or (best < 1e-8 and stall >= 8):
            break
    return D


@pytest.mark.parametrize("kind,n,basis", [("alkane", 1, "cc-pvdz"), ("water", 5, "6-31g")])
@pytest.mark.parametrize("skew", [1e-3, 1e-6])
def test_purification_of_a_matrix_that_is_not_symmetric(kind, n, basis, skew, tmp_path):
    """34 and 65 functions.  D D^2 is not symmetric then, and the loop ends at
    ||D - D^2|| near 1e-8 at the latest: 1e-7 on D.  (A loop that mirrors one
    triangle of D D^2 goes elsewhere, by about the skew.)"""
    atoms = mol.alkane(n) if kind == "alkane" else mol.water_cluster(n, 1)
    b = gb.BasisSet(mol.basis_file(basis), mol.write_xyz(atoms, str(tmp_path / "m.xyz")))
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.standard_normal((b.nbf, b.nbf)))
    e = np.concatenate([-rng.uniform(0.3, 11.0, b.nocc), rng.uniform(0.15, 4.0, b.nbf - b.nocc)])
    A = rng.standard_normal((b.nbf, b.nbf)) * skew
    F = (q * e) @ q.T + A - A.T
    p = gb.Purif(b)
    p.set_sx(np.eye(b.nbf), np.eye(b.nbf))
    D, _ = p.purify(F)
    assert np.abs(D - _purify_plain(F, b.nocc)).max() < 1e-7

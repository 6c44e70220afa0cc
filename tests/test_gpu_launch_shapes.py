"""The shapes a Fock launch can take -- small blocks claiming unit by unit, one
large block per SM, large blocks claiming chunks -- give the same F in every
kind of build: plain, sharded, incremental, with an exchange-only part, batched.

The small shape comes from the tuning table (one block per SM below every
occupancy limit); sums in another order leave 1e-11 on F, as between runs."""
import numpy as np
import pytest

import gtfock_b200 as gb
from gtfock_b200 import molecules as mol

pytestmark = pytest.mark.gpu

TOL = 1e-11
# units of 32 lanes from which the default launches of (ss|ss), the largest
# large block (32 warps), claim chunks: 16 rounds of the resident warps
CHUNKS = 148 * 32 * 16


@pytest.fixture(autouse=True)
def clean_table():
    gb.tune_clear()
    yield
    gb.tune_clear()


def _small_shapes(kind):
    """every launch of this kind on one small block per SM"""
    for x in range(6):
        for y in range(x + 1):
            for part in (0, 1):
                for b in range(40):
                    gb.load().gtf_tune_put(kind, x, y, part, 2.0 ** b, 1, 1, 0.0)


def _water24(tmp_path, **kw):
    b = gb.BasisSet(mol.basis_file("6-31g"), mol.write_xyz(mol.water_cluster(24, 7), str(tmp_path / "w24.xyz")))
    pf = gb.PFock(b, tolscr=1e-10, **kw)
    return b, pf


def _density(n, skew=0.0):
    a = np.random.default_rng(5).standard_normal((n, n)) * 0.05
    i = np.arange(n)
    a *= np.exp(-np.abs(i[:, None] - i[None, :]) / 20.0)
    return 0.5 * (a + a.T) + skew * (a - a.T) + np.eye(n) * 0.3


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["plain", "shards", "incremental", "nosymm"])
def test_chunked_builds_match_small_blocks(tmp_path, kind, precision):
    b, pf = _water24(tmp_path, symm=0 if kind == "nosymm" else 1)
    # FP32 quartets round the same in every shape; their number is what matters here
    pf.set_precision(precision, 1e-3)
    D = _density(b.nbf, 0.5 if kind == "nosymm" else 0.0)

    def build():
        if kind == "shards":
            parts = []
            for r in range(2):
                pf.set_shard(r, 2)
                parts.append(pf.compute_fock(D).copy())
            return sum(parts)
        if kind == "incremental":
            pf.set_incremental(True)
            pf.compute_fock(0.9 * D)
            F = pf.compute_fock(D).copy()
            pf.set_incremental(False)
            return F
        return pf.compute_fock(D).copy()

    F = build()
    ssss = [q for x, y, _, q in pf.class_stats() if (x, y) == (0, 0)][0]
    assert ssss / 32 > CHUNKS * (2 if kind == "shards" else 1)
    _small_shapes(0)
    ref = build()
    assert np.abs(F).max() > 1.0
    assert np.abs(F - ref).max() < TOL
    pf.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_large_blocks_of_batched_launches(tmp_path, monkeypatch, precision):
    """Two (H2O)16 and a small molecule in batched launches of large blocks
    (from 4 rounds of the resident warps on) and in small ones: the energies of
    the first iteration, whose density does not depend on F, within the 1e-11
    per element of F times the 16 x 13 functions' density."""
    monkeypatch.setenv("GTFOCK_SOLO_UNITS", str(1 << 40))
    files = [(mol.basis_file("6-31g"), mol.write_xyz(a, str(tmp_path / ("m%d.xyz" % k))))
             for k, a in enumerate([mol.water_cluster(16, 7), mol.water_cluster(16, 8), mol.alkane(2)])]
    energies = []
    for small in (False, True):
        if small:
            _small_shapes(1)
        bt = gb.Batch(len(files))
        slots = [bt.add(g, x, precision=precision, fp32_cutoff=1e-3, max_iters=2, etol=0.0) for g, x in files]
        bt.run()
        energies.append([bt.result(s)[0][:2] for s in slots])
        bt.close()
    for e, ref in zip(*energies):
        assert np.abs(np.array(e) - np.array(ref)).max() < 1e-9 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("n", [16, 32, 80, 96, 97, 98])
def test_batch_purification_at_its_sizes(tmp_path, n):
    """Hydrogen molecules in a row (97: with a water), one function per H: 96 is
    the largest job whose purification is one launch (all of its shared memory,
    6 x 6 elements per thread), 97 the first of the tiled path; 16, 32 and 80
    fill the 16-wide thread tiles exactly.  Converged densities against the
    one-job solver's: both loops stop at |dE| below 1e-12, |dD| about its root."""
    atoms = [("H", 0.0, 0.0, 3.0 * k + s) for k in range(n // 2 - (3 if n == 97 else 0)) for s in (0.0, 0.74)]
    if n == 97:
        atoms += [("O", 0.0, 6.0, 0.0), ("H", 0.0, 6.757, 0.586), ("H", 0.0, 5.243, 0.586)]
    gbs, xyz = mol.basis_file("sto-3g"), mol.write_xyz(atoms, str(tmp_path / "m.xyz"))
    assert gb.BasisSet(gbs, xyz).nbf == n
    bt = gb.Batch(1)
    slot = bt.add(gbs, xyz, max_iters=30, etol=0.0)
    bt.run()
    e, D = bt.result(slot)[0], bt.density(slot, n)
    bt.close()
    one = gb.SCFSolver(gbs, xyz)
    one.set_options(etol=0.0)
    ref, _ = one.solve(30)
    assert abs(e[-1] - ref[-1]) < 1e-9
    assert np.abs(D - one.density()).max() < 1e-6
    one.close()

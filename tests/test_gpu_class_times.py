"""Times per class pair of builds whose launches run side by side: each is the
time of that class's own launches, whatever else the build had under way."""
import numpy as np
import pytest

import gtfock_b200 as gb
from gtfock_b200 import molecules as mol

pytestmark = pytest.mark.gpu

DDSS, DDDD = (5, 0), (5, 5)


@pytest.mark.parametrize("incremental", [False, True])
def test_class_times_of_overlapped_builds(tmp_path, incremental):
    b = gb.BasisSet(mol.basis_file("cc-pvdz"), mol.write_xyz(mol.alkane(8), str(tmp_path / "m.xyz")))
    pf = gb.PFock(b, tolscr=1e-10)
    assert all(t == 0.0 for _, _, t, _ in pf.class_stats())   # nothing built yet
    if incremental:
        pf.set_incremental(True)
    D = np.eye(b.nbf) * 0.3 + 0.01
    F = pf.compute_fock(D).copy()
    stats = pf.class_stats()
    ms = {(x, y): t for x, y, t, q in stats if q > 0}
    assert len(ms) == 21 and min(ms.values()) > 0.0
    # 18 launches of 1296-integral quartets against one of 36-integral quartets
    assert ms[DDDD] > ms[DDSS]
    assert pf.class_stats() == stats                          # measured once
    assert np.array_equal(pf.get_mat(gb.MAT_F), F)
    assert np.abs(pf.compute_fock(D) - F).max() < 1e-11
    pf.close()

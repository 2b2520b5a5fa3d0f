"""The near field of the static multipoles in the FMM's E_M2D."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_waters,order", [(1500, 4), (4000, 8), (8000, 3)])
def test_near_field_of_neighbouring_leaves(n_waters, order, tmp_path):
    """Multipoles only within 5.5 bohr of the middle of the box, a corner of
    leaves at every depth: the sites as near (less than a leaf's side)
    have them in neighbouring leaves, no expansion contributes, and their field
    is the direct one but for the order of the sums (3e-14 of the field each
    way over water; limit 3e-13)."""
    w = synth.water_cluster(n_waters, seed=5)
    g = OMMPSystem(synth.write_mmp(str(tmp_path / "w.mmp"), w))
    x = g.cmm
    assert g.pol_atoms == g.mm_atoms
    r = np.linalg.norm(x - (x.min(axis=0) + 0.5 * np.max(x.max(axis=0) - x.min(axis=0))), axis=1)
    w.mult = np.where(r[:, None] < 5.5, w.mult, 0.0)
    path = synth.write_mmp(str(tmp_path / "z.mmp"), w)
    ref = OMMPSystem(path).e_m2d()
    g = OMMPSystem(path)
    g.set_fmm(True, order)
    e = g.e_m2d()
    near = r < 5.5
    assert np.count_nonzero(near) >= 5 and np.linalg.norm(ref[:, near]) > 0
    assert np.linalg.norm(e[:, near] - ref[:, near]) / np.linalg.norm(ref[:, near]) < 3e-13
    # the other sites do see expansions
    assert not np.array_equal(e[:, ~near], ref[:, ~near])

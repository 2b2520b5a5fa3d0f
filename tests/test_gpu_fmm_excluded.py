"""Excluded pairs under the FMM: the near field forms them (csrc/fmm_near.cu) and
the finishing pass takes them out again (csrc/kernels.cu) with the same
operations, so that a single dipole gives exactly nothing at the neighbours that
do not see it.  The cells of bonded neighbours touch: no expansion reaches from
one to the other."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("site", [1, 50, 150, 298])
def test_excluded_pairs_cancel(tmp_path, site):
    w = synth.chain_system(3, 100, 1500, seed=4)
    g = OMMPSystem(synth.write_mmp(str(tmp_path / "c.mmp"), w))
    g.set_fmm(True)
    x = np.zeros((g.pol_atoms, 3))
    x[site] = (0.3, -0.7, 0.9)
    y = g.tmatvec(x, dodiag=False)
    assert not y[[site - 1, site + 1]].any()
    assert y[[k for k in range(len(y)) if abs(k - site) > 5]].any(axis=1).all()

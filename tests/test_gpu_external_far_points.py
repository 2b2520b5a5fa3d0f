"""Points far outside the system, or not finite, beside ordinary ones
(csrc/external.cu): the ordinary points keep their values and the far ones have
those of plain FP64.

Tolerances: an ordinary point as in test_gpu_external_points, 1e-11 of the
largest value; a grid as wide as 2^22 bohr resolves 2^-49 bohr, 4e-16 of the
distance of a pair formed on it (5 bohr or more), so that 1e-13 of an ordinary
point's sum of terms (here at most ten times the largest value) holds beside
any other point: 1e-12.  A far point of a neutral system has a value of its
charges' cancelling sum: 1e-12 of the sum of their absolute terms."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [1e5, 3e6, 5e6, 1e8, 1e10, 1e13, np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("kind", ["water", "chain"])
def test_far_points(tmp_path, kind, far):
    w = synth.water_cluster(60, seed=3) if kind == "water" else synth.chain_system(2, 20, 50, seed=3)
    p = synth.write_mmp(str(tmp_path / "s.mmp"), w)
    g, o = OMMPSystem(p), OracleSystem(p)
    rng = np.random.default_rng(5)
    g.set_external_field(1e-3 * rng.standard_normal((g.pol_atoms, 3)))
    o.set_ipd(g.ipd)
    pts = o.cmm[rng.integers(len(o.cmm), size=150)] + rng.uniform(0.5, 8.0, (150, 3))
    out = np.array([[far, 1.0, 2.0], [3.0, far, far]])
    both = np.concatenate([pts[:70], out[:1], pts[70:], out[1:]])
    near = np.r_[0:70, 71:151]
    q = np.abs(o.q).sum()
    for which, pot, fld in ((0, g.potential_mmpol2ext, g.field_mmpol2ext), (1, g.potential_mm2ext, g.field_mm2ext),
                            (2, g.potential_pol2ext, g.field_pol2ext)):
        for get, ref, power in ((pot, o.potential_ext, 1), (fld, o.field_ext, 2)):
            v, r = get(both), ref(which, both)
            assert np.abs(v[near] - r[near]).max() <= 1e-12 * np.abs(r[near]).max()
            for k in (70, 151):
                if not np.isfinite(far):
                    assert not np.isfinite(v[k]).any()
                else:
                    assert np.abs(v[k] - r[k]).max() <= 1e-12 * q / far ** power

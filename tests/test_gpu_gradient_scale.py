"""The polarization gradient (csrc/grad_sym.cu) of weak charges and weak
dipoles: its terms are products of a static multipole, or a dipole, and a
dipole, and neither factor's size may cost bits of the fixed-point sums.

Tolerance: a pair's double-single terms are within 2^-44 of their value and
cancel at most about tenfold between the pairs of a site (random fields):
1e-12 of the gradient's largest value, against the oracle on the same dipoles."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nomm", [False, True])
@pytest.mark.parametrize("field", [1e-2, 1e-5, 1e-8, 1e-100])
@pytest.mark.parametrize("charges", [1.0, 1e-3, 0.0])
@pytest.mark.parametrize("kind", ["water", "chain"])
def test_matches_oracle(tmp_path, kind, charges, field, nomm):
    """nomm, AMOEBA: the P dipoles are zero and differ from the D ones."""
    if nomm and kind == "water" and charges == 0.0:
        pytest.skip("(D P' + P D') / 2 = 0: the gradient is exactly zero")
    w = synth.water_cluster(40, seed=6) if kind == "water" else synth.chain_system(1, 20, 30, seed=6)
    w.mult = w.mult * charges
    p = synth.write_mmp(str(tmp_path / "s.mmp"), w)
    g, o = OMMPSystem(p), OracleSystem(p)
    f = field * np.random.default_rng(1).standard_normal((g.pol_atoms, 3))
    g.set_external_field(f, nomm=nomm, solver="inversion")
    o.set_ipd(g.ipd)
    ref = o.polelec_geomgrad()
    assert np.abs(g.polelec_geomgrad() - ref).max() < 1e-12 * np.abs(ref).max()

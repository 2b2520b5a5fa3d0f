"""The inversion solver is linear in the field at any size, also where the
squares of its values leave the range of a double (csrc/engine.cu).

Tolerance: solutions of an FP64 solver, condition number (below 1e2 here)
times 1e-15, 1e-12."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-300, 1e-200, 1e-150, 1e150, 1e200, 0.0])
def test_scaled_field(tmp_path, scale):
    g = OMMPSystem(synth.write_mmp(str(tmp_path / "s.mmp"), synth.water_cluster(20, seed=2)))
    f = np.random.default_rng(1).standard_normal((g.pol_atoms, 3))
    g.set_external_field(f, nomm=True, solver="inversion")
    ref = g.ipd[0].copy()
    for _ in range(2):
        g.set_external_field(scale * f, nomm=True, solver="inversion")
        assert np.abs(g.ipd[0] - scale * ref).max() <= 1e-12 * scale * np.abs(ref).max()
    g.set_external_field(f, nomm=True, solver="inversion")
    assert np.abs(g.ipd[0] - ref).max() <= 1e-12 * np.abs(ref).max()

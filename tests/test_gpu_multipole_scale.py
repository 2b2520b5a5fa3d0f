"""The static-static energy and gradient (csrc/m2m.cu) scale with the square of
the multipoles at any size of them.

A power of two scales every multipole exactly, so that the results differ from
those of the unscaled system, scaled, by the roundings of the sums at most: the
kernels' 3.5e-14 of the gradient on either side, 1e-12; the energy cancels
further, 1e-11."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth

pytestmark = pytest.mark.gpu


def load(tmp_path, w, e):
    """The system with its multipoles times 2^e, to the last bit."""
    p = synth.write_mmp(str(tmp_path / "s.mmp"), w)
    lines = open(p).read().split("\n")
    first = 24 + 3 * w.mm_atoms
    for i in range(w.mm_atoms):
        q = [float(v) for v in lines[first + i].split()]
        lines[first + i] = " ".join("%.17e" % v for v in np.ldexp(q, e))
    open(p, "w").write("\n".join(lines))
    return OMMPSystem(p)


@pytest.mark.parametrize("kind", ["water", "chain"])
def test_scaled_multipoles(tmp_path, kind):
    w = synth.water_cluster(100, seed=3) if kind == "water" else synth.chain_system(1, 20, 80, seed=3)
    g = load(tmp_path, w, 0)
    energy, grad = g.get_fixedelec_energy(), g.fixedelec_geomgrad()
    for e in (-3, -20, -40, -60, -80, 10, 40):
        g = load(tmp_path, w, e)
        assert abs(np.ldexp(g.get_fixedelec_energy(), -2 * e) - energy) < 1e-11 * abs(energy)
        assert np.linalg.norm(np.ldexp(g.fixedelec_geomgrad(), -2 * e) - grad) < 1e-12 * np.linalg.norm(grad)

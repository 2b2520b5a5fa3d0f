"""External points at the edges of the kernel's tiles (csrc/external.cu): one
to a few hundred points and sites, points far outside the system and close to
its sites, against the CPU oracle.

Tolerance: a pair is within 2^-44 of its terms and the potential of neutral
molecules is down to a hundredth of them: 1e-11 of the largest value (the
oracle's own FP64 sums carry the same factor of 1e-16)."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,size,npoints", [("water", 1, 1), ("water", 11, 33), ("water", 43, 127),
                                               ("water", 86, 129), ("chain", 1, 5), ("chain", 26, 300)])
def test_matches_oracle(tmp_path, kind, size, npoints):
    if kind == "water":
        w = synth.water_cluster(size, seed=size)
    else:
        w = synth.chain_system(n_chains=2, chain_len=10, n_waters=size, seed=size)
    p = synth.write_mmp(str(tmp_path / "s.mmp"), w)
    g, o = OMMPSystem(p), OracleSystem(p)
    rng = np.random.default_rng(size)
    c = o.cmm
    near = c[rng.integers(len(c), size=npoints)] + rng.uniform(0.4, 1.5, (npoints, 3))
    far = rng.uniform(-1.0, 1.0, (npoints, 3)) * np.array([300.0, 3000.0, 30.0])
    ipd = rng.standard_normal((g.n_ipd, g.pol_atoms, 3))
    g.set_solver_tol(1e-12)
    g.set_external_field(ipd[0])
    o.set_ipd(g.ipd)
    for pts in (near, far, np.concatenate([far, near])):
        for which, pot, fld in ((0, g.potential_mmpol2ext, g.field_mmpol2ext), (1, g.potential_mm2ext, g.field_mm2ext),
                                (2, g.potential_pol2ext, g.field_pol2ext)):
            v, e = o.potential_ext(which, pts), o.field_ext(which, pts)
            assert np.abs(pot(pts) - v).max() <= 1e-11 * np.abs(v).max()
            assert np.abs(fld(pts) - e).max() <= 1e-11 * np.abs(e).max()


def test_small_dipoles(tmp_path):
    """The induced part scales with its dipoles down to 2^-400, bit for bit."""
    w = synth.water_cluster(50, seed=3)
    g = OMMPSystem(synth.write_mmp(str(tmp_path / "s.mmp"), w))
    x = np.random.default_rng(1).standard_normal((g.pol_atoms, 3))
    pts = g.cmm[:40] + 1.3
    out = []
    for e in (0, -400):
        g.clear_guess()
        g.set_external_field(np.ldexp(x, e), nomm=True, solver="inversion")
        out.append((np.ldexp(g.potential_pol2ext(pts), -e), np.ldexp(g.field_pol2ext(pts), -e)))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])

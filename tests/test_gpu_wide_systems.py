"""Systems wider than the split coordinates of the double-single kernels resolve
(a molecule parked far away): every pair is formed in FP64 then, and the results
are those of plain FP64; and back to the ordinary kernels when the system is
compact again, bit for bit.

Tolerances: FP64 sums of up to a thousand terms that cancel a few times, 1e-12
of the result's norm; the static energy is a cancelling sum of the charges'
terms, 1e-11 of it; a solve to 1e-12, 1e-9."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, solve_multi, synth
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def load(tmp_path, kind, size):
    if kind == "water":
        w = synth.water_cluster(size, seed=3)
    else:
        w = synth.chain_system(1, 20, size, seed=3)
    p = synth.write_mmp(str(tmp_path / "s.mmp"), w)
    return OMMPSystem(p), OracleSystem(p)


@pytest.mark.parametrize("far", [1e6, 3e7, 1e9, 1e12])
@pytest.mark.parametrize("kind,size", [("water", 60), ("water", 300), ("chain", 120)])
def test_far_molecule(tmp_path, kind, size, far):
    g, o = load(tmp_path, kind, size)
    c0 = g.cmm.copy()
    c = c0.copy()
    c[-3:] += [far, 0.5 * far, 0.0]
    rng = np.random.default_rng(2)
    x = rng.standard_normal((2, g.pol_atoms, 3))
    f = 1e-3 * rng.standard_normal((g.pol_atoms, 3))
    pts = c0[:50] + 3.0
    before = g.tmatvec(x), g.e_m2d(), g.potential_mm2ext(pts)
    g.update_coordinates(c)
    o.update_coordinates(c)
    ref = np.stack([o.tmatvec(x[0]), o.tmatvec(x[1])])
    for kernel in ("symmetric", "ordered", "auto"):
        g.set_fp64_kernel(kernel)
        assert rel(g.tmatvec(x), ref) < 1e-12
        assert rel(g.tmatvec(x[0]), ref[0]) < 1e-12
    assert rel(g.e_m2d(), o.e_m2d()) < 1e-12
    assert abs(g.get_fixedelec_energy() - o.get_fixedelec_energy()) < 1e-11 * abs(o.get_fixedelec_energy())
    assert rel(g.fixedelec_geomgrad(), o.fixedelec_geomgrad()) < 1e-11
    g.set_solver_tol(1e-12)
    g.set_external_field(f)
    o.set_ipd(g.ipd)
    assert rel(g.polelec_geomgrad(), o.polelec_geomgrad()) < 1e-11
    assert rel(g.potential_mmpol2ext(pts), o.potential_ext(0, pts)) < 1e-12
    assert rel(g.field_mmpol2ext(pts), o.field_ext(0, pts)) < 1e-12
    o.set_tol(1e-12)
    o.set_external_field(f)
    assert rel(g.ipd, o.ipd) < 1e-9
    g.update_coordinates(c0)
    after = g.tmatvec(x), g.e_m2d(), g.potential_mm2ext(pts)
    for a, b in zip(before, after):
        assert np.array_equal(a, b)


def test_products_of_a_large_wide_system(tmp_path):
    """2,403 sites: above the size of the symmetric product, and the shared
    launches of the multi-system engine, which always take it."""
    g, o = load(tmp_path, "water", 801)
    c = g.cmm.copy()
    c[-3:] += [1e9, 0.0, 0.0]
    g.update_coordinates(c)
    o.update_coordinates(c)
    x = np.random.default_rng(2).standard_normal((2, g.pol_atoms, 3))
    ref = np.stack([o.tmatvec(x[0]), o.tmatvec(x[1])])
    assert rel(g.tmatvec(x), ref) < 1e-12
    f = 1e-3 * x[0]
    g.set_solver_tol(1e-10)
    g.set_precision("mixed-ds")
    solve_multi([g], [f])
    e = o.e_m2d()
    for k in range(2):
        r = e[k] + f - o.tmatvec(g.ipd[k])
        assert np.sqrt((o.pol[:, None] * r * r).mean()) < 2e-10  # twice the solver's tolerance

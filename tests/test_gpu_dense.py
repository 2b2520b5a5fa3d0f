"""The inversion solver (FP32 inverse refined in FP64, csrc/dense.cu) at the
edges of its 64 x 64 blocks, its FP64 LU fall-back for a matrix that is not
positive definite, and the in-core product, against the CPU oracle.

Tolerances: a refined solution is that of an FP64 solver, condition number
(below 1e2 here) times 1e-15 on either side, 1e-12; the indefinite matrix has
a condition number up to 1e5: 1e-9."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth
from oracle.oracle import SOLVER_INVERSION, OracleSystem

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def pair(tmp_path, w):
    p = synth.write_mmp(str(tmp_path / "s.mmp"), w)
    g, o = OMMPSystem(p), OracleSystem(p)
    g.set_default_solver("inversion")
    o.set_default_solver(SOLVER_INVERSION)
    c = o.cmm
    ef, _, _ = synth.point_charge_field(c[o.polar_mm], w.box_center(), seed=4, n_charges=3, radius=3.0, guard=0.5,
                                        all_sites_bohr=c)
    return g, o, ef


@pytest.mark.parametrize("waters", [1, 7, 8, 14, 15, 57, 64])
def test_inversion_matches_oracle(tmp_path, waters):
    g, o, ef = pair(tmp_path, synth.water_cluster(waters, seed=waters))
    for k in range(2):  # a second field on the same geometry reuses the inverse
        g.set_external_field((1 + k) * ef)
        o.set_external_field((1 + k) * ef)
        assert rel(g.ipd, o.ipd) < 1e-12
    c = o.cmm + np.random.default_rng(waters).uniform(-0.05, 0.05, o.cmm.shape)
    g.update_coordinates(c)
    o.update_coordinates(c)
    g.set_external_field(ef)
    o.set_external_field(ef)
    assert rel(g.ipd, o.ipd) < 1e-12


def test_inversion_of_chains(tmp_path):
    g, o, ef = pair(tmp_path, synth.chain_system(n_chains=2, chain_len=15, n_waters=30, seed=8))
    g.set_external_field(ef)
    o.set_external_field(ef)
    assert rel(g.ipd, o.ipd) < 1e-12


def test_not_positive_definite(tmp_path):
    """Molecules at half their distances with thirty times the polarizability:
    T has negative eigenvalues and the solver takes the LU factors."""
    w = synth.water_cluster(30, seed=2)
    w.pol, w.coords = w.pol * 30.0, w.coords * 0.5
    g, o, ef = pair(tmp_path, w)
    n = o.pol_atoms
    T = np.stack([o.tmatvec(e.reshape(n, 3)).ravel() for e in np.eye(3 * n)])
    ev = np.linalg.eigvalsh(0.5 * (T + T.T))
    assert ev[0] < 0 and abs(ev).max() / abs(ev).min() < 1e5
    for _ in range(2):
        g.set_external_field(ef)
        o.set_external_field(ef)
        assert rel(g.ipd, o.ipd) < 1e-9


@pytest.mark.parametrize("waters", [1, 10, 43, 90])
def test_in_core_product(tmp_path, waters):
    g, o, _ = pair(tmp_path, synth.water_cluster(waters, seed=waters))
    x = np.random.default_rng(waters).standard_normal((2, o.pol_atoms, 3))
    for dodiag in (True, False):
        y = g.tmatvec(x, dodiag=dodiag, matv="incore")
        for k in range(2):
            assert rel(y[k], o.tmatvec(x[k], dodiag=dodiag)) < 1e-13 * (1 + 9 * (not dodiag))

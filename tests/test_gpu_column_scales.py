"""The columns of a product do not see each other's size: the dipoles of every
column of the symmetric product (csrc/tmu_sym.cu) and of the FMM's near field
(csrc/fmm_near.cu) have a scale of their own.

Tolerance as for the symmetric product (test_gpu_sym_product): 2e-13 of the
result's norm.  A column's arithmetic depends on its own scale only, so that
its values beside two partners of different size are the same bits."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu
TOL = 2e-13


def load(tmp_path, kind, size):
    if kind == "water":
        w = synth.water_cluster(size, seed=size)
    else:
        w = synth.chain_system(n_chains=3, chain_len=20, n_waters=size, seed=size)
    p = synth.write_mmp(str(tmp_path / "s.mmp"), w)
    return OMMPSystem(p), OracleSystem(p)


@pytest.mark.parametrize("ratio", [1e9, 1e-9, 1e18])
@pytest.mark.parametrize("kind,size", [("water", 43), ("water", 340), ("water", 801), ("chain", 352)])
def test_symmetric_product(tmp_path, kind, size, ratio):
    g, o = load(tmp_path, kind, size)
    g.set_fp64_kernel("symmetric")
    x = np.random.default_rng(size).standard_normal((2, o.pol_atoms, 3))
    x[1] *= ratio
    y = g.tmatvec(x)
    for k in range(2):
        ref = o.tmatvec(x[k])
        assert np.linalg.norm(y[k] - ref) < TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("nf", [2, 5, 6])
def test_batch_groups(tmp_path, nf):
    """2,403 sites: the FP64 CG of several columns takes the symmetric product
    in groups of two columns (two in one launch), an odd column alone."""
    g, _ = load(tmp_path, "water", 801)
    g.set_solver_tol(1e-6)
    rng = np.random.default_rng(nf)
    f = 1e-3 * rng.standard_normal((nf, g.pol_atoms, 3))
    out = []
    for ratio in (1.0, 1e5):
        s = f.copy()
        s[1::2] *= ratio
        out.append(np.asarray(g.set_external_fields_batch(s)[0])[0::2])
    assert np.array_equal(out[0], out[1])


def test_fmm(tmp_path):
    g, _ = load(tmp_path, "water", 1500)
    g.set_fmm(True)
    x = np.random.default_rng(3).standard_normal((2, g.pol_atoms, 3))
    y = g.tmatvec(x[0])
    for ratio in (1e9, 1e25):
        assert np.array_equal(g.tmatvec(np.stack([x[0], ratio * x[1]]))[0], y)

"""T.mu of FP64 accuracy (csrc/tmu_sym.cu) at the edges of its schedule: sizes
around its 32- and 128-site tiles, an odd and an even number of tiles, both
kernels (each unordered pair once; all ordered pairs), one and two columns,
AMOEBA and Wang-AL with excluded pairs, against the CPU oracle.

Tolerance: a double-single pair is within 2^-44 of its term (products and sums
of a few 2^-47 roundings), and the terms' absolute sum is at most a few times
the result: 2e-13 of the result's norm."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu
TOL = 2e-13


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def load(tmp_path, kind, size):
    if kind == "water":
        w = synth.water_cluster(size, seed=size)
    else:
        w = synth.chain_system(n_chains=3, chain_len=20, n_waters=size, seed=size)
    p = synth.write_mmp(str(tmp_path / "s.mmp"), w)
    return OMMPSystem(p), OracleSystem(p)


@pytest.mark.parametrize("kind,size", [("water", 1), ("water", 11), ("water", 43), ("water", 85), ("water", 128),
                                       ("water", 333), ("water", 340), ("water", 700), ("chain", 20), ("chain", 352)])
def test_matches_oracle(tmp_path, kind, size):
    g, o = load(tmp_path, kind, size)
    x = np.random.default_rng(size).standard_normal((2, o.pol_atoms, 3))
    ref = np.stack([o.tmatvec(x[0]), o.tmatvec(x[1])])
    for kernel in ("auto", "ordered", "symmetric"):
        g.set_fp64_kernel(kernel)
        assert rel(g.tmatvec(x), ref) < TOL
        assert rel(g.tmatvec(x[1]), ref[1]) < TOL
    assert rel(g.tmatvec_ds(x), ref) < TOL


@pytest.mark.parametrize("size", [100, 500])
def test_scale_does_not_matter(tmp_path, size):
    """Dipoles times a power of two give the product times it, bit for bit
    (the symmetric product scales by the largest magnitude), and one
    non-finite dipole makes the whole product non-finite."""
    g, o = load(tmp_path, "water", size)
    g.set_fp64_kernel("symmetric")
    x = np.random.default_rng(size).standard_normal((o.pol_atoms, 3))
    y = g.tmatvec(x)
    for e in (-300, -60, 60, 300):
        assert np.array_equal(g.tmatvec(np.ldexp(x, e)), np.ldexp(y, e))
    assert not g.tmatvec(np.zeros_like(x)).any()
    x[size, 1] = np.nan
    assert np.isnan(g.tmatvec(x)).all()


def test_offset_coordinates(tmp_path):
    """A system far from the origin: the same product as at the origin (the
    shift by 512 bohr is exact to 2^-44 bohr, and r^-3 of the closest pairs
    (about 1.8 bohr apart, damped) follows it within 1e-12)."""
    g, o = load(tmp_path, "water", 400)
    x = np.random.default_rng(2).standard_normal((o.pol_atoms, 3))
    y = g.tmatvec(x)
    g.update_coordinates(g.cmm + 512.0)
    assert rel(g.tmatvec(x), y) < 1e-12

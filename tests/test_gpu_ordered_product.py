"""T.mu over all ordered pairs (csrc/tmu_rows.cu): sizes around its rules (300
and 800 sites), around tiles of 128 sources and CTAs of 8 targets, one, two
and an odd number of columns, columns of very different scale, AMOEBA and
Wang-AL with excluded pairs, lists longer than their capacity (a compressed
system), against the CPU oracle.

Tolerance as for the symmetric product (test_gpu_sym_product): a
double-single pair is within 2^-44 of its term and the terms' absolute sum is
at most a few times the result, 2e-13 of the result's norm; the compressed
system's terms cancel further (its condition number is about 30 times that of
the others), 6e-12."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu
TOL = 2e-13


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def load(tmp_path, kind, size, squeeze=1.0):
    if kind == "water":
        w = synth.water_cluster(size, seed=size)
    else:
        w = synth.chain_system(n_chains=3, chain_len=20, n_waters=size, seed=size)
    w.coords = w.coords * squeeze
    p = synth.write_mmp(str(tmp_path / "s.mmp"), w)
    return OMMPSystem(p), OracleSystem(p)


@pytest.mark.parametrize("kind,size", [("water", 1), ("water", 3), ("water", 43), ("water", 99), ("water", 100),
                                       ("water", 266), ("water", 267), ("water", 300), ("water", 799), ("water", 801),
                                       ("chain", 20), ("chain", 120), ("chain", 352)])
def test_matches_oracle(tmp_path, kind, size):
    g, o = load(tmp_path, kind, size)
    g.set_fp64_kernel("ordered")
    x = np.random.default_rng(size).standard_normal((2, o.pol_atoms, 3))
    x[1] *= 1e9  # each column has its own scale
    ref = np.stack([o.tmatvec(x[0]), o.tmatvec(x[1])])
    y = g.tmatvec(x)
    for k in range(2):
        assert rel(y[k], ref[k]) < TOL
        assert rel(g.tmatvec(x[k]), ref[k]) < TOL
    assert np.all(g.tmatvec(np.zeros_like(x)) == 0.0)
    x[0, 0, 0] = np.nan
    assert np.isnan(g.tmatvec(x[0])).any()


@pytest.mark.parametrize("size", [120, 300])
def test_long_lists(tmp_path, size):
    """At 0.45 of its size a water cluster has some 200 sources within 6 bohr
    of a site."""
    g, o = load(tmp_path, "water", size, 0.45)
    g.set_fp64_kernel("ordered")
    x = np.random.default_rng(size).standard_normal((2, o.pol_atoms, 3))
    y = g.tmatvec(x)
    for k in range(2):
        ref = o.tmatvec(x[k])
        assert rel(y[k], ref) < 6e-12
        assert rel(g.tmatvec(x[k]), ref) < 6e-12

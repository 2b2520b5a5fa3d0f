"""Source-split partials summed before the finishing passes (k_sum_splits):
numbers of splits around its eight warps, few and many values, for the
external points (a few points against all sites), the static sums and the
permanent field of systems of different sizes, against the CPU oracle.

Tolerance: the sums keep FP64 rounding, 1e-12 of the result's norm as in the
tests of those sums; a single molecule's pairs are all excluded, where the
oracle skips them and the kernels cancel terms of order one: 1e-14 absolute.
Far from a neutral system the potentials cancel too: 1e-13 (a double-single
pair is within 2^-44 of its term) of the sum of the charges' absolute terms."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu
TOL = 1e-12


def rel(a, b):
    d, n = np.linalg.norm(np.asarray(a) - np.asarray(b)), np.linalg.norm(np.asarray(b))
    return d / n if n > 0.0 else d * TOL / 1e-14


@pytest.mark.parametrize("size", [1, 42, 43, 96, 97, 420, 1000])
@pytest.mark.parametrize("kind", ["water", "chain"])
def test_sums_of_splits(tmp_path, kind, size):
    if kind == "water":
        w = synth.water_cluster(size, seed=size)
    else:
        w = synth.chain_system(n_chains=2, chain_len=12, n_waters=size, seed=size)
    p = synth.write_mmp(str(tmp_path / "s.mmp"), w)
    g, o = OMMPSystem(p), OracleSystem(p)
    assert rel(g.e_m2d(), o.e_m2d()) < TOL
    assert abs(g.get_fixedelec_energy() - o.get_fixedelec_energy()) < TOL * max(1.0, abs(o.get_fixedelec_energy()))
    assert rel(g.fixedelec_geomgrad(), o.fixedelec_geomgrad()) < 1e-11
    rng = np.random.default_rng(size)
    for n in (1, 31, 33, 200):
        c = g.cmm.mean(0) + 40.0 + 5.0 * rng.standard_normal((n, 3))
        r = np.linalg.norm(c[:, None, :] - g.cmm[None, :, :], axis=2)
        q = np.abs(np.asarray(g.q).reshape(g.mm_atoms, -1)[:, 0])
        v, e = g.potential_mm2ext(c) - o.potential_ext(1, c), g.field_mm2ext(c) - o.field_ext(1, c)
        assert np.all(np.abs(v) < 1e-13 * (q / r).sum(1))
        assert np.all(np.linalg.norm(e, axis=1) < 1e-13 * (q / r ** 2).sum(1))

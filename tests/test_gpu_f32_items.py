"""The FP32 symmetric product's item space (csrc/tmu32.cu): sizes below one
round of CTAs (all units cut into sub-tiles), around one round and between
rounds, an odd and an even number of super-tiles, against the FP64 product.
The FP32 operator's documented bound is 1e-5 of T (relative)."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,size", [("water", 1), ("water", 86), ("water", 340), ("water", 2900), ("water", 2902),
                                       ("water", 3100), ("water", 5000), ("chain", 1000)])
def test_item_space(tmp_path, kind, size):
    if kind == "water":
        w = synth.water_cluster(size, seed=size)
    else:
        w = synth.chain_system(n_chains=6, chain_len=40, n_waters=size, seed=size)
    g = OMMPSystem(synth.write_mmp(str(tmp_path / "s.mmp"), w))
    g.set_fp32_kernel("symmetric")
    x = np.random.default_rng(size).standard_normal((2, g.pol_atoms, 3))
    ref = g.tmatvec(x)
    y = g.tmatvec_fp32(x)
    assert np.linalg.norm(y - ref) < 1e-5 * np.linalg.norm(ref)
    one = g.tmatvec_fp32(x[1])
    assert np.linalg.norm(one - ref[1]) < 1e-5 * np.linalg.norm(ref[1])
    assert np.array_equal(g.tmatvec_fp32(x), y)

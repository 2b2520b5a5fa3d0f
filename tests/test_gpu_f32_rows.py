"""The pairwise FP32 product (csrc/tmu32_rows.cu): sizes around its 128-source
tiles, 4 targets per CTA and the 32 sources between two compensations, 1 to 9
columns (groups of 4, 2 and 1), AMOEBA and Wang-AL, against the FP64 product.
The FP32 operator's documented bound is 1e-5 of T (relative)."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth

pytestmark = pytest.mark.gpu


def load(tmp_path, kind, size):
    if kind == "water":
        w = synth.water_cluster(size, seed=size)
    else:
        w = synth.chain_system(n_chains=3, chain_len=20, n_waters=size, seed=size)
    return OMMPSystem(synth.write_mmp(str(tmp_path / "s.mmp"), w))


@pytest.mark.parametrize("kind,size", [("water", 1), ("water", 2), ("water", 42), ("water", 43), ("water", 85),
                                       ("water", 342), ("water", 1200), ("chain", 20), ("chain", 352)])
def test_matches_fp64_product(tmp_path, kind, size):
    g = load(tmp_path, kind, size)
    g.set_fp32_kernel("pairwise")
    x = np.random.default_rng(size).standard_normal((2, g.pol_atoms, 3))
    ref = g.tmatvec(x)
    for y in (g.tmatvec_fp32(x), np.stack([g.tmatvec_fp32(x[0]), g.tmatvec_fp32(x[1])])):
        assert np.linalg.norm(y - ref) < 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("nf", [2, 3, 4, 7, 9])
def test_column_groups(tmp_path, nf):
    """Every column of a batch converges as the single solve does: to the
    mixed mode's tolerance on the FP64 residual."""
    g = load(tmp_path, "water", 85)
    g.set_fp32_kernel("pairwise")
    g.set_precision("mixed")
    g.set_solver_tol(1e-10)
    rng = np.random.default_rng(nf)
    fields = 1e-3 * rng.standard_normal((nf, g.pol_atoms, 3))
    one = np.ones((g.pol_atoms, 3))
    alpha = 1.0 / (g.tmatvec(one) - g.tmatvec(one, dodiag=False))
    for block in (True, False):
        g.set_block_cg(block)
        ipd = np.asarray(g.set_external_fields_batch(fields)[0])
        e = g.e_m2d()
        for k in range(nf):
            r = e[0] + fields[k] - g.tmatvec(np.ascontiguousarray(ipd[k][0]))
            assert np.sqrt((alpha * r * r).mean()) < 2e-10

"""The FMM product's kernels by expansion order and column count."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [5, 8, 10, 11, 12])
def test_fmm_columns_do_not_mix(order, tmp_path):
    """The FMM product of two columns is each column's own product bit for bit
    (its M2L kernels by order and column count), and it stays within the
    order's truncation of the direct product."""
    w = synth.water_cluster(1500, seed=5)
    g = OMMPSystem(synth.write_mmp(str(tmp_path / "w.mmp"), w))
    x = np.random.default_rng(order).standard_normal((2, g.pol_atoms, 3))
    d = g.tmatvec(x)
    g.set_fmm(True, order=order)
    y = g.tmatvec(x)
    for k in range(2):
        assert np.array_equal(y[k], g.tmatvec(x[k]))
    assert 0 < np.linalg.norm(y - d) / np.linalg.norm(d) < 0.02


# relative errors of the products of the same cluster by the M2L kernel that
# gave each (target term, source term) pair its own loads
_ERR = {2: 3.10e-3, 3: 1.75e-3, 4: 9.61e-4, 6: 3.26e-4, 7: 1.96e-4, 8: 1.26e-4, 9: 8.32e-5, 10: 5.24e-5}


@pytest.mark.parametrize("order", sorted(_ERR))
def test_fmm_truncation_by_order(order, tmp_path):
    """The FP32 M2L at each order (rows of 10 to 286 terms padded to 16 bytes,
    quads of target terms that straddle two orders, both launch shapes) keeps
    the truncation error that the order has: the same sums, so 1 % above."""
    w = synth.water_cluster(1500, seed=5)
    g = OMMPSystem(synth.write_mmp(str(tmp_path / "w.mmp"), w))
    x = np.random.default_rng(order).standard_normal((2, g.pol_atoms, 3))
    d = g.tmatvec(x)
    g.set_fmm(True, order=order)
    assert np.linalg.norm(g.tmatvec(x) - d) / np.linalg.norm(d) < 1.01 * _ERR[order]


# the same for 8,000 waters, whose trees have levels above the leaves'
_ERR_DEEP = {2: 5.77e-3, 3: 3.61e-3, 5: 1.41e-3, 8: 3.92e-4, 10: 1.91e-4, 12: 9.97e-5}


@pytest.mark.parametrize("order", sorted(_ERR_DEEP))
def test_fmm_truncation_with_translations(order, tmp_path):
    """M2M and L2L, one direction after the other, are the translations that
    sums over all three at once were: the truncation error stays, 1 % above."""
    w = synth.water_cluster(8000, seed=5)
    g = OMMPSystem(synth.write_mmp(str(tmp_path / "w.mmp"), w))
    x = np.random.default_rng(1).standard_normal((2, g.pol_atoms, 3))
    d = g.tmatvec(x)
    g.set_fmm(True, order=order)
    assert np.linalg.norm(g.tmatvec(x) - d) / np.linalg.norm(d) < 1.01 * _ERR_DEEP[order]

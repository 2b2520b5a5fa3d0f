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

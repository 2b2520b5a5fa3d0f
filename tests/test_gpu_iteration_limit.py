"""The FP64 CG at iteration limits of 0, 1 and a few after other solves, its
loop on the device and from the host (csrc/solvers.cu): a limit below 1 leaves
the starting dipoles and reports no iteration, as the reference does
(src/mod_solvers.F90:86-216), and a changed limit reaches a loop that was
captured before."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPError, OMMPSystem, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("size,kernel", [(20, "auto"), (100, "auto"), (300, "auto"), (300, "symmetric")])
def test_limits(tmp_path, size, kernel, graphs):
    g = OMMPSystem(synth.write_mmp(str(tmp_path / "s.mmp"), synth.water_cluster(size, seed=size)))
    g.set_fp64_kernel(kernel)
    g.set_use_graphs(graphs)
    f = 1e-3 * np.random.default_rng(1).standard_normal((g.pol_atoms, 3))
    g.set_external_field(f)
    full, ipd = g.iterations(0), g.ipd.copy()
    assert full > 4
    for limit in (0, 1, 0, 3, -1, full - 1, full, 0):
        g.set_solver_maxiter(limit)
        g.clear_guess()
        if 0 < limit < full:
            with pytest.raises(OMMPError):
                g.set_external_field(f)
        else:
            g.set_external_field(f)
        assert g.iterations(0) == max(0, limit)
        assert len(g.residual_history(0)) == max(0, limit)
        if limit < 1:
            assert not g.ipd.any()
        elif limit == full:
            assert np.array_equal(g.ipd, ipd)
    # a guess stays as it is
    g.set_solver_maxiter(200)
    g.set_external_field(f)
    g.set_solver_maxiter(0)
    ipd = g.ipd.copy()
    g.set_external_field(2 * f)
    assert np.array_equal(g.ipd, ipd) and g.iterations(0) == 0

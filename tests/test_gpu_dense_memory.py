"""Device memory of the inversion solver (csrc/engine.cu): a matrix that is not
positive definite is left to its LU factors, and the FP32 inverse that was tried
first holds no memory beside them: one dense matrix stays."""
import ctypes as C

import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, _lib, synth

pytestmark = pytest.mark.gpu


def free_bytes():
    f, t = C.c_int64(), C.c_int64()
    assert _lib.load().ommp_gpu_device_mem_info(C.byref(f), C.byref(t)) == 0
    return f.value


def test_factors_alone_stay(tmp_path):
    w = synth.water_cluster(400, seed=2)
    w.pol, w.coords = w.pol * 30.0, w.coords * 0.5  # T has negative eigenvalues
    g = OMMPSystem(synth.write_mmp(str(tmp_path / "s.mmp"), w))
    f = 1e-3 * np.random.default_rng(1).standard_normal((g.pol_atoms, 3))
    g.e_m2d()
    matrix = 8 * (3 * g.pol_atoms) ** 2
    before = free_bytes()
    for _ in range(2):
        g.set_external_field(f, solver="inversion")
        assert before - free_bytes() < 1.25 * matrix
    # a geometry with a positive definite T takes the inverse again, and leaves
    # it again
    g.update_coordinates(4.0 * g.cmm)
    g.set_external_field(f, solver="inversion")
    r = g.e_m2d()[0] + f - g.tmatvec(g.ipd[0])
    assert np.linalg.norm(r) < 1e-12 * np.linalg.norm(f)
    g.update_coordinates(0.25 * g.cmm)
    g.set_external_field(f, solver="inversion")
    assert before - free_bytes() < 1.25 * matrix

"""Device allocations that fail, without a GPU: the library's own objects linked
with a stand-in for the CUDA runtime (tests/host/fake_cuda.cpp) whose memory is
the host's and whose kernels do nothing.

Every size that a call allocates is made to fail in turn.  As long as it fails
the call either does without (each time) or reports an error (each time, never
going on with the buffer that it did not get), and once there is memory again
the same call succeeds."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from openmmpol_gb300 import OMMPError, OMMPSystem, _lib, build, synth


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    build.build()
    d = tmp_path_factory.mktemp("fake")
    obj, so = str(d / "fake.o"), str(d / "libommp_fake.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-I", build._cuda_include(), "-c",
                    os.path.join(ROOT, "tests", "host", "fake_cuda.cpp"), "-o", obj], check=True)
    objs = [os.path.join(build.OBJ, s + ".o") for s in build.CU_SOURCES + build.CXX_SOURCES]
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, *objs, obj, "-lpthread", "-ldl", "-lrt"], check=True)
    saved, _lib._lib = _lib._lib, None
    try:
        L = _lib.load(so)
        for name in ("fake_launches", "fake_instantiations", "fake_live"):
            getattr(L, name).restype = C.c_longlong
        L.fake_fail_bytes.argtypes = [C.c_longlong, C.c_longlong]
        yield L
    finally:
        _lib._lib = saved


@pytest.fixture(scope="module")
def path(tmp_path_factory):
    return synth.write_mmp(str(tmp_path_factory.mktemp("sys") / "w.mmp"), synth.water_cluster(1000, seed=3))


def fmm(g):
    g.set_fmm(True, order=8)
    g.set_fmm_lmax(8)


def tmatvec_fmm(g):
    fmm(g)
    g.tmatvec(np.ones((2, g.pol_atoms, 3)))


def e_m2d_fmm(g):
    fmm(g)
    g.e_m2d()


def other(**options):
    """A solve with another solver, product or precision."""
    def call(g):
        g.set_precision(options.get("precision", "fp64"))
        g.set_default_matv(options.get("matv", "direct"))
        f = np.ones((g.pol_atoms, 3))
        if "columns" in options:
            g.set_external_fields_batch(np.ones((options["columns"], *f.shape)))
        else:
            g.set_external_field(f, solver=options.get("solver", "cg"))
    return call


def geometry(g):
    g.update_coordinates(g.cmm)
    other(precision="mixed")(g)


CALLS = {
    "tmatvec_fmm": tmatvec_fmm,
    "e_m2d_fmm": e_m2d_fmm,
    "geometry": geometry,
    "incore": other(matv="incore"),
    "inversion": other(solver="inversion"),
    "diis": other(solver="diis"),
    "mixed": other(precision="mixed"),
    "mixed_batch": other(precision="mixed-ds", columns=5),
    "tmatvec": lambda g: g.tmatvec(np.ones((2, g.pol_atoms, 3))),
    "solve": lambda g: g.set_external_field(np.ones((g.pol_atoms, 3))),
    "batch": lambda g: g.set_external_fields_batch(np.ones((3, g.pol_atoms, 3))),
    "points": lambda g: g.potential_mm2ext(np.ones((300, 3))),
    "static_energy": lambda g: g.get_fixedelec_energy(),
    "static_gradient": lambda g: g.fixedelec_geomgrad(),
    "gradient": lambda g: g.polelec_geomgrad(),
}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_call_survives_failed_allocations(fake, path, name):
    call = CALLS[name]
    g = OMMPSystem(path)
    fake.fake_forget_sizes()
    call(g)
    sizes = (C.c_longlong * 256)()
    n = fake.fake_sizes(sizes, 256)
    g.close()
    live = fake.fake_live()
    wanted = [s for s in sizes[:n] if s > 8]
    # every allocation, by its size and the number of the same size before it
    for size, skip in sorted({(s, wanted[:k].count(s)) for k, s in enumerate(wanted)}):
        g = OMMPSystem(path)
        fake.fake_fail_bytes(size, skip)
        try:
            outcome = []
            for _ in range(3):
                try:
                    call(g)
                    outcome.append("ok")
                except OMMPError as e:
                    outcome.append(e.status)
        finally:
            fake.fake_fail_bytes(0, 0)
        assert len(set(outcome)) == 1, (size, skip, outcome)
        assert fake.fake_last_error() == 0, size  # nothing left for the next call to find
        call(g)
        g.close()
        assert fake.fake_live() == live, size


def test_fmm_streams_that_cannot_be_made(fake, path):
    """The FMM product's second stream and its two events are one set: while an
    event cannot be made the product reports it, and then it works."""
    g = OMMPSystem(path)
    live = fake.fake_live()
    fake.fake_fail_events(1)
    try:
        for k in range(2):
            with pytest.raises(OMMPError, match="streams"):
                tmatvec_fmm(g)
            if k == 0:  # the tree is there
                launches = fake.fake_launches()
        assert fake.fake_launches() == launches
    finally:
        fake.fake_fail_events(0)
    tmatvec_fmm(g)
    g.close()
    assert fake.fake_live() < live


def test_captured_loop_of_kernels_only(fake, path):
    """A CG loop whose captured body holds anything but kernels is not made into
    a graph: the solve goes from the host."""
    g = OMMPSystem(path)
    fake.fake_memset_node(1)
    try:
        made, launches = fake.fake_instantiations(), fake.fake_launches()
        for precision in ("fp64", "mixed"):
            other(precision=precision)(g)
        assert fake.fake_instantiations() == made and fake.fake_launches() > launches
    finally:
        fake.fake_memset_node(0)
    g.clear_guess()
    other()(g)
    assert fake.fake_instantiations() > made
    g.close()

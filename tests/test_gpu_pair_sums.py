"""Double-single pair sums of FP64 accuracy at the edges of their 32- and
128-site tiles, against the CPU oracle: the permanent field (csrc/m2d.cu), the
static energy and gradient (m2m.cu) and the polarization gradient
(grad_sym.cu), for AMOEBA water with all, some and few polarizable sites and
for Wang-AL chains.

Tolerances (2-norm): a pair is within 2^-44 of its largest term; the sums of
charge terms cancel to a tenth (field, forces) or a hundredth (static energy)
of their parts, and the oracle's own FP64 sums carry the same factors of
1e-16: 1e-12 for fields and forces, 1e-11 for the energy."""
import numpy as np
import pytest

from openmmpol_gb300 import OMMPSystem, synth
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def load(tmp_path, kind, size):
    if kind == "chain":
        w = synth.chain_system(n_chains=2, chain_len=25, n_waters=size, seed=size)
    else:
        w = synth.water_cluster(size, seed=size)
        if kind == "oxygens":  # hydrogens carry multipoles only
            w.pol[1::3] = w.pol[2::3] = 0.0
        elif kind == "few":  # whole tiles without a polarizable site
            w.pol[3 * (size // 8):] = 0.0
    p = synth.write_mmp(str(tmp_path / "s.mmp"), w)
    g, o = OMMPSystem(p), OracleSystem(p)
    c = o.cmm
    ef, _, _ = synth.point_charge_field(c[o.polar_mm], w.box_center(), seed=1, n_charges=4, radius=4.0, guard=0.5,
                                        all_sites_bohr=c)
    return g, o, ef


CASES = [("water", 1), ("water", 10), ("water", 11), ("water", 43), ("water", 86), ("water", 128), ("water", 171),
         ("oxygens", 11), ("oxygens", 130), ("few", 24), ("few", 200), ("chain", 1), ("chain", 26), ("chain", 70)]


@pytest.mark.parametrize("kind,size", CASES)
@pytest.mark.parametrize("precision", ["fp64", "mixed-ds"])
def test_matches_oracle(tmp_path, kind, size, precision):
    g, o, ef = load(tmp_path, kind, size)
    g.set_precision(precision)
    if size > 1 or kind != "water":
        assert rel(g.e_m2d(), o.e_m2d()) < 1e-12
        assert abs(g.get_fixedelec_energy() - o.get_fixedelec_energy()) <= 1e-11 * abs(o.get_fixedelec_energy())
        assert rel(g.fixedelec_geomgrad(), o.fixedelec_geomgrad()) < 1e-12
    g.set_external_field(ef)
    o.set_ipd(g.ipd)
    ref = o.polelec_geomgrad()
    gg = g.polelec_geomgrad()
    # a lone molecule has no force from itself: bounded by its dipoles' own terms
    scale = np.linalg.norm(ref) if size > 1 or kind != "water" else np.abs(g.ipd).max() ** 2
    assert np.linalg.norm(gg - ref) < 1e-12 * scale


def test_gradient_of_small_dipoles(tmp_path):
    """The static part of the gradient is linear in the dipoles: scaled far down
    (no permanent field), it keeps its relative accuracy."""
    g, o, ef = load(tmp_path, "water", 60)
    g.set_external_field(np.ldexp(ef, -100), nomm=True, solver="inversion")
    o.set_ipd(g.ipd)
    ref = o.polelec_geomgrad()
    assert np.abs(g.ipd).max() < 1e-28
    assert rel(g.polelec_geomgrad(), ref) < 1e-12

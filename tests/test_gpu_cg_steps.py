"""The fused conjugate-gradient steps (csrc/pcg.cu): solves at the sizes where
a launch shape changes (one CTA for the whole FP64 iteration up to 682 sites,
the symmetric product from 2,400, four lanes or one per site in the finishing
passes around 32,768), every inner preconditioner and FP32 product, one and
two columns, blocks of columns, and systems of different sizes and
preconditioners sharing the launches of the multi-system engine.

A solve ends when the rms of r.(alpha r) is below the tolerance by the
solver's own recursion; the true residual, from the FP64 product, differs by
rounding (CG, ~1e-13) or by a tenth of the tolerance (updated refinement
residuals): twice the tolerance.  The FP64 CG also leaves, like the reference
(src/mod_solvers.F90), as soon as |p.Tp| < 100 eps; r.(alpha r) is at most the
condition number of alpha T (below 4 here) times p.Tp then, so that the rms is
below sqrt(400 eps / 3n)."""
import numpy as np
import pytest

import openmmpol_gb300 as og
from openmmpol_gb300 import OMMPSystem, synth

pytestmark = pytest.mark.gpu
TOL = 1e-10
QUICK = np.sqrt(400 * np.finfo(float).eps)


def load(tmp_path, kind, size, name="s"):
    if kind == "water":
        w = synth.water_cluster(size, seed=size)
    else:
        w = synth.chain_system(n_chains=3, chain_len=20, n_waters=size, seed=size)
    g = OMMPSystem(synth.write_mmp(str(tmp_path / f"{name}.mmp"), w))
    g.set_solver_tol(TOL)
    return g


def field(g, seed):
    return 1e-3 * np.random.default_rng(seed).standard_normal((g.pol_atoms, 3))


def residual(g, f, ipd=None):
    one = np.ones((g.pol_atoms, 3))
    alpha = 1.0 / (g.tmatvec(one) - g.tmatvec(one, dodiag=False))
    mu = (g.ipd if ipd is None else ipd).reshape(-1, g.pol_atoms, 3)
    e = g.e_m2d().reshape(-1, g.pol_atoms, 3) + f
    out = []
    for k in range(mu.shape[0]):
        r = e[k] - g.tmatvec(mu[k])
        out.append(np.sqrt((alpha * r * r).mean()))
    return max(out)


@pytest.mark.parametrize("kind,size", [("water", 1), ("water", 227), ("water", 228), ("water", 333), ("water", 334),
                                       ("water", 500), ("chain", 20), ("chain", 300)])
def test_fp64_cg(tmp_path, kind, size):
    g = load(tmp_path, kind, size)
    f = field(g, size)
    bound = max(2 * TOL, QUICK / np.sqrt(3 * g.pol_atoms))
    for kernel in ("auto", "symmetric", "ordered"):
        g.set_fp64_kernel(kernel)
        g.clear_guess()
        g.set_external_field(f)
        assert residual(g, f) < bound
    g.set_external_field(1.1 * f)  # from the previous dipoles
    assert residual(g, 1.1 * f) < bound


@pytest.mark.parametrize("kind,size", [("water", 1), ("water", 85), ("water", 1000), ("chain", 300)])
@pytest.mark.parametrize("precond", ["diagonal", "block", "near"])
def test_inner_pcg(tmp_path, kind, size, precond):
    g = load(tmp_path, kind, size)
    g.set_precision("mixed")
    g.set_inner_preconditioner(precond)
    f = field(g, size)
    for kernel in ("pairwise", "tiled", "symmetric", "auto"):
        for graphs in (True, False):
            g.set_fp32_kernel(kernel)
            g.set_use_graphs(graphs)
            g.clear_guess()
            g.set_external_field(f)
            assert residual(g, f) < 2 * TOL


@pytest.mark.parametrize("size", [10922, 10923])  # one and four lanes per site from 32,768 sites down
def test_finishing_lanes(tmp_path, size):
    g = load(tmp_path, "water", size)
    f = field(g, size)
    for precision in ("fp64", "mixed"):
        g.set_precision(precision)
        g.clear_guess()
        g.set_external_field(f)
        assert residual(g, f) < max(2 * TOL, QUICK / np.sqrt(3 * g.pol_atoms) if precision == "fp64" else 0.0)


@pytest.mark.parametrize("precond", ["diagonal", "near"])
@pytest.mark.parametrize("nf", [3, 5])
def test_columns(tmp_path, nf, precond):
    g = load(tmp_path, "water", 200)
    g.set_precision("mixed")
    g.set_inner_preconditioner(precond)
    fields = np.stack([field(g, 10 + k) for k in range(nf)])
    for block in (True, False):
        g.set_block_cg(block)
        ipd = g.set_external_fields_batch(fields)[0]
        for k in range(nf):
            assert residual(g, fields[k], np.asarray(ipd)[k]) < 2 * TOL


def test_systems_sharing_launches(tmp_path):
    """More systems than one launch's table holds, of every preconditioner."""
    sizes = [1, 3, 20, 85, 90, 170, 228, 300, 341, 400, 450, 500, 20, 64, 128, 129, 11000, 7]
    systems, fields = [], []
    for k, n in enumerate(sizes):
        g = load(tmp_path, "chain" if k % 5 == 2 else "water", n, f"s{k}")
        g.set_precision("mixed-ds" if k % 2 else "mixed")
        g.set_inner_preconditioner(("diagonal", "block", "near")[k % 3])
        systems.append(g)
        fields.append(field(g, k))
    og.solve_multi(systems, fields)
    for g, f in zip(systems, fields):
        assert residual(g, f) < 2 * TOL


@pytest.mark.parametrize("kind,size", [("water", 340), ("water", 700), ("chain", 352)])
@pytest.mark.parametrize("nf", [3, 9, 16])
def test_column_groups(tmp_path, kind, size, nf):
    """The products of several pairs of columns (symmetric and ordered), and
    the tiled FP32 products of several groups, share a launch (odd counts
    leave a last column, 9 = 8 + 1)."""
    g = load(tmp_path, kind, size)
    g.set_precision("mixed")
    fields = np.stack([field(g, 40 + k) for k in range(nf)])
    for kernel in ("auto", "symmetric", "ordered"):
        g.set_fp64_kernel(kernel)
        ipd = np.asarray(g.set_external_fields_batch(fields)[0])
        for k in range(nf):
            assert residual(g, fields[k], ipd[k]) < 2 * TOL

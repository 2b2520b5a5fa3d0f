"""Performance cases: the calls a QM/MM or MD program makes of this library.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare(case, seed)`` builds what such a program holds before the call
(loaded systems, external fields, QM nuclei, grid points), ``run(state)`` is
one pass through the public entry points and returns everything it computes,
``work(case)`` the bytes and floating-point operations that the path cannot do
without, and ``exact(case, seed)`` the same outputs from plain 64-bit
PyTorch, without this library's code, where that is quick enough.

Kinds of case:

* ``solve``     one polarization solve in an external field (each SCF cycle of
                a QM/MM calculation), cold start, dipoles and energy;
* ``geometry``  a moved geometry: new coordinates, the solve, the energies and,
                where asked for, the forces (an MD or optimisation step);
* ``batch``     many fields on one geometry (several QM densities or states);
* ``gradient``  the polarization forces of a solved system;
* ``qmmm``      one QM/MM cycle with a QM helper: nuclear fields, the solve,
                the potential on a DFT-like grid, nuclear field gradients;
* ``multi``     several uneven systems solved together, as a server does.
"""
import math
import os
import tempfile

import numpy as np
import torch

import openmmpol_gb300 as og
from openmmpol_gb300 import synth

ANG2AU = 1.8897261245650
EXACT_MAX_SITES = 15100        # dense 64-bit solve: (3 n)^2 doubles
EXACT_MAX_GRAD_SITES = 10000


def listed():
    return [
        # the smallest solves: a cluster of 64 waters in the default mode
        # (FP64 CG to 1e-8), where launches and latency count
        dict(name="solve_192_fp64", kind="solve", system="water", size=64, precision="fp64", solver="cg",
             matv="direct", fmm=False, tol=1e-8),
        # a small solute with the dense solver at a new geometry
        dict(name="geometry_1500_inversion", kind="geometry", system="water", size=500, precision="fp64",
             solver="inversion", forces=False, tol=1e-8),
        # a solvated small molecule in the default mode, odd size
        dict(name="solve_5001_fp64", kind="solve", system="water", size=1667, precision="fp64", solver="cg",
             matv="direct", fmm=False, tol=1e-8),
        # a solvated chromophore, mixed precision, tight tolerance
        dict(name="solve_9003_mixed", kind="solve", system="water", size=3001, precision="mixed", solver="cg",
             matv="direct", fmm=False, tol=1e-10),
        # the benchmark's box: 30,000 waters, strict mixed precision
        dict(name="solve_90000_mixed", kind="solve", system="water", size=30000, precision="mixed", solver="cg",
             matv="direct", fmm=False, tol=1e-10),
        # a non-AMOEBA system (Wang-AL chains in water), double-single residuals
        dict(name="solve_chain_10200_mixed_ds", kind="solve", system="chain", size=2600, precision="mixed-ds",
             solver="cg", matv="direct", fmm=False, tol=1e-10),
        # a large box with the fast multipole method
        dict(name="solve_60000_fmm", kind="solve", system="water", size=20000, precision="fp64", solver="cg",
             matv="direct", fmm=True, tol=1e-8),
        # several QM densities on one geometry
        dict(name="batch_24x3003_mixed", kind="batch", system="water", size=1001, fields=24, precision="mixed",
             tol=1e-10),
        # polarization forces of a large box in the mixed modes
        dict(name="gradient_30000_mixed_ds", kind="gradient", system="water", size=10000, precision="mixed-ds",
             tol=1e-10),
        # one FP64 MD step: new coordinates, solve, energies, all forces
        dict(name="geometry_6000_fp64", kind="geometry", system="water", size=2000, precision="fp64",
             solver="cg", forces=True, tol=1e-8),
        # one QM/MM cycle: 40 nuclei, 20,001 grid points
        dict(name="qmmm_9000", kind="qmmm", system="water", size=3000, nuclei=40, points=20001,
             precision="mixed", tol=1e-10),
        # eight uneven systems together
        dict(name="multi_8_mixed_ds", kind="multi", system="water", count=8, smallest=100, largest=5000,
             precision="mixed-ds", tol=1e-10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "fmm", "geometry", "batch", "gradient", "qmmm", "multi"])
    if kind == "solve":
        prec = rng.choice(["fp64", "mixed", "mixed-ds"])
        c = dict(kind="solve", system=rng.choice(["water", "water", "chain"]), precision=prec, solver="cg",
                 matv="direct", fmm=False, tol=1e-8 if prec == "fp64" else 1e-10)
        top = {"fp64": 5000, "mixed": 20000, "mixed-ds": 30000}[prec]
        c["size"] = _log_int(rng, 12, top if c["system"] == "water" else 2600)
        if prec == "fp64" and c["size"] <= 600:
            c["solver"] = rng.choice(["cg", "diis"])
            c["matv"] = rng.choice(["direct", "incore"])
        return c
    if kind == "fmm":
        return dict(kind="solve", system="water", size=_log_int(rng, 2000, 20000), precision="fp64", solver="cg",
                    matv="direct", fmm=True, tol=1e-8)
    if kind == "geometry":
        solver = rng.choice(["cg", "cg", "inversion"])
        if solver == "inversion":
            return dict(kind="geometry", system="water", size=_log_int(rng, 12, 500), precision="fp64",
                        solver=solver, forces=False, tol=1e-8)
        prec = rng.choice(["fp64", "mixed", "mixed-ds"])
        return dict(kind="geometry", system="water", size=_log_int(rng, 12, 3000), precision=prec, solver="cg",
                    forces=True, tol=1e-8 if prec == "fp64" else 1e-10)
    if kind == "batch":
        return dict(kind="batch", system="water", size=_log_int(rng, 30, 2000), fields=rng.randint(2, 32),
                    precision=rng.choice(["fp64", "mixed", "mixed-ds"]), tol=1e-10)
    if kind == "gradient":
        prec = rng.choice(["fp64", "mixed-ds"])
        return dict(kind="gradient", system=rng.choice(["water", "water", "chain"]), precision=prec, tol=1e-10,
                    size=_log_int(rng, 12, 2600))
    if kind == "qmmm":
        return dict(kind="qmmm", system="water", size=_log_int(rng, 60, 5000), nuclei=rng.randint(3, 60),
                    points=_log_int(rng, 500, 40000), precision=rng.choice(["fp64", "mixed", "mixed-ds"]), tol=1e-10)
    small = _log_int(rng, 12, 300)
    return dict(kind="multi", system="water", count=rng.randint(2, 10), smallest=small,
                largest=_log_int(rng, 2 * small, 5000), precision=rng.choice(["mixed", "mixed-ds"]), tol=1e-10)


# --- systems -------------------------------------------------------------------
def _chain_shape(size):
    """(chains, sites per chain) of a chain system with `size` waters."""
    return max(1, size // 108), 100 if size >= 108 else max(4, size)


def _sites(case):
    if case["system"] == "water":
        return 3 * case["size"]
    nc, ln = _chain_shape(case["size"])
    return nc * ln + 3 * case["size"]


def _multi_sizes(case):
    k, a, b = case["count"], math.log(case["smallest"]), math.log(case["largest"])
    return [int(round(math.exp(a + (b - a) * i / max(1, k - 1)))) for i in range(k)]


def _make(system, size, seed):
    """The system's arrays, coordinates rounded as the .mmp file states them."""
    if system == "water":
        w = synth.water_cluster(size, seed=seed)
    else:
        nc, ln = _chain_shape(size)
        w = synth.chain_system(nc, ln, size, seed=seed)
    text = [" ".join(r) for r in np.char.mod("%.10f", w.coords)] if size < 200 else ["%.10f %.10f %.10f" % t for t in
                                                                                   map(tuple, w.coords.tolist())]
    w.coords = np.array(" ".join(text).split(), dtype=np.float64).reshape(-1, 3)
    return w, text


def _write(path, w, text):
    """A revision-3 .mmp file, as synth.write_mmp writes it."""
    mm = w.mm_atoms
    L = ["3", "0", "0", "1" if w.amoeba else "0", "0"] + ["0"] * 17 + [str(mm), "0"]
    L += [str(v) for v in w.z.tolist()]
    L += text
    L += ["1"] * mm
    fmt = " ".join(["%.8f"] * w.mult.shape[1])
    L += [fmt % tuple(m) for m in (w.mult[:3].tolist() if w.amoeba else w.mult.tolist())] * (mm // 3 if w.amoeba else 1)
    L += ["%.8f" % p for p in w.pol.tolist()]
    L += ["%d %d %d %d %d %d %d %d" % tuple(b) for b in w.bonds.tolist()]
    if w.amoeba:
        L += ["%d %d %d 117*0" % tuple(g) for g in w.groups.tolist()]
        L += ["%d %d %d %d" % tuple(f) for f in w.frames.tolist()]
    with open(path, "w") as f:
        f.write("\n".join(L))
        f.write("\n")


def _load(system, size, seed):
    w, text = _make(system, size, seed)
    fd, path = tempfile.mkstemp(suffix=".mmp")
    os.close(fd)
    try:
        _write(path, w, text)
        return w, og.OMMPSystem(path)
    finally:
        os.unlink(path)


def _field(w, seed):
    c = w.coords * ANG2AU
    ef, _, _ = synth.point_charge_field(c, w.box_center(), seed=seed, all_sites_bohr=c)
    return ef


def _nuclei(case, w, seed):
    """Positions (bohr), charges and numbers of QM nuclei near the centre."""
    c = w.coords * ANG2AU
    _, q, pos = synth.point_charge_field(c[:1], w.box_center(), seed=seed, n_charges=case["nuclei"], radius=8.0,
                                         all_sites_bohr=c)
    z = np.random.default_rng(seed).choice([1, 6, 7, 8], size=case["nuclei"]).astype(np.int32)
    return pos, z.astype(np.float64) + q, z


def _grid(case, w, pos, seed):
    """Points (bohr) around the nuclei at DFT-like distances, none within
    0.5 bohr of a site."""
    rng = np.random.default_rng(seed)
    c = w.coords * ANG2AU
    c = c[np.linalg.norm(c - pos.mean(0), axis=1) < 40.0]
    out = np.zeros((0, 3))
    while len(out) < case["points"]:
        k = 2048
        v = rng.standard_normal((k, 3))
        v *= (np.exp(rng.uniform(math.log(0.05), math.log(8.0), k)) / np.linalg.norm(v, axis=1))[:, None]
        p = pos[rng.integers(len(pos), size=k)] + v
        if len(c):
            r2 = (p * p).sum(1)[:, None] - 2.0 * p @ c.T + (c * c).sum(1)[None, :]
            p = p[r2.min(1) > 0.25]
        out = np.concatenate([out, p])
    return np.ascontiguousarray(out[: case["points"]])


def _setup(case, g):
    g.set_solver_tol(case["tol"])
    g.set_precision(case["precision"])


def prepare(case, seed):
    og.set_verbose(0)
    kind = case["kind"]
    if kind == "multi":
        ws, gs, fs = [], [], []
        for i, n in enumerate(_multi_sizes(case)):
            w, g = _load("water", n, seed * 16 + i)
            _setup(case, g)
            ws.append(w)
            gs.append(g)
            fs.append(_field(w, seed * 16 + i))
        return dict(case=case, systems=gs, fields=fs)
    w, g = _load(case["system"], case["size"], seed)
    _setup(case, g)
    s = dict(case=case, g=g)
    if kind == "solve":
        if case["matv"] != "direct":
            g.set_default_matv(case["matv"])
        if case["fmm"]:
            g.set_fmm(True)
        s["field"] = _field(w, seed)
    elif kind == "geometry":
        s["field"] = _field(w, seed)
        s["coords"] = w.coords * ANG2AU
    elif kind == "batch":
        s["fields"] = np.stack([_field(w, seed * 64 + k) for k in range(case["fields"])])
    elif kind == "gradient":
        g.set_external_field(_field(w, seed))
    elif kind == "qmmm":
        pos, q, z = _nuclei(case, w, seed)
        s["pos"] = pos
        s["helper"] = og.OMMPQmHelper(pos, q, z)
        s["grid"] = _grid(case, w, pos, seed)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "multi":
        for g in s["systems"]:
            g.clear_guess()
        e, _ = og.solve_multi(s["systems"], s["fields"])
        return dict(ipd=[g.ipd for g in s["systems"]], energy=e)
    g = s["g"]
    if kind == "solve":
        g.clear_guess()
        g.set_external_field(s["field"], solver=case["solver"])
        return dict(ipd=g.ipd, energy=g.get_polelec_energy())
    if kind == "geometry":
        g.update_coordinates(s["coords"])
        g.set_external_field(s["field"], solver=case["solver"])
        out = dict(ipd=g.ipd, energy=g.get_polelec_energy(), static=g.get_fixedelec_energy())
        if case["forces"]:
            out["pol_forces"] = g.polelec_geomgrad()
            out["static_forces"] = g.fixedelec_geomgrad()
        return out
    if kind == "batch":
        ipd, e = g.set_external_fields_batch(s["fields"])
        return dict(ipd=ipd, energy=e)
    if kind == "gradient":
        return dict(pol_forces=g.polelec_geomgrad())
    h = s["helper"]
    h.update_coord(s["pos"])
    h.prepare_qm_ele_ene(g)
    field = h.E_n2p
    g.clear_guess()
    g.set_external_field(field)
    h.prepare_qm_ele_grd(g)
    return dict(ipd=g.ipd, energy=g.get_polelec_energy(), E_n2p=field, V_m2n=h.V_m2n, V_grid=g.potential_mmpol2ext(s["grid"]),
                E_m2n=h.E_m2n, E_p2n=h.E_p2n, E_n2m=h.E_n2m, G_n2m=h.G_n2m, H_n2m=h.H_n2m)


# --- work ----------------------------------------------------------------------
def _solve_flops(case, n, cols=1):
    # conventional 45 flop per ordered pair and product; 8 products reach 1e-8
    # and 10 reach 1e-10 with a good preconditioner
    p = 45.0 * n * n
    its = 8 if case["tol"] > 1e-9 else 10
    if case.get("solver") == "inversion":
        return 2.0 / 3.0 * (3.0 * n) ** 3
    if case.get("fmm"):
        return its * 27.0 * 25.0 * 45.0 * n
    return its * p * cols


def work(case):
    kind = case["kind"]
    if kind == "multi":
        ns = [3 * k for k in _multi_sizes(case)]
        return {"bytes": sum(100.0 * n for n in ns), "flops": sum(_solve_flops(case, n) for n in ns)}
    n = _sites(case)
    per_pair_static = 100.0 if case["system"] == "water" else 30.0
    w = {"bytes": 8.0 * (3 + 3 + 2 + 6) * n, "flops": 0.0}
    if kind in ("solve", "qmmm"):
        w["flops"] = _solve_flops(case, n)
    if kind == "batch":
        w = {"bytes": 8.0 * 9 * n * case["fields"], "flops": _solve_flops(case, n, case["fields"])}
    if kind == "geometry":
        w["flops"] = _solve_flops(case, n) + 2 * per_pair_static * n * n
        if case["forces"]:
            w["flops"] += (302.0 + 300.0) * n * n
            w["bytes"] += 48.0 * n
    if kind == "gradient":
        w["flops"] = 302.0 * n * n
    if kind == "qmmm":
        w["flops"] += 60.0 * n * (case["points"] + 2.0 * case["nuclei"])
        w["bytes"] += 8.0 * (4.0 * case["points"] + 19.0 * n)
    return w


# --- the same in plain 64-bit PyTorch ------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Model:
    """One system in plain 64-bit PyTorch: AMOEBA water or Wang-AL chains."""

    def __init__(self, w):
        dev = _dev()
        self.amoeba = w.amoeba
        self.R = torch.tensor(w.coords * ANG2AU, dtype=torch.float64, device=dev)
        self.n = len(w.coords)
        pol = np.array([float("%.8f" % p) for p in w.pol])
        self.alpha = torch.tensor(pol * ANG2AU ** 3 if w.amoeba else pol, dtype=torch.float64, device=dev)
        self.th = self.alpha ** (1.0 / 6.0) * (1.0 if w.amoeba else math.sqrt(2.5874))
        mult = np.array([[float("%.8f" % v) for v in r] for r in (w.mult[:3] if w.amoeba else w.mult)])
        if w.amoeba:
            mult[:, 4:] /= 3.0
            mult = np.tile(mult, (self.n // 3, 1))
            self.local = torch.tensor(mult, dtype=torch.float64, device=dev)
            ex = [(i, j) for i in range(3) for j in range(3) if i != j]
            base = 3 * np.arange(self.n // 3)
            self.ex = torch.tensor(np.concatenate([np.stack([base + i, base + j], 1) for i, j in ex]), device=dev)
        else:
            self.q = torch.tensor(mult[:, 0], dtype=torch.float64, device=dev)
            nb = [[int(b) - 1 for b in r if b] for r in w.bonds]
            ex = set()
            for i, r in enumerate(nb):  # one and two bonds apart
                for j in r:
                    ex.add((i, j))
                    ex.update((i, k) for k in nb[j] if k != i)
            self.ex = torch.tensor(sorted(ex), device=dev)

    def lab(self, R):
        """q [n], mu [n, 3], Q [n, 3, 3] in the lab frame (bisector on O,
        z-then-x on H)."""
        O, H1, H2 = R[0::3], R[1::3], R[2::3]

        def frame(u, v):
            ez = u / u.norm(dim=1, keepdim=True)
            ex = v - (v * ez).sum(1, keepdim=True) * ez
            ex = ex / ex.norm(dim=1, keepdim=True)
            return torch.stack([ex, torch.linalg.cross(ez, ex), ez], dim=2)

        a, b = H1 - O, H2 - O
        na, nb = a.norm(dim=1, keepdim=True), b.norm(dim=1, keepdim=True)
        F = torch.stack([frame(nb * a + na * b, b), frame(O - H1, H2 - H1), frame(O - H2, H1 - H2)], 1).reshape(-1, 3, 3)
        m = self.local
        Q0 = m[:, [4, 5, 7, 5, 6, 8, 7, 8, 9]].reshape(-1, 3, 3)
        return m[:, 0], (F @ m[:, 1:4, None])[:, :, 0], F @ Q0 @ F.transpose(1, 2)

    def chunks(self, cols=None):
        step = max(1, int(1.2e7 // (cols or self.n)))
        return [(a, min(self.n, a + step)) for a in range(0, self.n, step)]

    def kernels(self, R, a, b, damped=True):
        """d [rows, n, 3] and r^-3, r^-5, r^-7 (damped), the self pairs zero."""
        d = R[a:b, None, :] - R[None, :, :]
        me = torch.arange(a, b, device=R.device)
        eye = torch.zeros(b - a, self.n, dtype=torch.bool, device=R.device)
        eye[torch.arange(b - a, device=R.device), me] = True
        r2 = (d * d).sum(-1).masked_fill(eye, 1.0)
        r = r2.sqrt()
        k1 = 1.0 / r
        k3 = k1 / r2
        k5 = k3 / r2
        k7 = k5 / r2
        if damped:
            u = r / (self.th[a:b, None] * self.th[None, :])
            if self.amoeba:
                x = 0.39 * u ** 3
                e = torch.exp(-x)
                k3, k5, k7 = k3 * (1 - e), k5 * (1 - (1 + x) * e), k7 * (1 - (1 + x + 0.6 * x * x) * e)
            else:
                c = u.clamp(max=1.0)
                k3, k5 = k3 * (4 * c ** 3 - 3 * c ** 4), k5 * c ** 4
        out = [k.masked_fill(eye, 0.0) for k in (k1, k3, k5, k7)]
        return d, out

    def excluded(self, a, b):
        e = self.ex[(self.ex[:, 0] >= a) & (self.ex[:, 0] < b)]
        m = torch.ones(b - a, self.n, dtype=torch.float64, device=e.device)
        m[e[:, 0] - a, e[:, 1]] = 0.0
        return m

    def static_field_rows(self, R, lab, a, b):
        d, (_, k3, k5, k7) = self.kernels(R, a, b)
        s = self.excluded(a, b)
        if not self.amoeba:
            return torch.einsum("ij,ijk->ik", s * k3 * self.q[None, :], d)
        q, mu, Q = lab
        k3, k5, k7 = s * k3, s * k5, s * k7
        md = torch.einsum("ijk,jk->ij", d, mu)
        t = torch.einsum("jkl,ijl->ijk", Q, d)
        c = q[None, :] * k3 + 3 * md * k5 + 15 * (t * d).sum(-1) * k7
        return torch.einsum("ij,ijk->ik", c, d) - k3 @ mu - 6 * torch.einsum("ij,ijk->ik", k5, t)

    def pol_field_rows(self, R, x, a, b):
        """Field of the dipoles x [n, 3] at the rows."""
        d, (_, k3, k5, _) = self.kernels(R, a, b)
        if not self.amoeba:
            s = self.excluded(a, b)
            k3, k5 = s * k3, s * k5
        md = torch.einsum("ijk,jk->ij", d, x)
        return 3 * torch.einsum("ij,ijk->ik", k5 * md, d) - k3 @ x

    def solve(self, fields):
        """E_M2D and the dipoles [len(fields), n, 3], residual near 1e-15."""
        lab = self.lab(self.R) if self.amoeba else None
        E = torch.cat([self.static_field_rows(self.R, lab, a, b) for a, b in self.chunks()])
        n = self.n
        T = torch.empty(3 * n, 3 * n, dtype=torch.float64, device=self.R.device)
        for a, b in self.chunks():
            d, (_, k3, k5, _) = self.kernels(self.R, a, b)
            if not self.amoeba:
                s = self.excluded(a, b)
                k3, k5 = s * k3, s * k5
            blk = -3 * k5[:, :, None, None] * d[:, :, :, None] * d[:, :, None, :]
            for k in range(3):
                blk[:, :, k, k] += k3
            T[3 * a:3 * b] = blk.permute(0, 2, 1, 3).reshape(3 * (b - a), 3 * n)
        al = self.alpha.repeat_interleave(3)[:, None]
        T.diagonal().add_(1.0 / al[:, 0])
        rhs = torch.stack([(E + torch.as_tensor(f, dtype=torch.float64, device=E.device)).reshape(-1) for f in fields], 1)
        x = al * rhs
        r = rhs - T @ x
        z = al * r
        p = z.clone()
        g = (r * z).sum(0)
        g0 = g.clone()
        for _ in range(200):
            h = T @ p
            st = g / (p * h).sum(0)
            x = x + st * p
            r = r - st * h
            z = al * r
            gn = (r * z).sum(0)
            if bool((gn <= 1e-31 * g0).all()):
                break
            p = z + (gn / g) * p
            g = gn
        return E, x.T.reshape(len(fields), n, 3)

    def forces(self, mu):
        """Gradient of the polarization energy at the dipoles mu."""
        R = self.R.clone().requires_grad_(True)
        total = torch.zeros_like(self.R)
        for a, b in self.chunks(8 * self.n):
            lab = self.lab(R) if self.amoeba else None
            u = 0.5 * (mu[a:b] * self.pol_field_rows(R, mu, a, b)).sum() + \
                (mu[a:b] * self.static_field_rows(R, lab, a, b)).sum()
            total -= torch.autograd.grad(u, R)[0]
        return total

    def static_rows(self, R, a, b):
        """Energy of the rows' multipoles in the others', each pair once per row."""
        q, m, Q = self.lab(R)
        d, (k1, k3, k5, k7) = self.kernels(R, a, b, damped=False)
        r2 = (d * d).sum(-1)
        k9 = torch.where(k7 > 0, k7 / torch.where(k7 > 0, r2, torch.ones_like(r2)), k7)
        s = self.excluded(a, b)
        qi, mi, Qi = q[a:b], m[a:b], Q[a:b]
        bj = torch.einsum("ijk,jk->ij", d, m)
        ai = torch.einsum("ijk,ik->ij", d, mi)
        tj = torch.einsum("jkl,ijl->ijk", Q, d)
        ti = torch.einsum("ikl,ijl->ijk", Qi, d)
        sj, si = (tj * d).sum(-1), (ti * d).sum(-1)
        V = q[None] * k1 + bj * k3 + 3 * sj * k5
        c = q[None] * k3 + 3 * bj * k5 + 15 * sj * k7
        u = qi[:, None] * V - c * ai + (mi @ m.T) * k3 + 6 * k5 * torch.einsum("ik,ijk->ij", mi, tj)
        u = u + 3 * q[None] * k5 * si - 6 * k5 * torch.einsum("ijk,jk->ij", ti, m) + 15 * bj * si * k7
        u = u - 60 * k7 * (ti * tj).sum(-1) + 105 * si * sj * k9 + 6 * k5 * (Qi.reshape(-1, 9) @ Q.reshape(-1, 9).T)
        return (0.5 * s * u).sum()

    def static(self, grad):
        R = self.R.clone().requires_grad_(grad)
        e, total = 0.0, torch.zeros_like(self.R)
        for a, b in self.chunks(8 * self.n):
            u = self.static_rows(R, a, b)
            e += float(u.detach())
            if grad:
                total += torch.autograd.grad(u, R)[0]
        return e, total

    def potential(self, mu, pts, field):
        """Potential (or field) of the static multipoles and of the dipoles
        mu at pts, separately."""
        P = torch.as_tensor(pts, dtype=torch.float64, device=self.R.device)
        q, m, Q = self.lab(self.R)
        out = [[], []]
        for a in range(0, len(P), max(1, int(1.2e7 // self.n))):
            d = P[a:a + max(1, int(1.2e7 // self.n)), None, :] - self.R[None]
            r2 = (d * d).sum(-1)
            k1 = r2.rsqrt()
            k3 = k1 / r2
            k5 = k3 / r2
            k7 = k5 / r2
            md = torch.einsum("ijk,jk->ij", d, m)
            t = torch.einsum("jkl,ijl->ijk", Q, d)
            s = (t * d).sum(-1)
            pd = torch.einsum("ijk,jk->ij", d, mu)
            if field:
                c = q[None] * k3 + 3 * md * k5 + 15 * s * k7
                out[0].append(torch.einsum("ij,ijk->ik", c, d) - k3 @ m - 6 * torch.einsum("ij,ijk->ik", k5, t))
                out[1].append(3 * torch.einsum("ij,ijk->ik", k5 * pd, d) - k3 @ mu)
            else:
                out[0].append((q[None] * k1 + md * k3 + 3 * s * k5).sum(1))
                out[1].append((pd * k3).sum(1))
        return [torch.cat(o) for o in out]


def _exact_nuclei(R, pos, q):
    """Field, its gradient (xx, xy, yy, xz, yz, zz) and Hessian (the same order,
    xxx, xxy, xxz, xyy, xyz, xzz, yyy, yyz, yzz, zzz) of the nuclei at R."""
    d = R[:, None, :] - torch.as_tensor(pos, device=R.device)[None]
    q = torch.as_tensor(q, device=R.device)[None]
    r2 = (d * d).sum(-1)
    k3 = q * r2 ** -1.5
    k5, k7 = k3 / r2, k3 / r2 / r2
    x = d.unbind(-1)
    E = torch.einsum("ij,ijk->ik", k3, d)
    G = torch.stack([(3 * k5 * x[a] * x[b] - (k3 if a == b else 0.0)).sum(1)
                     for a, b in ((0, 0), (0, 1), (1, 1), (0, 2), (1, 2), (2, 2))], 1)
    H = []
    for a, b, c in ((0, 0, 0), (0, 0, 1), (0, 0, 2), (0, 1, 1), (0, 1, 2), (0, 2, 2), (1, 1, 1), (1, 1, 2), (1, 2, 2),
                    (2, 2, 2)):
        e = 15 * k7 * x[a] * x[b] * x[c]
        for i, j, k in ((a, b, c), (a, c, b), (b, c, a)):
            if i == j:
                e = e - 3 * k5 * x[k]
        H.append(e.sum(1))
    return E, G, torch.stack(H, 1)


def _np(t):
    return t.detach().cpu().numpy()


def _sets(model, mu):
    """Dipoles [k, n, 3] as the library returns them (D and P for AMOEBA)."""
    return np.repeat(_np(mu)[:, None], 2 if model.amoeba else 1, axis=1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "multi":
        if 3 * case["largest"] > EXACT_MAX_SITES:
            return None
        ipd, en = [], []
        for i, n in enumerate(_multi_sizes(case)):
            w, _ = _make("water", n, seed * 16 + i)
            m = _Model(w)
            E, mu = m.solve([_field(w, seed * 16 + i)])
            ipd.append(_sets(m, mu)[0])
            en.append(float(-0.5 * (mu[0] * E).sum()))
        return dict(ipd=ipd, energy=np.array(en))
    n = _sites(case)
    if n > EXACT_MAX_SITES or case.get("fmm"):
        return None
    w, _ = _make(case["system"], case["size"], seed)
    m = _Model(w)
    if kind == "batch":
        E, mu = m.solve([_field(w, seed * 64 + k) for k in range(case["fields"])])
        return dict(ipd=_sets(m, mu), energy=_np(-0.5 * (mu * E[None]).sum((1, 2))))
    if kind == "qmmm":
        pos, q, _ = _nuclei(case, w, seed)
        En, Gn, Hn = _exact_nuclei(m.R, pos, q)
        E, mu = m.solve([En])
        V = m.potential(mu[0], pos, False)
        Vg = m.potential(mu[0], _grid(case, w, pos, seed), False)
        F = m.potential(mu[0], pos, True)
        return dict(ipd=_sets(m, mu)[0], energy=float(-0.5 * (mu[0] * E).sum()), E_n2p=_np(En), V_m2n=_np(V[0]),
                    V_grid=_np(Vg[0] + Vg[1]), E_m2n=_np(F[0]), E_p2n=_np(F[1]), E_n2m=_np(En), G_n2m=_np(Gn),
                    H_n2m=_np(Hn))
    E, mu = m.solve([_field(w, seed)])
    if kind == "gradient":
        return dict(pol_forces=_np(m.forces(mu[0]))) if n <= EXACT_MAX_GRAD_SITES else None
    out = dict(ipd=_sets(m, mu)[0], energy=float(-0.5 * (mu[0] * E).sum()))
    if kind == "geometry":
        e, g = m.static(case["forces"])
        out["static"] = e
        if case["forces"]:
            out["pol_forces"] = _np(m.forces(mu[0]))
            out["static_forces"] = _np(g)
    return out

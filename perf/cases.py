"""The work that users of this framework have it do, as cases that can be timed.

Every case goes through the Python entry points: md.atoms / md.nvt /
md.min_lbfgs, and the System and Batch handles behind them.  A pass starts
from the same positions and velocities each time, so it can be repeated.

Mixed-precision systems hold FP32 forces and hand everything out in double
arrays; their outputs are given as float32, the type they were computed in.
The outputs of FP64 systems are given as they come.
"""
import math
import os
import tempfile

import numpy as np
import torch

from mapp4py_gb300 import _lib, md, precond

KB = 8.617330350e-5          # eV/K
FS = 1.0 / 10.180505671156723  # 1 fs in A sqrt(amu/eV)
MASS = np.array([63.5, 63.5])
NR = NRHO = 5000
RC, DR, DRHO = 5.5, 5.5 / 5000, 0.01
SKIN = 0.5
ROW = 54.0  # neighbours inside the cutoff of an FCC atom, for work()


# ------------------------------------------------------------------ cases
def _nvt(name, precision, n, steps, T, **more):
    c = {"name": name, "kind": "nvt", "precision": precision, "nx": n[0], "ny": n[1], "nz": n[2], "steps": steps,
         "T": T, "sigma": 0.05, "vac": 0.0, "tilt": 0.0, "xB": 0.5, "pairwise": False, "api": "system"}
    c.update(more)
    return c


def listed():
    return [
        # one force call on a small cell with new positions: a driver that
        # moves the atoms itself and asks for energy, forces and stress
        {"name": "force_fp64_500", "kind": "force", "precision": "fp64", "nx": 5, "ny": 5, "nz": 5, "sigma": 0.05,
         "vac": 0.0, "tilt": 0.0, "xB": 0.5, "pairwise": False},
        # md.nvt at its default precision on a small single-element crystal
        _nvt("md_nvt_fp64_4000", "fp64", (10, 10, 10), 100, 300.0, xB=0.0, sigma=0.0, api="md"),
        # the same precision on a large alloy (a reference trajectory)
        _nvt("nvt_fp64_256000", "fp64", (40, 40, 40), 10, 600.0),
        # mixed-precision MD of a small cell, where launches count
        _nvt("md_nvt_mixed_4000", "mixed", (10, 10, 10), 100, 600.0, api="md"),
        # a strained, tilted cell with vacancies and a Finnis-Sinclair
        # potential (a density function for every pair of elements)
        _nvt("nvt_mixed_fs_tilted", "mixed", (20, 20, 20), 100, 600.0, vac=0.01, tilt=0.02, pairwise=True),
        # MD of a quarter of a million atoms
        _nvt("nvt_mixed_256000", "mixed", (40, 40, 40), 50, 600.0),
        # the headline workload: NVT of two million atoms
        _nvt("nvt_mixed_2048000", "mixed", (80, 80, 80), 50, 600.0),
        # many independent cells of 500 to 32,000 atoms at their own temperatures
        {"name": "batch_nvt_128", "kind": "batch_nvt", "cells": 128, "nmin": 500, "nmax": 32000, "steps": 20},
        # md.min_lbfgs at its defaults on a small disordered cell
        {"name": "md_lbfgs_fp64_4000", "kind": "lbfgs", "precision": "fp64", "nx": 10, "ny": 10, "nz": 10,
         "sigma": 0.1, "vac": 0.01, "tilt": 0.0, "xB": 0.5, "pairwise": False, "m": 2, "iters": 10, "api": "md"},
        # the first iterations of relaxing a large disordered alloy
        {"name": "lbfgs_mixed_253000", "kind": "lbfgs", "precision": "mixed", "nx": 40, "ny": 40, "nz": 40,
         "sigma": 0.15, "vac": 0.01, "tilt": 0.0, "xB": 0.5, "pairwise": False, "m": 10, "iters": 10,
         "api": "system"},
        # relaxing many cells at once with the learned preconditioner
        {"name": "batch_lbfgs_64", "kind": "batch_lbfgs", "cells": 64, "nmin": 1000, "nmax": 16000, "m": 10,
         "iters": 10, "net": True},
        # constant-stress MD: the box moves and the list is built every step
        {"name": "nst_mixed_32000", "kind": "nst", "precision": "mixed", "nx": 20, "ny": 20, "nz": 20,
         "sigma": 0.05, "vac": 0.0, "tilt": 0.0, "xB": 0.5, "pairwise": False, "T": 600.0, "steps": 20},
    ]


def draw(rng):
    def side(most):
        # repeats per axis from 4 up, near a log-uniform volume
        cells = math.exp(rng.uniform(math.log(64.0), math.log(float(most) ** 3)))
        s = cells ** (1.0 / 3.0)
        return [max(4, int(round(s * math.exp(rng.uniform(-0.25, 0.25))))) for _ in range(3)]

    def shape(c, most):
        n = side(most)
        while n[0] * n[1] * n[2] > most ** 3:
            n[n.index(max(n))] -= 1
        c.update(nx=n[0], ny=n[1], nz=n[2], sigma=rng.uniform(0.03, 0.12), vac=rng.choice([0.0, rng.uniform(0.0, 0.03)]),
                 tilt=rng.choice([0.0, 0.0, rng.uniform(0.005, 0.03)]), xB=rng.uniform(0.0, 1.0),
                 pairwise=rng.random() < 0.25)
        return c

    kind = rng.choice(["force", "nvt", "nvt", "nvt", "nvt", "batch_nvt", "lbfgs", "batch_lbfgs", "nst"])
    if kind == "force":
        return shape({"kind": kind, "precision": rng.choice(["fp64", "mixed"])}, 50)
    if kind == "nvt":
        p = rng.choice(["fp64", "mixed", "mixed"])
        c = shape({"kind": kind, "precision": p, "api": rng.choice(["system", "md"])}, 40 if p == "fp64" else 78)
        c.update(steps=rng.randint(8, 12) if p == "fp64" else rng.randint(8, 50), T=rng.uniform(100.0, 1200.0))
        return c
    if kind == "batch_nvt":
        return {"kind": kind, "cells": rng.randint(2, 120), "nmin": 500, "nmax": rng.choice([4000, 16000, 30000]),
                "steps": rng.randint(8, 20)}
    if kind == "lbfgs":
        p = rng.choice(["fp64", "mixed"])
        c = shape({"kind": kind, "precision": p, "api": rng.choice(["system", "md"])}, 20 if p == "fp64" else 39)
        c.update(m=rng.choice([2, 5, 10]), iters=rng.randint(4, 8))
        return c
    if kind == "batch_lbfgs":
        return {"kind": kind, "cells": rng.randint(2, 60), "nmin": 1000, "nmax": rng.choice([4000, 16000]), "m": 10,
                "iters": rng.randint(4, 8), "net": rng.random() < 0.5}
    c = shape({"kind": "nst", "precision": rng.choice(["fp64", "mixed"])}, 19)
    c.update(T=rng.uniform(200.0, 900.0), steps=rng.randint(8, 20))
    return c


# ------------------------------------------------------------------ inputs
def _knots(pairwise):
    """F, rho[source][at], rphi on the grids of an analytic A/B alloy: Morse
    pair term, exponential density, -c sqrt(rho) embedding, cubic switch."""
    r = np.arange(NR) * DR
    rh = np.arange(NRHO) * DRHO
    t = np.clip((r - 5.0) / 0.5, 0.0, 1.0)
    sw = 1.0 - 3.0 * t * t + 2.0 * t * t * t
    par = ((0.35, 2.55, 1.2), (0.42, 2.75, 1.5))
    F = np.stack([-p[2] * np.sqrt(rh) for p in par])
    ph = [p[0] * (np.exp(-2.8 * (r - p[1])) - 2.0 * np.exp(-1.4 * (r - p[1]))) * sw for p in par]
    de = [np.exp(-3.0 * (r / p[1] - 1.0)) * sw for p in par]
    # a Finnis-Sinclair potential: the density of a source also depends on the element it acts at
    rho = np.stack([np.stack([de[i] * (1.0 if i == j or not pairwise else 0.9 + 0.1 * i) for j in range(2)])
                    for i in range(2)])
    rphi = np.stack([np.stack([r * 0.5 * (ph[i] + ph[j]) for j in range(2)]) for i in range(2)])
    return F, rho, rphi


def _force_field(pairwise):
    F, rho, rphi = _knots(pairwise)
    return _lib.ForceField.knots(NR, NRHO, DR, DRHO, F, rho, rphi)


def _setfl(atoms, pairwise):
    """The potential given to md.atoms as a setfl (or Finnis-Sinclair) file."""
    F, rho, rphi = _knots(pairwise)
    fd, path = tempfile.mkstemp(suffix=".fs" if pairwise else ".setfl")
    with os.fdopen(fd, "w") as f:
        f.write("analytic A/B alloy\nMorse pair term, exponential density\ncubic switch over 5.0-5.5 A\n2 A B\n")
        f.write("%d %.17e %d %.17e %.17e\n" % (NRHO, DRHO, NR, DR, RC))

        def block(a):
            f.write("\n".join("%.17e" % v for v in a) + "\n")

        for i in range(2):
            f.write("29 63.5 3.615 fcc\n")
            block(F[i])
            for j in range(2 if pairwise else 1):
                block(rho[i, j])
        for i in range(2):
            for j in range(i + 1):
                block(rphi[i, j])
    (atoms.ff_eam_fs if pairwise else atoms.ff_eam_setfl)(path)
    os.unlink(path)


_BASIS = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])


def _cell(n, rng, xB, sigma, vac, tilt, T):
    """FCC repeats with random elements, vacancies, a lower-triangular strain,
    noise and Maxwell-Boltzmann velocities: H, x, elem, v."""
    a = 3.615
    g = np.stack(np.meshgrid(*(np.arange(k) for k in n), indexing="ij"), -1).reshape(-1, 1, 3)
    x = ((g + _BASIS).reshape(-1, 3)) * a
    H = np.diag([k * a for k in n]).astype(np.float64)
    elem = (rng.random(len(x)) < xB).astype(np.uint8)
    if vac > 0.0:
        keep = np.ones(len(x), dtype=bool)
        keep[rng.choice(len(x), int(round(vac * len(x))), replace=False)] = False
        x, elem = x[keep], elem[keep]
    if tilt > 0.0:
        E = np.eye(3) + np.tril(rng.uniform(-tilt, tilt, (3, 3)))
        H, x = H @ E, x @ E
    if sigma > 0.0:
        x = x + rng.normal(0.0, sigma, x.shape)
    s = x @ np.linalg.inv(H)
    x = np.ascontiguousarray((s - np.floor(s)) @ H)
    v = rng.standard_normal(x.shape) * np.sqrt(KB * T / MASS[elem])[:, None]
    return H, x, elem, v


def _inputs(case, seed):
    """The cells of a case and their temperatures, from the seed alone."""
    rng = np.random.default_rng(seed)
    if not case["kind"].startswith("batch"):
        T = case.get("T", 300.0)
        return [_cell((case["nx"], case["ny"], case["nz"]), rng, case["xB"], case["sigma"], case["vac"], case["tilt"],
                      T)], np.array([T])
    relax = case["kind"] == "batch_lbfgs"
    size = np.random.default_rng(case["cells"])  # the cells' sizes belong to the case, what is in them to the seed
    cells, temps = [], []
    for k in range(case["cells"]):
        # sizes spread over the logarithm of the range, shapes and disorder drawn
        lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
        m = math.exp(lo + (hi - lo) * (k + size.random()) / case["cells"])
        side = (m / 4.0) ** (1.0 / 3.0) * np.exp(size.normal(0.0, 0.2, 3))
        n = [max(4, int(round(v))) for v in side]
        vac = size.uniform(0.0, 0.03 if relax else 0.02)
        T = rng.uniform(100.0, 1200.0)
        cells.append(_cell(n, rng, rng.random(), rng.uniform(0.05, 0.2) if relax else 0.05, vac,
                           0.02 if relax else 0.0, T))
        temps.append(T)
    return cells, np.array(temps)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available() and a.size > 300000)
    t.numpy()[...] = a
    return t.numpy()


def prepare(case, seed):
    cells, temps = _inputs(case, seed)
    st = {"case": case, "temps": temps}
    if case["kind"].startswith("batch"):
        st["ff"] = _force_field(False)
        b = _lib.Batch(st["ff"], [(c[0], c[1], c[2]) for c in cells], MASS)
        st["x"] = _pinned(np.concatenate([c[1] for c in cells]))
        st["v"] = _pinned(np.concatenate([c[3] for c in cells]))
        st["out"] = [_pinned(np.empty_like(st["x"])) for _ in range(3)]
        b.autotune()
        st["sys"] = b
        st["net"] = precond.load() if case.get("net") else None  # the network that ships with the framework
        return st
    H, x, elem, v = cells[0]
    if case.get("api") == "md":
        a = md.atoms(H, x, elem, ("A", "B"), MASS, x_d=v)
        a.precision = case["precision"]
        a.kB = KB
        _setfl(a, case["pairwise"])
        st.update(atoms=a, x=x, v=v)
        # the first run makes the device state
        if case["kind"] == "lbfgs":
            md.min_lbfgs(m=case["m"]).run(a, 0)
        else:
            sim = md.nvt(case["T"], FS)
            sim.ntally = 0
            sim.run(a, 0)
        return st
    st["ff"] = _force_field(case["pairwise"])
    s = _lib.System(st["ff"], H, x, elem, MASS, SKIN, _lib.MIXED if case["precision"] == "mixed" else _lib.FP64)
    if case["precision"] == "mixed" and s.n >= 50000:  # as md.atoms does
        s.set_x(x)
        s.autotune()
    st.update(sys=s, H=H, x=_pinned(x), v=_pinned(v), out=[_pinned(np.empty_like(x)) for _ in range(3)])
    return st


# ------------------------------------------------------------------ a pass
def _given(case, d):
    """Outputs in the type they were computed in (see the top)."""
    if case.get("precision", "mixed") == "fp64":
        return d
    return {k: torch.from_numpy(np.ascontiguousarray(v)).to(torch.float32) for k, v in d.items()}


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "force":
        s = st["sys"]
        s.set_x(st["x"])
        s.build()
        pe, vir = s.force()
        return _given(case, {"pe": np.array([pe]), "virial": vir, "f": s.get_f(st["out"][2])})
    if kind == "batch_nvt":
        b = st["sys"]
        b.set_x(st["x"])
        b.set_v(st["v"])
        th, _ = b.nvt_run(st["temps"], FS, KB, case["steps"], thermo=True)
        xo, vo, fo = st["out"]
        return _given(case, {"thermo": th, "x": b.get_x(xo), "v": b.get_v(vo), "f": b.get_f(fo)})
    if kind == "batch_lbfgs":
        b = st["sys"]
        b.set_x(st["x"])
        r = b.lbfgs_run(m=case["m"], f_tol=1e-4, nsteps=case["iters"], net=st["net"])
        return _given(case, {"pe": np.array([c["pe"] for c in r]), "x": b.get_x(st["out"][0]),
                             "f": b.get_f(st["out"][2])})
    if kind == "lbfgs" and case["api"] == "system":
        s = st["sys"]
        s.set_x(st["x"])
        r = s.lbfgs_run(m=case["m"], f_tol=1e-4, nsteps=case["iters"])
        return _given(case, {"pe": np.array([r["pe"]]), "x": s.get_x(st["out"][0]), "f": s.get_f(st["out"][2])})
    if kind == "nvt" and case["api"] == "system":
        xo, vo, fo = st["out"]
        th, _ = st["sys"].nvt_run_host(st["x"], st["v"], case["T"], FS, KB, case["steps"], thermo=True, x_out=xo,
                                       v_out=vo, f_out=fo)
        return _given(case, {"thermo": th, "x": xo, "v": vo, "f": fo})
    if kind == "nst":
        s = st["sys"]
        s.set_box(st["H"])
        s.set_x(st["x"])
        s.set_v(st["v"])
        th, VH, eta, etaS = s.nst_run(np.zeros((3, 3)), case["T"], FS, KB, case["steps"])
        xo, vo, fo = st["out"]
        return _given(case, {"thermo": th, "H": s.get_box(), "V_H": VH, "x": s.get_x(xo), "v": s.get_v(vo),
                             "f": s.get_f(fo)})
    a = st["atoms"]
    a.x[...] = st["x"]
    if kind == "lbfgs":
        r = md.min_lbfgs(m=case["m"], e_tol=0.0, f_tol=1e-4).run(a, case["iters"])
        return _given(case, {"pe": np.array([r["pe"]]), "x": a.x, "f": a.f})
    a.x_d[...] = st["v"]
    sim = md.nvt(case["T"], FS)
    sim.ntally = 0
    sim.run(a, case["steps"])
    return _given(case, {"pe": np.array([a.pe]), "S_pe": a.S_pe, "x": a.x, "v": a.x_d, "f": a.f})


def work(case):
    """Bytes and operations that a pass cannot do without: the host arrays in
    and out once, and for each evaluation of the forces positions read,
    forces and state written; ~60 operations for each pair inside the cutoff
    (distance, three spline values, the force), each pair once."""
    if case["kind"].startswith("batch"):
        lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
        n = case["cells"] * (math.exp(hi) - math.exp(lo)) / (hi - lo)
    else:
        n = 4.0 * case["nx"] * case["ny"] * case["nz"] * (1.0 - case["vac"])
    evals = {"force": 1}.get(case["kind"], case.get("steps", case.get("iters", 0)) + 1)
    io = {"force": 48.0, "lbfgs": 72.0, "batch_lbfgs": 72.0}.get(case["kind"], 120.0)
    state = 48.0 if case["kind"] == "force" else 96.0  # x, v (or the search direction) read and written
    return {"bytes": n * (io + state * evals), "flops": n * evals * (ROW / 2.0 * 60.0 + 40.0)}


# ------------------------------------------------------------------ in 64 bits
class _Plain:
    """EAM energy, forces and virial of cells in torch FP64: cubic Hermite
    splines through the knots (five-point derivatives), every pair by both
    atoms, periodic images by bins of the reach."""

    def __init__(self, cells, pairwise, reach):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        F, rho, rphi = _knots(pairwise)
        self.F, self.rho, self.rphi = (self._spline(a) for a in (F, rho, rphi))
        self.cut2 = []
        for a in range(2):
            for b in range(2):
                nz = [np.flatnonzero(t)[-1] for t in (rphi[a, b], rho[a, b], rho[b, a])]
                self.cut2.append((max(nz) * DR) ** 2)
        self.count = [len(c[1]) for c in cells]
        self.cell = torch.repeat_interleave(torch.arange(len(cells), device=self.dev),
                                            torch.tensor(self.count, device=self.dev))
        self.elem = torch.from_numpy(np.concatenate([c[2] for c in cells]).astype(np.int64)).to(self.dev)
        self.pairs, base = [], 0
        for H, x, _, _ in cells:
            for i, j, sh in self._near(H, torch.from_numpy(x).to(self.dev), reach):
                self.pairs.append((i + base, j + base, sh))
            base += len(x)
        if len(self.pairs) > 64:  # many small cells: one batch of pairs
            self.pairs = [tuple(torch.cat([p[k] for p in self.pairs]) for k in range(3))]

    def _spline(self, a):
        f = torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)
        d = torch.empty_like(f)
        d[..., 2:-2] = ((f[..., :-4] - f[..., 4:]) + 8.0 * (f[..., 3:-1] - f[..., 1:-3])) / 12.0
        d[..., 0] = f[..., 1] - f[..., 0]
        d[..., 1] = 0.5 * (f[..., 2] - f[..., 0])
        d[..., -2] = 0.5 * (f[..., -1] - f[..., -3])
        d[..., -1] = f[..., -1] - f[..., -2]
        step = f[..., 1:] - f[..., :-1]
        c2 = 3.0 * step - 2.0 * d[..., :-1] - d[..., 1:]
        c3 = d[..., :-1] + d[..., 1:] - 2.0 * step
        return torch.stack([f[..., :-1], d[..., :-1], c2, c3], -1).reshape(-1, 4)

    def _near(self, H, x, reach):
        """(i, j, image vector) of the pairs closer than reach, by blocks of atoms"""
        Ht = torch.from_numpy(H).to(self.dev)
        B = torch.linalg.inv(Ht)
        depth = torch.linalg.norm(B, dim=0).cpu().numpy()
        nb = [max(1, int(1.0 / (reach * d))) for d in depth]
        # a box thinner than the reach needs more than one layer of images
        lay = [max(1, math.ceil(reach * d)) if n == 1 else 1 for n, d in zip(nb, depth)]
        s = x @ B
        fl = torch.floor(s)
        b = torch.stack([((s - fl)[:, d] * nb[d]).long().clamp_(0, nb[d] - 1) for d in range(3)], 1)
        flat = b[:, 0] + nb[0] * (b[:, 1] + nb[1] * b[:, 2])
        order = torch.argsort(flat, stable=True)
        cnt = torch.bincount(flat, minlength=nb[0] * nb[1] * nb[2])
        start = torch.cumsum(cnt, 0) - cnt
        most = int(cnt.max())
        slot = torch.arange(most, device=self.dev)
        nbt = torch.tensor(nb, device=self.dev)
        got = []
        block = max(1, 24_000_000 // most)
        for lo in range(0, len(x), block):
            i = torch.arange(lo, min(lo + block, len(x)), device=self.dev)
            found = []
            for k in range(-lay[0], lay[0] + 1):
                for m in range(-lay[1], lay[1] + 1):
                    for n in range(-lay[2], lay[2] + 1):
                        u = b[i] + torch.tensor([k, m, n], device=self.dev)
                        im = torch.div(u, nbt, rounding_mode="floor")
                        w = u - im * nbt
                        wf = w[:, 0] + nb[0] * (w[:, 1] + nb[1] * w[:, 2])
                        ok = slot[None, :] < cnt[wf][:, None]
                        at = (start[wf][:, None] + slot[None, :]).clamp_(max=len(x) - 1)
                        j = order[at]
                        # image of j's wrapped position beside i's wrapped position
                        sh = (im[:, None, :] - fl[j] + fl[i][:, None, :]).double() @ Ht
                        d = x[i][:, None, :] - x[j] - sh
                        r2 = (d * d).sum(-1)
                        ok &= (r2 < reach * reach) & (r2 > 1e-12)
                        q, p = torch.nonzero(ok, as_tuple=True)
                        found.append((i[q], j[q, p], sh[q, p]))
            got.append(tuple(torch.cat([f[k] for f in found]) for k in range(3)))
        return got

    def _at(self, tab, which, r, n, step):
        p = r / step
        m = p.long().clamp_(max=n - 2)
        p = (p - m).clamp_(max=1.0)
        c = tab[which * (n - 1) + m]
        return (((c[:, 3] * p + c[:, 2]) * p + c[:, 1]) * p + c[:, 0],
                ((3.0 * c[:, 3] * p + 2.0 * c[:, 2]) * p + c[:, 1]) / step)

    def __call__(self, x):
        """pe and virial (xx, xy, xz, yy, yz, zz) per cell, forces"""
        N, nc = len(x), len(self.count)
        rho = torch.zeros(N, dtype=torch.float64, device=self.dev)
        cut2 = torch.tensor(self.cut2, dtype=torch.float64, device=self.dev)

        def inside():
            for i, j, sh in self.pairs:
                d = x[i] - x[j] - sh
                r2 = (d * d).sum(-1)
                t = self.elem[i] * 2 + self.elem[j]
                k = torch.nonzero(r2 < cut2[t]).flatten()
                i, j, t, d = i[k], j[k], t[k], d[k]
                yield i, j, t, (self.elem[j] * 2 + self.elem[i]), d, r2[k].sqrt()

        for i, j, t, u, d, r in inside():
            rho.index_add_(0, i, self._at(self.rho, u, r, NR, DR)[0])
        F, dF = self._at(self.F, self.elem, rho, NRHO, DRHO)
        top = NRHO * DRHO
        F = torch.where(rho > top, F + dF * (rho - top), F)
        pe = torch.zeros(nc, dtype=torch.float64, device=self.dev).index_add_(0, self.cell, F)
        vir = torch.zeros(nc, 6, dtype=torch.float64, device=self.dev)
        f = torch.zeros(N, 3, dtype=torch.float64, device=self.dev)
        for i, j, t, u, d, r in inside():
            z, dz = self._at(self.rphi, t, r, NR, DR)
            phi = z / r
            g = -((dz - phi) / r + dF[i] * self._at(self.rho, u, r, NR, DR)[1] +
                  dF[j] * self._at(self.rho, t, r, NR, DR)[1]) / r
            v = g[:, None] * d
            f.index_add_(0, i, v)
            c = self.cell[i]
            pe.index_add_(0, c, 0.5 * phi)
            if nc == 1:
                w = 0.5 * (v.T @ d)
                vir += torch.stack([w[0, 0], w[0, 1], w[0, 2], w[1, 1], w[1, 2], w[2, 2]])
            else:
                vir.index_add_(0, c, 0.5 * torch.stack([v[:, 0] * d[:, 0], v[:, 0] * d[:, 1], v[:, 0] * d[:, 2],
                                                        v[:, 1] * d[:, 1], v[:, 1] * d[:, 2], v[:, 2] * d[:, 2]], 1))
        return pe, vir, f


def _chain(eta, tr, ndof, ddt, freq):
    """Half a step of a three-link Nose-Hoover chain for every cell (arrays):
    the velocity factor; eta changes in place."""
    def phi(a):
        return np.where(np.abs(a) < 1e-9, 1.0, np.expm1(a) / np.where(a == 0.0, 1.0, a))

    h = 0.5 * ddt
    eta[2] += h * (eta[1] ** 2 - freq)
    eta[1] += h * phi(-eta[2] * h) * (-eta[2] * eta[1] + eta[0] ** 2 - freq)
    eta[0] += h * phi(-eta[1] * h) * (-eta[1] * eta[0] + freq * (tr - 1.0))
    fac = np.exp(-ddt * eta[0])
    tr = tr * fac * fac
    eta[0] += h * phi(-eta[1] * h) * (-eta[1] * eta[0] + freq * (tr - 1.0))
    eta[1] += h * phi(-eta[2] * h) * (-eta[2] * eta[1] + ndof * eta[0] ** 2 - freq)
    eta[2] += h * (eta[1] ** 2 - freq)
    return fac


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("force", "nvt", "batch_nvt"):
        # a minimiser's steps and a moving box's are a path of accepted
        # trials and list images, which no formula gives
        return None
    cells, temps = _inputs(case, seed)
    pairwise = case.get("pairwise", False)
    plain = _Plain(cells, pairwise, RC + (0.1 if kind == "force" else 1.3))
    dev = plain.dev
    x = torch.from_numpy(np.concatenate([c[1] for c in cells])).to(dev)
    if kind == "force":
        pe, vir, f = plain(x)
        return {"pe": pe, "virial": vir[0], "f": f}
    v = torch.from_numpy(np.concatenate([c[3] for c in cells])).to(dev)
    mass = torch.from_numpy(MASS).to(dev)[plain.elem][:, None]
    nc, cell, n = len(cells), plain.cell, np.array(plain.count, dtype=np.float64)

    def kinetic():
        m = mass[:, 0]
        q = torch.stack([m * v[:, a] * v[:, b] for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))], 1)
        return torch.zeros(nc, 6, dtype=torch.float64, device=dev).index_add_(0, cell, q).cpu().numpy()

    ndof = 3.0 * n
    freq, ddt = 1.0 / (100.0 * FS) ** 2, 0.5 * FS
    eta = np.zeros((3, nc))
    pe, vir, f = plain(x)
    kin = kinetic()
    T = (kin[:, 0] + kin[:, 3] + kin[:, 5]) / (ndof * KB)
    fac = np.ones(nc)
    rows = []

    def note():
        rows.append(np.concatenate([pe.cpu().numpy()[:, None], T[:, None], kin, vir.cpu().numpy()], 1))

    note()
    count = torch.from_numpy(n).to(dev)[:, None]
    for _ in range(case["steps"]):
        k = _chain(eta, T / temps, ndof, ddt, freq)
        T, fac = T * k * k, fac * k
        v = v * torch.from_numpy(fac).to(dev)[cell][:, None] + f * (0.5 * FS) / mass
        dx = v * FS
        x = x + dx - (torch.zeros(nc, 3, dtype=torch.float64, device=dev).index_add_(0, cell, dx) / count)[cell]
        pe, vir, f = plain(x)
        v = v + f * (0.5 * FS) / mass
        kin = kinetic()
        T = (kin[:, 0] + kin[:, 3] + kin[:, 5]) / (ndof * KB)
        fac = _chain(eta, T / temps, ndof, ddt, freq)
        kin, T = kin * (fac * fac)[:, None], T * fac * fac
        note()
    v = v * torch.from_numpy(fac).to(dev)[cell][:, None]
    # positions come back wrapped or not, as the last list build left them
    d = {"x": None, "v": v, "f": f}
    if case.get("api") == "md":
        vol = float(np.prod(np.diag(cells[0][0])))
        w = (-vir[0] / vol).cpu().numpy()
        d.update(pe=pe, S_pe=np.array([[w[0], w[1], w[2]], [w[1], w[3], w[4]], [w[2], w[4], w[5]]]))
    elif kind == "nvt":
        d["thermo"] = np.stack([r[0] for r in rows])
    else:
        d["thermo"] = np.stack([r[:, :2] for r in rows])
    return d

"""The two forms of the FP64 passes of one cell: pairs computed once with a
record of each, and the full rows that a system takes where it keeps no
records.  Forces, MD, relaxations and constant-stress MD over the full rows,
against the oracle at the tolerances of the pair form's tests, and the two
forms against each other (another order of the same sums)."""
import numpy as np
import pytest

import oracle as O
from mapp4py_gb300 import _lib, synth

pytestmark = pytest.mark.gpu


def _cell(cells=(6, 5, 5), T=600.0):
    return synth.alloy(cells, xB=0.4, sigma=0.05, T=T, seed=6)


def _sys(potentials, c, mode, precision=_lib.FP64):
    path, _ = potentials[("A", "B")]
    s = _lib.System(_lib.ForceField.setfl(path), c.H, c.x, c.elem, c.masses, skin=0.5, precision=precision)
    assert s.pair_records() == (1 if precision == _lib.FP64 else 0)
    if mode is not None:
        assert s.pair_records(mode) == mode
    s.set_v(c.v)
    return s


def _oracle(potentials, c):
    path, _ = potentials[("A", "B")]
    o = O.System(O.Eam.setfl(path), c.H, c.x, c.elem, c.masses, skin=0.5)
    o.v = c.v
    return o


# 32, 16, 8 and 4 lanes an atom
@pytest.mark.parametrize("cells", [(3, 3, 4), (7, 7, 8), (9, 9, 9), (14, 14, 14)])
def test_forces_and_energies(potentials, cells):
    c = _cell(cells)
    o = _oracle(potentials, c)
    pe_o, vir_o = o.force()
    s = _sys(potentials, c, 0)
    pe, vir = s.force()
    assert abs(pe - pe_o) <= 1e-12 * abs(pe_o)
    assert np.max(np.abs(vir - vir_o)) <= 1e-11 * np.max(np.abs(vir_o))
    assert np.max(np.abs(s.get_f() - o.f)) <= 1e-10 * max(1.0, np.max(np.abs(o.f)))
    assert abs(s.energy() - pe_o) <= 1e-12 * abs(pe_o)
    rho, _ = s.rho_dF()
    assert s.pair_records(1) == 1
    pe1, vir1 = s.force()
    assert abs(pe1 - pe) <= 1e-12 * abs(pe)
    rho1, _ = s.rho_dF()
    assert np.max(np.abs(rho1 - rho)) <= 1e-13 * np.max(rho)


# without and with a step graph
@pytest.mark.parametrize("nsteps", [5, 40])
def test_nvt(potentials, nsteps):
    c = _cell()
    o = _oracle(potentials, c)
    th_o, eta_o, _ = o.nvt_run(600.0, synth.FS, synth.KB, nsteps, t_relax=100 * synth.FS)
    s = _sys(potentials, c, 0)
    th, eta = s.nvt_run(600.0, synth.FS, synth.KB, nsteps, thermo=True)
    for k in (0, 1):
        assert np.max(np.abs(th[:, k] - th_o[:, k])) <= 1e-10 * np.max(np.abs(th_o[:, k]))
    assert np.max(np.abs(th[:, 8:] - th_o[:, 8:])) <= 1e-9 * np.max(np.abs(th_o[:, 8:]))
    pe, _ = s.force()  # the last row is the energy of the positions reached
    assert abs(th[-1, 0] - pe) <= 1e-12 * abs(pe)


@pytest.mark.parametrize("method", ["lbfgs", "cg"])
def test_relaxation(potentials, method):
    c = _cell(T=0.0)
    out = []
    for mode in (0, 1):
        s = _sys(potentials, c, mode)
        r = s.lbfgs_run(m=5, nsteps=5) if method == "lbfgs" else s.cg_run(nsteps=5)
        out.append((r, s.get_x()))
    (a, xa), (b, xb) = out
    assert (a["niter"], a["n_energy"], a["err"]) == (b["niter"], b["n_energy"], b["err"])
    # five iterations magnify the last bits; test_gpu_work allows the same
    assert abs(a["pe"] - b["pe"]) <= 1e-11 * abs(a["pe"])
    assert np.max(np.abs(xa - xb)) <= 1e-8


def test_constant_stress(potentials):
    c = _cell(T=300.0)
    nan = np.nan
    S = np.array([[0.0, nan, nan], [nan, 0.0, nan], [nan, nan, 0.0]])
    th = [_sys(potentials, c, mode).nst_run(S, 300.0, synth.FS, synth.KB, 20)[0] for mode in (0, 1)]
    assert np.max(np.abs(th[0][:, 0] - th[1][:, 0])) <= 1e-10 * np.max(np.abs(th[1][:, 0]))
    assert np.max(np.abs(th[0][:, 14:] - th[1][:, 14:])) <= 1e-10


def test_choice(potentials):
    c = _cell()
    s = _sys(potentials, c, None)
    s.force()
    f = s.get_f()
    for mode in (0, 1, 1, 0, 1):  # the list follows each choice
        assert s.pair_records(mode) == mode == s.pair_records()
        s.force()
        assert np.max(np.abs(s.get_f() - f)) <= 1e-10 * np.max(np.abs(f))
    s.nvt_begin(600.0, synth.FS, synth.KB, 10)
    with pytest.raises(_lib.MappgError):
        s.pair_records(0)
    assert s.pair_records() == 1
    s.nvt_steps(10)
    s.nvt_end()
    with pytest.raises(_lib.MappgError):
        s.pair_records(2)
    m = _sys(potentials, c, 0, precision=_lib.MIXED)
    with pytest.raises(_lib.MappgError):
        m.pair_records(1)
    m.force()

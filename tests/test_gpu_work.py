"""The minimizers' vectors live in a workspace kept with the system: runs of
other sizes before and after, and runs started inside another one's iteration
function, leave a run's results as they are."""
import numpy as np
import pytest

from mapp4py_gb300 import _lib, synth

pytestmark = pytest.mark.gpu


def _sys(potentials, precision):
    path, _ = potentials[("A", "B")]
    c = synth.alloy((7, 6, 6), xB=0.3, sigma=0.15, seed=11)
    return c, _lib.System(_lib.ForceField.setfl(path), c.H, c.x, c.elem, c.masses, skin=0.5, precision=precision)


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
def test_runs_of_other_sizes_leave_no_trace(potentials, precision):
    _, fresh = _sys(potentials, precision)
    a = fresh.lbfgs_run(m=5, nsteps=8)
    c, s = _sys(potentials, precision)
    for run in (lambda: s.lbfgs_run(m=1, nsteps=3), lambda: s.lbfgs_run(m=20, nsteps=4), lambda: s.cg_run(nsteps=3)):
        run()
    s.set_x(c.x)
    b = s.lbfgs_run(m=5, nsteps=8)
    assert (a["niter"], a["n_energy"]) == (b["niter"], b["n_energy"])
    # FP64 line-search energies; the mixed forces' FP32 rounding moves x by ~1e-6 of a step
    assert abs(a["pe"] - b["pe"]) <= (1e-11 if precision == _lib.FP64 else 1e-7) * abs(a["pe"])
    assert np.max(np.abs(fresh.get_x() - s.get_x())) <= (1e-8 if precision == _lib.FP64 else 1e-3)


def test_a_run_inside_the_iteration_function(potentials):
    _, plain = _sys(potentials, _lib.FP64)
    a = plain.lbfgs_run(m=5, nsteps=6)
    _, s = _sys(potentials, _lib.FP64)
    seen = []

    def inner(step):
        seen.append(s.cg_run(nsteps=0)["pe"])

    s.set_hook(inner, 2)
    b = s.lbfgs_run(m=5, nsteps=6)
    assert len(seen) == 3 and a["niter"] == b["niter"]
    assert abs(a["pe"] - b["pe"]) <= 1e-9 * abs(a["pe"])

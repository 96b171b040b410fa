"""The thermostat chain at the end of an MD step against the oracle: chain
lengths and iteration counts beside the default, and couplings so stiff that
the chain's arguments leave the range of its polynomials.  Tolerances: the
FP64 trajectory's 1e-10 relative (as the NVT parity tests), the mixed path's
temperature 1e-6 relative over 12 steps (FP32 forces, ~1e-7 a step)."""
import numpy as np
import pytest

import oracle as O
from mapp4py_gb300 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,niters,relax", [(1, 1, 100.0), (2, 1, 100.0), (3, 1, 100.0), (3, 2, 20.0), (5, 1, 50.0),
                                            (3, 1, 0.9), (4, 3, 0.9)])
@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
def test_chain_follows_oracle(potentials, precision, L, niters, relax):
    path, _ = potentials[("A", "B")]
    c = synth.alloy((4, 5, 4), xB=0.5, sigma=0.05, T=600.0, seed=9)
    eta0 = 0.02 * np.arange(1, L + 1)
    kw = dict(t_relax=relax * synth.FS, L=L, niters=niters)
    o = O.System(O.Eam.setfl(path), c.H, c.x, c.elem, c.masses, skin=0.5)
    o.v = c.v
    th_o, eta_o, _ = o.nvt_run(700.0, synth.FS, synth.KB, 12, eta=eta0.copy(), **kw)
    s = _lib.System(_lib.ForceField.setfl(path), c.H, c.x, c.elem, c.masses, precision=precision)
    s.set_v(c.v)
    th, eta = s.nvt_run(700.0, synth.FS, synth.KB, 12, eta=eta0.copy(), thermo=True, **kw)
    rel = 1e-10 if precision == _lib.FP64 else 1e-6
    assert np.max(np.abs(th[:, 1] - th_o[:, 1])) <= rel * np.max(np.abs(th_o[:, 1]))
    if precision == _lib.FP64:  # a stiff chain takes a temperature's FP32 rounding far beyond it
        assert np.max(np.abs(eta - eta_o)) <= rel * np.max(np.abs(eta_o))


@pytest.mark.parametrize("cells", [(3, 3, 3), (5, 4, 6), (11, 11, 11), (16, 17, 16)])
@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
def test_energy_and_virial_of_the_last_step(potentials, precision, cells):
    """An MD step's energy and virial (added up where the step closes) against
    a force call at the positions that the step reached."""
    path, _ = potentials[("A", "B")]
    c = synth.alloy(cells, xB=0.5, sigma=0.05, T=600.0, seed=9)
    s = _lib.System(_lib.ForceField.setfl(path), c.H, c.x, c.elem, c.masses, precision=precision)
    s.set_v(c.v)
    th, _ = s.nvt_run(700.0, synth.FS, synth.KB, 7, thermo=True)
    pe, vir = s.force()
    # sums in another order; mixed: positions rounded to FP32 in another frame
    rel, relv = (1e-13, 1e-12) if precision == _lib.FP64 else (1e-7, 1e-5)
    assert abs(th[-1, 0] - pe) <= rel * abs(pe)
    assert np.max(np.abs(th[-1, 8:] - vir)) <= relv * np.sqrt(s.n) * np.max(np.abs(vir))

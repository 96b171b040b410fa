"""Calls between the start of an MD run and its first step.  A list build
there takes the displacement that the run's steps have left in the positions
out of them, and there has been none.  Atoms that the build moved would be
away by the shift; else the positions agree to the FP32 forces' rounding
(another row order: ~1e-6 of a force, 1e-4 A/fs^2 of acceleration, over ten
steps of 1 fs below 1e-8 A)."""
import ctypes as C

import numpy as np
import pytest

from mapp4py_gb300 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.fixture
def spoiled_memory():
    """Device memory that other work has used and given back: every second of
    a row of blocks is free again and holds 0.37, for the allocations to come."""
    rt = C.CDLL("libcudart.so")
    n = (1 << 20) // 8  # MB blocks, as large as a system's partial sums
    src = np.full(n, 0.37)
    blocks = [C.c_void_p() for _ in range(64)]
    for p in blocks:
        assert rt.cudaMalloc(C.byref(p), C.c_size_t(8 * n)) == 0
        assert rt.cudaMemcpy(p, src.ctypes.data_as(C.c_void_p), C.c_size_t(8 * n), 1) == 0
    for p in blocks[::2]:
        rt.cudaFree(p)
    yield
    for p in blocks[1::2]:
        rt.cudaFree(p)


def _sys(potentials, cells):
    path, _ = potentials[("A", "B")]
    c = synth.alloy(cells, xB=0.4, sigma=0.05, T=600.0, seed=5)
    s = _lib.System(_lib.ForceField.setfl(path), c.H, c.x, c.elem, c.masses, precision=_lib.MIXED)
    s.set_v(c.v)
    return c, s


# one cluster bins the first, four kernels the second; with and without a step graph
@pytest.mark.parametrize("cells,nsteps", [((5, 5, 5), 10), ((5, 5, 5), 4), ((14, 13, 13), 10)])
def test_build_before_the_first_step(potentials, spoiled_memory, cells, nsteps):
    x = []
    for build in (False, True):
        c, s = _sys(potentials, cells)
        s.nvt_begin(600.0, synth.FS, synth.KB, nsteps)
        if build:
            s.build()
        s.nvt_steps(nsteps)
        s.nvt_end()
        x.append(s.get_x())
    d = x[1] - x[0]
    d -= np.round(d @ np.linalg.inv(c.H)) @ c.H
    assert np.max(np.abs(d)) <= 1e-8


def test_relaxation_after_an_unfinished_run(potentials, spoiled_memory):
    out = []
    for begun in (False, True):
        c, s = _sys(potentials, (5, 5, 5))
        if begun:
            s.nvt_begin(600.0, synth.FS, synth.KB, 10)
        r = s.lbfgs_run(m=5, nsteps=3)
        out.append((r["pe"], s.get_x()))
    assert abs(out[1][0] - out[0][0]) <= 1e-7 * abs(out[0][0])
    d = out[1][1] - out[0][1]
    d -= np.round(d @ np.linalg.inv(c.H)) @ c.H
    assert np.max(np.abs(d)) <= 1e-5

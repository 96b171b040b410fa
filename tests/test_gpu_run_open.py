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


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
def test_rows_that_grow_before_the_first_step(potentials, precision):
    """The rows of a thin gas are short.  A begun run whose atoms are put
    close together has its rows moved by the build that follows: its step
    graph is taken again.  The steps are those of a run begun there (FP64 to
    the trajectory's 1e-10; mixed bits differ in nothing but the frame)."""
    path, _ = potentials[("A", "B")]
    c = synth.alloy((5, 5, 5), xB=0.4, sigma=0.05, T=300.0, seed=5)
    H = np.diag([90.0] * 3)
    rng = np.random.default_rng(2)
    thin = rng.random((c.natoms, 3)) @ H
    close = c.x + 30.0
    ff = _lib.ForceField.setfl(path)
    out = []
    for moved in (False, True):
        s = _lib.System(ff, H, thin if moved else close, c.elem, c.masses, precision=precision)
        s.set_v(c.v)
        if not moved:
            s.build()
        cap = s.stats()["capacity"]
        s.nvt_begin(300.0, synth.FS, synth.KB, 20)
        if moved:
            s.set_x(close)
            s.force()
            assert s.stats()["capacity"] > cap
        s.nvt_steps(20)
        s.nvt_end()
        out.append((s.get_x(), s.get_v()))
    tol = 1e-10 if precision == _lib.FP64 else 1e-6
    for a, b in zip(*out):
        assert np.max(np.abs(a - b)) <= tol * max(1.0, np.max(np.abs(a)))


def test_tuning_a_batch_is_refused_in_a_run(potentials):
    """... and leaves the chunks that the run's graphs walk."""
    path, _ = potentials[("A", "B")]
    cs = [synth.alloy(k, xB=0.4, sigma=0.05, T=300.0, seed=3) for k in ((4, 4, 4), (5, 4, 4), (6, 5, 5))]
    ff = _lib.ForceField.setfl(path)
    x = []
    for disturbed in (False, True):
        b = _lib.Batch(ff, [(c.H, c.x, c.elem) for c in cs], cs[0].masses)
        b.set_v(np.concatenate([c.v for c in cs]))
        b.nvt_begin([300.0, 400.0, 500.0], synth.FS, synth.KB, 12)
        chunk = b.tuning()["atoms_per_chunk"]
        if disturbed:
            with pytest.raises(_lib.MappgError):
                b.autotune()
        assert b.tuning()["atoms_per_chunk"] == chunk
        b.nvt_steps(12)
        b.nvt_end()
        x.append(b.get_x())
    assert np.array_equal(x[0], x[1])

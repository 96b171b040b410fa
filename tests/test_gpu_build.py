"""Neighbour sets of the list builder where its staging changes shape: rows
and candidates beyond what a block holds on chip, bins of more atoms than a
block takes at a time, empty bins, single atoms, tilted boxes.  The sets equal
the oracle's exactly."""
import numpy as np
import pytest

import oracle as O
from mapp4py_gb300 import _lib, synth
from test_gpu_parity import keys

pytestmark = pytest.mark.gpu


def _cell(kind):
    rng = np.random.default_rng(17)
    if kind == "wide":  # a reach of 10.5 A: ~400 entries a row, several tiles of candidates
        c = synth.alloy((7, 6, 8), xB=0.5, sigma=0.1, seed=3)
        return c.H, c.x, c.elem, 5.0
    if kind == "wide_tilted":
        H = np.array([[26.0, 0, 0], [3.0, 25.0, 0], [-2.0, 4.0, 27.0]])
        return H, synth.wrap(H, rng.random((1400, 3)) @ H), (rng.random(1400) < 0.5).astype(np.uint8), 5.0
    if kind == "cluster":  # one bin holds 300 atoms, all of them neighbours: rows of 299
        x = 20.0 + rng.uniform(-1.4, 1.4, (300, 3))
        return np.diag([43.0, 41.0, 40.0]), x, (rng.random(300) < 0.5).astype(np.uint8), 0.5
    if kind == "gas":  # mostly empty bins, rows of 0 to a few entries
        H = np.array([[61.0, 0, 0], [5.0, 55.0, 0], [0.0, -7.0, 50.0]])
        return H, rng.random((257, 3)) @ H, (rng.random(257) < 0.5).astype(np.uint8), 0.5
    if kind == "one":  # an atom and its own images
        return np.diag([6.6, 7.0, 9.0]), np.array([[6.5, 0.1, 4.0]]), np.zeros(1, np.uint8), 0.9
    raise KeyError(kind)


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
@pytest.mark.parametrize("kind", ["wide", "wide_tilted", "cluster", "gas", "one"])
def test_neighbor_sets_at_the_builders_edges(potentials, kind, precision):
    path, _ = potentials[("A", "B")]
    H, x, elem, skin = _cell(kind)
    masses = [synth.MASS, synth.MASS]
    o = O.System(O.Eam.setfl(path), H, x, elem, masses, skin=skin, pair_wise=False)
    o.init_dynamic()
    s = _lib.System(_lib.ForceField.setfl(path), H, x, elem, masses, skin=skin, precision=precision)
    s.build()
    assert np.array_equal(keys(*s.neighbors()), keys(*o.neighbors()))


def test_batch_rows_equal_single_cells_at_the_builders_edges(potentials):
    path, _ = potentials[("A", "B")]
    ff = _lib.ForceField.setfl(path)
    masses = [synth.MASS, synth.MASS]
    cells = [_cell(k)[:3] for k in ("wide", "cluster", "gas", "wide_tilted")]
    b = _lib.Batch(ff, cells, masses, skin=5.0)
    b.build()
    cnt, ent = b.neighbors()
    at = np.concatenate([[0], np.cumsum(cnt)])
    for k, (H, x, elem) in enumerate(cells):
        lo, hi = b.offsets[k], b.offsets[k + 1]
        e = ent[at[lo]:at[hi]].copy()
        e[:, 0] -= lo
        s = _lib.System(ff, H, x, elem, masses, skin=5.0, precision=_lib.MIXED)
        assert np.array_equal(keys(cnt[lo:hi], e), keys(*s.neighbors()))


@pytest.mark.parametrize("cells,skin", [((2, 4, 5), 0.5), ((4, 4, 5), 6.5), ((7, 6, 6), 0.5), ((9, 9, 8), 0.5)])
def test_fp64_pairs_by_owner_match_the_oracle(potentials, cells, skin):
    """Forces, energy and virial with every pair computed once: 32, 16 and 8
    lanes an atom, several images of one neighbour (a side of 7.2 A), lists
    longer than the lanes' mask (a reach of 12 A: ~300 pairs owned)."""
    path, _ = potentials[("A", "B")]
    c = synth.alloy(cells, xB=0.4, sigma=0.08, vac=0.02, seed=6)
    o = O.System(O.Eam.setfl(path), c.H, c.x, c.elem, c.masses, skin=0.5)
    pe_o, vir_o = o.force()
    s = _lib.System(_lib.ForceField.setfl(path), c.H, c.x, c.elem, c.masses, skin=skin)
    pe, vir = s.force()
    assert abs(pe - pe_o) <= 1e-12 * abs(pe_o)
    assert np.max(np.abs(vir - vir_o)) <= 1e-11 * np.max(np.abs(vir_o))
    assert np.max(np.abs(s.get_f() - o.f)) <= 1e-10 * max(1.0, np.max(np.abs(o.f)))
    assert abs(s.energy() - pe_o) <= 1e-12 * abs(pe_o)


@pytest.mark.parametrize("precision", [_lib.FP64, _lib.MIXED])
@pytest.mark.parametrize("n", [5, 13, 32, 33, 160, 161, 200, 257])
def test_neighbor_sets_of_one_crowded_bin(potentials, n, precision):
    """Every remainder of the atoms a warp tests together, and rows around the
    number of candidates it notes and around the row it puts together on chip."""
    path, _ = potentials[("A", "B")]
    rng = np.random.default_rng(n)
    x = 20.0 + rng.uniform(-1.4, 1.4, (n, 3))
    H, elem, masses = np.diag([43.0, 41.0, 40.0]), (rng.random(n) < 0.5).astype(np.uint8), [synth.MASS, synth.MASS]
    o = O.System(O.Eam.setfl(path), H, x, elem, masses, skin=0.5, pair_wise=False)
    o.init_dynamic()
    s = _lib.System(_lib.ForceField.setfl(path), H, x, elem, masses, skin=0.5, precision=precision)
    s.build()
    assert np.array_equal(keys(*s.neighbors()), keys(*o.neighbors()))


@pytest.mark.parametrize("n,bins", [(1, (4, 4, 4)), (33, (4, 5, 6)), (1025, (16, 16, 8)), (8191, (12, 13, 13)),
                                    (8192, (16, 16, 8)), (8193, (16, 16, 8)), (700, (13, 13, 13))])
def test_neighbor_sets_where_binning_changes_kernels(potentials, n, bins):
    """Around the largest system that one cluster of blocks bins, by atoms and
    by bins, and a second build from moved positions."""
    path, rc = potentials[("A", "B")]
    rng = np.random.default_rng(n)
    ff = _lib.ForceField.setfl(path)
    H = np.diag([b * 6.2 for b in bins])
    H[1, 0] = 1.3
    x, elem, masses = rng.random((n, 3)) @ H, (rng.random(n) < 0.5).astype(np.uint8), [synth.MASS, synth.MASS]
    s = _lib.System(ff, H, x, elem, masses, skin=0.5, precision=_lib.MIXED)
    for _ in range(2):
        s.set_x(x)
        s.build()
        o = O.System(O.Eam.setfl(path), H, x, elem, masses, skin=0.5, pair_wise=False)
        o.init_dynamic()
        assert np.array_equal(keys(*s.neighbors()), keys(*o.neighbors()))
        x = rng.random((n, 3)) @ H


@pytest.mark.parametrize("n", [1, 3, 4, 5, 161, 300, 900])
def test_neighbor_sets_of_a_crowded_bin_among_many(potentials, n):
    """The same edges where the bins are many and a block has fewer warps:
    900 atoms in one bin need several tiles of candidates."""
    path, _ = potentials[("A", "B")]
    rng = np.random.default_rng(n)
    x = np.concatenate([20.0 + rng.uniform(-1.4, 1.4, (n, 3)), rng.random((300, 3)) * 50.0])
    H, elem = np.diag([50.0, 50.5, 51.0]), (rng.random(n + 300) < 0.5).astype(np.uint8)
    o = O.System(O.Eam.setfl(path), H, x, elem, [synth.MASS, synth.MASS], skin=0.5, pair_wise=False)
    o.init_dynamic()
    s = _lib.System(_lib.ForceField.setfl(path), H, x, elem, [synth.MASS, synth.MASS], skin=0.5, precision=_lib.MIXED)
    s.build()
    assert np.array_equal(keys(*s.neighbors()), keys(*o.neighbors()))

"""The mixed passes add their FP32 terms up to energies no worse than an FP64
sum.  Atoms out of each other's reach whose embedding energies are 1, 2^-24
and 2^-48: any order of FP64 additions gives their sum exactly, a sum kept
in two floats loses the last."""
import numpy as np
import pytest

from mapp4py_gb300 import _lib

pytestmark = pytest.mark.gpu

F0 = (1.0, 2.0 ** -24, 2.0 ** -48)


@pytest.fixture(scope="module")
def ff():
    nr, nrho, dr, drho = 120, 50, 0.05, 0.1
    tail = np.maximum(0.0, 1.0 - dr * np.arange(nr) / 5.0) ** 3
    F = np.repeat(np.array(F0)[:, None], nrho, axis=1)
    pairs = np.broadcast_to(tail, (3, 3, nr)).copy()
    return _lib.ForceField.knots(nr, nrho, dr, drho, F, pairs, pairs)


def _cell(order):
    x = 6.0 + 12.0 * np.array([[0, 0, 0], [1, 0, 0], [0, 1, 1]], dtype=np.float64)
    return np.diag([24.0] * 3), x, np.array(order, dtype=np.uint8)


ORDERS = [(0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)]


@pytest.mark.parametrize("order", ORDERS)
def test_energy_of_one_cell(ff, order):
    H, x, elem = _cell(order)
    s = _lib.System(ff, H, x, elem, [1.0] * 3, precision=_lib.MIXED)
    pe, _ = s.force()
    assert pe == sum(F0)
    assert s.energy() == sum(F0)


def test_energies_of_a_batch(ff):
    b = _lib.Batch(ff, [_cell(o) for o in ORDERS], [1.0] * 3)
    pe, _ = b.force()
    assert np.all(pe == sum(F0))
    assert np.all(b.energy() == sum(F0))

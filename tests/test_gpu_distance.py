"""The FP64 passes' distances are correctly rounded roots.  Atoms in pairs,
each along x and out of reach of the others: an atom's density is then one
spline value, formed here from the positions in the kernel's operations (its
fused multiply-adds by exact rationals, rounded once), and equals it bit for
bit."""
from decimal import Decimal, localcontext
from fractions import Fraction

import numpy as np
import pytest

from mapp4py_gb300 import _lib, synth

pytestmark = pytest.mark.gpu


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _both(c, p):
    """Value and derivative per knot of a spline record."""
    b2 = _fma(c[3], p, c[2])
    b1 = _fma(b2, p, c[1])
    return _fma(b1, p, c[0]), _fma(_fma(c[3], p, b2), p, b1)


def _rsqrt(x):
    """The double next to 1/sqrt(x)."""
    with localcontext() as ctx:
        ctx.prec = 60
        return float(1 / Decimal(x).sqrt())


def _density(ff, rho_tab, r):
    q = r * (1.0 / ff.dr)
    m = min(int(q), ff.nr - 2)
    p = min(q - m, 1.0)
    w = [float(v) for v in rho_tab[m]]
    return _fma(_fma(_fma(w[3], p, w[2]), p, w[1]), p, w[0])


def _pairs(side, seed):
    rng = np.random.default_rng(seed)
    at = 13.0 * np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) + 2.0
    x = np.repeat(at, 2, axis=0)
    x[0::2, 0] += rng.random(len(at))
    x[1::2, 0] = x[0::2, 0] + rng.uniform(1.8, 5.4, len(at))
    return np.diag([13.0 * side] * 3), x


# 32, 16, 8 and 4 lanes an atom
@pytest.mark.parametrize("side", [6, 9, 12, 19])
def test_density_of_atom_pairs(potentials, side):
    path, _ = potentials[("A",)]
    ff = _lib.ForceField.setfl(path)
    H, x = _pairs(side, side)
    s = _lib.System(ff, H, x, np.zeros(len(x), np.uint8), [synth.MASS], skin=0.5)
    s.force()
    rho, _ = s.rho_dF()
    xw = s.get_x()
    d = xw[0::2] - xw[1::2]
    assert np.all(d[:, 1:] == 0.0)
    tab = ff.tables()[1][0, 0]
    want = np.repeat([_density(ff, tab, float(r)) for r in np.sqrt(d[:, 0] * d[:, 0])], 2)
    assert np.count_nonzero(rho != want) == 0


@pytest.mark.parametrize("side", [6, 12])
def test_force_of_atom_pairs(potentials, side):
    """The same for forces, with 1/r the correctly rounded one.  The kernel's
    is within 0.508 ulp (what CUDA's own reciprocal root has), so it may round
    the other way for two distances in a hundred at most."""
    path, _ = potentials[("A",)]
    ff = _lib.ForceField.setfl(path)
    H, x = _pairs(side, side + 100)
    s = _lib.System(ff, H, x, np.zeros(len(x), np.uint8), [synth.MASS], skin=0.5)
    s.force()
    _, dF = s.rho_dF()
    f, xw = s.get_f(), s.get_x()
    assert np.all(f[:, 1:] == 0.0) and np.array_equal(f[0::2], -f[1::2])
    tab, ztab = ff.tables()[1][0, 0], ff.tables()[2][0, 0]
    dri = 1.0 / ff.dr
    other = 0
    for k in range(len(x) // 2):
        dx = float(xw[2 * k, 0] - xw[2 * k + 1, 0])
        rsq = dx * dx
        rinv = _rsqrt(rsq)
        q = float(np.sqrt(rsq)) * dri
        m = min(int(q), ff.nr - 2)
        p = min(q - m, 1.0)
        _, d = _both([float(v) for v in tab[m]], p)
        z, dz = _both([float(v) for v in ztab[m]], p)
        phi, g = z * rinv, -rinv * dri
        A, B = -(_fma(dz, dri, -phi) * rinv) * rinv, d * g
        fi, fj = float(dF[2 * k]), float(dF[2 * k + 1])
        # either atom may own the pair
        want = {_fma(fj, B, _fma(fi, B, A)) * dx, _fma(fi, B, _fma(fj, B, A)) * dx}
        other += float(f[2 * k, 0]) not in want
    assert other <= 0.02 * (len(x) // 2)


def test_density_of_coincident_atoms(potentials):
    """Two atoms at one place: no force or energy, but the density at r = 0."""
    path, _ = potentials[("A",)]
    ff = _lib.ForceField.setfl(path)
    x = np.array([[5.0, 6.0, 7.0], [5.0, 6.0, 7.0], [15.0, 15.0, 15.0]])
    s = _lib.System(ff, np.diag([25.0] * 3), x, np.zeros(3, np.uint8), [synth.MASS], skin=0.5)
    with pytest.raises(_lib.MappgError):
        s.force()
    rho, _ = s.rho_dF()
    assert np.array_equal(rho, [_density(ff, ff.tables()[1][0, 0], 0.0)] * 2 + [0.0])

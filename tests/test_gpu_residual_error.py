"""The MIXED refinement's residual against exact rational arithmetic: the error of A x on uniform
grids, isolated by a right-hand side that is A x rounded to FP64, so that what is left is a few
rounding errors and the FP32 store rounds only those."""
from fractions import Fraction

import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu


def exact_ax(x, h):
    """Zero-gradient rows of -div grad on compact x: a list of rationals per cell (C order)."""
    w = [1 / (Fraction(d) * Fraction(d)) for d in h]
    f = np.array([Fraction(v) for v in x.ravel()], dtype=object).reshape(x.shape)
    y = np.zeros(x.shape, dtype=object) + Fraction(0)
    for a in range(3):
        d = np.diff(f, axis=a) * w[a]
        lo, hi = [slice(None)] * 3, [slice(None)] * 3
        lo[a], hi[a] = slice(0, -1), slice(1, None)
        y[tuple(lo)] -= d
        y[tuple(hi)] += d
    return y


def errors(x, h, **kw):
    """(computed - exact) residual in units of 2^-53 of w max|x| (w: the largest 1/h^2), per cell,
    and w."""
    nx, ny, nz = x.shape
    with cg.Solver(nx=nx, ny=ny, nz=nz, lx=nx * h[0], ly=ny * h[1], lz=nz * h[2], cx=nx * h[0] / 2, cy=ny * h[1] / 2,
                   radius=min(h[:2]), precision="mixed", solver="bicgstab", **kw) as s:
        ax = exact_ax(x, [s.cfg.lx / nx, s.cfg.ly / ny, s.cfg.lz / nz])
        b = np.array([float(v) for v in ax.ravel()])
        got = s.residual(b, x.ravel())
    want = [Fraction(v) - e for v, e in zip(b, ax.ravel())]
    w = max(1.0 / (d * d) for d in h)
    return np.array([float(Fraction(float(g)) - e) for g, e in zip(got, want)]).reshape(x.shape) / 2.0 ** -53 / w


@pytest.mark.parametrize("shape,h", [((12, 10, 24), (0.3, 0.7, 0.45)), ((9, 7, 66), (0.11, 0.13, 0.17))])
def test_rounding_is_not_one_sided(shape, h):
    """x uniform in [1, 2): its integers are exact, so the errors are the products', the conversion's
    and the store's, each rounded to nearest: the mean over 2880 and 4158 cells lies within 5 of
    its standard deviations of zero (errors of neighbouring cells are independent: each is a
    rounding of another number)."""
    e = errors(1.0 + np.random.default_rng(7).random(shape), h).ravel()
    assert abs(e.mean()) <= 5 * e.std() / np.sqrt(e.size), (e.mean(), e.std())

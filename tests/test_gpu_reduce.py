"""The block reduction's integer warp sum at the ends of its range: the drag and lift sums of
cfdgb_op_update_uf against math.fsum of the force field the same call returns.

The warp sum adds mantissas shifted to the warp's largest exponent (rounding at most 1/32 ulp
of the largest value a lane) and falls back to FP64 additions near the ends of the exponent
range; thread and block sums are FP64 additions of at most a few dozen values.  Together the
error is below 64 ulp of the sum of magnitudes."""
import math

import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu

NX, NY, NZ, LZ = 23, 11, 7, 7.0


def forces(us, vs):
    with cg.Solver(nx=NX, ny=NY, nz=NZ, lx=float(NX), ly=float(NY), lz=LZ, cx=8.0, cy=5.0, dt=0.5) as s:
        z = s.zeros()
        f = np.zeros((3,) + s.shape)
        eta = np.ones(s.shape)
        out = [s.zeros() for _ in range(3)]
        cd, cl = s.update_uf(eta, z, us(s.shape), vs(s.shape), z, *out, f)
    return cd, cl, f


def check(got, f):
    vals = (f[2:-2, 2:-2, 2:-2] * (-2.0 / LZ)).ravel()
    want, size = math.fsum(vals), math.fsum(np.abs(vals))
    assert abs(got - want) <= 64 * 2.0 ** -53 * size, (got, want, size)


@pytest.mark.parametrize("scale", [1.0, 1e-3, 1e150, 1e-150, 1e-279, 1e-290, 1e-305, 1e300])
def test_force_sums_at_every_magnitude(scale):
    rng = np.random.default_rng(3)
    spread = lambda sh: scale * rng.standard_normal(sh) * 2.0 ** rng.integers(-70, 1, sh)
    cd, cl, f = forces(spread, lambda sh: scale * rng.standard_normal(sh))
    check(cd, f[0])
    check(cl, f[1])


def test_force_sums_of_few_and_cancelling_values():
    """Zeros in most warps, one value alone, and values that cancel to their last place."""
    def one(sh):
        a = np.zeros(sh)
        a[5, 4, 3] = 0.1
        return a

    def cancel(sh):
        a = np.zeros(sh)
        a[3, 3, 3], a[3, 3, 4], a[9, 9, 8] = 1.0 + 2.0 ** -52, -1.0, 2.0 ** -60
        return a

    cd, cl, f = forces(one, cancel)
    assert cd == f[0].sum() * -2.0 / LZ != 0.0
    check(cl, f[1])
    assert cl != 0.0


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_values_reach_the_sum(bad):
    def poke(sh):
        a = np.ones(sh)
        a[6, 5, 4] = bad
        return a

    cd, cl, _ = forces(poke, lambda sh: np.ones(sh))
    assert not math.isfinite(cd) and math.isfinite(cl)

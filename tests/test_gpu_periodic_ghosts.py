"""The periodic z ghost fill on pairs of values (an even nz), single values (odd) and the thin grids
below four cells: after a step the two ghost layers on each side are exactly the images nz cells
away, in every field and over the whole padded plane."""
import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nz", [3, 4, 5, 6, 9, 16])
def test_ghosts_are_the_images(nz, precision):
    kw = dict(nx=21, ny=18, nz=nz, lx=8.0, ly=6.0, lz=0.3 * nz, cx=2.0, cy=3.0, dt=0.01, solver="jacobi", seed=2,
              amp=1e-2, tol=1e-9, precision=precision, **cg.BOUNDARY_SET)
    with cg.Solver(**kw) as s:
        s.init_fields()
        s.step(3)
        f = s.get_fields()
    for k in "uvwp":
        a = f[k]
        assert np.ptp(a) > 0 and np.all(np.isfinite(a)), k
        np.testing.assert_array_equal(a[:, :, :2], a[:, :, nz:nz + 2], err_msg=k)
        np.testing.assert_array_equal(a[:, :, nz + 2:], a[:, :, 2:4], err_msg=k)

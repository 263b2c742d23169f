"""QUICK convection-diffusion (the marching kernel) bit for bit against the oracle where its
tiles can go wrong: grids smaller than a tile, ragged rows and chunks, k lines split over two
tiles, one-cell remainders, periodic z, the stretched grid, divisors that need the double
correction (spacings of 0.3), and the eddy viscosity.  Fields change sign from cell to cell, so
both upwind branches run in every warp, and hold exact zeros."""
import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DT, RE = 0.004, 90.0


def fields(shape, seed):
    rng = np.random.default_rng(seed)
    out = [rng.standard_normal(shape) for _ in range(6)]
    for a in out:
        a[rng.random(shape) < 0.05] = 0.0
    return out


@pytest.mark.parametrize("h", [0.25, 0.3])
@pytest.mark.parametrize("dims", [(3, 3, 3), (5, 64, 3), (4, 7, 63), (9, 100, 5), (6, 5, 127), (5, 4, 128), (5, 6, 129),
                                  (7, 3, 300), (33, 17, 12), (160, 9, 7)])
@pytest.mark.parametrize("bc_z", ["zero_gradient", "periodic"])
def test_every_tile_shape(dims, h, bc_z):
    nx, ny, nz = dims
    lx, ly, lz = nx * h, ny * h, nz * h
    g = O.Grid(nx, ny, nz, lx, ly, lz, lx / 4, bc_z=bc_z)
    with cg.Solver(nx=nx, ny=ny, nz=nz, lx=lx, ly=ly, lz=lz, cx=lx / 4, cy=ly / 2, Re=RE, dt=DT, bc_z=bc_z) as s:
        f = fields(s.shape, nx + ny + nz)
        got, ref = [a.copy() for a in f[3:]], [a.copy() for a in f[3:]]
        s.convection_diffusion(*f[:3], *got)
    O.convection_diffusion(g, DT, 1.0 / RE, *f[:3], *ref)
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)


def test_stretched_grid_with_eddy_viscosity():
    dims = dict(nx=112, ny=104, nz=5, lx=17.0, ly=12.0, lz=3.0)
    g = O.Grid(112, 104, 5, 17.0, 12.0, 3.0, 6.5, gridder="sml")
    for les in (0, 1):
        with cg.Solver(grid="sml", cx=6.5, cy=6.0, Re=RE, dt=DT, les=les, **dims) as s:
            f = fields(s.shape, 5)
            got, ref = [a.copy() for a in f[3:]], [a.copy() for a in f[3:]]
            s.convection_diffusion(*f[:3], *got)
            nut = s.smagorinsky(*f[:3]) if les else None
        O.convection_diffusion(g, DT, 1.0 / RE, *f[:3], *ref, nut=nut)
        for a, b in zip(got, ref):
            np.testing.assert_array_equal(a, b)

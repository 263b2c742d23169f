"""The FP64 V-cycle's pair passes (levels with an even nz) where they can go wrong: one pair a
row, odd rows and planes, levels that halve along some axes only, no halving along z, rows wider
than a warp, both row scalings, periodic z.  The preconditioner changes the path to the
solution, not the solution: every solve ends below 1e-10, in a few dozen iterations, with the
plain FP64 BiCGSTAB's fields (two solves at 1e-10 agree to 1e-7 on these grids)."""
import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu

SHAPES = [(16, 8, 4), (12, 6, 10), (16, 10, 6), (9, 8, 8), (8, 7, 6), (24, 20, 2 * 7), (16, 12, 5), (40, 24, 72),
          (64, 32, 16), (6, 4, 258)]


@pytest.mark.parametrize("solver", ["bicgstab", "jacobi"])
@pytest.mark.parametrize("shape", SHAPES)
def test_fp64_vcycle_on_ragged_levels(shape, solver):
    nx, ny, nz = shape
    dom = dict(nx=nx, ny=ny, nz=nz, lx=float(nx), ly=float(ny), lz=0.8 * nz, cx=nx / 2.0, cy=ny / 2.0, radius=0.75,
               project_rhs=1, seed=3, amp=1e-3, dt=0.01, tol=1e-10, solver=solver, maxit=20000)
    check(dom)


@pytest.mark.parametrize("solver", ["bicgstab", "jacobi"])
@pytest.mark.parametrize("shape", [(16, 8, 4), (24, 12, 4), (32, 16, 8), (20, 10, 16)])
def test_fp64_vcycle_with_periodic_z(shape, solver):
    nx, ny, nz = shape
    dom = dict(nx=nx, ny=ny, nz=nz, lx=float(nx), ly=float(ny), lz=0.8 * nz, cx=nx / 2.0, cy=ny / 2.0, radius=0.75,
               seed=3, amp=1e-3, dt=0.01, tol=1e-10, solver=solver, maxit=20000, **cg.BOUNDARY_SET)
    check(dom)


def check(dom):
    runs = {}
    for key, kw in (("mg", dict(precond="multigrid")), ("plain", {})):
        with cg.Solver(**kw, **dom) as s:
            s.init_fields()
            st = s.step(3)
            runs[key] = (s.get_fields(), st)
    st = runs["mg"][1]
    assert all(r.status == 0 and r.relres < 1e-10 for r in st[1:]), [(r.status, r.relres) for r in st]
    assert all(r.iters <= 40 for r in st[1:]), [r.iters for r in st]
    core = (slice(2, -2),) * 3
    a, b = runs["mg"][0], runs["plain"][0]
    scale = np.sqrt(sum(np.linalg.norm(b[k][core]) ** 2 for k in "uvw"))
    for k in "uvw":
        assert np.linalg.norm(a[k][core] - b[k][core]) <= 1e-7 * scale, k
    p, q = a["p"][core], b["p"][core]
    assert np.linalg.norm((p - p.mean()) - (q - q.mean())) <= 1e-6 * np.linalg.norm(q - q.mean())

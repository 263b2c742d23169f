"""The MIXED refinement's residual from 64-bit integers where its pairs, rows and shuffles can go
wrong: one pair a row, rows that fill a warp or not, rows over several tiles, an odd number of
rows, one plane a chunk, anisotropic spacings, periodic z, both row scalings; and the FMA chain
it leaves to (odd nz, the stretched grid are other tests').  A wrong residual anywhere would make
the refinement converge to another solution: against the FP64 run of the same case the pressure
agrees to 1e-5 and the velocity to 1e-6 (the FP32 stencil's error; measured ~1e-7 and ~1e-8),
and every solve ends below 1e-10 in that residual."""
import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bset", [False, True], ids=["table", "boundary_set"])
@pytest.mark.parametrize("solver", ["bicgstab", "jacobi", "cg"])
@pytest.mark.parametrize("shape", [(5, 3, 4), (6, 5, 6), (9, 7, 10), (40, 9, 64), (12, 33, 66), (7, 5, 130), (33, 16, 12),
                                   (160, 3, 8)])
def test_mixed_solution_matches_fp64(shape, solver, bset):
    nx, ny, nz = shape
    kw = dict(nx=nx, ny=ny, nz=nz, lx=0.5 * nx, ly=0.5 * ny, lz=0.2 * nz, cx=0.15 * nx, cy=0.25 * ny, radius=0.4,
              dt=0.01, solver=solver, seed=3, amp=1e-3, maxit=20000, tol=1e-10,
              **(cg.BOUNDARY_SET if bset else dict(project_rhs=1)))
    out = []
    for precision in ("mixed", "fp64"):
        with cg.Solver(precision=precision, **kw) as s:
            s.init_fields()
            st = s.step(3)
            out.append(s.get_fields())
        assert all(r.status == 0 and r.relres < 1e-10 for r in st[1:]), [(r.status, r.relres) for r in st]
    core = (slice(2, -2),) * 3
    a, b = out
    scale = np.sqrt(sum(np.linalg.norm(b[k][core]) ** 2 for k in "uvw"))
    for k in "uvw":
        assert np.linalg.norm(a[k][core] - b[k][core]) <= 1e-6 * scale, k
    p, q = a["p"][core], b["p"][core]
    assert np.linalg.norm((p - p.mean()) - (q - q.mean())) <= 1e-5 * np.linalg.norm(q - q.mean())

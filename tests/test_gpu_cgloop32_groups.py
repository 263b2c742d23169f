"""FP32 CG sweeps in one cooperative launch with four quads a thread (more than 8192 cells a
multiprocessor), on whole and ragged ranges, against a kernel a phase; and which of the two a grid
takes.  Both runs end below 1e-11 in the FP64 residual, so the fields agree to 1e-8 of the velocity
and 1e-7 of the mean-free pressure (its constant and the solve error, a few hundred times the
tolerance on these grids)."""
import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu


def run(monkeypatch, loop, shape, bset, tol=1e-11):
    nx, ny, nz = shape
    if loop:
        monkeypatch.delenv("CFDGB_NO_LOOP", raising=False)
    else:
        monkeypatch.setenv("CFDGB_NO_LOOP", "1")
    with cg.Solver(nx=nx, ny=ny, nz=nz, lx=0.5 * nx, ly=0.5 * ny, lz=0.4 * nz, cx=0.15 * nx, cy=0.25 * ny, radius=0.4,
                   dt=0.01, precision="mixed", solver="cg", tol=tol, seed=5, amp=1e-3, maxit=20000,
                   **(cg.BOUNDARY_SET if bset else dict(project_rhs=1))) as s:
        s.init_fields()
        st = s.step(3)
        f = s.get_fields()
        ran = {k for k, v in s.kernel_stats().items() if v[1] > 0}
    assert all(r.status == 0 and r.relres < tol for r in st[1:]), [(r.status, r.relres) for r in st]
    return f, ran


@pytest.mark.parametrize("bset", [False, True], ids=["table", "boundary_set"])
@pytest.mark.parametrize("shape", [(200, 130, 64), (201, 131, 52)])
def test_four_quads_a_thread_match_a_kernel_a_phase(monkeypatch, shape, bset):
    a, ran = run(monkeypatch, True, shape, bset)
    assert "cg_loop32" in ran and "cg_pq32" not in ran
    b, ran = run(monkeypatch, False, shape, bset)
    assert "cg_pq32" in ran and "cg_loop32" not in ran
    core = (slice(2, -2),) * 3
    scale = np.sqrt(sum(np.linalg.norm(b[k][core]) ** 2 for k in "uvw"))
    for k in "uvw":
        assert np.linalg.norm(a[k][core] - b[k][core]) <= 1e-8 * scale, k
    p, q = a["p"][core], b["p"][core]
    assert np.linalg.norm((p - p.mean()) - (q - q.mean())) <= 1e-7 * np.linalg.norm(q - q.mean())


@pytest.mark.parametrize("shape,loop", [((3, 3, 3), True), ((64, 76, 17), True), ((40, 160, 128), True),
                                        ((12, 200, 160), False), ((160, 128, 128), False)])
def test_which_form_a_grid_takes(monkeypatch, shape, loop):
    """Planes or grids beyond a multiprocessor's shared memory and registers stay on a kernel a
    phase."""
    ran = run(monkeypatch, True, shape, False, 1e-6)[1]
    assert ("cg_loop32" in ran, "cg_pq32" in ran) == (loop, not loop)

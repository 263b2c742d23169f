"""FP32 CG sweeps in one cooperative launch, where their partition can go wrong: fewer cells than a
warp, ranges shorter than a plane and longer than two, a last block of a few cells, every number of
groups a thread (quads 1, 2, 4; single cells 4, 16), periodic z, and planes too large for the
shared memory (left to a kernel a phase).  Against the same run with a kernel a phase
(CFDGB_NO_LOOP): both end below 1e-11 in the FP64 residual, so the fields agree to 1e-8 of the
velocity and 1e-7 of the mean-free pressure (its constant and the solve error, a few hundred times
the tolerance on these grids).  And the failure path of the barrier's wait."""
import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (5, 4, 4), (11, 7, 5), (97, 13, 4), (64, 76, 16), (64, 76, 17), (120, 70, 64), (150, 120, 64),
          (130, 100, 61), (12, 200, 160)]


def run(monkeypatch, loop, **kw):
    if loop:
        monkeypatch.delenv("CFDGB_NO_LOOP", raising=False)
    else:
        monkeypatch.setenv("CFDGB_NO_LOOP", "1")
    with cg.Solver(precision="mixed", solver="cg", tol=1e-11, seed=5, amp=1e-3, maxit=20000, **kw) as s:
        s.init_fields()
        st = s.step(3)
        f = s.get_fields()
    assert all(r.status == 0 and r.relres < 1e-11 for r in st[1:]), [(r.status, r.relres) for r in st]
    return f


@pytest.mark.parametrize("bset", [False, True], ids=["table", "boundary_set"])
@pytest.mark.parametrize("shape", SHAPES)
def test_one_launch_matches_a_kernel_a_phase(monkeypatch, shape, bset):
    nx, ny, nz = shape
    kw = dict(nx=nx, ny=ny, nz=nz, lx=0.5 * nx, ly=0.5 * ny, lz=0.4 * nz, cx=0.15 * nx, cy=0.25 * ny, radius=0.4,
              dt=0.01, **(cg.BOUNDARY_SET if bset else dict(project_rhs=1)))
    a = run(monkeypatch, True, **kw)
    b = run(monkeypatch, False, **kw)
    core = (slice(2, -2),) * 3
    scale = np.sqrt(sum(np.linalg.norm(b[k][core]) ** 2 for k in "uvw"))
    for k in "uvw":
        assert np.linalg.norm(a[k][core] - b[k][core]) <= 1e-8 * scale, k
    p, q = a["p"][core], b["p"][core]
    assert np.linalg.norm((p - p.mean()) - (q - q.mean())) <= 1e-7 * np.linalg.norm(q - q.mean())


def test_wait_that_runs_out_ends_the_launch(monkeypatch):
    monkeypatch.setenv("CFDGB_TEST_WAIT_FAULT", "1")
    kw = dict(nx=64, ny=32, nz=16, lx=32.0, ly=16.0, lz=8.0, cx=8.0, cy=8.0, dt=0.01, project_rhs=1)
    with cg.Solver(precision="mixed", solver="cg", tol=1e-11, seed=5, amp=1e-3, **kw) as s:
        s.init_fields()
        with pytest.raises(cg.CfdgbError, match="bounded wait between blocks"):
            s.step(2)
    monkeypatch.delenv("CFDGB_TEST_WAIT_FAULT")
    with cg.Solver(precision="mixed", solver="cg", tol=1e-11, seed=5, amp=1e-3, **kw) as s:
        s.init_fields()
        assert s.step(2)[1].status == 0


def test_pipeline_wait_that_runs_out_ends_the_launch(monkeypatch):
    """The kernels a phase that larger grids take keep their own bounded waits."""
    monkeypatch.setenv("CFDGB_NO_LOOP", "1")
    monkeypatch.setenv("CFDGB_TEST_WAIT_FAULT", "1")
    kw = dict(nx=128, ny=64, nz=16, lx=32.0, ly=16.0, lz=4.0, cx=8.0, cy=8.0)
    s = cg.Solver(precision="mixed", solver="cg", **kw)
    monkeypatch.delenv("CFDGB_TEST_WAIT_FAULT")
    with s:
        s.init_fields()
        s.step(1)  # step 1 has no pressure solve
        with pytest.raises(cg.CfdgbError, match="FP32 stencil pipeline"):
            s.step(1)
        s.init_fields()
        assert [r.status for r in s.step(3)] == [0, 0, 0]

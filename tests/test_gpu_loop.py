"""The FP64 Krylov iterations in one cooperative launch, where their partition can go wrong:
fewer cells than a warp, a last block of a few cells, the change from one cell a thread to
several, periodic z, the stretched grid's factored rows (both scalings), CG.  Against the same
run with a kernel a phase (CFDGB_NO_LOOP): the same iteration on another summation order, so at
1e-11 the fields agree to 1e-8 of the velocity and the mean-free pressure (the solve error, a
few hundred times the tolerance on these grids).  And the failure path of the barrier's wait."""
import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu


def run(monkeypatch, loop, **kw):
    if loop:
        monkeypatch.delenv("CFDGB_NO_LOOP", raising=False)
    else:
        monkeypatch.setenv("CFDGB_NO_LOOP", "1")
    with cg.Solver(tol=1e-11, seed=5, amp=1e-3, maxit=20000, **kw) as s:
        s.init_fields()
        st = s.step(3)
        f = s.get_fields()
    assert all(r.status == 0 and r.relres < 1e-11 for r in st[1:]), [(r.status, r.relres) for r in st]
    return f, st


def agree(a, b):
    core = (slice(2, -2),) * 3
    scale = np.sqrt(sum(np.linalg.norm(b[k][core]) ** 2 for k in "uvw"))
    for k in "uvw":
        assert np.linalg.norm(a[k][core] - b[k][core]) <= 1e-8 * scale, k
    p, q = a["p"][core], b["p"][core]
    assert np.linalg.norm((p - p.mean()) - (q - q.mean())) <= 1e-8 * np.linalg.norm(q - q.mean())


SHAPES = [(3, 3, 3), (5, 4, 3), (11, 7, 5), (97, 13, 4), (64, 76, 16), (64, 76, 17), (50, 40, 41)]


@pytest.mark.parametrize("bset", [False, True], ids=["table", "boundary_set"])
@pytest.mark.parametrize("solver", ["bicgstab", "jacobi", "cg"])
@pytest.mark.parametrize("shape", SHAPES)
def test_one_launch_matches_a_kernel_a_phase(monkeypatch, shape, solver, bset):
    nx, ny, nz = shape
    kw = dict(nx=nx, ny=ny, nz=nz, lx=0.5 * nx, ly=0.5 * ny, lz=0.4 * nz, cx=0.15 * nx, cy=0.25 * ny, radius=0.4,
              dt=0.01, solver=solver, **(cg.BOUNDARY_SET if bset else dict(project_rhs=1)))
    a, _ = run(monkeypatch, True, **kw)
    b, _ = run(monkeypatch, False, **kw)
    agree(a, b)


@pytest.mark.parametrize("nz", [4, 9])
def test_stretched_grid(monkeypatch, nz):
    """Jacobi-scaled rows on the boundary set (consistent there); one cell a thread and several."""
    kw = dict(nx=112, ny=104, nz=nz, lx=17.0, ly=12.0, lz=3.0, cx=6.5, cy=6.0, grid="sml", Re=100.0, dt=0.005,
              solver="jacobi", **cg.BOUNDARY_SET)
    a, _ = run(monkeypatch, True, **kw)
    b, _ = run(monkeypatch, False, **kw)
    agree(a, b)


def test_stretched_grid_unscaled_rows(monkeypatch):
    """SPE rows: step 2 of the unperturbed run carries the solve that converges on this grid."""
    out = []
    for loop in (True, False):
        if loop:
            monkeypatch.delenv("CFDGB_NO_LOOP", raising=False)
        else:
            monkeypatch.setenv("CFDGB_NO_LOOP", "1")
        with cg.Solver(nx=120, ny=110, nz=9, lx=17.0, ly=12.0, lz=3.0, cx=6.5, cy=6.0, grid="sml", Re=100.0, dt=0.005,
                       solver="bicgstab", tol=1e-11, maxit=20000) as s:
            s.init_fields()
            st = s.step(2)
            out.append(s.get_fields())
        assert st[1].status == 0 and st[1].relres < 1e-11
    agree(*out)


@pytest.mark.parametrize("solver", ["jacobi", "cg"])
@pytest.mark.parametrize("graph", [True, False])
def test_barrier_wait_timeout_is_reported_and_the_context_recovers(monkeypatch, solver, graph):
    kw = dict(nx=128, ny=64, nz=16, lx=32.0, ly=16.0, lz=4.0, cx=8.0, cy=8.0, solver=solver)
    if not graph:
        monkeypatch.setenv("CFDGB_NO_STEP_GRAPH", "1")
    monkeypatch.setenv("CFDGB_TEST_WAIT_FAULT", "1")
    s = cg.Solver(**kw)
    monkeypatch.delenv("CFDGB_TEST_WAIT_FAULT")
    with s:
        s.init_fields()
        s.step(1)  # step 1 has no pressure solve
        with pytest.raises(cg.CfdgbError) as e:
            s.step(1)
        assert e.value.status == cg.ECUDA
        s.init_fields()
        st = s.step(3)
        f = s.get_fields()
    with cg.Solver(**kw) as ref:
        ref.init_fields()
        st_ref = ref.step(3)
        f_ref = ref.get_fields()
    assert [(r.status, r.iters, r.cd) for r in st] == [(r.status, r.iters, r.cd) for r in st_ref]
    for k in "uvwp":
        np.testing.assert_array_equal(f[k], f_ref[k])

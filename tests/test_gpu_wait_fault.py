"""A wait between the blocks of the one-launch Krylov iterations that runs out, beyond the one
case that ends in block 0: it is reported whichever block left last and whatever the other steps
of the call return, and it belongs to that solve alone.  CFDGB_TEST_WAIT_FAULT (read at
cfdgb_create) makes one bounded wait of the next launch run out after half a millisecond."""
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu

KW = dict(nx=128, ny=64, nz=16, lx=32.0, ly=16.0, lz=4.0, cx=8.0, cy=8.0)


def started(monkeypatch, request, graph, **kw):
    if not graph:
        monkeypatch.setenv("CFDGB_NO_STEP_GRAPH", "1")
    monkeypatch.setenv("CFDGB_TEST_WAIT_FAULT", request)
    s = cg.Solver(**{**KW, **kw})
    monkeypatch.delenv("CFDGB_TEST_WAIT_FAULT")
    s.init_fields()
    s.step(1)  # step 1 has no pressure solve
    return s


@pytest.mark.parametrize("solver", ["jacobi", "cg"])
def test_the_next_solve_starts_clean(monkeypatch, solver):
    """No cfdgb_init_fields in between: the fault is the failed solve's own.  (Host-driven: there
    the failed step ends before it corrects the velocity with an unfinished pressure.)"""
    with started(monkeypatch, "1", False, solver=solver) as s:
        with pytest.raises(cg.CfdgbError, match="bounded wait between blocks") as e:
            s.step(1)
        assert e.value.status == cg.ECUDA
        assert [r.status for r in s.step(2)] == [0, 0]


@pytest.mark.parametrize("solver", ["jacobi", "cg"])
@pytest.mark.parametrize("graph", [True, False])
def test_block_0_leaving_last_does_not_hide_it(monkeypatch, solver, graph):
    """Request 2: the solve carries the fault of a block that gave up at the chunk's last barrier;
    block 0, whose own waits all ended, writes the solve's scalars after that."""
    with started(monkeypatch, "2", graph, solver=solver) as s:
        with pytest.raises(cg.CfdgbError, match="bounded wait between blocks") as e:
            s.step(1)
        assert e.value.status == cg.ECUDA


@pytest.mark.parametrize("solver", ["jacobi", "cg"])
@pytest.mark.parametrize("graph", [True, False])
def test_capped_steps_of_the_same_call_do_not_hide_it(monkeypatch, solver, graph):
    """Callers accept CFDGB_ENOCONV, the lower status: the call must still end with CFDGB_ECUDA."""
    with started(monkeypatch, "1", graph, solver=solver, tol=1e-13, maxit=5) as s:
        with pytest.raises(cg.CfdgbError, match="bounded wait between blocks") as e:
            s.step(4, allow_noconv=True)
        assert e.value.status == cg.ECUDA

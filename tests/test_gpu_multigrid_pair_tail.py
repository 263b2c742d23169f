"""Which one-block tail a V-cycle takes, and the pair tail alone against the general one: the plan is
read from the trace, and CFDGB_MG_GENERAL_TAIL changes that kernel only (the marching kernels stay), so
a difference is the tail's.  Every value is formed by the same rounded sequence: runs agree bit for
bit.  Pairs along z, y (nz odd) and x (ny and nz odd), one, two and three pairs a thread, coarsest
levels whose inverse fits shared memory or not; a coarsest level of more than 256 cells has no dense
inverse and keeps the general tail."""
import re

import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu

PAIRS = [(32, 16, 8), (40, 24, 10), (120, 40, 12), (64, 9, 9), (16, 176, 4), (24, 24, 18), (96, 4, 16), (64, 24, 5),
         (48, 16, 9), (64, 13, 7), (12, 12, 96)]
GENERAL = [(30, 20, 9), (28, 15, 7), (72, 13, 5), (36, 60, 6)]
PERIODIC = [(32, 16, 8), (16, 176, 4), (96, 4, 16)]


def run(shape, solver, bset, capfd):
    nx, ny, nz = shape
    capfd.readouterr()
    with cg.Solver(nx=nx, ny=ny, nz=nz, lx=0.27 * nx, ly=0.23 * ny, lz=0.19 * nz, cx=0.1 * nx, cy=0.115 * ny,
                   radius=0.3, dt=0.01, solver=solver, precision="mixed", precond="multigrid", seed=5, amp=1e-3,
                   tol=1e-8, **(cg.BOUNDARY_SET if bset else dict(project_rhs=1))) as s:
        plan = re.search(r"multigrid: .* in one block(.*)", capfd.readouterr().err).group(1).strip()
        s.init_fields()
        st = s.step(2)
        return plan, [(r.iters, r.outer, r.relres) for r in st], s.get_fields(), s.launch_count()


@pytest.mark.parametrize("solver", ["bicgstab", "jacobi"])
@pytest.mark.parametrize("shape,bset", [(q, False) for q in PAIRS] + [(q, True) for q in PERIODIC])
def test_pair_tail_runs_and_matches_the_general_one(shape, bset, solver, monkeypatch, capfd):
    monkeypatch.setenv("CFDGB_TRACE", "1")
    plan, st, f, n = run(shape, solver, bset, capfd)
    assert plan == "on cell pairs"
    monkeypatch.setenv("CFDGB_MG_GENERAL_TAIL", "1")
    plan, st2, f2, n2 = run(shape, solver, bset, capfd)
    assert plan == ""
    assert st == st2 and n == n2
    for k in "uvwp":
        assert np.array_equal(f[k], f2[k]), (k, float(np.abs(f[k] - f2[k]).max()))


@pytest.mark.parametrize("shape", GENERAL)
def test_levels_without_a_dense_inverse_keep_the_general_tail(shape, monkeypatch, capfd):
    monkeypatch.setenv("CFDGB_TRACE", "1")
    assert run(shape, "bicgstab", False, capfd)[0] == ""

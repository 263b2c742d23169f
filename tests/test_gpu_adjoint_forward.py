"""The objective that cfdgb_forward returns against the drag that cfdgb_step reports on the same run:
FP64 takes the same arithmetic (equal but for the order of the average's additions), MIXED another
form of the refinement's residual, so the two agree as solves to the tolerance do: 1e-8 for
1e-11, a few hundred times the tolerance on this grid."""
import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,precond,bound", [("fp64", "none", 1e-14), ("fp64", "multigrid", 1e-14),
                                                     ("mixed", "none", 1e-8), ("mixed", "multigrid", 1e-8)])
def test_objective_is_the_mean_drag_of_the_steps(precision, precond, bound):
    kw = dict(nx=64, ny=32, nz=8, lx=16.0, ly=8.0, lz=2.0, cx=4.0, cy=4.0, Re=100.0, dt=0.005, tol=1e-11,
              solver="jacobi", project_rhs=1, precision=precision, precond=precond)
    with cg.Solver(**kw) as s:
        s.init_fields()
        cd = np.array([r.cd for r in s.step(8)])
        s.init_fields()
        J = s.forward(8, 5, 8, 3)
    want = cd[4:].mean()
    assert abs(J - want) <= bound * abs(want), (J, want)

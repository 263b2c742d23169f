"""Contexts stepped by threads of their own at the same time, each with its one-launch iterations (a
block on every multiprocessor, with grid barriers): their launches take turns on the GPU, and every
result is the one the context gives alone, bit for bit."""
import threading

import numpy as np
import pytest

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

pytestmark = pytest.mark.gpu

KINDS = [dict(nx=96, ny=48, nz=4, solver="bicgstab"), dict(nx=64, ny=76, nz=17, solver="cg"),
         dict(nx=64, ny=76, nz=16, solver="jacobi"), dict(nx=97, ny=48, nz=16, solver="cg", precision="mixed"),
         dict(nx=96, ny=48, nz=4, solver="bicgstab", precision="mixed"),
         dict(nx=96, ny=48, nz=16, solver="jacobi", precision="mixed", precond="multigrid")]


def steps(kw, seed, out, key):
    n = {a: kw[f"n{a}"] for a in "xyz"}
    try:
        with cg.Solver(lx=0.25 * n["x"], ly=0.25 * n["y"], lz=0.25 * n["z"], cx=0.06 * n["x"], cy=0.125 * n["y"],
                       dt=0.005, tol=1e-9, seed=seed, amp=1e-3, project_rhs=1, maxit=20000, **kw) as s:
            s.init_fields()
            st = s.step(6)
            out[key] = ([(r.status, r.iters, r.relres, r.cd) for r in st], s.get_fields())
    except Exception as e:  # raised in the test's thread
        out[key] = e


def test_threads_give_the_results_of_one_context_at_a_time():
    jobs = [(q, seed) for q in range(len(KINDS)) for seed in (1, 2)]
    alone, together = {}, {}
    for q, seed in jobs:
        steps(KINDS[q], seed, alone, (q, seed))
    threads = [threading.Thread(target=steps, args=(KINDS[q], seed, together, (q, seed))) for q, seed in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for key in jobs:
        for r in (alone[key], together[key]):
            assert not isinstance(r, Exception), (key, r)
        assert alone[key][0] == together[key][0], key
        assert all(r[0] == 0 for r in alone[key][0]), key
        for k in "uvwp":
            np.testing.assert_array_equal(alone[key][1][k], together[key][1][k])

"""bench.py's end-to-end leg without a GPU: a solve at its iteration cap is counted, not raised."""
from types import SimpleNamespace as S

import numpy as np

import bench


class FakeError(RuntimeError):
    pass


class FakeSolver:
    """Steps whose 7th solve hits the cap; raises as the binding does unless told not to."""
    shape, cells, stream = (5, 5, 5), 1, 0

    def __init__(self, **kw):
        self.kw, self.n = kw, 0

    def __enter__(self):
        return self

    def __exit__(self, *a):
        pass

    def init_fields(self):
        pass

    def set_fields(self, *a):
        pass

    def get_fields(self, host):
        return host

    def step(self, n, allow_noconv=False):
        out = []
        for _ in range(n):
            self.n += 1
            capped = self.n == 7
            out.append(S(step=self.n, iters=self.kw["maxit"] if capped else 9, status=-3 if capped else 0,
                         relres=3e-8 if capped else 5e-9))
            if capped and not allow_noconv:
                raise FakeError("cfdgb status -3: step finished with status -3")
        return out


class FakeEvent:
    def __init__(self, enable_timing):
        pass

    def record(self, stream):
        pass

    def elapsed_time(self, other):
        return 250.0


def fakes():
    cuda = S(ExternalStream=lambda s: s, Event=FakeEvent, synchronize=lambda: None)
    torch = S(cuda=cuda, float64=None, empty=lambda shape, dtype, pin_memory: S(numpy=lambda: np.zeros(shape)))
    return S(Solver=FakeSolver, CfdgbError=FakeError), torch, S(world=1, barrier=lambda: None, max=lambda x: x)


def test_a_capped_solve_is_counted():
    line = bench.e2e_line(*fakes(), "c2", 5, 3, 5000)
    assert line["value"] == bench.cells_of("c2") * 5 / 0.25
    assert line["h2d_bytes_per_step"] == line["d2h_bytes_per_step"] == 4 * 8 * 125
    assert (line["capped_solves"], line["unconverged_solves"]) == (1, 1)
    assert line["failure"].startswith("1 of 5 timed solves")


def test_no_failure_is_named_when_every_solve_converged():
    line = bench.e2e_line(*fakes(), "c2", 3, 3, 5000)
    assert line["capped_solves"] == line["unconverged_solves"] == 0 and "failure" not in line


def test_the_warm_up_may_hold_the_capped_solve():
    line = bench.e2e_line(*fakes(), "c2", 2, 8, 5000)
    assert line["capped_solves"] == 0

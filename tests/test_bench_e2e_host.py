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
            out.append(S(step=self.n, iters=self.kw.get("maxit", 5000) if capped else 9, status=-3 if capped else 0,
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


def test_one_launch_kernels_have_a_roofline(tmp_path):
    """Grids of up to a few million cells run their Krylov iterations in cg_loop64, bicg_loop64 and
    cg_loop32: words and flops an iteration, times the iterations a launch."""
    cells = 1_000_000
    for name, word, flops in (("bicg_loop64", 19, 48), ("cg_loop64", 11, 23)):
        prof = {name: (40.0, 8), "update_uf": (1.0, 4)}  # 8 launches of 5 ms, 100 iterations each
        r, share = bench.roofline(prof, cells, 8, "64", 5000.0, "measured", tmp_path / "none", 800)
        assert r["kernel"] == name and r["avg_launch_us"] == 5000.0
        assert r["achieved"] == round(word * 8 * cells * 100 / 5e-3 / 1e9, 1)
        assert share == {name: round(40 / 41, 4), "update_uf": round(1 / 41, 4)}
        a = bench.alu_roofline(prof, cells, {"fp64_tflops": 2.0}, 800)
        assert a["kernel"] == name and a["achieved"] == round(flops * cells * 100 / 5e-3 / 1e12, 4)
    r, _ = bench.roofline({"cg_loop32": (2.0, 4)}, cells, 4, "32", 5000.0, "measured", tmp_path / "none", 200)
    assert r["kernel"] == "cg_loop32" and r["achieved"] == round(10 * 4 * cells * 50 / 5e-4 / 1e9, 1)

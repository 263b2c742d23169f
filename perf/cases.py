"""The work this framework is used for, as cases that can be timed and compared.

Three kinds of pass, each through the public Python binding:

  run      a short simulation: host fields in (pinned), `steps` projection steps, fields out
           (pinned), as a coupled host program calls it.
  poisson  the allocation-free Poisson solve on device buffers of the caller.
  adjoint  the drag-gradient pair forward + backward with checkpoints.

Grids are those of the package's own configurations and tests (96x48x4, 120x40x12,
256x128x32, 256x128x64, 512x256x64, 768x384x96, 1024x512x128, the stretched 190x210x40) and
generic odd ones.  Perturbed runs on the zero-gradient boundary table project the right-hand
side (`project_rhs`), which keeps their Neumann problem solvable; the others run the boundary
set with the convective outflow.  Poisson tolerances are tight (1e-11, 1e-12) so that two
correct solves of a step agree: at a loose one the fields differ by the solve error itself.
The pressure of an all-Neumann problem is free up to a constant.  FP64 solves hold it to FP64
rounding (the V-cycle's own linear map where one preconditions), MIXED ones only to that of an
FP32 mean, so a MIXED run fetches u, v and w, which the pressure's gradient corrects, and the
forces, as programs that gather flow statistics do.
"""
import ctypes as C
import math

import numpy as np
import torch

import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg

AMP = 1e-3  # of the seeded perturbation of u, v, w


def _run(name, nx, ny, nz, h, solver, precision, steps, precond="none", bset=False, grid="uniform", Re=200.0,
         dt=0.002, tol=1e-12):
    return dict(name=name, kind="run", nx=nx, ny=ny, nz=nz, h=h, solver=solver, precision=precision, steps=steps,
                precond=precond, bset=bset, grid=grid, Re=Re, dt=dt, tol=tol)


def listed():
    return [
        # the drop-in default on the reference's own small case: launches and latency count
        _run("fp64 small", 96, 48, 4, 0.25, "bicgstab", "fp64", 10, Re=100.0, dt=0.005),
        # a service that may not allocate: one solve on its own device buffers
        dict(name="static poisson", kind="poisson", nx=40, ny=24, nz=16, h=0.25, solver="jacobi", tol=1e-12),
        # FP64 CG on an odd grid (no vector width divides a row)
        _run("fp64 cg odd", 151, 77, 27, 0.125, "cg", "fp64", 4),
        # the reference's algorithm in FP64 on the gradient workload's grid
        _run("fp64 jacobi", 256, 128, 32, 0.09375, "jacobi", "fp64", 3, Re=100.0, dt=0.004),
        # the reference's default stretched grid
        _run("fp64 stretched", 190, 210, 40, 0.0, "jacobi", "fp64", 3, bset=True, grid="sml", Re=40.0),
        # FP64 throughout with the V-cycle: who needs FP64 kernels but not the reference's iteration
        _run("fp64 multigrid", 512, 256, 64, 0.0625, "jacobi", "fp64", 4, precond="multigrid", bset=True),
        # small and ragged MIXED multigrid run: latency, levels that do not all halve
        _run("mixed multigrid ragged", 120, 40, 12, 0.25, "jacobi", "mixed", 8, precond="multigrid", Re=100.0,
             dt=0.005),
        # production precision and solver on the 8.4 M cell grid
        _run("mixed multigrid", 512, 256, 64, 0.0625, "jacobi", "mixed", 8, precond="multigrid", bset=True),
        # 28 M cells, the gradient stress workload's aspect and nz (96: not a power of two)
        _run("mixed multigrid nz96", 768, 384, 96, 0.0625, "bicgstab", "mixed", 5, precond="multigrid", Re=300.0,
             dt=0.001, tol=1e-11),
        # the largest: 67 M cells
        _run("mixed multigrid large", 1024, 512, 128, 0.03125, "jacobi", "mixed", 5, precond="multigrid", bset=True,
             Re=300.0, dt=0.001, tol=1e-11),
        # FP32 CG sweeps in FP64 refinement
        _run("mixed cg", 256, 128, 64, 0.125, "cg", "mixed", 3, tol=1e-11),
        # forward and backward: drag gradient with respect to inlet profile and solid fraction
        dict(name="adjoint mixed multigrid", kind="adjoint", nx=256, ny=128, nz=32, h=0.09375, solver="jacobi",
             precision="mixed", precond="multigrid", steps=8, first=5, ckpt=4, Re=100.0, dt=0.004, tol=1e-12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fp64", "fp64 multigrid", "mixed", "mixed multigrid", "mixed multigrid", "stretched", "poisson",
                       "adjoint"])
    h = rng.choice([0.0625, 0.09375, 0.125, 0.25])
    if kind == "poisson":
        n = _log(rng, 9, 64)
        return dict(kind="poisson", nx=n, ny=_log(rng, 7, 60), nz=_log(rng, 5, 64), h=h,
                    solver=rng.choice(["bicgstab", "jacobi"]), tol=1e-12)
    if kind == "adjoint":
        m = rng.choice([1, 2, 3, 4])
        return dict(kind="adjoint", nx=64 * m, ny=32 * m, nz=8 * rng.randint(1, 4), h=0.375 / m, solver="jacobi",
                    precision=rng.choice(["fp64", "mixed"]), precond="multigrid", steps=rng.randint(4, 8), first=3,
                    ckpt=rng.randint(2, 4), Re=100.0, dt=0.004, tol=1e-12)
    bset = rng.random() < 0.5
    if kind == "stretched":
        c = _run("", 2 * rng.randint(56, 95), 2 * rng.randint(52, 105), rng.randint(8, 40), 0.0, "jacobi", "fp64", 3,
                 bset=True, grid="sml", Re=40.0)
    elif kind == "fp64":
        c = _run("", _log(rng, 48, 256), _log(rng, 24, 128), _log(rng, 4, 40), h,
                 rng.choice(["bicgstab", "jacobi", "cg"]), "fp64", 3, bset=bset)
    elif kind == "mixed":
        c = _run("", _log(rng, 48, 256), _log(rng, 24, 128), _log(rng, 4, 64), h,
                 rng.choice(["bicgstab", "jacobi", "cg"]), "mixed", 3, bset=bset, tol=1e-11)
    else:  # grids that coarsen: a small odd or even base, halved a few times
        k = 2 ** rng.randint(3, 5)
        # (periodic z: nz halves down to one)
        m = rng.choice([2, 4]) if bset else rng.randint(2, 6)
        c = _run("", k * rng.randint(6, 16), k * rng.randint(3, 8), (k // 2) * m, h,
                 rng.choice(["bicgstab", "jacobi"]), "mixed" if kind == "mixed multigrid" else "fp64",
                 rng.randint(3, 6), precond="multigrid", bset=bset, tol=1e-11)
    del c["name"]
    return c


def _lengths(c):
    if c.get("grid") == "sml":
        return 17.0, 12.0, 3.0
    return c["nx"] * c["h"], c["ny"] * c["h"], c["nz"] * c["h"]


def _solver(c, seed):
    lx, ly, lz = _lengths(c)
    kw = dict(cg.BOUNDARY_SET) if c.get("bset") else dict(project_rhs=1)
    cx = 6.5 if c.get("grid") == "sml" else lx / 4
    return cg.Solver(nx=c["nx"], ny=c["ny"], nz=c["nz"], lx=lx, ly=ly, lz=lz, cx=cx, cy=ly / 2, radius=0.5,
                     Re=c["Re"], dt=c["dt"], solver=c["solver"], precision=c["precision"], precond=c["precond"],
                     tol=c["tol"], grid=c.get("grid", "uniform"), maxit=20000, seed=seed, amp=AMP, **kw)


def _initial(c, seed):
    """u, v, w (1, 0, 0 plus a uniform perturbation of the interior) and p = 0, padded, on the GPU."""
    shape = (c["nx"] + 4, c["ny"] + 4, c["nz"] + 4)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    f = torch.zeros((4,) + shape, dtype=torch.float64, device="cuda")
    f[0] = 1.0
    for a in range(3):
        f[a, 2:-2, 2:-2, 2:-2] += AMP * (2 * torch.rand((c["nx"], c["ny"], c["nz"]), generator=gen, device="cuda",
                                                        dtype=torch.float64) - 1)
    return f


def _inlet(c, seed):
    gen = torch.Generator().manual_seed(seed)
    return 1.0 + AMP * (2 * torch.rand((c["ny"], c["nz"]), generator=gen, dtype=torch.float64) - 1)


def _poisson_data(c, seed):
    """A consistent right-hand side (sums to zero) and a warm start, unscaled rows."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    shape = (c["nx"], c["ny"], c["nz"])
    b = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
    x0 = 0.01 * torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
    return b - b.mean(), x0


def _diag(c):
    """The diagonal of the uniform-grid Neumann operator."""
    d = torch.zeros((c["nx"], c["ny"], c["nz"]), dtype=torch.float64, device="cuda")
    for a in range(3):
        e = torch.full((d.shape[a],), 2.0, dtype=torch.float64, device="cuda")
        e[0] = e[-1] = 1.0
        d += (e / c["h"] ** 2).reshape([-1 if q == a else 1 for q in range(3)])
    return d


def prepare(c, seed):
    st = dict(case=c)
    if c["kind"] == "poisson":
        b, x0 = _poisson_data(c, seed)
        if c["solver"] == "jacobi":
            b = b / _diag(c)
        st.update(b=b.contiguous(), x0=x0, x=torch.empty_like(x0), lib=cg.load_library())
        return st
    s = st["solver"] = _solver(c, seed)
    if c["kind"] == "adjoint":
        s.set_inlet(_inlet(c, seed).numpy())
        init = torch.zeros((4,) + s.shape, dtype=torch.float64).pin_memory()
        init[0] = 1.0
        st["init"] = init.numpy()
        return st
    f = _initial(c, seed)
    init = torch.empty(f.shape, dtype=torch.float64, pin_memory=True)
    st["init"] = init.copy_(f).numpy()
    shape = f.shape if c["precision"] == "fp64" else f[:3].shape
    st["out"] = torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()
    return st


def run(st):
    c = st["case"]
    if c["kind"] == "poisson":
        x, it, rr = st["x"], C.c_int(), C.c_double()
        x.copy_(st["x0"])
        rc = st["lib"].cfdgb_poisson_solve_static(
            c["nx"], c["ny"], c["nz"], c["h"], c["h"], c["h"], cg.SOLVERS[c["solver"]], c["tol"], 5000,
            C.c_void_p(st["b"].data_ptr()), C.c_void_p(x.data_ptr()),
            C.c_void_p(torch.cuda.current_stream().cuda_stream), C.byref(it), C.byref(rr))
        if rc != 0:
            raise RuntimeError("poisson solve: status %d" % rc)
        return x
    s = st["solver"]
    if c["kind"] == "adjoint":
        s.init_fields(*st["init"])
        J = s.forward(c["steps"], c["first"], c["steps"], c["ckpt"])
        g_in, g_eta = s.backward()
        return dict(J=np.array(J), inlet=g_in, eta=g_eta)
    s.init_fields(*st["init"])
    r = s.step(c["steps"])
    out = st["out"]
    s.get_fields(dict(zip("uvwp", out)))
    got = dict(velocity=out[:3], forces=np.array([(q.cd, q.cl) for q in r]))
    return dict(got, p=out[3]) if len(out) > 3 else got


def work(c):
    """Per cell and step: the state (u, v, w, p) and the solver's warm start read and written once,
    about 330 operations of convection, diffusion, right-hand side and correction, and a Poisson
    solve of 100 operations a cell (a few multigrid cycles)."""
    n = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "poisson":
        return dict(bytes=24 * n, flops=100 * n)
    steps = c["steps"] * (3 if c["kind"] == "adjoint" else 1)  # backward: recompute and transpose
    return dict(bytes=n * (80 * steps + 64), flops=430 * n * steps)


# ---- the same in plain torch, FP64 ----------------------------------------------------------------------------------


class _Grid:
    """Metrics of the padded grid (two ghost layers) and the exact Poisson solve."""

    def __init__(self, c):
        self.n = (c["nx"], c["ny"], c["nz"])
        self.pz = bool(c.get("bset"))
        fine = [(0.3, 100, -4), (0.3, 100, 0), None] if c.get("grid") == "sml" else [None] * 3
        self.X, self.D, self.S = [], [], []
        for a, (n, l, f) in enumerate(zip(self.n, _lengths(c), fine)):
            if f is None:
                d = np.full(n, l / n)
            else:  # `cells` fine cells over part of the axis, shifted, coarse ones on both sides
                part, cells, off = f
                coarse, left = (l - part * l) / (n - cells), (n - cells) // 2 + off
                d = np.full(n, coarse)
                d[left:left + cells] = part * l / cells
            x = np.concatenate([[0.0], np.cumsum(d)])
            x = np.concatenate([[x[0] - 2 * d[0], x[0] - d[0]], x, [x[-1] + d[-1], x[-1] + 2 * d[-1]]])
            D = np.concatenate([[d[0]] * 2, d, [d[-1]] * 2])
            S = np.empty(n + 4)
            S[2:n + 1] = (d[:-1] + d[1:]) / 2  # between the centres of cells i and i + 1
            S[:2], S[n + 1:] = S[2], S[n]
            shape = [-1 if q == a else 1 for q in range(3)]
            self.X.append(x)
            self.D.append(torch.tensor(D, device="cuda").reshape(shape))
            self.S.append(torch.tensor(S, device="cuda").reshape(shape))
        self.eig = None

    def at(self, m, a, o, ext):
        """Metric array m[a] at the faces of an extent, shifted by o along its axis."""
        return m[a].narrow(a, 2 + o, ext[a])

    def solve(self, b):
        """A x = b, the component along the constant left at zero in the eigenbasis: A is a Kronecker
        sum of three tridiagonal matrices, each symmetric under the weights D."""
        if self.eig is None:
            self.eig = []
            for a, n in enumerate(self.n):
                D, S = self.D[a].flatten(), self.S[a].flatten()
                lo, hi = 1 / S[1:n + 1], 1 / S[2:n + 2]
                per = self.pz and a == 2
                if not per:
                    lo[0] = hi[-1] = 0
                w = D[2:n + 2].sqrt()
                T = torch.diag(lo + hi) - torch.diag(lo[1:], -1) - torch.diag(hi[:-1], 1)
                if per:
                    T[0, -1] -= lo[0]
                    T[-1, 0] -= hi[-1]
                lam, Q = torch.linalg.eigh(T / w[:, None] / w[None, :])
                lam[0] = 0
                self.eig.append((lam, Q / w[:, None], (Q * w[:, None]).T.contiguous()))
        (lx, vx, ix), (ly, vy, iy), (lz, vz, iz) = self.eig

        def apply(x, mx, my, mz):
            x = torch.matmul(x, mz.T)
            x = torch.matmul(my, x)
            return torch.matmul(mx, x.reshape(x.shape[0], -1)).reshape(x.shape)

        lam = lx[:, None, None] + ly[:, None] + lz
        lam[0, 0, 0] = math.inf
        return apply(apply(b, ix, iy, iz) / lam, vx, vy, vz)

    def diag(self):
        d = 0
        for a, n in enumerate(self.n):
            D, S = self.D[a].flatten(), self.S[a].flatten()
            lo, hi = 1 / (D[2:n + 2] * S[1:n + 1]), 1 / (D[2:n + 2] * S[2:n + 2])
            if not (self.pz and a == 2):
                lo[0] = hi[-1] = 0
            d = d + (lo + hi).reshape(self.D[a].shape[:a] + (-1,) + self.D[a].shape[a + 1:])
        return d

    def volume(self):
        return self.D[0][2:-2] * self.D[1][:, 2:-2] * self.D[2][:, :, 2:-2]

    def solid(self, c):
        """Solid fraction of the cylinder: 100 x 100 samples in the cells its circle can cut."""
        lx, ly, _ = _lengths(c)
        cx, cy, R = (6.5 if c.get("grid") == "sml" else lx / 4), ly / 2, 0.5
        eta = torch.zeros([m + 4 for m in self.n], dtype=torch.float64, device="cuda")
        sub = (np.arange(100) + 0.5) / 100
        X, Y = self.X[0], self.X[1]
        col = np.zeros((self.n[0], self.n[1]))
        for i in range(self.n[0]):
            a = X[i + 2] + (X[i + 3] - X[i + 2]) * sub - cx
            if abs(a).min() > R + 1:
                continue
            for j in range(self.n[1]):
                b = Y[j + 2] + (Y[j + 3] - Y[j + 2]) * sub - cy
                dx, dy = X[i + 3] - X[i + 2], Y[j + 3] - Y[j + 2]
                dist = math.hypot((X[i + 2] + X[i + 3]) / 2 - cx, (Y[j + 2] + Y[j + 3]) / 2 - cy)
                if abs(dist - R) < math.hypot(dx, dy) / 2:
                    col[i, j] = np.mean(np.hypot(a[:, None], b[None, :]) <= R)
                else:
                    col[i, j] = float(dist <= R)
        eta[2:-2, 2:-2, 0:-1] = torch.tensor(col, device="cuda")[:, :, None]
        return eta


def _shift(f, o, ext):
    return f[2 + o[0]:2 + o[0] + ext[0], 2 + o[1]:2 + o[1] + ext[1], 2 + o[2]:2 + o[2] + ext[2]]


def _unit(a, o):
    return tuple(o if q == a else 0 for q in range(3))


def _add(*os):
    return tuple(sum(q) for q in zip(*os))


def _convection_diffusion(g, U, nu, dt):
    """u*, v*, w*: explicit Euler, QUICK convection, central diffusion; other entries as U's."""
    out = []
    for A in range(3):
        ext = [n - (1 if q == A and not (g.pz and A == 2) else 0) for q, n in enumerate(g.n)]
        phi, conv, diff = U[A], 0, 0
        half = 0.5 * g.at(g.S, A, 0, ext) / g.at(g.D, A, 0, ext)
        for b in range(3):
            own = b == A
            M, N = (g.D, g.S) if own else (g.S, g.D)  # spacings between the values, between the faces' own
            s0 = 1 if own else 0

            def m(o):
                return g.at(M, b, o + s0, ext)

            def face(o):  # between the values at o and o + 1
                f = [_shift(phi, _unit(b, o + q), ext) for q in (-1, 0, 1, 2)]
                if own:
                    vel = 0.5 * (f[1] + f[2])
                else:
                    v0, v1 = _shift(U[b], _unit(b, o), ext), _shift(U[b], _add(_unit(b, o), _unit(A, 1)), ext)
                    vel = v0 + (v1 - v0) * half
                k = 0.125 * m(o) ** 2
                up = k * ((f[2] - f[1]) / m(o) - (f[1] - f[0]) / m(o - 1)) / g.at(N, b, o, ext)
                dn = k * ((f[3] - f[2]) / m(o + 1) - (f[2] - f[1]) / m(o)) / g.at(N, b, o + 1, ext)
                return 0.5 * (f[1] + f[2]) - torch.where(vel > 0, up, dn), vel

            (P, vp), (Q, vn) = face(0), face(-1)
            f = [_shift(phi, _unit(b, q), ext) for q in (-1, 0, 1)]
            d = g.at(N, b, 0, ext)
            conv = conv + ((P * P - Q * Q) if own else (P * vp - Q * vn)) / d
            diff = diff + ((f[2] - f[1]) / m(0) - (f[1] - f[0]) / m(-1)) / d
        r = phi.clone()
        _shift(r, (0, 0, 0), ext).copy_(_shift(phi, (0, 0, 0), ext) + dt * (nu * diff - conv))
        out.append(r)
    return out


def _boundary(g, c, U, p, inlet, old, dt):
    """Ghost fill, x faces then y then z; old: the state before the step (None at init)."""
    u, v, w = [f.clone() for f in U]
    p = p.clone()
    I = slice(2, -2)
    wall = 0.0 if c.get("bset") else 1.0
    u_out, v_out, w_out = u[-4, I, I], v[-3, I, I], w[-3, I, I]
    if c.get("bset"):  # convective outlet, then the uniform correction that balances the net flux
        if old is not None:
            cu, cv = dt / g.D[0].flatten()[-3], dt / g.S[0].flatten()[-3]
            u_out = (old[0][-3, I, I] + cu * u_out) / (1 + cu)
            v_out = (old[1][-2, I, I] + cv * v_out) / (1 + cv)
            w_out = (old[2][-2, I, I] + cv * w_out) / (1 + cv)
        area = (g.D[1] * g.D[2])[0, I, I]
        u_out = u_out + ((inlet - u_out) * area).sum() / area.sum()
    u[0:2, I, I] = inlet
    v[0:2, I, I], w[0:2, I, I] = -v[2:3, I, I], -w[2:3, I, I]
    u[-3:, I, I], v[-2:, I, I], w[-2:, I, I] = u_out, v_out, w_out
    p[0:2, I, I], p[-2:, I, I] = p[2:3, I, I].clone(), p[-3:-2, I, I].clone()
    for f in (u, w, p):
        f[I, 0:2, I], f[I, -2:, I] = f[I, 2:3, I].clone(), f[I, -3:-2, I].clone()
    v[I, 0:2, I], v[I, -3:, I] = wall * v[I, 2:3, I].clone(), wall * v[I, -4:-3, I].clone()
    if g.pz:
        for f in (u, v, w, p):
            f[:, :, :2], f[:, :, -2:] = f[:, :, -4:-2].clone(), f[:, :, 2:4].clone()
    else:
        for f in (u, v, p):
            f[I, I, 0:2], f[I, I, -2:] = f[I, I, 2:3].clone(), f[I, I, -3:-2].clone()
        w[I, I, 0:2], w[I, I, -3:] = w[I, I, 2:3].clone(), w[I, I, -4:-3].clone()
    return [u, v, w], p


def _simulate(c, U, p, inlet, eta, g):
    """`steps` projection steps; fields, pressure and (Cd, Cl) of each step."""
    dt, lz, first = c["dt"], _lengths(c)[2], U
    U, p = _boundary(g, c, U, p, inlet, None, dt)
    vol, I = g.volume(), slice(2, -2)
    weight = vol * g.diag() if c["solver"] == "jacobi" and c["precision"] == "fp64" else torch.ones_like(vol)
    forces = []
    for step in range(c["steps"]):
        S = _convection_diffusion(g, U, 1.0 / c["Re"], dt)
        if step > 0:
            div = 0
            for a in range(3):
                div = div + (_shift(S[a], (0, 0, 0), g.n) - _shift(S[a], _unit(a, -1), g.n)) / g.at(g.D, a, 0, g.n)
            if g.pz:  # the bottom face is the image of the top one
                div = div.clone()
                div[:, :, 0] += (S[2][I, I, 1] - S[2][I, I, -3]) / g.D[2].flatten()[2]
            b = -div / dt
            if not c.get("bset"):
                b = b - b.mean()
            x = g.solve(b)
            x = x - (weight * x).sum() / weight.sum()
            p = p.clone()
            p[I, I, I] = x
            if g.pz:
                p[I, I, -2] = x[:, :, 0]
        V, F = [], []
        for a in range(3):
            ext = [n - (1 if q == a and not (g.pz and a == 2) else 0) for q, n in enumerate(g.n)]
            o, e = (0, 0, 0), _unit(a, 1)
            t = _shift(S[a], o, ext) - dt * (_shift(p, e, ext) - _shift(p, o, ext)) / g.at(g.S, a, 0, ext)
            e0, e1 = _shift(eta, o, ext), _shift(eta, e, ext)
            if g.pz and a == 2:
                e1 = torch.cat([e1[:, :, :-1], e0[:, :, :1]], 2)
            frac = e0 + (e1 - e0) * (0.5 * g.at(g.S, a, 0, ext) / g.at(g.D, a, 0, ext))
            f = first[a].clone()  # the last face along an axis keeps its initial value until the ghost fill
            _shift(f, o, ext).copy_((1 - frac) * t)
            V.append(f)
            F.append((frac * t * vol[:ext[0], :ext[1], :ext[2]]).sum() * (2 / (lz * dt)))
        forces.append(torch.stack(F[:2]))
        U, p = _boundary(g, c, V, p, inlet, U, dt)
    return U, p, torch.stack(forces)


def exact(c, seed):
    if c["kind"] == "poisson":
        b, x0 = _poisson_data(c, seed)
        x = _Grid(c).solve(b)
        weight = _diag(c) if c["solver"] == "jacobi" else torch.ones_like(x)
        return x + (weight * (x0 - x)).sum() / weight.sum()
    g = _Grid(c)
    eta = g.solid(c)
    if c["kind"] == "adjoint":
        inlet = _inlet(c, seed).cuda().requires_grad_()
        eta.requires_grad_()
        f = torch.zeros([4] + [n + 4 for n in g.n], dtype=torch.float64, device="cuda")
        f[0] = 1.0
        J = _simulate(c, list(f[:3]), f[3], inlet, eta, g)[2][c["first"] - 1:, 0].mean()
        J.backward()
        return dict(J=J.detach().cpu().numpy(), inlet=inlet.grad.cpu().numpy(), eta=eta.grad.cpu().numpy())
    f = _initial(c, seed)
    with torch.no_grad():
        U, p, forces = _simulate(c, list(f[:3]), f[3], torch.ones((), dtype=torch.float64, device="cuda"), eta, g)
    got = dict(velocity=torch.stack(U).cpu().numpy(), forces=forces.cpu().numpy())
    if c["precision"] == "fp64":  # the constant a V-cycle leaves in the pressure is the iteration's own
        got["p"] = None if c["precond"] == "multigrid" else p.cpu().numpy()
    return got

"""The work that users of this framework have it do, as measurable cases.

Every case goes through a public entry point (``FDMOperator.solve`` /
``solve_device``, ``PararealOperator.run``, the learned coarse propagator,
``ResidualCNN``) with the plan, operator or model that a program keeps
between its calls.  ``exact`` restates each computation in plain torch in 64
bits.  Problems, sizes and step sizes are those of the repository's own
benchmark and test problems.
"""

from __future__ import annotations

import math
import warnings

import numpy as np
import torch

import pararealml_gb300 as ns
from pararealml_gb300.learned import HC, LAYERS, LAYOUT, CNNCoarseOperator, ResidualCNN, init_params
from pararealml_gb300.operators import fdm
from pararealml_gb300.operators.parareal import PararealOperator

CH_D, CH_GAMMA = 0.1, 0.01
SW = {"h": 1.0, "b": 0.01, "v": 0.1, "f": 0.0, "g": 9.81}
WAVE_C = 0.7
NS_RE = 5000.0


def listed():
    return [
        # the reference's own small example: every one of 800 forward Euler
        # steps of a 65^2 mesh kept; one step is a few microseconds
        dict(name="diffusion_65_fe_f64", kind="diffusion_solve", n=64, steps=800),
        # a batch of initial states advanced to their end (serial fine solves
        # of the batched Parareal workload), single and double precision
        dict(name="diffusion_257x64_rk4_f32", kind="explicit", eq="diffusion", n=256, batch=64, steps=100,
             integrator="RK4", dtype="float32", keep="final"),
        dict(name="diffusion_257x16_rk4_f64", kind="explicit", eq="diffusion", n=256, batch=16, steps=100,
             integrator="RK4", dtype="float64", keep="final"),
        # the headline: large Cahn-Hilliard, every step kept, in the
        # reference's precision and in the bandwidth-oriented one
        dict(name="cahn_hilliard_1025_f64", kind="explicit", eq="cahn_hilliard", n=1024, batch=1, steps=100,
             integrator="RK4", dtype="float64", keep="full"),
        dict(name="cahn_hilliard_1025_f32", kind="explicit", eq="cahn_hilliard", n=1024, batch=1, steps=200,
             integrator="RK4", dtype="float32", keep="full"),
        # the largest mesh of the shallow-water ensemble: a four-stage step of
        # three coupled components
        dict(name="shallow_water_513x16_f32", kind="explicit", eq="shallow_water", n=512, batch=16, steps=32,
             integrator="RK4", dtype="float32", keep="final"),
        # a 3D mesh, double precision
        dict(name="diffusion3d_97_rk4_f64", kind="explicit3d", eq="diffusion", n=96, batch=1, steps=20,
             integrator="RK4", dtype="float64", keep="final"),
        # parallel in time: 32 slices, RK4 fine and forward Euler coarse
        # operator, two iterations
        dict(name="parareal_257_s32_f64", kind="parareal", n=256, slices=32, fine_per_slice=50, iterations=2),
        # implicit steps: each an element-wise secant solve
        dict(name="backward_euler_257_f64", kind="implicit", n=256, steps=3, method="BackwardEulerMethod"),
        # the reference's Navier-Stokes example: a Jacobi solve after each step
        dict(name="navier_stokes_101x81_f64", kind="navier_stokes", nx=100, ny=80, steps=2),
        # a training step of the learned coarse operator, forward and backward
        dict(name="cnn_train_257x16", kind="cnn_train", n=256, batch=16),
        # the learned coarse operator applied eight times in a row
        dict(name="cnn_coarse_257", kind="cnn_coarse", n=256, batch=1, steps=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["diffusion_solve", "diffusion", "diffusion", "cahn_hilliard", "cahn_hilliard",
                       "shallow_water", "shallow_water", "explicit3d", "parareal", "implicit", "navier_stokes",
                       "cnn_train", "cnn_coarse"])
    if kind == "diffusion_solve":
        return dict(kind=kind, n=_log_int(rng, 16, 160), steps=_log_int(rng, 100, 800))
    if kind == "diffusion":
        n = _log_int(rng, 32, 384)
        return dict(kind="explicit", eq=kind, n=n, batch=max(1, min(96, int(rng.uniform(0.05, 1.0) * 4e6 / (n * n)))),
                    steps=_log_int(rng, 20, 100), integrator=rng.choice(["RK4", "RK4", "ForwardEulerMethod"]),
                    dtype=rng.choice(["float32", "float64"]), keep="final")
    if kind == "cahn_hilliard":
        n = _log_int(rng, 64, 1024)
        return dict(kind="explicit", eq=kind, n=n, batch=rng.choice([1, 1, 2, 5]) if n < 500 else 1,
                    steps=_log_int(rng, 20, 100), integrator=rng.choice(["RK4", "ForwardEulerMethod"]),
                    dtype=rng.choice(["float32", "float64"]), keep=rng.choice(["full", "final"]))
    if kind == "shallow_water":
        n = _log_int(rng, 40, 512)
        return dict(kind="explicit", eq=kind, n=n, batch=max(1, min(64, int(rng.uniform(0.05, 1.0) * 4e6 / (n * n)))),
                    steps=_log_int(rng, 8, 32), integrator="RK4", dtype=rng.choice(["float32", "float32", "float64"])
                    if n < 200 else "float32", keep="final")
    if kind == "explicit3d":
        return dict(kind=kind, eq=rng.choice(["diffusion", "wave"]), n=_log_int(rng, 12, 96), batch=1,
                    steps=_log_int(rng, 4, 20), integrator=rng.choice(["RK4", "ForwardEulerMethod"]),
                    dtype=rng.choice(["float32", "float64"]), keep="final")
    if kind == "parareal":
        return dict(kind=kind, n=_log_int(rng, 48, 256), slices=rng.choice([8, 16, 32]),
                    fine_per_slice=rng.choice([20, 50]), iterations=rng.choice([1, 2, 3]))
    if kind == "implicit":
        return dict(kind=kind, n=_log_int(rng, 24, 256), steps=rng.choice([1, 2, 3]),
                    method=rng.choice(["BackwardEulerMethod", "CrankNicolsonMethod"]))
    if kind == "navier_stokes":
        return dict(kind=kind, nx=rng.randint(24, 90), ny=rng.randint(24, 90), steps=1)
    n = _log_int(rng, 40, 256)
    if kind == "cnn_train":
        return dict(kind=kind, n=n, batch=max(1, int(rng.uniform(0.1, 1.0) * 1e6 / (n * n))))
    return dict(kind=kind, n=n, batch=rng.choice([1, 1, 3]), steps=rng.choice([2, 5, 8]))


# --------------------------------------------------------------------------
# problems


def _geometry(c):
    """(mesh extents, cells, steps) of a case's mesh."""
    k = c["kind"]
    if k == "explicit" and c["eq"] == "shallow_water":
        return [64.0] * 2, [c["n"]] * 2
    if k in ("parareal", "cnn_train", "cnn_coarse"):
        return [0.25 * c["n"]] * 2, [c["n"]] * 2
    if k == "explicit" and c["eq"] == "cahn_hilliard":
        return [0.0625 * c["n"]] * 2, [c["n"]] * 2
    if k == "explicit3d":
        return [4.0] * 3, [c["n"]] * 3
    if k == "navier_stokes":
        return [0.05 * c["nx"], 0.05 * c["ny"]], [c["nx"], c["ny"]]
    return [10.0] * 2, [c["n"]] * 2


def _d_x(c):
    length, n = _geometry(c)
    return [length[a] / n[a] for a in range(len(n))]


def _d_t(c):
    dx = _d_x(c)[0]
    k = c["kind"]
    if k == "implicit":
        return 1e-3
    if k == "navier_stokes":
        return 0.05
    if k == "parareal":
        return 1e-3
    eq = "diffusion" if k == "diffusion_solve" else c["eq"]
    if eq == "cahn_hilliard":
        return 1e-4
    if eq == "shallow_water":
        return 0.4 * dx / math.sqrt(SW["g"] * SW["h"])
    if eq == "wave":
        return 0.2 * dx
    return 0.06 * dx * dx


def _cp(c):
    length, n = _geometry(c)
    mesh = ns.Mesh([(0.0, x) for x in length], _d_x(c))
    k = c["kind"]
    dims = len(n)
    eq = c.get("eq", {"diffusion_solve": "diffusion", "implicit": "diffusion", "navier_stokes": "navier_stokes"}.get(
        k, "cahn_hilliard"))
    if eq == "cahn_hilliard":
        de = ns.CahnHilliardEquation(2, CH_D, CH_GAMMA)
        bc = ns.NeumannBoundaryCondition(lambda x, t: np.zeros((len(x), 2)), is_static=True)
    elif eq == "shallow_water":
        de = ns.ShallowWaterEquation(SW["h"], SW["b"], SW["v"], SW["f"], SW["g"])
        bc = ns.NeumannBoundaryCondition(ns.vectorize_bc_function(lambda x, t: (0.0, None, None)), is_static=True)
    elif eq == "wave":
        de = ns.WaveEquation(dims, WAVE_C)
        bc = ns.NeumannBoundaryCondition(lambda x, t: np.zeros((len(x), 2)), is_static=True)
    elif eq == "navier_stokes":
        de = ns.NavierStokesEquation(NS_RE)

        def face(w, psi):
            return ns.DirichletBoundaryCondition(ns.vectorize_bc_function(lambda x, t: (w, psi, None, None)), is_static=True)

        return ns.ConstrainedProblem(de, mesh, [(face(1.0, 0.1), face(0.0, 0.0)), (face(0.0, 0.0), face(0.0, 0.0))])
    else:
        de = ns.DiffusionEquation(dims, 1.0)
        bc = ns.DirichletBoundaryCondition(lambda x, t: np.zeros((len(x), 1)), is_static=True)
    return ns.ConstrainedProblem(de, mesh, [(bc, bc)] * dims)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (2 ** 31) + 17)


def _uniform(g, shape, lo, hi):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _bumps(c, batch, seed, lo, hi, var_lo, var_hi, peak_lo, peak_hi):
    """Gaussian bumps (batch, *vertices) of random centre, variance and peak."""
    length, n = _geometry(c)
    g = _gen(seed)
    out = _uniform(g, (batch,) + (1,) * len(n), peak_lo, peak_hi).expand((batch,) + tuple(k + 1 for k in n)).clone()
    var = _uniform(g, (batch,) + (1,) * len(n), var_lo, var_hi)
    for a in range(len(n)):
        centre = _uniform(g, (batch,) + (1,) * len(n), lo * length[a], hi * length[a])
        x = torch.linspace(0.0, length[a], n[a] + 1, dtype=torch.float64, device="cuda")
        x = x.reshape((1,) * (1 + a) + (-1,) + (1,) * (len(n) - 1 - a))
        out = out * torch.exp(-0.5 * (x - centre) ** 2 / var)
    return out


def _zero_faces(y):
    """y (batch, *vertices) with zero on every face, in place."""
    for a in range(1, y.dim()):
        y.select(a, 0).zero_()
        y.select(a, y.shape[a] - 1).zero_()
    return y


def _initial(c, seed):
    """Initial states (batch, *vertices, components) in float64 on the GPU."""
    k, batch = c["kind"], c.get("batch", 1)
    eq = c.get("eq", "cahn_hilliard" if k in ("parareal", "cnn_train", "cnn_coarse") else "diffusion")
    if k == "navier_stokes":
        w = _bumps(c, 1, seed, 0.3, 0.7, 0.1, 0.4, 0.5, 1.5)
        y = torch.zeros(w.shape + (4,), dtype=torch.float64, device="cuda")
        y[..., 0] = w
        for comp, value in ((0, 1.0), (1, 0.1)):
            y[:, 0, :, comp] = value
            y[:, -1, :, comp] = 0.0
            y[:, :, 0, comp] = 0.0
            y[:, :, -1, comp] = 0.0
        return y
    if eq == "cahn_hilliard":
        shape = (batch,) + tuple(n + 1 for n in _geometry(c)[1])
        conc = _uniform(_gen(seed), shape, -0.1, 0.1)
        mu = conc ** 3 - conc - CH_GAMMA * _lap(conc, _d_x(c), True)
        return torch.stack([conc, mu], dim=-1)
    if eq == "shallow_water":
        h = _bumps(c, batch, seed, 0.125, 0.875, 1.0, 6.0, 0.05, 0.2)
        return torch.stack([h, torch.zeros_like(h), torch.zeros_like(h)], dim=-1)
    y = _bumps(c, batch, seed, 0.2, 0.8, 0.3, 1.0, 0.5, 1.5)
    if eq == "wave":
        return torch.stack([y, torch.zeros_like(y)], dim=-1)
    return _zero_faces(y)[..., None]


def _operator(c, dtype, **kw):
    name = c.get("integrator") or c.get("method") or "RK4"
    return fdm.FDMOperator(getattr(fdm, name)(), fdm.ThreePointCentralDifferenceMethod(), _d_t(c), dtype=dtype, **kw)


def _planar(y, pitch, dtype):
    """(batch, *vertices, C) -> the device layout (batch, C, nx, pitch)."""
    b, nx, ny, comps = y.shape
    out = torch.zeros((b, comps, nx, pitch), dtype=dtype, device="cuda")
    out[..., :ny] = y.permute(0, 3, 1, 2)
    return out


def _cnn(c, seed):
    model = ResidualCNN(init_params(int(seed) % 100003))
    model.set_scales([15.0, 3.0], [0.01, 0.02])
    return model


# --------------------------------------------------------------------------


def prepare(case, seed):
    c = case
    k = c["kind"]
    if k in ("cnn_train", "cnn_coarse"):
        nv = c["n"] + 1
        pitch = -(-nv // 32) * 32
        u = _planar(_initial(c, seed), pitch, torch.float32)
        model = _cnn(c, seed)
        if k == "cnn_train":
            noise = torch.randn(u.shape, generator=_gen(seed + 1), device="cuda", dtype=torch.float32)
            return {"case": c, "model": model, "u": u, "target": u + 0.01 * noise, "y": torch.zeros_like(u)}
        cp = _cp(c)
        base = fdm.FDMOperator(fdm.ForwardEulerMethod(), fdm.ThreePointCentralDifferenceMethod(), 0.0125, dtype="float32")
        op = CNNCoarseOperator(0.05, model, base=base, dtype="float32")
        return {"case": c, "cp": cp, "op": op, "propagate": op.coarse_propagator(cp, c["batch"], c["steps"]), "u": u,
                "out": torch.zeros_like(u)}
    cp = _cp(c)
    y0 = _initial(c, seed)
    if k == "parareal":
        fine = fdm.FDMOperator(fdm.RK4(), fdm.ThreePointCentralDifferenceMethod(), _d_t(c))
        coarse = fdm.FDMOperator(fdm.ForwardEulerMethod(), fdm.ThreePointCentralDifferenceMethod(),
                                 _d_t(c) * c["fine_per_slice"] / _coarse_steps(c))
        op = PararealOperator(fine, coarse, 0.0, c["iterations"], n_slices=c["slices"], trajectory="final")
        return {"case": c, "cp": cp, "op": op, "y0": y0, "t": (0.0, _d_t(c) * c["fine_per_slice"] * c["slices"])}
    if k == "explicit" or k == "explicit3d":
        op = _operator(c, c["dtype"], trajectory=c["keep"])
        op.plan(cp, c["batch"])
        return {"case": c, "cp": cp, "op": op, "y0": y0}
    ic = ns.DiscreteInitialCondition(cp, y0[0].cpu().numpy(), True)
    ivp = ns.InitialValueProblem(cp, (0.0, c["steps"] * _d_t(c)), ic)
    op = _operator(dict(c, integrator="ForwardEulerMethod") if k == "diffusion_solve" else c, "float64",
                   keep_on_device=k == "diffusion_solve")
    op.plan(cp, 1)
    return {"case": c, "op": op, "ivp": ivp, "seed": int(seed) % (2 ** 31)}


def _coarse_steps(c):
    return -(-c["fine_per_slice"] // 20)  # forward Euler is stable up to steps of about 0.02


def run(state):
    c = state["case"]
    k = c["kind"]
    if k in ("explicit", "explicit3d"):
        traj = state["op"].solve_device(state["cp"], state["y0"], 0.0, c["steps"])
        return traj[..., :c["n"] + 1]  # the row padding holds nothing
    if k == "diffusion_solve":
        return state["op"].solve(state["ivp"]).device_y
    if k == "implicit":
        with warnings.catch_warnings():
            warnings.simplefilter("ignore", RuntimeWarning)  # slow secant convergence is reported as one
            return state["op"].solve(state["ivp"]).discrete_y()
    if k == "navier_stokes":
        np.random.seed(state["seed"])  # the Jacobi solves start from numpy's generator
        return state["op"].solve(state["ivp"]).discrete_y()
    if k == "parareal":
        return state["op"].run(state["cp"], state["y0"], state["t"])["final"]
    n = c["n"] + 1
    if k == "cnn_coarse":
        state["propagate"](state["u"], state["out"], 0.0)
        return state["out"][..., :n]
    model = state["model"]
    model.forward(state["u"], state["y"], n, n)
    model.loss_and_dy(state["y"], state["target"], n, n)
    model.backward(state["u"], n, n)
    return [state["y"][..., :n], model.grads]


def work(case):
    c = case
    k = c["kind"]
    length, n = _geometry(c)
    v = math.prod(x + 1 for x in n)
    if k == "cnn_train":
        v *= c["batch"]
        flops = 2 * 9 * (2 * HC + 4 * HC * HC + HC * 2) * v
        return {"bytes": 3 * 2 * 4 * v + 2 * 4 * sum(math.prod(s) for _, _, _, s in LAYOUT), "flops": 3 * flops}
    if k == "cnn_coarse":
        v *= c["batch"]
        flops = 2 * 9 * (2 * HC + 4 * HC * HC + HC * 2) * v * c["steps"]
        return {"bytes": 2 * 2 * 4 * v, "flops": flops}
    if k == "parareal":
        steps = c["iterations"] * c["slices"] * (c["fine_per_slice"] + _coarse_steps(c))
        return {"bytes": 2 * 2 * 8 * v, "flops": 20 * v * steps}
    if k == "implicit":
        return {"bytes": 8 * v * (1 + c["steps"]), "flops": 25 * 25 * v * c["steps"]}
    if k == "navier_stokes":
        return {"bytes": 4 * 8 * v * (1 + c["steps"]), "flops": v * c["steps"] * (4 * 20 + 8 * 40 * min(c["nx"], c["ny"]))}
    eq = "diffusion" if k == "diffusion_solve" else c["eq"]
    comps = {"diffusion": 1, "wave": 2, "cahn_hilliard": 2, "shallow_water": 3}[eq]
    flops = {"diffusion": 7, "wave": 7, "cahn_hilliard": 20, "shallow_water": 60}[eq] + (3 if k == "explicit3d" else 0)
    stages = 4 if c.get("integrator", "ForwardEulerMethod") == "RK4" and eq != "cahn_hilliard" else 1
    size = 8 if c.get("dtype", "float64") == "float64" else 4
    saved = 1 if c.get("keep") == "final" else c["steps"]
    batch = c.get("batch", 1)
    return {"bytes": batch * comps * v * (8 + size * saved), "flops": batch * v * c["steps"] * stages * (flops + 4 * comps)}


# --------------------------------------------------------------------------
# the same in plain torch, 64 bits


def _ends(y, a, neumann):
    """Previous and next values along axis a: zero outside the mesh, or the
    mirrored value on a zero-flux face."""
    prev, nxt = torch.zeros_like(y), torch.zeros_like(y)
    n = y.shape[a]
    prev.narrow(a, 1, n - 1).copy_(y.narrow(a, 0, n - 1))
    nxt.narrow(a, 0, n - 1).copy_(y.narrow(a, 1, n - 1))
    if neumann:
        prev.select(a, 0).copy_(y.select(a, 1))
        nxt.select(a, n - 1).copy_(y.select(a, n - 2))
    return prev, nxt


def _lap(y, d_x, neumann):
    """Laplacian of y (batch, *vertices)."""
    out = 0.0
    for a, h in enumerate(d_x):
        prev, nxt = _ends(y, a + 1, neumann)
        out = out + ((nxt - 2.0 * y) + prev) / (h * h)
    return out


def _grad(y, a, h, neumann):
    prev, nxt = _ends(y, a + 1, neumann)
    return (nxt - prev) / (2.0 * h)


def _rk4(y, f, dt, fix=lambda y: y):
    k1 = f(y)
    k2 = f(fix(y + 0.5 * dt * k1))
    k3 = f(fix(y + 0.5 * dt * k2))
    k4 = f(fix(y + dt * k3))
    return fix(y + dt / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4))


def _stepper(eq, d_x, dt, rk4):
    """One explicit step of a state (components, batch, *vertices)."""
    if eq == "cahn_hilliard":  # dc/dt reads mu alone, which no stage changes

        def step(y):
            c, mu = y[0], y[1]
            return torch.stack([c + dt * CH_D * _lap(mu, d_x, True), c ** 3 - c - CH_GAMMA * _lap(c, d_x, True)])

        return step
    if eq == "shallow_water":

        def f(y):
            h, u, v = y
            hx, hy = _grad(h, 0, d_x[0], True), _grad(h, 1, d_x[1], True)
            ux, uy = _grad(u, 0, d_x[0], False), _grad(u, 1, d_x[1], False)
            vx, vy = _grad(v, 0, d_x[0], False), _grad(v, 1, d_x[1], False)
            return torch.stack([
                -SW["h"] * (ux + vy) - h * ux - u * hx - h * vy - v * hy,
                SW["v"] * _lap(u, d_x, False) - u * ux - v * uy - SW["g"] * hx - SW["b"] * u + SW["f"] * v,
                SW["v"] * _lap(v, d_x, False) - u * vx - v * vy - SW["g"] * hy - SW["b"] * v - SW["f"] * u])

        fix = lambda y: y  # noqa: E731
    elif eq == "wave":

        def f(y):
            return torch.stack([y[1], WAVE_C ** 2 * _lap(y[0], d_x, True)])

        # zero-flux faces constrain both components' derivatives only
        fix = lambda y: y  # noqa: E731
    else:

        def f(y):
            return _lap(y[0], d_x, False)[None]

        fix = lambda y: _zero_faces(y[0].clone())[None]  # noqa: E731
    if rk4:
        return lambda y: _rk4(y, f, dt, fix)
    return lambda y: fix(y + dt * f(y))


def _secant(y, f, dt, fix, a, tol=1.48e-8, limit=50):
    """The element-wise secant solve of one implicit step."""
    dx = float(np.finfo(float).eps ** 0.33)
    f0 = f(y)
    p = fix(y + dt * f0)
    p1 = p * (1.0 + dx) + torch.where(p >= 0, dx, -dx)
    forward = (1.0 - a) * dt * f0 if a != 1.0 else 0.0
    residual = lambda x: x - fix(y + a * dt * f(x) + forward)  # noqa: E731
    q0, q1 = residual(p), residual(p1)
    active = torch.ones_like(p, dtype=torch.bool)
    for _ in range(limit):
        nz = q1 != q0
        if not bool(nz.any()):
            return (p1 + p) / 2.0
        d = torch.where(nz, q1 * (p1 - p) / torch.where(nz, q1 - q0, torch.ones_like(q0)), torch.zeros_like(q0))
        new = torch.where(nz, p1 - d, p)
        new = torch.where(~nz & active, (p1 + p) / 2.0, new)
        active = active & nz
        p, p1 = p1, new
        if not bool((nz & (d.abs() >= tol)).any()):
            return p1
        q0, q1 = q1, residual(p1)
    return p


def _jacobi(lap, start, d_x, fix, tol=1e-3):
    """Jacobi iterations of a Poisson problem until the change is small."""
    y = fix(start)
    inv = [1.0 / (h * h) for h in d_x]
    scale = 1.0 / sum(2.0 * i for i in inv)
    while True:
        acc = 0.0
        for a, i in enumerate(inv):
            prev, nxt = _ends(y, a + 1, False)
            acc = acc + (prev + nxt) * i
        new = fix((acc - lap) * scale)
        done = not float(torch.linalg.vector_norm(new - y)) > tol
        y = new
        if done:
            return y


def _lid_faces(y, lower):
    y = y.clone()
    y[:, 0, :] = lower
    y[:, -1, :] = 0.0
    y[:, :, 0] = 0.0
    y[:, :, -1] = 0.0
    return y


def _net(params, s_in, s_out, u, base):
    """The network's 64-bit forward pass on u (batch, 2, H, W)."""
    def conv(x, l):
        w = params[f"w{l}"]  # [9][ci][co]
        return torch.nn.functional.conv2d(x, w.reshape(3, 3, w.shape[1], w.shape[2]).permute(3, 2, 0, 1),
                                          params[f"b{l}"], padding=1)

    x = u * s_in[None, :, None, None]
    for l in range(LAYERS - 1):
        x = torch.relu(conv(x, l))
    return base + s_out[None, :, None, None] * conv(x, LAYERS - 1)


def exact(case, seed):
    c = case
    k = c["kind"]
    dt, d_x = (_d_t(c) if k not in ("cnn_train", "cnn_coarse") else 0.0125), _d_x(c)
    y0 = _initial(c, seed)
    if k in ("cnn_train", "cnn_coarse"):
        # the inputs as they are stored (float32), the arithmetic in 64 bits
        u = y0.float().double().permute(0, 3, 1, 2)
        params = {key: torch.from_numpy(np.asarray(v, dtype=np.float32).astype(np.float64)).cuda().requires_grad_(k == "cnn_train")
                  for key, v in init_params(int(seed) % 100003).items()}
        s_in = torch.tensor([15.0, 3.0], device="cuda").double()
        s_out = torch.tensor([0.01, 0.02], device="cuda").double()
        if k == "cnn_coarse":
            step = _stepper("cahn_hilliard", d_x, dt, False)
            for _ in range(c["steps"]):
                b = u.permute(1, 0, 2, 3)
                for _ in range(4):
                    b = step(b)
                u = _net(params, s_in, s_out, u, b.permute(1, 0, 2, 3))
            return u
        grads = {key: torch.zeros_like(v) for key, v in params.items()}
        n = c["n"] + 1
        pitch = -(-n // 32) * 32
        noise = torch.randn(tuple(u.shape[:3]) + (pitch,), generator=_gen(seed + 1), device="cuda", dtype=torch.float32)
        target = (u.float() + 0.01 * noise[..., :n]).double()
        out = torch.empty_like(u)
        for b in range(u.shape[0]):  # one state at a time: the graph of all would be large
            y = _net(params, s_in, s_out, u[b:b + 1], u[b:b + 1])
            loss = ((y - target[b:b + 1]) ** 2).sum() / u.numel()
            for key, g in zip(params, torch.autograd.grad(loss, list(params.values()))):
                grads[key] += g
            out[b] = y.detach()[0]
        flat = torch.cat([grads[f"{kind}{l}"].reshape(-1) for kind, l, _, _ in LAYOUT])
        return [out, flat]
    if k in ("explicit", "explicit3d", "diffusion_solve"):
        eq = c.get("eq", "diffusion")
        step = _stepper(eq, d_x, dt, c.get("integrator") == "RK4")
        y = y0.movedim(-1, 0)
        full = k == "diffusion_solve" or c["keep"] == "full"
        # kept in the result's own layout: planar device states, or vertices last
        kept = []
        for _ in range(c["steps"]):
            y = step(y)
            if full:
                kept.append(y)
        if not full:
            kept = [y]
        out = torch.stack(kept)  # (saved, C, batch, *vertices)
        if k == "diffusion_solve":
            return out[:, 0, 0, ..., None]
        out = out.transpose(1, 2)  # (saved, batch, C, *vertices)
        if k == "explicit3d":
            return out.reshape(tuple(out.shape[:3]) + (-1, out.shape[-1]))  # planes stacked as rows
        return out
    if k == "parareal":
        fine = _stepper("cahn_hilliard", d_x, dt, True)
        n_g = _coarse_steps(c)
        coarse_step = _stepper("cahn_hilliard", d_x, dt * c["fine_per_slice"] / n_g, False)
        s = c["slices"]

        def coarse(y):
            for _ in range(n_g):
                y = coarse_step(y)
            return y

        u = [y0.movedim(-1, 0)]
        g_old = []
        for j in range(s):
            g_old.append(coarse(u[j]))
            u.append(g_old[j])
        for i in range(min(s, c["iterations"])):
            f = torch.cat(u[i:s], dim=1)  # the open slices at once
            for _ in range(c["fine_per_slice"]):
                f = fine(f)
            corr = {i + m: f[:, m:m + 1] - g_old[i + m] for m in range(s - i)}
            u[i + 1] = g_old[i] + corr[i]
            for j in range(i + 1, s):
                g_old[j] = coarse(u[j])
                u[j + 1] = g_old[j] + corr[j]
        return u[s].movedim(0, -1)
    if k == "implicit":
        f = lambda y: _lap(y, d_x, False)  # noqa: E731
        fix = lambda y: _zero_faces(y.clone())  # noqa: E731
        y, out = y0[..., 0], []
        for _ in range(c["steps"]):
            y = _secant(y, f, dt, fix, 1.0 if c["method"] == "BackwardEulerMethod" else 0.5)
            out.append(y[0, ..., None])
        return torch.stack(out)
    # navier_stokes
    state = np.random.RandomState(int(seed) % (2 ** 31))
    w, psi, u, v = y0.movedim(-1, 0)
    out = []
    for _ in range(c["steps"]):
        def f(y):
            return (_lap(y, d_x, False) / NS_RE - u * _grad(y, 0, d_x[0], False) - v * _grad(y, 1, d_x[1], False))

        start = torch.from_numpy(state.random_sample(tuple(psi.shape[1:]) + (1,)))[..., 0].cuda()[None]
        new = (_rk4(w, f, dt, lambda y: _lid_faces(y, 1.0)),
               _jacobi(-w, start, d_x, lambda y: _lid_faces(y, 0.1)),
               _grad(psi, 1, d_x[1], False), -_grad(psi, 0, d_x[0], False))
        w, psi, u, v = new
        out.append(torch.stack([x[0] for x in new], dim=-1))
    return torch.stack(out)

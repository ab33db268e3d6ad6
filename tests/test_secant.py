"""The fused secant iteration of the implicit integrators (``prml_secant_solve``
and the generated secant kernels) and the constant-divisor division they use.

CPU: ``quot`` (csrc/fdm_step.cuh), restated in exact rational arithmetic with
one rounding per operation, equals the correctly rounded quotient.  GPU: mesh
sizes around the kernel's tiles, batches, an instance whose residuals never
change (every element to the midpoint) and the iteration limit, against the
oracle at the bar of the implicit tests (1e-12, equal iteration counts)."""

import math
import random
import warnings
from fractions import Fraction

import numpy as np
import pytest

import pararealml_gb300 as ns
import problems
from golden_cases import rel_l2
from oracle import fdm as orc
from pararealml_gb300.operators import fdm

REL_F64 = 1e-12


def _quot(x, d, y):
    fma = lambda a, b, c: float(Fraction(a) * Fraction(b) + Fraction(c))  # noqa: E731
    q = x * y
    q = fma(fma(-q, d, x), y, q)
    return fma(fma(-q, d, x), y, q)


def test_constant_division_is_correctly_rounded():
    rng = random.Random(7)
    for _ in range(20000):
        d = rng.uniform(1.0, 2.0) * 2.0 ** rng.randint(-30, 30)
        x = rng.uniform(1.0, 2.0) * 2.0 ** rng.randint(-200, 200) * rng.choice((-1.0, 1.0))
        assert _quot(x, d, 1.0 / d) == x / d
    for _ in range(20000):  # quotients close to the midpoint of two floats
        d = rng.uniform(1.0, 2.0)
        m = rng.uniform(1.0, 2.0)
        x = float(Fraction(d) * (Fraction(m) + Fraction(math.ulp(m)) / 2))
        for k in (x, math.nextafter(x, 9.0), math.nextafter(x, 0.0)):
            assert _quot(k, d, 1.0 / d) == k / d


def _oracle(cp, y0, kind, d_t, steps, **kw):
    st = orc.FDMStepper(cp, kind, d_t, **kw)
    y, out = np.array(y0), []
    for i in range(steps):
        y = st.step(i * d_t, y)
        out.append(y)
    return np.stack(out), st.secant_iterations


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(3, 3), (8, 32), (9, 33), (7, 65), (40, 31)])
@pytest.mark.parametrize("kind", ["be", "cn"])
def test_tiles_and_batches(nx, ny, kind):
    import torch

    bc = ns.DirichletBoundaryCondition(lambda x, t: 0.1 * x[:, :1], is_static=True)
    free = ns.NeumannBoundaryCondition(lambda x, t: np.full((len(x), 1), 0.05), is_static=True)
    mesh = ns.Mesh([(0.0, 1.0), (0.0, 1.3)], [1.0 / (nx - 1), 1.3 / (ny - 1)])
    cp = ns.ConstrainedProblem(ns.DiffusionEquation(2, 0.3), mesh, [(bc, free), (free, bc)])
    rng = np.random.default_rng(nx * ny)
    y0 = np.stack([ns.DiscreteInitialCondition(cp, s * rng.random((nx, ny, 1)), True).discrete_y_0(True)
                   for s in (1.0, 0.05, 4.0)])
    d_t = 0.4 / (0.3 * ((nx - 1) ** 2 + ((ny - 1) / 1.3) ** 2))
    integ = fdm.BackwardEulerMethod() if kind == "be" else fdm.CrankNicolsonMethod(0.6)
    op = fdm.FDMOperator(integ, fdm.ThreePointCentralDifferenceMethod(), d_t)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        traj = op.solve_device(cp, torch.tensor(y0, device="cuda"), 0.0, 2)
        plan = op.plan(cp, 3)
        got = plan.unpack(traj, 6).cpu().numpy().reshape(2, 3, nx, ny, 1)
        for b in range(3):
            want, its = _oracle(cp, y0[b], kind, d_t, 2, **({} if kind == "be" else {"cn_a": 0.6}))
            assert [i[b] for i in plan.secant_iterations] == its
            assert rel_l2(got[:, b], want) < REL_F64


@pytest.mark.gpu
@pytest.mark.parametrize("y0", [3.0, 0.0])
def test_residuals_that_never_change_go_to_the_midpoint(y0):
    """dy/dt = 2 y at d_t = 0.5: the residual x - (y + x) is -y for every x."""
    cp = ns.ConstrainedProblem(ns.PopulationGrowthEquation(2.0))
    ivp = ns.InitialValueProblem(cp, (0.0, 0.5), ns.ConstantInitialCondition(cp, [y0]))
    op = fdm.FDMOperator(fdm.BackwardEulerMethod(), fdm.ThreePointCentralDifferenceMethod(), 0.5)

    def outcome(run):
        with warnings.catch_warnings(record=True) as w:
            warnings.simplefilter("always")
            y = run()
        return y, [str(x.message) for x in w if issubclass(x.category, RuntimeWarning)]

    got, got_w = outcome(lambda: op.solve(ivp).discrete_y())
    want, want_w = outcome(lambda: _oracle(cp, [y0], "be", 0.5, 1)[0])
    assert np.array_equal(got, want) and got_w == want_w


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [1, 2, 9, 17])
def test_iteration_limit_returns_the_previous_iterate(limit):
    ivp = problems.diffusion_2d(ns, n=20, t_end=0.04)
    cp = ivp.constrained_problem
    op = fdm.FDMOperator(fdm.BackwardEulerMethod(1e-13, limit), fdm.ThreePointCentralDifferenceMethod(), 0.02)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        try:
            want, _ = _oracle(cp, ivp.initial_condition.discrete_y_0(True), "be", 0.02, 2, secant_tol=1e-13,
                              secant_maxiter=limit)
        except RuntimeError as e:
            with pytest.raises(RuntimeError, match="all failed to converge"):
                op.solve(ivp)
            assert "all failed to converge" in str(e)
            return
        assert rel_l2(op.solve(ivp).discrete_y(), want) < REL_F64

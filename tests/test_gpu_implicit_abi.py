"""An implicit step driven from outside with the element-wise functions of the C
ABI (``prml_implicit_predict / residual / update / stop / finish`` around
``prml_fdm_rhs``), as the header documents the loop, against the package's own
step (one launch per secant iteration): the same iteration counts and, with
the same operations in the same order, the same bits."""

import ctypes
import warnings

import numpy as np
import pytest

import pararealml_gb300 as ns
from pararealml_gb300 import _native
from pararealml_gb300.operators import fdm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["be", "cn"])
@pytest.mark.parametrize("limit", [50, 7])
def test_documented_loop_equals_the_package_step(kind, limit):
    import torch

    bc = ns.DirichletBoundaryCondition(lambda x, t: 0.1 * x[:, :1], is_static=True)
    free = ns.NeumannBoundaryCondition(lambda x, t: np.full((len(x), 1), 0.05), is_static=True)
    cp = ns.ConstrainedProblem(ns.DiffusionEquation(2, 0.3), ns.Mesh([(0.0, 1.0), (0.0, 1.3)], [1.0 / 16, 1.3 / 32]),
                               [(bc, free), (free, bc)])
    batch, d_t = 3, 0.4 / (0.3 * (16 ** 2 + (32 / 1.3) ** 2))
    rng = np.random.default_rng(6)
    y0 = np.stack([ns.DiscreteInitialCondition(cp, s * rng.random((17, 33, 1)), True).discrete_y_0(True)
                   for s in (1.0, 0.05, 4.0)])
    integ = fdm.BackwardEulerMethod(1.48e-8, limit) if kind == "be" else fdm.CrankNicolsonMethod(0.6, 1.48e-8, limit)
    plan = fdm.FDMOperator(integ, fdm.ThreePointCentralDifferenceMethod(), d_t).plan(cp, batch)
    start, want = plan.new_state(1), plan.new_state(1)
    plan.pack_device(torch.tensor(y0, device="cuda"), start[0])
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        try:
            plan.run(start[0], want, 1, 0.0, d_t)
        except RuntimeError as e:  # the limit: every element of an instance failed
            assert limit == 7 and "failed to converge" in str(e)
    its = list(plan.secant_iterations[0])

    lib, ip, s = _native.lib(), plan._ip, plan.implicit
    ip.batch, ip.dt, ip.a, ip.tol, ip.crank_nicolson = batch, d_t, s["a"], s["tol"], int(s["crank_nicolson"])
    ip.dirichlet = plan.params.dirichlet
    bufs = plan.new_state(9)
    p, p1, q0, q1, fu, f, f0, res, out = (b.data_ptr() for b in bufs)
    flags = torch.zeros(batch * plan.inst, dtype=torch.uint8, device="cuda")
    counters = torch.zeros((batch, 4), dtype=torch.int32, device="cuda")
    stats = torch.zeros((batch, 4), dtype=torch.float64, device="cuda")
    counts = torch.zeros(batch, dtype=torch.int32, device="cuda")
    counter = torch.zeros(1, dtype=torch.int32, device="cuda")
    y, stream = start.data_ptr(), plan.stream_handle()
    ref = ctypes.byref(ip)

    def check(rc):
        _native.check(rc, "implicit")

    def residual(x, q, prev):
        plan.rhs(x, f, d_t)
        check(lib.prml_implicit_residual(ref, x, y, f, fu, q, prev, counters.data_ptr(), stream))

    def stop(xs, xo, force):
        check(lib.prml_implicit_stop(ref, xs, xo, flags.data_ptr(), counters.data_ptr(), counter.data_ptr(), force, res,
                                     stats.data_ptr(), counts.data_ptr(), stream))

    plan.rhs(y, f0, 0.0)
    check(lib.prml_implicit_predict(ref, y, f0, fu, p, p1, flags.data_ptr(), counters.data_ptr(), stream))
    residual(p, q0, None)
    residual(p1, q1, q0)
    for it in range(1, limit + 1):
        check(lib.prml_implicit_update(ref, p, p1, q0, q1, flags.data_ptr(), counters.data_ptr(), stream))
        stop(p, p1, 0)
        p, p1 = p1, p
        if it == limit:
            stop(p, p1, 1)
            break
        q0, q1 = q1, q0
        residual(p1, q1, q0)
    check(lib.prml_implicit_finish(ref, res, f0, out, stream))
    torch.cuda.synchronize()
    assert [int(v) for v in counts.cpu()] == its
    assert torch.equal(bufs[8][..., :plan.ny], want[0][..., :plan.ny])
    total = stats[:, 1].cpu().numpy()
    assert np.all(total == 17 * 33)

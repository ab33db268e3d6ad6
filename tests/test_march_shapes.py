"""Marching kernels on calls beside the ones of test_march.py: meshes of more
rows than a grid has, and several instances (of a batch below the plan's
capacity, with start times of their own) per launch.  In float64 the results
equal the staged kernels' bit for bit (the same operations in the same
order); in float32 they differ by contraction only, at most steps x 16
roundings of 2^-24 relative L2."""

import numpy as np
import pytest

import pararealml_gb300 as ns
import problems
from golden_cases import rel_l2
from pararealml_gb300 import codegen
from pararealml_gb300.operators import fdm

pytestmark = pytest.mark.gpu

STAGED = (16, 32, 128)


def _plan(cp, integ, d_t, dtype, batch, tile):
    op = fdm.FDMOperator(getattr(fdm, integ)(), fdm.ThreePointCentralDifferenceMethod(), d_t, dtype=dtype, tile=tile)
    return op.plan(cp, batch)


def test_more_rows_than_a_grid_dimension_of_small_tiles():
    """280,001 x 5 vertices, RK4 (every kernel of the autotuner takes part)."""
    import torch

    bc = ns.DirichletBoundaryCondition(lambda x, t: np.zeros((len(x), 1)), is_static=True)
    mesh = ns.Mesh([(0.0, 2800.0), (0.0, 0.04)], [0.01, 0.01])
    cp = ns.ConstrainedProblem(ns.DiffusionEquation(2, 1.0), mesh, [(bc, bc)] * 2)
    y0 = torch.rand((1,) + tuple(cp.mesh.vertices_shape) + (1,), dtype=torch.float64, device="cuda")
    got = []
    for tile in (STAGED, codegen.march_tile(4, 1, 4), None):
        op = fdm.FDMOperator(fdm.RK4(), fdm.ThreePointCentralDifferenceMethod(), 1e-6, tile=tile, trajectory="final")
        got.append(op.solve_device(cp, y0, 0.0, 3))
    assert torch.equal(got[0][..., :5], got[1][..., :5]) and torch.equal(got[0][..., :5], got[2][..., :5])


_BATCHED = {
    # name: (problem, integrator, d_t, instances of the plan)
    "shallow_water": (lambda: problems.shallow_water_2d(ns, n=70), "RK4", 0.01, 3),
    "diffusion_7_strips": (lambda: problems.diffusion_2d(ns, n=210), "RK4", 1e-4, 7),
    "wave_dynamic": (lambda: problems.dynamic_bc_wave_2d(ns, nx=45, ny=91), "RK4", 0.001, 3),
    "wave_dynamic_fe": (lambda: problems.dynamic_bc_wave_2d(ns, nx=66, ny=21), "ForwardEulerMethod", 0.001, 7),
    "cahn_hilliard": (lambda: problems.cahn_hilliard_2d(ns, n=131, length=32.75), "RK4", 1e-4, 7),
}


def _states(plan, cp, ivp, batch, seed):
    """``batch`` different states of the plan's layout with the problem's Dirichlet values."""
    import torch

    rng = np.random.default_rng(seed)
    y = ivp.initial_condition.discrete_y_0(True)
    y = np.stack([y * rng.uniform(0.5, 1.5) + 0.05 * rng.standard_normal(y.shape) for _ in range(batch)])
    state = plan.new_state(1)
    plan.pack_device(torch.tensor(y, device="cuda"), state[0, :batch])
    return state


@pytest.mark.parametrize("every", [1, 4])
@pytest.mark.parametrize("name", sorted(_BATCHED))
def test_several_instances(name, every):
    """All instances of a plan, and all but one of them; time-dependent
    conditions with a start time and a boundary table per instance."""
    import torch

    build, integ, d_t, batch = _BATCHED[name]
    ivp = build()
    cp = ivp.constrained_problem
    steps = 4
    for dtype in ("float64", "float32"):
        gen = _plan(cp, integ, d_t, dtype, batch, None).module.gen
        for run in (batch, batch - 1):
            want = None
            for tile in [STAGED] + [t for t in gen.march_kernels if t[0] in (4, 24)]:
                plan = _plan(cp, integ, d_t, dtype, batch, tile)
                y0 = _states(plan, cp, ivp, batch, 5)
                kw = {}
                if plan.low.dynamic:
                    start = np.arange(batch) % 3
                    plan.preset_tables(0.0, d_t, steps + 2)
                    offset = torch.tensor(start * d_t, device="cuda")
                    slots = torch.tensor(2 * start, dtype=torch.int32, device="cuda")
                    kw = {"t_offset_ptr": offset.data_ptr(), "bc_inst_slot_ptr": slots.data_ptr()}
                out = plan.new_state(steps // every)
                out.fill_(float("nan"))
                plan.run(y0, out, steps, 0.0, d_t, save_every=every, batch=run,
                         traj_step_stride=batch * plan.inst, **kw)
                torch.cuda.synchronize()
                plan.check_status()
                # instances that do not take part are left alone
                assert bool(torch.isnan(out[:, run:]).all())
                got = out[:, :run, ..., :plan.ny].double().cpu().numpy()
                if want is None:
                    want = got
                    assert np.isfinite(got).all() and not any(np.array_equal(got[:, 0], got[:, b]) for b in range(1, run))
                elif dtype == "float64":
                    assert np.array_equal(got, want), (tile, run)
                else:
                    for b in range(run):
                        assert rel_l2(got[:, b], want[:, b]) < steps * 16 * 2.0 ** -24, (tile, run, b)

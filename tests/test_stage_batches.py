"""Stage kernels of 3D meshes with several instances per launch, all of a
plan's and fewer: in float64 the whole-step kernels' results bit for bit (the
same operations in the same order); in float32 they differ by contraction
only, at most steps x 16 roundings of 2^-24 relative L2."""

import numpy as np
import pytest

import pararealml_gb300 as ns
import problems
from golden_cases import rel_l2
from pararealml_gb300.operators import fdm

pytestmark = pytest.mark.gpu

_CASES = {
    "rk4": (lambda: problems.diffusion_3d_mixed(ns, n=(9, 13, 35)), "RK4", 0.001, 3),
    "midpoint": (lambda: problems.diffusion_3d_mixed(ns, n=(5, 4, 6)), "ExplicitMidpointMethod", 0.001, 7),
    "fe": (lambda: problems.diffusion_3d_mixed(ns, n=(8, 7, 65)), "ForwardEulerMethod", 0.0001, 7),
    "vector_field": (lambda: problems.curvilinear_vector_field(ns, "SPHERICAL"), "RK4", 0.001, 3),
}


@pytest.mark.parametrize("every", [1, 4])
@pytest.mark.parametrize("name", sorted(_CASES))
def test_several_instances(name, every):
    import torch

    build, integ, d_t, batch = _CASES[name]
    ivp = build()
    cp = ivp.constrained_problem
    rng = np.random.default_rng(9)
    y = ivp.initial_condition.discrete_y_0(True)
    y = torch.tensor(np.stack([y * rng.uniform(0.5, 1.5) + 0.05 * rng.standard_normal(y.shape) for _ in range(batch)]),
                     device="cuda")
    steps = 4

    def plan_of(dtype, tile):
        op = fdm.FDMOperator(getattr(fdm, integ)(), fdm.ThreePointCentralDifferenceMethod(), d_t, dtype=dtype, tile=tile)
        return op.plan(cp, batch)

    for dtype in ("float64", "float32"):
        gen = plan_of(dtype, None).module.gen
        assert gen.stage_kernels
        for run in (batch, batch - 1):
            want = None
            for tile in [next(iter(gen.step_kernels))] + list(gen.stage_kernels):
                plan = plan_of(dtype, tile)
                state, out = plan.new_state(1), plan.new_state(steps // every)
                plan.pack_device(y, state[0])
                out.fill_(float("nan"))
                plan.run(state, out, steps, 0.0, d_t, save_every=every, batch=run)  # slots of ``run`` instances
                torch.cuda.synchronize()
                flat, saved = out.flatten(0, 1), steps // every * run
                assert bool(torch.isnan(flat[saved:]).all())
                got = flat[:saved].unflatten(0, (-1, run))[..., :plan.ny].double().cpu().numpy()
                if want is None:
                    want = got
                    assert np.isfinite(got).all() and not any(np.array_equal(got[:, 0], got[:, b]) for b in range(1, run))
                elif dtype == "float64":
                    assert np.array_equal(got, want), (tile, run)
                else:
                    for b in range(run):
                        assert rel_l2(got[:, b], want[:, b]) < steps * 16 * 2.0 ** -24, (tile, run, b)

"""3D runs where the stage kernels' three work states do not fit: the tuned
whole-step kernel, which needs none, takes the run.

CPU: the choice, with the allocator and the launches replaced.  GPU: with an
allocator that refuses the work states, the same bits as with them (float64:
the same operations in the same order)."""

import types

import numpy as np
import pytest

import pararealml_gb300 as ns
import problems
from pararealml_gb300 import codegen, engine
from pararealml_gb300.operators import fdm

STAGE = (1, 2, 128, 1, 1, "s")
WHOLE = (8, 32, 256, 1, 2)


def test_a_run_without_room_takes_the_whole_step_kernel():
    torch = pytest.importorskip("torch")
    plan = object.__new__(engine.StencilPlan)
    plan.secant_iterations, plan.secant_warnings, plan.jacobi_iterations = [], [], []
    plan.low = types.SimpleNamespace(dynamic=False, lap_idx=())
    plan.tile, plan.implicit, plan.inst, plan.batch, plan._user_ctas = None, None, 64, 1, 0
    plan._tuned, plan._tuned_ctas, plan._tuned_whole = {True: STAGE}, {True: 0}, {True: (WHOLE, 304)}
    plan.params = types.SimpleNamespace(batch=1, t_offset=0, dirichlet=0, neumann=0, max_ctas=0)
    launched = []

    def launch(tile, *args):
        if codegen.is_stage(tile):
            raise torch.cuda.OutOfMemoryError("no room")
        launched.append((tile, plan.params.max_ctas, args))

    plan._launch = launch
    plan.run(1024, 2048, 4, 0.0, 0.1)
    assert [x[:2] for x in launched] == [(WHOLE, 304)] and launched[0][2][:2] == (1024, 64)
    assert (plan.last_tile, plan.last_ctas) == (WHOLE, 304)
    plan.tile = STAGE  # the caller's own choice fails as it is
    with pytest.raises(torch.cuda.OutOfMemoryError):
        plan.run(1024, 2048, 4, 0.0, 0.1)


@pytest.mark.gpu
@pytest.mark.parametrize("when", ["run", "tuning"])
def test_without_work_states(monkeypatch, when):
    import torch

    ivp = problems.diffusion_3d_mixed(ns, n=(21, 24, 35), t_end=0.012)
    tuned = {}

    def solve(refuse, cache):
        monkeypatch.setattr(engine, "_tune_cache_load", lambda: cache)
        monkeypatch.setattr(engine, "_tune_cache_store", lambda key, entry: cache.update({key: entry}))
        op = fdm.FDMOperator(fdm.RK4(), fdm.ThreePointCentralDifferenceMethod(), 0.001)
        plan = op.plan(ivp.constrained_problem, 1)
        launch, new_state, inside = plan._launch, plan.new_state, [False]

        def launching(tile, *args):
            inside[0] = codegen.is_stage(tile)
            try:
                launch(tile, *args)
            finally:
                inside[0] = False

        def states(n=1):
            if inside[0] and refuse:
                raise torch.cuda.OutOfMemoryError("no room")
            return new_state(n)

        plan._launch, plan.new_state = launching, states
        return op.solve(ivp).discrete_y(), plan.last_tile

    want, tile = solve(False, tuned)
    assert codegen.is_stage(tile)  # faster by far on this mesh
    got, tile = solve(True, tuned if when == "run" else {})
    assert not codegen.is_stage(tile)
    assert np.array_equal(got, want)

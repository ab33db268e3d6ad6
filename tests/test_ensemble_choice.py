"""Ensembles on streams: kernels tuned alone are kept only where the whole
advance, all groups side by side, is faster with them."""

import types

import pytest

import pararealml_gb300 as ns
import problems
from pararealml_gb300.ensemble import EnsembleSolver
from pararealml_gb300.operators import fdm
from pararealml_gb300 import codegen, engine

STAGED, RESIDENT = (16, 32, 256), codegen.RESIDENT_TILE


class _Plan:
    tuned_choices = engine.StencilPlan.tuned_choices
    set_tuned = engine.StencilPlan.set_tuned
    tile = implicit = None

    def __init__(self, pick):
        self.module = types.SimpleNamespace(gen=types.SimpleNamespace(step_kernels={STAGED: ("n", 0)}))
        self._tuned, self._tuned_ctas = {False: pick}, {False: 0}
        self._tuned_whole = {False: (STAGED, 304)}


@pytest.mark.parametrize("tuned_ms,staged_ms,keeps", [(1.0, 2.0, True), (2.0, 1.0, False)])
def test_the_faster_advance_decides(tuned_ms, staged_ms, keeps):
    solver = EnsembleSolver(fdm.RK4(), fdm.ThreePointCentralDifferenceMethod())
    plans = [_Plan(STAGED), _Plan(RESIDENT)]
    solver._groups = [{"plan": p, "n_steps": 4} for p in plans]
    solver._time_replay = lambda: tuned_ms if plans[1]._tuned[False] == RESIDENT else staged_ms
    solver._choose_kernels()
    assert (plans[1]._tuned[False], plans[1]._tuned_ctas[False]) == ((RESIDENT, 0) if keeps else (STAGED, 304))
    assert (plans[0]._tuned[False], plans[0]._tuned_ctas[False]) == (STAGED, 0)


def test_nothing_is_timed_where_there_is_nothing_to_choose():
    solver = EnsembleSolver(fdm.RK4(), fdm.ThreePointCentralDifferenceMethod())
    solver._time_replay = lambda: pytest.fail("timed")
    solver._groups = [{"plan": _Plan(RESIDENT), "n_steps": 4}]  # one group: tuned as it runs
    solver._choose_kernels()
    solver._groups = [{"plan": _Plan(STAGED), "n_steps": 4} for _ in range(2)]
    solver._choose_kernels()


@pytest.mark.gpu
@pytest.mark.parametrize("use_graph", [True, False])
def test_small_meshes_side_by_side(use_graph):
    """Meshes whose tuned kernels are resident ones: the results of single
    solves bit for bit, whichever set is kept (float64)."""
    import numpy as np

    ivps, d_ts = problems.shallow_water_ensemble(ns, n_instances=9, sizes=(16, 32, 48), t_end=0.5, seed=11)
    solver = EnsembleSolver(fdm.RK4(), fdm.ThreePointCentralDifferenceMethod(), dtype="float64", launch="streams",
                            use_graph=use_graph)
    solver.setup(ivps, d_ts)
    for _ in range(3):
        solver.advance()
    for ivp, d_t, y in zip(ivps, d_ts, solver.final_states()):
        op = fdm.FDMOperator(fdm.RK4(), fdm.ThreePointCentralDifferenceMethod(), d_t, trajectory="final", tile=STAGED)
        assert np.array_equal(y, op.solve(ivp).discrete_y()[-1])

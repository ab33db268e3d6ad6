"""The time of a secant iteration grows with the mesh no faster than its work:
every CTA of a launch reports to the same few counters, which must not become
the bound on large meshes."""

import warnings

import numpy as np
import pytest

import pararealml_gb300 as ns
from pararealml_gb300.operators import fdm

pytestmark = pytest.mark.gpu


def test_time_of_an_iteration_grows_with_the_work():
    """Backward Euler diffusion (50 iterations, the limit, on both meshes): four
    times the vertices may take twice four times as long."""
    import torch

    def us_per_iteration(n):
        bc = ns.DirichletBoundaryCondition(lambda x, t: np.zeros((len(x), 1)), is_static=True)
        cp = ns.ConstrainedProblem(ns.DiffusionEquation(2, 1.0), ns.Mesh([(0.0, 10.0)] * 2, [10.0 / n] * 2), [(bc, bc)] * 2)
        op = fdm.FDMOperator(fdm.BackwardEulerMethod(), fdm.ThreePointCentralDifferenceMethod(), 1e-3)
        g = np.exp(-0.5 * (np.linspace(0.0, 10.0, n + 1) - 4.7) ** 2)
        y0 = torch.tensor(np.outer(g, g)[None, ..., None], device="cuda")
        best = float("inf")
        with warnings.catch_warnings():
            warnings.simplefilter("ignore", RuntimeWarning)
            for _ in range(4):  # the first one compiles
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                op.solve_device(cp, y0, 0.0, 3)
                b.record()
                b.synchronize()
                best = min(best, a.elapsed_time(b) * 1e3)
        return best / sum(its[0] for its in op.plan(cp, 1).secant_iterations)

    assert us_per_iteration(512) < 8 * us_per_iteration(256)

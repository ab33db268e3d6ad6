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

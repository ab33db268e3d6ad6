"""Marching step kernels (``march_body``): a warp walks a strip of columns down
the rows with every integrator stage (or several time steps) in registers.

CPU: every global access of every job stays inside the state and each vertex
is stored exactly once.  GPU: in float64 the results equal the staged
kernels' bit for bit (the same operations in the same order) on ragged meshes
with every kind of face, for every shape of kernel; in float32 they differ by
contraction only: at most 12 steps x 16 roundings of 2^-24, 1.2e-5.
"""

import numpy as np
import pytest

import pararealml_gb300 as ns
import problems
from golden_cases import rel_l2
from pararealml_gb300 import codegen
from pararealml_gb300.operators import fdm

REL_F32 = 12 * 16 * 2.0 ** -24
STAGED = (16, 32, 128)


def _shapes(esize):
    multi = [(vw, depth, 1) for vw in codegen.MARCH_MULTI[esize] for depth in (2, 4)]
    return multi + [(vw, depth, depth) for vw, depth in codegen.MARCH_SINGLE[esize]]


def _jobs(tile, nx, ny, rows, edge_rows):
    """(first row, chunk rows, first column) of every job, as march_body takes them."""
    vw = tile[6]
    hl = (32 * vw - tile[1]) // (2 * vw)
    strips = -(-ny // tile[1])
    edges = min(2, strips)
    for strip in range(strips):
        edge = strip == 0 or (edges == 2 and strip == strips - 1)
        n = edge_rows if edge else rows
        for chunk in range(-(-nx // n)):
            yield chunk * n, n, strip * tile[1] - hl * vw


@pytest.mark.parametrize("esize", [4, 8])
@pytest.mark.parametrize("nx,ny,batch", [(3, 3, 1), (5, 40, 3), (40, 5, 1), (17, 57, 1), (65, 65, 2), (130, 257, 1)])
def test_accesses_stay_inside_the_state(esize, nx, ny, batch):
    pitch = -(-ny // 32) * 32
    for vw, depth, steps in _shapes(esize):
        for jobs in codegen.MARCH_JOBS[::2]:
            tile = codegen.march_tile(jobs, vw, depth, steps)
            hl = (32 * vw - tile[1]) // (2 * vw)
            assert hl * vw >= depth and (tile[1] * esize) % min(16, vw * esize) == 0
            rows, edge_rows = codegen.march_rows(tile, nx, ny, batch, esize, 152)
            assert 1 <= rows <= nx and 1 <= edge_rows <= nx
            seen = np.zeros((nx, ny), dtype=int)
            for r0, n, c0 in _jobs(tile, nx, ny, rows, edge_rows):
                r1 = min(r0 + n, nx)
                for lane in range(32):
                    gj0 = c0 + lane * vw
                    if 0 <= gj0 < ny:  # the vectors a lane loads start inside the mesh
                        assert gj0 % vw == 0 and gj0 + vw <= pitch
                    if hl <= lane < 32 - hl and gj0 < ny:  # and stores
                        assert gj0 >= 0
                        seen[r0:r1, gj0:min(gj0 + vw, ny)] += 1
            assert np.all(seen == 1), (tile, rows, edge_rows)


def test_where_marching_kernels_exist():
    """2D meshes without Jacobi rows; multi-stage systems of dy/dt rows only."""
    def kernels(ivp, integ, dtype="f64", **kw):
        return codegen.generate_source(codegen.lower_problem(ivp.constrained_problem), integ, dtype, **kw).march_kernels

    assert kernels(problems.shallow_water_2d(ns, n=16), codegen.RK4)
    assert kernels(problems.cahn_hilliard_2d(ns, n=16), codegen.RK4)  # one stage: mu is an LHS.Y row
    assert not kernels(problems.cahn_hilliard_2d(ns, n=16), codegen.RK4, "f32c")
    assert not kernels(problems.convection_diffusion_1d(ns, n=20), codegen.RK4)
    assert not kernels(problems.navier_stokes_2d(ns), codegen.RK4)
    assert not kernels(problems.diffusion_2d(ns, n=16), codegen.FORWARD_EULER, exact_div=True)


_CASES = {
    "diffusion": (lambda: problems.diffusion_2d(ns, n=57, t_end=0.012), "RK4", 0.001),
    "diffusion_5x5": (lambda: problems.diffusion_2d(ns, n=4, t_end=0.012), "RK4", 0.001),
    "diffusion_5x5_fe": (lambda: problems.diffusion_2d(ns, n=4, t_end=0.012), "ForwardEulerMethod", 0.001),
    "shallow_water": (lambda: problems.shallow_water_2d(ns, n=70, t_end=0.12), "RK4", 0.01),
    "wave_partial_faces": (lambda: problems.mixed_bc_wave_2d(ns, nx=77, ny=145, t_end=0.012), "RK4", 0.001),
    "wave_midpoint": (lambda: problems.mixed_bc_wave_2d(ns, nx=45, ny=77, t_end=0.012), "ExplicitMidpointMethod", 0.001),
    "wave_dynamic_faces": (lambda: problems.dynamic_bc_wave_2d(ns, nx=26, ny=91, t_end=0.012), "RK4", 0.001),
    "wave_dynamic_fe": (lambda: problems.dynamic_bc_wave_2d(ns, nx=66, ny=21, t_end=0.012), "ForwardEulerMethod", 0.001),
    "burgers_cauchy": (lambda: problems.burgers_2d(ns, n=24, t_end=0.012), "RK4", 0.001),
    "polar": (lambda: problems.polar_shallow_water(ns, t_end=0.012), "RK4", 0.001),
    "cahn_hilliard": (lambda: problems.cahn_hilliard_2d(ns, n=131, length=32.75, t_end=0.012), "RK4", 0.001),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(_CASES))
def test_marching_kernels_equal_the_staged_kernels(name):
    build, integ, d_t = _CASES[name]
    ivp = build()

    def solve(dtype, tile, trajectory):
        op = fdm.FDMOperator(getattr(fdm, integ)(), fdm.ThreePointCentralDifferenceMethod(), d_t, dtype=dtype,
                             tile=tile, trajectory=trajectory)
        return op.solve(ivp).discrete_y(), op.plan(ivp.constrained_problem, 1).module.gen

    for dtype in ("float64", "float32"):
        for trajectory in ("full", 4, "final"):
            want, gen = solve(dtype, STAGED, trajectory)
            for tile in gen.march_kernels:
                if tile[0] not in (4, 24):  # few long jobs, many short ones
                    continue
                got, _ = solve(dtype, tile, trajectory)
                if dtype == "float64":
                    assert np.array_equal(got, want), (tile, trajectory, float(np.max(np.abs(got - want))))
                else:
                    assert rel_l2(got, want) < REL_F32, (tile, trajectory)

"""Resident step kernel (``resident_body``): a small 2D mesh in the shared
memory of one thread-block cluster per instance, all steps in one launch.

CPU: which meshes it takes and how their rows are dealt.  GPU: in float64 the
results equal the staged kernels' bit for bit (the same operations in the same
order) on ragged bands with every kind of face; in float32 they differ by
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


@pytest.mark.parametrize("most", [2, 8, 16])
def test_every_cta_of_a_cluster_holds_rows(most):
    for nx in (2, 3, 5, 16, 17, 31, 65, 101, 181, 500):
        for ny in (3, 40, 65, 181):
            shape = codegen.resident_shape(nx, ny, 2, 8, 4, most)
            if shape is None:
                assert nx * ny > codegen.RESIDENT_VERTICES[8] or 4 * 2 * (-(-nx // most) + 2) * (ny + 2) * 8 > codegen.RESIDENT_SMEM
                continue
            cluster, band = shape
            assert 2 <= cluster <= most and cluster * band >= nx > (cluster - 1) * band
    assert codegen.resident_shape(1, 65, 1, 8, 1, 16) is None  # nothing to split
    assert codegen.resident_shape(65, 65, 1, 8, 1, 0) is None  # no clusters on the device
    assert codegen.resident_shape(257, 257, 1, 8, 1, 16) is None


def test_where_the_resident_kernel_exists():
    def kernels(ivp, integ, dtype="f64", **kw):
        return codegen.generate_source(codegen.lower_problem(ivp.constrained_problem), integ, dtype, **kw).resident_kernels

    assert kernels(problems.diffusion_2d(ns, n=16), codegen.RK4)
    assert kernels(problems.cahn_hilliard_2d(ns, n=16), codegen.RK4, "f32")
    assert not kernels(problems.cahn_hilliard_2d(ns, n=16), codegen.RK4, "f32c")
    assert not kernels(problems.convection_diffusion_1d(ns, n=20), codegen.RK4)
    assert not kernels(problems.navier_stokes_2d(ns), codegen.RK4)
    assert not kernels(problems.diffusion_2d(ns, n=16), codegen.FORWARD_EULER, exact_div=True)


_CASES = {
    "diffusion": (lambda: problems.diffusion_2d(ns, n=57, t_end=0.012), "RK4", 0.001),
    "diffusion_5x5": (lambda: problems.diffusion_2d(ns, n=4, t_end=0.012), "RK4", 0.001),
    "diffusion_97_fe": (lambda: problems.diffusion_2d(ns, n=96, t_end=0.0012), "ForwardEulerMethod", 0.0001),
    "shallow_water": (lambda: problems.shallow_water_2d(ns, n=70, t_end=0.12), "RK4", 0.01),
    "wave_partial_faces": (lambda: problems.mixed_bc_wave_2d(ns, nx=67, ny=145, t_end=0.012), "RK4", 0.001),
    "wave_midpoint": (lambda: problems.mixed_bc_wave_2d(ns, nx=45, ny=77, t_end=0.012), "ExplicitMidpointMethod", 0.001),
    "wave_dynamic_faces": (lambda: problems.dynamic_bc_wave_2d(ns, nx=26, ny=91, t_end=0.012), "RK4", 0.001),
    "wave_dynamic_fe": (lambda: problems.dynamic_bc_wave_2d(ns, nx=66, ny=21, t_end=0.012), "ForwardEulerMethod", 0.001),
    "burgers_cauchy": (lambda: problems.burgers_2d(ns, n=24, t_end=0.012), "RK4", 0.001),
    "polar": (lambda: problems.polar_shallow_water(ns, t_end=0.012), "RK4", 0.001),
    "cahn_hilliard": (lambda: problems.cahn_hilliard_2d(ns, n=91, length=22.75, t_end=0.012), "RK4", 0.001),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(_CASES))
def test_resident_kernel_equals_the_staged_kernels(name):
    build, integ, d_t = _CASES[name]
    ivp = build()

    def solve(dtype, tile, trajectory):
        op = fdm.FDMOperator(getattr(fdm, integ)(), fdm.ThreePointCentralDifferenceMethod(), d_t, dtype=dtype,
                             tile=tile, trajectory=trajectory)
        return op.solve(ivp).discrete_y()

    for dtype in ("float64", "float32"):
        for trajectory in ("full", 4, "final"):
            want = solve(dtype, STAGED, trajectory)
            got = solve(dtype, codegen.RESIDENT_TILE, trajectory)
            if dtype == "float64":
                assert np.array_equal(got, want), (trajectory, float(np.max(np.abs(got - want))))
            else:
                assert rel_l2(got, want) < REL_F32, trajectory


@pytest.mark.gpu
def test_more_instances_than_clusters_fit_and_long_runs():
    """24 instances of 16 CTAs (more than the GPU holds at once) and more steps
    than one launch takes, against the staged kernel bit for bit."""
    import torch

    ivp = problems.diffusion_2d(ns, n=33)
    cp = ivp.constrained_problem
    rng = np.random.default_rng(3)
    y0 = rng.random((24,) + tuple(cp.mesh.vertices_shape) + (1,))
    out = []
    for tile in (STAGED, codegen.RESIDENT_TILE):
        op = fdm.FDMOperator(fdm.ForwardEulerMethod(), fdm.ThreePointCentralDifferenceMethod(), 1e-5, tile=tile)
        plan = op.plan(cp, 24)
        start = plan.new_state(1)
        plan.pack(y0, start[0])
        traj = plan.new_state(5)
        plan.run(start[0], traj, 20000, 0.0, 1e-5, 4000, work=plan.new_state(2))
        torch.cuda.synchronize()
        out.append(plan.unpack(traj, 5 * 24).cpu().numpy())
    assert np.array_equal(out[0], out[1])

"""Kernels launched once per integrator stage of a multi-stage step
on 3D meshes (``stage_body3``).

CPU: for which problems they exist and which vertices a thread holds.  GPU: in
float64 the results equal the whole-step kernels' bit for bit (the same
operations in the same order, through memory instead of registers) on ragged
meshes with every kind of face; in float32 they differ by contraction only:
at most 12 steps x 16 roundings of 2^-24, 1.2e-5.
"""

import numpy as np
import pytest

import pararealml_gb300 as ns
import problems
from golden_cases import rel_l2
from pararealml_gb300 import codegen
from pararealml_gb300.operators import fdm

REL_F32 = 12 * 16 * 2.0 ** -24


def _gen(ivp, integ, dtype="f64", **kw):
    return codegen.generate_source(codegen.lower_problem(ivp.constrained_problem), integ, dtype, **kw)


def test_where_stage_kernels_exist():
    """3D steps whose right-hand side every stage evaluates anew, with nothing solved between the steps."""
    assert _gen(problems.diffusion_3d_mixed(ns), codegen.RK4).stage_kernels
    assert _gen(problems.diffusion_3d_mixed(ns), codegen.FORWARD_EULER).stage_kernels
    assert not _gen(problems.cahn_hilliard_3d(ns), codegen.RK4).stage_kernels  # one stage is the step
    assert not _gen(problems.diffusion_3d_mixed(ns), codegen.FORWARD_EULER, exact_div=True).stage_kernels
    assert not _gen(problems.diffusion_2d(ns, n=16), codegen.RK4).stage_kernels


def _threads(n, esize, planes):
    """(plane, row, first column) of every thread of an instance, as stage_body3 takes them."""
    vw = 16 // esize
    vecs = -(-n[2] // vw)
    jobs = -(-n[0] // planes) * n[1] * vecs
    for job in range(-(-jobs // codegen.STAGE_THREADS) * codegen.STAGE_THREADS):
        line, vec = divmod(min(job, jobs - 1), vecs)
        chunk, row = divmod(line, n[1])
        yield job < jobs, chunk * planes, row, vec * vw


@pytest.mark.parametrize("esize", [4, 8])
@pytest.mark.parametrize("n", [(3, 3, 3), (9, 14, 35), (5, 6, 64), (4, 3, 33)])
def test_accesses_stay_inside_the_state(n, esize):
    """Every vertex is stored once; a lane whose neighbour column is inside
    the mesh finds it in the neighbouring lane or is the warp's first or last."""
    vw, pitch = 16 // esize, -(-n[2] // 32) * 32
    for planes in codegen.STAGE_PLANES:
        seen = np.zeros(n, dtype=int)
        prev = None
        for t, (active, k, i, j) in enumerate(_threads(n, esize, planes)):
            assert 0 <= k < n[0] and 0 <= i < n[1] and j + vw <= pitch
            if t % 32 and j > 0 and active:
                assert prev == (k, i, j - vw)
            prev = (k, i, j)
            if active:
                seen[k:k + planes, i, j:j + vw] += 1
        assert np.all(seen == 1)


_CASES = {
    "diffusion_3d": (lambda: problems.diffusion_3d_mixed(ns, n=(9, 13, 35), t_end=0.012), "RK4", 0.001),
    "diffusion_3d_equal_steps": (lambda: problems.diffusion_3d_mixed(ns, n=(8, 12, 14), t_end=0.012), "RK4", 0.001),
    "cahn_hilliard_fe": (lambda: problems.cahn_hilliard_3d(ns, t_end=0.012), "ForwardEulerMethod", 0.001),
    "diffusion_3d_midpoint": (lambda: problems.diffusion_3d_mixed(ns, n=(5, 4, 6), t_end=0.012),
                              "ExplicitMidpointMethod", 0.001),
    "diffusion_3d_fe": (lambda: problems.diffusion_3d_mixed(ns, n=(8, 7, 65), t_end=0.0012), "ForwardEulerMethod", 0.0001),
    "vector_field": (lambda: problems.curvilinear_vector_field(ns, "SPHERICAL", t_end=0.012), "RK4", 0.001),
    "cylindrical": (lambda: problems.curvilinear_diffusion_3d(ns, "CYLINDRICAL", t_end=0.012), "RK4", 0.001),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(_CASES))
def test_stage_kernels_equal_whole_step_kernels(name):
    build, integ, d_t = _CASES[name]
    ivp = build()

    def solve(dtype, tile, trajectory):
        op = fdm.FDMOperator(getattr(fdm, integ)(), fdm.ThreePointCentralDifferenceMethod(), d_t, dtype=dtype,
                             tile=tile, trajectory=trajectory)
        return op.solve(ivp).discrete_y(), op.plan(ivp.constrained_problem, 1).module.gen

    for dtype in ("float64", "float32"):
        whole = next(iter(solve(dtype, None, "final")[1].step_kernels))
        for trajectory in ("full", 4, "final"):
            want, gen = solve(dtype, whole, trajectory)
            assert gen.stage_kernels
            for tile in gen.stage_kernels:
                got, _ = solve(dtype, tile, trajectory)
                if dtype == "float64":
                    assert np.array_equal(got, want), (tile, trajectory, float(np.max(np.abs(got - want))))
                else:
                    assert rel_l2(got, want) < REL_F32, (tile, trajectory)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["diffusion_3d", "diffusion_3d_equal_steps", "cahn_hilliard_fe"])
def test_fused_order_on_3d_meshes(name):
    """Fused operation order against the reference's on the same device, with
    whole-step and stage kernels: at most 12 steps x 4 stages x 24 roundings
    of 2^-53 of a diffusing state, 1.3e-13 relative L2."""
    build, integ, d_t = _CASES[name]
    ivp = build()

    def solve(op_order, kind):
        op = fdm.FDMOperator(getattr(fdm, integ)(), fdm.ThreePointCentralDifferenceMethod(), d_t, op_order=op_order)
        gen = op.plan(ivp.constrained_problem, 1).module.gen
        kernels = getattr(gen, kind)
        if not kernels:
            return None
        op = fdm.FDMOperator(getattr(fdm, integ)(), fdm.ThreePointCentralDifferenceMethod(), d_t, op_order=op_order,
                             tile=next(iter(kernels)))
        return op.solve(ivp).discrete_y()

    want = solve("reference", "step_kernels")
    for kind in ("step_kernels", "stage_kernels"):
        got = solve("fused", kind)
        assert got is None or rel_l2(got, want) < 12 * 4 * 24 * 2.0 ** -53

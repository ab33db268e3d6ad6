"""The anti-Laplacian on one thread-block cluster per instance: mesh sizes on
both sides of the kernel's edges (clusters of fewer CTAs where a CTA would
own less than one halo, one / two / four vertices per thread, the largest
mesh it takes and the next one, which runs on the grid-wide kernel), every
coordinate system, batches beyond the resident clusters, and the stop inside,
at the end and after several blocks of 16 iterations.  Against the oracle:
float64 iteration for iteration and within 1e-12 relative L2; float32 within
an iteration and 1e-4 (its rounding of the estimates), as for the other
kernels."""

import numpy as np
import pytest

import pararealml_gb300 as ns
import problems
from golden_cases import rel_l2
from oracle import fdm as orc
from test_gpu_jacobi import REL_F64, _device_solve, _oracle_solve, _plan, _smooth_rhs

pytestmark = pytest.mark.gpu


def _mesh(system, n):
    lo = {"CARTESIAN": (0.0, -1.0, 0.3), "POLAR": (1.0, 0.0), "SPHERICAL": (1.0, 0.0, 0.6)}[system]
    length = {"CARTESIAN": (2.0, 2.5, 1.4), "POLAR": (2.0, 3.0), "SPHERICAL": (2.0, 3.0, 1.8)}[system]
    return ([(lo[a], lo[a] + length[a]) for a in range(len(n))], [length[a] / (n[a] - 1) for a in range(len(n))])


def _first_change(ivp, lap, init):
    one, _ = _oracle_solve(ivp, lap, init, 1e9)
    c = orc.FDMStepper(ivp.constrained_problem, "rk4", 0.01).yc(0.0)
    return float(np.linalg.norm(one - orc.apply_y_constraints(c[[1]], init.copy())))


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("system,n", [
    ("CARTESIAN", (3,)), ("CARTESIAN", (40,)), ("CARTESIAN", (3, 3)), ("CARTESIAN", (5, 4)), ("CARTESIAN", (4, 70)),
    ("CARTESIAN", (17, 33)), ("CARTESIAN", (64, 128)), ("CARTESIAN", (65, 127)), ("CARTESIAN", (128, 128)),
    ("CARTESIAN", (181, 181)), ("CARTESIAN", (182, 181)), ("CARTESIAN", (9, 10, 11)), ("CARTESIAN", (31, 32, 33)),
    ("POLAR", (41, 50)), ("SPHERICAL", (9, 8, 10)),
])
def test_cluster_solve_matches_the_oracle(system, n, dtype):
    ivp = problems.jacobi_system(ns, system, len(n), mesh=_mesh(system, n))
    rng = np.random.default_rng(3)
    lap = _smooth_rhs(ivp, rng)
    init = rng.random(lap.shape)
    tol = 0.03 * _first_change(ivp, lap, init)
    want, its = _oracle_solve(ivp, lap, init, tol)
    got, dev = _device_solve(_plan(ivp, tol=tol, dtype=dtype), lap[None], [init])
    if dtype == "float64":
        assert dev == [its] and rel_l2(got[0], want) < REL_F64
    else:
        assert abs(dev[0] - its) <= 1 and rel_l2(got[0], want) < 1e-4


def test_batch_beyond_the_resident_clusters_and_stop_positions():
    """Forty instances whose tolerances (through the scale of their data) stop
    them at different iterations of a block."""
    ivp = problems.jacobi_system(ns, "CARTESIAN", 2, mesh=_mesh("CARTESIAN", (21, 26)))
    rng = np.random.default_rng(8)
    scales = np.geomspace(0.05, 20.0, 40)
    laps = [_smooth_rhs(ivp, rng, s) for s in scales]
    inits = [rng.random(laps[0].shape) * s for s in scales]
    got, its = _device_solve(_plan(ivp, batch=40, tol=0.02), np.stack(laps), inits)
    for b in range(40):
        want, n = _oracle_solve(ivp, laps[b], inits[b], 0.02)
        assert its[b] == n and rel_l2(got[b], want) < REL_F64, b
    assert len({n % 16 for n in its}) > 8

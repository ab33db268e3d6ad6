"""The change norms that the CTAs of a cluster exchange every 16 Jacobi
iterations (``jacobi_cluster``) when the last block is a short one, as an
iteration limit that is no multiple of 16 makes it.

CPU: with one CTA as late as the waits of the kernel allow and the others as
early, no CTA's sums are overwritten before the late one has read them.  GPU:
solves that stop in, or are cut off by, a second or third block of a few
iterations, against the oracle (float64, 1e-12 relative L2)."""

import pathlib
import re

import numpy as np
import pytest

import pararealml_gb300 as ns
import problems
from golden_cases import rel_l2
from oracle import fdm as orc
from pararealml_gb300 import _native

SOURCE = pathlib.Path(_native.__file__).parent / "csrc" / "prml_jacobi.cu"
BLOCK = 16


def _copies():
    """Copies of the exchanged sums that the kernel declares."""
    text = SOURCE.read_text()
    dims = re.search(r"__shared__ double cpart((?:\[\w+\])+)", text).group(1).strip("[]").split("][")
    if len(dims) < 3:
        return 1
    return int(re.search(rf"constexpr int {dims[0]} = (\d+);", text).group(1))


def _overwritten(ctas, late, blocks, copies):
    """Whether a CTA can send the sums of block n + 1 over those of block n
    that CTA ``late`` has yet to read.  After the cluster barrier of block n a
    CTA waits for nobody but its two neighbours' halos: d ranks away from one
    that has not begun block n + 1 it completes d - 1 iterations of it, and
    may send that block's sums if that is all of it.  It cannot pass that
    block's cluster barrier, so no later block's sums are in flight."""
    for n in range(len(blocks) - 1):
        if n % copies != (n + 1) % copies:
            continue
        for rank in range(ctas):
            if rank != late and abs(rank - late) - 1 >= blocks[n + 1]:
                return True
    return False


@pytest.mark.parametrize("ctas", [2, 3, 8, 16])
@pytest.mark.parametrize("limit", [16, 17, 20, 32, 35, 47, 1_000_000])
def test_no_sum_is_overwritten_before_it_is_read(ctas, limit):
    full, rest = divmod(limit, BLOCK)
    blocks = [BLOCK] * min(full, 4) + ([rest] if rest else [])
    for late in range(ctas):
        assert not _overwritten(ctas, late, blocks, _copies())


def _changes(ivp, lap, init, count):
    """2-norm of the change of each of the first ``count`` iterations."""
    st = orc.FDMStepper(ivp.constrained_problem, "rk4", 0.01)
    idx = st.rhs.lap_idx
    yc, dbc = st.yc(0.0)[idx], orc._dbc(st.dyc(0.0)[:, idx], lap.ndim - 1, lap.shape[-1])
    y = init.copy()
    orc.apply_y_constraints(yc, y)
    out = []
    for _ in range(count):
        new = orc.anti_laplacian_estimate(st.rhs.cs, y, lap, st.rhs.d_x, dbc, st.rhs.grids)
        orc.apply_y_constraints(yc, new)
        out.append(float(np.linalg.norm(new - y)))
        y = new
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [17, 20, 35])
def test_limits_that_leave_a_short_last_block(limit):
    """101 x 81 vertices: 16 CTAs.  The tolerances put the stop on the first
    and last iteration of the short block, and beyond the limit."""
    from test_gpu_jacobi import REL_F64, _device_solve, _oracle_solve, _plan, _smooth_rhs

    mesh = ([(-2.5, 2.5), (0.0, 4.0)], [0.05, 0.05])
    ivp = problems.jacobi_system(ns, "CARTESIAN", 2, mesh=mesh)
    rng = np.random.default_rng(limit)
    lap = _smooth_rhs(ivp, rng)
    init = rng.random(lap.shape)
    change = _changes(ivp, lap, init, limit + 1)
    assert all(a > b for a, b in zip(change, change[1:]))
    plan = _plan(ivp)
    plan.jacobi_max_iterations = limit
    for stop in (limit // BLOCK * BLOCK + 1, limit, limit + 1):
        tol = 0.5 * (change[stop - 1] + change[stop - 2])
        want, n = _oracle_solve(ivp, lap, init, tol)
        assert n == stop
        plan.jacobi_tol = tol
        for _ in range(20):
            if stop > limit:
                with pytest.raises(_native.ConvergenceError):
                    _device_solve(plan, lap[None], [init])
                assert plan.jacobi_iterations[-1] == [-1]
            else:
                got, its = _device_solve(plan, lap[None], [init])
                assert its == [n] and rel_l2(got[0], want) < REL_F64

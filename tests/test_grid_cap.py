"""``max_ctas``: no launch of a step kernel has more CTAs than the caller
allows, whichever kernel family takes the step.

CPU: with a cap the autotuner chooses among the kernels whose CTAs walk over
their tiles.  GPU: marching, stage and resident kernels under a cap launch at
most that many CTAs and give the uncapped results bit for bit (the same
operations; only the launches are cut differently)."""

import ctypes
import types

import numpy as np
import pytest

import pararealml_gb300 as ns
import problems
from pararealml_gb300 import codegen, engine
from pararealml_gb300.operators import fdm


def _gen(ivp, integ, dtype="f64"):
    return codegen.generate_source(codegen.lower_problem(ivp.constrained_problem), integ, dtype, fast=True)


def tuning_plan(monkeypatch, gen, cost, stored):
    """A plan whose autotune() runs on a clock that ``cost(tile)`` advances
    per launch, with ``stored`` as the cache; and the set of tiles it times."""
    torch = pytest.importorskip("torch")
    clock, timed = [0.0], set()

    class Event:
        def __init__(self, enable_timing=True):
            pass

        def record(self):
            self.t = clock[0]

        def synchronize(self):
            pass

        def elapsed_time(self, other):
            return other.t - self.t

    class State:
        zero_ = lambda self: self  # noqa: E731
        data_ptr = lambda self: 0  # noqa: E731
        __getitem__ = lambda self, i: self  # noqa: E731

    def occupancy(kernel, threads, occ):
        occ._obj.value = 1
        return 0

    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "get_device_properties",
                        lambda dev: types.SimpleNamespace(multi_processor_count=152, name="GPU"))
    monkeypatch.setattr(engine._native, "lib", lambda: types.SimpleNamespace(prml_kernel_occupancy=occupancy))
    monkeypatch.setattr(engine._native, "check", lambda rc, what: None)
    monkeypatch.setattr(engine, "_tune_cache_load", lambda: stored)
    monkeypatch.setattr(engine, "_tune_cache_store", lambda key, entry: stored.update({key: entry}))
    plan = object.__new__(engine.StencilPlan)
    plan.tile, plan._tuned, plan._tuned_ctas, plan._tuned_whole, plan._resident = None, {}, {}, {}, (4, 4)
    plan.module = types.SimpleNamespace(gen=gen)
    plan.nz, plan.rows, plan.ny, plan.C, plan.esize, plan.batch, plan.inst = 1, 17, 17, 1, 8, 1, 1
    plan.device, plan._user_ctas = "cuda", 0
    plan.params = types.SimpleNamespace(bc_stride=0, max_ctas=0)
    plan.new_state = lambda n: State()
    plan._step_kernel = lambda tile: tile
    plan.resident_shape = lambda: (4, 5)

    def launch(tile, *a):
        timed.add(tile)
        clock[0] += cost(tile)

    plan._launch = launch
    return plan, timed


@pytest.mark.parametrize("cap", [0, 3])
@pytest.mark.parametrize("build,integ", [
    (lambda: problems.diffusion_3d_mixed(ns), codegen.RK4),
    (lambda: problems.diffusion_2d(ns, n=16), codegen.FORWARD_EULER),
])
def test_a_cap_leaves_the_walking_kernels_to_the_autotuner(monkeypatch, build, integ, cap):
    """Stage and resident kernels are the fastest, and are timed only without a cap."""
    gen = _gen(build(), integ)
    special = {**gen.stage_kernels, **gen.resident_kernels}
    assert special
    plan, timed = tuning_plan(monkeypatch, gen, lambda tile: 0.1 if tile in special else 0.2, {})
    plan.limit_ctas(cap)
    best = plan.autotune(1e-4)
    assert (best in special) == (cap == 0) and bool(timed & set(special)) == (cap == 0)
    # an operator with a cap does not take the pick of one without, nor the other way round
    plan.limit_ctas(0 if cap else 3)
    assert (plan.autotune(1e-4) in special) == (cap != 0)


class _Node(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("smem", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def _grids(record):
    """CTAs of every kernel launch that ``record()`` makes, from a CUDA graph."""
    import torch

    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        record()
    cu = ctypes.CDLL("libcuda.so.1")
    raw, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t()
    assert cu.cuGraphGetNodes(raw, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert cu.cuGraphGetNodes(raw, nodes, ctypes.byref(count)) == 0
    out = []
    for node in nodes:
        kind = ctypes.c_int()
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value == 0:
            p = _Node()
            assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(p)) == 0
            out.append(p.grid[0] * p.grid[1] * p.grid[2])
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("kind,build,integ,cap", [
    ("stage_kernels", lambda: problems.diffusion_3d_mixed(ns, n=(9, 13, 35)), "RK4", 3),
    ("stage_kernels", lambda: problems.diffusion_3d_mixed(ns, n=(8, 7, 65)), "ForwardEulerMethod", 5),
    ("march_kernels", lambda: problems.mixed_bc_wave_2d(ns, nx=45, ny=77), "RK4", 3),
    ("march_kernels", lambda: problems.cahn_hilliard_2d(ns, n=131, length=32.75), "RK4", 5),
    ("resident_kernels", lambda: problems.dynamic_bc_wave_2d(ns, nx=26, ny=21), "RK4", 3),
    ("resident_kernels", lambda: problems.diffusion_2d(ns, n=20), "ForwardEulerMethod", 40),
])
def test_launches_stay_within_the_cap(kind, build, integ, cap):
    import torch

    ivp = build()
    cp = ivp.constrained_problem
    gen = _gen(ivp, {"RK4": codegen.RK4, "ForwardEulerMethod": codegen.FORWARD_EULER}[integ])
    y0 = ivp.initial_condition.discrete_y_0(True)
    batch = 7
    y = torch.tensor(np.stack([y0 * (1.0 + 0.1 * b) for b in range(batch)]), device="cuda")
    for tile in list(getattr(gen, kind))[:3]:
        got = {}
        for ctas in (0, cap):
            op = fdm.FDMOperator(getattr(fdm, integ)(), fdm.ThreePointCentralDifferenceMethod(), 1e-4, tile=tile,
                                 max_ctas=ctas)
            plan = op.plan(cp, batch)
            state, out = plan.new_state(1), plan.new_state(3)
            plan.pack_device(y, state[0])
            plan.run(state[0], out, 3, 0.0, 1e-4)
            torch.cuda.synchronize()
            grids = _grids(lambda: plan.run(state[0], out, 3, 0.0, 1e-4))
            assert grids and (ctas == 0 or max(grids) <= ctas), (tile, grids)
            plan.check_status()
            got[ctas] = plan.unpack(out, 3 * batch).cpu().numpy()
        assert np.array_equal(got[0], got[cap]), tile


@pytest.mark.gpu
def test_a_cap_below_a_cluster_is_refused():
    ivp = problems.diffusion_2d(ns, n=20)
    op = fdm.FDMOperator(fdm.RK4(), fdm.ThreePointCentralDifferenceMethod(), 1e-4, tile=codegen.RESIDENT_TILE, max_ctas=1)
    with pytest.raises(ValueError, match="max_ctas"):
        op.solve(ivp)

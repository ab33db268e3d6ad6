"""Picks stored by the autotuner are taken only where it would offer them now:
on the same device, under the same rule, and among the kernels that can run."""

import pytest

import pararealml_gb300 as ns
import problems
from pararealml_gb300 import codegen, engine
from test_grid_cap import _gen, tuning_plan


def test_a_stored_resident_kernel_that_cannot_run_is_not_taken(monkeypatch):
    gen = _gen(problems.diffusion_2d(ns, n=16), codegen.FORWARD_EULER)
    resident = set(gen.resident_kernels)
    stored = {}
    plan, timed = tuning_plan(monkeypatch, gen, lambda tile: 0.1 if tile in resident else 0.2, stored)
    assert plan.autotune(1e-4) in resident
    plan, timed = tuning_plan(monkeypatch, gen, lambda tile: 0.2, stored)
    assert plan.autotune(1e-4) in resident and not timed  # the stored pick
    plan, timed = tuning_plan(monkeypatch, gen, lambda tile: 0.2, stored)
    plan.resident_shape = lambda: None  # a driver or device without the clusters
    assert plan.autotune(1e-4) not in resident and timed


@pytest.mark.parametrize("change", ["device", "SMs", "rule"])
def test_a_pick_of_another_device_or_rule_is_not_taken(monkeypatch, change):
    torch = pytest.importorskip("torch")
    gen = _gen(problems.diffusion_2d(ns, n=16), codegen.FORWARD_EULER)
    stored = {}
    plan, _ = tuning_plan(monkeypatch, gen, lambda tile: 0.1, stored)
    plan.autotune(1e-4)
    plan, timed = tuning_plan(monkeypatch, gen, lambda tile: 0.1, stored)
    device = torch.cuda.get_device_properties("cuda")
    if change == "device":
        device.name = "another"
    elif change == "SMs":
        device.multi_processor_count = 148
    else:
        monkeypatch.setattr(engine.StencilPlan, "TUNE_RULE", 1)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda dev: device)
    plan.autotune(1e-4)
    assert timed


def test_the_stored_picks_are_parsed_once_per_change(monkeypatch, tmp_path):
    parses = []
    load = engine.json.load
    monkeypatch.setattr(engine.json, "load", lambda f: (parses.append(1), load(f))[1])
    monkeypatch.setattr(engine._native, "JIT_CACHE_DIR", str(tmp_path))
    assert engine._tune_cache_load() == {} and not parses
    engine._tune_cache_store("a", {"tile": [1]})
    for _ in range(3):
        assert engine._tune_cache_load() == {"a": {"tile": [1]}}
    assert len(parses) == 1
    engine._tune_cache_store("b", {"tile": [2]})
    assert engine._tune_cache_load() == {"a": {"tile": [1]}, "b": {"tile": [2]}} and len(parses) == 2
    (tmp_path / "autotune.json").write_text("not json")
    assert engine._tune_cache_load() == {}

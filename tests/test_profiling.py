"""The profiling hooks are live: ranges around plan / table build / launch show up in a chrome trace."""

import glob
import json
import os

import torch
from torch.distributed.tensor.placement_types import Shard

from etha_b200.comm.planner import plan_m2m
from etha_b200.utils.profiling import ProfilingSpec, maybe_enable_profiling, nvtx_range


def test_chrome_trace_contains_the_named_ranges(tmp_path):
    spec = ProfilingSpec(enable_profiling=True, dump_folder=str(tmp_path), save_traces_folder="traces/plan",
                         profile_freq=3, warmup_steps=1, active_steps=2)
    with maybe_enable_profiling(spec, rank=0) as prof:
        assert prof is not None
        for _ in range(3):
            with nvtx_range("etha.plan"):
                plan_m2m(torch.arange(4), (Shard(0),), torch.arange(4, 8), (Shard(1),))
            prof.step()
    files = glob.glob(os.path.join(str(tmp_path), "traces", "plan", "rank0_step*.json"))
    assert files, "no chrome trace was written"
    names = {e.get("name") for e in json.load(open(files[0]))["traceEvents"]}
    assert "etha.plan" in names


def test_profiling_off_yields_none(tmp_path):
    with maybe_enable_profiling(ProfilingSpec(enable_profiling=False, dump_folder=str(tmp_path))) as prof:
        assert prof is None
    assert not os.listdir(tmp_path)


def test_a_range_decorates_functions():
    """Every call opens a range of its own; calls may nest (the profiler folds those into one)."""
    depth = []

    @nvtx_range("etha.step")
    def step(n):
        depth.append(n)
        return step(n - 1) + n if n else 0

    with torch.profiler.profile() as prof:
        assert [step(0), step(0), step(3)] == [0, 0, 6]
    assert depth == [0, 0, 3, 2, 1, 0]
    assert [e.count for e in prof.key_averages() if e.key == "etha.step"] == [3]


def test_other_observers_see_the_ranges(tmp_path):
    """Not only the autograd profiler listens to record_function."""
    path = str(tmp_path / "trace.json")
    observer = torch.profiler.ExecutionTraceObserver().register_callback(path)
    observer.start()
    with nvtx_range("etha.observed"):
        torch.zeros(1)
    observer.stop()
    with nvtx_range("etha.unobserved"):
        torch.zeros(1)
    observer.unregister_callback()
    names = {n["name"] for n in json.load(open(path))["nodes"]}
    assert "etha.observed" in names and "etha.unobserved" not in names


def test_a_failed_push_does_not_turn_nvtx_off(monkeypatch):
    pushed = []

    def push(name):
        if not pushed:
            pushed.append(None)
            raise RuntimeError("first push fails")
        pushed.append(name)

    monkeypatch.setattr(nvtx_range, "_nvtx", nvtx_range._nvtx)
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch.cuda.nvtx, "range_push", push)
    monkeypatch.setattr(torch.cuda.nvtx, "range_pop", lambda: pushed.pop())
    with nvtx_range("a"):
        assert pushed == [None]
    with nvtx_range("b"):
        assert pushed == [None, "b"]
    assert pushed == [None]

"""Which intake a transpiled network gets: arrival bits where they and what making them holds at once fit half of the
device's free memory, else the scanning form, which a plan of arrival bits carries along (saved and loaded too)."""

import itertools

import numpy as np
import pytest
import torch

from naer2_b200 import _lib, population
from naer2_b200.transpiler import JitRuntime, PlannedNetwork, load_plan, plan_of, save_plan
from naer2_b200.transpiler import runtime as jit_runtime
from naer2_b200.transpiler.runtime import arrival_bytes, arrivals_need, scan_form
from test_arrivals import _exact, _plastic


@pytest.fixture(autouse=True)
def _own_seeds(monkeypatch):
    """Populations made here draw their default seeds from a count of their own."""
    monkeypatch.setattr(population, "_SEEDS", itertools.count(1 << 20))


@pytest.mark.parametrize("make", [_plastic, _exact])
def test_a_plan_carries_the_scanning_form(monkeypatch, tmp_path, make):
    plan = plan_of(make(33, 4)[0])
    save_plan(plan, tmp_path / "plan.npz")
    loaded = scan_form(load_plan(tmp_path / "plan.npz"))
    form = scan_form(plan)
    population._SEEDS = itertools.count(1 << 20)
    monkeypatch.setattr(jit_runtime, "ARRIVAL_BYTES", 0)
    want = plan_of(make(33, 4)[0])
    assert "window" not in form and "window" not in want and "window" not in loaded
    for a, b, c in zip(form["pops"], want["pops"], loaded["pops"]):
        assert {k: v for k, v in a.items() if k != "conns"} == {k: v for k, v in b.items() if k != "conns"}
        assert a["source"] == c["source"] and a["fields"] == c["fields"] and "outs" not in c


def test_the_need_counts_the_tables_and_the_largest_connections_making():
    plan = plan_of(_exact(33, 4)[0])
    sizes = [(p["n"], len(c["link"]), plan["pops"][c["src"]]["depth"]) for p in plan["pops"] for c in p["conns"]]
    assert arrivals_need(plan) == sum(arrival_bytes(*s) for s in sizes) + jit_runtime.BUILD_BYTES * max(s[1] for s in sizes)


@pytest.mark.gpu
@pytest.mark.parametrize("make", [_plastic, _exact])
@pytest.mark.parametrize("through_file", [False, True])
def test_little_free_memory_scans(cuda, monkeypatch, tmp_path, make, through_file):
    def run():
        population._SEEDS = itertools.count(1 << 20)
        net, _ = make(33, 4)
        net.record(50)
        if through_file:
            save_plan(plan_of(net), tmp_path / "plan.npz")
            states = [{a: p.state_tensor(a).clone() for a in p.dynamic_attrs} for p in net.populations]
            net = PlannedNetwork(load_plan(tmp_path / "plan.npz"), states, net.device, record_steps=50)
        net.run_steps(50)
        rt = net.runtime
        assert isinstance(rt, JitRuntime)
        return [rt.raster_words(p) for p in net.populations] + [t.cpu().numpy() for p in net.populations
                                                                for _, t in sorted(p._state.items())], rt

    want, rt = run()
    assert rt.window is not None
    need = arrivals_need(rt.plan)
    monkeypatch.setattr(jit_runtime, "SMALL_BYTES", 0)
    monkeypatch.setattr(_lib, "free_bytes", lambda device: 2 * need)
    _, rt = run()
    assert rt.window is not None
    monkeypatch.setattr(_lib, "free_bytes", lambda device: 2 * need - 2)
    got, rt = run()
    assert rt.window is None and not any("outs" in p for p in rt.plan["pops"])
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.gpu
def test_making_the_bits_holds_what_is_counted(cuda):
    """The peak of arrival_form over a connection's links, against BUILD_BYTES."""
    n, k = 4000, 500
    g = torch.Generator(device=cuda).manual_seed(1)
    ptr = (torch.arange(n + 1, device=cuda) * k).int()
    link = torch.randint(0, 3000, (n * k,), generator=g, device=cuda) | (torch.randint(1, 32, (n * k,), generator=g, device=cuda) << 24)
    link = link.int()
    jit_runtime.arrival_form(ptr, link, 3000, 31)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats(cuda)
    before = torch.cuda.memory_allocated(cuda)
    f = jit_runtime.arrival_form(ptr, link, 3000, 31)
    peak = torch.cuda.max_memory_allocated(cuda) - before
    assert f["bad"] == 0 and peak <= jit_runtime.BUILD_BYTES * n * k

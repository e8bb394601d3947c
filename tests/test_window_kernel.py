"""The window kernel's source: one copy of the step's code for the populations that run the same text, no sizes in it
(networks that differ in their sizes alone share a compiled kernel), none at all where its code would take in more
connections than WINDOW_INTAKES. On the GPU, networks of several kinds of populations and several of each give the
scanning intake's results bit for bit."""

import itertools
import re
import subprocess

import numpy as np
import pytest
import torch

from naer2_b200 import population
from naer2_b200.build import ARCH, nvcc
from naer2_b200.patterns import fixed_indegree
from naer2_b200.transpiler import JitRuntime, plan_of
from naer2_b200.transpiler import runtime as jit_runtime
from tests.dsl_models import PairSTDP, Pacemaker, Syn, TraceLIF


@pytest.fixture(autouse=True)
def _own_seeds(monkeypatch):
    """Populations made here draw their default seeds from a count of their own."""
    monkeypatch.setattr(population, "_SEEDS", itertools.count(1 << 20))


def _net(sizes, thetas, edge=Syn, k=3, sources=0):
    """Every population of TraceLIF connected to every one; `sources` Pacemakers connected to each."""
    g = torch.Generator().manual_seed(len(sizes))
    pops = [TraceLIF(theta=th) * n for n, th in zip(sizes, thetas)]
    fibres = [Pacemaker(period=3 + i) * (20 + i) for i in range(sources)]
    for i, p in enumerate(pops + fibres):
        p.seed = 1 + i
    for s, t in itertools.product(fibres + pops, pops):
        c = s >> edge() @ fixed_indegree(k, seed=1) >> t
        c.weight = 0.1 + 0.5 * torch.rand(c.shape, generator=g)
        c.delay = (torch.randint(1, 5, c.shape, generator=g) * 0.1).double()
    net = pops[0].network
    net.resolution = 0.1
    return net


def _copies(plan):
    return len(re.findall(r"^namespace n2p\d+ \{", plan["window"]["source"], re.M))


def test_networks_of_other_sizes_share_the_kernel():
    a, b = plan_of(_net((100, 37), (1.0, 1.0))), plan_of(_net((900, 1), (1.0, 1.0)))
    assert a["window"]["source"] == b["window"]["source"] and _copies(a) == 1
    assert a["window"]["order"] == [0, 1] and a["window"]["counts"] == [2]


def test_populations_of_one_text_share_its_code():
    plan = plan_of(_net((40, 50, 60, 70), (1.0, 2.0, 1.0, 1.0)))
    assert _copies(plan) == 2
    assert plan["window"]["order"] == [0, 2, 3, 1] and plan["window"]["counts"] == [3, 1]
    # 8 connections into each: one text of them is within WINDOW_INTAKES, two are not
    assert _copies(plan_of(_net((40,) * 8, (1.0,) * 8))) == 1
    assert "window" not in plan_of(_net((40,) * 8, (1.0,) * 7 + (2.0,)))


def _run(make, edge, steps):
    net = make()
    net.record(steps)
    for part in (1, 20, steps - 21):
        net.run_steps(part)
    rt = net.runtime
    assert isinstance(rt, JitRuntime)
    out = [rt.raster_words(p) for p in net.populations]
    out += [t.cpu().numpy() for p in net.populations for _, t in sorted(p._state.items())]
    out += [np.array(sorted(rt.counters().items(), key=str), dtype=object), np.array(rt.status())]
    if edge is PairSTDP:
        out += [rt.edge_state(c, "weight").cpu().numpy() for c in net.connections]
    return out, rt


@pytest.mark.gpu
@pytest.mark.parametrize("sizes, thetas, edge, sources", [
    ((33, 64, 1), (0.4, 0.4, 0.4), Syn, 1), ((40, 31, 65, 7), (0.4, 0.6, 0.4, 0.6), Syn, 0),
    ((90, 33, 40), (0.5, 0.5, 0.7), PairSTDP, 1), ((50,) * 7, (0.4,) * 7, Syn, 1)])
def test_populations_that_share_code_match_the_scanning_intake(cuda, monkeypatch, sizes, thetas, edge, sources):
    def make():
        net = _net(sizes, thetas, edge, sources=sources)
        for i, p in enumerate(net.populations):
            if "v" in p.dynamic_attrs:
                p.v = 0.9 * torch.rand(len(p.shape), generator=torch.Generator().manual_seed(i))
        return net

    got, rt = _run(make, edge, 60)
    assert (rt.window is not None) == ("window" in rt.plan)
    monkeypatch.setattr(jit_runtime, "ARRIVAL_BYTES", 0)
    want, rt = _run(make, edge, 60)
    assert rt.window is None
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert sum(int(np.unpackbits(w.view(np.uint8)).sum()) for w in want[:len(sizes)]) > 50


@pytest.mark.parametrize("pops, per", [(4, 4500), (8, 2300), (8, 1700)])
def test_full_networks_spill_no_registers(tmp_path, pops, per):
    """At three and four blocks per SM, with as many connections as a window kernel takes in."""
    plan = plan_of(_net((per,) * pops, (1.0,) * pops, k=1))
    src = tmp_path / "window.cu"
    src.write_text(plan["window"]["source"])
    out = subprocess.run([nvcc(), *ARCH, "-std=c++17", "--fmad=false", "-Xptxas", "-v", "-cubin", "-o",
                          str(tmp_path / "window.cubin"), str(src)], capture_output=True, text=True, check=True)
    assert "0 bytes spill stores, 0 bytes spill loads" in out.stderr, out.stderr

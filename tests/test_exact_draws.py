"""Random draws of an exact-time network over arrival bits are keyed as the scanning intake keys them (the send hook is
lowered twice there: after each group of arrivals, then at the step's end): the call sites in the generated source on the
CPU, rasters and state bit for bit on the GPU, of populations with and without incoming connections."""

import itertools
import random
import re

import numpy as np
import pytest
import torch

import naer2_b200 as n2
from naer2_b200 import population, receives as r
from naer2_b200.patterns import fixed_indegree
from naer2_b200.transpiler import JitRuntime, plan_of
from naer2_b200.transpiler import runtime as jit_runtime
from tests.dsl_models import DecayLIF, Syn


@pytest.fixture(autouse=True)
def _own_seeds(monkeypatch):
    """Populations made here draw their default seeds from a count of their own."""
    monkeypatch.setattr(population, "_SEEDS", itertools.count(1 << 20))


@n2.node
class RandomFibre:
    """Fires by its own draw, at a drawn time inside the step; counts what it receives."""

    def __init__(self, p: float = 0.08):
        self.p = p
        self.got: float = 0.0

    def update(self, time: n2.time):
        self.got = self.got * 0.5

    def send(self, time: n2.time):
        if random.random() < self.p:
            n2.spike(time - 0.1 * random.random())

    def receive(self, time: n2.time, edge: r.edge, source: r.source):
        self.got += edge.weight


def _net(feedback):
    g = torch.Generator().manual_seed(3)
    src, tgt = RandomFibre() * 50, DecayLIF(theta=0.5, tau=3.0, t_ref=0.25) * 40
    src.seed, tgt.seed = 1, 2
    pairs = [(src, tgt, 12)] + ([(tgt, src, 4)] if feedback else [])
    for s, t, k in pairs:
        c = s >> Syn() @ fixed_indegree(k, seed=12) >> t
        c.weight = 0.1 + 0.3 * torch.rand(c.shape, generator=g)
        c.delay = (torch.randint(1, 5, c.shape, generator=g) * 0.1).double()
    net = src.network
    net.resolution = 0.1
    net.exact = True
    return net


@pytest.mark.parametrize("feedback", [False, True])
def test_call_sites_are_the_scanning_intakes(monkeypatch, feedback):
    def sites():
        return [[int(x) for x in re.findall(r"n2_uniform\(p, j, n, (\d+)u", p["source"])] for p in plan_of(_net(feedback))["pops"]]

    got = sites()
    monkeypatch.setattr(jit_runtime, "ARRIVAL_BYTES", 0)
    want = sites()
    for a, b in zip(got, want):
        assert a[-2:] == b[-2:]  # the step's own send
        assert not feedback or a == b


@pytest.mark.gpu
@pytest.mark.parametrize("feedback", [False, True])
def test_draws_give_the_scanning_intakes_spikes(cuda, monkeypatch, feedback):
    def run():
        net = _net(feedback)
        net.record(60)
        for part in (1, 20, 39):
            net.run_steps(part)
        rt = net.runtime
        assert isinstance(rt, JitRuntime)
        out = [rt.raster_words(p) for p in net.populations] + [rt.spike_times(p)[0] for p in net.populations]
        return out + [t.cpu().numpy() for p in net.populations for _, t in sorted(p._state.items())], rt

    got, rt = run()
    assert rt.window is not None
    monkeypatch.setattr(jit_runtime, "WINDOW_BLOCKS", 0)
    steps, _ = run()
    monkeypatch.setattr(jit_runtime, "ARRIVAL_BYTES", 0)
    want, _ = run()
    for a, b, c in zip(got, steps, want):
        assert np.array_equal(a, c) and np.array_equal(b, c)
    assert all(int(np.unpackbits(w.view(np.uint8)).sum()) > 20 for w in want[:2])

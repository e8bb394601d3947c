"""The generated arrival kernels' branches on size, against the scanning intake, bit for bit: connections whose rows and
words are not held ahead, outgoing connections past the cached row bounds, links with their delays in an array of their
own, more edge attributes than are loaded ahead of the hooks; as a window and as launches per population."""

import itertools

import numpy as np
import pytest
import torch

import naer2_b200 as n2
from naer2_b200 import population, receives as r
from naer2_b200.patterns import fixed_indegree
from naer2_b200.transpiler import JitRuntime, arrival
from naer2_b200.transpiler import runtime as jit_runtime
from tests.dsl_models import DecayLIF, JitterPacemaker, Pacemaker, PairSTDP, Syn, TraceLIF

pytestmark = pytest.mark.gpu


@n2.edge
class Wide:
    """A link of ten values, all of them its own."""

    def __init__(self, weight: float = 0.1):
        self.weight = weight
        self.a, self.b, self.c, self.d, self.e, self.f, self.g, self.h, self.i = 0.1, 0.2, 0.3, 0.4, 0.5, 0.6, 0.7, 0.8, 0.9

    def forward(self, time: n2.time, dst: r.destination):
        self.a = self.a * 0.9 + self.i
        self.b = self.b * 0.8 + self.a
        self.c = self.c * 0.7 + self.b
        self.d = self.d * 0.6 + self.c
        self.e = self.e * 0.5 + self.d
        self.f = self.f * 0.4 + self.e
        self.g = self.g * 0.3 + self.f
        self.h = self.h * 0.2 + self.g
        self.i = self.i * 0.1 + 0.01 * self.h
        self.weight = min(self.weight + 0.001 * self.i, 0.5)

    def backward(self):
        pass


@pytest.fixture(autouse=True)
def _own_seeds(monkeypatch):
    """Populations made here draw their default seeds from a count of their own."""
    monkeypatch.setattr(population, "_SEEDS", itertools.count(1 << 20))


def _net(exact, edge, sources, hub):
    """`sources` input populations into one target, which sends to itself and to `hub` more populations."""
    g = torch.Generator().manual_seed(sources + hub)
    fibre, cell = (JitterPacemaker, DecayLIF) if exact else (Pacemaker, TraceLIF)
    pops = [fibre(period=3 + i % 4) * (30 + i) for i in range(sources)]
    tgt = cell(theta=0.8) * 70
    more = [cell(theta=0.9) * (10 + i) for i in range(hub)]
    for i, p in enumerate(pops + [tgt] + more):
        p.seed = 1 + i
    for i, (s, t) in enumerate([(p, tgt) for p in pops] + [(tgt, tgt)] + [(tgt, m) for m in more]):
        c = s >> edge() @ fixed_indegree(2 + i % 5 * 20 if t is tgt else 9, seed=i) >> t
        c.weight = 0.05 + 0.2 * torch.rand(c.shape, generator=g)
        c.delay = (torch.randint(1, 6, c.shape, generator=g) * 0.1).double()
    for p in pops:
        p.phase = torch.randint(0, 3, (len(p.shape),), generator=g, dtype=torch.int32)
        if exact:
            p.jitter = (0.1 * torch.rand(len(p.shape), generator=g)).float()
    net = tgt.network
    net.resolution = 0.1
    net.exact = exact
    return net


def _run(exact, edge, sources, hub):
    population._SEEDS = itertools.count(1 << 20)
    net = _net(exact, edge, sources, hub)
    net.record(50)
    for part in (1, 20, 29):
        net.run_steps(part)
    rt = net.runtime
    assert isinstance(rt, JitRuntime)
    out = [rt.raster_words(p) for p in net.populations]
    out += [t.cpu().numpy() for p in net.populations for _, t in sorted(p._state.items())]
    out += [rt.edge_state(c, a).cpu().numpy() for c in net.connections for a in ("weight", "i", "x_pre")
            if (id(c), a) in rt.edge_arrays]
    return out + [np.array(sorted(rt.counters().items(), key=str), dtype=object), np.array(rt.status())], rt


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("edge, sources, hub, ahead, packed", [
    (Syn, 10, 10, (8, 4), 1 << 24), (PairSTDP, 4, 9, (2, 2), 1 << 24), (Syn, 3, 1, (2, 1), 0), (Wide, 2, 0, (8, 4), 0),
    (Wide, 5, 1, (0, 0), 1 << 24)])
def test_size_branches_match_the_scanning_intake(cuda, monkeypatch, exact, edge, sources, hub, ahead, packed):
    if exact and edge is PairSTDP:
        edge = Syn  # (its hooks read the clocked neuron's trace)
    monkeypatch.setattr(arrival, "AHEAD", ahead)
    monkeypatch.setattr(arrival, "WINDOW_INTAKES", 64)
    monkeypatch.setattr(arrival, "WINDOW_POPS", 64)
    monkeypatch.setattr(jit_runtime, "PACKED_BITS", packed)
    got, rt = _run(exact, edge, sources, hub)
    assert rt.window is not None
    monkeypatch.setattr(jit_runtime, "WINDOW_BLOCKS", 0)
    steps, rt = _run(exact, edge, sources, hub)
    assert rt.window is None and any("outs" in p for p in rt.plan["pops"])
    monkeypatch.setattr(jit_runtime, "ARRIVAL_BYTES", 0)
    want, rt = _run(exact, edge, sources, hub)
    assert not any("outs" in p for p in rt.plan["pops"])
    assert len(got) == len(want)
    for a, b, c in zip(got, steps, want):
        assert np.array_equal(a, c) and np.array_equal(b, c)
    assert sum(int(np.unpackbits(w.view(np.uint8)).sum()) for w in want[sources:sources + 1 + hub]) > 20

"""A transpiled network's steps captured into a CUDA graph: a graph replayed, replayed again at once, and followed by
eager steps gives, bit for bit, what the launches of one population and step at a time give in the same order. (The
window kernel's barrier starts each launch from nothing, so no launch counts on what the host did before it.)"""

import itertools

import numpy as np
import pytest
import torch

from naer2_b200 import population
from naer2_b200.patterns import fixed_indegree
from naer2_b200.transpiler import runtime as jit_runtime
from tests.dsl_models import PairSTDP, Pacemaker, TraceLIF

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _own_seeds(monkeypatch):
    """Populations made here draw their default seeds from a count of their own."""
    monkeypatch.setattr(population, "_SEEDS", itertools.count(1 << 20))


def _run(replays):
    g = torch.Generator().manual_seed(5)
    src, tgt = Pacemaker(period=3) * 300, TraceLIF(theta=1.2) * 700
    src.seed, tgt.seed = 1, 2
    c = src >> PairSTDP() @ fixed_indegree(40, seed=10) >> tgt
    c.weight = 0.2 + 0.6 * torch.rand(c.shape, generator=g)
    c.delay = (torch.randint(1, 6, c.shape, generator=g) * 0.1).double()
    src.phase = torch.randint(0, 3, (300,), generator=g, dtype=torch.int32)
    net = src.network
    net.resolution = 0.1
    net.record(60)
    net.run_steps(10)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        net.run_steps(7)
    for _ in range(replays):
        graph.replay()
    net.run_steps(1)
    net.run_steps(12)
    torch.cuda.synchronize()
    rt = net.runtime
    net.check()
    out = [rt.raster_words(p) for p in net.populations]
    out += [t.cpu().numpy() for p in net.populations for _, t in sorted(p._state.items())]
    out += [rt.edge_state(c, a).cpu().numpy() for a in ("weight", "x_pre", "t_last")]
    return out, rt, graph


@pytest.mark.parametrize("replays", [1, 3])
def test_captured_steps_replay(cuda, monkeypatch, replays):
    got, rt, _ = _run(replays)
    assert rt.window is not None
    monkeypatch.setattr(jit_runtime, "WINDOW_BLOCKS", 0)
    want, rt, _ = _run(replays)
    assert rt.window is None
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert sum(int(np.unpackbits(w.view(np.uint8)).sum()) for w in got[:2]) > 100


def test_long_runs_are_several_launches(cuda, monkeypatch):
    def run(net_steps):
        population._SEEDS = itertools.count(1 << 20)
        src, tgt = Pacemaker(period=7) * 50, TraceLIF(theta=1.2) * 60
        src.seed, tgt.seed = 1, 2
        c = src >> PairSTDP() @ fixed_indegree(12, seed=10) >> tgt
        c.weight, c.delay = 0.2, 0.3
        net = src.network
        net.resolution = 0.1
        for n in net_steps:
            net.run_steps(n)
        rt = net.runtime
        return [t.cpu().numpy() for p in net.populations for _, t in sorted(p._state.items())] + [
            rt.edge_state(c, "weight").cpu().numpy(), np.array(rt.counters()["events"])], rt

    got, rt = run([2100])
    assert rt.window is not None and rt.launches == 3
    want, _ = run([700] * 3)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert int(want[-1]) > 1000

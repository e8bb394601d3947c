"""Which networks run their steps in chunks (csrc/naer2b.cu, chunk_steps) and how that is chosen: Network.steps_per_barrier
and Network.block, the slots kept for it, the tuner's candidates. Every choice gives the oracle's rasters and state."""

import itertools

import pytest
import torch

from naer2_b200 import population
from naer2_b200.models import LIF, Poisson_source
from naer2_b200.networks import brunel
from naer2_b200.patterns import fixed_indegree
from naer2_b200.runtime import lookahead
from naer2_b200.tune import autotune
from test_chunks_gpu import _net
from test_parity_gpu import assert_identical, run_both

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _own_seeds(monkeypatch):
    """Populations made here draw their default seeds from a count of their own."""
    monkeypatch.setattr(population, "_SEEDS", itertools.count(1 << 20))


def _same(net, steps=90, persistent=True):
    gr, orr, gs, os_, cnt, ev = run_both(net, steps, chunk=41, persistent=persistent)
    assert sum(int(r.sum()) for r in gr) > 0
    assert_identical(gr, orr, gs, os_)
    assert cnt["events"] == ev


@pytest.mark.parametrize("spb, block", [(None, None), (1, None), (2, 64), (3, 256), (5, 128), (40, 64)])
def test_every_choice_gives_the_oracles_results(cuda, spb, block):
    net = _net(900, 7, 12, seed=3)
    net.steps_per_barrier, net.block = spb, block
    _same(net)
    rt = net.runtime
    assert lookahead(net, rt.desc) == (7 if spb is None else min(spb, 7))
    # 12 steps of delay in 16 slots; up to 32 with the steps between two barriers
    assert {rt.cpop[k].acc_depth for k in (1, 2)} == ({16} if spb in (1, 2, 3) else {32})
    net.close()


@pytest.mark.parametrize("change", ["per step", "many connections", "rows"])
def test_slots_are_kept_for_chunks_alone(cuda, change):
    net = _net(300, 2 if change == "rows" else 15, 15, seed=3)
    if change == "many connections":
        a = net.populations[1]
        for i in range(60):
            c = a >> fixed_indegree(2, seed=i) >> a
            c.weight, c.delay = 0.01, 1.5
    if change == "rows":  # two steps between barriers, 1,300 links per neuron: past the rule's line
        a = net.populations[1]
        c = a >> fixed_indegree(2400, seed=1) >> a
        c.weight, c.delay = 0.0005, 0.2
    _same(net, persistent=change != "per step")
    rt = net.runtime
    assert lookahead(net, rt.desc) == 1 and {rt.cpop[k].acc_depth for k in (1, 2)} == {16}
    net.close()


def test_more_outgoing_connections_than_are_walked_together(cuda):
    """A population of 11 outgoing connections: its rows past the eighth are looked up in the tables, in chunks too."""
    g = torch.Generator().manual_seed(5)
    src = Poisson_source(rate=200.0) * 50
    src.seed = 1
    for i in range(11):
        t = LIF(tau=20.0, theta=20.0, V_r=10.0, t_ref=2.0, ext_rate=20.0, ext_weight=0.1) * (40 + i)
        t.seed = 2 + i
        t.V = 20.0 * torch.rand(40 + i, generator=g)
        c = src >> fixed_indegree(6, seed=i) >> t
        c.weight = 0.4 * torch.rand(c.shape, generator=g)
        c.delay = (torch.randint(5, 9, c.shape, generator=g) * 0.1).double()
    net = src.network
    net.resolution = 0.1
    _same(net)
    assert lookahead(net, net.runtime.desc) == 5
    net.close()


def test_the_tuner_tries_the_barrier_per_step(cuda):
    net, _ = brunel.build(**brunel.CONFIG0, seed=4)
    report = autotune(net, steps=100, warmup=20)
    tried = {(t["block"], t.get("steps_per_barrier")) for t in report["trials"]}
    assert {(None, None), (128, 1), (256, 1), (128, None), (256, None)} <= tried
    best = min(t["us_per_step"] for t in report["trials"])
    assert report["chosen"]["us_per_step"] == best
    assert (net.block, net.steps_per_barrier) == (report["chosen"]["block"], report["chosen"]["steps_per_barrier"])
    _same(net, 120)
    net.close()

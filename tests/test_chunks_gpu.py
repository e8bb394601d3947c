"""Networks whose every link has a delay of several steps run those steps without a grid barrier between them
(csrc/n2b_device.cuh, chunk_kernel): rasters and state must be the oracle's bit for bit for chunks of 2 steps and of
the most a chunk holds, delays that spread past the smallest, windows that cut chunks short, tiles of every width,
fewer blocks than tiles, sources that fire densely, both neuron models, weights per link and shared."""

import itertools

import numpy as np
import pytest
import torch

from naer2_b200 import population
from naer2_b200.models import LIF, PD14_neuron, Poisson_source
from naer2_b200.patterns import fixed_indegree, fixed_outdegree
from naer2_b200.runtime import describe
from test_parity_gpu import assert_identical, run_both

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _own_seeds(monkeypatch):
    """Populations made here draw their default seeds from a count of their own."""
    monkeypatch.setattr(population, "_SEEDS", itertools.count(1 << 20))


def _net(n, lo, hi, seed, rate=1.0):
    """Sources, LIF and PD14 neurons with delays of lo..hi steps on every link."""
    g = torch.Generator().manual_seed(seed)
    src = Poisson_source(rate=rate) * max(1, n // 3)
    a = LIF(tau=20.0, theta=20.0, V_r=10.0, t_ref=2.0, ext_rate=20.0, ext_weight=0.1) * n
    b = PD14_neuron(K_cortical=1600) * max(1, n // 2 + 1)
    src.seed, a.seed, b.seed = 1, 2, 3
    a.V = 20.0 * torch.rand(n, generator=g)
    b.potential = -65.0 + 15.0 * torch.rand(len(b), generator=g)
    k = 0
    for s, t, w in ((src, a, 0.4), (src, b, 0.2), (a, a, 0.3), (a, b, 0.1), (b, a, -0.5), (b, b, -0.2)):
        k += 1
        c = s >> (fixed_indegree(5, seed=k) if k % 2 else fixed_outdegree(k=4, seed=k)) >> t
        c.weight = w if k % 3 else w * (0.5 + torch.rand(c.shape, generator=g))
        c.delay = (torch.randint(lo, hi + 1, c.shape, generator=g) * 0.1).double()
    net = src.network
    net.resolution = 0.1
    return net


@pytest.mark.parametrize("n, lo, hi, grid, window", [
    (1, 2, 2, None, 100), (33, 2, 9, None, 7), (300, 3, 3, None, 100), (300, 15, 15, 2, 50), (1000, 15, 31, None, 100),
    (700, 40, 60, None, 33), (2500, 7, 20, 5, 100), (5200, 15, 15, None, 100), (11000, 15, 15, None, 100),
    (44000, 4, 5, None, 100)])
def test_chunks_of_steps_match_the_oracle(cuda, n, lo, hi, grid, window):
    net = _net(n, lo, hi, seed=n)
    net.grid, net.window = grid, window
    d = describe(net)
    assert d.lookahead == min(lo, 32)
    steps = 150 if n < 20000 else 60
    gr, orr, gs, os_, cnt, ev = run_both(net, steps, chunk=41)
    assert sum(int(r.sum()) for r in gr[1:]) > 0 or n == 1
    assert_identical(gr, orr, gs, os_)
    assert cnt["events"] == ev and cnt["spikes"] == sum(int(r.sum()) for r in gr)
    net.close()


def test_a_source_that_fires_at_every_step(cuda):
    """Every source neuron in every step: a chunk's spike list is full."""
    net = _net(400, 32, 33, seed=5, rate=1e4)
    gr, orr, gs, os_, cnt, ev = run_both(net, 130)
    assert gr[0].all()
    assert_identical(gr, orr, gs, os_)
    assert cnt["events"] == ev

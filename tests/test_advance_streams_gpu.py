"""n2b_advance orders a network's steps with the stream they are asked for on: after what is already there, before what
comes next, on any stream and from several threads, each call whole."""

import itertools
import threading

import pytest
import torch

from naer2_b200 import population
from naer2_b200.networks import brunel

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _own_seeds(monkeypatch):
    """Populations made here draw their default seeds from a count of their own."""
    monkeypatch.setattr(population, "_SEEDS", itertools.count(1 << 20))


def _net(delay):
    net, pops = brunel.build(**dict(brunel.CONFIG0, delay=delay), seed=4)
    net.window = 20
    net.runtime
    torch.cuda.synchronize()
    return net, pops


@pytest.mark.parametrize("delay", [1.5, "uniform"])
def test_steps_on_a_users_stream(cuda, delay):
    """The state is written on the stream behind a long wait, just before the steps, and read just after them."""
    out = []
    for busy in (False, True):
        net, pops = _net(delay)
        stream = torch.cuda.Stream(cuda)
        with torch.cuda.stream(stream):
            V = pops["E"].state_tensor("V")
            for n in (1, 20, 47):
                if busy:
                    torch.cuda._sleep(20_000_000)
                V.mul_(0.5).add_(7.0)
                net.run_steps(n)
                out.append(V.clone())
                if not busy:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        net.close()
    for a, b in zip(out[:3], out[3:]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("delay", [1.5, "uniform"])
def test_steps_from_two_threads(cuda, delay):
    """Two threads on streams of their own advance one network: all the steps are made, each once."""
    net, pops = _net(delay)
    rt = net.runtime

    def work(n):
        with torch.cuda.stream(torch.cuda.Stream(cuda)):
            for _ in range(60):
                rt.advance(n)

    threads = [threading.Thread(target=work, args=(n,)) for n in (1, 23)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    got, counts = {k: p.state_tensor("V").clone() for k, p in pops.items()}, net.counters()
    net.close()
    net, pops = _net(delay)
    net.run_steps(60 * 24)
    torch.cuda.synchronize()
    assert counts == net.counters()
    for k, p in pops.items():
        assert torch.equal(got[k], p.state_tensor("V"))
    net.close()

"""The transpiled intake over arrival bits: its tables on the CPU (every link in one outgoing row, its bit its own),
and on the GPU against the form that looks every link's source up (`ARRIVAL_BYTES` = 0), whose results it must
give bit for bit: rows below, at and past a word's 32 links, more arrivals in one step than a thread's list or a
neuron's event queue holds, plastic edges, exact times, and plans saved and loaded."""

import itertools

import numpy as np
import pytest
import torch

from naer2_b200 import population
from naer2_b200.patterns import fixed_indegree
from naer2_b200.transpiler import JitRuntime, PlannedNetwork, load_plan, plan_of, save_plan
from naer2_b200.transpiler import runtime as jit_runtime
from naer2_b200.transpiler.runtime import arrival_bytes, arrival_form
from tests.dsl_models import DecayLIF, JitterPacemaker, PairSTDP, Pacemaker, Syn, TraceLIF


@pytest.fixture(autouse=True)
def _own_seeds(monkeypatch):
    """Populations made here draw their default seeds from a count of their own."""
    monkeypatch.setattr(population, "_SEEDS", itertools.count(1 << 20))


@pytest.mark.parametrize("n_src, n_tgt, longest, mask, bad", [(1, 1, 1, 1, 0), (7, 5, 0, 3, 0), (40, 30, 31, 15, 0),
                                                              (40, 30, 65, 31, 3), (300, 9, 700, 255, 0)])
def test_arrival_form_gives_every_link_a_bit_of_its_own(n_src, n_tgt, longest, mask, bad):
    g = np.random.default_rng(n_src + longest)
    lens = g.integers(0, longest + 1, n_tgt)
    ptr = np.concatenate([[0], np.cumsum(lens)])
    n = int(ptr[-1])
    src, dly = g.integers(0, n_src, n), g.integers(1, mask + 1, n)
    if bad:  # a delay of 0, a delay past the ring, a source past the population
        dly[0], dly[1], src[2] = 0, mask + 1, n_src
    link = torch.from_numpy(((dly << 24) | src).astype(np.uint32).view(np.int32).copy())
    f = arrival_form(torch.from_numpy(ptr.astype(np.int32)), link, n_src, mask)
    wptr = f["wptr"].numpy()
    assert np.array_equal(np.diff(wptr), (lens + 31) // 32) and f["words"] == wptr[-1] and f["bad"] == bad
    row = np.repeat(np.arange(n_tgt), lens)
    pos = 32 * wptr[row] + (np.arange(n) - ptr[row])
    good = np.ones(n, bool)
    good[:bad] = False
    out_src = np.repeat(np.arange(n_src), np.diff(f["out_ptr"].numpy()))
    got_pos = f["pos"].numpy().view(np.uint32).astype(np.int64)
    got_dly = got_pos >> 24 if f["dly"] is None else f["dly"].numpy()  # at most 2^24 bits to a slot: packed
    got = list(zip(out_src, got_dly, got_pos & 0xFFFFFF if f["dly"] is None else got_pos))
    assert sorted(got) == sorted(zip(src[good], dly[good], pos[good]))
    top = int(dly[good].max()) if good.any() else 1
    assert f["depth"] == top + 1
    assert 4 * f["depth"] * f["words"] + 5 * n <= arrival_bytes(n_tgt, n, mask + 1)


def _plastic(k, period):
    g = torch.Generator().manual_seed(k)
    src, tgt = Pacemaker(period=period) * 45, TraceLIF(theta=0.4 * k / period + 0.5) * 37
    src.seed, tgt.seed = 1, 2
    c = src >> PairSTDP() @ fixed_indegree(k, seed=10) >> tgt
    c.weight = 0.2 + 0.6 * torch.rand(c.shape, generator=g)
    c.delay = (torch.randint(1, 4, c.shape, generator=g) * 0.1).double()
    src.phase = torch.randint(0, period, (45,), generator=g, dtype=torch.int32)
    net = src.network
    net.resolution = 0.1
    return net, c


def _exact(k, period):
    g = torch.Generator().manual_seed(k)
    src, tgt = JitterPacemaker(period=period) * 60, DecayLIF(theta=0.2 * k / period + 0.3, tau=3.0, t_ref=0.25) * 50
    src.seed, tgt.seed = 1, 2
    for s, kk in ((src, k), (tgt, 3)):
        c = s >> Syn() @ fixed_indegree(kk, seed=12) >> tgt
        c.weight = 0.1 + 0.3 * torch.rand(c.shape, generator=g)
        c.delay = (torch.randint(1, 5, c.shape, generator=g) * 0.1).double()
    src.phase = torch.randint(0, period, (60,), generator=g, dtype=torch.int32)
    src.jitter = (0.1 * torch.rand(60, generator=g)).float()
    net = src.network
    net.resolution = 0.1
    net.exact = True
    return net, None


def _run(make, k, period, steps, through_file=None):
    net, edge = make(k, period)
    net.record(steps)
    if through_file is not None:
        plan = plan_of(net)
        save_plan(plan, through_file)
        states = [{a: p.state_tensor(a).clone() for a in p.dynamic_attrs} for p in net.populations]
        net = PlannedNetwork(load_plan(through_file), states, net.device, record_steps=steps)
    for part in (1, steps // 3, steps - 1 - steps // 3):  # windows of several lengths
        net.run_steps(part)
    rt = net.runtime
    assert isinstance(rt, JitRuntime)
    out = [rt.raster_words(p) for p in net.populations]
    out += [t.cpu().numpy() for p in net.populations for _, t in sorted(p._state.items())]
    out += [rt.spike_times(p)[0] for p in net.populations]
    out += [np.array(sum(rt.status())), np.array(sorted(rt.counters().items(), key=str), dtype=object)]
    if edge is not None and through_file is None:
        out += [rt.edge_state(edge, a).cpu().numpy() for a in ("weight", "x_pre", "t_last")]
    return out, rt


@pytest.mark.gpu
@pytest.mark.parametrize("make, k, period", [(_plastic, 1, 3), (_plastic, 31, 4), (_plastic, 32, 1), (_plastic, 33, 1),
                                             (_plastic, 300, 1), (_plastic, 300, 9), (_exact, 5, 4), (_exact, 33, 4),
                                             (_exact, 90, 1)])
def test_arrival_bits_give_the_scanning_intake_bit_for_bit(cuda, monkeypatch, tmp_path, make, k, period):
    got, rt = _run(make, k, period, 61)
    assert all("outs" in p for p in rt.plan["pops"])
    assert rt.window is not None  # a window of steps per launch
    loaded, _ = _run(make, k, period, 61, through_file=tmp_path / "plan.npz")
    monkeypatch.setattr(jit_runtime, "WINDOW_BLOCKS", 0)
    steps, rt = _run(make, k, period, 61)
    assert rt.window is None and all("outs" in p for p in rt.plan["pops"])  # one launch per population and step
    monkeypatch.setattr(jit_runtime, "ARRIVAL_BYTES", 0)
    want, rt = _run(make, k, period, 61)
    assert not any("outs" in p for p in rt.plan["pops"])
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and np.array_equal(a, b)
    for a, b in zip(steps, want):
        assert a.dtype == b.dtype and np.array_equal(a, b)
    for a, b in zip(loaded, want):
        assert np.array_equal(a, b)
    assert sum(int(np.unpackbits(w.view(np.uint8)).sum()) for w in want[:2]) > 50


@pytest.mark.gpu
def test_a_window_whose_barrier_gives_up_reports_it(cuda):
    """A 1 ns limit makes a block's wait give up while every block still arrives: check() raises, later windows do
    not run, and reset_counters clears the stop."""
    net, _ = _plastic(33, 1)
    net.barrier_limit_ns = 1
    net.run_steps(200)
    assert net.runtime.window is not None
    with pytest.raises(RuntimeError, match="grid barrier"):
        net.check()
    net.runtime.reset_counters()
    net.barrier_limit_ns = 0
    net.run_steps(20)
    net.check()

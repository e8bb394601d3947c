"""A transpiled network whose window kernel does not compile steps by one launch per population, one whose arrival kernels
do not, or whose parameters do not fit a kernel, looks its links' sources up: the same results, bit for bit."""

import itertools

import numpy as np
import pytest
import torch

from naer2_b200 import population
from naer2_b200.patterns import fixed_indegree
from naer2_b200.transpiler import JitRuntime
from naer2_b200.transpiler import runtime as jit_runtime
from tests.dsl_models import Pacemaker, Syn, TraceLIF
from test_arrivals import _exact, _plastic

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _own_seeds(monkeypatch):
    """Populations made here draw their default seeds from a count of their own."""
    monkeypatch.setattr(population, "_SEEDS", itertools.count(1 << 20))


def _run(make):
    population._SEEDS = itertools.count(1 << 20)
    net, edge = make(33, 4)
    net.record(50)
    net.run_steps(50)
    rt = net.runtime
    assert isinstance(rt, JitRuntime)
    out = [rt.raster_words(p) for p in net.populations]
    out += [t.cpu().numpy() for p in net.populations for _, t in sorted(p._state.items())]
    return out + ([] if edge is None else [rt.edge_state(edge, "weight").cpu().numpy()]), rt


@pytest.mark.parametrize("make", [_plastic, _exact])
@pytest.mark.parametrize("refused", ["window", "arrivals", "parameters"])
def test_what_does_not_compile_is_stepped_another_way(cuda, monkeypatch, make, refused):
    want, rt = _run(make)
    assert rt.window is not None
    compiled = jit_runtime.compile_source

    def compile_source(source, device, name=b"n2b_user_step"):
        if name == b"n2b_user_window" or (refused == "arrivals" and "n2_deliver" in source):
            raise RuntimeError("refused")
        return compiled(source, device, name)

    if refused == "parameters":
        monkeypatch.setattr(jit_runtime, "PARAMS_BYTES", 64)
        got, rt = _run(make)
    else:
        monkeypatch.setattr(jit_runtime, "compile_source", compile_source)
        with pytest.warns(UserWarning, match="refused"):
            got, rt = _run(make)
    assert rt.window is None and any("outs" in p for p in rt.plan["pops"]) == (refused == "window")
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_a_source_of_700_connections(cuda):
    """Its arrival kernel would take more parameters than a launch holds."""
    src = Pacemaker(period=3) * 20
    src.seed = 1
    targets = [TraceLIF(theta=1e9) * 2 for _ in range(700)]
    for i, t in enumerate(targets):
        t.seed = 2
        c = src >> Syn() @ fixed_indegree(3, seed=7) >> t
        c.weight, c.delay = 0.25, 0.1 * (1 + i % 3)
    net = src.network
    net.resolution = 0.1
    net.run_steps(13)
    net.check()
    v = [t.state_tensor("v").cpu() for t in targets]
    assert not any("outs" in p for p in net.runtime.plan["pops"])
    assert all(torch.equal(x, v[i % 3]) for i, x in enumerate(v)) and float(v[0].sum()) > 0

"""The stop word of the cooperative step kernels (set by a block whose barrier wait gave up) is read by one thread of each
block, which all its threads then follow: in the library's source and in the generated window kernel on the CPU. On the
GPU, windows whose waits give up one after the other (a 1 ns limit) end, say so, and leave a network that runs on."""

import itertools
import pathlib
import re

import pytest
import torch

from naer2_b200 import _lib, population
from naer2_b200.networks import brunel
from naer2_b200.patterns import fixed_indegree
from naer2_b200.transpiler import plan_of
from tests.dsl_models import Pacemaker, Syn, TraceLIF

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture(autouse=True)
def _own_seeds(monkeypatch):
    """Populations made here draw their default seeds from a count of their own."""
    monkeypatch.setattr(population, "_SEEDS", itertools.count(1 << 20))


def _user_net():
    src, tgt = Pacemaker(period=2) * 70, TraceLIF(theta=1.5) * 90
    src.seed, tgt.seed = 1, 2
    c = src >> Syn() @ fixed_indegree(20, seed=10) >> tgt
    c.weight, c.delay = 0.2, 0.2
    net = src.network
    net.resolution = 0.1
    return net


def test_one_thread_reads_the_stop_word():
    """Outside the barrier's wait (one thread already), no kernel that holds a grid barrier reads it per thread."""
    text = (ROOT / "naer2_b200" / "csrc" / "n2b_device.cuh").read_text()
    reads = [m.start() for m in re.finditer(r"\*\(volatile unsigned \*\)\((?:a\.barrier|bar) \+ BAR_ABORT\)", text)]
    assert len(reads) >= 2
    for at in reads:
        line = text[text.rindex("\n", 0, at):text.index("\n", at)]
        assert "threadIdx.x == 0 ? " in line or "(spin & 15) == 15" in line, line
    assert text.count("= stop_word(a)") == text.count("if (__syncthreads_or(stop))") == 2
    window = plan_of(_user_net())["window"]["source"]
    kernel = window[window.index("n2b_user_window"):]
    assert "const u32 stop = threadIdx.x == 0 ? *(volatile u32 *)(w.grid.bar + 32) : 0u;" in kernel
    assert kernel.count("volatile") == 1 and "if (WINDOW && __syncthreads_or(stop)) return;" in window


@pytest.mark.gpu
@pytest.mark.parametrize("delay", [1.5, "uniform", "hooks"])
def test_windows_that_give_up_in_turn(cuda, delay):
    net = _user_net() if delay == "hooks" else brunel.build(**dict(brunel.CONFIG0, delay=delay), eta=6.0, seed=11)[0]
    net.barrier_limit_ns = 1
    stops = 0
    for _ in range(8):
        for _ in range(4):
            net.run_steps(100)  # (queued: a window may start while the one before it stops)
        torch.cuda.synchronize()
        rt = net.runtime
        stops += int(rt.bar[33]) if delay == "hooks" else rt.status()[_lib.ERR_BARRIER]
        rt.reset_counters()
    assert stops >= 1
    if delay == "hooks":
        net.barrier_limit_ns = 0
        net.run_steps(50)
        net.check()
    net.close()

"""Workloads of this framework for timing: what its users have it do, through its public entry points.

Three families, over the sizes of this repository's own configurations (naer2_b200/networks), benchmark and tests:
  - stepping networks of the built-in models (`Network.run_steps` / `Network.step`): Brunel's model A, the PD14
    microcircuit, many uneven instances batched in one network, a densely driven population that pulls its input;
  - stepping networks of the user's own models (hooks compiled at run time): clocked, with plastic edges, and
    event-driven at exact spike times;
  - the recurrent LIF layer: plain forward, a training step, and its input projection alone (forward and backward).
A case is a dict of plain values; `path` names the family's member, the rest its sizes.
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

import naer2_b200 as n2
from naer2_b200 import receives as r
from naer2_b200.bptt import SpikeEvents
from naer2_b200.networks import batched, bptt_task, brunel, driven, pd14
from naer2_b200.patterns import fixed_indegree

DT = 0.1  # ms per step of every network


# ---------------------------------------------------------------------------------------------- the user's own models


@n2.node
class Afferent:
    """A Poisson input fibre, its draw made in its own hook."""

    def __init__(self, p: float = 0.01):
        self.p = p
        self.last: float = 0.0

    def update(self, time: n2.time):
        pass

    def send(self, time: n2.time):
        if random.random() < self.p:
            n2.spike()
            self.last = time

    def receive(self, time: n2.time, edge: r.edge, source: r.source):
        pass


@n2.node
class TraceLIF:
    """A leaky neuron with a postsynaptic trace for its plastic inputs."""

    def __init__(self, decay: float = 0.98, theta: float = 1.0, tau_post: float = 20.0):
        self.decay, self.theta, self.tau_post = decay, theta, tau_post
        self.v: float = 0.0
        self.y_post: float = 0.0
        self.t_post: float = 0.0

    def update(self, time: n2.time):
        self.v = self.v * self.decay

    def send(self, time: n2.time):
        if self.v >= self.theta:
            n2.spike()
            self.v = 0.0
            self.y_post = self.y_post * math.exp((self.t_post - time) / self.tau_post) + 1.0
            self.t_post = time

    def receive(self, time: n2.time, edge: r.edge, source: r.source):
        self.v += edge.weight


@n2.edge
class PairSTDP:
    """Pair-based plasticity: depression at an arrival, potentiation when the target fires."""

    def __init__(self, weight: float = 0.02, tau_pre: float = 20.0, tau_post: float = 20.0, a_plus: float = 0.0005,
                 a_minus: float = 0.0005, w_max: float = 0.05):
        self.weight = weight
        self.x_pre = 0.0
        self.t_last = 0.0
        self.tau_pre, self.tau_post, self.a_plus, self.a_minus, self.w_max = tau_pre, tau_post, a_plus, a_minus, w_max

    def forward(self, time: n2.time, dst: r.destination):
        self.x_pre = self.x_pre * math.exp((self.t_last - time) / self.tau_pre) + 1.0
        self.t_last = time
        y = dst.y_post * math.exp((dst.t_post - time) / self.tau_post)
        self.weight = max(self.weight - self.a_minus * y, 0.0)

    def backward(self, time: n2.time, dst: r.destination):
        x = self.x_pre * math.exp((self.t_last - time) / self.tau_pre)
        self.weight = min(self.weight + self.a_plus * x, self.w_max)


@n2.edge
class Synapse:
    def __init__(self, weight: float = 0.1):
        self.weight = weight

    def forward(self):
        pass

    def backward(self):
        pass


@n2.node
class JitterPacemaker:
    """An input that fires every `period` steps at its own time inside the step."""

    def __init__(self, period: int = 40):
        self.period = period
        self.phase: int = 0
        self.jitter: float = 0.0

    def update(self, time: n2.time):
        self.phase = self.phase + 1
        self.jitter = self.jitter * 0.9 + 0.005

    def send(self, time: n2.time):
        if self.phase % self.period == 0:
            n2.spike(time - self.jitter)

    def receive(self, time: n2.time, edge: r.edge, source: r.source):
        pass


@n2.node
class DecayLIF:
    """A leaky neuron that decays exactly between its arrivals."""

    def __init__(self, tau: float = 10.0, theta: float = 1.0, v_reset: float = 0.0, t_ref: float = 1.0):
        self.tau, self.theta, self.v_reset, self.t_ref = tau, theta, v_reset, t_ref
        self.v: float = 0.0
        self.last: float = 0.0
        self.ref_end: float = 0.0

    def update(self, time: n2.time):
        pass

    def send(self, time: n2.time):
        if self.v >= self.theta:
            n2.spike(time)
            self.v = self.v_reset
            self.ref_end = time + self.t_ref
            self.last = time + self.t_ref

    def receive(self, time: n2.time, edge: r.edge, source: r.source):
        if time >= self.ref_end:
            self.v = self.v * math.exp((self.last - time) / self.tau) + edge.weight
            self.last = time


# ---------------------------------------------------------------------------------------------- the cases


def listed():
    return [
        # a closed loop that steps one dt at a time (reads the state, acts, steps again): launch latency
        dict(name="brunel_1k_one_step", path="brunel", ne=800, ce=80, delay="fixed", steps=1, record=False),
        # the small test network over one default window, spikes recorded (its single delay of 1.5 ms)
        dict(name="brunel_1k_window", path="brunel", ne=800, ce=80, delay="fixed", steps=100, record=True),
        # the usual size: Brunel's model A at 12,500 neurons, delays 1-20 steps, a window and a remainder
        dict(name="brunel_12k", path="brunel", ne=10000, ce=1000, delay="uniform", steps=130, record=True),
        # the cortical microcircuit, weights and delays per link
        dict(name="pd14_half", path="pd14", scale=0.5, steps=100, record=True),
        # a parameter scan: uneven networks stepped together
        dict(name="batched_10", path="batched", instances=10, steps=50),
        # a dense input, pulled
        dict(name="driven_pull", path="driven", n_in=2000, n=10000, k_in=500, steps=100),
        # the usual size with the user's own neuron model
        dict(name="hooks_12k", path="hooks", ne=10000, ce=1000, steps=50),
        # plastic inputs, an odd size
        dict(name="hooks_stdp", path="plastic", n_pre=1999, n=1501, k=150, steps=100),
        # event-driven delivery at exact spike times
        dict(name="hooks_exact", path="exact", n_pre=1000, n=3001, k=100, steps=100),
        # inference, an odd and smaller layer
        dict(name="layer_infer_odd", path="infer", batch=24, steps=151, channels=333, hidden=320, readouts=11),
        # the training step of the benchmark's configuration
        dict(name="layer_train", path="train", batch=128, steps=500, channels=700, hidden=1024, readouts=20),
        # the input projection alone, forward and backward
        dict(name="projection", path="project", batch=128, steps=250, channels=700, hidden=1024, readouts=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["brunel", "brunel", "pd14", "batched", "driven", "hooks", "hooks", "plastic", "exact", "infer",
                       "train", "project"])
    if path == "brunel":
        ne = _log(rng, 500, 12000)
        return dict(path=path, ne=ne, ce=max(8, min(1000, ne // 10)), delay=rng.choice(["fixed", "uniform"]),
                    steps=_log(rng, 1, 200), record=rng.random() < 0.5)
    if path == "pd14":
        return dict(path=path, scale=round(math.exp(rng.uniform(math.log(0.02), math.log(0.5))), 4),
                    steps=rng.randint(20, 100), record=rng.random() < 0.5)
    if path == "batched":
        return dict(path=path, instances=rng.randint(2, 10), steps=rng.randint(10, 50))
    if path == "driven":
        n = _log(rng, 1000, 10000)
        return dict(path=path, n_in=_log(rng, 300, 2500), n=n, k_in=_log(rng, 100, 600), steps=rng.randint(20, 100))
    if path == "hooks":
        ne = _log(rng, 500, 10000)
        return dict(path=path, ne=ne, ce=max(8, min(1000, ne // 10)), steps=_log(rng, 5, 60))
    if path == "plastic":
        return dict(path=path, n_pre=_log(rng, 300, 4000), n=_log(rng, 200, 4000), k=_log(rng, 30, 200),
                    steps=_log(rng, 10, 100))
    if path == "exact":
        return dict(path=path, n_pre=_log(rng, 300, 2000), n=_log(rng, 300, 5000), k=_log(rng, 30, 120),
                    steps=_log(rng, 10, 100))
    return dict(path=path, batch=8 * _log(rng, 1, 16), steps=_log(rng, 50, 400), channels=_log(rng, 100, 700),
                hidden=32 * _log(rng, 2, 32), readouts=rng.randint(2, 20))


# ---------------------------------------------------------------------------------------------- inputs


def _brunel(case, seed, dev, hooks=False):
    ne, ce = case["ne"], case["ce"]
    net, pops = brunel.build(NE=ne, NI=ne // 4, CE=ce, CI=max(1, ce // 4), seed=seed, device=dev, transpiled=hooks,
                             delay=1.5 if case.get("delay") == "fixed" else "uniform")
    return net, {name: (p, ("V", "ref")) for name, p in pops.items()}


def _plastic(case, seed, dev):
    g = torch.Generator(device="cpu").manual_seed(seed)
    src, tgt = Afferent(p=0.004) * case["n_pre"], TraceLIF() * case["n"]
    src.seed, tgt.seed = (seed << 8) | 1, (seed << 8) | 2
    c = src >> PairSTDP() @ fixed_indegree(case["k"], seed=(seed << 8) | 3, device=dev) >> tgt
    c.weight = 0.01 + 0.03 * torch.rand(c.shape, generator=g)
    c.delay = ((torch.randint(1, 16, c.shape, generator=g) * DT).double()).to(dev)
    net = src.network
    net.resolution = DT
    tgt.v = torch.rand(case["n"], generator=g)
    return net, {"post": (tgt, ("v", "y_post", "t_post"))}, c


def _exact_times(case, seed, dev):
    g = torch.Generator(device="cpu").manual_seed(seed)
    src, tgt = JitterPacemaker() * case["n_pre"], DecayLIF(theta=0.5) * case["n"]
    src.seed, tgt.seed = (seed << 8) | 1, (seed << 8) | 2
    for s, k, w in ((src, case["k"], 0.25), (tgt, max(2, case["k"] // 4), 0.05)):
        c = s >> Synapse() @ fixed_indegree(k, seed=(seed << 8) | (3 + (s is tgt)), device=dev) >> tgt
        c.weight = (w * (0.2 + torch.rand(c.shape, generator=g))).to(dev)
        c.delay = ((torch.randint(1, 21, c.shape, generator=g) * DT).double()).to(dev)
    src.phase = torch.randint(0, 40, (case["n_pre"],), generator=g, dtype=torch.int32)
    src.jitter = (0.05 * torch.rand(case["n_pre"], generator=g)).float()
    net = src.network
    net.resolution = DT
    net.exact = True
    return net, {"post": (tgt, ("v", "last", "ref_end"))}


def _layer(case, seed, dev, density=0.1):
    kw = dict(batch=case["batch"], steps=case["steps"], channels=case["channels"], hidden=case["hidden"],
              readouts=case["readouts"], density=density, classes=case["readouts"])
    return bptt_task.build(seed=seed, device=dev, **kw)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    path = case["path"]
    if path in ("infer", "train", "project"):
        layer, x, y = _layer(case, seed, dev, density=0.01 if path == "project" else 0.1)
        state = {"path": path, "layer": layer, "x": SpikeEvents.from_dense(x), "y": y}
        if path == "project":
            g = torch.Generator(device=dev).manual_seed(seed + 11)
            state["du"] = torch.randn(case["steps"], case["batch"], case["hidden"], generator=g, device=dev)
        return state
    plastic = None
    if path == "brunel":
        net, pops = _brunel(case, seed, dev)
    elif path == "hooks":
        net, pops = _brunel(case, seed, dev, hooks=True)
    elif path == "plastic":
        net, pops, plastic = _plastic(case, seed, dev)
    elif path == "exact":
        net, pops = _exact_times(case, seed, dev)
    elif path == "pd14":
        net, pl = pd14.build(scale=case["scale"], seed=seed, device=dev)
        pops = {n: (p, ("potential", "current", "ref")) for n, p in zip(pd14.NAMES, pl)}
    elif path == "batched":
        # the scan's sizes and parameters are its own, its draws the seed's
        parts = [brunel.build(**dict(p, seed=(seed << 12) | (b + 1)), device=dev)
                 for b, p in enumerate(batched.instance_params(b) for b in range(case["instances"]))]
        net, parts = parts[0][0], [p for _, p in parts]
        for part in parts[1:]:
            net += part["E"].network
        pops = {f"{k}{b}": (p, ("V", "ref")) for b, part in enumerate(parts) for k, p in part.items()}
    elif path == "driven":
        net, pl = driven.build(N_in=case["n_in"], N=case["n"], K_in=case["k_in"], J_in=0.1 * 5 / case["k_in"] * 0.1,
                               seed=seed, device=dev)
        for c in net.connections:
            if c._source is pl["in"]:
                c.mode = "pull"
        pops = {k: (pl[k], ("V", "ref")) for k in ("E", "I")}
    else:
        raise ValueError(path)
    record = case.get("record", True)
    if record:
        net.record(case["steps"])
    state = {"path": path, "net": net, "pops": pops, "steps": case["steps"], "record": record, "plastic": plastic}
    net.runtime  # the buffers and kernels of the network, built once
    return state


# ---------------------------------------------------------------------------------------------- one pass


def run(state):
    path = state["path"]
    if path == "infer":
        m, t = state["layer"].infer(state["x"])
        return {"m": m, "t": t}
    if path == "train":
        layer = state["layer"]
        layer.zero_grad(set_to_none=True)
        m = layer(state["x"])
        loss = torch.nn.functional.cross_entropy(m, state["y"])
        loss.backward()
        return {"m": m.detach(), "loss": loss.detach(), "w_in": layer.w_in.grad, "w_rec": layer.w_rec.grad,
                "w_out": layer.w_out.grad}
    if path == "project":
        layer = state["layer"]
        layer.zero_grad(set_to_none=True)
        u = layer.current(state["x"])
        u.backward(state["du"])
        return {"u": u.detach(), "w_in": layer.w_in.grad}
    net = state["net"]
    if state["record"]:
        net.record(state["steps"])
    if state["steps"] == 1:
        net.step(DT)
    else:
        net.run_steps(state["steps"])
    out = {name: {a: p.state_tensor(a) for a in attrs} for name, (p, attrs) in state["pops"].items()}
    if state["record"]:
        rt = net.runtime
        for name, (p, _) in state["pops"].items():
            out[name]["spikes"] = rt.rasters[rt.pops.index(p)]
    if state["plastic"] is not None:
        out["weight"] = net.runtime.edge_state(state["plastic"], "weight")
    return out


# ---------------------------------------------------------------------------------------------- the work of one pass


def work(case):
    """Bytes and operations of one pass. A network: per neuron and step its membrane and arrival slot read and
    written (16 bytes, with a synaptic current 32), per synaptic event its link (9 bytes: target, delay, weight), at
    rates that these networks settle at. The layer: its input current, spikes and gradients once."""
    path = case["path"]
    if path in ("infer", "train", "project"):
        T, B, C, H, R = (case[k] for k in ("steps", "batch", "channels", "hidden", "readouts"))
        u, w_in, nnz_in = 4.0 * T * B * H, 4.0 * C * H, 0.006 * T * B * C
        if path == "project":
            return {"bytes": 2 * u + 2 * w_in + 2 * 4 * nnz_in, "flops": 2 * nnz_in * H}
        nnz = 0.1 * H * H
        spikes = 0.03 * T * B * H  # about 30 Hz
        fwd = {"bytes": 2 * u + w_in + 4 * nnz_in + 6 * nnz, "flops": spikes * 0.1 * H + 4 * T * B * H + nnz_in * H}
        if path == "infer":
            return fwd
        # the adjoint: every link of every step carries a gradient, the weights' only where the source spiked
        return {"bytes": fwd["bytes"] + 3 * u + T * B * H / 8 + 2 * w_in + 12 * nnz,
                "flops": fwd["flops"] + 2 * T * B * nnz + spikes * 0.1 * H + nnz_in * H}
    steps = case["steps"]
    if path in ("brunel", "hooks"):
        n, per = 1.25 * case["ne"], 1.25 * case["ce"]
        rate, state = 0.004, 16
    elif path == "pd14":
        n, per = 77169 * case["scale"], 3870 * case["scale"]
        rate, state = 0.0004, 32
    elif path == "batched":
        sizes = [batched.instance_params(b) for b in range(case["instances"])]
        n = sum(p["NE"] + p["NI"] for p in sizes)
        per = sum((p["NE"] + p["NI"]) * (p["CE"] + p["CI"]) for p in sizes) / n
        rate, state = 0.01, 16
    elif path == "driven":
        n, per, rate, state = case["n"], case["k_in"], 0.39, 16
    elif path == "plastic":
        n, per, rate, state = case["n"], case["k"], 0.004, 24
    else:
        n, per, rate, state = case["n"], 1.25 * case["k"], 0.025, 24
    events = n * per * rate * steps
    return {"bytes": n * state * steps + 9 * events, "flops": 2 * events + 4 * n * steps}


# ---------------------------------------------------------------------------------------------- in 64 bits


class _Spike(torch.autograd.Function):
    """Heaviside forward, the fast sigmoid's derivative backward."""

    @staticmethod
    def forward(ctx, x, slope):
        ctx.save_for_backward(x)
        ctx.slope = slope
        return (x >= 0).to(x.dtype)

    @staticmethod
    def backward(ctx, g):
        (x,) = ctx.saved_tensors
        return g / (1.0 + ctx.slope * x.abs()) ** 2, None


def exact(case, seed):
    """The layer in dense float64 autograd. The networks have no such value: their spikes are whole numbers, and
    their states follow them."""
    if case["path"] not in ("infer", "train", "project"):
        return None
    dev = torch.device("cuda", torch.cuda.current_device())
    layer, x, y = _layer(case, seed, dev, density=0.01 if case["path"] == "project" else 0.1)
    w_in, w_rec, w_out = (p.detach().double().requires_grad_() for p in (layer.w_in, layer.w_rec, layer.w_out))
    u = torch.matmul(x.double(), w_in)
    if case["path"] == "project":
        g = torch.Generator(device=dev).manual_seed(seed + 11)
        du = torch.randn(case["steps"], case["batch"], case["hidden"], generator=g, device=dev)
        u.backward(du.double())
        return {"u": u.detach(), "w_in": w_in.grad}
    wiring, H = layer.wiring, case["hidden"]
    pre, post, delay = (torch.from_numpy(np.asarray(a)).to(dev) for a in (wiring.pre, wiring.post, wiring.delay))
    D = 5
    W = torch.zeros(D * H, H, dtype=torch.float64, device=dev).index_put(((delay - 1) * H + pre, post), w_rec)
    alpha, beta, theta, slope = layer.alpha, layer.beta, layer.theta, layer.slope
    B, R = case["batch"], case["readouts"]
    V = torch.zeros(B, H, dtype=torch.float64, device=dev)
    O = torch.zeros(B, R, dtype=torch.float64, device=dev)
    zero = torch.zeros(B, H, dtype=torch.float64, device=dev)
    hist, Os = [zero] * D, []  # hist[d - 1]: the spikes d steps ago
    with torch.set_grad_enabled(case["path"] == "train"):
        for t in range(case["steps"]):
            vp = alpha * V + u[t] + torch.cat(hist, 1) @ W
            s = _Spike.apply(vp - theta, slope)
            V = vp - theta * s
            O = beta * O + s @ w_out
            hist = [s] + hist[:-1]
            Os.append(O)
        m, ts = torch.stack(Os).max(dim=0)
        if case["path"] == "infer":
            return {"m": m, "t": None}
        loss = torch.nn.functional.cross_entropy(m, y)
    loss.backward()
    return {"m": m.detach(), "loss": loss.detach(), "w_in": w_in.grad, "w_rec": w_rec.grad, "w_out": w_out.grad}

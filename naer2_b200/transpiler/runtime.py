"""The run-time compiled path: a network whose populations' hooks are lowered to CUDA and compiled with
NVRTC (reference naer2/runtime.py:213-526, PopulationRuntime, which builds and launches the generated
Gluon kernels; here one generated step kernel per population, `n2b_jit_*` in the C ABI).

Built by Network.runtime when a population's model has no built-in kernel (models.params_of raises). Every
population of such a network runs its own transpiled hooks -- built-in models included, as their hooks
state them in Python. The interface Network uses is NetworkRuntime's: advance, start_recording, raster,
spikes, status, check, counters, reset_counters, close.
"""

from __future__ import annotations

import ast
import ctypes
import functools
import hashlib
import warnings

import numpy as np
import torch

from .. import _lib, receives
from ..hook import assigned_members
from ..topology import delay_steps, pull_form
from . import arrival
from .template import NPB_C, build_source, ctype_of, edge_hook_context, hook_context, params_type, scan

BLOCK = 128  # exact-time intake without arrival bits: one thread per neuron
# A network's intake reads arrival bits (one bit per link and arrival slot, set by the spikes' deliveries) as long
# as they and the outgoing rows take at most this much, and half of the device's free memory with what making them
# holds at once (BUILD_BYTES per link of a connection: int64 columns and a sort, 52 measured); past it, every neuron
# looks its whole incoming row up in its sources' spike rings, which needs no more memory than the links. At 12,500
# neurons of 1,250 links and 32 slots the bits are 64 MB, the rows 78 MB.
ARRIVAL_BYTES = 32 << 30
BUILD_BYTES = 72
SMALL_BYTES = 64 << 20  # less than this is taken without asking the device (0.7 ms)
PACKED_BITS = 1 << 24  # bits of a slot whose places leave a link word's top 8 bits to the delay
PARAMS_BYTES = 32764  # a kernel's parameters at most (48 bytes per outgoing connection, 40 to 64 per incoming one)
# A window kernel holds every block of the network at once: 592 blocks (18,944 neurons) are four per SM, 64 registers
# a thread, which the step's code needs (five per SM would be 51). Larger networks, those of more than
# arrival.WINDOW_POPS populations or, over the distinct ones, arrival.WINDOW_INTAKES connections, and devices that hold
# fewer blocks step by one launch per population.
WINDOW_BLOCKS, WINDOW_SMS = 592, 148
WINDOW_STEPS = 1024  # steps of one launch of it at most (8 ms at 7.5 us a step): other streams' launches come in between
BARRIER_LIMIT_NS = 2_000_000_000  # how long a window's block waits at its grid barrier before it gives up
_CACHE: dict = {}  # (source hash, device) -> n2b_jit_kernel handle, for the process's lifetime


def compile_source(source: str, device: int, name: bytes = b"n2b_user_step") -> ctypes.c_void_p:
    key = (hashlib.sha256(source.encode()).hexdigest(), device)
    if key not in _CACHE:
        lib = _lib.load()
        h = ctypes.c_void_p()
        _lib.check(lib.n2b_jit_compile(source.encode(), name, None, 0, device, ctypes.byref(h)),
                   "n2b_jit_compile")
        _CACHE[key] = h
    return _CACHE[key]


def trivial(hook) -> bool:
    """A hook whose body does nothing (pass / a docstring)."""
    if hook is None:
        return True
    return all(isinstance(st, ast.Pass) or (isinstance(st, ast.Expr) and isinstance(st.value, ast.Constant))
               for st in hook.ast.body)


class EdgePlan:
    """What a connection's hooks read and write of its links. recv: {receive-facing name: edge name};
    per_link: edge names held per link (assigned by the edge hooks, or set as per-link tensors); written:
    those the edge hooks assign; static: {edge name: value} of the rest; forward / backward: the edge's
    non-trivial hooks (or None)."""

    def __init__(self, conn, receive_hook):
        from ..hook import used_members

        fabric = conn.fabric
        rename = {hook_name: real for real, hook_name in (conn._fabric_map or {}).items()}
        edge_param = receive_hook.parameter_type_to_name.get(receives.edge, "edge") if receive_hook else "edge"
        names = used_members(receive_hook.ast, edge_param) if receive_hook is not None else set()
        self.recv = {h: rename.get(h, h) for h in sorted(names)}
        has_edge = fabric.instance is not None
        self.forward = None if not has_edge or trivial(fabric.edge["forward"]) else fabric.edge["forward"]
        self.backward = None if not has_edge or trivial(fabric.edge["backward"]) else fabric.edge["backward"]
        used, written = set(self.recv.values()), set()
        for h in (self.forward, self.backward):
            if h is not None:
                used |= used_members(h.ast, "self")
                written |= h.assigned_members
        self.written = sorted(written)
        self.per_link, self.static = [], {}
        for name in sorted(used):
            v = fabric.value(name)
            if v is None:
                raise ValueError(f"{conn!r}: edge.{name} is read but the connection has no such attribute")
            if name in written or (isinstance(v, torch.Tensor) and v.numel() != 1):
                self.per_link.append(name)
            else:
                self.static[name] = float(v.item() if isinstance(v, torch.Tensor) else v)

    def initial(self, conn, name: str, n_links: int) -> torch.Tensor:
        """A per-link array's starting values, canonical order, float32 on the CPU."""
        v = conn.fabric.value(name)
        if isinstance(v, torch.Tensor) and v.numel() == n_links:
            return v.detach().reshape(-1).to("cpu", torch.float32)
        return torch.full((n_links,), float(v.item() if isinstance(v, torch.Tensor) else v), dtype=torch.float32)


def arrival_bytes(n_tgt: int, n_links: int, depth: int) -> int:
    """Device bytes of a connection's arrival bits (`depth` slots of one bit per link, rows starting words of their
    own) and outgoing rows (5 bytes per link), at most."""
    return depth * 4 * (n_links // 32 + n_tgt) + 5 * n_links


def arrival_form(ptr: torch.Tensor, link: torch.Tensor, n_src: int, mask: int) -> dict:
    """The arrival bits of one connection, from its pull CSR: `wptr` int32 [n_tgt + 1], each row's first word in a
    slot; `words` per slot; `depth`, the slots (the largest delay + 1: a slot is read and cleared in the step before
    the first that can set it again); the outgoing rows `out_ptr` int32 [n_src + 1], `pos` int32 (uint32 bits: the
    link's bit in a slot) and `dly` uint8, links of a source in pull order -- with at most 2^24 bits to a slot the
    delay is in the top 8 bits of `pos` and `dly` is None; `bad`: links whose source or delay (1 .. mask) is out of
    range, in no outgoing row."""
    dev = link.device
    n_tgt = len(ptr) - 1
    ptr = ptr.to(torch.int64)
    lens = ptr.diff()
    wptr = torch.zeros(n_tgt + 1, dtype=torch.int64, device=dev)
    wptr[1:] = torch.cumsum((lens + 31) // 32, 0)
    n_links = int(ptr[-1]) if n_tgt else 0
    link = link[:n_links]
    src, dly = link & 0xFFFFFF, (link >> 24) & 0xFF
    pos = torch.repeat_interleave(wptr[:-1] * 32 - ptr[:-1], lens) + torch.arange(n_links, device=dev)
    good = (dly >= 1) & (dly <= mask) & (src < n_src)
    bad = n_links - int(good.sum())
    if bad:
        src, dly, pos = src[good], dly[good], pos[good]
    order = torch.argsort(src, stable=True)
    out_ptr = torch.zeros(n_src + 1, dtype=torch.int64, device=dev)
    out_ptr[1:] = torch.cumsum(torch.bincount(src, minlength=n_src)[:n_src], 0)
    dly = dly[order]
    top = int(dly.max()) if dly.numel() else 1
    pos, words = pos[order], int(wptr[-1])
    packed = 32 * words <= PACKED_BITS
    if packed:
        pos = pos | (dly.to(torch.int64) << 24)
    return {"wptr": wptr.to(torch.int32), "words": words, "depth": top + 1,
            "out_ptr": out_ptr.to(torch.int32),
            "pos": torch.where(pos >= 2 ** 31, pos - 2 ** 32, pos).to(torch.int32),
            "dly": None if packed else dly.to(torch.uint8), "bad": bad}


def scan_form(plan: dict) -> dict:
    """A plan of arrival bits as one of the scanning intake, which needs no memory beside the links."""
    out = {key: v for key, v in plan.items() if key != "window"}
    out["pops"] = [{**{key: v for key, v in p.items() if key not in ("outs", "scan")}, **p["scan"]} for p in plan["pops"]]
    return out


def arrivals_need(plan: dict) -> int:
    """Device bytes of a plan's arrival bits and outgoing rows, and of building the largest connection's."""
    pops = plan["pops"]
    sizes = [(arrival_bytes(p["n"], len(c["link"]), pops[c["src"]]["depth"]), BUILD_BYTES * len(c["link"]))
             for p in pops for c in p["conns"]]
    return sum(t for t, _ in sizes) + max((b for _, b in sizes), default=0)


def plan_of(net, intake: str | None = None) -> dict:
    """The transpiled form of a network, everything its step kernels need and nothing of its Python model classes:
    per population its CUDA source, the Params fields with the values of the scalar ones, its state attributes
    (name -> "float" / "int" / "bool"), size, seed and spike-ring depth, and (networks whose intake reads arrival
    bits) its outgoing connections; per incoming connection (in order) its
    source population, pull CSR (int32 ptr, uint32 link words) and per-link edge arrays (pull order) with the
    pull permutation. JitRuntime builds from it; save_plan / load_plan keep it in a file, so that a network can
    be transpiled where its model classes are and stepped where only the plan is. A plan of arrival bits carries the
    scanning intake's sources along ("scan"), but with intake "arrivals"; "scan" is a plan of the latter alone."""
    dev = net.device if net.device is not None else torch.device("cpu")
    dt = float(net.resolution)
    pops = list(net.populations)
    index = {id(p): k for k, p in enumerate(pops)}
    words = [(len(p.shape) + 31) // 32 for p in pops]
    # spike-bit ring depth of each population: above every delay of its outgoing connections
    steps_of, max_out = {}, [1] * len(pops)
    for c in net.connections:
        topo = c.fabric.topology
        steps = delay_steps(c.fabric.value("delay"), len(topo), dt, device=topo.target_indices.device)
        steps_of[id(c)] = steps
        if len(topo):
            s = index[id(c._source)]
            max_out[s] = max(max_out[s], int(steps.max()))
    depth = [max(2, 1 << int(np.ceil(np.log2(m + 1)))) for m in max_out]
    exact = bool(getattr(net, "exact", False))
    plan = {"dt": dt, "exact": exact, "pops": []}
    incoming_of = [[c for c in net.connections if c._target is p] for p in pops]
    outs = [[] for _ in pops]  # each population's outgoing connections: (target population, its connection)
    for k, conns in enumerate(incoming_of):
        for ci, c in enumerate(conns):
            outs[index[id(c._source)]].append([k, ci])
    arrivals = sum(arrival_bytes(len(p.shape), len(c.fabric.topology), depth[index[id(c._source)]])
                   for p, conns in zip(pops, incoming_of) for c in conns) <= ARRIVAL_BYTES and intake != "scan"
    total = sum(arrival.blocks_of(len(p.shape)) for p in pops)
    per_sm = -(-total // WINDOW_SMS)
    ahead = arrival.AHEAD_FEW if 2 * WINDOW_SMS < total <= WINDOW_BLOCKS else arrival.AHEAD
    bodies, edges = [], 0  # arrival bits: the populations' part of the window kernel, edge attributes they stage
    for k, p in enumerate(pops):
        node, conns, name = p.node, incoming_of[k], type(p.instance).__name__

        def lowered() -> tuple[list, dict]:
            """The incoming connections and the hooks as a source takes them (their draws' call sites count from here)."""
            incoming, site = [], 0
            for c in conns:
                port = c._target_port or "receive"
                hook = node.receive.get(port)
                if hook is None:
                    raise ValueError(f"{p!r} has no receive port {port!r}")
                ep = EdgePlan(c, hook)
                dyn = [h for h, real in ep.recv.items() if real in ep.per_link]
                stat = {h: ep.static[real] for h, real in ep.recv.items() if real not in ep.per_link}
                ctx = hook_context(p, hook, dyn, stat, site_base=site)
                site += 32
                inc = {"receive": (hook.ast, ctx), "edge_dynamic": ep.per_link, "edge_written": ep.written,
                       "alias": {h: real for h, real in ep.recv.items() if real in ep.per_link and h != real},
                       "forward": None, "backward": None, "conn": c, "plan": ep}
                for kind in ("forward", "backward"):
                    eh = getattr(ep, kind)
                    if eh is not None:
                        inc[kind] = (eh.ast, edge_hook_context(p, eh, ep.per_link, ep.static))
                if ep.backward is not None:
                    dst = ep.backward.parameter_type_to_name.get(receives.destination)
                    inc["backward_writes"] = dst is not None and bool(assigned_members(ep.backward.ast, dst))
                incoming.append(inc)
            return incoming, {"update": (node.update.ast, hook_context(p, node.update, site_base=site)),
                              "send": (node.send.ast, hook_context(p, node.send, site_base=site + 32))}

        if not arrivals or intake is None:
            incoming, hooks = lowered()
            src, fields = build_source(name, dict(p.dynamic_attrs), hooks, incoming, exact=exact, n=len(p.shape))
            scanning = {"source": src, "fields": [(f, ctype) for f, ctype, _ in fields]}
        if arrivals:
            incoming, hooks = lowered()
            src, fields, body = arrival.build(name, dict(p.dynamic_attrs), hooks, incoming, len(outs[k]), exact, ahead)
            bodies.append(body)
            edges = max(edges, arrival.staged(incoming, exact))
        attrs = {a: ("bool" if py is bool else "int" if py is int else "float") for a, py in p.dynamic_attrs.items()}
        entry = {"name": name, "n": len(p.shape), "words": words[k], "depth": depth[k],
                 "seed": int(p.seed) & 0xFFFFFFFFFFFFFFFF, "source": src,
                 "fields": [(name, ctype) for name, ctype, _ in fields], "attrs": attrs, "conns": []}
        if arrivals:
            entry["outs"] = outs[k]
            if intake is None:
                entry["scan"] = scanning
        for inc in incoming:
            c = inc["conn"]
            topo = c.fabric.topology
            ptr, link, perm = pull_form(topo, steps_of[id(c)], len(p.shape))
            ep = inc["plan"]
            per_link = {}
            for e in ep.per_link:
                v = ep.initial(c, e, len(topo))
                per_link[e] = (v[perm.cpu()] if v.numel() else torch.zeros(0)).to(torch.float32)
            entry["conns"].append({"src": index[id(c._source)], "ptr": ptr.to(torch.int32).cpu(),
                                   "link": link.to(torch.int32).cpu(), "perm": perm.cpu(), "per_link": per_link,
                                   "written": list(ep.written), "conn_id": id(c)})
        plan["pops"].append(entry)
    if arrivals and 0 < total <= WINDOW_BLOCKS and len(pops) <= arrival.WINDOW_POPS:
        kinds = sorted(set(bodies), key=bodies.index)  # populations of one text share its code
        if sum(len(incoming_of[bodies.index(b)]) for b in kinds) <= arrival.WINDOW_INTAKES:
            order = sorted(range(len(pops)), key=lambda k: (kinds.index(bodies[k]), k))
            counts = [bodies.count(b) for b in kinds]
            plan["window"] = {"source": arrival.window_source(exact, list(zip(kinds, counts)), edges, per_sm),
                              "order": order, "counts": counts}
    plan["device"] = dev
    return plan


def save_plan(plan: dict, path) -> None:
    """A plan in one .npz file: its structure as JSON, its arrays beside it."""
    import json

    arrays, meta = {}, {"dt": plan["dt"], "exact": plan["exact"], "pops": []}
    if "window" in plan:
        meta["window_kernel"] = plan["window"]
    for k, p in enumerate(plan["pops"]):
        m = {key: p[key] for key in ("name", "n", "words", "depth", "seed", "source", "fields", "attrs", "outs",
                                      "scan") if key in p}
        m["conns"] = []
        for ci, c in enumerate(p["conns"]):
            for key in ("ptr", "link", "perm"):
                arrays[f"p{k}_c{ci}_{key}"] = c[key].numpy()
            for e, v in c["per_link"].items():
                arrays[f"p{k}_c{ci}_e_{e}"] = v.numpy()
            m["conns"].append({"src": c["src"], "per_link": list(c["per_link"]), "written": c["written"]})
        meta["pops"].append(m)
    arrays["plan_json"] = np.frombuffer(json.dumps(meta).encode(), dtype=np.uint8)
    np.savez_compressed(path, **arrays)


def load_plan(path) -> dict:
    import json

    z = np.load(path)
    meta = json.loads(bytes(z["plan_json"]).decode())
    plan = {"dt": meta["dt"], "exact": meta["exact"], "pops": []}
    if "window_kernel" in meta:  # (an older plan's, under "window", takes other parameters: it steps without)
        plan["window"] = meta["window_kernel"]
    for k, m in enumerate(meta["pops"]):
        p = dict(m)
        p["fields"] = [tuple(f) for f in m["fields"]]
        if "scan" in m:
            p["scan"] = {"source": m["scan"]["source"], "fields": [tuple(f) for f in m["scan"]["fields"]]}
        p["conns"] = []
        for ci, c in enumerate(m["conns"]):
            p["conns"].append({"src": c["src"], "written": c["written"], "conn_id": None,
                               "ptr": torch.from_numpy(z[f"p{k}_c{ci}_ptr"]),
                               "link": torch.from_numpy(z[f"p{k}_c{ci}_link"]),
                               "perm": torch.from_numpy(z[f"p{k}_c{ci}_perm"]),
                               "per_link": {e: torch.from_numpy(z[f"p{k}_c{ci}_e_{e}"]) for e in c["per_link"]}})
        plan["pops"].append(p)
    return plan


_CTYPES = {"long long": ctypes.c_int64, "float": ctypes.c_float, "int": ctypes.c_int32, "u32": ctypes.c_uint32}


@functools.lru_cache(maxsize=256)
def _params_struct(fields: tuple):
    """The ctypes Params structure of a plan's fields (pointers as void *)."""
    def ctype(ct):
        if ct.startswith("N2Out["):
            return arrival.Out * int(ct[6:-1])
        return ctypes.c_void_p if ct.endswith("*") else _CTYPES[ct]

    return params_type([(name, ct, ctype(ct)) for name, ct in fields])


def _window_type(window: dict, types: list):
    """The parameter block of a plan's window kernel, `types` the populations' Params."""
    kinds, at = [], 0
    for count in window["counts"]:
        kinds.append((types[window["order"][at]], count))
        at += count
    return arrival.window_type(tuple(kinds))


class JitRuntime:
    """The step kernels of a transpiled network: built from `net` (its plan made on the spot), or from a saved
    plan (`plan`; `net` then a PlannedNetwork holding the plan's state)."""

    def __init__(self, net, plan: dict | None = None):
        self.net = net
        dev = self.device = net.device
        dindex = dev.index if dev.index is not None else 0
        scanning = None  # the plan's other form (plans of an older version have none)
        if plan is None:
            plan, scanning = plan_of(net, "arrivals"), lambda: plan_of(net, "scan")
        elif any("scan" in p for p in plan["pops"]):
            scanning = functools.partial(scan_form, plan)
        # arrival bits where they, and making them, take half of what is free on the device at most
        if scanning and any("outs" in p for p in plan["pops"]):
            need = arrivals_need(plan)
            if need > SMALL_BYTES and need > _lib.free_bytes(dev) // 2:
                plan, scanning = scanning(), None
        plan, window_kernel, self.kernels = self._compiled(plan, scanning, dindex)
        self.plan = plan
        dt = self.dt = float(plan["dt"])
        pops = self.pops = list(net.populations)
        self.keep = []
        words = self.words = [p["words"] for p in plan["pops"]]
        depth = self.depth = [p["depth"] for p in plan["pops"]]
        self.bits = [torch.zeros(d * w, dtype=torch.int32, device=dev) for d, w in zip(depth, words)]
        # each spike's time within its step (event-driven intake reads it; the clocked one ignores it)
        self.offs = [torch.zeros(d * max(1, p["n"]), dtype=torch.float32, device=dev)
                     for d, p in zip(depth, plan["pops"])]
        self.exact = bool(plan["exact"])
        self.err = torch.zeros(len(pops), dtype=torch.int32, device=dev)
        self.counters_t = torch.zeros(len(pops), 2, dtype=torch.int64, device=dev)
        self.record_rows = int(net.record_steps)
        self.rec_step0 = net.step_count
        self.rasters = [torch.zeros(max(1, self.record_rows) * w, dtype=torch.int32, device=dev) for w in words]
        self.raster_offs = [torch.zeros(max(1, self.record_rows) * max(1, p["n"]), dtype=torch.float32,
                                        device=dev) for p in plan["pops"]]
        self.params, self.sources = [], []
        forms = []  # per population, its incoming connections' arrival forms
        self.edge_arrays = {}  # (connection id, edge name) -> (per-link values in pull order, pull permutation)
        tdtype = {"bool": torch.bool, "int": torch.int32, "float": torch.float32}
        for k, (p, pp) in enumerate(zip(pops, plan["pops"])):
            self.sources.append(pp["source"])
            P = _params_struct(tuple(pp["fields"]))()
            P.n, P.words, P.bit_mask = pp["n"], words[k], depth[k] - 1
            P.seed_lo, P.seed_hi = pp["seed"] & 0xFFFFFFFF, (pp["seed"] >> 32) & 0xFFFFFFFF
            for a, ty in pp["attrs"].items():
                t = p.state_tensor(a, dev)
                if t.dtype != tdtype[ty]:
                    t = t.to(tdtype[ty])
                if not t.is_contiguous():
                    t = t.contiguous()
                p._state[a] = t
                setattr(P, f"s_{a}", t.data_ptr())
            P.bits, P.raster = self.bits[k].data_ptr(), self.rasters[k].data_ptr()
            P.off, P.raster_off = self.offs[k].data_ptr(), self.raster_offs[k].data_ptr()
            P.raster_steps, P.rec0 = self.record_rows, self.rec_step0
            P.err = self.err[k:].data_ptr()
            P.counters = self.counters_t[k].data_ptr()
            bad = 0
            forms.append([])
            for ci, c in enumerate(pp["conns"]):
                s = c["src"]
                have = {f for f, _ in pp["fields"] if f.startswith(f"c{ci}_")}
                ptr = self._dev(c["ptr"])
                setattr(P, f"c{ci}_ptr", ptr.data_ptr())
                if f"c{ci}_link" in have:
                    link = self._dev(c["link"] if c["link"].numel() else torch.zeros(1, dtype=torch.int32))
                    values = {"link": link.data_ptr(), "src_bits": self.bits[s].data_ptr(), "src_words": words[s],
                              "src_mask": depth[s] - 1, "src_off": self.offs[s].data_ptr(),
                              "src_n": plan["pops"][s]["n"]}
                    for name, v in values.items():
                        if f"c{ci}_{name}" in have:
                            setattr(P, f"c{ci}_{name}", v)
                if "outs" in pp:
                    f = arrival_form(ptr, c["link"].to(dev), plan["pops"][s]["n"], depth[s] - 1)
                    bad += f["bad"]
                    f["arr"] = torch.zeros(max(1, f["depth"] * f["words"]), dtype=torch.int32, device=dev)
                    self.keep += [f[x] for x in ("wptr", "out_ptr", "pos", "dly", "arr")]  # (dly may be None)
                    setattr(P, f"c{ci}_wptr", f["wptr"].data_ptr())
                    setattr(P, f"c{ci}_arr", f["arr"].data_ptr())
                    setattr(P, f"c{ci}_arr_words", f["words"])
                    setattr(P, f"c{ci}_arr_depth", f["depth"])
                    forms[k].append(f)
                for e, v in c["per_link"].items():
                    v = self._dev(v if v.numel() else torch.zeros(1))
                    self.edge_arrays[(c["conn_id"], e)] = (v, c["perm"])
                    setattr(P, f"c{ci}_e_{e}", v.data_ptr())
            if "outs" in pp:
                P.bad = bad
            self.params.append(P)
        for P, pp in zip(self.params, plan["pops"]):
            for o, (tgt, ci) in enumerate(pp.get("outs", ())):
                f = forms[tgt][ci]
                P.outs[o] = arrival.Out(ptr=f["out_ptr"].data_ptr(), pos=f["pos"].data_ptr(),
                                        dly=f["dly"].data_ptr() if f["dly"] is not None else None,
                                        arr=f["arr"].data_ptr(), words=f["words"], depth=f["depth"])
        self.window = self.window_kernel = None  # the window kernel and its parameter block
        self.window_grid = sum(arrival.blocks_of(p["n"]) for p in plan["pops"])
        self.bar = torch.zeros(64, dtype=torch.int32, device=dev)  # its grid barrier (N2Grid)
        if window_kernel is not None:
            self._window(plan["window"], window_kernel)
        self.stream = torch.cuda.Stream(device=dev)
        self._s = ctypes.c_void_p(self.stream.cuda_stream)
        self.launches = 0

    def _compiled(self, plan: dict, scanning, dindex: int) -> tuple:
        """(the plan's form to run, its window kernel or None, else its step kernels). The window kernel where it
        compiles, its parameters fit and the device holds all its blocks at once; else a kernel per population, of the
        scanning intake where those of the arrival bits do not compile or their parameters do not fit."""
        types = [_params_struct(tuple(p["fields"])) for p in plan["pops"]]
        if scanning and any(ctypes.sizeof(t) > PARAMS_BYTES for t in types):
            return self._compiled(scanning(), None, dindex)
        if "window" in plan and ctypes.sizeof(_window_type(plan["window"], types)) <= arrival.WINDOW_PARAMS:
            try:
                kern, blocks = compile_source(plan["window"]["source"], dindex, b"n2b_user_window"), ctypes.c_int32()
                _lib.check(_lib.load().n2b_jit_resident_blocks(kern, arrival.THREADS, ctypes.byref(blocks)),
                           "n2b_jit_resident_blocks")
                if blocks.value >= sum(arrival.blocks_of(p["n"]) for p in plan["pops"]):
                    return plan, kern, []
            except RuntimeError as e:
                warnings.warn(f"no window kernel ({e}): one launch per population and step", stacklevel=4)
        try:
            return plan, None, [compile_source(p["source"], dindex) for p in plan["pops"]]
        except RuntimeError as e:
            if not scanning or not any("outs" in p for p in plan["pops"]):
                raise
            warnings.warn(f"no arrival bits ({e}): every link's source is looked up", stacklevel=4)
            return self._compiled(scanning(), None, dindex)

    def _window(self, plan: dict, kern: ctypes.c_void_p) -> None:
        """The window kernel's parameter block."""
        self.window_kernel, self.window = kern, _window_type(plan, [type(P) for P in self.params])()
        self.window.dt = self.dt
        self.window.grid.bar = self.bar.data_ptr()
        self.window_slots = []  # per population in the block's order: (its index, its kind, its place among them)
        for g, count in enumerate(plan["counts"]):
            self.window_slots += [(plan["order"][len(self.window_slots) + i], g, i) for i in range(count)]
        for at, (k, _, _) in enumerate(self.window_slots):
            self.window.first[at + 1] = self.window.first[at] + arrival.blocks_of(self.plan["pops"][k]["n"])

    def _dev(self, t):
        t = t.to(self.device).contiguous()
        self.keep.append(t)
        return t

    # ------------------------------------------------------------------ stepping

    def advance(self, n_steps: int) -> None:
        """Steps step_count .. step_count + n_steps - 1: a launch of the window kernel per WINDOW_STEPS or, without it, per step one
        launch per population, in order, the whole window in one library call (n2b_jit_launch_window writes each
        launch's step and times)."""
        n_steps = int(n_steps)
        if n_steps <= 0:
            return
        self.stream.wait_stream(torch.cuda.current_stream(self.device))
        step = self.net.step_count
        if self.window is not None:
            self._advance_window(step, n_steps)
        else:
            self._advance_steps(step, n_steps)
        last = step + n_steps - 1
        for P in self.params:  # (the fields as the last launch had them)
            P.step, P.t, P.t0 = last, (last + 1) * self.dt, last * self.dt
        torch.cuda.current_stream(self.device).wait_stream(self.stream)

    def _advance_window(self, step: int, n_steps: int) -> None:
        lib, W = _lib.load(), self.window
        W.grid.limit_ns = int(getattr(self.net, "barrier_limit_ns", 0) or BARRIER_LIMIT_NS)
        for k, g, i in self.window_slots:
            getattr(W, f"p{g}")[i] = self.params[k]
        for first in range(0, n_steps, WINDOW_STEPS):
            W.step0, W.n_steps = step + first, min(WINDOW_STEPS, n_steps - first)
            _lib.check(lib.n2b_jit_launch_cooperative(self.window_kernel, self.window_grid, arrival.THREADS,
                                                      ctypes.addressof(W), ctypes.sizeof(W), self._s),
                       "n2b_jit_launch_cooperative")
            self.launches += 1

    def _advance_steps(self, step: int, n_steps: int) -> None:
        k = len(self.kernels)
        grids, blocks = (ctypes.c_uint32 * k)(), (ctypes.c_uint32 * k)()
        kerns, params, sizes = (ctypes.c_void_p * k)(), (ctypes.c_void_p * k)(), (ctypes.c_size_t * k)()
        for i, (kern, P, pp) in enumerate(zip(self.kernels, self.params, self.plan["pops"])):
            size = pp["n"]
            if "outs" in pp:
                per, blocks[i] = arrival.NPB_C, arrival.THREADS
            elif self.exact:
                per, blocks[i] = BLOCK, BLOCK
            else:
                per, blocks[i] = NPB_C, scan(size) * NPB_C
            grids[i] = (size + per - 1) // per
            kerns[i] = kern.value
            params[i] = ctypes.addressof(P)
            sizes[i] = ctypes.sizeof(P)
        _lib.check(_lib.load().n2b_jit_launch_window(kerns, grids, blocks, params, sizes, k, step, n_steps, self.dt,
                                                     self._s), "n2b_jit_launch_window")
        self.launches += n_steps * sum(1 for g in grids if g)

    def start_recording(self, steps: int) -> None:
        if self.record_rows == 0 or steps > self.record_rows:
            raise RuntimeError("recording needs Network.record(steps) before the first step "
                               f"(this runtime keeps {self.record_rows} rows)")
        self.rec_step0 = self.net.step_count
        for P in self.params:
            P.rec0 = self.rec_step0

    # ------------------------------------------------------------------ results

    def raster_words(self, pop) -> np.ndarray:
        k = self.pops.index(pop)
        words = self.words[k]
        rows = min(self.record_rows, self.net.step_count - self.rec_step0)
        if rows <= 0:
            return np.zeros((0, words), dtype=np.uint32)
        self.stream.synchronize()
        return self.rasters[k][: rows * words].cpu().numpy().view(np.uint32).reshape(rows, words)

    def raster(self, pop) -> np.ndarray:
        w = self.raster_words(pop)
        n = len(pop.shape)
        bits = np.unpackbits(w.view(np.uint8).reshape(len(w), -1, 4), axis=2, bitorder="little")
        return bits.reshape(len(w), -1)[:, :n].astype(bool)

    def spikes(self, pop):
        steps, ids = np.nonzero(self.raster(pop))
        return steps.astype(np.int64) + self.rec_step0, ids.astype(np.int64)

    def edge_state(self, conn, name: str) -> torch.Tensor:
        """A per-link edge value (a weight the edge hooks change, ...) in canonical link order."""
        if (id(conn), name) not in self.edge_arrays:
            raise KeyError(f"{name} is not held per link on this connection")
        self.stream.synchronize()
        v, perm = self.edge_arrays[(id(conn), name)]
        out = torch.empty_like(v)
        if perm.numel():
            out[perm.to(v.device)] = v[: perm.numel()]
        return out[: perm.numel()]

    def spike_times(self, pop) -> tuple:
        """(times ms float32, neuron ids) of the recorded spikes: each spike's step start plus its time within
        the step (the end of the step for a spike of the clocked send; its own time in the event-driven intake)."""
        raster = self.raster(pop)
        steps, ids = np.nonzero(raster)
        k = self.pops.index(pop)
        n = len(pop.shape)
        offs = self.raster_offs[k][: len(raster) * n].cpu().numpy()
        o = offs[steps * n + ids]
        t0 = ((steps + self.rec_step0) * self.dt).astype(np.float32)
        return (t0 + o).astype(np.float32), ids.astype(np.int64)

    def status(self) -> list:
        self.stream.synchronize()
        return self.err.cpu().tolist()

    def check(self) -> None:
        bad = sum(self.status())
        if bad:
            raise RuntimeError(f"{bad} links with a delay outside their source's spike ring")
        stops = int(self.bar[33])
        if stops:
            raise RuntimeError(f"a window of steps stopped: {stops} grid barrier wait(s) gave up (the run is "
                               "incomplete; reset_counters clears the stop)")

    def counters(self) -> dict:
        self.stream.synchronize()
        c = self.counters_t.cpu().numpy()
        return {"events": int(c[:, 0].sum()), "spikes": int(c[:, 1].sum()),
                "per_population": [int(x) for x in c[:, 1]]}

    def reset_counters(self) -> None:
        self.stream.synchronize()
        self.counters_t.zero_()
        self.err.zero_()
        self.bar.zero_()

    def close(self) -> None:
        self.stream.synchronize()
        self.kernels = []


class PlannedPopulation:
    """A population as a plan describes it: its size, seed and state tensors, no model class."""

    def __init__(self, entry: dict, state: dict):
        self.name = entry["name"]
        self.shape = range(entry["n"])
        self.seed = entry["seed"]
        self._state = dict(state)

    def state_tensor(self, attr: str, device=None) -> torch.Tensor:
        t = self._state[attr]
        if device is not None and t.device != torch.device(device):
            t = self._state[attr] = t.to(device)
        return t

    def __repr__(self):
        return f"PlannedPopulation({self.name} x {len(self.shape)})"


class PlannedNetwork:
    """Steps a saved plan (plan_of / save_plan / load_plan): the step kernels of a transpiled network, run where
    its Python model classes are not. states: per population {attribute: tensor [n]} (the initial state)."""

    def __init__(self, plan: dict, states: list, device, record_steps: int = 0):
        self.device = torch.device(device)
        self.resolution = float(plan["dt"])
        self.exact = bool(plan["exact"])
        self.step_count = 0
        self.record_steps = int(record_steps)
        self.populations = [PlannedPopulation(p, st) for p, st in zip(plan["pops"], states)]
        self.runtime = JitRuntime(self, plan)

    def run_steps(self, n_steps: int) -> None:
        self.runtime.advance(n_steps)
        self.step_count += int(n_steps)

    def close(self) -> None:
        self.runtime.close()

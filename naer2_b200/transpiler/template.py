"""The step-kernel template of a transpiled population (reference naer2/transpiler/templates/fused_template.py:
85-371, the Gluon kernel it fills: pull -> deliver -> update/send -> emit).

One launch per population per step n (time t = (n + 1) dt, the end of the step), 32 neurons per block; clocked
intake: scan(n) threads per neuron (the neuron's first thread runs its hooks); exact-time intake: one thread per
neuron, three more warps for the deliveries.
  1. intake and receive: for each incoming connection (in the network's order), the neuron's pull row (its
     incoming links, canonical order within the row); a link whose source spiked at step n - d runs the
     connection's receive hook once, with its per-link edge values, in link order. Which links those are is read
     from the connection's arrival bits: one bit per incoming link and arrival slot n mod D, every row starting a
     word of its own, set by the spikes' deliveries and cleared here (clocked: the SCAN threads list the arrivals
     of their share of the row's words, the hooks then run over the lists);
  2. update, then send (n2.spike() anywhere marks the neuron as firing at step n);
  3. the spike-bit word of the block's 32 neurons into the population's spike-bit ring slot n mod depth (and the
     raster), the state back to memory, and the spike / arrival counters;
  4. delivery: the block's spikes set the arrival bits of their outgoing links (link by delay d: slot
     (n + d) mod D), one 32-bit reduction per link.
A step's work is its spikes' links and one bit per link of the intake; a kernel that looks every incoming link's
source up in its spike ring (the form `arrivals=False`, kept for networks whose arrival bits would not fit, see
runtime.ARRIVAL_BYTES) reads 32 times that. Measured, us per step, links looked up -> arrival bits: 12,500 neurons
of 1,250 links (47 spikes a step) 92 -> 19; 1,501 neurons of 150 plastic links 33 -> 11 (a fired neuron's edge
backward hooks by a group of warps instead of its one thread); 3,001 event-driven neurons of 125 links 73 -> 36.
What remains is the chain of one step: two launches of memory latencies.
The source is self-contained (NVRTC compiles it with no includes); its one parameter is the `Params` block,
mirrored field by field by the ctypes structure `params_type` builds, so that the host fills it directly.
"""

from __future__ import annotations

import ctypes

from .cuda import HookContext, lower_hook

_PRELUDE = r'''
typedef unsigned int u32;
typedef unsigned long long u64;

// Philox4x32-10 (Salmon et al., SC 2011): the first output word of counter (c0..c3) under key (k0, k1).
__device__ __forceinline__ u32 n2_philox_w0(u32 c0, u32 c1, u32 c2, u32 c3, u32 k0, u32 k1) {
    #pragma unroll
    for (int r = 0; r < 10; ++r) {
        const u32 h0 = __umulhi(0xD2511F53u, c0), l0 = 0xD2511F53u * c0;
        const u32 h1 = __umulhi(0xCD9E8D57u, c2), l1 = 0xCD9E8D57u * c2;
        const u32 n0 = h1 ^ c1 ^ k0, n2 = h0 ^ c3 ^ k1;
        c0 = n0; c1 = l1; c2 = n2; c3 = l0;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    return c0;
}

// Python's % on floats: the result takes the sign of the divisor.
__device__ __forceinline__ float n2_pymod(float a, float b) {
    float r = fmodf(a, b);
    if (r != 0.f && ((r < 0.f) != (b < 0.f))) r += b;
    return r;
}
'''


def ctype_of(py) -> tuple[str, object, object]:
    """(C type, ctypes type, torch dtype) of a dynamic attribute's Python type."""
    import torch

    if py is bool:
        return "bool", ctypes.c_bool, torch.bool
    if py is int:
        return "int", ctypes.c_int32, torch.int32
    return "float", ctypes.c_float, torch.float32


NPB_C = 32  # neurons per block (one spike-bit word); clocked intake: scan(n) * NPB_C threads
EXACT_THREADS = 128  # exact-time intake over arrival bits: the block's threads (the first NPB_C run the hooks)
LIST_WORDS = 4096  # clocked intake: the block's arrival lists (u32), SCAN * CAP per neuron
OUT_CACHED = 8  # outgoing connections whose row bounds a block loads ahead of its spikes

# The outgoing rows of one connection, as its source's kernel delivers along them.
_DELIVER = r'''
struct N2Out {
    const int *ptr;            // rows per source neuron
    const u32 *pos;            // per link: its bit among a slot's words
    const unsigned char *dly;  // per link: its delay in steps
    u32 *arr;                  // the arrival bits, [mask + 1][words]
    long long words;
    int mask, pad;
};

// The links of one row r0 .. r1, strided over `nthr` threads (this one `at`): set each link's bit in the arrival
// slot of its step. Four links' loads are in flight before their reductions: a row is a chain of memory
// latencies, not of bandwidth.
__device__ __forceinline__ void n2_deliver(const N2Out &o, long long n, int r0, int r1, int at, int nthr) {
    for (int l = r0 + at; l < r1; l += 4 * nthr) {
        u32 pos[4], d[4];
        #pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int q = l + k * nthr;
            d[k] = q < r1 ? o.dly[q] : 0u;
            pos[k] = q < r1 ? o.pos[q] : 0u;
        }
        #pragma unroll
        for (int k = 0; k < 4; ++k)
            if (d[k]) atomicOr(o.arr + (size_t)((n + d[k]) & o.mask) * o.words + (pos[k] >> 5), 1u << (pos[k] & 31u));
    }
}
'''


def deliver_code(n_out: int, threads: int) -> str:
    """The block's deliveries: `fw` holds its spiking neurons' bits. Every (spike, connection) row is walked by one
    warp or, with fewer rows than warps, by a group of them (a power of two), so that a row of 1,000 links is a
    few loads per lane whatever the block's spikes."""
    if not n_out:
        return ""
    cached = min(n_out, OUT_CACHED)
    rows = ("const int r0 = o < {0} ? n2_optr[o][q] : O.ptr[jq], r1 = o < {0} ? n2_optr[o][q + 1] : O.ptr[jq + 1];"
            .format(cached) if n_out > cached else "const int r0 = n2_optr[o][q], r1 = n2_optr[o][q + 1];")
    return f"""    // the spikes' outgoing rows
{_rows_loop(f"__popc(fw) * {n_out}", threads)}        const int o = i % {n_out};
        u32 m = fw;
        for (int k = i / {n_out}; k > 0; --k) m &= m - 1;
        const int q = __ffs(m) - 1, jq = (int)blockIdx.x * NPB_C + q;
        const N2Out &O = p.outs[o];
        {rows}
        n2_deliver(O, n, r0, r1, (int)threadIdx.x % (32 * g), 32 * g);
    }}
    }}
"""


def _rows_loop(rows: str, threads: int) -> str:
    """The head of a block's loop over `rows` rows (i), each by a group of g warps (fewer rows than warps) or one."""
    return f"""    if (fw) {{
    const int rows = {rows};
    int g = 1;
    while (2 * g * rows <= {threads // 32}) g *= 2;
    for (int i = (int)(threadIdx.x >> 5) / g; i < rows; i += {threads // 32} / g) {{
"""


def out_rows_code(n_out: int, threads: int) -> str:
    """The row bounds of the block's neurons in its first OUT_CACHED outgoing connections, loaded under the intake."""
    cached = min(n_out, OUT_CACHED)
    if not cached:
        return ""
    return f"""    __shared__ int n2_optr[{cached}][NPB_C + 1];
    for (int k = threadIdx.x; k < {cached} * (NPB_C + 1); k += {threads}) {{
        const int q = k % (NPB_C + 1);
        n2_optr[k / (NPB_C + 1)][q] = p.outs[k / (NPB_C + 1)].ptr[min((int)blockIdx.x * NPB_C + q, p.n)];
    }}
"""


MAX_ARRIVALS = 64  # exact-time intake: arrivals a neuron can hold in one step (more are counted, dropped)


def _arrival_body(pop_name: str, c: int, inc: dict) -> str:
    """One arrival of connection c: the link's edge values, edge forward, receive, edge values stored."""
    body = ""
    if inc.get("forward") is not None:
        fn, ctx = inc["forward"]
        body += lower_hook(fn, ctx, f"{pop_name} edge forward (connection {c})")
    body += "".join(f"const float e_{h} = e_{real};\n" for h, real in inc.get("alias", {}).items())
    if inc["receive"] is not None:
        fn, ctx = inc["receive"]
        body += lower_hook(fn, ctx, f"{pop_name} receive (connection {c})")
    body += "".join(f"p.c{c}_e_{e}[l] = e_{e};\n" for e in inc.get("edge_written", ()))
    return body


def scan(n: int) -> int:
    """Clocked intake: threads scanning one neuron's incoming row, for a population of n neurons (more for small
    populations, so that their blocks still fill the GPU)."""
    return 32 if n <= 4096 else 8


ROWS_AHEAD = 8  # incoming connections whose row bounds a thread loads ahead of its step


def _prologue(incoming: list, live: str, row: str) -> str:
    """Before anything the previous launch wrote is read: the next launch may be scheduled and this one's static row
    bounds are loaded while the previous launch is still running (n2b_jit_launch_window launches such kernels
    with programmatic stream serialization); griddepcontrol.wait returns once it has finished."""
    out = ['    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");\n']
    for c, inc in enumerate(incoming[:ROWS_AHEAD]):
        if inc["receive"] is not None or inc.get("forward") is not None:
            out.append(f"    const int c{c}_r0 = {live} ? p.c{c}_ptr[{row}] : 0, c{c}_w0 = {live} ? p.c{c}_wptr[{row}] : 0, "
                       f"c{c}_w1 = {live} ? p.c{c}_wptr[{row} + 1] : 0;\n")
    return "".join(out)


def _row_bounds(c: int, live: str, row: str) -> str:
    if c < ROWS_AHEAD:
        return f"const int r0 = c{c}_r0, w0 = c{c}_w0, w1 = c{c}_w1;"
    return (f"const int r0 = {live} ? p.c{c}_ptr[{row}] : 0, w0 = {live} ? p.c{c}_wptr[{row}] : 0, "
            f"w1 = {live} ? p.c{c}_wptr[{row} + 1] : 0;")


_WAIT = '    asm volatile("griddepcontrol.wait;" ::: "memory");\n'


def _scan_intake(c: int, arrival: str) -> str:
    """Connection c's arrivals without arrival bits: the SCAN threads look their row segment's sources up in the
    spike ring and list the arrivals; the owner runs the hooks over the lists (a segment with more than CAP
    arrivals is walked again, link by link)."""
    hit = (f"(p.c{c}_src_bits[(size_t)(m & p.c{c}_src_mask) * p.c{c}_src_words + (src >> 5)] >> (src & 31)) & 1u")
    at = arrival.replace("\n", "\n                        ").rstrip() + "\n"
    return f"""    {{  // connection {c}: scan
        const int r0 = live ? p.c{c}_ptr[j] : 0, r1 = live ? p.c{c}_ptr[j + 1] : 0;
        const int seg = (r1 - r0 + SCAN - 1) / SCAN;
        const int a = min(r1, r0 + sc * seg), b = min(r1, a + seg);
        int cnt = 0;
        for (int l = a; l < b; ++l) {{
            const u32 w = p.c{c}_link[l];
            const int src = (int)(w & 0xFFFFFFu), d = (int)(w >> 24);
            if (d < 1 || d > p.c{c}_src_mask) {{ atomicAdd(p.err, 1); continue; }}
            const long long m = n - d;
            if (m < 0 || !({hit})) continue;
            if (cnt < CAP) s_list[(jl * SCAN + sc) * CAP + cnt] = (u32)l;
            ++cnt;
        }}
        s_cnt[jl * SCAN + sc] = cnt;
        __syncthreads();
        if (live && own) {{  // the hooks, in link order
            for (int s = 0; s < SCAN; ++s) {{
                const int cs = s_cnt[jl * SCAN + s];
                if (cs <= CAP) {{
                    for (int i = 0; i < cs; ++i) {{
                        const int l = (int)s_list[(jl * SCAN + s) * CAP + i];
                        {at}                    }}
                }} else {{  // the segment again, one link at a time
                    const int as = min(r1, r0 + s * seg), bs = min(r1, as + seg);
                    for (int l = as; l < bs; ++l) {{
                        const u32 w = p.c{c}_link[l];
                        const int src = (int)(w & 0xFFFFFFu), d = (int)(w >> 24);
                        if (d < 1 || d > p.c{c}_src_mask) continue;
                        const long long m = n - d;
                        if (m < 0 || !({hit})) continue;
                        {at}                    }}
                }}
            }}
        }}
        link_k = 0xFFFFFFu;
        __syncthreads();  // the lists are rewritten by the next connection
    }}
"""


def _bits_intake(c: int, arrival: str) -> str:
    """Connection c's arrivals from its arrival bits: each of the neuron's SCAN threads (neighbouring lanes of a
    warp) takes a run of the row's words, four loads in flight, lists the links of its set bits and clears them,
    as long as its list holds a whole word's; the words after that stay set for the owner, which runs the hooks
    over the lists in word order and then over such words, i.e. in link order throughout."""
    at = arrival.replace("\n", "\n                    ").rstrip() + "\n"
    return f"""    {{  // connection {c}: its arrival bits
        {_row_bounds(c, "live", "j")}
        u32 *arr = p.c{c}_arr + (size_t)(n & p.c{c}_arr_mask) * p.c{c}_arr_words;
        const int seg = (w1 - w0 + SCAN - 1) / SCAN;
        const int a = min(w1, w0 + sc * seg), b = min(w1, a + seg);
        u32 *list = s_list + (jl * SCAN + sc) * CAP;
        int cnt = 0;
        bool left = false;  // words left for the owner
        for (int k = a; k < b; k += 4) {{
            u32 x[4];
            #pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = k + i < b ? __ldcg(arr + k + i) : 0u;
            #pragma unroll
            for (int i = 0; i < 4; ++i) {{
                left = left || (x[i] && cnt + __popc(x[i]) > CAP);
                if (!x[i] || left) continue;
                for (u32 v = x[i]; v; v &= v - 1) list[cnt++] = (u32)(r0 + 32 * (k + i - w0) + __ffs(v) - 1);
                arr[k + i] = 0u;
            }}
        }}
        s_cnt[jl * SCAN + sc] = left ? ~cnt : cnt;
        const u32 some = __ballot_sync(0xffffffffu, cnt || left);  // also orders the lists before the owner's reads
        __syncwarp();
        if (live && own) {{  // the hooks, in link order
            for (u32 segs = (some >> (threadIdx.x & 31)) & (u32)((1ull << SCAN) - 1); segs; segs &= segs - 1) {{
                const int s = __ffs(segs) - 1;
                const int cs = s_cnt[jl * SCAN + s], listed = cs < 0 ? ~cs : cs;
                for (int i = 0; i < listed; ++i) {{
                    const int l = (int)s_list[(jl * SCAN + s) * CAP + i];
                    {at}                }}
                if (cs >= 0) continue;
                const int as = min(w1, w0 + s * seg), bs = min(w1, as + seg);
                for (int k = as; k < bs; ++k) {{
                    u32 v = __ldcg(arr + k);  // (the listed words are clear)
                    if (v) arr[k] = 0u;
                    for (; v; v &= v - 1) {{
                    const int l = r0 + 32 * (k - w0) + __ffs(v) - 1;
                    {at}                    }}
                }}
            }}
        }}
        link_k = 0xFFFFFFu;
        __syncwarp();  // the lists are rewritten by the next connection
    }}
"""


def _clocked_kernel(pop_name: str, attrs: dict, hooks: dict, incoming: list, n: int, arrivals: bool,
                    n_out: int) -> str:
    """The clocked step kernel: SCAN threads per neuron find the step's arrivals of each incoming connection
    (`_bits_intake`, or `_scan_intake` without arrival bits) and list them in shared memory; the neuron's first
    thread (the owner) runs the hooks over the lists in segment order, i.e. in link order, with the same arrival
    numbers and draws as one link at a time. SCAN = scan(n), CAP = LIST_WORDS / (NPB_C * SCAN). Edge backward
    hooks that assign nothing of the destination are run for a fired neuron's links by the whole block (a link's
    hook touches that link alone), the others by the owner, link by link."""
    SCAN = scan(n)
    CAP = LIST_WORDS // (NPB_C * SCAN)
    threads = SCAN * NPB_C
    src = [f"constexpr int SCAN = {SCAN}, NPB_C = {NPB_C}, CAP = {CAP};\n\n"]
    src.append(f'// population {pop_name}\nextern "C" __global__ void __launch_bounds__({threads}) '
               "n2b_user_step(const __grid_constant__ Params p) {\n")
    src.append("""    __shared__ u32 s_list[NPB_C * SCAN * CAP];
    __shared__ int s_cnt[NPB_C * SCAN];
    __shared__ u32 s_word, s_arrivals;
    const int jl = threadIdx.x / SCAN, sc = threadIdx.x % SCAN;
    const int j = blockIdx.x * NPB_C + jl;
    const bool live = j < p.n, own = sc == 0;
    const long long n = p.step;
    const float t = p.t;
    bool fired = false;
    float spike_t = t;
    u32 arrived = 0;
    u32 link_k = 0xFFFFFFu;
    if (threadIdx.x == 0) { s_word = 0u; s_arrivals = 0u; }
""")
    if arrivals:
        src.append(_prologue(incoming, "live", "j"))
        src.append(out_rows_code(n_out, threads))
        src.append(_WAIT)
        src.append("    if (p.bad && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(p.err, p.bad);\n")
    for a, py in attrs.items():
        ct, _, _ = ctype_of(py)
        src.append(f"    {ct} s_{a} = (live && own) ? p.s_{a}[j] : ({ct})0;\n")
    src.append("    __syncthreads();\n")
    for c, inc in enumerate(incoming):
        if inc["receive"] is None and inc.get("forward") is None:
            continue
        loads = "".join(f"float e_{e} = p.c{c}_e_{e}[l];\n" for e in inc["edge_dynamic"])
        arrival = loads + "link_k = arrived++;\n" + "{\n" + _arrival_body(pop_name, c, inc) + "}\n"
        src.append((_bits_intake if arrivals else _scan_intake)(c, arrival))
    src.append("    if (live && own) {\n")
    for name in ("update", "send"):
        fn, ctx = hooks[name]
        body = lower_hook(fn, ctx, f"{pop_name} {name}")
        src.append("        " + body.replace("\n", "\n        ").rstrip() + "\n")
    backward = [(c, inc) for c, inc in enumerate(incoming) if inc.get("backward") is not None]
    shared = arrivals and backward and not any(inc.get("backward_writes", True) for _, inc in backward)
    if backward and not shared:  # the neuron fired: every incoming link's edge backward hook at its spike's time
        src.append("        if (fired) {\n            const float t = spike_t;\n")
        for c, inc in backward:
            src.append(_backward_loop(pop_name, c, inc, "j", "0", "1", " " * 12))
        src.append("        }\n")
    src.append("""        if (fired) {
            const float o = spike_t - p.t0;  // the spike's time within its step
            p.off[(size_t)(n & p.bit_mask) * p.n + j] = o;
            const long long r = n - p.rec0;
            if (p.raster_off && r >= 0 && r < p.raster_steps) p.raster_off[(size_t)r * p.n + j] = o;
            atomicOr(&s_word, 1u << jl);
        }
        if (arrived) atomicAdd(&s_arrivals, arrived);
    }
""")
    if shared:  # what the backward hooks read of the fired neurons
        read = [a for a in attrs if any(f"s_{a}" in _backward_body(pop_name, c, inc) for c, inc in backward)]
        src.append("    __shared__ float n2_spike_t[NPB_C];\n")
        for a in read:
            src.append(f"    __shared__ {ctype_of(attrs[a])[0]} n2d_{a}[NPB_C];\n")
        src.append("    if (fired) {\n        n2_spike_t[jl] = spike_t;\n")
        src += [f"        n2d_{a}[jl] = s_{a};\n" for a in read]
        src.append("    }\n")
    src.append("""    __syncthreads();
    const u32 fw = s_word;
    if (threadIdx.x == 0) {  // the block's 32 neurons: one spike-bit word
        const int word = blockIdx.x;
        if (word < p.words) {
            p.bits[(size_t)(n & p.bit_mask) * p.words + word] = fw;
            const long long r = n - p.rec0;
            if (p.raster && r >= 0 && r < p.raster_steps) p.raster[(size_t)r * p.words + word] = fw;
        }
        if (fw) atomicAdd(p.counters + 1, (u64)__popc(fw));
        if (s_arrivals) atomicAdd(p.counters, (u64)s_arrivals);
    }
""")
    for a in attrs:
        src.append(f"    if (live && own) p.s_{a}[j] = s_{a};\n")
    if arrivals:
        src.append(deliver_code(n_out, threads))
    if shared:
        src.append("    // the fired neurons' incoming links: edge backward at the spike's time\n")
        src.append(_rows_loop("__popc(fw)", threads))
        src.append("""        u32 m = fw;
        for (int k = i; k > 0; --k) m &= m - 1;
        const int q = __ffs(m) - 1, jq = (int)blockIdx.x * NPB_C + q;
        const float t = n2_spike_t[q];
""")
        src += [f"        const {ctype_of(attrs[a])[0]} s_{a} = n2d_{a}[q];\n" for a in read]
        for c, inc in backward:
            src.append(_backward_loop(pop_name, c, inc, "jq", "(int)threadIdx.x % (32 * g)", "32 * g", " " * 8))
        src.append("    }\n    }\n")
    src.append("}\n")
    return "".join(src)


def _backward_body(pop_name: str, c: int, inc: dict) -> str:
    fn, ctx = inc["backward"]
    return (lower_hook(fn, ctx, f"{pop_name} edge backward (connection {c})") +
            "".join(f"p.c{c}_e_{e}[l] = e_{e};\n" for e in inc.get("edge_written", ())))


def _backward_loop(pop_name: str, c: int, inc: dict, j: str, first: str, step: str, pad: str) -> str:
    """Connection c's edge backward hook over the incoming links of neuron `j`: first, first + step, ..."""
    loads = "".join(f"{pad}    float e_{e} = p.c{c}_e_{e}[l];\n" for e in inc["edge_dynamic"])
    body = _backward_body(pop_name, c, inc).replace("\n", f"\n{pad}    ").rstrip()
    return (f"{pad}for (int l = p.c{c}_ptr[{j}] + {first}; l < p.c{c}_ptr[{j} + 1]; l += {step}) {{\n{loads}"
            f"{pad}    {body}\n{pad}}}\n")


def build_source(pop_name: str, attrs: dict, hooks: dict, incoming: list, exact: bool = False,
                 n: int = 1 << 30, arrivals: bool = False, n_out: int = 0) -> tuple[str, list]:
    """(CUDA source, params fields [(name, C type, ctypes type)]) of one population.

    attrs: dynamic attr -> python type; hooks: {"update": (fn_ast, ctx), "send": (fn_ast, ctx)};
    incoming: one dict per incoming connection: "receive": (fn_ast, ctx) or None; "edge_dynamic": the per-link
    arrays by the edge's own attribute names; "edge_written": those the edge hooks assign (stored back);
    "alias": {receive-facing name: edge name} where they differ; "forward" / "backward": (fn_ast, ctx) of the
    edge hooks or None; "backward_writes": whether the backward hook assigns the destination's state.

    n: the population's size (the clocked intake's threads per neuron, `scan(n)`).

    arrivals: the intake reads the connections' arrival bits, which the spikes' deliveries set (`n_out`: the
    population's outgoing connections, Params.outs); otherwise every incoming link's source is looked up.

    exact: event-driven intake at exact times. Every spike carries its time (its offset in its step, in the
    population's offset ring); a link of delay d delivers it at that time plus d steps. A neuron collects its
    arrivals of the step, sorts them by time (stable: connection order, then link order, among equal times),
    runs receive (and edge forward) for each at its own time and send after each group of equal times; then
    update and send at the end of the step, as in the clocked intake."""
    fields = [("step", "long long", ctypes.c_int64), ("rec0", "long long", ctypes.c_int64),
              ("raster_steps", "long long", ctypes.c_int64), ("t", "float", ctypes.c_float),
              ("t0", "float", ctypes.c_float),
              ("n", "int", ctypes.c_int32), ("words", "int", ctypes.c_int32), ("bit_mask", "int", ctypes.c_int32),
              ("seed_lo", "u32", ctypes.c_uint32), ("seed_hi", "u32", ctypes.c_uint32)]
    for a, py in attrs.items():
        ct, cty, _ = ctype_of(py)
        fields.append((f"s_{a}", f"{ct} *", ctypes.c_void_p))
    fields += [("bits", "u32 *", ctypes.c_void_p), ("off", "float *", ctypes.c_void_p),
               ("raster", "u32 *", ctypes.c_void_p), ("raster_off", "float *", ctypes.c_void_p),
               ("err", "int *", ctypes.c_void_p),
               ("counters", "u64 *", ctypes.c_void_p)]
    if arrivals:
        fields.append(("bad", "int", ctypes.c_int32))  # incoming links out of range: counted every step
    for c, inc in enumerate(incoming):
        fields.append((f"c{c}_ptr", "const int *", ctypes.c_void_p))
        if arrivals:
            fields += [(f"c{c}_wptr", "const int *", ctypes.c_void_p), (f"c{c}_arr", "u32 *", ctypes.c_void_p),
                       (f"c{c}_arr_words", "long long", ctypes.c_int64), (f"c{c}_arr_mask", "int", ctypes.c_int32)]
        else:
            fields += [(f"c{c}_src_bits", "const u32 *", ctypes.c_void_p), (f"c{c}_src_words", "int", ctypes.c_int32)]
        if exact or not arrivals:
            fields += [(f"c{c}_link", "const u32 *", ctypes.c_void_p),
                       (f"c{c}_src_off", "const float *", ctypes.c_void_p),
                       (f"c{c}_src_mask", "int", ctypes.c_int32), (f"c{c}_src_n", "int", ctypes.c_int32)]
        for e in inc["edge_dynamic"]:
            fields.append((f"c{c}_e_{e}", "float *" if e in inc.get("edge_written", ()) else "const float *",
                           ctypes.c_void_p))
    if arrivals and n_out:
        fields.append(("outs", f"N2Out[{n_out}]", Out * n_out))

    src = [_PRELUDE]
    if arrivals:
        src.append(_DELIVER)
    src.append("struct Params {\n")
    for name, ct, _ in fields:
        src.append(f"    {ct.split('[')[0]} {name}{'[' + ct.split('[')[1] if '[' in ct else ''};\n")
    src.append("};\n\n")
    src.append(r'''// uniform in [0, 1): 24 bits of the draw for (neuron j, step n, call site, link k)
__device__ __forceinline__ float n2_uniform(const Params &p, int j, long long n, u32 site, u32 k) {
    const u32 w = n2_philox_w0((u32)j, (u32)n, (u32)((u64)n >> 32), (site << 24) | (k & 0xFFFFFFu), p.seed_lo,
                               p.seed_hi);
    return (float)(w >> 8) * 5.9604644775390625e-08f;
}

''')
    if not exact:
        src.append(_clocked_kernel(pop_name, attrs, hooks, incoming, n, arrivals, n_out))
        return "".join(src), fields
    # arrival bits: 32 neurons per block (one per lane of its first warp), the other warps for the deliveries only
    threads = EXACT_THREADS if arrivals else 128
    if arrivals:
        src.append(f"constexpr int NPB_C = {NPB_C};\n\n")
    src.append(f'// population {pop_name}\nextern "C" __global__ void __launch_bounds__({threads}) n2b_user_step('
               "const __grid_constant__ Params p) {\n")
    if arrivals:
        src.append("    const int j = blockIdx.x * NPB_C + (int)threadIdx.x;\n"
                   "    const bool live = threadIdx.x < NPB_C && j < p.n;\n")
    else:
        src.append("    const int j = blockIdx.x * blockDim.x + threadIdx.x;\n    const bool live = j < p.n;\n")
    src.append("    const long long n = p.step;\n    const float t = p.t;\n")
    src.append("    bool fired = false;\n    float spike_t = t;\n    u32 arrived = 0;\n    u32 link_k = 0xFFFFFFu;\n")
    if arrivals:
        src.append("    __shared__ u32 s_word;\n")
        src.append(_prologue(incoming, "live", "j"))
        src.append(out_rows_code(n_out, threads))
        src.append(_WAIT)
        src.append("    if (p.bad && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(p.err, p.bad);\n")
    for a, py in attrs.items():
        ct, _, _ = ctype_of(py)
        src.append(f"    {ct} s_{a} = live ? p.s_{a}[j] : ({ct})0;\n")
    src.append("    if (live) {\n")
    src.append(_exact_intake(pop_name, incoming, hooks, arrivals))
    for name in ("update", "send"):
        fn, ctx = hooks[name]
        body = lower_hook(fn, ctx, f"{pop_name} {name}")
        src.append("        " + body.replace("\n", "\n        ").rstrip() + "\n")
    backward = [(c, inc) for c, inc in enumerate(incoming) if inc.get("backward") is not None]
    if backward:  # the neuron fired: every incoming link's edge backward hook at its spike's time
        src.append("        if (fired) {\n            const float t = spike_t;\n")
        for c, inc in backward:
            src.append(_backward_loop(pop_name, c, inc, "j", "0", "1", " " * 12))
        src.append("        }\n")
    src.append("    }\n")
    src.append("""    if (live && fired) {
        const float o = spike_t - p.t0;  // the spike's time within its step
        p.off[(size_t)(n & p.bit_mask) * p.n + j] = o;
        const long long r = n - p.rec0;
        if (p.raster_off && r >= 0 && r < p.raster_steps) p.raster_off[(size_t)r * p.n + j] = o;
    }
""")
    word = "blockIdx.x" if arrivals else "j >> 5"
    if arrivals:
        src.append("    if (threadIdx.x < 32) {\n")
    src.append(f'''    const u32 b = __ballot_sync(0xffffffffu, live && fired);
    const u32 arrivals = __reduce_add_sync(0xffffffffu, arrived);
    if ((threadIdx.x & 31) == 0) {{
        const int word = {word};
        if (word < p.words) {{
            p.bits[(size_t)(n & p.bit_mask) * p.words + word] = b;
            const long long r = n - p.rec0;
            if (p.raster && r >= 0 && r < p.raster_steps) p.raster[(size_t)r * p.words + word] = b;
        }}
        if (b) atomicAdd(p.counters + 1, (u64)__popc(b));
        if (arrivals) atomicAdd(p.counters, (u64)arrivals);
    }}
''')
    if arrivals:
        src.append("    if (threadIdx.x == 0) s_word = b;\n    }\n")
    for a in attrs:
        src.append(f"    if (live) p.s_{a}[j] = s_{a};\n")
    if arrivals:
        src.append("    __syncthreads();\n    const u32 fw = s_word;\n")
        src.append(deliver_code(n_out, threads))
    src.append("}\n")
    return "".join(src), fields


def _exact_intake(pop_name: str, incoming: list, hooks: dict, arrivals: bool) -> str:
    """The event-driven intake: collect the step's arrivals with their times (from the connections' arrival bits, or
    by looking every incoming link's source up), sort, deliver in time order."""
    out = [f"""        float a_t[{MAX_ARRIVALS}];
        int a_c[{MAX_ARRIVALS}], a_l[{MAX_ARRIVALS}];
        int na = 0;
"""]
    for c, inc in enumerate(incoming):
        if inc["receive"] is None and inc.get("forward") is None:
            continue
        insert = f"""            const float tau = p.t0 + p.c{c}_src_off[slot * p.c{c}_src_n + src];
            if (na == {MAX_ARRIVALS}) {{ atomicAdd(p.err, 1); continue; }}
            int k = na++;
            while (k > 0 && a_t[k - 1] > tau) {{ a_t[k] = a_t[k - 1]; a_c[k] = a_c[k - 1]; a_l[k] = a_l[k - 1]; --k; }}
            a_t[k] = tau; a_c[k] = {c}; a_l[k] = l;
"""
        if arrivals:
            out.append(f"""        {{  // connection {c}: its arrival bits, four words in flight
        {_row_bounds(c, "true", "j")}
        u32 *arr = p.c{c}_arr + (size_t)(n & p.c{c}_arr_mask) * p.c{c}_arr_words;
        for (int wk = w0; wk < w1; wk += 4) {{
            u32 x[4];
            #pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = wk + i < w1 ? __ldcg(arr + wk + i) : 0u;
            #pragma unroll
            for (int i = 0; i < 4; ++i) {{
            if (x[i]) arr[wk + i] = 0u;
            for (u32 v = x[i]; v; v &= v - 1) {{
            const int l = r0 + 32 * (wk + i - w0) + __ffs(v) - 1;
            const u32 w = p.c{c}_link[l];
            const int src = (int)(w & 0xFFFFFFu), d = (int)(w >> 24);
            const size_t slot = (size_t)((n - d) & p.c{c}_src_mask);
{insert}            }}
            }}
        }}
        }}
""")
        else:
            out.append(f"""        for (int l = p.c{c}_ptr[j]; l < p.c{c}_ptr[j + 1]; ++l) {{
            const u32 w = p.c{c}_link[l];
            const int src = (int)(w & 0xFFFFFFu), d = (int)(w >> 24);
            if (d < 1 || d > p.c{c}_src_mask) {{ atomicAdd(p.err, 1); continue; }}
            const long long m = n - d;
            if (m < 0) continue;
            const size_t slot = (size_t)(m & p.c{c}_src_mask);
            if (!((p.c{c}_src_bits[slot * p.c{c}_src_words + (src >> 5)] >> (src & 31)) & 1u)) continue;
{insert}        }}
""")
    out.append("""        for (int i = 0; i < na;) {
            const float tau = a_t[i];
            int e = i;
            while (e < na && a_t[e] == tau) ++e;
            for (int k = i; k < e; ++k) {
                const int l = a_l[k];
                const float t = tau;
                link_k = arrived++;
                switch (a_c[k]) {
""")
    for c, inc in enumerate(incoming):
        if inc["receive"] is None and inc.get("forward") is None:
            continue
        loads = "".join(f"float e_{x} = p.c{c}_e_{x}[l];\n" for x in inc["edge_dynamic"])
        body = loads + _arrival_body(pop_name, c, inc)
        out.append(f"                case {c}: {{\n                    " +
                   body.replace("\n", "\n                    ").rstrip() + "\n                } break;\n")
    fn, ctx = hooks["send"]
    send = lower_hook(fn, ctx, f"{pop_name} send")
    out.append("""                default: break;
                }
            }
            {
                const float t = tau;
                """ + send.replace("\n", "\n                ").rstrip() + """
            }
            i = e;
        }
        link_k = 0xFFFFFFu;
""")
    return "".join(out)


class Out(ctypes.Structure):
    """One outgoing connection (the source's N2Out)."""
    _fields_ = [("ptr", ctypes.c_void_p), ("pos", ctypes.c_void_p), ("dly", ctypes.c_void_p),
                ("arr", ctypes.c_void_p), ("words", ctypes.c_int64), ("mask", ctypes.c_int32),
                ("pad", ctypes.c_int32)]


def params_type(fields: list):
    """The ctypes structure of a Params block."""
    return type("Params", (ctypes.Structure,), {"_fields_": [(name, cty) for name, _, cty in fields]})


def edge_hook_context(pop, hook, per_link: list, edge_static: dict) -> HookContext:
    """An edge hook's names: self = the link (per-link arrays, the edge's static values), the destination =
    the target neuron's state; the source's state and random draws are refused."""
    from .. import receives
    from .cuda import Root

    names = {ty: nm for ty, nm in hook.parameter_type_to_name.items()}
    static = {k: v for k, v in pop.instance.__dict__.items()
              if k not in pop.dynamic_attrs and isinstance(v, (int, float, bool))}
    roots = {"self": Root("e_", {n: float for n in per_link}, dict(edge_static), True, "the link")}
    if receives.destination in names:
        roots[names[receives.destination]] = Root("s_", dict(pop.dynamic_attrs), static, True,
                                                  "the destination neuron")
    return HookContext(time_name=names.get(receives.time), source_name=names.get(receives.source), roots=roots,
                       random=False)


def hook_context(pop, hook, edge_dynamic=(), edge_static=None, site_base: int = 0) -> HookContext:
    """The names a hook's body may use, from its signature and the population's attributes."""
    from .. import receives

    names = {ty: nm for ty, nm in hook.parameter_type_to_name.items()}
    static = {k: v for k, v in pop.instance.__dict__.items()
              if k not in pop.dynamic_attrs and isinstance(v, (int, float, bool))}
    return HookContext(self_attrs=dict(pop.dynamic_attrs), self_static=static,
                       time_name=names.get(receives.time), edge_name=names.get(receives.edge),
                       source_name=names.get(receives.source), edge_dynamic=set(edge_dynamic),
                       edge_static=dict(edge_static or {}), site_base=site_base)

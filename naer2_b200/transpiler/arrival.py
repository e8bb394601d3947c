"""The step kernels of a transpiled network over arrival bits: their CUDA source (template.py's other form looks
every incoming link's source up in its spike ring instead).

Per connection, one bit per incoming link and arrival slot n mod D, every pull row starting a word of its own. A
population's step n, 32 neurons per block, SCAN threads per neuron:
  1. intake and receive: for each incoming connection (in the network's order), the links whose bit of slot n is
     set, in link order, run the connection's hooks once each; the bits are cleared as they are read. Exact times:
     the arrivals of every connection are collected with their times, sorted, and delivered in time order;
  2. update, then send (n2.spike() anywhere marks the neuron as firing at step n), by the neuron's first thread;
  3. the spike-bit word of the block's 32 neurons into the population's spike-bit ring slot n mod depth (and the
     raster), and the spike / arrival counters;
  4. delivery: the block's spikes set the bits of their outgoing links (delay d: slot (n + d) mod D), one 32-bit
     reduction per link; a fired neuron's edge backward hooks run over its incoming links.
A step's work is its spikes' links and one bit per link of the intake; looking the links up reads 32 times that.

Two kernels run it. `n2b_user_step` (a population's `source`) is one step of one population. `n2b_user_window`
(`window_source`) is a window of steps of the whole network in one cooperative launch: every block keeps its 32
neurons' state in registers and its row bounds throughout, and the steps are separated by a grid barrier (bounded: a
wait that gives up sets an abort word, and the kernel winds down). A step is a chain of memory latencies, so what it
costs is the launches around it and the loads that a launch starts with. Measured, us per step, links looked up ->
arrival bits, one launch per population -> window: 12,500 neurons of 1,250 links (47 spikes a step) 92 -> 19.4 ->
8.3; 1,501 neurons of 150 plastic links 33 -> 11.2 -> 6.8; 3,001 event-driven neurons of 125 links 73 -> 36 ->
14.5.
"""

from __future__ import annotations

import ctypes

from .cuda import lower_hook
from .template import _PRELUDE, MAX_ARRIVALS, NPB_C, UNIFORM, _arrival_body, base_fields, ctype_of

SCAN = 8  # threads per neuron: a row of 1,250 links is 40 words, five to a thread
THREADS = NPB_C * SCAN
CAP = 16  # clocked intake: arrivals a thread lists of one connection (more stay in their words for the owner)
OUT_CACHED = 8  # outgoing connections whose row bounds a block holds in shared memory
PIECE = 256  # links of a row that a warp delivers at once, eight loads a lane in flight
WORDS_AHEAD = 4  # incoming connections whose arrival words are loaded together at a step's start
ROWS_AHEAD = 8  # incoming connections whose row bounds a thread holds
WINDOW_PARAMS = 16384  # bytes of a window kernel's parameter block at most
WINDOW_POPS = 16  # populations of a window kernel at most (each is a copy of the step's code)

_COMMON = r'''
struct N2Out {
    const int *ptr;            // rows per source neuron
    const u32 *pos;            // per link: its bit among a slot's words (dly null: its delay in the top 8 bits)
    const unsigned char *dly;  // per link: its delay in steps, of connections with more than 2^24 bits to a slot
    u32 *arr;                  // the arrival bits, [mask + 1][words]
    long long words;
    int mask, pad;
};

constexpr int SCAN = @SCAN@, NPB_C = @NPB@, CAP = @CAP@, MAX_ARRIVALS = @MAXA@, OUT_CACHED = @OUTC@, PIECE = @PIECE@;

// A block's shared scratch. Clocked: the arrivals that each thread listed; exact times: each neuron's arrivals.
struct N2Scratch {
    u32 word, arrivals;
    int optr[OUT_CACHED][NPB_C + 1];
    float spike_t[NPB_C];
@LISTS@
};

// One warp, the links r0 .. r1 (at most PIECE) of a row: set each one's bit in the arrival slot of its step. Every
// link's load is in flight before the first reduction: a row is a chain of memory latencies, not of bandwidth.
__device__ __forceinline__ void n2_deliver(const N2Out &o, long long n, int r0, int r1) {
    u32 pos[PIECE / 32], d[PIECE / 32];
    const int l0 = r0 + (int)(threadIdx.x & 31);
    if (o.dly) {
        #pragma unroll
        for (int k = 0; k < PIECE / 32; ++k) {
            const int l = l0 + 32 * k;
            d[k] = l < r1 ? __ldg(o.dly + l) : 0u;
            pos[k] = l < r1 ? __ldg(o.pos + l) : 0u;
        }
    } else {
        #pragma unroll
        for (int k = 0; k < PIECE / 32; ++k) pos[k] = l0 + 32 * k < r1 ? __ldg(o.pos + l0 + 32 * k) : 0u;
        #pragma unroll
        for (int k = 0; k < PIECE / 32; ++k) {
            d[k] = pos[k] >> 24;
            pos[k] &= 0xFFFFFFu;
        }
    }
    #pragma unroll
    for (int k = 0; k < PIECE / 32; ++k)
        if (d[k]) atomicOr(o.arr + (size_t)((n + d[k]) & o.mask) * o.words + (pos[k] >> 5), 1u << (pos[k] & 31u));
}

// The grid barrier of a window: `bar[0]` counts arrivals, `bar[32]` is set when a wait gave up (bar[33]: how many).
struct N2Grid {
    u32 *bar;
    u64 limit_ns;
    u32 base, pad;  // the count before this window
};

__device__ __forceinline__ u64 n2_clock() {
    u64 t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool n2_grid_sync(const N2Grid &g, int k) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const u32 target = g.base + (u32)(k + 1) * gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(g.bar) : "memory");
        int ok = 1;
        u64 t0 = 0;
        for (int spin = 0;; ++spin) {
            u32 v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(g.bar) : "memory");
            if ((int)(v - target) >= 0) break;
            if ((spin & 15) == 15 && *(volatile u32 *)(g.bar + 32)) { ok = 0; break; }
            if (spin == 0) t0 = n2_clock();
            else if (n2_clock() - t0 > g.limit_ns) {
                atomicExch(g.bar + 32, 1u);
                atomicAdd(g.bar + 33, 1u);
                ok = 0;
                break;
            }
            __nanosleep(20);
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}
'''

_LISTS = {False: "    u32 list[NPB_C * SCAN * CAP];\n    int cnt[NPB_C * SCAN];",
          True: "    float a_t[NPB_C][MAX_ARRIVALS];\n    int a_l[NPB_C][MAX_ARRIVALS];\n"
                "    unsigned short a_c[NPB_C][MAX_ARRIVALS];\n    unsigned char a_o[NPB_C][MAX_ARRIVALS];"}


class Out(ctypes.Structure):
    """One outgoing connection (the source's N2Out)."""
    _fields_ = [("ptr", ctypes.c_void_p), ("pos", ctypes.c_void_p), ("dly", ctypes.c_void_p),
                ("arr", ctypes.c_void_p), ("words", ctypes.c_int64), ("mask", ctypes.c_int32),
                ("pad", ctypes.c_int32)]


class Grid(ctypes.Structure):
    """A window's grid barrier (N2Grid)."""
    _fields_ = [("bar", ctypes.c_void_p), ("limit_ns", ctypes.c_uint64), ("base", ctypes.c_uint32),
                ("pad", ctypes.c_uint32)]


def common(exact: bool) -> str:
    text = _COMMON.replace("@LISTS@", _LISTS[exact])
    for key, v in (("SCAN", SCAN), ("NPB", NPB_C), ("CAP", CAP), ("MAXA", MAX_ARRIVALS), ("OUTC", OUT_CACHED), ("PIECE", PIECE)):
        text = text.replace(f"@{key}@", str(v))
    return text


def indent(text: str, pad: int) -> str:
    return text.replace("\n", "\n" + " " * pad).rstrip() + "\n"


def takes(inc: dict) -> bool:
    """Whether an arrival on the connection runs anything."""
    return inc["receive"] is not None or inc.get("forward") is not None


def _row_bounds(c: int) -> str:
    """Connection c's row of neuron j: its first link, its words."""
    return (f"c{c}_r0 = live ? p.c{c}_ptr[j] : 0, c{c}_w0 = live ? p.c{c}_wptr[j] : 0, "
            f"c{c}_w1 = live ? p.c{c}_wptr[j + 1] : 0;\n")


def _words_of(c: int) -> str:
    """The row's bounds, its slot, and this thread's run of its words."""
    again = "" if c < ROWS_AHEAD else f"            const int {_row_bounds(c)}"
    return f"""{again}            const int r0 = c{c}_r0, w0 = c{c}_w0, w1 = c{c}_w1;
            u32 *arr = p.c{c}_arr + (size_t)(n & p.c{c}_arr_mask) * p.c{c}_arr_words;
            const int seg = (w1 - w0 + SCAN - 1) / SCAN;
            const int a = min(w1, w0 + sc * seg), b = min(w1, a + seg);
""" + (f"            u32 (&x)[4] = x{c};\n" if c < WORDS_AHEAD else f"            u32 x[4];\n{_first_words('arr', 'a', 'b', 12)}")


def _first_words(arr: str, a: str, b: str, pad: int) -> str:
    return (" " * pad + "#pragma unroll\n" + " " * pad +
            f"for (int i = 0; i < 4; ++i) x[i] = {a} + i < {b} ? __ldcg({arr} + {a} + i) : 0u;\n")


def _words_ahead(incoming: list) -> str:
    """The first connections' first words, loaded together: their latencies overlap."""
    out = ""
    for c, inc in enumerate(incoming[:WORDS_AHEAD]):
        if takes(inc):
            out += f"""        u32 x{c}[4];
        {{
            const u32 *arr = p.c{c}_arr + (size_t)(n & p.c{c}_arr_mask) * p.c{c}_arr_words;
            const int seg = (c{c}_w1 - c{c}_w0 + SCAN - 1) / SCAN;
            const int a = min(c{c}_w1, c{c}_w0 + sc * seg), b = min(c{c}_w1, a + seg);
            u32 (&x)[4] = x{c};
{_first_words('arr', 'a', 'b', 12)}        }}
"""
    return out


def _prefetch(c: int, inc: dict) -> str:
    """The listed link's edge values towards the SM, ahead of the owner's loads."""
    return "".join(f'asm volatile("prefetch.global.L1 [%0];" ::"l"(p.c{c}_e_{e} + l)); ' for e in inc["edge_dynamic"])


def _clocked_intake(c: int, inc: dict, arrival: str) -> str:
    """Connection c's arrivals: each of the neuron's SCAN threads (neighbouring lanes of a warp) lists the links of
    its words' set bits and clears them, as long as its list holds a whole word's; the words after that stay set for
    the owner, which runs the hooks over the lists in word order and then over such words, i.e. in link order."""
    return f"""        {{  // connection {c}
{_words_of(c)}            u32 *list = s.list + (jl * SCAN + sc) * CAP;
            int cnt = 0;
            bool left = false;  // words left for the owner
            for (int k = a; k < b; k += 4) {{
                #pragma unroll
                for (int i = 0; i < 4; ++i) {{
                    if (k > a) x[i] = k + i < b ? __ldcg(arr + k + i) : 0u;
                    left = left || (x[i] && cnt + __popc(x[i]) > CAP);
                    if (!x[i] || left) continue;
                    for (u32 v = x[i]; v; v &= v - 1) {{
                        const int l = r0 + 32 * (k + i - w0) + __ffs(v) - 1;
                        list[cnt++] = (u32)l;
                        {_prefetch(c, inc)}
                    }}
                    arr[k + i] = 0u;
                }}
            }}
            s.cnt[jl * SCAN + sc] = left ? ~cnt : cnt;
            const u32 some = __ballot_sync(0xffffffffu, cnt || left);
            __syncwarp();
            if (live && own) {{  // the hooks, in link order
                for (u32 segs = (some >> (threadIdx.x & 31)) & ((1u << SCAN) - 1); segs; segs &= segs - 1) {{
                    const int q = __ffs(segs) - 1;
                    const int cs = s.cnt[jl * SCAN + q], listed = cs < 0 ? ~cs : cs;
                    for (int i = 0; i < listed; ++i) {{
                        const int l = (int)s.list[(jl * SCAN + q) * CAP + i];
                        {indent(arrival, 24)}                    }}
                    if (cs >= 0) continue;
                    const int as = min(w1, w0 + q * seg), bs = min(w1, as + seg);
                    for (int k = as; k < bs; ++k) {{
                        u32 v = __ldcg(arr + k);  // (the listed words are clear)
                        if (v) arr[k] = 0u;
                        for (; v; v &= v - 1) {{
                            const int l = r0 + 32 * (k - w0) + __ffs(v) - 1;
                            {indent(arrival, 28)}                        }}
                    }}
                }}
            }}
            link_k = 0xFFFFFFu;
            __syncwarp();  // the lists are rewritten by the next connection
        }}
"""


def _exact_collect(c: int, inc: dict) -> str:
    """Connection c's arrivals of the step into the neuron's list, in link order, with their times; past
    MAX_ARRIVALS they are counted and dropped."""
    return f"""        {{  // connection {c}
{_words_of(c)}            int mine = 0;
            #pragma unroll
            for (int i = 0; i < 4; ++i) mine += __popc(x[i]);
            for (int k = a + 4; k < b; ++k) mine += __popc(__ldcg(arr + k));
            int at = mine;
            #pragma unroll
            for (int o = 1; o < SCAN; o <<= 1) {{
                const int v = __shfl_up_sync(0xffffffffu, at, o, SCAN);
                if (sc >= o) at += v;
            }}
            const int total = __shfl_sync(0xffffffffu, at, SCAN - 1, SCAN);
            at += na - mine;
            na += total;
            for (int k = a; mine > 0 && k < b; ++k) {{
                u32 v = k - a < 4 ? (k - a < 2 ? (k == a ? x[0] : x[1]) : (k - a == 2 ? x[2] : x[3])) : __ldcg(arr + k);
                if (v) arr[k] = 0u;
                for (; v; v &= v - 1, ++at) {{
                    if (at >= MAX_ARRIVALS) {{ atomicAdd(p.err, 1); continue; }}
                    const int l = r0 + 32 * (k - w0) + __ffs(v) - 1;
                    const u32 w = __ldg(p.c{c}_link + l);
                    {_prefetch(c, inc)}
                    const int src = (int)(w & 0xFFFFFFu), d = (int)(w >> 24);
                    s.a_t[jl][at] = t0 + __ldcg(p.c{c}_src_off + (size_t)((n - d) & p.c{c}_src_mask) * p.c{c}_src_n + src);
                    s.a_l[jl][at] = l;
                    s.a_c[jl][at] = {c};
                }}
            }}
        }}
"""


_EXACT_SORT = """        // by time, equal times in the order they were listed: each arrival's rank, the SCAN threads together
        na = min(na, MAX_ARRIVALS);
        __syncwarp();
        bool odd = false;  // (a time that is not a number has no rank)
        for (int e = sc; e < na; e += SCAN) {
            const float te = s.a_t[jl][e];
            int rank = 0;
            for (int k = 0; k < na; ++k) {
                const float tk = s.a_t[jl][k];
                rank += tk < te || (tk == te && k < e);
                odd = odd || tk != tk;
            }
            s.a_o[jl][rank] = (unsigned char)e;
        }
        __syncwarp();
        if (own && odd) {
            for (int e = 0; e < na; ++e) {
                const float te = s.a_t[jl][e];
                int k = e;
                while (k > 0 && s.a_t[jl][s.a_o[jl][k - 1]] > te) { s.a_o[jl][k] = s.a_o[jl][k - 1]; --k; }
                s.a_o[jl][k] = (unsigned char)e;
            }
        }
"""


def _exact_deliver(pop_name: str, incoming: list, hooks: dict) -> str:
    """The owner: receive (and edge forward) for each arrival at its own time, send after each group of equal ones."""
    cases = "".join(
        f"""                    case {c}: {{
                        {indent("".join(f"float e_{e} = p.c{c}_e_{e}[l];" + chr(10) for e in inc["edge_dynamic"])
                                + _arrival_body(pop_name, c, inc), 24)}                    }} break;
""" for c, inc in enumerate(incoming) if takes(inc))
    fn, ctx = hooks["send"]
    return f"""        if (live && own) {{
            for (int i = 0; i < na;) {{
                const float tau = s.a_t[jl][s.a_o[jl][i]];
                int e = i;
                while (e < na && s.a_t[jl][s.a_o[jl][e]] == tau) ++e;
                e = max(e, i + 1);
                for (int k = i; k < e; ++k) {{
                    const int o = s.a_o[jl][k], l = s.a_l[jl][o];
                    const float t = tau;
                    link_k = arrived++;
                    switch (s.a_c[jl][o]) {{
{cases}                    default: break;
                    }}
                }}
                {{
                    const float t = tau;
                    {indent(lower_hook(fn, ctx, f"{pop_name} send"), 20)}                }}
                i = e;
            }}
            link_k = 0xFFFFFFu;
        }}
        __syncwarp();
"""


def _rows_loop(rows: str) -> str:
    """The head of a block's loop over `rows` rows (i), each by a group of g warps (fewer rows than warps) or one."""
    return f"""        if (fw) {{
        const int rows = {rows};
        int g = 1;
        while (2 * g * rows <= {THREADS // 32}) g *= 2;
        for (int i = (int)(threadIdx.x >> 5) / g; i < rows; i += {THREADS // 32} / g) {{
"""


def _deliver_code(n_out: int) -> str:
    """The block's deliveries: its spikes' rows in pieces of PIECE links, dealt out to its warps in turn, so that two
    or three spikes in one block (the step's slowest) are still a piece or two per warp."""
    if not n_out:
        return ""
    rows = ("const int r0 = o < OUT_CACHED ? s.optr[o][q] : O.ptr[blk * NPB_C + q], r1 = o < OUT_CACHED ? "
            "s.optr[o][q + 1] : O.ptr[blk * NPB_C + q + 1];"
            if n_out > OUT_CACHED else "const int r0 = s.optr[o][q], r1 = s.optr[o][q + 1];")
    return f"""        int turn = (int)(threadIdx.x >> 5);  // the spikes' outgoing rows: this warp's next piece
        for (u32 m = fw; m; m &= m - 1) {{
            const int q = __ffs(m) - 1;
            for (int o = 0; o < {n_out}; ++o) {{
                const N2Out &O = p.outs[o];
                {rows}
                const int pieces = (r1 - r0 + PIECE - 1) / PIECE;
                for (; turn < pieces; turn += {THREADS // 32})
                    n2_deliver(O, n, r0 + turn * PIECE, min(r1, r0 + (turn + 1) * PIECE));
                turn -= pieces;
            }}
        }}
"""


def _backward_body(pop_name: str, c: int, inc: dict) -> str:
    fn, ctx = inc["backward"]
    return (lower_hook(fn, ctx, f"{pop_name} edge backward (connection {c})") +
            "".join(f"p.c{c}_e_{e}[l] = e_{e};\n" for e in inc.get("edge_written", ())))


def _backward_loop(pop_name: str, c: int, inc: dict, j: str, first: str, step: str) -> str:
    """Connection c's edge backward hook over the incoming links of neuron `j`: first, first + step, ..."""
    pad = " " * 12
    loads = "".join(f"{pad}    float e_{e} = p.c{c}_e_{e}[l];\n" for e in inc["edge_dynamic"])
    body = _backward_body(pop_name, c, inc).replace("\n", f"\n{pad}    ").rstrip()
    return (f"{pad}for (int l = p.c{c}_ptr[{j}] + {first}; l < p.c{c}_ptr[{j} + 1]; l += {step}) {{\n{loads}"
            f"{pad}    {body}\n{pad}}}\n")


def params_fields(attrs: dict, incoming: list, n_out: int, exact: bool) -> list:
    fields = base_fields(attrs)
    fields.append(("bad", "int", ctypes.c_int32))  # incoming links out of range: counted every step
    for c, inc in enumerate(incoming):
        fields += [(f"c{c}_ptr", "const int *", ctypes.c_void_p), (f"c{c}_wptr", "const int *", ctypes.c_void_p),
                   (f"c{c}_arr", "u32 *", ctypes.c_void_p), (f"c{c}_arr_words", "long long", ctypes.c_int64),
                   (f"c{c}_arr_mask", "int", ctypes.c_int32)]
        if exact:
            fields += [(f"c{c}_link", "const u32 *", ctypes.c_void_p),
                       (f"c{c}_src_off", "const float *", ctypes.c_void_p),
                       (f"c{c}_src_mask", "int", ctypes.c_int32), (f"c{c}_src_n", "int", ctypes.c_int32)]
        for e in inc["edge_dynamic"]:
            fields.append((f"c{c}_e_{e}", "float *" if e in inc.get("edge_written", ()) else "const float *",
                           ctypes.c_void_p))
    if n_out:
        fields.append(("outs", f"N2Out[{n_out}]", Out * n_out))
    return fields


def population(pop_name: str, attrs: dict, hooks: dict, incoming: list, n_out: int, exact: bool, fields: list) -> str:
    """A population's Params and its steps: `n2_steps`, n_steps of them from step n for the block `blk` (WINDOW: a
    grid barrier between them). Edge backward hooks that assign nothing of the destination run for a fired neuron's
    links on a group of warps (a link's hook touches that link alone), the others on the owner, link by link."""
    src = ["struct Params {\n"]
    src += [f"    {ct.split('[')[0]} {name}{'[' + ct.split('[')[1] if '[' in ct else ''};\n" for name, ct, _ in fields]
    src += ["};\n\n", UNIFORM]
    src.append(f"""// population {pop_name}
template <bool WINDOW>
__device__ __forceinline__ void n2_steps(const Params &p, N2Scratch &s, const int blk, long long n, const int n_steps,
                                         const double dt, const N2Grid &grid) {{
    const int jl = threadIdx.x / SCAN, sc = threadIdx.x % SCAN;
    const int j = blk * NPB_C + jl;
    const bool live = j < p.n, own = sc == 0;
""")
    # what no launch writes, then (one step per launch) the launch before this one: the next launch may be scheduled
    # and the row bounds loaded while it is still running
    src.append('    if (!WINDOW) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");\n')
    src += [f"    const int {_row_bounds(c)}" for c, inc in enumerate(incoming[:ROWS_AHEAD]) if takes(inc)]
    if n_out:
        src.append(f"""    for (int k = threadIdx.x; k < {min(n_out, OUT_CACHED)} * (NPB_C + 1); k += {THREADS}) {{
        const int q = k % (NPB_C + 1);
        s.optr[k / (NPB_C + 1)][q] = p.outs[k / (NPB_C + 1)].ptr[min(blk * NPB_C + q, p.n)];
    }}
""")
    src.append('    if (!WINDOW) asm volatile("griddepcontrol.wait;" ::: "memory");\n')
    for a, py in attrs.items():
        ct, _, _ = ctype_of(py)
        src.append(f"    {ct} s_{a} = (live && own) ? p.s_{a}[j] : ({ct})0;\n")
    backward = [(c, inc) for c, inc in enumerate(incoming) if inc.get("backward") is not None]
    shared = backward and not any(inc.get("backward_writes", True) for _, inc in backward)
    read = [a for a in attrs if any(f"s_{a}" in _backward_body(pop_name, c, inc) for c, inc in backward)] if shared else []
    src += [f"    __shared__ {ctype_of(attrs[a])[0]} n2d_{a}[NPB_C];\n" for a in read]
    src.append("""    u64 spikes = 0, events = 0;  // the block's, counted by its first thread
    for (int step = 0;; ++step, ++n) {
        const float t = WINDOW ? (float)((double)(n + 1) * dt) : p.t, t0 = WINDOW ? (float)((double)n * dt) : p.t0;
        bool fired = false;
        float spike_t = t;
        u32 arrived = 0;
        u32 link_k = 0xFFFFFFu;
@WORDS@        if (threadIdx.x == 0) {
            s.word = 0u;
            s.arrivals = 0u;
            if (p.bad && blk == 0) atomicAdd(p.err, p.bad);
        }
        __syncthreads();
""".replace("@WORDS@", _words_ahead(incoming)))
    if exact:
        src.append("        int na = 0;  // the neuron's arrivals of the step\n")
        src += [_exact_collect(c, inc) for c, inc in enumerate(incoming) if takes(inc)]
        if any(takes(inc) for inc in incoming):
            src += [_EXACT_SORT, _exact_deliver(pop_name, incoming, hooks)]
    else:
        for c, inc in enumerate(incoming):
            if takes(inc):
                loads = "".join(f"float e_{e} = p.c{c}_e_{e}[l];\n" for e in inc["edge_dynamic"])
                body = "link_k = arrived++;\n{\n" + _arrival_body(pop_name, c, inc) + "}\n"
                src.append(_clocked_intake(c, inc, loads + body))
    src.append("        if (live && own) {\n")
    for name in ("update", "send"):
        fn, ctx = hooks[name]
        src.append("            " + indent(lower_hook(fn, ctx, f"{pop_name} {name}"), 12))
    if backward and not shared:  # the neuron fired: every incoming link's edge backward hook at its spike's time
        src.append("            if (fired) {\n            const float t = spike_t;\n")
        src += [_backward_loop(pop_name, c, inc, "j", "0", "1") for c, inc in backward]
        src.append("            }\n")
    src.append("""            if (fired) {
                const float o = spike_t - t0;  // the spike's time within its step
                p.off[(size_t)(n & p.bit_mask) * p.n + j] = o;
                const long long r = n - p.rec0;
                if (p.raster_off && r >= 0 && r < p.raster_steps) p.raster_off[(size_t)r * p.n + j] = o;
                atomicOr(&s.word, 1u << jl);
""")
    if shared:
        src.append("                s.spike_t[jl] = spike_t;\n")
        src += [f"                n2d_{a}[jl] = s_{a};\n" for a in read]
    src.append("""            }
            if (arrived) atomicAdd(&s.arrivals, arrived);
        }
        __syncthreads();
        const u32 fw = s.word;
        if (threadIdx.x == 0) {  // the block's 32 neurons: one spike-bit word
            if (blk < p.words) {
                p.bits[(size_t)(n & p.bit_mask) * p.words + blk] = fw;
                const long long r = n - p.rec0;
                if (p.raster && r >= 0 && r < p.raster_steps) p.raster[(size_t)r * p.words + blk] = fw;
            }
            spikes += __popc(fw);
            events += s.arrivals;
        }
""")
    src.append(_deliver_code(n_out))
    if shared:
        src.append("        // the fired neurons' incoming links: edge backward at the spike's time\n")
        src.append(_rows_loop("__popc(fw)"))
        src.append("""            u32 m = fw;
            for (int k = i; k > 0; --k) m &= m - 1;
            const int q = __ffs(m) - 1, jq = blk * NPB_C + q;
            const float t = s.spike_t[q];
""")
        src += [f"            const {ctype_of(attrs[a])[0]} s_{a} = n2d_{a}[q];\n" for a in read]
        src += [_backward_loop(pop_name, c, inc, "jq", "(int)threadIdx.x % (32 * g)", "32 * g") for c, inc in backward]
        src.append("        }\n        }\n")
    src.append("""        if (!WINDOW || step + 1 == n_steps) break;
        if (!n2_grid_sync(grid, step)) break;
    }
""")
    src += [f"    if (live && own) p.s_{a}[j] = s_{a};\n" for a in attrs]
    src.append("    if (spikes) atomicAdd(p.counters + 1, spikes);\n    if (events) atomicAdd(p.counters, events);\n}\n")
    return "".join(src)


STEP_KERNEL = f"""
extern "C" __global__ void __launch_bounds__({THREADS}) n2b_user_step(const __grid_constant__ Params p) {{
    __shared__ N2Scratch s;
    n2_steps<false>(p, s, (int)blockIdx.x, p.step, 1, 0.0, N2Grid{{}});
}}
"""


def build(pop_name: str, attrs: dict, hooks: dict, incoming: list, n_out: int, exact: bool) -> tuple[str, list, str]:
    """(step kernel source, params fields, `population` text) of one population; the arguments are build_source's
    (template.py), with "backward_writes" per incoming connection: whether its backward hook assigns the
    destination's state, and n_out: the population's outgoing connections."""
    fields = params_fields(attrs, incoming, n_out, exact)
    body = population(pop_name, attrs, hooks, incoming, n_out, exact, fields)
    return _PRELUDE + common(exact) + body + STEP_KERNEL, fields, body


def blocks_of(n: int) -> int:
    return (n + NPB_C - 1) // NPB_C


def window_source(exact: bool, bodies: list, sizes: list, per_sm: int) -> str:
    """The window kernel over every population: `bodies` their `population` texts, `sizes` their neurons."""
    src = [_PRELUDE, common(exact)]
    src += [f"namespace n2p{k} {{\n{body}}}\n\n" for k, body in enumerate(bodies)]
    src.append("struct Window {\n    long long step0;\n    double dt;\n    N2Grid grid;\n    long long n_steps;\n")
    src += [f"    n2p{k}::Params p{k};\n" for k in range(len(bodies))]
    src.append(f"""}};

extern "C" __global__ void __launch_bounds__({THREADS}, {per_sm}) n2b_user_window(const __grid_constant__ Window w) {{
    __shared__ N2Scratch s;
    if (*(volatile u32 *)(w.grid.bar + 32)) return;  // an earlier window gave up: nothing runs
    const int b = (int)blockIdx.x;
""")
    first = 0
    for k, n in enumerate(sizes):
        if n:
            src.append(f"    if (b >= {first} && b < {first + blocks_of(n)}) n2p{k}::n2_steps<true>(w.p{k}, s, b - {first}, "
                       "w.step0, (int)w.n_steps, w.dt, w.grid);\n")
        first += blocks_of(n)
    src.append("}\n")
    return "".join(src)


def window_type(params: list):
    """The ctypes structure of a Window over the populations' Params types."""
    return type("Window", (ctypes.Structure,), {
        "_fields_": [("step0", ctypes.c_int64), ("dt", ctypes.c_double), ("grid", Grid), ("n_steps", ctypes.c_int64)]
                    + [(f"p{k}", t) for k, t in enumerate(params)]})

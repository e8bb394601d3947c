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
7.3; 1,501 neurons of 150 plastic links 33 -> 11.2 -> 6.1; 3,001 event-driven neurons of 125 links 73 -> 36 ->
11.6.
"""

from __future__ import annotations

import ctypes
import functools

from .cuda import lower_hook
from .template import _PRELUDE, MAX_ARRIVALS, NPB_C, UNIFORM, _arrival_body, base_fields, ctype_of

SCAN = 8  # threads per neuron: a row of 1,000 links is 32 words, four to a thread
THREADS = NPB_C * SCAN
CHUNK = 4 * SCAN  # words of a row taken at once, four to a thread
EDGE_CAP = {False: 16, True: MAX_ARRIVALS}  # arrivals whose edge values are loaded ahead of their hooks (by exact)
EDGE_ATTRS = {False: 8, True: 2}  # ... of at most so many edge attributes
OUT_CACHED = 8  # outgoing connections whose row bounds a block holds in shared memory
PIECE = 256  # links of a row that a warp delivers at once, eight loads a lane in flight
# (incoming connections whose row bounds a thread holds, those of them whose arrival words are loaded together at a
# step's start). Four blocks on an SM leave a thread 64 registers, three 80: with (8, 4), 4 connections spill 56 bytes at
# 64 and 8 connections 224, with (2, 2) none.
AHEAD, AHEAD_FEW = (8, 4), (2, 2)
WINDOW_PARAMS = 16384  # bytes of a window kernel's parameter block at most
WINDOW_POPS = 16  # populations of a window kernel at most
WINDOW_INTAKES = 8  # connections that the code of a window kernel takes in at most, over its distinct populations

_COMMON = r'''
struct N2Out {
    const int *ptr;            // rows per source neuron
    const u32 *pos;            // per link: its bit among a slot's words (dly null: its delay in the top 8 bits)
    const unsigned char *dly;  // per link: its delay in steps, of connections with more than 2^24 bits to a slot
    u32 *arr;                  // the arrival bits, [depth][words]
    long long words;
    int depth, pad;            // slots: the largest delay + 1 (step n's is n mod depth)
};

constexpr int SCAN = @SCAN@, NPB_C = @NPB@, CHUNK = 4 * SCAN, MAX_ARRIVALS = @MAXA@, OUT_CACHED = @OUTC@, PIECE = @PIECE@;
constexpr int EDGE_CAP = @ECAP@;

// A block's shared scratch. Clocked: each neuron's arrival words of a chunk; exact times: each neuron's arrivals.
struct N2Scratch {
    u32 word, arrivals;
    int optr[OUT_CACHED][NPB_C + 1];
    float spike_t[NPB_C];
@LISTS@
};

// One warp, the links r0 .. r1 (at most PIECE) of a row: set each one's bit in the arrival slot of its step. Every
// link's load is in flight before the first reduction: a row is a chain of memory latencies, not of bandwidth.
__device__ __forceinline__ void n2_deliver(const N2Out &o, long long n, int r0, int r1) {
    const u32 now = (u32)((u64)n % (u32)o.depth);
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
        if (d[k]) {
            const u32 slot = now + d[k] < (u32)o.depth ? now + d[k] : now + d[k] - (u32)o.depth;
            atomicOr(o.arr + (size_t)slot * o.words + (pos[k] >> 5), 1u << (pos[k] & 31u));
        }
}

// The grid barrier of a window: `bar[0]` counts its arrivals, `bar[32]` is set when a wait gave up (bar[33]: how many).
// The count wraps to 0 at the launch's last arrival, so that every launch starts from 0, a captured one's replay too
// (cleared by the last block out it cost each launch a round trip more: 28.9 us of 28.5 for a few steps).
struct N2Grid {
    u32 *bar;
    u64 limit_ns;
};

__device__ __forceinline__ u64 n2_clock() {
    u64 t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Barrier k of a launch of n_steps > k + 1 steps. Its last one is passed at 0: the count stays there.
__device__ __forceinline__ bool n2_grid_sync(const N2Grid &g, int k, int n_steps) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const u32 all = (u32)(n_steps - 1) * gridDim.x, target = (u32)(k + 1) * gridDim.x;
        asm volatile("red.release.gpu.global.inc.u32 [%0], %1;" ::"l"(g.bar), "r"(all - 1u) : "memory");
        int ok = 1;
        u64 t0 = 0;
        for (int spin = 0;; ++spin) {
            u32 v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(g.bar) : "memory");
            if (target == all ? v == 0u : v >= target) break;
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

_LISTS = {False: "    u32 words[NPB_C][CHUNK];",
          True: "    float a_t[NPB_C][MAX_ARRIVALS];\n    int a_l[NPB_C][MAX_ARRIVALS];\n"
                "    unsigned short a_c[NPB_C][MAX_ARRIVALS];\n    unsigned char a_o[NPB_C][MAX_ARRIVALS];"}


class Out(ctypes.Structure):
    """One outgoing connection (the source's N2Out)."""
    _fields_ = [("ptr", ctypes.c_void_p), ("pos", ctypes.c_void_p), ("dly", ctypes.c_void_p),
                ("arr", ctypes.c_void_p), ("words", ctypes.c_int64), ("depth", ctypes.c_int32),
                ("pad", ctypes.c_int32)]


class Grid(ctypes.Structure):
    """A window's grid barrier (N2Grid)."""
    _fields_ = [("bar", ctypes.c_void_p), ("limit_ns", ctypes.c_uint64)]


def common(exact: bool, edges: int) -> str:
    """The text shared by a network's populations; edges: edge attributes held in the scratch (`staged`)."""
    lists = _LISTS[exact] + (f"\n    float e[{edges}][NPB_C][EDGE_CAP];" if edges else "")
    text = _COMMON.replace("@LISTS@", lists)
    for key, v in (("SCAN", SCAN), ("NPB", NPB_C), ("MAXA", MAX_ARRIVALS), ("OUTC", OUT_CACHED), ("PIECE", PIECE),
                   ("ECAP", EDGE_CAP[exact])):
        text = text.replace(f"@{key}@", str(v))
    return text


def staged(incoming: list, exact: bool) -> int:
    """Edge attributes of these connections whose values are loaded ahead of the hooks, at most EDGE_ATTRS."""
    return min(EDGE_ATTRS[exact], max((len(inc["edge_dynamic"]) for inc in incoming if takes(inc)), default=0))


def indent(text: str, pad: int) -> str:
    return text.replace("\n", "\n" + " " * pad).rstrip() + "\n"


def takes(inc: dict) -> bool:
    """Whether an arrival on the connection runs anything."""
    return inc["receive"] is not None or inc.get("forward") is not None


def _row_bounds(c: int) -> str:
    """Connection c's row of neuron j: its first link, its words."""
    return (f"c{c}_r0 = live ? p.c{c}_ptr[j] : 0, c{c}_w0 = live ? p.c{c}_wptr[j] : 0, "
            f"c{c}_w1 = live ? p.c{c}_wptr[j + 1] : 0;\n")


def _chunk_head(c: int, ahead: tuple) -> str:
    """The loop over a row's words in chunks (the same number of them for the whole warp): word kb + SCAN i + sc is
    x[i] of the neuron's thread sc, four loads in flight; the first connections' first chunk is loaded already."""
    again = "" if c < ahead[0] else f"            const int {_row_bounds(c)}"
    if c >= ahead[0]:
        again += f"            const int c{c}_rounds = {_rounds(c)};\n"
    first = f"x{c}[i]" if c < ahead[1] else "w0 + SCAN * i + sc < w1 ? __ldcg(arr + w0 + SCAN * i + sc) : 0u"
    return f"""{again}            const int r0 = c{c}_r0, w0 = c{c}_w0, w1 = c{c}_w1;
            u32 *arr = p.c{c}_arr + (size_t)slot{c} * p.c{c}_arr_words;
            u32 x[4];
            #pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = {first};
            for (int kb = 0, round = 0; round < c{c}_rounds; ++round, kb += CHUNK) {{
                #pragma unroll
                for (int i = 0; i < 4; ++i) {{
                    const int k = w0 + kb + SCAN * i + sc;
                    if (round) x[i] = k < w1 ? __ldcg(arr + k) : 0u;
                    if (x[i]) arr[k] = 0u;
                }}
"""


def _rounds(c: int) -> str:
    return f"(int)(__reduce_max_sync(0xffffffffu, (u32)(c{c}_w1 - c{c}_w0)) + CHUNK - 1) / CHUNK"


def _words_ahead(incoming: list, ahead: tuple) -> str:
    """The first connections' first words, loaded together: their latencies overlap."""
    return "".join(f"""        u32 x{c}[4];
        {{
            const u32 *arr = p.c{c}_arr + (size_t)slot{c} * p.c{c}_arr_words + c{c}_w0;
            #pragma unroll
            for (int i = 0; i < 4; ++i) x{c}[i] = SCAN * i + sc < c{c}_w1 - c{c}_w0 ? __ldcg(arr + SCAN * i + sc) : 0u;
        }}
""" for c, inc in enumerate(incoming[:ahead[1]]) if takes(inc))


# Each thread's first arrival (start[i]) of its word i among the neuron's arrivals of the chunk, in word order, and
# their number (total): counts of two words to a register, scanned over the neuron's threads.
_RANKS = """                u32 n01 = __popc(x[0]) | __popc(x[1]) << 16, n23 = __popc(x[2]) | __popc(x[3]) << 16;
                const u32 own01 = n01, own23 = n23;
                #pragma unroll
                for (int o = 1; o < SCAN; o <<= 1) {
                    const u32 u01 = __shfl_up_sync(0xffffffffu, n01, o, SCAN), u23 = __shfl_up_sync(0xffffffffu, n23, o, SCAN);
                    if (sc >= o) { n01 += u01; n23 += u23; }
                }
                const u32 t01 = __shfl_sync(0xffffffffu, n01, SCAN - 1, SCAN), t23 = __shfl_sync(0xffffffffu, n23, SCAN - 1, SCAN);
                n01 -= own01;
                n23 -= own23;
                const int h0 = t01 & 0xFFFFu, h1 = h0 + (t01 >> 16), h2 = h1 + (t23 & 0xFFFFu), total = h2 + (t23 >> 16);
                const int start[4] = {(int)(n01 & 0xFFFFu), h0 + (int)(n01 >> 16), h1 + (int)(n23 & 0xFFFFu), h2 + (int)(n23 >> 16)};
"""


def _stage_edges(c: int, inc: dict, exact: bool, at: str, pad: int) -> str:
    """The edge values of link l into the scratch's place `at`."""
    return "".join(" " * pad + f"s.e[{a}][jl][{at}] = p.c{c}_e_{e}[l];\n"
                   for a, e in enumerate(inc["edge_dynamic"][:EDGE_ATTRS[exact]]))


def _clocked_intake(c: int, inc: dict, body: str, ahead: tuple) -> str:
    """Connection c's arrivals: the neuron's threads put their words with a set bit into shared memory and clear
    them; the neuron's first thread (the owner) runs the hooks over the words' bits, i.e. in link order. Edge values
    are loaded by the threads together, ahead of the owner's chain of hooks (of the chunk's first EDGE_CAP arrivals)."""
    edges = inc["edge_dynamic"]
    stage, loads = "", ""
    if edges:
        stage = _RANKS + f"""                #pragma unroll
                for (int i = 0; i < 4; ++i) {{
                    int at = start[i];
                    for (u32 v = x[i]; v && at < EDGE_CAP; v &= v - 1, ++at) {{
                        const int l = r0 + 32 * (kb + SCAN * i + sc) + __ffs(v) - 1;
{_stage_edges(c, inc, False, "at", 24)}                    }}
                }}
"""
        for a, e in enumerate(edges):
            loads += (f"float e_{e} = at < EDGE_CAP ? s.e[{a}][jl][at] : p.c{c}_e_{e}[l];\n" if a < EDGE_ATTRS[False]
                      else f"float e_{e} = p.c{c}_e_{e}[l];\n")
    run = loads + ("++at;\n" if edges else "") + "link_k = arrived++;\n{\n" + body + "}\n"
    return f"""        {{  // connection {c}
{_chunk_head(c, ahead)}{stage}                u32 some = 0u;  // the neuron's words of the chunk with a set bit
                #pragma unroll
                for (int i = 0; i < 4; ++i) {{
                    some |= ((__ballot_sync(0xffffffffu, x[i] != 0u) >> (threadIdx.x & 31 & ~(SCAN - 1))) & ((1u << SCAN) - 1)) << (SCAN * i);
                    if (x[i]) s.words[jl][SCAN * i + sc] = x[i];
                }}
                __syncwarp();
                if (own) {{  // the hooks, in link order
                    {"int at = 0;" if edges else ""}
                    for (; some; some &= some - 1) {{
                        const int k = __ffs(some) - 1;
                        for (u32 v = s.words[jl][k]; v; v &= v - 1) {{
                            const int l = r0 + 32 * (kb + k) + __ffs(v) - 1;
                            {indent(run, 28)}                        }}
                    }}
                }}
                __syncwarp();  // the words are rewritten by the next chunk
            }}
            link_k = 0xFFFFFFu;
        }}
"""


def _exact_collect(c: int, inc: dict, ahead: tuple) -> str:
    """Connection c's arrivals of the step into the neuron's list, in link order; past MAX_ARRIVALS they are counted
    and dropped."""
    return f"""        {{  // connection {c}
{_chunk_head(c, ahead)}{_RANKS}                #pragma unroll
                for (int i = 0; i < 4; ++i) {{
                    int at = na + start[i];
                    for (u32 v = x[i]; v; v &= v - 1, ++at) {{
                        if (at >= MAX_ARRIVALS) {{ atomicAdd(p.err, 1); continue; }}
                        s.a_l[jl][at] = r0 + 32 * (kb + SCAN * i + sc) + __ffs(v) - 1;
                        s.a_c[jl][at] = {c};
                    }}
                }}
                na += total;
            }}
        }}
"""


def _exact_times(incoming: list) -> str:
    """The listed arrivals' times and edge values: the SCAN threads take one each, so that their loads (the link, then
    its source's spike) overlap."""
    cases = "".join(f"""                case {c}: {{
                    const u32 w = __ldg(p.c{c}_link + l);
{_stage_edges(c, inc, True, "e", 20)}                    const int src = (int)(w & 0xFFFFFFu), d = (int)(w >> 24);
                    s.a_t[jl][e] = t0 + __ldcg(p.c{c}_src_off + (size_t)((n - d) & p.c{c}_src_mask) * p.c{c}_src_n + src);
                }} break;
""" for c, inc in enumerate(incoming) if takes(inc))
    return f"""        na = min(na, MAX_ARRIVALS);
        __syncwarp();
        for (int e = sc; e < na; e += SCAN) {{
            const int l = s.a_l[jl][e];
            switch (s.a_c[jl][e]) {{
{cases}                default: break;
            }}
        }}
"""


_EXACT_SORT = """        // by time, equal times in the order they were listed: each arrival's rank, the SCAN threads together
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


def _exact_loads(c: int, inc: dict) -> str:
    return "".join(f"float e_{e} = s.e[{a}][jl][o];\n" if a < EDGE_ATTRS[True] else f"float e_{e} = p.c{c}_e_{e}[l];\n"
                   for a, e in enumerate(inc["edge_dynamic"]))


def _exact_deliver(pop_name: str, incoming: list, hooks: dict) -> str:
    """The owner: receive (and edge forward) for each arrival at its own time, send after each group of equal ones."""
    cases = "".join(
        f"""                    case {c}: {{
                        {indent(_exact_loads(c, inc) + _arrival_body(pop_name, c, inc), 24)}                    }} break;
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
                   (f"c{c}_arr_depth", "int", ctypes.c_int32)]
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


def population(pop_name: str, attrs: dict, hooks: dict, incoming: list, n_out: int, exact: bool, fields: list,
               ahead: tuple) -> str:
    """A population's Params and its steps: `n2_steps`, n_steps of them from step n for the block `blk` (WINDOW: a
    grid barrier between them). Edge backward hooks that assign nothing of the destination run for a fired neuron's
    links on a group of warps (a link's hook touches that link alone), the others on the owner, link by link."""
    src = ["struct Params {\n"]
    src += [f"    {ct.split('[')[0]} {name}{'[' + ct.split('[')[1] if '[' in ct else ''};\n" for name, ct, _ in fields]
    src += ["};\n\n", UNIFORM]
    src.append(f"""// population {pop_name}
template <bool WINDOW>
__device__ __forceinline__ void n2_steps(const Params &p, N2Scratch &s, const int blk, long long n, const int n_steps,
                                         const double dt, const N2Grid &grid, const u32 stop) {{
    const int jl = threadIdx.x / SCAN, sc = threadIdx.x % SCAN;
    const int j = blk * NPB_C + jl;
    const bool live = j < p.n, own = sc == 0;
""")
    # what no launch writes, then (one step per launch) the launch before this one: the next launch may be scheduled
    # and the row bounds loaded while it is still running
    src.append('    if (!WINDOW) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");\n')
    src += [f"    const int {_row_bounds(c)}    const int c{c}_rounds = {_rounds(c)};\n"
            for c, inc in enumerate(incoming[:ahead[0]]) if takes(inc)]
    if n_out:
        src.append(f"""    for (int k = threadIdx.x; k < {min(n_out, OUT_CACHED)} * (NPB_C + 1); k += {THREADS}) {{
        const int q = k % (NPB_C + 1);
        s.optr[k / (NPB_C + 1)][q] = p.outs[k / (NPB_C + 1)].ptr[min(blk * NPB_C + q, p.n)];
    }}
""")
    src.append('    if (!WINDOW) asm volatile("griddepcontrol.wait;" ::: "memory");\n'
               "    if (WINDOW && __syncthreads_or(stop)) return;  // an earlier window gave up: nothing runs\n")
    for a, py in attrs.items():
        ct, _, _ = ctype_of(py)
        src.append(f"    {ct} s_{a} = (live && own) ? p.s_{a}[j] : ({ct})0;\n")
    backward = [(c, inc) for c, inc in enumerate(incoming) if inc.get("backward") is not None]
    shared = backward and not any(inc.get("backward_writes", True) for _, inc in backward)
    read = [a for a in attrs if any(f"s_{a}" in _backward_body(pop_name, c, inc) for c, inc in backward)] if shared else []
    src += [f"    __shared__ {ctype_of(attrs[a])[0]} n2d_{a}[NPB_C];\n" for a in read]
    # each connection's slot of the step, kept as the steps go on
    src += [f"    int slot{c} = (int)((u64)n % (u32)p.c{c}_arr_depth);\n" for c, inc in enumerate(incoming) if takes(inc)]
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
""".replace("@WORDS@", _words_ahead(incoming, ahead)))
    if exact:
        src.append("        int na = 0;  // the neuron's arrivals of the step\n")
        src += [_exact_collect(c, inc, ahead) for c, inc in enumerate(incoming) if takes(inc)]
        if any(takes(inc) for inc in incoming):
            src += [_exact_times(incoming), _EXACT_SORT, _exact_deliver(pop_name, incoming, hooks)]
        else:  # the send of a time group has call sites of its own: without groups the step's send keeps its numbers
            fn, ctx = hooks["send"]
            lower_hook(fn, ctx, f"{pop_name} send")
    else:
        for c, inc in enumerate(incoming):
            if takes(inc):
                src.append(_clocked_intake(c, inc, _arrival_body(pop_name, c, inc), ahead))
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
        if (!n2_grid_sync(grid, step, n_steps)) break;
""")
    src += [f"        if (++slot{c} == p.c{c}_arr_depth) slot{c} = 0;\n" for c, inc in enumerate(incoming) if takes(inc)]
    src.append("    }\n")
    src += [f"    if (live && own) p.s_{a}[j] = s_{a};\n" for a in attrs]
    src.append("    if (spikes) atomicAdd(p.counters + 1, spikes);\n    if (events) atomicAdd(p.counters, events);\n}\n")
    return "".join(src)


STEP_KERNEL = f"""
extern "C" __global__ void __launch_bounds__({THREADS}) n2b_user_step(const __grid_constant__ Params p) {{
    __shared__ N2Scratch s;
    n2_steps<false>(p, s, (int)blockIdx.x, p.step, 1, 0.0, N2Grid{{}}, 0u);
}}
"""


def build(pop_name: str, attrs: dict, hooks: dict, incoming: list, n_out: int, exact: bool,
          ahead: tuple = AHEAD) -> tuple[str, list, str]:
    """(step kernel source, params fields, `population` text) of one population; the arguments are build_source's
    (template.py), with "backward_writes" per incoming connection: whether its backward hook assigns the
    destination's state, n_out: the population's outgoing connections, and `ahead` (AHEAD)."""
    fields = params_fields(attrs, incoming, n_out, exact)
    body = population(pop_name, attrs, hooks, incoming, n_out, exact, fields, ahead)
    return _PRELUDE + common(exact, staged(incoming, exact)) + body + STEP_KERNEL, fields, body


def blocks_of(n: int) -> int:
    return (n + NPB_C - 1) // NPB_C


def window_source(exact: bool, kinds: list, edges: int, per_sm: int) -> str:
    """The window kernel: `kinds` its distinct `population` texts and how many populations run each, in the order of the
    parameter block (populations of one kind share its code); `edges` the most edge attributes that one of them stages;
    `per_sm` the blocks that an SM holds at once. The populations' sizes are parameters: networks that differ in them
    alone share the kernel."""
    src = [_PRELUDE, common(exact, edges)]
    src += [f"namespace n2p{g} {{\n{body}}}\n\n" for g, (body, _) in enumerate(kinds)]
    src.append("struct Window {\n    long long step0;\n    double dt;\n    N2Grid grid;\n    long long n_steps;\n")
    src.append(f"    int first[{sum(count for _, count in kinds) + 1}];  // each population's first block, then their number\n")
    src += [f"    n2p{g}::Params p{g}[{count}];\n" for g, (_, count) in enumerate(kinds)]
    src.append(f"""}};

extern "C" __global__ void __launch_bounds__({THREADS}, {per_sm}) n2b_user_window(const __grid_constant__ Window w) {{
    __shared__ N2Scratch s;
    // set when an earlier window gave up (one thread reads for the block: another block may set it meanwhile)
    const u32 stop = threadIdx.x == 0 ? *(volatile u32 *)(w.grid.bar + 32) : 0u;
    int k = 0;
    while ((int)blockIdx.x >= w.first[k + 1]) ++k;
    const int b = (int)blockIdx.x - w.first[k];
""")
    before = 0
    for g, (_, count) in enumerate(kinds):
        src.append(f"    if (k >= {before} && k < {before + count}) n2p{g}::n2_steps<true>(w.p{g}[{f'k - {before}' if count > 1 else 0}], "
                   "s, b, w.step0, (int)w.n_steps, w.dt, w.grid, stop);\n")
        before += count
    src.append("}\n")
    return "".join(src)


@functools.lru_cache(maxsize=64)
def window_type(kinds: tuple):
    """The ctypes structure of a Window: per kind its Params type and its number of populations."""
    return type("Window", (ctypes.Structure,), {
        "_fields_": [("step0", ctypes.c_int64), ("dt", ctypes.c_double), ("grid", Grid), ("n_steps", ctypes.c_int64),
                     ("first", ctypes.c_int32 * (sum(count for _, count in kinds) + 1))]
                    + [(f"p{g}", t * count) for g, (t, count) in enumerate(kinds)]})

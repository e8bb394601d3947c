// Surrogate-gradient BPTT of a recurrent LIF layer with delayed sparse recurrence (include/naer2b.h,
// n2b_bptt_*). No counterpart in the reference: naer2 has no differentiable path.
//
// Model, per sample b, hidden neuron i, step t (dt = 1 step):
//   R[t][i]     = sum over incoming links k of i: w_k * s[t - d_k][pre_k]          (d_k in 1..5 steps)
//   Vpre[t][i]  = alpha * V[t-1][i] + U[t][i] + R[t][i]                             (U: input current)
//   s[t][i]     = Vpre >= theta  (spiking)   |   f(Vpre - theta), f(x) = x / (1 + slope |x|)  (smooth)
//   V[t][i]     = Vpre - theta * s[t][i]                                            (subtractive reset)
//   O[t][r]     = beta * O[t-1][r] + sum_i w_out[i][r] * s[t][i];   m[r] = max_t O[t][r] at t*[r]
// Backward (q = dL/dVpre, g = f'(Vpre - theta) = 1 / (1 + slope |Vpre - theta|)^2, the fast-sigmoid
// surrogate in the spiking model, the true derivative in the smooth one; the reset is differentiated):
//   o[t][r]  = dm[r] * [t == t*[r]] + beta * o[t+1][r]
//   q[t][i]  = alpha q[t+1][i] + g[t][i] * (sum_{k out of i} w_k q[t + d_k][post_k]
//                                           + sum_r w_out[i][r] o[t][r] - theta alpha q[t+1][i])
//   dU[t][i] = q[t][i];  dw_k = sum_t,b s[t - d_k][pre_k] q[t][post_k];  dw_out[i][r] = sum_t,b s[t][i] o[t][r]
//
// Layout: a group of 8 CTAs runs 8 samples; CTA `rank` owns hidden neurons [rank*HC, rank*HC + HC), HC = H/8.
// Spiking forward (fwd_group_kernel) and adjoint (bwd_kernel): eight threads per neuron, groups of one cooperative
// launch (one CTA per SM: at that size only 15 clusters of 8 are resident on 148 SMs, but every group must be) that
// exchange a step's spikes, or its q, through the L2. The smooth model, rows that do not fit a CTA's shared memory, short
// sequences and many groups (scans) take fwd_kernel: four threads per neuron (two samples each), the group a
// thread-block cluster, every CTA writing its neurons' entries into all 8 CTAs' spike rings (distributed shared memory)
// before one cluster barrier.
// The forward keeps the last spikes of all H neurons for its 8 samples in shared memory (one byte of 8 sample bits per
// neuron, or 8 floats in the smooth model). Backward: what it needs of the forward is the surrogate's derivative of
// every step. Up to FULL_TAPE_BYTES the forward keeps them; past that each K-step segment is first recomputed from its
// membrane checkpoint and the stored spikes by two grid-wide kernels (the recurrent inputs of all its steps at once,
// then one membrane scan per neuron and sample; same arithmetic, same order: the same Vpre bit for bit). The adjoint
// runs all steps, or the segment, backwards in one cooperative launch: q of all neurons is exchanged through a two-slot
// ring in global memory, and each neuron pushes its outgoing rows' q sums into a 6-slot ring of its own partials,
// kept in global memory between the segments' launches.
// Every sum has a fixed order (no float atomics), so results are bit-for-bit reproducible.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>

#include "../../include/naer2b.h"

namespace cg = cooperative_groups;

namespace n2b_bptt {

constexpr int NS = 8;          // samples per cluster
constexpr int CL = 8;          // CTAs per cluster
constexpr int NT = 4;          // threads per neuron
constexpr int SPT = NS / NT;   // samples per thread
constexpr int RING = 6;        // spike / partial ring slots (delays 1..5)
constexpr int MAXD = 5;
constexpr unsigned FULL = 0xffffffffu;

struct Args {
    int B, T, H, R, K, HC, NC, nseg, nnz;
    float alpha, beta, theta, slope;
    int tape, csr_smem;
    const int32_t *in_ptr;
    const uint16_t *in_code;
    const float *in_w;
    const int32_t *out_grp;  // [H][MAXD + 1]: row start of each delay 1..5, then the row end
    const uint16_t *out_code;
    const float *out_w;
    const float *U;     // [T][B][H]
    uint8_t *s_bits;    // [T][NC][H]      (spiking)
    float *s_f;         // [T][NC][H][8]   (smooth)
    float *v_ckpt;      // [nseg][B][H]
    float *g_seg;       // [K][B][H]: the segment's recurrent input, then its surrogate derivatives
    unsigned long long *xw;  // [NC][XSLOTS][H / 4]: the forward's published words
    float *tot;         // [T][B][R]: every step's readout sums
    float *g_all;       // [T][B][H]: every step's surrogate derivatives, or null (segments recomputed)
    float *dU;          // [T][B][H]
    const float *w_out; // [H][R]
    float *m;           // [B][R]
    int32_t *tstar;     // [B][R]
    const float *dm;    // [B][R]
    const int32_t *tstar_in;
    float *dwp;         // [NC][nnz] per-cluster dw, out order
    float *dwo_p;       // [NC][H][R]
    float *part_st;     // [NC * CL][RING][HC][NS] the adjoint's partial ring between segments
    float *q_st;        // [B][H] q[t0] of the last segment done
    float *o_st;        // [B][R] the readout adjoint at t0
    float *qx;          // [NC][2][H][8] the adjoint's q exchange ring (slot t & 1)
    uint32_t *qflag;    // [NC][2][H / 4] its flags, one per warp (cleared before a call's first launch)
    float *o_all;       // [T][B][R]: every step's readout adjoint (all steps in one launch)
    int32_t *err;       // [N2B_BPTT_ERR_WORDS]
    int wait_polls;     // polls before a wait of the per-step exchange gives up
};

__device__ __forceinline__ float surrogate(float x, float slope) {
    const float a = __fadd_rn(1.f, __fmul_rn(slope, fabsf(x)));
    return __fdiv_rn(1.f, __fmul_rn(a, a));
}

__device__ __forceinline__ float smooth_spike(float x, float slope) {
    return __fdiv_rn(x, __fadd_rn(1.f, __fmul_rn(slope, fabsf(x))));
}

// v[k] of a thread's two samples: (sub's samples 2 sub, 2 sub + 1) with compile-time indices only.
__device__ __forceinline__ void mine(const float v[NS], int sub, float &x0, float &x1) {
    x0 = sub == 0 ? v[0] : sub == 1 ? v[2] : sub == 2 ? v[4] : v[6];
    x1 = sub == 0 ? v[1] : sub == 1 ? v[3] : sub == 2 ? v[5] : v[7];
}

// Shared-memory layout of the forward kernel (identical in every CTA, so that remote addresses match).
struct FwdSmem {
    size_t ring, xbuf, wout, ptr, code, w, total;
};
__host__ __device__ inline FwdSmem fwd_smem(int H, int HC, int R, bool smooth, bool csr_smem, int in_cta_max) {
    FwdSmem L{};
    size_t o = 0;
    auto a16 = [](size_t x) { return (x + 15) & ~size_t(15); };
    L.ring = o; o = a16(o + (smooth ? sizeof(float) * RING * H * NS : (size_t)RING * H));
    L.xbuf = o; o = a16(o + sizeof(float) * 2 * CL * NS * R);
    L.wout = o; o = a16(o + sizeof(float) * HC * R);
    L.ptr = o; o = a16(o + sizeof(int32_t) * (HC + 1));
    L.code = o; o = a16(o + (csr_smem ? sizeof(uint16_t) * in_cta_max : 0));
    L.w = o; o = a16(o + (csr_smem ? sizeof(float) * in_cta_max : 0));
    L.total = o;
    return L;
}

struct BwdSmem {
    size_t pnew, part, dwo, obuf, grp, code, w, dw, total;
};
__host__ __device__ inline BwdSmem bwd_smem(int H, int HC, int R, int out_cta_max, bool full) {
    BwdSmem L{};
    size_t o = 0;
    auto a16 = [](size_t x) { return (x + 15) & ~size_t(15); };
    L.pnew = o; o = a16(o + sizeof(float) * H * NS);
    L.part = o; o = a16(o + sizeof(float) * RING * HC * NS);
    L.dwo = o; o = a16(o + (full ? 0 : sizeof(float) * HC * R));
    L.obuf = o; o = a16(o + (full ? 0 : sizeof(float) * 2 * NS * R));  // o[t] in half t & 1
    L.grp = o; o = a16(o + sizeof(int32_t) * HC * (MAXD + 1));
    L.code = o; o = a16(o + sizeof(uint16_t) * out_cta_max);
    L.w = o; o = a16(o + sizeof(float) * out_cta_max);
    L.dw = o; o = a16(o + sizeof(float) * out_cta_max);
    L.total = o;
    return L;
}

// The forward's exchange between a group's CTAs, step by step: four neurons' spikes are published as one 64-bit word, the
// step's number + 1 beside the 32 bits, and every CTA polls the words themselves (one write and one read through the
// L2; no fence, counter or barrier). The words are cleared before a call's first launch. Polls are bounded, here and in
// the adjoint: one that gives up counts in err[3] and sets the CTA's `aborted`, after which it polls no more -- it
// publishes its own words all the same, so that neither it nor the CTAs that wait for them can hang.
constexpr int XCHG_SPIN_LIMIT = 1 << 21;  // default polls (n2b_bptt_desc.wait_polls = 0): about a second
__device__ __forceinline__ void publish(unsigned long long *p, uint32_t word, uint32_t tag) {
    const unsigned long long v = ((unsigned long long)tag << 32) | word;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// The word published under `tag`, polled for at most `limit` times.
__device__ __forceinline__ bool await(const unsigned long long *p, uint32_t tag, int limit, uint32_t &word) {
    for (int it = 0; it < limit; ++it) {
        unsigned long long v;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
        if ((uint32_t)(v >> 32) == tag) {
            word = (uint32_t)v;
            return true;
        }
    }
    return false;
}

// The spikes that the incoming links read: the forward's shared-memory ring (6 slots, the slot of step t in
// t mod 6; slots of steps before 0 are still zero), or the stored spikes of every step (recompute).
struct RingSrc {
    const unsigned char *ring;
    int H, tbase;  // t mod 6
    __device__ __forceinline__ int slot(int d) const {
        const int sl = tbase - d;
        return sl < 0 ? sl + RING : sl;
    }
};
struct TapeSrc {
    const uint8_t *bits;
    const float *f;
    int H, NC, q, t;
};

// R for the 8 samples of one neuron: this thread's share of its incoming row (links rs + sub, rs + sub + NT,
// ...), then the NT shares added pairwise ((s0 + s1) + (s2 + s3), the same value in all NT lanes).
// CHECKED: every code is checked (a bad one counted and skipped); otherwise the rows were validated when they
// were copied (bad links replaced by a zero-weight link). Both give the same sums for the same rows.
template <bool SMOOTH, bool CHECKED, class Src>
__device__ __forceinline__ void gather_in(const Args &a, const Src &src, const uint16_t *code, const float *w,
                                          int rs, int re, int sub, float acc[NS]) {
#pragma unroll
    for (int b = 0; b < NS; ++b) acc[b] = 0.f;
#pragma unroll 2
    for (int l = rs + sub; l < re; l += NT) {
        const uint32_t c = code[l];
        const float wl = w[l];
        const int pre = (int)(c & 0x7FFu), d = (int)(c >> 11);
        if (CHECKED && (d < 1 || d > MAXD || pre >= a.H)) {
            atomicAdd(a.err + 0, 1);
            continue;
        }
        if constexpr (SMOOTH) {
            float s[NS];
            if constexpr (std::is_same<Src, RingSrc>::value) {
                const float4 *p = reinterpret_cast<const float4 *>(src.ring) + ((size_t)src.slot(d) * src.H + pre) * 2;
                const float4 x = p[0], y = p[1];
                s[0] = x.x; s[1] = x.y; s[2] = x.z; s[3] = x.w; s[4] = y.x; s[5] = y.y; s[6] = y.z; s[7] = y.w;
            } else {
                const int tt = src.t - d;
                if (tt < 0) continue;
                const float4 *p = reinterpret_cast<const float4 *>(src.f) + (((size_t)tt * src.NC + src.q) * src.H + pre) * 2;
                const float4 x = p[0], y = p[1];
                s[0] = x.x; s[1] = x.y; s[2] = x.z; s[3] = x.w; s[4] = y.x; s[5] = y.y; s[6] = y.z; s[7] = y.w;
            }
#pragma unroll
            for (int b = 0; b < NS; ++b) acc[b] = __fadd_rn(acc[b], __fmul_rn(wl, s[b]));
        } else {
            uint32_t byte;
            if constexpr (std::is_same<Src, RingSrc>::value) {
                byte = src.ring[(size_t)src.slot(d) * src.H + pre];
            } else {
                const int tt = src.t - d;
                byte = tt >= 0 ? src.bits[((size_t)tt * src.NC + src.q) * src.H + pre] : 0u;
            }
            if (!byte) continue;
#pragma unroll
            for (int b = 0; b < NS; ++b)
                if ((byte >> b) & 1u) acc[b] = __fadd_rn(acc[b], wl);
        }
    }
#pragma unroll
    for (int b = 0; b < NS; ++b) acc[b] = __fadd_rn(acc[b], __shfl_xor_sync(FULL, acc[b], 1));
#pragma unroll
    for (int b = 0; b < NS; ++b) acc[b] = __fadd_rn(acc[b], __shfl_xor_sync(FULL, acc[b], 2));
}

// One membrane step of one sample: returns the spike value, updates V, gives Vpre.
template <bool SMOOTH>
__device__ __forceinline__ float lif_step(const Args &a, float &V, float u, float r, float &vpre) {
    const float vp = __fadd_rn(__fadd_rn(__fmul_rn(a.alpha, V), u), r);
    float s;
    if constexpr (SMOOTH) s = smooth_spike(__fadd_rn(vp, -a.theta), a.slope);
    else s = vp >= a.theta ? 1.f : 0.f;
    V = __fadd_rn(vp, -__fmul_rn(a.theta, s));
    vpre = vp;
    return s;
}

// ------------------------------------------------------------------------------------------------ forward

// DERIV: it keeps the surrogate derivatives of every step (a.g_all; a kernel of its own: 4% of the plain forward).
template <bool SMOOTH, bool DERIV>
__global__ void __launch_bounds__(512) fwd_kernel(const __grid_constant__ Args a, int in_cta_max) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int q = (int)blockIdx.x / CL;
    const int H = a.H, HC = a.HC, R = a.R, B = a.B;
    const int h0 = rank * HC;
    const bool csr = a.csr_smem != 0;
    const FwdSmem L = fwd_smem(H, HC, R, SMOOTH, csr, in_cta_max);
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned char *ring = smem + L.ring;
    float *xbuf = reinterpret_cast<float *>(smem + L.xbuf);
    float *wout = reinterpret_cast<float *>(smem + L.wout);
    int32_t *lptr = reinterpret_cast<int32_t *>(smem + L.ptr);
    const int tid = threadIdx.x, nthr = blockDim.x;

    for (size_t k = tid; k < (L.xbuf - L.ring) / 4; k += nthr) reinterpret_cast<uint32_t *>(ring)[k] = 0u;
    for (int k = tid; k < HC * R; k += nthr) wout[k] = a.w_out[(size_t)h0 * R + k];
    const int base = a.in_ptr[h0];
    for (int k = tid; k <= HC; k += nthr) lptr[k] = a.in_ptr[h0 + k] - base;
    const uint16_t *gcode = a.in_code + base;
    const float *gw = a.in_w + base;
    const int n_in = a.in_ptr[h0 + HC] - base;
    const bool in_smem = csr && n_in <= in_cta_max;
    if (csr && !in_smem && tid == 0) atomicAdd(a.err + 2, 1);  // a wrong in_cta_max: the rows stay global
    uint16_t *sc = reinterpret_cast<uint16_t *>(smem + L.code);
    float *sw = reinterpret_cast<float *>(smem + L.w);
    if (in_smem) {
        for (int k = tid; k < n_in; k += nthr) {  // validated once: a bad link becomes a zero-weight link
            const uint32_t c = gcode[k];
            const bool bad = (c >> 11) < 1 || (c >> 11) > MAXD || (c & 0x7FFu) >= (uint32_t)H;
            if (bad) atomicAdd(a.err + 0, 1);
            sc[k] = bad ? (uint16_t)(1u << 11) : (uint16_t)c;
            sw[k] = bad ? 0.f : gw[k];
        }
    }
    __syncthreads();
    cl.sync();  // every CTA's shared memory is initialised before any remote write reaches it

    const bool nt = tid < NT * HC;
    const int pl = nt ? tid / NT : 0, sub = tid % NT;
    const int post = h0 + pl;
    const int rs = nt ? lptr[pl] : 0, re = nt ? lptr[pl + 1] : 0;
    float V0 = 0.f, V1 = 0.f;
    const bool ro = tid < NS * R;
    const int rb = ro ? tid / R : 0, rr = ro ? tid % R : 0;
    float O = 0.f, mx = -INFINITY;
    int ts = -1;
    const size_t bq = (size_t)q * NS + SPT * sub;  // this thread's first sample

    for (int t = 0; t < a.T; ++t) {
        if (!DERIV && a.tape && t % a.K == 0 && nt) {
            a.v_ckpt[((size_t)(t / a.K) * B + bq) * H + post] = V0;
            a.v_ckpt[((size_t)(t / a.K) * B + bq + 1) * H + post] = V1;
        }
        float acc[NS];
        const RingSrc src{ring, H, t % RING};
        if (in_smem) gather_in<SMOOTH, false>(a, src, sc, sw, rs, re, sub, acc);
        else gather_in<SMOOTH, true>(a, src, gcode, gw, rs, re, sub, acc);
        float r0, r1, s0 = 0.f, s1 = 0.f, vp;
        mine(acc, sub, r0, r1);
        if (nt) {
            const float u0 = __ldg(a.U + ((size_t)t * B + bq) * H + post);
            const float u1 = __ldg(a.U + ((size_t)t * B + bq + 1) * H + post);
            float vp1;
            s0 = lif_step<SMOOTH>(a, V0, u0, r0, vp);
            s1 = lif_step<SMOOTH>(a, V1, u1, r1, vp1);
            if constexpr (DERIV) {
                float *g = a.g_all + ((size_t)t * B + bq) * H + post;
                __stcs(g, surrogate(__fadd_rn(vp, -a.theta), a.slope));
                __stcs(g + H, surrogate(__fadd_rn(vp1, -a.theta), a.slope));
            }
        }
        const int slot = t % RING;
        if constexpr (SMOOTH) {
            if (nt) {
                const float2 v = make_float2(s0, s1);
                float2 *dst = reinterpret_cast<float2 *>(ring) + ((size_t)slot * H + post) * 4 + sub;
                for (int k = 0; k < CL; ++k) *cl.map_shared_rank(dst, k) = v;
                if (a.tape) reinterpret_cast<float2 *>(a.s_f)[(((size_t)t * a.NC + q) * H + post) * 4 + sub] = v;
            }
        } else {
            uint32_t bits = ((s0 != 0.f) ? 1u : 0u) | ((s1 != 0.f) ? 2u : 0u);
            bits <<= SPT * sub;
            bits |= __shfl_xor_sync(FULL, bits, 1);
            bits |= __shfl_xor_sync(FULL, bits, 2);
            if (nt) {
                unsigned char *dst = ring + (size_t)slot * H + post;
                for (int k = sub; k < CL; k += NT) *cl.map_shared_rank(dst, k) = (unsigned char)bits;
                if (a.tape && sub == 0) a.s_bits[((size_t)t * a.NC + q) * H + post] = (uint8_t)bits;
            }
        }
        __syncthreads();  // this CTA's own neurons' entries are in its ring
        if (ro) {
            float sum = 0.f;
            if constexpr (SMOOTH) {
                const float *rf = reinterpret_cast<const float *>(ring) + ((size_t)slot * H + h0) * NS + rb;
                for (int p = 0; p < HC; ++p) sum = __fadd_rn(sum, __fmul_rn(rf[(size_t)p * NS], wout[p * R + rr]));
            } else {  // four neurons' bytes per word, neurons in ascending order
                const uint32_t *rw = reinterpret_cast<const uint32_t *>(ring + (size_t)slot * H + h0);
                for (int k = 0; k < HC / 4; ++k) {
                    const uint32_t word = rw[k];
                    if (!word) continue;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if ((word >> (8 * j + rb)) & 1u) sum = __fadd_rn(sum, wout[(4 * k + j) * R + rr]);
                }
            }
            float *dst = xbuf + (((size_t)(t & 1) * CL + rank) * NS + rb) * R + rr;
            *cl.map_shared_rank(dst, 0) = sum;
        }
        cl.sync();  // step t's spikes in every ring, its readout partials in rank 0
        if (rank == 0 && ro) {
            float tot = 0.f;
            for (int k = 0; k < CL; ++k) tot = __fadd_rn(tot, xbuf[(((size_t)(t & 1) * CL + k) * NS + rb) * R + rr]);
            O = __fadd_rn(__fmul_rn(a.beta, O), tot);
            if (O > mx) {
                mx = O;
                ts = t;
            }
        }
    }
    if (rank == 0 && ro) {
        a.m[(size_t)(q * NS + rb) * R + rr] = mx;
        a.tstar[(size_t)(q * NS + rb) * R + rr] = ts;
    }
    cl.sync();  // no CTA leaves while another may still address its shared memory
}

// ------------------------------------------------------------------------------------------------ forward, by spikes

// The spiking forward with the incoming rows in shared memory: a group of 8 CTAs of one cooperative launch, a CTA per
// SM (clusters of 8 would not do: 16 of them do not fit 148 SMs one CTA each, and two CTAs on an SM halve the pace of
// their groups, and so of the launch). A step is a chain -- the group's spikes of the step before, each row's look at
// its sources, the sums in link order, the new spikes -- of which little is arithmetic, so:
//   - a warp publishes its four neurons' spikes as one 64-bit word, the step's number beside the 32 bits, and every
//     CTA polls the group's words themselves: one write and one read through the L2, no fence, counter or barrier;
//   - which of a row's links of delay 2..5 have a spike (one byte load and a bit each; the codes are the byte's address
//     past the step's, four to a 64-bit load) is found before the step's words are there;
//   - only those links and the delay-1 links are then added, in link order: fwd_kernel's sums bit for bit (a link
//     without a spike adds nothing there either);
//   - the input currents are loaded two steps ahead, and the readout is a pair of kernels of its own over the spikes
//     (its sums do not feed the recurrence).
// Measured at batch 128, 500 steps, 1024 hidden neurons of 102 links, 1.9% of them spiking: 4.18 ms in fwd_kernel, 1.71 ms
// here (1.9 with the readout's kernels).
constexpr int NB = NS;        // threads per neuron: one sample each; in the link loops four link shares times two halves
constexpr int LS = NB / 2;    // of the samples
constexpr int SLOTS = 8;      // spike ring slots in shared memory (t & 7)
constexpr int XSLOTS = 4;     // slots of the group's published words (t & 3)
constexpr int WORD_LINKS = 32, MASK_LINKS = 2 * WORD_LINKS;  // links of a share with a place in its masks
constexpr int NEAR_REGS = 4;  // delay-1 links a thread holds in registers (a share has about five, two lanes look at them)
constexpr size_t SMEM_MAX = 227 * 1024;

struct ScanSmem {
    size_t ring, ptr, row, code, w, total;
};
__host__ __device__ inline int scan_stride(int H) {  // bytes of a ring slot: a power of two
    int s = 32;
    while (s < H) s *= 2;
    return s;
}
__host__ __device__ inline ScanSmem scan_smem(int H, int HC, int in_cta_max) {
    ScanSmem L{};
    size_t o = 0;
    auto a16 = [](size_t x) { return (x + 15) & ~size_t(15); };
    L.ring = o; o = a16(o + (size_t)SLOTS * scan_stride(H));
    L.ptr = o; o = a16(o + sizeof(int32_t) * (HC + 1));
    L.row = o; o = a16(o + sizeof(int32_t) * (HC + 1));
    // each of a row's NT shares padded to whole 64-bit loads (of a row of len links: at most len + 15 codes)
    L.code = o; o = a16(o + sizeof(uint16_t) * ((size_t)in_cta_max + 15 * HC));
    L.w = o; o = a16(o + sizeof(float) * in_cta_max);
    L.total = o;
    return L;
}
// Codes of one share of a row of len links, padded.
__host__ __device__ inline int scan_share(int len) { return ((len + NT - 1) / NT + 3) / 4 * 4; }

// Of four bytes, which have a bit in their low nibble, as four bits.
__device__ __forceinline__ uint32_t low_nibbles(uint32_t x) {
    const uint32_t t = (((x & 0x0F0F0F0Fu) + 0x0F0F0F0Fu) >> 4) & 0x01010101u;  // 15 + a nibble carries unless it is 0
    return (t * 0x00204081u) >> 21 & 0xFu;                                      // bits 0, 8, 16, 24 to 21 .. 24
}

__global__ void __launch_bounds__(NB * 128) fwd_group_kernel(const __grid_constant__ Args a, int in_cta_max, int g0) {
    const int rank = (int)blockIdx.x % CL;
    const int q = g0 + (int)blockIdx.x / CL;
    const int H = a.H, HC = a.HC, B = a.B;
    const int h0 = rank * HC, stride = scan_stride(H);
    const ScanSmem L = scan_smem(H, HC, in_cta_max);
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned char *ring = smem + L.ring;
    int32_t *lptr = reinterpret_cast<int32_t *>(smem + L.ptr);
    int32_t *row = reinterpret_cast<int32_t *>(smem + L.row);
    uint16_t *code = reinterpret_cast<uint16_t *>(smem + L.code);
    float *w = reinterpret_cast<float *>(smem + L.w);
    __shared__ int aborted;
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31;

    if (tid == 0) aborted = 0;
    for (size_t k = tid; k < L.ptr / 4; k += nthr) reinterpret_cast<uint32_t *>(ring)[k] = 0u;
    const int base = a.in_ptr[h0];
    for (int k = tid; k <= HC; k += nthr) lptr[k] = a.in_ptr[h0 + k] - base;
    __syncthreads();
    const bool in_smem = lptr[HC] <= in_cta_max;
    if (!in_smem && tid == 0) atomicAdd(a.err + 2, 1);  // a wrong in_cta_max: the rows stay global
    if (in_smem && tid < 32) {  // each row's first code
        int sum = 0;
        for (int p0 = 0; p0 < HC; p0 += 32) {
            const int p = p0 + lane;
            const int n = p < HC ? NT * scan_share(lptr[p + 1] - lptr[p]) : 0;
            int incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += v;
            }
            if (p < HC) row[p] = sum + incl - n;
            sum += __shfl_sync(FULL, incl, 31);
        }
    }
    __syncthreads();
    for (int p = tid / 32; in_smem && p < HC; p += nthr / 32) {  // a warp per row: its links, validated once
        const int rs = lptr[p], len = lptr[p + 1] - rs, share = scan_share(len);
        for (int k = lane; k < NT * share; k += 32) {  // share k / share, link number k % share of it
            const int l = (k % share) * NT + k / share;
            uint32_t c = 1u << 11;  // padding and bad links: a link of weight 0, one step from neuron 0
            if (l < len) {
                const uint32_t g = a.in_code[base + rs + l];
                const bool bad = (g >> 11) < 1 || (g >> 11) > MAXD || (g & 0x7FFu) >= (uint32_t)H;
                if (bad) atomicAdd(a.err + 0, 1);
                else c = g;
                w[rs + l] = bad ? 0.f : a.in_w[base + rs + l];
            }
            // the byte of step t - d is at ((t + 8 - d) & 7) * stride + pre
            code[row[p] + k] = (uint16_t)((SLOTS - (c >> 11)) * stride + (c & 0x7FFu));
        }
    }
    __syncthreads();

    const unsigned mask = (unsigned)(SLOTS * stride - 1);
    const bool nt = tid < NB * HC;
    const int pl = nt ? tid / NB : 0;                     // the thread's neuron
    const int half = (tid >> 2) & 1, sub = tid % LS;      // in the link loops: its half of the samples, its share
    const int own = tid % NB;                             // its sample (LS half + sub)
    const int post = h0 + pl;
    const int len = nt ? lptr[pl + 1] - lptr[pl] : 0;
    const int links = len > sub ? (len - sub + NT - 1) / NT : 0;  // of this share
    const int kept = in_smem ? links : 0;
    const uint16_t *sc = code + (in_smem ? row[pl] + sub * scan_share(lptr[pl + 1] - lptr[pl]) : 0);
    const float *sw = w + lptr[pl] + sub;
    // the codes this lane looks at before the step's words are there, of the share's first 32 links: the two halves'
    // lanes take every other group of four (padding and links past the share's end are masked out below)
    uint2 codes[WORD_LINKS / 8];
#pragma unroll
    for (int g = 0; g < WORD_LINKS / 8; ++g) {
        const int i = 8 * g + 4 * half;
        codes[g] = i < kept ? *reinterpret_cast<const uint2 *>(sc + i) : make_uint2(0u, 0u);
    }
    // the share's links of delay 1 (their spikes come with the step's words), by place; of its first 32 links' the
    // two halves' lanes hold every other one's code (and place, in the bits above 16), those past the registers stay in `rest`
    uint32_t near[2] = {0u, 0u}, rest = 0u, held[NEAR_REGS];
    {
        int k = 0;
        for (int i = 0; i < min(kept, MASK_LINKS); ++i) {
            if (sc[i] < (SLOTS - 1) * stride) continue;
            near[i / WORD_LINKS] |= 1u << (i % WORD_LINKS);
            if (i < WORD_LINKS && k++ >= 2 * NEAR_REGS) rest |= 1u << i;
        }
#pragma unroll
        for (int h = 0; h < NEAR_REGS; ++h) {
            uint32_t m = near[0];
            for (int j = 2 * h + half; j > 0 && m; --j) m &= m - 1;
            const int i = m ? __ffs(m) - 1 : 0;
            held[h] = m ? sc[i] | (uint32_t)i << 16 | 1u << 31 : 0u;
        }
    }
    uint32_t *ring32 = reinterpret_cast<uint32_t *>(ring);
    unsigned long long *xw = a.xw + (size_t)q * XSLOTS * (H / 4);
    const float *u = a.U + ((size_t)q * NS + own) * H + post;
    const size_t ustep = (size_t)B * H;
    float V = 0.f, u0 = nt ? __ldcs(u) : 0.f, u1 = (nt && a.T > 1) ? __ldcs(u + ustep) : 0.f;
    const unsigned nib = 0xFu << (LS * half);
    for (int t = 0; t < a.T; ++t) {
        const float u2 = (nt && t + 2 < a.T) ? __ldcs(u + (size_t)(t + 2) * ustep) : 0.f;
        if (a.tape && !a.g_all && t % a.K == 0 && nt)
            a.v_ckpt[((size_t)(t / a.K) * B + (size_t)q * NS + own) * H + post] = V;
        const unsigned tb = (unsigned)(t & (SLOTS - 1)) * stride;
        // which of the share's links of delay 2..5 have a spike, in either half of the samples (each lane for every
        // other group of four links; the halves exchange)
        uint32_t hit[2] = {0u, 0u};
        {
            uint32_t lo = 0u, hi = 0u;
#pragma unroll
            for (int g = 0; g < WORD_LINKS / 8; ++g) {
                const uint2 c4 = codes[g];
                const uint32_t b0 = ring[(tb + (c4.x & 0xFFFFu)) & mask], b1 = ring[(tb + (c4.x >> 16)) & mask];
                const uint32_t b2 = ring[(tb + (c4.y & 0xFFFFu)) & mask], b3 = ring[(tb + (c4.y >> 16)) & mask];
                const uint32_t all = b0 | b1 << 8 | b2 << 16 | b3 << 24;
                lo |= low_nibbles(all) << (8 * g);
                hi |= low_nibbles(all >> 4) << (8 * g);
            }
            lo <<= 4 * half;
            hi <<= 4 * half;
            hit[0] = (half ? hi : lo) | __shfl_xor_sync(FULL, half ? lo : hi, LS);
            hit[0] &= (kept < WORD_LINKS ? (1u << kept) - 1u : ~0u) & ~near[0];
        }
        if (__any_sync(FULL, kept > WORD_LINKS)) {  // rows of more than 128 links
            for (int i = WORD_LINKS; i < min(kept, MASK_LINKS); ++i)
                if (ring[(tb + sc[i]) & mask] & nib) hit[1] |= 1u << (i - WORD_LINKS);
            hit[1] |= near[1];
        }
        if (t > 0) {  // the group's spikes of step t - 1
            if (tid < H / 4) {
                uint32_t word = 0u;
                if (!*(volatile int *)&aborted &&
                    !await(xw + (size_t)((t - 1) % XSLOTS) * (H / 4) + tid, (uint32_t)t, a.wait_polls, word)) {
                    atomicAdd(a.err + 3, 1);
                    *(volatile int *)&aborted = 1;
                }
                ring32[((t - 1) & (SLOTS - 1)) * (stride / 4) + tid] = word;
            }
            __syncthreads();
        }
        {  // ... and of its links of delay 1
            uint32_t lo = 0u, hi = 0u;
#pragma unroll
            for (int h = 0; h < NEAR_REGS; ++h) {
                const uint32_t byte = ring[(tb + (held[h] & 0xFFFFu)) & mask], bit = (held[h] >> 31) << (held[h] >> 16 & 31u);
                if (byte & 0x0Fu) lo |= bit;
                if (byte & 0xF0u) hi |= bit;
            }
            hit[0] |= (half ? hi : lo) | __shfl_xor_sync(FULL, half ? lo : hi, LS);
            for (uint32_t m = rest; m; m &= m - 1) {
                const int i = __ffs(m) - 1;
                if (ring[(tb + sc[i]) & mask] & nib) hit[0] |= 1u << i;
            }
        }
        float acc[LS] = {0.f, 0.f, 0.f, 0.f};
        auto add = [&](uint32_t byte, float wl) {
            const uint32_t b = byte & nib;
            if (b & 0x11u) acc[0] = __fadd_rn(acc[0], wl);
            if (b & 0x22u) acc[1] = __fadd_rn(acc[1], wl);
            if (b & 0x44u) acc[2] = __fadd_rn(acc[2], wl);
            if (b & 0x88u) acc[3] = __fadd_rn(acc[3], wl);
        };
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            uint32_t h = hit[m];
            while (h) {  // two links' loads at a time
                const int i = m * WORD_LINKS + __ffs(h) - 1;
                h &= h - 1;
                const int j = h ? m * WORD_LINKS + __ffs(h) - 1 : i;
                const uint32_t bi = ring[(tb + sc[i]) & mask], bj = h ? ring[(tb + sc[j]) & mask] : 0u;
                const float wi = sw[NT * i], wj = sw[NT * j];
                h &= h - 1;
                add(bi, wi);
                add(bj, wj);
            }
        }
        for (int i = in_smem ? MASK_LINKS : 0; i < links; ++i) {  // links past the masks, or every link from memory
            if (in_smem) {
                add(ring[(tb + sc[i]) & mask], sw[NT * i]);
                continue;
            }
            const uint32_t g = a.in_code[base + lptr[pl] + sub + NT * i];
            const int pre = (int)(g & 0x7FFu), d = (int)(g >> 11);
            if (d < 1 || d > MAXD || pre >= H) {
                if (half == 0) atomicAdd(a.err + 0, 1);
                continue;
            }
            add(ring[(tb + (unsigned)((SLOTS - d) * stride + pre)) & mask], a.in_w[base + lptr[pl] + sub + NT * i]);
        }
        __syncwarp();
        // the shares added pairwise, (s0 + s1) + (s2 + s3); the lane keeps its own sample's
#pragma unroll
        for (int b = 0; b < LS; ++b) acc[b] = __fadd_rn(acc[b], __shfl_xor_sync(FULL, acc[b], 1));
#pragma unroll
        for (int b = 0; b < LS; ++b) acc[b] = __fadd_rn(acc[b], __shfl_xor_sync(FULL, acc[b], 2));
        float vp = 0.f, sp = 0.f;
        if (nt) sp = lif_step<false>(a, V, u0, sub == 0 ? acc[0] : sub == 1 ? acc[1] : sub == 2 ? acc[2] : acc[3], vp);
        u0 = u1;
        u1 = u2;
        // the warp's four neurons' bytes, samples in lane order
        const uint32_t word = __ballot_sync(FULL, sp != 0.f);
        if (lane == 0 && nt) {
            publish(xw + (size_t)(t % XSLOTS) * (H / 4) + (post >> 2), word, (uint32_t)t + 1u);
            *reinterpret_cast<uint32_t *>(a.s_bits + ((size_t)t * a.NC + q) * H + post) = word;
        }
        if (a.tape && a.g_all && nt)
            __stcs(a.g_all + ((size_t)t * B + (size_t)q * NS + own) * H + post, surrogate(__fadd_rn(vp, -a.theta), a.slope));
    }
}

// The readout of every step, from the stored spikes: a block per (step, group), its 8 samples' spikes as bit masks,
// then a thread per (sample, readout): sum over each eighth of the neurons in ascending order, the eighths added in
// order (as the CTAs of fwd_kernel sum and add).
constexpr int READOUT_THREADS = 256;
__global__ void __launch_bounds__(READOUT_THREADS) readout_kernel(const __grid_constant__ Args a) {
    __shared__ uint32_t bits[NS][32];
    const int t = blockIdx.x / a.NC, q = blockIdx.x % a.NC, lane = threadIdx.x & 31;
    const uint8_t *src = a.s_bits + ((size_t)t * a.NC + q) * a.H;
    for (int g = threadIdx.x / 32; g < a.H / 32; g += READOUT_THREADS / 32) {
        const uint32_t byte = src[32 * g + lane];
#pragma unroll
        for (int b = 0; b < NS; ++b) {
            const uint32_t m = __ballot_sync(FULL, (byte >> b) & 1u);
            if (lane == b) bits[b][g] = m;
        }
    }
    __syncthreads();
    for (int pair = threadIdx.x; pair < NS * a.R; pair += READOUT_THREADS) {
        const int b = pair / a.R;
        const float *w = a.w_out + pair % a.R;
        float tot = 0.f, sum = 0.f;
        int end = a.HC;  // of the eighth being summed
        for (int g = 0; g < a.H / 32; ++g)
            for (uint32_t m = bits[b][g]; m; m &= m - 1) {
                const int n = 32 * g + __ffs(m) - 1;
                if (n >= end) {  // (an eighth without a spike adds 0)
                    tot = __fadd_rn(tot, sum);
                    sum = 0.f;
                    while (n >= end) end += a.HC;
                }
                sum = __fadd_rn(sum, __ldg(w + (size_t)n * a.R));
            }
        a.tot[((size_t)t * a.NC + q) * NS * a.R + pair] = __fadd_rn(tot, sum);
    }
}

// The readouts over time: a thread per (sample, readout); MAX_AHEAD steps' sums loaded together (the loads' latency is
// what it costs).
constexpr int MAX_AHEAD = 32;
__global__ void __launch_bounds__(32) readout_max_kernel(const __grid_constant__ Args a) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, n = a.B * a.R;
    if (k >= n) return;
    float O = 0.f, mx = -INFINITY;
    int ts = -1;
    float next[MAX_AHEAD];
#pragma unroll
    for (int j = 0; j < MAX_AHEAD; ++j) next[j] = j < a.T ? a.tot[(size_t)j * n + k] : 0.f;
    for (int t0 = 0; t0 < a.T; t0 += MAX_AHEAD) {
        float v[MAX_AHEAD];
#pragma unroll
        for (int j = 0; j < MAX_AHEAD; ++j) {
            v[j] = next[j];
            const int t = t0 + MAX_AHEAD + j;
            next[j] = t < a.T ? a.tot[(size_t)t * n + k] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < MAX_AHEAD; ++j) {
            if (t0 + j >= a.T) break;
            O = __fadd_rn(__fmul_rn(a.beta, O), v[j]);
            if (O > mx) {
                mx = O;
                ts = t0 + j;
            }
        }
    }
    a.m[k] = mx;
    a.tstar[k] = ts;
}

// ------------------------------------------------------------------------------------------------ recompute

// The recurrent input R of every step of a segment [t0, t1) from the stored spikes: NT threads per
// (chunk of TC steps, cluster, neuron); each thread decodes its share of the neuron's incoming row once and
// applies every link to the TC steps of its chunk, then the NT shares are added as the forward adds them
// ((s0 + s1) + (s2 + s3), links in the forward's order within each share): the same sums bit for bit.
// A link with a bad code (counted by the forward) is clamped into range here instead of checked per step.
// Spiking model: a block is blockDim / NT neurons of one (chunk, cluster); it first stages the spike bytes of
// the MAXD + TC - 1 steps its links read, of every neuron of the cluster, as one 16-byte row per neuron in
// shared memory (steps before 0 as zero), so that a link's TC steps are one 128-bit load. Launch: grid
// (H / (blockDim / NT), NC, chunks).
constexpr int TC = 5;
constexpr int RWIN = MAXD + TC - 1;  // steps tc - MAXD .. tc + TC - 2
static_assert(RWIN <= 16, "a staged row is 16 bytes");

template <bool SMOOTH>
__global__ void __launch_bounds__(256) recompute_r_kernel(const __grid_constant__ Args a, int t0, int t1) {
    extern __shared__ __align__(16) unsigned char rows[];  // spiking: [H][16] bytes
    const int ppb = blockDim.x / NT;  // neurons per block
    const int q = blockIdx.y, tc = t0 + blockIdx.z * TC;
    const int post = blockIdx.x * ppb + threadIdx.x / NT, sub = threadIdx.x % NT;
    const int rs = a.in_ptr[post], re = a.in_ptr[post + 1];
    const int kend = min(TC, t1 - tc);  // steps of this chunk inside the segment
    float acc[TC][NS];
#pragma unroll
    for (int k = 0; k < TC; ++k)
#pragma unroll
        for (int b = 0; b < NS; ++b) acc[k][b] = 0.f;
    if constexpr (SMOOTH) {
        const int row = a.NC * a.H;  // entries between two steps of the stored spikes
        for (int l = rs + sub; l < re; l += NT) {
            const uint32_t c = a.in_code[l];
            const float wl = a.in_w[l];
            const int pre = min((int)(c & 0x7FFu), a.H - 1), d = min(max((int)(c >> 11), 1), MAXD);
            const int base = (tc - d) * row + q * a.H + pre;  // step tc - d
#pragma unroll
            for (int k = 0; k < TC; ++k) {
                if (tc + k - d < 0 || k >= kend) continue;
                const float4 *p = reinterpret_cast<const float4 *>(a.s_f) + (size_t)(base + k * row) * 2;
                const float4 x = p[0], y = p[1];
                const float sv[NS] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
                for (int b = 0; b < NS; ++b) acc[k][b] = __fadd_rn(acc[k][b], __fmul_rn(wl, sv[b]));
            }
        }
    } else {
        // stage: thread j packs the RWIN bytes of neurons j, j + blockDim, ... (coalesced byte loads per step)
        for (int pre = threadIdx.x; pre < a.H; pre += blockDim.x) {
            uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int sidx = 0; sidx < RWIN; ++sidx) {
                const int tt = tc - MAXD + sidx;
                const uint32_t byte = (tt >= 0 && tt < a.T) ? a.s_bits[((size_t)tt * a.NC + q) * a.H + pre] : 0u;
                w[sidx / 4] |= byte << (8 * (sidx % 4));
            }
            reinterpret_cast<uint4 *>(rows)[pre] = make_uint4(w[0], w[1], w[2], w[3]);
        }
        __syncthreads();
        for (int l = rs + sub; l < re; l += NT) {
            const uint32_t c = a.in_code[l];
            const float wl = a.in_w[l];
            const int pre = min((int)(c & 0x7FFu), a.H - 1), d = min(max((int)(c >> 11), 1), MAXD);
            const uint4 v = reinterpret_cast<const uint4 *>(rows)[pre];
            const uint64_t lo = ((uint64_t)v.y << 32) | v.x, hi = ((uint64_t)v.w << 32) | v.z;
            const int sh = 8 * (MAXD - d);  // byte of step tc - d
            const uint64_t win = sh ? (lo >> sh) | (hi << (64 - sh)) : lo;  // steps tc - d ...
            if (!(win & ((1ull << (8 * TC)) - 1))) continue;
            // branch-free: a clear bit adds +0.0f, which leaves a sum that started at +0 unchanged bit for bit
            // (it is never -0), so the sums stay the forward's
#pragma unroll
            for (int k = 0; k < TC; ++k) {
                const uint32_t byte = k < kend ? (uint32_t)(win >> (8 * k)) & 0xffu : 0u;
#pragma unroll
                for (int b = 0; b < NS; ++b) acc[k][b] = __fadd_rn(acc[k][b], ((byte >> b) & 1u) ? wl : 0.f);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < TC; ++k) {
#pragma unroll
        for (int b = 0; b < NS; ++b) acc[k][b] = __fadd_rn(acc[k][b], __shfl_xor_sync(FULL, acc[k][b], 1));
#pragma unroll
        for (int b = 0; b < NS; ++b) acc[k][b] = __fadd_rn(acc[k][b], __shfl_xor_sync(FULL, acc[k][b], 2));
    }
    const size_t bq = (size_t)q * NS + SPT * sub;
#pragma unroll
    for (int k = 0; k < TC; ++k) {
        if (k >= kend) break;
        float r0, r1;
        mine(acc[k], sub, r0, r1);
        a.g_seg[((size_t)(tc + k - t0) * a.B + bq) * a.H + post] = r0;
        a.g_seg[((size_t)(tc + k - t0) * a.B + bq + 1) * a.H + post] = r1;
    }
}

// The membrane of the segment from its checkpoint, one thread per (sample, neuron): Vpre as the forward made it,
// its surrogate derivative over R in g_seg, and a check that the stored spike is the one Vpre gives.
template <bool SMOOTH>
__global__ void __launch_bounds__(256) recompute_v_kernel(const __grid_constant__ Args a, int seg, int t0, int t1) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.B * a.H) return;
    const int b = k / a.H, j = k % a.H, q = b / NS, bl = b % NS;
    float V = a.v_ckpt[(size_t)seg * a.B * a.H + k];
    int bad = 0;
    for (int t = t0; t < t1; ++t) {
        float *gp = a.g_seg + (size_t)(t - t0) * a.B * a.H + k;
        const float u = __ldg(a.U + (size_t)t * a.B * a.H + k);
        float vp;
        const float s = lif_step<SMOOTH>(a, V, u, *gp, vp);
        float stored;
        if constexpr (SMOOTH) stored = a.s_f[(((size_t)t * a.NC + q) * a.H + j) * NS + bl];
        else stored = ((a.s_bits[((size_t)t * a.NC + q) * a.H + j] >> bl) & 1u) ? 1.f : 0.f;
        bad += s != stored;
        *gp = surrogate(__fadd_rn(vp, -a.theta), a.slope);
    }
    if (bad) atomicAdd(a.err + 1, bad);  // the recompute differs from the forward
}

// ------------------------------------------------------------------------------------------------ adjoint

// The adjoint's threads: NB per neuron, one sample each -- or, in the link loops, LS link shares of a row times two
// halves of the samples, a 16-byte load of a q row per lane. A step is bound by shared memory: 13,000 links per CTA
// read 32 bytes of q each. What else the loads cost is kept down: a quarter warp reads four links of one neuron, whose
// rows lie in different banks (32 bytes each, targets distinct mod 4: bank_order in bptt.py), lanes past a row's end
// load nothing, and every neuron's loop ends at its own row. At 1024 hidden neurons of 102 links, 128 samples and
// 500 steps: 5.3 ms (with 4 threads a neuron, a recomputation of each segment and a cluster barrier per step 6.9).

// One delay group of a neuron's outgoing row: acc[b] += w q[post][4 half + b] over this lane's share of the links
// (gs + sub, gs + sub + LS, ...). With DW (some lane's neuron spiked at the links' step), the lanes with `dwl` also
// add sum_b s[b] q[post][b] to dw[l]: each half its samples' sum, then the pair's to dw by half 0. A skipped code
// (0xFFFF) adds nothing. Every lane of the warp calls it; the loop's length is the warp's.
template <bool SMOOTH, bool DW>
__device__ __forceinline__ void out_group(const uint16_t *ocode, const float *ow, const float *pnew, float *dw,
                                          int gs, int ge, int sub, int half, bool dwl, uint32_t sbyte,
                                          const float sf[LS], float acc[LS]) {
    const int rounds = (int)__reduce_max_sync(FULL, (unsigned)max(0, (ge - gs - sub + LS - 1) / LS));
    const float4 *rows = reinterpret_cast<const float4 *>(pnew) + half;
    int l = gs + sub;
#pragma unroll 2
    for (int k = 0; k < rounds; ++k, l += LS) {
        const uint32_t c = l < ge ? ocode[l] : 0xFFFFu;
        const bool ok = c != 0xFFFFu;
        float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
        float wl = 0.f;
        if (ok) {
            y = rows[2 * (c & 0x7FFu)];  // < H: checked when the rows were copied
            wl = ow[l];
        }
        acc[0] = __fmaf_rn(wl, y.x, acc[0]);
        acc[1] = __fmaf_rn(wl, y.y, acc[1]);
        acc[2] = __fmaf_rn(wl, y.z, acc[2]);
        acc[3] = __fmaf_rn(wl, y.w, acc[3]);
        if constexpr (DW) {
            float dk = 0.f;
            if constexpr (SMOOTH) {
                dk = __fmaf_rn(sf[3], y.w, __fmaf_rn(sf[2], y.z, __fmaf_rn(sf[1], y.y, __fmul_rn(sf[0], y.x))));
            } else {
                if (sbyte & 1u) dk = y.x;
                if (sbyte & 2u) dk = __fadd_rn(dk, y.y);
                if (sbyte & 4u) dk = __fadd_rn(dk, y.z);
                if (sbyte & 8u) dk = __fadd_rn(dk, y.w);
            }
            dk = __fadd_rn(dk, __shfl_xor_sync(FULL, dk, 1));
            if (dwl && ok && half == 0) dw[l] = __fadd_rn(dw[l], dk);
        }
    }
}

// The adjoint of the steps [t0, t1), run backwards; `first`: the last steps of the sequence (state starts at
// zero), else the state of the segment after it is loaded (partial ring, q, readout adjoint, dw, dw_out).
// Each step, every warp writes the q[t] of its four neurons into slot t & 1 of the group's ring in global memory and
// releases a flag (the step's number + 1) after them; later (the links of q[t + 1] in between) every CTA polls the group's
// flags and copies the q[t] of all H neurons into its own shared buffer (pnew). Two slots suffice: a slot t & 1 is written
// only after its CTA has every q[t + 1], which each CTA releases after its copy of q[t + 2]. (Published like the
// forward's words, q would be twice the bytes to copy: 5.75 ms for the kernel at the workload's size, 5.26 this way.)
// The launch is cooperative, so the CTAs of a group are resident together; `g0` is the launch's first group.
// FULL: all steps in one launch. What of a step does not depend on q is then made beforehand by kernels of its own --
// the readout's part of dL/ds (readout_dV_kernel, left in dU, where q[t] takes its place) and dw_out (dwo_kernel).
template <bool SMOOTH, bool FULL>
__global__ void __launch_bounds__(NB * 128) bwd_kernel(const __grid_constant__ Args a, int out_cta_max, int t0, int t1,
                                                       int first, int g0) {
    const int rank = (int)blockIdx.x % CL;
    const int q = g0 + (int)blockIdx.x / CL;
    const int H = a.H, HC = a.HC, R = a.R, B = a.B;
    const int h0 = rank * HC;
    const BwdSmem L = bwd_smem(H, HC, R, out_cta_max, FULL);
    extern __shared__ __align__(16) unsigned char smem[];
    float *pnew = reinterpret_cast<float *>(smem + L.pnew);
    float *part = reinterpret_cast<float *>(smem + L.part);
    const float *wout = a.w_out + (size_t)h0 * R;  // read through L1
    float *dwo = reinterpret_cast<float *>(smem + L.dwo);
    float *obuf = reinterpret_cast<float *>(smem + L.obuf);
    int32_t *grp = reinterpret_cast<int32_t *>(smem + L.grp);
    uint16_t *ocode = reinterpret_cast<uint16_t *>(smem + L.code);
    float *ow = reinterpret_cast<float *>(smem + L.w);
    float *dw = reinterpret_cast<float *>(smem + L.dw);
    const int tid = threadIdx.x, nthr = blockDim.x;
    float *part_st = a.part_st + ((size_t)q * CL + rank) * RING * HC * NS;  // this group's CTA, in any launch

    const bool nt = tid < NB * HC;
    const int pl = nt ? tid / NB : 0;                 // the thread's neuron
    const int half = tid & 1, sub = (tid >> 1) % LS;  // in the link loops: its half of the samples, its share
    const int own = LS * half + sub;                  // its sample
    const int me = h0 + pl;                           // its neuron (the pre of its outgoing row)
    const int obase = a.out_grp[(size_t)h0 * (MAXD + 1)];
    const int on_all = a.out_grp[(size_t)(h0 + HC - 1) * (MAXD + 1) + MAXD] - obase;
    const int on = min(on_all, out_cta_max);  // a wrong out_cta_max: the links past it are skipped, counted
    if (on_all > on && tid == 0) atomicAdd(a.err + 2, 1);
    for (size_t k = tid; k < L.total / 4; k += nthr) reinterpret_cast<uint32_t *>(smem)[k] = 0u;
    __syncthreads();
    for (int k = tid; k < HC * (MAXD + 1); k += nthr) grp[k] = min(a.out_grp[(size_t)h0 * (MAXD + 1) + k] - obase, on);
    // the outgoing rows, validated once: a link whose target is out of range or whose delay is not its group's
    // becomes the code 0xFFFF (skipped) and is counted
    if (nt) {
        for (int d = 1; d <= MAXD; ++d) {
            const int gs = min(a.out_grp[(size_t)me * (MAXD + 1) + d - 1] - obase, on);
            const int ge = min(a.out_grp[(size_t)me * (MAXD + 1) + d] - obase, on);
            for (int l = gs + own; l < ge; l += NB) {
                const uint32_t c = a.out_code[obase + l];
                const bool bad = (int)(c >> 11) != d || (c & 0x7FFu) >= (uint32_t)H;
                if (bad) atomicAdd(a.err + 0, 1);
                ocode[l] = bad ? (uint16_t)0xFFFFu : (uint16_t)c;
                ow[l] = a.out_w[obase + l];
            }
        }
    }
    if (!first) {
        for (int k = tid; k < RING * HC * NS; k += nthr) part[k] = part_st[k];
        for (int k = tid; k < on; k += nthr) dw[k] = a.dwp[(size_t)q * a.nnz + obase + k];
        for (int k = tid; k < HC * R; k += nthr) dwo[k] = a.dwo_p[((size_t)q * H + h0) * R + k];
    }
    __shared__ int aborted;
    if (tid == 0) aborted = 0;
    __syncthreads();

    const size_t bq = (size_t)q * NS + own;  // this thread's sample
    const bool ro = !FULL && tid < NS * R;
    const int rb = ro ? tid / R : 0, rr = ro ? tid % R : 0;
    const float dmv = ro ? a.dm[(size_t)(q * NS + rb) * R + rr] : 0.f;
    const int tsv = ro ? a.tstar_in[(size_t)(q * NS + rb) * R + rr] : -1;
    float o = (ro && !first) ? a.o_st[(size_t)(q * NS + rb) * R + rr] : 0.f;
    float qp = (nt && !first) ? a.q_st[bq * H + me] : 0.f;  // q[t + 1] of this thread's sample

    // this neuron's spikes at step tt (0 before step 0): the 8 samples' bits, or (smooth) the floats of this lane's
    // half of the samples
    auto spikes_at = [&](int tt, float out[LS]) -> uint32_t {
        if constexpr (SMOOTH) {
#pragma unroll
            for (int b = 0; b < LS; ++b) out[b] = 0.f;
            if (tt < 0 || !nt) return 0u;
            const float4 x = reinterpret_cast<const float4 *>(a.s_f)[(((size_t)tt * a.NC + q) * H + me) * 2 + half];
            out[0] = x.x; out[1] = x.y; out[2] = x.z; out[3] = x.w;
            return 0xffu;
        } else {
            (void)out;
            return (tt < 0 || !nt) ? 0u : a.s_bits[((size_t)tt * a.NC + q) * H + me];
        }
    };
    uint64_t hist = 0;      // spiking: byte d - 1 = the 8 samples' spikes at t - d
    float histf[MAXD][LS];  // smooth: histf[d - 1] = spikes at t - d
    for (int d = 1; d <= MAXD; ++d) {
        const uint32_t byte = spikes_at(t1 - 1 - d, histf[d - 1]);
        if constexpr (!SMOOTH) hist |= (uint64_t)byte << (8 * (d - 1));
    }
    // the surrogate derivatives and spikes of the next step down, loaded one step ahead
    auto g_at = [&](int tt) { return nt ? __ldcs(a.g_seg + ((size_t)(tt - t0) * B + bq) * H + me) : 0.f; };
    float gn = g_at(t1 - 1);
    auto y_at = [&](int tt) { return (FULL && nt) ? a.dU[((size_t)tt * B + bq) * H + me] : 0.f; };
    float yn = y_at(t1 - 1);
    float stn[LS];
    uint32_t sbn = spikes_at(t1 - 1, stn);
    // outgoing rows of neuron me, delay group d, at step u (q[u] in pnew): partial[u - d] += w q[u][post];
    // dw += s[u - d][me] q[u][post] (sbyte, sf: the spikes at u - d). Every thread of the CTA calls it.
    auto out_rows = [&](int u, int d, uint32_t sbyte, const float *sf) {
        float acc[LS];
#pragma unroll
        for (int b = 0; b < LS; ++b) acc[b] = 0.f;
        const int gs = nt ? grp[pl * (MAXD + 1) + d - 1] : 0, ge = nt ? grp[pl * (MAXD + 1) + d] : 0;
        if (__any_sync(FULL, sbyte != 0u))  // the same branch for the whole warp
            out_group<SMOOTH, true>(ocode, ow, pnew, dw, gs, ge, sub, half, sbyte != 0u, sbyte >> (LS * half), sf, acc);
        else
            out_group<SMOOTH, false>(ocode, ow, pnew, dw, gs, ge, sub, half, false, 0u, sf, acc);
        // the shares added pairwise, two samples fewer to carry each time: ends with the lane's sample 4 half + sub
        const float k0 = (sub & 1) ? acc[1] : acc[0], k1 = (sub & 1) ? acc[3] : acc[2];
        const float s0 = (sub & 1) ? acc[0] : acc[1], s1 = (sub & 1) ? acc[2] : acc[3];
        const float e0 = __fadd_rn(k0, __shfl_xor_sync(FULL, s0, 2)), e1 = __fadd_rn(k1, __shfl_xor_sync(FULL, s1, 2));
        const float x = __fadd_rn((sub & 2) ? e1 : e0, __shfl_xor_sync(FULL, (sub & 2) ? e0 : e1, 4));
        if (nt && u - d >= 0) {
            float *pp = part + ((size_t)((u - d) % RING) * HC + pl) * NS + LS * half + sub;
            *pp = __fadd_rn(*pp, x);
        }
    };
    // the readout adjoint o[t] does not depend on q: it is made one step ahead, into the other half of obuf, so
    // that no barrier is needed for it (the half of o[t - 1] was last read at step t + 1, three barriers back)
    if (ro) {
        o = __fadd_rn(t1 - 1 == tsv ? dmv : 0.f, __fmul_rn(a.beta, o));
        obuf[(size_t)((t1 - 1) & 1) * NS * R + rb * R + rr] = o;
    }
    if (!FULL) __syncthreads();  // o[t1 - 1] ready
    for (int t = t1 - 1; t >= t0; --t) {
        const float *ob = obuf + (size_t)(t & 1) * NS * R;  // o[t]
        float st[LS];
#pragma unroll
        for (int b = 0; b < LS; ++b) st[b] = stn[b];
        const uint32_t sbyte_t = sbn;
        const float gc = gn, yc = yn;
        if (t > t0) {
            gn = g_at(t - 1);
            yn = y_at(t - 1);
            sbn = spikes_at(t - 1, stn);
        }
        float *slot = a.qx + ((size_t)q * 2 + (t & 1)) * H * NS;
        uint32_t *flags = a.qflag + ((size_t)q * 2 + (t & 1)) * (H / 4);
        if (nt) {
            float *pp = part + ((size_t)(t % RING) * HC + pl) * NS + own;
            float sh = *pp;
            if constexpr (FULL) {
                sh = __fadd_rn(sh, yc);
            } else {
#pragma unroll 4
                for (int r = 0; r < R; ++r) sh = __fmaf_rn(__ldg(wout + pl * R + r), ob[own * R + r], sh);
            }
            *pp = 0.f;
            const float ap = __fmul_rn(a.alpha, qp);
            qp = __fmaf_rn(gc, __fmaf_rn(-a.theta, ap, sh), ap);
            slot[(size_t)me * NS + own] = qp;
        }
        __syncwarp();
        if (nt && (tid & 31) == 0)
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flags + me / 4), "r"((uint32_t)t + 1u) : "memory");
        // while the group's other values arrive: what nothing waits for
        if (nt) {
            __stcs(a.dU + ((size_t)t * B + bq) * H + me, qp);
            // dw_out: this neuron's spikes at t times o[t]; each of its NB threads takes an eighth of the readouts
            if (!FULL && sbyte_t) {
                if constexpr (SMOOTH) {
                    // a lane holds half of the samples' spikes: its half's sum to the readout, the halves in turn
                    for (int r = sub; r < R; r += LS) {
                        float acc = 0.f;
#pragma unroll
                        for (int b = 0; b < LS; ++b) acc = __fmaf_rn(st[b], ob[(LS * half + b) * R + r], acc);
                        acc = __fadd_rn(acc, __shfl_xor_sync(3u << (tid & 30), acc, 1));
                        if (half == 0) dwo[pl * R + r] = __fadd_rn(dwo[pl * R + r], acc);
                    }
                } else {
                    for (int r = own; r < R; r += NB) {
                        float acc = dwo[pl * R + r];
                        for (uint32_t m = sbyte_t; m; m &= m - 1) acc = __fadd_rn(acc, ob[(__ffs(m) - 1) * R + r]);
                        dwo[pl * R + r] = acc;
                    }
                }
            }
        }
        if (ro && t > t0) {  // o[t - 1]; o keeps o[t0] for the segment before this one
            o = __fadd_rn(t - 1 == tsv ? dmv : 0.f, __fmul_rn(a.beta, o));
            obuf[(size_t)((t - 1) & 1) * NS * R + rb * R + rr] = o;
        }
        // step t + 1's delay groups 2..5 (pnew still holds q[t + 1]; their partials are for steps t - 1 and earlier,
        // so only the delay-1 group waits for q[t])
        if (t + 1 < t1) {
#pragma unroll
            for (int d = 2; d <= MAXD; ++d)
                out_rows(t + 1, d, SMOOTH ? 0xffu : (uint32_t)((hist >> (8 * (d - 2))) & 0xffu), histf[d - 2]);
        }
        if (tid < H / 4 && !*(volatile int *)&aborted) {
            bool there = false;
            for (int it = 0; it < a.wait_polls && !there; ++it) {
                uint32_t v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flags + tid) : "memory");
                there = v == (uint32_t)t + 1u;
            }
            if (!there) {
                atomicAdd(a.err + 3, 1);
                *(volatile int *)&aborted = 1;
            }
        }
        __syncthreads();  // every CTA's q[t] written, every read of q[t + 1] done: q[t] (past L1) into pnew
        for (int j = tid; j < H * (NS / 4); j += nthr)
            reinterpret_cast<float4 *>(pnew)[j] = __ldcg(reinterpret_cast<const float4 *>(slot) + j);
        __syncthreads();
        out_rows(t, 1, SMOOTH ? 0xffu : (uint32_t)(hist & 0xffu), histf[0]);
        // the spike history of step t - 1: delays 1..5 reach t - 2 .. t - 6
        if constexpr (SMOOTH) {
            for (int d = 1; d <= MAXD; ++d) spikes_at(t - 1 - d, histf[d - 1]);
        } else {
            const uint32_t byte = spikes_at(t - 1 - MAXD, histf[0]);
            hist = (hist >> 8) | ((uint64_t)byte << (8 * (MAXD - 1)));
        }
    }
    // step t0's delay groups 2..5 (q[t0] is still in pnew)
#pragma unroll
    for (int d = 2; d <= MAXD; ++d)
        out_rows(t0, d, SMOOTH ? 0xffu : (uint32_t)((hist >> (8 * (d - 2))) & 0xffu), histf[d - 2]);
    // the state for the segment before this one
    __syncthreads();
    for (int k = tid; k < on; k += nthr) a.dwp[(size_t)q * a.nnz + obase + k] = dw[k];
    if constexpr (!FULL) {
        for (int k = tid; k < RING * HC * NS; k += nthr) part_st[k] = part[k];
        for (int k = tid; k < HC * R; k += nthr) a.dwo_p[((size_t)q * H + h0) * R + k] = dwo[k];
        if (nt) a.q_st[bq * H + me] = qp;
        if (ro && rank == 0) a.o_st[(size_t)(q * NS + rb) * R + rr] = o;
    }
}

// FULL, before the adjoint: the readout adjoint of every step, a thread per (sample, readout), last step first.
__global__ void __launch_bounds__(64) readout_adjoint_kernel(const __grid_constant__ Args a) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, n = a.B * a.R;
    if (k >= n) return;
    const float dm = a.dm[k];
    const int ts = a.tstar_in[k];
    float o = 0.f;
    for (int t = a.T - 1; t >= 0; --t) {
        o = __fadd_rn(t == ts ? dm : 0.f, __fmul_rn(a.beta, o));
        a.o_all[(size_t)t * n + k] = o;
    }
}

// FULL, before the adjoint: dU[t][b][i] = sum_r w_out[i][r] o[t][b][r], a thread per two neurons with their rows of w_out
// in registers (R4 groups of four readouts), DV_ROWS (t, b) rows per block. Bound by the write of dU.
constexpr int DV_ROWS = 32;
template <int R4>
__global__ void __launch_bounds__(256) readout_dV_kernel(const __grid_constant__ Args a) {
    __shared__ float4 o[DV_ROWS][R4];
    const int pairs = a.H / 2, i = blockIdx.y * blockDim.x + threadIdx.x, n = a.T * a.B;
    const int r0 = blockIdx.x * DV_ROWS, rows = min(DV_ROWS, n - r0);
    for (int k = threadIdx.x; k < DV_ROWS * R4 * 4; k += blockDim.x) {
        const int row = k / (R4 * 4), r = k % (R4 * 4);
        reinterpret_cast<float *>(o)[k] = (row < rows && r < a.R) ? a.o_all[(size_t)(r0 + row) * a.R + r] : 0.f;
    }
    float w[2][R4 * 4];
#pragma unroll
    for (int r = 0; r < R4 * 4; ++r) {
        const bool in = i < pairs && r < a.R;
        w[0][r] = in ? a.w_out[(size_t)(2 * i) * a.R + r] : 0.f;
        w[1][r] = in ? a.w_out[(size_t)(2 * i + 1) * a.R + r] : 0.f;
    }
    __syncthreads();
    if (i >= pairs) return;
    const bool wide = (reinterpret_cast<uintptr_t>(a.dU) & 7) == 0;  // the caller's buffer (H is even: so every row)
    for (int k = 0; k < rows; ++k) {
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int r = 0; r < R4; ++r) {
            const float4 v = o[k][r];
            s0 = __fmaf_rn(w[0][4 * r], v.x, s0);
            s1 = __fmaf_rn(w[1][4 * r], v.x, s1);
            s0 = __fmaf_rn(w[0][4 * r + 1], v.y, s0);
            s1 = __fmaf_rn(w[1][4 * r + 1], v.y, s1);
            s0 = __fmaf_rn(w[0][4 * r + 2], v.z, s0);
            s1 = __fmaf_rn(w[1][4 * r + 2], v.z, s1);
            s0 = __fmaf_rn(w[0][4 * r + 3], v.w, s0);
            s1 = __fmaf_rn(w[1][4 * r + 3], v.w, s1);
        }
        float *at = a.dU + (size_t)(r0 + k) * a.H + 2 * i;
        if (wide) {
            __stcs(reinterpret_cast<float2 *>(at), make_float2(s0, s1));
        } else {
            __stcs(at, s0);
            __stcs(at + 1, s1);
        }
    }
}

// FULL: dw_out's partial sums, chunk c of NC of the (step, group) pairs: dwo_p[c][i][r] = sum over the chunk's spikes of
// neuron i of o[t][b][r]. A warp per four neurons (one word of spikes per step and group), a lane per readout. T pairs to
// a chunk: chunks of whole steps left all but T of the NC of them empty in short sequences of large batches.
__global__ void __launch_bounds__(256) dwo_kernel(const __grid_constant__ Args a) {
    const int lane = threadIdx.x & 31, word = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, c = blockIdx.y;
    if (word >= a.H / 4) return;
    const size_t p0 = (size_t)c * a.T;  // the chunk's first pair
    const uint32_t *src = reinterpret_cast<const uint32_t *>(a.s_bits) + word;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k0 = 0; k0 < a.T; k0 += 32) {
        // 32 pairs' words, a lane each; then those with a spike, in order
        const uint32_t mine = k0 + lane < a.T ? src[(p0 + k0 + lane) * (a.H / 4)] : 0u;
        for (uint32_t some = __ballot_sync(FULL, mine != 0u); some; some &= some - 1) {
            const int k = k0 + __ffs(some) - 1;
            const uint32_t w = __shfl_sync(FULL, mine, k - k0);
            const float *o = a.o_all + (p0 + k) * NS * a.R + lane;  // (t, q): samples 8q ..
            for (uint32_t m = w; m; m &= m - 1) {
                const int bit = __ffs(m) - 1;
                const float v = lane < a.R ? __ldg(o + (bit & 7) * a.R) : 0.f;
                if (bit < 8) acc[0] = __fadd_rn(acc[0], v);
                else if (bit < 16) acc[1] = __fadd_rn(acc[1], v);
                else if (bit < 24) acc[2] = __fadd_rn(acc[2], v);
                else acc[3] = __fadd_rn(acc[3], v);
            }
        }
    }
    if (lane < a.R)
#pragma unroll
        for (int j = 0; j < 4; ++j) a.dwo_p[((size_t)c * a.H + 4 * word + j) * a.R + lane] = acc[j];
}

// dw_rec in the caller's (incoming, canonical) order: the clusters' partials added in cluster order.
__global__ void reduce_dw_kernel(const float *dwp, const int32_t *perm, int nnz, int NC, float *dw) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nnz) return;
    float s = 0.f;
    for (int c = 0; c < NC; ++c) s = __fadd_rn(s, dwp[(size_t)c * nnz + l]);
    dw[perm[l]] = s;
}

__global__ void reduce_dwo_kernel(const float *dwo_p, int n, int NC, float *dwo) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    float s = 0.f;
    for (int c = 0; c < NC; ++c) s = __fadd_rn(s, dwo_p[(size_t)c * n + k]);
    dwo[k] = s;
}

__global__ void gather_kernel(const float *src, const int32_t *perm, int n, float *dst) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l < n) dst[l] = src[perm[l]];
}

// ------------------------------------------------------------------------------------------------ input projection

// U[r] = sum over the spiking channels c of input row r (ascending) of w_in[c]: H / 4 threads per row, one float4
// of hidden units each, blockDim / (H / 4) rows per block; the channel indices of a row four at a time, then their
// weight rows. An index outside [0, C) adds nothing (the event lists are checked when they are built).
__global__ void __launch_bounds__(256) project_fwd_kernel(const int32_t *row_ptr, const int32_t *ch, int rows,
                                                          int C, int H, const float *w, float *u) {
    const int h4 = H / 4;
    const int r = blockIdx.x * (blockDim.x / h4) + threadIdx.x / h4, c4 = threadIdx.x % h4;
    if (r >= rows) return;
    const int k0 = row_ptr[r], k1 = row_ptr[r + 1];
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = k0; k < k1; k += 4) {
        int c[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = k + j < k1 ? __ldg(ch + k + j) : -1;
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            v[j] = (c[j] >= 0 && c[j] < C) ? __ldg(reinterpret_cast<const float4 *>(w + (size_t)c[j] * H) + c4)
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (c[j] < 0 || c[j] >= C) continue;
            acc.x = __fadd_rn(acc.x, v[j].x);
            acc.y = __fadd_rn(acc.y, v[j].y);
            acc.z = __fadd_rn(acc.z, v[j].z);
            acc.w = __fadd_rn(acc.w, v[j].w);
        }
    }
    reinterpret_cast<float4 *>(u + (size_t)r * H)[c4] = acc;
}

// dw_in, first pass: chunk k (rows row_idx[chunk_ptr[k] .. chunk_ptr[k + 1]) of one channel, ascending) summed
// into partials[k]; a block per chunk, H / 4 threads, four rows' loads in flight. A row outside [0, rows) adds
// nothing.
__global__ void __launch_bounds__(256) project_bwd_chunk_kernel(const int32_t *chunk_ptr, const int32_t *row_idx,
                                                                int rows, int H, const float *du, float *partials) {
    const int k = blockIdx.x, c4 = threadIdx.x;
    const int j0 = chunk_ptr[k], j1 = chunk_ptr[k + 1];
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = j0; j < j1; j += 4) {
        int r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) r[i] = j + i < j1 ? __ldg(row_idx + j + i) : -1;
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            v[i] = (r[i] >= 0 && r[i] < rows) ? __ldcs(reinterpret_cast<const float4 *>(du + (size_t)r[i] * H) + c4)
                                              : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (r[i] < 0 || r[i] >= rows) continue;
            acc.x = __fadd_rn(acc.x, v[i].x);
            acc.y = __fadd_rn(acc.y, v[i].y);
            acc.z = __fadd_rn(acc.z, v[i].z);
            acc.w = __fadd_rn(acc.w, v[i].w);
        }
    }
    reinterpret_cast<float4 *>(partials + (size_t)k * H)[c4] = acc;
}

// dw_in, second pass: channel c's chunks (ch_chunk[c] .. ch_chunk[c + 1]) added in chunk order.
__global__ void project_bwd_reduce_kernel(const int32_t *ch_chunk, int C, int H, const float *partials, float *dw) {
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)C * H) return;
    const int c = (int)(e / H), h = (int)(e % H);
    float s = 0.f;
    for (int k = ch_chunk[c]; k < ch_chunk[c + 1]; ++k) s = __fadd_rn(s, partials[(size_t)k * H + h]);
    dw[e] = s;
}

}  // namespace n2b_bptt

// ------------------------------------------------------------------------------------------------ host

namespace n2b_host {
int set_error(int code, const std::string &msg);
}

namespace {

using namespace n2b_bptt;

int bfail(int code, const std::string &msg) { return n2b_host::set_error(code, msg); }
int bcuda(cudaError_t e, const char *what) {
    return n2b_host::set_error(N2B_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
}
#define B_CUDA(call)                                    \
    do {                                                \
        cudaError_t _e = (call);                        \
        if (_e != cudaSuccess) return bcuda(_e, #call); \
    } while (0)

// A taped forward keeps the surrogate derivatives of every step when they take at most this much (the workload's
// 128 x 500 x 1024 are 262 MB): 0.04 ms of writes under the forward instead of 0.18 ms of recomputing per segment of
// 50 steps, of which the adjoint hides half. Larger layers, and those asked for it (desc.segments: their tape would leave
// the program too little memory), keep the membrane every `checkpoint` steps and recompute.
constexpr size_t FULL_TAPE_BYTES = (size_t)4 << 30;

struct WsLayout {
    size_t spikes, xw, tot, vck, gseg, outw, dwp, dwo, part, qst, ost, qx, qflag, err, total;
};

size_t a256(size_t x) { return (x + 255) & ~size_t(255); }

int check_desc(const n2b_bptt_desc *d) {
    if (!d) return bfail(N2B_EINVAL, "desc is NULL");
    if (d->batch <= 0 || d->batch % NS) return bfail(N2B_EINVAL, "batch must be a positive multiple of 8");
    if (d->hidden <= 0 || d->hidden % 32 || d->hidden > 1024)
        return bfail(N2B_EINVAL, "hidden must be a multiple of 32, at most 1024");
    if (d->readouts <= 0 || d->readouts > 32) return bfail(N2B_EINVAL, "readouts must be in 1..32");
    if (d->steps <= 0 || d->checkpoint <= 0) return bfail(N2B_EINVAL, "steps and checkpoint must be positive");
    if ((int64_t)d->steps * (d->batch / NS) * d->hidden >= ((int64_t)1 << 31))
        return bfail(N2B_EINVAL, "steps x batch / 8 x hidden must stay below 2^31");
    if (d->smooth && d->hidden > 256) return bfail(N2B_EINVAL, "the smooth model is for hidden <= 256");
    if (d->nnz < 0 || (d->nnz > 0 && (!d->in_code || !d->out_code || !d->out_perm)))
        return bfail(N2B_EINVAL, "missing link arrays");
    if (!d->in_ptr || !d->out_grp) return bfail(N2B_EINVAL, "missing row arrays");
    if (d->in_cta_max < 0 || d->out_cta_max < 0) return bfail(N2B_EINVAL, "negative link counts");
    if (d->wait_polls < 0) return bfail(N2B_EINVAL, "wait_polls < 0");
    return N2B_OK;
}

// A spiking layer whose incoming rows fit a CTA's shared memory.
bool rows_fit(const n2b_bptt_desc *d) {
    return !d->smooth && scan_smem(d->hidden, d->hidden / CL, d->in_cta_max).total <= SMEM_MAX - 1024;
}

// The forward runs fwd_group_kernel, else fwd_kernel (the same results). Its launches and set-up cost 13 us more, and its
// CTAs lose against fwd_kernel's clusters where several of them share an SM. Measured, fwd_kernel over it, plain forwards
// at 5% / 10% of the neurons spiking a step:
//   steps: 5 0.3-0.7, 12 0.7-1.2, 16 0.9-1.3 / 0.7-1.15, 24 1.04-1.55 / 1.0-1.36, 50 1.2-1.9, 300 1.3-2.1;
//   a CTA per SM (18 groups of 8 samples) 1.04-2.1 at 1,024 neurons, 19 groups 0.89-1.09 / 0.80-0.96; at 512 neurons 16
//   groups 1.33-1.88, 19 groups 1.02-1.26 / 0.98-1.16, 64 groups 0.66-0.75; at 256 neurons 32 groups 1.06-1.34 / 1.01-1.28,
//   64 groups 0.78-1.01; at 64 neurons 64 groups 1.04-1.33.
constexpr int SMS = 148, GROUP_STEPS = 24, GROUP_THREADS = 512;  // (threads of its CTAs per SM, where there are several)
bool scans(const n2b_bptt_desc *d) {
    const int64_t ctas = (int64_t)(d->batch / NS) * CL;
    return rows_fit(d) && d->steps >= GROUP_STEPS && (ctas <= SMS || ctas * d->hidden <= (int64_t)GROUP_THREADS * SMS);
}

bool full_tape(const n2b_bptt_desc *d) {
    return !d->segments && rows_fit(d) && sizeof(float) * (size_t)d->steps * d->batch * d->hidden <= FULL_TAPE_BYTES;
}

WsLayout ws_layout(const n2b_bptt_desc *d) {
    WsLayout L{};
    const size_t T = d->steps, B = d->batch, H = d->hidden, R = d->readouts, NC = B / NS;
    const size_t nseg = (T + d->checkpoint - 1) / d->checkpoint, K = std::min<size_t>(d->checkpoint, T);
    size_t o = 0;
    L.spikes = o; o = a256(o + (d->smooth ? sizeof(float) * T * NC * H * NS : T * NC * H));
    L.xw = o; o = a256(o + (scans(d) ? sizeof(unsigned long long) * NC * XSLOTS * (H / 4) : 0));
    L.tot = o; o = a256(o + (scans(d) || full_tape(d) ? sizeof(float) * T * B * R : 0));
    L.vck = o; o = a256(o + (full_tape(d) ? 0 : sizeof(float) * nseg * B * H));
    // every step, or two segments: one recomputed, one run back
    L.gseg = o; o = a256(o + sizeof(float) * (full_tape(d) ? T : 2 * K) * B * H);
    L.outw = o; o = a256(o + sizeof(float) * std::max<size_t>(d->nnz, 1));
    L.dwp = o; o = a256(o + sizeof(float) * NC * std::max<size_t>(d->nnz, 1));
    L.dwo = o; o = a256(o + sizeof(float) * NC * H * R);
    L.part = o; o = a256(o + sizeof(float) * NC * CL * RING * (H / CL) * NS);
    L.qst = o; o = a256(o + sizeof(float) * B * H);
    L.ost = o; o = a256(o + sizeof(float) * B * R);
    L.qx = o; o = a256(o + sizeof(float) * NC * 2 * H * NS);
    L.qflag = o; o = a256(o + sizeof(uint32_t) * NC * 2 * (H / 4));
    L.err = o; o = a256(o + sizeof(int32_t) * N2B_BPTT_ERR_WORDS);
    L.total = o;
    return L;
}

// n2b_bptt_infer's scratch: what fwd_group_kernel and the readout's kernels hand on.
struct PlainLayout {
    size_t spikes, xw, tot, total;
};
PlainLayout plain_layout(const n2b_bptt_desc *d) {
    PlainLayout L{};
    if (!scans(d)) return L;  // fwd_kernel keeps nothing in memory
    const size_t T = d->steps, B = d->batch, H = d->hidden, NC = B / NS;
    size_t o = 0;
    L.spikes = o; o = a256(o + T * NC * H);
    L.xw = o; o = a256(o + sizeof(unsigned long long) * NC * XSLOTS * (H / 4));
    L.tot = o; o = a256(o + sizeof(float) * T * B * d->readouts);
    L.total = o;
    return L;
}

int threads_of(const n2b_bptt_desc *d, int per_neuron) {
    const int n = std::max(per_neuron * (d->hidden / CL), NS * d->readouts);
    return (n + 31) / 32 * 32;
}

Args sizes_of(const n2b_bptt_desc *d) {
    Args a{};
    a.B = d->batch;
    a.T = d->steps;
    a.H = d->hidden;
    a.R = d->readouts;
    a.K = d->checkpoint;
    a.HC = d->hidden / CL;
    a.NC = d->batch / NS;
    a.nseg = (d->steps + d->checkpoint - 1) / d->checkpoint;
    a.nnz = d->nnz;
    a.alpha = d->alpha;
    a.beta = d->beta;
    a.theta = d->theta;
    a.slope = d->slope;
    a.in_ptr = d->in_ptr;
    a.in_code = d->in_code;
    a.out_grp = d->out_grp;
    a.out_code = d->out_code;
    a.wait_polls = d->wait_polls > 0 ? d->wait_polls : XCHG_SPIN_LIMIT;
    return a;
}

Args args_of(const n2b_bptt_desc *d, char *ws, const WsLayout &L) {
    Args a = sizes_of(d);
    a.s_bits = reinterpret_cast<uint8_t *>(ws + L.spikes);
    a.s_f = reinterpret_cast<float *>(ws + L.spikes);
    a.xw = reinterpret_cast<unsigned long long *>(ws + L.xw);
    a.tot = reinterpret_cast<float *>(ws + L.tot);
    a.v_ckpt = reinterpret_cast<float *>(ws + L.vck);
    a.g_seg = reinterpret_cast<float *>(ws + L.gseg);
    a.g_all = full_tape(d) ? a.g_seg : nullptr;
    a.out_w = reinterpret_cast<float *>(ws + L.outw);
    a.dwp = reinterpret_cast<float *>(ws + L.dwp);
    a.dwo_p = reinterpret_cast<float *>(ws + L.dwo);
    a.part_st = reinterpret_cast<float *>(ws + L.part);
    a.q_st = reinterpret_cast<float *>(ws + L.qst);
    a.o_st = reinterpret_cast<float *>(ws + L.ost);
    a.qx = reinterpret_cast<float *>(ws + L.qx);
    a.qflag = reinterpret_cast<uint32_t *>(ws + L.qflag);
    a.o_all = a.tot;
    a.err = reinterpret_cast<int32_t *>(ws + L.err);
    return a;
}

int check_ws(const n2b_bptt_desc *d, void *ws, size_t bytes, WsLayout &L) {
    int rc = check_desc(d);
    if (rc) return rc;
    L = ws_layout(d);
    if (!ws || (reinterpret_cast<uintptr_t>(ws) & 255)) return bfail(N2B_EINVAL, "workspace must be 256-byte aligned");
    if (bytes < L.total) return bfail(N2B_ESPACE, "workspace too small: need " + std::to_string(L.total) + " bytes");
    return N2B_OK;
}

template <class Kern, class... Rest>
int launch_cluster(Kern kern, int grid, int threads, size_t smem, cudaStream_t s, const Args &a, Rest... rest) {
    if (smem > 227 * 1024) return bfail(N2B_EINVAL, "shared memory need " + std::to_string(smem) + " bytes > 227 KiB");
    B_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    B_CUDA(cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg));
    if (clusters < 1) return bfail(N2B_ECUDA, "a cluster of 8 CTAs of this size cannot be resident");
    B_CUDA(cudaLaunchKernelEx(&cfg, kern, a, rest...));
    return N2B_OK;
}

// The groups of 8 CTAs that one cooperative launch of `kern` can hold (all resident at once).
template <class Kern>
int coop_groups(Kern kern, int threads, size_t smem, int &groups) {
    if (smem > 227 * 1024) return bfail(N2B_EINVAL, "shared memory need " + std::to_string(smem) + " bytes > 227 KiB");
    B_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int dev = 0, sms = 0, per_sm = 0;
    B_CUDA(cudaGetDevice(&dev));
    B_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    B_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
    groups = per_sm * sms / CL;
    if (groups < 1) return bfail(N2B_ECUDA, "a group of 8 CTAs of this size cannot be resident");
    return N2B_OK;
}

// The backward's two internal streams on a device, made on first use and kept: the adjoint on the highest
// priority, the next segment's recompute on the lowest, so that when both are ready the adjoint's CTAs are placed
// first and the recompute fills the SMs the adjoint leaves free.
struct SideStreams {
    cudaStream_t hi = nullptr, lo = nullptr;
};
int side_streams(SideStreams &out) {
    static std::mutex mu;
    static SideStreams per_dev[64];
    int dev = 0;
    B_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return bfail(N2B_EINVAL, "device index above 63");
    std::lock_guard<std::mutex> lock(mu);
    SideStreams &st = per_dev[dev];
    if (!st.hi) {
        int least = 0, greatest = 0;
        B_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
        B_CUDA(cudaStreamCreateWithPriority(&st.hi, cudaStreamNonBlocking, greatest));
        B_CUDA(cudaStreamCreateWithPriority(&st.lo, cudaStreamNonBlocking, least));
    }
    out = st;
    return N2B_OK;
}

// Events of one backward call, destroyed on every return (pending work keeps them alive as long as it needs).
struct CallEvents {
    cudaEvent_t e[6] = {};
    ~CallEvents() {
        for (cudaEvent_t x : e)
            if (x) cudaEventDestroy(x);
    }
};

template <class Kern, class... Rest>
int launch_coop(Kern kern, int grid, int threads, size_t smem, cudaStream_t s, const Args &a, Rest... rest) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    B_CUDA(cudaLaunchKernelEx(&cfg, kern, a, rest...));
    return N2B_OK;
}

// The forward's launches. `group`: fwd_group_kernel and the readout's kernels, over a's spikes, words and readout sums;
// else fwd_kernel, which without a tape writes m, tstar and the error words alone.
int run_forward(const n2b_bptt_desc *d, Args a, bool group, cudaStream_t s) {
    B_CUDA(cudaMemsetAsync(a.err, 0, sizeof(int32_t) * N2B_BPTT_ERR_WORDS, s));
    if (group) {
        const int NC = d->batch / NS, gthreads = (NB * (d->hidden / CL) + 31) / 32 * 32;
        const size_t smem = scan_smem(d->hidden, d->hidden / CL, d->in_cta_max).total;
        int per_launch = 0;  // groups per cooperative launch
        int rc = coop_groups(fwd_group_kernel, gthreads, smem, per_launch);
        if (rc) return rc;
        B_CUDA(cudaMemsetAsync(a.xw, 0, sizeof(unsigned long long) * NC * XSLOTS * (d->hidden / 4), s));
        for (int g0 = 0; g0 < NC; g0 += per_launch) {
            rc = launch_coop(fwd_group_kernel, std::min(per_launch, NC - g0) * CL, gthreads, smem, s, a, d->in_cta_max,
                             g0);
            if (rc) return rc;
        }
        readout_kernel<<<(unsigned)(d->steps * NC), READOUT_THREADS, 0, s>>>(a);  // (below 2^26: check_desc)
        B_CUDA(cudaGetLastError());
        readout_max_kernel<<<(unsigned)((d->batch * d->readouts + 31) / 32), 32, 0, s>>>(a);
        B_CUDA(cudaGetLastError());
        return N2B_OK;
    }
    const bool smooth = d->smooth != 0;
    const int grid = (d->batch / NS) * CL, threads = threads_of(d, NT);
    FwdSmem S = fwd_smem(d->hidden, d->hidden / CL, d->readouts, smooth, true, d->in_cta_max);
    a.csr_smem = S.total <= 200 * 1024;
    if (!a.csr_smem) S = fwd_smem(d->hidden, d->hidden / CL, d->readouts, smooth, false, 0);
    return smooth              ? launch_cluster(fwd_kernel<true, false>, grid, threads, S.total, s, a, d->in_cta_max)
           : a.tape && a.g_all ? launch_cluster(fwd_kernel<false, true>, grid, threads, S.total, s, a, d->in_cta_max)
                               : launch_cluster(fwd_kernel<false, false>, grid, threads, S.total, s, a, d->in_cta_max);
}

}  // namespace

extern "C" {

int n2b_bptt_workspace_bytes(const n2b_bptt_desc *d, size_t *bytes) {
    if (!bytes) return bfail(N2B_EINVAL, "bytes is NULL");
    int rc = check_desc(d);
    if (rc) return rc;
    *bytes = ws_layout(d).total;
    return N2B_OK;
}

int n2b_bptt_forward(const n2b_bptt_desc *d, const float *u, const float *w_rec, const float *w_out, int32_t tape,
                     float *m, int32_t *tstar, void *workspace, size_t workspace_bytes, void *stream) {
    WsLayout L;
    int rc = check_ws(d, workspace, workspace_bytes, L);
    if (rc) return rc;
    if (!u || !w_out || !m || !tstar || (d->nnz > 0 && !w_rec)) return bfail(N2B_EINVAL, "missing arguments");
    Args a = args_of(d, static_cast<char *>(workspace), L);
    a.tape = tape != 0;
    a.U = u;
    a.in_w = w_rec;
    a.w_out = w_out;
    a.m = m;
    a.tstar = tstar;
    // without a tape nothing of the workspace but the error words is written (calls and a backward may overlap)
    return run_forward(d, a, tape && scans(d), reinterpret_cast<cudaStream_t>(stream));
}

int n2b_bptt_infer_bytes(const n2b_bptt_desc *d, size_t *bytes) {
    if (!bytes) return bfail(N2B_EINVAL, "bytes is NULL");
    int rc = check_desc(d);
    if (rc) return rc;
    *bytes = plain_layout(d).total;
    return N2B_OK;
}

int n2b_bptt_infer(const n2b_bptt_desc *d, const float *u, const float *w_rec, const float *w_out, float *m,
                   int32_t *tstar, int32_t *err, void *scratch, size_t scratch_bytes, void *stream) {
    int rc = check_desc(d);
    if (rc) return rc;
    if (!u || !w_out || !m || !tstar || !err || (d->nnz > 0 && !w_rec)) return bfail(N2B_EINVAL, "missing arguments");
    const PlainLayout L = plain_layout(d);
    if (L.total > 0 && (!scratch || (reinterpret_cast<uintptr_t>(scratch) & 255)))
        return bfail(N2B_EINVAL, "scratch must be 256-byte aligned");
    if (scratch_bytes < L.total) return bfail(N2B_ESPACE, "scratch too small: need " + std::to_string(L.total) + " bytes");
    char *at = static_cast<char *>(scratch);
    Args a = sizes_of(d);
    a.U = u;
    a.in_w = w_rec;
    a.w_out = w_out;
    a.m = m;
    a.tstar = tstar;
    a.err = err;
    if (L.total > 0) {
        a.s_bits = reinterpret_cast<uint8_t *>(at + L.spikes);
        a.xw = reinterpret_cast<unsigned long long *>(at + L.xw);
        a.tot = reinterpret_cast<float *>(at + L.tot);
    }
    return run_forward(d, a, scans(d), reinterpret_cast<cudaStream_t>(stream));
}

int n2b_bptt_backward(const n2b_bptt_desc *d, const float *u, const float *w_rec, const float *w_out,
                      const float *dm, const int32_t *tstar, float *du, float *dw_rec, float *dw_out,
                      void *workspace, size_t workspace_bytes, void *stream) {
    WsLayout L;
    int rc = check_ws(d, workspace, workspace_bytes, L);
    if (rc) return rc;
    if (!u || !w_out || !dm || !tstar || !du || !dw_out || (d->nnz > 0 && (!w_rec || !dw_rec)))
        return bfail(N2B_EINVAL, "missing arguments");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    char *ws = static_cast<char *>(workspace);
    Args a = args_of(d, ws, L);
    a.U = u;
    a.in_w = w_rec;
    a.w_out = w_out;
    a.dm = dm;
    a.tstar_in = tstar;
    a.dU = du;
    if (d->nnz > 0) {  // the weights in outgoing order
        gather_kernel<<<(d->nnz + 255) / 256, 256, 0, s>>>(w_rec, d->out_perm, d->nnz,
                                                           reinterpret_cast<float *>(ws + L.outw));
        B_CUDA(cudaGetLastError());
    }
    const bool smooth = d->smooth != 0;
    const int NC = d->batch / NS, threads = threads_of(d, NB);
    const bool full = full_tape(d);  // the adjoint of all steps in one launch, nothing to recompute
    BwdSmem S = bwd_smem(d->hidden, d->hidden / CL, d->readouts, d->out_cta_max, full);
    // Other kernels run beside the adjoint (dw_out's, the next segment's recomputation). Where several of its CTAs fit an
    // SM it would be placed around theirs, two and more to one SM and none to the next, at the pace of the fullest: it
    // asks for so much shared memory that an SM holds just its share. 50 steps of 128 samples: 256 neurons 403 -> 285 us,
    // 512 neurons 505 -> 375.
    const int share = (NC * CL + SMS - 1) / SMS;
    const bool spread = full && d->hidden <= 512 && share <= 3;
    if (spread) S.total = std::max(S.total, SMEM_MAX / (share + 1) + 2048);
    const int K = full ? d->steps : d->checkpoint, nseg = full ? 1 : a.nseg;
    const int rthreads = d->hidden % 64 == 0 ? 256 : 128;  // whole neurons of NT threads; hidden % 32 == 0
    const size_t rsmem = smooth ? 0 : (size_t)16 * d->hidden;  // the staged spike rows
    int per_launch = 0;  // groups per cooperative launch
    rc = smooth ? coop_groups(bwd_kernel<true, false>, threads, S.total, per_launch)
         : full ? coop_groups(bwd_kernel<false, true>, threads, S.total, per_launch)
                : coop_groups(bwd_kernel<false, false>, threads, S.total, per_launch);
    if (rc) return rc;
    SideStreams st;
    rc = side_streams(st);
    if (rc) return rc;
    CallEvents ev;  // fork, recomputed[2], adjoint done[2], join
    for (cudaEvent_t &x : ev.e) B_CUDA(cudaEventCreateWithFlags(&x, cudaEventDisableTiming));
    cudaEvent_t fork = ev.e[0], join = ev.e[5], *rec = ev.e + 1, *adj = ev.e + 3;
    B_CUDA(cudaEventRecord(fork, s));
    B_CUDA(cudaStreamWaitEvent(st.hi, fork, 0));
    B_CUDA(cudaStreamWaitEvent(st.lo, fork, 0));
    float *gbuf[2] = {a.g_seg, full ? a.g_seg : a.g_seg + (size_t)std::min(K, d->steps) * d->batch * d->hidden};
    // segment seg recomputed from its checkpoint into gbuf[seg & 1] on the low-priority stream
    auto recompute = [&](int seg) -> int {
        const int t0 = seg * K, t1 = std::min(d->steps, t0 + K);
        Args ra = a;
        ra.g_seg = gbuf[seg & 1];
        const dim3 rgrid((unsigned)(d->hidden / (rthreads / NT)), (unsigned)NC, (unsigned)((t1 - t0 + TC - 1) / TC));
        const unsigned vblocks = (unsigned)((d->batch * d->hidden + 255) / 256);
        if (smooth) {
            recompute_r_kernel<true><<<rgrid, rthreads, 0, st.lo>>>(ra, t0, t1);
            recompute_v_kernel<true><<<vblocks, 256, 0, st.lo>>>(ra, seg, t0, t1);
        } else {
            recompute_r_kernel<false><<<rgrid, rthreads, rsmem, st.lo>>>(ra, t0, t1);
            recompute_v_kernel<false><<<vblocks, 256, 0, st.lo>>>(ra, seg, t0, t1);
        }
        B_CUDA(cudaGetLastError());
        B_CUDA(cudaEventRecord(rec[seg & 1], st.lo));
        return N2B_OK;
    };
    // Segments run backwards. The recompute of segment seg - 1 overlaps the adjoint of seg; it reuses the buffer
    // of seg + 1, so it waits for that adjoint.
    B_CUDA(cudaMemsetAsync(a.qflag, 0, sizeof(uint32_t) * NC * 2 * (d->hidden / 4), st.hi));
    if (full) {  // what does not depend on q: the readout's part of dU on this stream, dw_out beside the adjoint
        readout_adjoint_kernel<<<(unsigned)((d->batch * d->readouts + 63) / 64), 64, 0, st.hi>>>(a);
        B_CUDA(cudaGetLastError());
        B_CUDA(cudaEventRecord(rec[0], st.hi));
        B_CUDA(cudaStreamWaitEvent(st.lo, rec[0], 0));
        // (with the adjoint's partition of shared memory and L1: an SM that runs it takes the adjoint's CTA at once)
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)((d->hidden / 4 + 7) / 8), (unsigned)NC);
        cfg.blockDim = dim3(256);
        cfg.stream = st.lo;
        cudaLaunchAttribute carveout[1];
        carveout[0].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        carveout[0].val.sharedMemCarveout = 100;
        cfg.attrs = carveout;
        cfg.numAttrs = spread ? 1 : 0;
        B_CUDA(cudaLaunchKernelEx(&cfg, dwo_kernel, a));
        B_CUDA(cudaEventRecord(rec[1], st.lo));
        const int vthreads = std::min(256, d->hidden / 2);
        const dim3 vgrid((unsigned)(((int64_t)d->steps * d->batch + DV_ROWS - 1) / DV_ROWS),
                         (unsigned)((d->hidden / 2 + vthreads - 1) / vthreads));
        switch ((d->readouts + 3) / 4) {
            case 1: readout_dV_kernel<1><<<vgrid, vthreads, 0, st.hi>>>(a); break;
            case 2: readout_dV_kernel<2><<<vgrid, vthreads, 0, st.hi>>>(a); break;
            case 3: readout_dV_kernel<3><<<vgrid, vthreads, 0, st.hi>>>(a); break;
            case 4: readout_dV_kernel<4><<<vgrid, vthreads, 0, st.hi>>>(a); break;
            case 5: readout_dV_kernel<5><<<vgrid, vthreads, 0, st.hi>>>(a); break;
            case 6: readout_dV_kernel<6><<<vgrid, vthreads, 0, st.hi>>>(a); break;
            case 7: readout_dV_kernel<7><<<vgrid, vthreads, 0, st.hi>>>(a); break;
            default: readout_dV_kernel<8><<<vgrid, vthreads, 0, st.hi>>>(a); break;
        }
        B_CUDA(cudaGetLastError());
    } else {
        rc = recompute(nseg - 1);
    }
    if (rc) return rc;
    for (int seg = nseg - 1; seg >= 0; --seg) {
        const int t0 = seg * K, t1 = std::min(d->steps, t0 + K);
        const int first = seg == nseg - 1;
        Args ba = a;
        ba.g_seg = gbuf[seg & 1];
        if (!full) B_CUDA(cudaStreamWaitEvent(st.hi, rec[seg & 1], 0));
        for (int g0 = 0; g0 < NC; g0 += per_launch) {
            const int grid = std::min(per_launch, NC - g0) * CL;
            rc = smooth ? launch_coop(bwd_kernel<true, false>, grid, threads, S.total, st.hi, ba, d->out_cta_max, t0,
                                      t1, first, g0)
                 : full ? launch_coop(bwd_kernel<false, true>, grid, threads, S.total, st.hi, ba, d->out_cta_max, t0, t1,
                                      first, g0)
                        : launch_coop(bwd_kernel<false, false>, grid, threads, S.total, st.hi, ba, d->out_cta_max, t0,
                                      t1, first, g0);
            if (rc) return rc;
        }
        B_CUDA(cudaEventRecord(adj[seg & 1], st.hi));
        if (seg > 0) {
            if (seg + 1 < nseg) B_CUDA(cudaStreamWaitEvent(st.lo, adj[(seg + 1) & 1], 0));
            rc = recompute(seg - 1);
            if (rc) return rc;
        }
    }
    if (d->nnz > 0) {
        reduce_dw_kernel<<<(d->nnz + 255) / 256, 256, 0, st.hi>>>(a.dwp, d->out_perm, d->nnz, NC, dw_rec);
        B_CUDA(cudaGetLastError());
    }
    const int n = d->hidden * d->readouts;
    if (full) B_CUDA(cudaStreamWaitEvent(st.hi, rec[1], 0));
    reduce_dwo_kernel<<<(n + 255) / 256, 256, 0, st.hi>>>(a.dwo_p, n, NC, dw_out);
    B_CUDA(cudaGetLastError());
    B_CUDA(cudaEventRecord(join, st.hi));
    B_CUDA(cudaStreamWaitEvent(s, join, 0));
    return N2B_OK;
}

int n2b_bptt_status(const n2b_bptt_desc *d, void *workspace, size_t workspace_bytes, int32_t *words, void *stream) {
    WsLayout L;
    int rc = check_ws(d, workspace, workspace_bytes, L);
    if (rc) return rc;
    if (!words) return bfail(N2B_EINVAL, "words is NULL");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    int32_t host[N2B_BPTT_ERR_WORDS];
    B_CUDA(cudaMemcpyAsync(host, static_cast<char *>(workspace) + L.err, sizeof(host), cudaMemcpyDeviceToHost, s));
    B_CUDA(cudaStreamSynchronize(s));
    for (int k = 0; k < N2B_BPTT_ERR_WORDS; ++k) words[k] = host[k];
    return N2B_OK;
}

int n2b_bptt_spikes(const n2b_bptt_desc *d, void *workspace, size_t workspace_bytes, void *out, void *stream) {
    WsLayout L;
    int rc = check_ws(d, workspace, workspace_bytes, L);
    if (rc) return rc;
    if (!out) return bfail(N2B_EINVAL, "out is NULL");
    const size_t T = d->steps, NC = d->batch / NS, H = d->hidden;
    const size_t n = d->smooth ? sizeof(float) * T * NC * H * NS : T * NC * H;
    B_CUDA(cudaMemcpyAsync(out, static_cast<char *>(workspace) + L.spikes, n, cudaMemcpyDeviceToDevice,
                           reinterpret_cast<cudaStream_t>(stream)));
    return N2B_OK;
}

int n2b_project_forward(const int32_t *row_ptr, const int32_t *channel, int32_t rows, int32_t channels,
                        int32_t hidden, const float *w_in, float *u, void *stream) {
    if (rows < 0 || channels <= 0 || hidden <= 0 || hidden % 4 || hidden > 1024)
        return bfail(N2B_EINVAL, "project: rows >= 0, channels > 0, hidden a multiple of 4 up to 1024");
    if (rows == 0) return N2B_OK;
    if (!row_ptr || !channel || !w_in || !u) return bfail(N2B_EINVAL, "project: missing arguments");
    if ((reinterpret_cast<uintptr_t>(w_in) | reinterpret_cast<uintptr_t>(u)) & 15)
        return bfail(N2B_EINVAL, "project: w_in and u must be 16-byte aligned");
    const int h4 = hidden / 4, rpb = std::max(1, 256 / h4);
    project_fwd_kernel<<<(unsigned)((rows + rpb - 1) / rpb), (unsigned)(rpb * h4), 0,
                         reinterpret_cast<cudaStream_t>(stream)>>>(row_ptr, channel, rows, channels, hidden, w_in, u);
    B_CUDA(cudaGetLastError());
    return N2B_OK;
}

int n2b_project_backward(const int32_t *chunk_ptr, int32_t n_chunks, const int32_t *row_idx,
                         const int32_t *channel_chunk, int32_t channels, int32_t rows, int32_t hidden,
                         const float *du, float *partials, float *dw_in, void *stream) {
    if (n_chunks < 0 || rows < 0 || channels <= 0 || hidden <= 0 || hidden % 4 || hidden > 1024)
        return bfail(N2B_EINVAL, "project: n_chunks, rows >= 0, channels > 0, hidden a multiple of 4 up to 1024");
    if (!channel_chunk || !dw_in || (n_chunks > 0 && (!chunk_ptr || !row_idx || !du || !partials)))
        return bfail(N2B_EINVAL, "project: missing arguments");
    if ((reinterpret_cast<uintptr_t>(du) | reinterpret_cast<uintptr_t>(partials)) & 15)
        return bfail(N2B_EINVAL, "project: du and partials must be 16-byte aligned");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (n_chunks > 0) {
        project_bwd_chunk_kernel<<<(unsigned)n_chunks, (unsigned)(hidden / 4), 0, s>>>(chunk_ptr, row_idx, rows,
                                                                                     hidden, du, partials);
        B_CUDA(cudaGetLastError());
    }
    const size_t n = (size_t)channels * hidden;
    project_bwd_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(channel_chunk, channels, hidden, partials,
                                                                          dw_in);
    B_CUDA(cudaGetLastError());
    return N2B_OK;
}

}  // extern "C"

/*
 * rsc_nodes.cuh -- pulse formation on the triangle range weight, summed on
 * the nodes of the gate grid.
 *
 * The triangle whose half width is a whole number n of gate spacings is
 * linear in range between neighbouring gate origins: the weight a scatterer
 * has in gate k is the interpolation, between the two nodes E_m <= r < E_m+1
 * it lies between, of the weights W(k, m) of gate k at the nodes.  So a
 * scatterer adds its signal to two nodes with the weights (E_m+1 - r) and
 * (r - E_m) over the spacing, both exact differences times one reciprocal,
 * and the last block forms every gate from its 2 n - 1 nodes.  The work per
 * scatterer does not depend on n: a pulse sampled finely in range costs what
 * a coarse one does.  The nodes are the gate origins the reference's running
 * sum gives (rs.cl:1214), continued evenly on both sides.  Where that sum
 * drifts from the spacing, the triangle's ends miss the nodes and the plain
 * sums stay gate by gate (node_slip in rsc.cu); the compensated ones use the
 * even grid and end where the table does.
 *
 * Each warp takes a contiguous piece of the state, 64 neighbours at a time,
 * lane l holding scatterers l and l + 32.  A state in spatial order keeps a
 * run within two neighbouring intervals, so the warp holds the sums of their
 * three nodes in registers, lane by lane, and reduces them across its lanes
 * only when a run leaves them.
 *
 * What bounds it: the issue of its instructions.  README scale (2,001,920
 * scatterers, 40 gates, n = 2): 13.0 M warp instructions, 24.9 us alone,
 * against 22.0 M and 35.0 us for the sums gate by gate (k_pulse_group); the
 * step beside the advance 67.1 -> 57.6 us.  500,000 scatterers on 240 gates
 * (n = 12, which the gate window did not hold: every gate visited) 441 ->
 * 19 us.  The signal's quotients and roots share one range check per
 * scatterer instead of one each.  Written on packed pairs instead of two
 * scalar scatterers it issued 10% fewer instructions (each constant of a
 * packed operation costs its moves) but needed 77-104 registers and was
 * slower (26.9 us); runs staged in shared memory by cp.async (the addresses
 * and the copies' own loads cost more than the latency they hid) 31.0.
 */
#ifndef SIMRADAR_GB300_RSC_NODES_CUH
#define SIMRADAR_GB300_RSC_NODES_CUH

#include "rsc_pulse.cuh"

namespace rsc {

/* Largest half width of the triangle, in gate spacings. */
constexpr int kNodeMaxN = 64;

/* A scatterer's signal: its range, and signal x angular weight of each lane
 * (Ih, Qh, Iv, Qv). */
struct Sig {
    float r, s[4];
};

/* signal_plain.  The range, the phase and the angular weight are its values
 * bit for bit (rsc_mid.cuh; the three direction cosines share one reciprocal);
 * 1 / r^2 is taken of the squared range and joins the angular weight before
 * the rotation, whose sums are fused.  False when a scatterer is beyond 60
 * degrees off the beam, closer than 2^-30 m or at a phase above 6e6 rad: the
 * caller takes signal_plain. */
__device__ __forceinline__ bool signal_plain_mid(const PulseArgs &P, const float4 &p, const float4 &x, Sig &o) {
    const float *sd = P.sim;
    const float s = p.x * p.x + p.y * p.y + p.z * p.z;
    const float r = sqrt_mid(s);
    /* the cosine of the beam angle, each direction cosine rounded */
    const float y = rcp_mid(r);
    const float dot = sd[0] * div_by(p.x, r, y) + sd[1] * div_by(p.y, r, y) + sd[2] * div_by(p.z, r, y);
    const float phase = r * sd[4];
    /* 1 / r^2, as the reciprocal of the squared range */
    float k = rcp_mid(s);
    /* acos(dot) = 2 asin(sqrt((1 - dot) / 2)), 0 past 1 (rsm_acosf); the
     * doubling joins the table's scale, which is exact */
    const float z = fmaxf(fmaf(dot, -0.5f, 0.5f), 0.0f);
    const float sz = sqrt_from(z, rsqrt_approx(fmaxf(z, 0x1p-80f)));
    const float half = fmaf(sz * z, rsm_asin_poly(z), sz), scale = 2.0f * P.awd[0];
    const float raw0 = cl_clamp(fmaf(half, scale, P.awd[1] + 0.0f), 0.0f, P.awd[2]);
    const float raw1 = cl_clamp(fmaf(half, scale, P.awd[1] + 1.0f), 0.0f, P.awd[2]);
    k = k * cl_mix(__ldg(P.aw + (uint32_t)raw0), __ldg(P.aw + (uint32_t)raw1), raw0 - floorf(raw0));
    /* sine and cosine (rsm_sincosf): adding 1.5 x 2^23 rounds to the integer,
     * whose low bits are then the sum's */
    const float qm = __fadd_rn(phase * RSM_TWO_OVER_PI, 12582912.0f);
    const float q = qm - 12582912.0f;
    float t = fmaf(-q, RSM_PIO2_1, phase);
    t = fmaf(-q, RSM_PIO2_2, t);
    t = fmaf(-q, RSM_PIO2_3, t);
    float ss, cc;
    {
        const float w = t * t;
        float ps = fmaf(0x1.71de3ap-19f, w, -0x1.a01a02p-13f);   /* rsm_sincos_reduced */
        ps = fmaf(ps, w, 0x1.111112p-7f);
        ps = fmaf(ps, w, -0x1.555556p-3f);
        const float sn = fmaf(t * w, ps, t);
        float pc = fmaf(-0x1.27e4fcp-22f, w, 0x1.a01a02p-16f);
        pc = fmaf(pc, w, -0x1.6c16c2p-10f);
        pc = fmaf(pc, w, 0x1.555556p-5f);
        pc = fmaf(pc, w, -0.5f);
        const float cs = fmaf(w, pc, 1.0f);
        const unsigned b = __float_as_uint(qm);
        const bool swap = (b & 1u) != 0u;
        ss = __uint_as_float(__float_as_uint(swap ? cs : sn) ^ ((b & 2u) << 30)) * k;
        cc = __uint_as_float(__float_as_uint(swap ? sn : cs) ^ (((b + 1u) & 2u) << 30)) * k;
    }
    o.r = r;
    o.s[0] = fmaf(x.x, cc, x.y * ss);
    o.s[1] = fmaf(x.y, cc, -(x.x * ss));
    o.s[2] = fmaf(x.z, cc, x.w * ss);
    o.s[3] = fmaf(x.w, cc, -(x.z * ss));
    return dot > 0.5f && dot <= 0x1.00002p+0f && s > 0x1p-60f && fabsf(phase) < 6.0e6f;
}

/* The sum of four values over the warp's lanes: the sum of value c in lanes
 * 8 c .. 8 c + 7 (six shuffles). */
__device__ __forceinline__ float warp_sum4(unsigned lane, float v0, float v1, float v2, float v3) {
    const bool h16 = (lane & 16u) != 0;
    float k0 = h16 ? v2 : v0, k1 = h16 ? v3 : v1;
    k0 = k0 + __shfl_xor_sync(0xffffffffu, h16 ? v0 : v2, 16);
    k1 = k1 + __shfl_xor_sync(0xffffffffu, h16 ? v1 : v3, 16);
    const bool h8 = (lane & 8u) != 0;
    float k = h8 ? k1 : k0;
    k = k + __shfl_xor_sync(0xffffffffu, h8 ? k0 : k1, 8);
    k = k + __shfl_xor_sync(0xffffffffu, k, 4);
    k = k + __shfl_xor_sync(0xffffffffu, k, 2);
    return k + __shfl_xor_sync(0xffffffffu, k, 1);
}

/* Nodes of a pulse of G gates: m = -n .. G + n - 1, at index m + n. */
__host__ __device__ __forceinline__ unsigned node_count(unsigned G, int n) { return G + 2u * (unsigned)n; }
__host__ __device__ __forceinline__ size_t node_smem_bytes(unsigned G, int n, bool compensated) {
    return (size_t)node_count(G, n) * (compensated ? 8 * sizeof(double) : 4 * sizeof(double) + sizeof(float));
}

/* 4 blocks of 256 per SM at 64 registers, nothing spilled.  README scale,
 * pulse alone: 24.9 us; 26.9 with 3 blocks at 77 registers, 24.8 with 2 of
 * 512, 28.1 with 8 of 128. */
constexpr int kNodeThreads = 256, kNodeMinBlocks = 4;

/* The compensated form: 3 blocks at 80 registers (40 bytes spilled) against 2
 * at 115: a dwell of 3 pulses of 8.4 M scatterers 919 us against 941, of 2 of
 * 33.7 M 3449 against 3486. */
constexpr int kCompMinBlocks = 3;

/* Runs a warp should have at least: a small state takes fewer blocks
 * (131,072 scatterers, pulses read back: 17.8 us per step with 1, 18.3 with
 * 2, 21.3 with 3). */
constexpr unsigned kNodeRuns = 1;

/* Copies of the nodes' sums that single scatterers are added to (a power of
 * two): blocks share a copy, so that few meet in an address. */
constexpr unsigned kNodeCopies = 8;
__host__ __device__ __forceinline__ unsigned node_copies(unsigned G, int n) {
    unsigned c = kNodeCopies;
    while (c > 1 && c * node_count(G, n) > 1024u) c >>= 1;
    return c;
}

/* Scatterers of a run that make a window worth moving to them (a move costs a
 * reduction of its sums, about what eight scatterers alone cost). */
constexpr int kNodePart = 8;
/* ... in runs of their own piece.  The other runs (sparse debris: a run spans
 * several intervals; a state in the caller's order) move it for no fewer than
 * this, and a run with as many in the window lets the rest go one by one
 * without looking further (60,000 drops and 3 x 800 debris: 161 us for 8
 * steps against 175 when sparse runs were taken window by window). */
constexpr int kNodeMost = 40;

/* A warp's window of three nodes and their sums, lane by lane (plain form). */
struct NodeWindow {
    float E0, E1, E2, i0, i1;
    int c;              /* node index of E0, -1: none yet */
    float acc[3][4];

    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int m = 0; m < 3; m++) {
#pragma unroll
            for (int l = 0; l < 4; l++) acc[m][l] = 0.0f;
        }
    }
    __device__ __forceinline__ void move(const PulseArgs &P, int node) {
        c = node;
        E0 = __ldg(P.node + node);
        E1 = __ldg(P.node + node + 1);
        E2 = __ldg(P.node + node + 2);
        i0 = 1.0f / (E1 - E0);
        i1 = 1.0f / (E2 - E1);
        clear();
    }
    __device__ __forceinline__ bool holds(float r) const { return r >= E0 && r < E2; }
    /* a scatterer at a range in [E0, E2) weighed onto the three nodes */
    __device__ __forceinline__ void add(const Sig &g) {
        const float w0 = fmaxf((E1 - g.r) * i0, 0.0f);
        const float w1 = fminf((g.r - E0) * i0, (E2 - g.r) * i1);
        const float w2 = fmaxf((g.r - E1) * i1, 0.0f);
        fma_pair(w0, g.s[0], g.s[1], acc[0][0], acc[0][1]);
        fma_pair(w0, g.s[2], g.s[3], acc[0][2], acc[0][3]);
        fma_pair(w1, g.s[0], g.s[1], acc[1][0], acc[1][1]);
        fma_pair(w1, g.s[2], g.s[3], acc[1][2], acc[1][3]);
        fma_pair(w2, g.s[0], g.s[1], acc[2][0], acc[2][1]);
        fma_pair(w2, g.s[2], g.s[3], acc[2][2], acc[2][3]);
    }
    /* the lanes' sums into the block's bins */
    __device__ __forceinline__ void flush(double *bins, unsigned lane) {
        if (c < 0) return;
#pragma unroll
        for (int m = 0; m < 3; m++) {
            const float k = warp_sum4(lane, acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
            if ((lane & 7u) == 0u && k != 0.0f) atomicAdd(bins + 4 * (c + m) + (lane >> 3), (double)k);
        }
        c = -1;
    }
};

/* ---- the compensated form ----
 * The same walk over the state with double-float sums.  Bound by instruction
 * issue (FP32 adds and FMAs of the double-floats): README scale 36.6 M warp
 * instructions and 59.6 us alone, against 61.9 M and 88.4 us for moments per
 * interval reduced across the warp for every run of 64 with signal_comp's
 * terms; 8.4 M scatterers at 30 km 266 -> 202 us; 77,777 on gates 7.5 m apart
 * (too many for the gate window: every gate visited) 119 -> 15 us.  A gate's
 * error against FP64 is what it was or less (rms 8.4e-9 of the sum of |x| on a
 * 21,536-scatterer scene, both forms: the output's rounding; 1,000 pulses of
 * 8.4 M at 30 km 2.3e-8 of the gate, 2.7e-8 before). */

/* Add the double-float (h, l) to the double-float sum (S, s). */
__device__ __forceinline__ void df_acc(float &S, float &s, float h, float l) {
    float a, e;
    two_sum(S, h, a, e);
    S = a;
    s = s + (e + l);
}

/* The sum of four double-floats over the warp's lanes, the sum of value c in
 * lanes 8 c .. 8 c + 7, heads added error-free. */
__device__ __forceinline__ void warp_sum4_df(unsigned lane, const float *v, const float *u, float &S, float &s) {
    const bool h16 = (lane & 16u) != 0, h8 = (lane & 8u) != 0;
    float k0 = h16 ? v[2] : v[0], k1 = h16 ? v[3] : v[1], t0 = h16 ? u[2] : u[0], t1 = h16 ? u[3] : u[1];
    df_acc(k0, t0, __shfl_xor_sync(0xffffffffu, h16 ? v[0] : v[2], 16),
           __shfl_xor_sync(0xffffffffu, h16 ? u[0] : u[2], 16));
    df_acc(k1, t1, __shfl_xor_sync(0xffffffffu, h16 ? v[1] : v[3], 16),
           __shfl_xor_sync(0xffffffffu, h16 ? u[1] : u[3], 16));
    S = h8 ? k1 : k0;
    s = h8 ? t1 : t0;
    df_acc(S, s, __shfl_xor_sync(0xffffffffu, h8 ? k0 : k1, 8), __shfl_xor_sync(0xffffffffu, h8 ? t0 : t1, 8));
#pragma unroll
    for (int off = 4; off > 0; off >>= 1)
        df_acc(S, s, __shfl_xor_sync(0xffffffffu, S, off), __shfl_xor_sync(0xffffffffu, s, off));
}

/* Node j of the even grid, rs + (j - n) delta, as a double-float. */
__device__ __forceinline__ void comp_node(const PulseArgs &P, int j, float &h, float &l) {
    float a, b, s, e;
    two_prod((float)(j - P.mom_n), P.rdelta, a, b);
    two_sum(P.rs, a, s, e);
    fast_two_sum(s, e + b, h, l);
}

/* f 2^-896 as a double: its exponent as it stands under the wider bias, exact
 * for subnormal values too.  (The FP64 units' conversions issue at 1/64 of the
 * FP32 rate: 8.4 M scatterers, 3 steps, 1,025 us with them, 930 without.)  An
 * infinity or NaN stays one in the head of a double-float, which makes the
 * sum one whatever the tail gives. */
constexpr double kWideScale = 0x1p896;
template <bool HEAD>
__device__ __forceinline__ double wide_of(float f) {
    const unsigned b = __float_as_uint(f), m = b & 0x7fffffffu;
    unsigned hi = (m >> 3) | (b & 0x80000000u);
    if (HEAD && m >= 0x7f800000u) hi |= 0x7ff00000u;
    return __hiloint2double((int)hi, (int)(b << 29));
}
/* The same of a double of FP32's range. */
__device__ __forceinline__ double wide_scaled(double v) {
    const unsigned hi = (unsigned)__double2hiint(v), m = hi & 0x7fffffffu;
    if (m - 0x38100000u >= 0x0fe00000u) return v * (1.0 / kWideScale);   /* beyond FP32's normal numbers */
    return __hiloint2double((int)(hi - 0x38000000u), __double2loint(v));
}
/* And back, as a double-float: 24 bits of head, cut off, and 29 of tail; false
 * beyond FP32's range. */
__device__ __forceinline__ bool wide_split(double d, float &h, float &l) {
    const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
    const unsigned s = hi & 0x80000000u, m = hi & 0x7fffffffu, e = m >> 20;
    h = __uint_as_float(s | (m << 3) | (lo >> 29));
    l = e > 23u ? __uint_as_float(s | ((e - 23u) << 23)) * ((float)(lo & 0x1fffffffu) * 0x1p-29f) : 0.0f;
    return e < 0xffu;
}
__device__ __forceinline__ bool not_zero(double d) {
    return (((unsigned)__double2hiint(d) & 0x7fffffffu) | (unsigned)__double2loint(d)) != 0u;
}

/* A double-float into a sum in L2 (of 2^-896 times the values), as two
 * reductions: the additions happen there, not in the SM's few FP64 lanes.  (As atomicAdd through a generic
 * pointer each waited for its answer: 3 us per scatterer.) */
__device__ __forceinline__ void red_add(double *o, double v) {
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(o), "d"(v) : "memory");
}
__device__ __forceinline__ void red_add_df(double *o, float h, float l) {
    red_add(o, wide_of<true>(h));
    red_add(o, wide_of<false>(l));
}

/* The compensated sums of an interval [E_j, E_j+1) between two nodes of the
 * even grid: Sum x and Sum (r - E_j) x of its terms x, per lane, from which
 * the last block forms every gate exactly (the triangle's end lies where its
 * table's scale puts it, a few ulps off the node: an interval's own line is
 * right up to there, where node sums would mix it with its neighbour's).
 * Doubles acc64[8 j + l] and acc64[8 j + 4 + l], scaled as wide_of. */
constexpr unsigned kCompSums = 8;

/* A warp's window of two intervals beside the node E, with t = r - E: below
 * it (side 0) and above (side 1) the sums of x and of |t| x. */
struct CompWindow {
    float Eh, El;
    int c;              /* the lower interval, -1: none yet */
    float X[2][4], x[2][4], T[2][4], t[2][4];

    __device__ __forceinline__ void move(const PulseArgs &P, int j) {
        c = j;
        comp_node(P, j + 1, Eh, El);
#pragma unroll
        for (int q = 0; q < 2; q++) {
#pragma unroll
            for (int l = 0; l < 4; l++) X[q][l] = x[q][l] = T[q][l] = t[q][l] = 0.0f;
        }
    }
    __device__ __forceinline__ void offset(const CompSig &g, float &th, float &tl) const {
        float e;
        two_sum(g.r, -Eh, th, e);
        tl = e + (g.rl - El);
    }
    template <int Q>
    __device__ __forceinline__ void add_side(const CompSig &g, float dh, float dl) {
#pragma unroll
        for (int l = 0; l < 4; l++) {
            float ph, pl;
            df_acc(X[Q][l], x[Q][l], g.s[l], g.u[l]);
            df_mul_pair(g.s[l], g.u[l], dh, dl, ph, pl);
            df_acc(T[Q][l], t[Q][l], ph, pl);
        }
    }
    __device__ __forceinline__ void add(const CompSig &g, float th, float tl) {
        /* a run in spatial order mostly lies on one side */
        if (th + tl >= 0.0f) add_side<1>(g, th, tl);
        else add_side<0>(g, -th, -tl);
    }
    __device__ __forceinline__ void flush(const PulseArgs &P, unsigned lane) {
        if (c < 0) return;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (!__any_sync(0xffffffffu, X[q][0] != 0.0f || X[q][1] != 0.0f || X[q][2] != 0.0f || X[q][3] != 0.0f)) continue;
            float a, b, d, e;
            warp_sum4_df(lane, X[q], x[q], a, b);
            warp_sum4_df(lane, T[q], t[q], d, e);
            if ((lane & 7u) == 0u) {
                if (q == 0) {
                    /* |t| = delta - (r - E_j) */
                    float mh, ml;
                    df_mul_pair(a, b, P.rdelta, 0.0f, mh, ml);
                    df_acc(mh, ml, -d, -e);
                    d = mh;
                    e = ml;
                }
                double *o = P.acc64 + kCompSums * (unsigned)(c + q) + (lane >> 3);
                red_add_df(o, a, b);
                red_add_df(o + 4, d, e);
            }
        }
        c = -1;
    }
};

/* The interval of a range to one (comp_stray puts it right), -1 off the nodes. */
__device__ __forceinline__ int comp_interval(const PulseArgs &P, float r) {
    const int last = (int)node_count(P.G, P.mom_n) - 2;
    const float jf = floorf((r - P.rs) * P.inv_delta) + (float)P.mom_n;
    return jf >= -1.0f && jf <= (float)(last + 1) ? min(max((int)jf, 0), last) : -1;
}
__device__ __noinline__ void comp_stray(const PulseArgs &P, int j, const CompSig &g) {
    const float delta = P.rdelta;
    const int last = (int)node_count(P.G, P.mom_n) - 2;
    float a, b, c, d, uh, ul;
    comp_node(P, j, c, d);
    two_sum(g.r, -c, uh, ul);
    ul = ul + (g.rl - d);
    /* The quotient can be one off beside a node.  Which side is decided on the
     * double-float less the node's offset, not on the rounded uh + ul, which is
     * delta up to half an ulp below it: the next interval's offset would be
     * negative there and the scatterer in neither. */
    two_sum(uh, -delta, a, b);
    if (uh + ul < 0.0f) {
        j--;
        two_sum(uh, delta, uh, b);
        ul = ul + b;
    } else if (a + (b + ul) >= 0.0f) {
        j++;
        uh = a;
        ul = b + ul;
    }
    if (j < 0 || j > last) return;
    double *o = P.acc64 + kCompSums * (unsigned)j;
#pragma unroll 1
    for (int l = 0; l < 4; l++) {
        df_mul_pair(g.s[l], g.u[l], uh, ul, a, b);
        red_add_df(o + l, g.s[l], g.u[l]);
        red_add_df(o + 4 + l, a, b);
    }
}

/* Non-finite values: their lanes of every gate NaN (0 x NaN in pass 1), the
 * scatterer's finite lanes kept; false when its range is not finite and
 * nothing is left of it. */
__device__ __noinline__ bool comp_non_finite(const PulseArgs &P, CompSig &g) {
    double *gate = P.acc64 + kCompSums * (size_t)node_count(P.G, P.mom_n);
    const bool range = fabsf(g.r) < INFINITY;
    for (int l = 0; l < 4; l++) {
        if (range && fabsf(g.s[l]) < INFINITY && fabsf(g.u[l]) < INFINITY) continue;
        g.s[l] = g.u[l] = 0.0f;
        for (unsigned k = 0; k < P.G; k++) atomicAdd(gate + 4 * k + l, (double)NAN);
    }
    return range;
}

/* A run the window does not hold whole: as node_settle. */
__device__ __forceinline__ void comp_settle(const PulseArgs &P, CompWindow &W, CompSig *g, unsigned in, int part,
                                            unsigned lane) {
    int j[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        j[q] = -1;
        if (!((in >> q) & 1u)) continue;
        bool live = true;
        if (!(fabsf(g[q].r) < INFINITY) || !finite4(g[q].s) || !finite4(g[q].u)) live = comp_non_finite(P, g[q]);
        if (live) j[q] = comp_interval(P, g[q].r);
    }
    for (;;) {
        const unsigned l0 = __ballot_sync(0xffffffffu, j[0] >= 0), l1 = __ballot_sync(0xffffffffu, j[1] >= 0);
        if ((l0 | l1) == 0u) return;
        const auto within = [&](int c) {
            return __popc(__ballot_sync(0xffffffffu, j[0] >= 0 && (unsigned)(j[0] - c) < 2u)) +
                   __popc(__ballot_sync(0xffffffffu, j[1] >= 0 && (unsigned)(j[1] - c) < 2u));
        };
        int here = W.c < 0 ? 0 : within(W.c);
        if (here < part) {
            int best = 0, at = 0;
            unsigned t0 = l0, t1 = l1;
#pragma unroll 1
            for (int t = 0; t < 4 && best < part && (t0 | t1) != 0u; t++) {
                const int src = __ffs(t0 ? t0 : t1) - 1;
                const int cand = __shfl_sync(0xffffffffu, t0 ? j[0] : j[1], src);
                const int a = within(cand - 1), b = within(cand);
                best = max(a, b);
                at = a > b ? cand - 1 : cand;
                if (t0) t0 &= ~(0x1ffu << (src & ~7));
                else t1 &= ~(0x1ffu << (src & ~7));
            }
            if (best < part) {
                if (j[0] >= 0) comp_stray(P, j[0], g[0]);
                if (j[1] >= 0) comp_stray(P, j[1], g[1]);
                return;
            }
            W.flush(P, lane);
            W.move(P, min(max(at, 0), (int)node_count(P.G, P.mom_n) - 3));
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (j[q] >= 0 && (unsigned)(j[q] - W.c) < 2u) {
                float th, tl;
                W.offset(g[q], th, tl);
                /* one off beside the window's end: by itself */
                if (fabsf(th + tl) <= P.rdelta) W.add(g[q], th, tl);
                else comp_stray(P, j[q], g[q]);
                j[q] = -1;
            }
        }
    }
}

/* A scatterer with a non-finite signal reaches every gate, its weight there
 * as pass 1 forms it (0 x NaN is NaN): straight into the grid's sums of the
 * gates, which the last block adds to what the nodes give. */
__device__ __noinline__ void node_non_finite(const PulseArgs &P, float r, float v0, float v1, float v2, float v3) {
    double *gate = P.acc64 + 4 * (size_t)node_count(P.G, P.mom_n);
    for (unsigned k = 0; k < P.G; k++) {
        const float w = range_weight(P, r - __ldg(P.rk + k));
        atomicAdd(gate + 4 * k + 0, (double)(w * v0));
        atomicAdd(gate + 4 * k + 1, (double)(w * v1));
        atomicAdd(gate + 4 * k + 2, (double)(w * v2));
        atomicAdd(gate + 4 * k + 3, (double)(w * v3));
    }
}

/* Index of the interval [E_j, E_j+1) that holds r, -1 outside the nodes. */
__device__ __forceinline__ int node_interval(const PulseArgs &P, float r) {
    const int last = (int)node_count(P.G, P.mom_n) - 2;
    const float jf = floorf((r - __ldg(P.node)) * P.inv_delta);
    if (!(jf >= -1.0f && jf <= (float)(last + 1))) return -1;
    int j = min(max((int)jf, 0), last);
    /* the quotient can be one off beside a node */
    if (r < __ldg(P.node + j)) j--;
    else if (r >= __ldg(P.node + j + 1)) j++;
    return j > last ? -1 : j;
}

/* One scatterer, in interval j, by itself: eight FP64 reductions in L2 (scaled
 * as wide_of), which nothing waits for.  (2,000,000 out of spatial order on 512
 * gates 1.5 m apart, which all go this way: 799 us; 273 as two reductions of
 * four FP32 values, whose sums of 1e5 terms lose three digits; 4,082 with every
 * gate visited.) */
__device__ __forceinline__ void node_stray(const PulseArgs &P, double *stray, int j, float r, const float *v) {
    const float a = __ldg(P.node + j), b = __ldg(P.node + j + 1), i = 1.0f / (b - a);
    const float wa = (b - r) * i, wb = (r - a) * i;
    double *o = stray + 4 * (unsigned)j;
#pragma unroll
    for (int l = 0; l < 4; l++) {
        red_add(o + l, wide_of<true>(wa * v[l]));
        red_add(o + 4 + l, wide_of<true>(wb * v[l]));
    }
}

/* A lane's scatterer by itself: to every gate when not finite, nowhere when
 * it reaches none. */
__device__ __forceinline__ bool sig_finite(const Sig &g) { return fabsf(g.r) < INFINITY && finite4(g.s); }
__device__ __forceinline__ void node_alone(const PulseArgs &P, const Sig &g, double *stray) {
    if (!sig_finite(g)) {
        node_non_finite(P, g.r, g.s[0], g.s[1], g.s[2], g.s[3]);
        return;
    }
    const int j = node_interval(P, g.r);
    if (j >= 0) node_stray(P, stray, j, g.r, g.s);
}

/* A run the window holds little of.  Scatterers that reach no gate drop out
 * and non-finite ones go to every gate; what the window, or one moved to
 * where a good part of the run lies, holds is added to it, and the rest --
 * debris, scatterers respawned elsewhere since the last sort -- one by one. */
__device__ __forceinline__ void node_settle(const PulseArgs &P, NodeWindow &W, const Sig *g, unsigned in, int part,
                                            double *bins, double *stray, unsigned lane) {
    int j[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        j[q] = -1;
        if (!((in >> q) & 1u)) continue;
        if (!sig_finite(g[q])) {
            node_non_finite(P, g[q].r, g[q].s[0], g[q].s[1], g[q].s[2], g[q].s[3]);
        } else {
            j[q] = node_interval(P, g[q].r);
        }
    }
    for (;;) {
        const unsigned l0 = __ballot_sync(0xffffffffu, j[0] >= 0), l1 = __ballot_sync(0xffffffffu, j[1] >= 0);
        if ((l0 | l1) == 0u) return;
        const auto within = [&](int c) {
            return __popc(__ballot_sync(0xffffffffu, j[0] >= 0 && (unsigned)(j[0] - c) < 2u)) +
                   __popc(__ballot_sync(0xffffffffu, j[1] >= 0 && (unsigned)(j[1] - c) < 2u));
        };
        if (W.c < 0 || within(W.c) < part) {
            /* where a few of those left lie: any of them may be astray */
            int best = 0, at = 0;
            unsigned t0 = l0, t1 = l1;
#pragma unroll 1
            for (int t = 0; t < 4 && best < part && (t0 | t1) != 0u; t++) {
                const int src = __ffs(t0 ? t0 : t1) - 1;
                const int cand = __shfl_sync(0xffffffffu, t0 ? j[0] : j[1], src);
                const int a = within(cand - 1), b = within(cand);
                best = max(a, b);
                at = a > b ? cand - 1 : cand;
                /* the next a quarter of the run on */
                if (t0) t0 &= ~(0x1ffu << (src & ~7));
                else t1 &= ~(0x1ffu << (src & ~7));
            }
            if (best < part) {
                if (j[0] >= 0) node_stray(P, stray, j[0], g[0].r, g[0].s);
                if (j[1] >= 0) node_stray(P, stray, j[1], g[1].r, g[1].s);
                return;
            }
            W.flush(bins, lane);
            W.move(P, min(max(at, 0), (int)node_count(P.G, P.mom_n) - 3));
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (j[q] >= 0 && (unsigned)(j[q] - W.c) < 2u) {
                W.add(g[q]);
                j[q] = -1;
            }
        }
    }
}

/* The end of a block whose sums are on their way to the grid's accumulator:
 * the last block forms the gates and leaves accumulator and counter at zero.
 * A chain of round trips to L2 at the end of every pulse: the sums
 * (reductions nothing waits for), the ticket, the loads, all of them before
 * the first gate is formed (393,225 scatterers: 333.5 -> 328.5 us for 10
 * steps; 500,000 on gates 2.5 m apart: 140 -> 137.7 for 4, against generic
 * atomics, a fence on both sides of the ticket and the gates' own sums loaded
 * one by one).  STRAY: scatterers may have gone to P.stray. */
template <int MODE, bool STRAY>
__device__ __forceinline__ void node_gates(const PulseArgs &P, double *bins, unsigned nblk) {
    const unsigned nodes = node_count(P.G, P.mom_n), outs = P.G * 4;
    __shared__ bool s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        /* after the barrier this orders every thread's reductions before the
         * ticket, and the last block's reads after it */
        unsigned t;
        asm volatile("atom.global.add.acq_rel.gpu.u32 %0, [%1], 1;" : "=r"(t) : "l"(P.counter) : "memory");
        s_last = t == nblk - 1;
    }
    __syncthreads();
    if (!s_last) return;
    /* the first of this thread's outputs' single contributions, on its way
     * together with the sums */
    double *extra = P.acc64 + (size_t)(MODE == 1 ? kCompSums : 4u) * nodes;
    const unsigned first = MODE == 1 ? threadIdx.x : 2 * threadIdx.x;
    const double e0 = first < outs ? __ldcg(extra + first) : 0.0;
    const double f0 = MODE == 0 && first < outs ? __ldcg(extra + first + 1) : 0.0;
    if constexpr (MODE == 1) {
        const unsigned all = nodes * kCompSums;
#pragma unroll 4
        for (unsigned o = threadIdx.x; o < all; o += blockDim.x) bins[o] = __ldcg(P.acc64 + o) * kWideScale;
        __syncthreads();
        for (unsigned o = threadIdx.x; o < all; o += blockDim.x) P.acc64[o] = 0.0;
        const double s = (double)P.rwd[0], ds = (double)P.rdelta * s;
        for (unsigned o = threadIdx.x; o < outs; o += blockDim.x) {
            const unsigned k = o >> 2, l = o & 3u, n = (unsigned)P.mom_n;
            double sum = 0.0;
            /* gate k lies at index k + n: the intervals n below it, where the
             * weight is 1 - (m delta - u) s, and n above, 1 - (m delta + u) s */
            for (unsigned m = 0; m < n; m++) {
                const double *lo = bins + kCompSums * (k + n - 1 - m) + l, *hi = bins + kCompSums * (k + n + m) + l;
                sum = fma(1.0 - (double)(m + 1) * ds, lo[0], sum);
                sum = fma(1.0 - (double)m * ds, hi[0], sum);
                sum = fma(s, lo[4] - hi[4], sum);
            }
            const double e = o == threadIdx.x ? e0 : __ldcg(extra + o);
            if (e != 0.0) extra[o] = 0.0;
            reinterpret_cast<float *>(P.pulse)[o] = (float)(sum + e);
        }
        if (threadIdx.x == 0) *P.counter = 0u;
        return;
    }
    /* each node's sum as a double-float, over bins[o], whose sums are out: the
     * FP64 units of the one block add 2 numbers a cycle (500,000 scatterers on
     * 240 gates, 4 pulses: 138 us, 136 with FP32 sums) */
    float2 *sums = reinterpret_cast<float2 *>(bins);
    float *at_node = reinterpret_cast<float *>(sums + 4 * nodes);
    const unsigned copies = node_copies(P.G, P.mom_n);
    bool fits = true;
    /* the loads of several sums in flight at once: no store or branch between them */
#pragma unroll 4
    for (unsigned o = threadIdx.x; o < nodes * 4; o += blockDim.x) {
        double d[STRAY ? kNodeCopies + 1 : 1];
        d[0] = __ldcg(P.acc64 + o);
#pragma unroll
        for (unsigned c = 0; STRAY && c < kNodeCopies; c++) {
            d[c + 1] = c < copies ? __ldcg(P.stray + (size_t)c * 4 * nodes + o) : 0.0;
        }
        float h, l;
        fits = wide_split(d[0], h, l) && fits;
#pragma unroll
        for (unsigned c = 0; STRAY && c < kNodeCopies; c++) {
            float a, b;
            fits = wide_split(d[c + 1], a, b) && fits;
            df_acc(h, l, a, b);
        }
        sums[o] = make_float2(h, l);
    }
    for (unsigned o = threadIdx.x; o < nodes; o += blockDim.x) at_node[o] = __ldg(P.node + o);
    if (__syncthreads_or(!fits)) {
        for (unsigned o = threadIdx.x; o < nodes * 4; o += blockDim.x) {
            double v = __ldcg(P.acc64 + o);
            for (unsigned c = 0; STRAY && c < copies; c++) v = v + __ldcg(P.stray + (size_t)c * 4 * nodes + o);
            v = v * kWideScale;
            const float h = (float)v;
            sums[o] = make_float2(h, fabsf(h) < INFINITY ? (float)(v - (double)h) : 0.0f);
        }
        __syncthreads();
    }
    for (unsigned o = threadIdx.x; o < nodes * 4; o += blockDim.x) P.acc64[o] = 0.0;
    for (unsigned o = threadIdx.x; STRAY && o < 2 * nodes * copies; o += blockDim.x) {
        reinterpret_cast<double2 *>(P.stray)[o] = make_double2(0.0, 0.0);
    }
    /* two values of a gate per thread, which share its weights */
    const int n = P.mom_n;
    const float4 *two = reinterpret_cast<const float4 *>(sums);
    for (unsigned o = threadIdx.x; o < P.G * 2; o += blockDim.x) {
        const unsigned k = o >> 1, half = o & 1u;
        const float rk = __ldg(P.rk + k);
        float sum[2] = {0.0f, 0.0f}, low[2] = {0.0f, 0.0f};
        const unsigned end = min(k + 2u * (unsigned)n + 1u, nodes);
#pragma unroll 4
        for (unsigned at = k; at < end; at++) {
            const float w = fmaxf(1.0f - fabsf(at_node[at] - rk) * P.rwd[0], 0.0f);
            const float4 x = two[2 * at + half];
            const float a = x.x * w, b = x.z * w;
            df_acc(sum[0], low[0], a, fmaf(x.y, w, fmaf(x.x, w, -a)));
            df_acc(sum[1], low[1], b, fmaf(x.w, w, fmaf(x.z, w, -b)));
        }
        float2 g = make_float2(sum[0] + low[0], sum[1] + low[1]);
        const double e = o == threadIdx.x ? e0 : __ldcg(extra + 2 * o), f = o == threadIdx.x ? f0 : __ldcg(extra + 2 * o + 1);
        if (not_zero(e) || not_zero(f)) {   /* not finite */
            g = make_float2((float)((double)g.x + e), (float)((double)g.y + f));
            extra[2 * o] = extra[2 * o + 1] = 0.0;
        }
        reinterpret_cast<float2 *>(P.pulse)[o] = g;
    }
    if (threadIdx.x == 0) *P.counter = 0u;
}

/* The block's node sums into the grid's accumulator, and the gates. */
template <int MODE>
__device__ __forceinline__ void node_finish(const PulseArgs &P, double *bins, unsigned nblk) {
    if (MODE == 0) {
        const unsigned nodes = node_count(P.G, P.mom_n);
        __syncthreads();
        for (unsigned o = threadIdx.x; o < nodes * 4; o += blockDim.x) {
            const double v = bins[o];
            if (not_zero(v)) red_add(P.acc64 + o, wide_scaled(v));
        }
    }
    node_gates<MODE, true>(P, bins, nblk);
}

/* A run of 64 into the warp's window. */
__device__ __forceinline__ void node_run(const PulseArgs &P, NodeWindow &W, const float4 *p, const float4 *x, unsigned in,
                                         int part, double *bins, double *stray, unsigned lane) {
    Sig g[2];
    bool held[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        if (!signal_plain_mid(P, p[q], x[q], g[q])) {
            Sig32 sg;
            signal_plain(P, p[q], x[q], sg);
            g[q].r = sg.r;
#pragma unroll
            for (int l = 0; l < 4; l++) g[q].s[l] = sg.s.v[l];
        }
        /* NaN or an infinity in any lane makes the sum NaN */
        const float f = fmaf(g[q].s[0], 0.0f, fmaf(g[q].s[1], 0.0f, fmaf(g[q].s[2], 0.0f, g[q].s[3] * 0.0f)));
        held[q] = W.holds(g[q].r) && f == 0.0f;
    }
    if (__all_sync(0xffffffffu, held[0] && held[1])) {
        W.add(g[0]);
        W.add(g[1]);
    } else if (__popc(__ballot_sync(0xffffffffu, held[0])) + __popc(__ballot_sync(0xffffffffu, held[1])) >=
               kNodeMost) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (held[q]) W.add(g[q]);
            else if ((in >> q) & 1u) node_alone(P, g[q], stray);
        }
    } else {
        node_settle(P, W, g, in, part, bins, stray, lane);
    }
}
/* A beam and wave number whose terms are finite for every scatterer that
 * comp_run may skip: |b| of 2^-20 to 2^20, |k| below 2^12 (a phase below 2^32).
 * NaN and infinities are neither. */
__device__ __forceinline__ bool comp_tame(const PulseArgs &P) {
    const float *sd = P.sim;
    return fabsf(sd[0]) < 0x1p20f && fabsf(sd[1]) < 0x1p20f && fabsf(sd[2]) < 0x1p20f && fabsf(sd[4]) < 0x1p12f &&
           P.ib2_hi < 0x1p40f;
}

__device__ __forceinline__ void comp_run(const PulseArgs &P, CompWindow &W, const float4 *p, const float4 *x, unsigned in,
                                         int part, bool tame, unsigned lane) {
    /* nothing to do when no scatterer of the run reaches a gate and none has
     * a term that is not finite, which would reach all of them: backscatter
     * below 2^30 (2^98 times it is finite), ranges of 2^-10 to 2^20 m, and a
     * pulse that comp_tame */
    bool live = !tame;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const float r2 = fmaf(p[q].x, p[q].x, fmaf(p[q].y, p[q].y, p[q].z * p[q].z));
        const float f = fmaf(x[q].x, 0x1p98f, fmaf(x[q].y, 0x1p98f, fmaf(x[q].z, 0x1p98f, x[q].w * 0x1p98f)));
        live = live || !(fabsf(f) < INFINITY && ((r2 > 0x1p-20f && r2 < P.reach_lo2) || (r2 > P.reach_hi2 && r2 < 0x1p40f)));
    }
    if (!__any_sync(0xffffffffu, live)) return;
    CompSig g[2];
    float th[2], tl[2];
    bool held[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        signal_comp_any(P, p[q], x[q], g[q]);
        /* NaN or an infinity in any lane makes the sum NaN (a tail is finite
         * where its head is) */
        const float f = fmaf(g[q].s[0], 0.0f, fmaf(g[q].s[1], 0.0f, fmaf(g[q].s[2], 0.0f, g[q].s[3] * 0.0f)));
        W.offset(g[q], th[q], tl[q]);
        const float t = th[q] + tl[q];
        held[q] = t >= -P.rdelta && t < P.rdelta && f == 0.0f;
    }
    if (__popc(__ballot_sync(0xffffffffu, held[0])) + __popc(__ballot_sync(0xffffffffu, held[1])) >= kNodeMost) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (held[q]) {
                W.add(g[q], th[q], tl[q]);
            } else if ((in >> q) & 1u) {
                bool live = true;
                if (!(fabsf(g[q].r) < INFINITY) || !finite4(g[q].s) || !finite4(g[q].u)) live = comp_non_finite(P, g[q]);
                const int j = live ? comp_interval(P, g[q].r) : -1;
                if (j >= 0) comp_stray(P, j, g[q]);
            }
        }
    } else {
        comp_settle(P, W, g, in, part, lane);
    }
}

template <int MODE>   /* RSC_PULSE_PLAIN, RSC_PULSE_COMPENSATED */
__device__ __forceinline__ void node_body(const PulseArgs &P, unsigned blk, unsigned nblk) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *bins = reinterpret_cast<double *>(smem_raw);
    const unsigned nodes = node_count(P.G, P.mom_n);
    double *stray = P.stray + (size_t)4 * nodes * (blk & (node_copies(P.G, P.mom_n) - 1u));
    if (MODE == 0) {
        for (unsigned o = threadIdx.x; o < nodes * 4; o += blockDim.x) bins[o] = 0.0;
        __syncthreads();
    }
    const unsigned lane = threadIdx.x & 31u;
    const unsigned long long n = P.n, runs = (n + 63ull) / 64ull, whole = n / 64ull;
    const unsigned long long warps = (unsigned long long)nblk * (blockDim.x >> 5);
    const unsigned long long me = (unsigned long long)blk * (blockDim.x >> 5) + (threadIdx.x >> 5);
    /* a contiguous piece of the runs in spatial order, and every warps-th of
     * the others, which cost more each */
    const unsigned long long lead = P.lead / 64ull;
    const unsigned long long last = lead * (me + 1) / warps;
    NodeWindow W;
    CompWindow C;
    if (MODE == 0) {
        W.c = -1;
        W.E0 = W.E1 = W.E2 = NAN;
        W.i0 = W.i1 = 0.0f;
        W.clear();
    } else {
        C.move(P, 0);
        C.c = -1;
        C.Eh = NAN;
    }
    const bool tame = MODE == 1 && comp_tame(P);
    const auto next = [&](unsigned long long r) {
        r++;
        return r == last ? lead + me : (r > last ? r + (warps - 1) : r);
    };
    unsigned long long run = lead * me / warps;
    if (run == last) run = lead + me;
    for (; run < runs; run = next(run)) {
        const float4 *pp = P.pos + run * 64ull + lane, *xx = P.rcs + run * 64ull + lane;
        float4 p[2], x[2];
        unsigned in = 3u;
        if (run < whole) {
            p[0] = __ldg(pp);
            p[1] = __ldg(pp + 32);
            x[0] = __ldg(xx);
            x[1] = __ldg(xx + 32);
        } else {
            /* past the end: the last scatterer with no backscatter */
            const unsigned left = (unsigned)(n - run * 64ull);
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const bool past = lane + 32u * q >= left;
                p[q] = __ldg(past ? P.pos + (n - 1) : pp + 32 * q);
                x[q] = past ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : __ldg(xx + 32 * q);
                if (past) in &= ~(1u << q);
            }
        }
        const int part = run < lead ? kNodePart : kNodeMost;
        if constexpr (MODE == 0) {
            node_run(P, W, p, x, in, part, bins, stray, lane);
        } else {
            comp_run(P, C, p, x, in, part, tame, lane);
        }
    }
    if (MODE == 0) W.flush(bins, lane);
    else C.flush(P, lane);
    node_finish<MODE>(P, bins, nblk);
}

__global__ void __launch_bounds__(kNodeThreads, kNodeMinBlocks) k_pulse_nodes(const PulseArgs P) {
    node_body<0>(P, blockIdx.x, gridDim.x);
}

__global__ void __launch_bounds__(kNodeThreads, kCompMinBlocks) k_pulse_nodes_comp(const PulseArgs P) {
    node_body<1>(P, blockIdx.x, gridDim.x);
}

/* ---- the plain form on a state in the caller's order ----
 * No run lies together, so every scatterer goes to its two nodes by itself: 8
 * additions to the warp's own node sums in shared memory, lane l's node next
 * to the next lane's.  Bound by those additions (compare and swap, lane after
 * lane where they meet), so fewer is faster: the gates' own sums take 4 for
 * each gate a scatterer reaches, or a visit to every gate when the gate window
 * does not hold them.  2,000,000 scatterers: n = 2 59 -> 41 us, n = 4 126 (as
 * reductions in L2, which meet in a few addresses) -> 41; 300,000 from the
 * caller's own buffers, n = 4 100 -> 27.  With 3 and 2 blocks per SM 43 and 56
 * instead of 41. */
__host__ __device__ __forceinline__ size_t node_any_smem_bytes(unsigned G, int n, int warps) {
    const size_t own = (size_t)node_count(G, n) * (1 + 4 * (size_t)warps) * sizeof(float), last = node_smem_bytes(G, n, false);
    return own > last ? own : last;   /* the last block's sums of the nodes take the place of the warps' */
}
/* ... while 4 blocks fit an SM with it. */
constexpr size_t kNodeAnyMost = 54 * 1024;
/* Narrower triangles reach two gates, whose own sums are as few (2,000,000:
 * 41.5 us on the nodes, 41.3 there; 30,000: 10.5, 8.7). */
constexpr int kNodeAnyLeast = 2;

__device__ __forceinline__ void node_any_add(const PulseArgs &P, const float *E, int last, float *mine, unsigned nodes,
                                             const float4 &p, const float4 &x) {
    Sig g;
    if (!signal_plain_mid(P, p, x, g)) {
        Sig32 sg;
        signal_plain(P, p, x, sg);
        g.r = sg.r;
#pragma unroll
        for (int l = 0; l < 4; l++) g.s[l] = sg.s.v[l];
    }
    if (!sig_finite(g)) {
        node_non_finite(P, g.r, g.s[0], g.s[1], g.s[2], g.s[3]);
        return;
    }
    /* node_interval and node_stray, on the nodes in shared memory */
    const float jf = floorf((g.r - E[0]) * P.inv_delta);
    if (!(jf >= -1.0f && jf <= (float)(last + 1))) return;
    int j = min(max((int)jf, 0), last);
    if (g.r < E[j]) j--;
    else if (g.r >= E[j + 1]) j++;
    if (j < 0 || j > last) return;
    const float a = E[j], b = E[j + 1], i = 1.0f / (b - a);
    const float wa = (b - g.r) * i, wb = (g.r - a) * i;
#pragma unroll
    for (int l = 0; l < 4; l++) {
        float *o = mine + (size_t)l * nodes + j;
        atomicAdd(o, wa * g.s[l]);
        atomicAdd(o + 1, wb * g.s[l]);
    }
}

__global__ void __launch_bounds__(kNodeThreads, kNodeMinBlocks) k_pulse_nodes_any(const PulseArgs P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const unsigned nodes = node_count(P.G, P.mom_n), nwarps = blockDim.x >> 5, warp = threadIdx.x >> 5;
    const unsigned lane = threadIdx.x & 31u;
    float *E = reinterpret_cast<float *>(smem_raw), *sums = E + nodes, *mine = sums + (size_t)warp * 4 * nodes;
    for (unsigned o = threadIdx.x; o < nodes; o += blockDim.x) E[o] = __ldg(P.node + o);
    for (unsigned o = threadIdx.x; o < nwarps * 4 * nodes; o += blockDim.x) sums[o] = 0.0f;
    __syncthreads();
    const int last = (int)nodes - 2;
    const unsigned long long n = P.n, stride = (unsigned long long)gridDim.x * blockDim.x * 2ull;
    for (unsigned long long base = ((unsigned long long)blockIdx.x * nwarps + warp) * 64ull + lane; base < n; base += stride) {
        const bool two = base + 32ull < n;
        const float4 p0 = __ldg(P.pos + base), x0 = __ldg(P.rcs + base);
        float4 p1 = p0, x1 = x0;
        if (two) {
            p1 = __ldg(P.pos + base + 32);
            x1 = __ldg(P.rcs + base + 32);
        }
        node_any_add(P, E, last, mine, nodes, p0, x0);
        if (two) node_any_add(P, E, last, mine, nodes, p1, x1);
    }
    __syncthreads();
    for (unsigned o = threadIdx.x; o < nodes * 4; o += blockDim.x) {
        const unsigned at = (o & 3u) * nodes + (o >> 2);
        float v = 0.0f;
        for (unsigned w = 0; w < nwarps; w++) v = v + sums[(size_t)w * 4 * nodes + at];
        if (v != 0.0f) red_add(P.acc64 + o, wide_of<true>(v));
    }
    node_gates<0, false>(P, reinterpret_cast<double *>(smem_raw), gridDim.x);
}

}  // namespace rsc

#endif

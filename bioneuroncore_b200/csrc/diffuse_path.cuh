// diffuse_path.cuh -- step 2.5 for networks whose components are unbranched (a soma with
// one dendrite and one axon, plain cables, single segments); included by diffuse.cu.
//
// A component's segments in path order couple only to the slots before and after them,
// so a warp holds 32 x R consecutive slots (whole components end to end, R per lane): the
// potentials and the solves' stencils in registers, the ions in the warp's own rows of
// shared memory, a neighbour's value a register, a shuffle or a row entry away.  No CTA
// barrier, no incidence lists.  What bounds it is instruction issue and, behind it,
// instruction fetch (71% of issue slots at 24 warps per SM and 1.28M segments, 44% in the
// form for few warps at 55k): about 8,600 lane slots of instructions per segment and tick,
// a third of them V_m sweeps at 7 FP32 instructions and 2 / R shuffles, where the CTA-tile
// kernel runs 27,000 (a sweep there is about 32: shared loads and a store, a barrier, range
// checks).  So loops over ions and sweeps stay rolled: unrolled,
// 1.28M segments of 64-segment neurons took 502-548 us.
// Measured, step 2.5 per tick, this kernel against the CTA-tile kernel: 1.28M segments
// (64 per neuron) 459 us against 1,198; 55k (37 per neuron) 66 against 128; 2,048 (32 per
// neuron) 34 against 116; an uneven ensemble of 418k 169 against 451.
//
// The arithmetic is k_diffusion's, bit for bit:
//  * a segment has at most two connections, and a sum of two terms is the same in either
//    order; only the phi_e diagonal has three terms, and keeps connection order (bit 31
//    of pt_seg);
//  * a connection is taken from slot to next slot whatever its stored direction: with its
//    ends exchanged the potential difference and every flux change sign exactly;
//  * a Jacobi sweep maps an iterate to the next one, so once a sweep returns its iterate
//    unchanged in every bit, the remaining sweeps of the 50 would too and are not run;
//  * (float)(0.5 (double)a + ...) of two floats, and a float plus a float rounded through
//    double, are the float operations (the double keeps 2 x 24 + 2 bits);
//  * ion 5 has diffusion coefficient 0: its fluxes are zeros unless a concentration or its
//    product with a Bernoulli value is not finite;
//  * divisions by a value used many times are Markstein's correction of a * (1 / b)
//    (div_rn_f), their range conditions checked once per solve or sub-step instead of
//    per division.  Warps with a value outside them take the kSafe code, which divides.

// z^2 D and z * 96.485 per ion, as the products evaluate in float; and which of the rows
// PathRows::b holds an ion's Bernoulli values at -z x and z x
__constant__ float kZ2D[7] = {1.0f * 1.0f * 1.33f, 1.0f * 1.0f * 1.96f, 2.0f * 2.0f * 0.22f, -1.0f * -1.0f * 2.03f,
                              2.0f * 2.0f * 0.10f, -1.0f * -1.0f * 0.0f, 1.0f * 1.0f * 9.31f};
__constant__ float kZF[7] = {1.0f * 96.485f, 1.0f * 96.485f, 2.0f * 96.485f, -1.0f * 96.485f,
                             2.0f * 96.485f, -1.0f * 96.485f, 1.0f * 96.485f};
__constant__ int kBm[7] = {0, 0, 2, 1, 2, 1, 0};
__constant__ int kBp[7] = {1, 1, 3, 0, 3, 0, 1};

// Values of the lanes holding the slots before and after this lane's.  The warp's last
// slot has no connection to a next one, so the rotation's wrapped values are never used.
template <typename T> __device__ __forceinline__ T from_prev(T v) {
    return __shfl_sync(0xFFFFFFFFu, v, (int)((threadIdx.x + 31u) & 31u));
}
template <typename T> __device__ __forceinline__ T from_next(T v) {
    return __shfl_sync(0xFFFFFFFFu, v, (int)((threadIdx.x + 1u) & 31u));
}

// sg_bernoulli at -x, x, -2x and 2x.  The warp takes the cheapest form that serves all its
// connections: all arguments in the linear range; all where the exponential needs no
// argument reduction; all within 50, where it needs the reduction but none of dm_exp's
// range checks; else the general function.
__device__ __forceinline__ float bernoulli_of(float v, double e, float linear) {
    const float r = (float)((double)v / (e - 1.0));
    return fabsf(v) < 1e-3f ? linear : r;
}
__device__ __noinline__ float path_bernoulli_any(float v) { return sg_bernoulli(v); }

// One warp's rows in shared memory, each a value per slot: what a sub-step touches once is
// kept here, so that registers (80 a thread) allow 24 warps per SM.  A lane reads its own
// slots and, after a __syncwarp, its neighbours'.  The two extra words let the warp's last
// slot read a next one (never used: it has no connection).
template <int R>
struct __align__(16) PathRows {
    float in[7][32 * R];
    float out[7][32 * R];
    float coef[7][32 * R];   // D area dt_sub / length of the connection to the next slot
    float f[7][32 * R];      // its fluxes
    float b[4][32 * R];      // its Bernoulli values at -x, x, -2x, 2x
    float pad[4];
};

template <int R> __device__ __forceinline__ void row_get(const float* row, uint32_t l, float (&x)[R]) {
    if constexpr (R == 2) {
        const float2 v = reinterpret_cast<const float2*>(row)[l];
        x[0] = v.x; x[1] = v.y;
    } else if constexpr (R == 4) {
        const float4 v = reinterpret_cast<const float4*>(row)[l];
        x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    } else {
#pragma unroll
        for (int s = 0; s < R; s++) x[s] = row[l * R + s];
    }
}
template <int R> __device__ __forceinline__ void row_put(float* row, uint32_t l, const float (&x)[R]) {
    if constexpr (R == 2) reinterpret_cast<float2*>(row)[l] = make_float2(x[0], x[1]);
    else if constexpr (R == 4) reinterpret_cast<float4*>(row)[l] = make_float4(x[0], x[1], x[2], x[3]);
    else
#pragma unroll
        for (int s = 0; s < R; s++) row[l * R + s] = x[s];
}
// the value before this lane's first slot (lane 0: 0)
template <int R> __device__ __forceinline__ float row_prev(const float* row, uint32_t l) {
    return l ? row[l * R - 1] : 0.0f;
}

template <int R>
__device__ __forceinline__ void bernoulli_four(const float (&x)[R], PathRows<R>& p, uint32_t l) {
    float m = 0.0f;
    bool num = true;
#pragma unroll
    for (int s = 0; s < R; s++) {
        m = fmaxf(m, fabsf(x[s]));
        num &= x[s] == x[s];
    }
    const float m2 = num ? 2.0f * m : 1e30f;
    const bool lin = __all_sync(0xFFFFFFFFu, m2 < 1e-3f), small = __all_sync(0xFFFFFFFFu, m2 < 0.34f),
               mid = __all_sync(0xFFFFFFFFu, m2 < 50.0f);
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
        float bm[R], bp[R];
#pragma unroll
        for (int s = 0; s < R; s++) {
            const float v = k ? 2.0f * x[s] : x[s];
            bm[s] = 1.0f - 0.5f * -v;
            bp[s] = 1.0f - 0.5f * v;
        }
        if (small) {
            if (!lin) {
#pragma unroll
                for (int s = 0; s < R; s++) {
                    const float v = k ? 2.0f * x[s] : x[s];
                    bm[s] = bernoulli_of(-v, dm_exp_taylor((double)-v), bm[s]);
                    bp[s] = bernoulli_of(v, dm_exp_taylor((double)v), bp[s]);
                }
            }
        } else if (mid) {
#pragma unroll
            for (int s = 0; s < R; s++) {
                const float v = k ? 2.0f * x[s] : x[s];
                bm[s] = bernoulli_of(-v, dm_exp_mid((double)-v), bm[s]);
                bp[s] = bernoulli_of(v, dm_exp_mid((double)v), bp[s]);
            }
        } else {
#pragma unroll
            for (int s = 0; s < R; s++) {
                const float v = k ? 2.0f * x[s] : x[s];
                bm[s] = path_bernoulli_any(-v);
                bp[s] = path_bernoulli_any(v);
            }
        }
        row_put<R>(p.b[2 * k], l, bm);
        row_put<R>(p.b[2 * k + 1], l, bp);
    }
}

// x over vf (rounded as the division, for a finite x; see div_by_float), given yv = 1 / vf
__device__ __forceinline__ double over(double x, double vf, double yv) {
    const double q0 = x * yv;
    return __fma_rn(__fma_rn(-q0, vf, x), yv, q0);
}

// The ions' fluxes of one intracellular sub-step (rows f, zero where there is no
// connection) applied (diffusion_kernel.h:152-238); ie: each connection's Nernst-Planck
// current.  kSafe: divide, and handle ion 5.
template <int R, bool kSafe, int kUQ>
__device__ __forceinline__ void path_apply_intra(PathRows<R>& p, uint32_t l, const bool (&has)[R], bool hasL0,
                                                 const float (&vf)[R], float dt_sub, float ydts, float (&ie)[R]) {
#pragma unroll
    for (int s = 0; s < R; s++) ie[s] = 0.0f;
    double yv[R];
#pragma unroll
    for (int s = 0; s < R; s++) yv[s] = 1.0 / (double)vf[s];
#pragma unroll kUQ
    for (int q = 0; q < 7; q++) {
        if (!kSafe && q == 5) continue;
        float f[R], x[R];
        row_get<R>(p.f[q], l, f);
        row_get<R>(p.in[q], l, x);
        const float fprev = row_prev<R>(p.f[q], l);
#pragma unroll
        for (int s = 0; s < R; s++) {
            const float a = kZF[q] * f[s];
            const double fr = (double)f[s], fl = (double)(s ? f[s ? s - 1 : 0] : fprev);
            double acc;
            if (kSafe) {
                if (has[s]) ie[s] += a / dt_sub;
                acc = 0.0;
                if (s ? has[s ? s - 1 : 0] : hasL0) acc += fl / (double)vf[s];
                if (has[s]) acc -= fr / (double)vf[s];
            } else {
                const float q0 = a * ydts;
                ie[s] += __fmaf_rn(__fmaf_rn(-q0, dt_sub, a), ydts, q0);
                acc = over(fl, (double)vf[s], yv[s]) - over(fr, (double)vf[s], yv[s]);
            }
            x[s] = x[s] + (float)acc;
        }
        row_put<R>(p.in[q], l, x);
    }
}

// One extracellular sub-step (diffusion_kernel.h:244-281).  The extracellular volume is
// 0.25 vf exactly, so a flux over it is four times the flux over vf.
template <int R, bool kSafe, int kUQ>
__device__ __forceinline__ void path_extra(PathRows<R>& p, uint32_t l, const bool (&has)[R], bool hasL0,
                                           const float (&vf)[R], const double (&yv)[R]) {
#pragma unroll kUQ
    for (int q = 0; q < 7; q++) {
        if (!kSafe && q == 5) continue;
        float x[R], co[R], bm[R], bp[R];
        row_get<R>(p.b[kBm[q]], l, bm);
        row_get<R>(p.b[kBp[q]], l, bp);
        row_get<R>(p.out[q], l, x);
        row_get<R>(p.coef[q], l, co);
        const float nxt = p.out[q][l * R + R];
        double f[R], c[R + 1];
#pragma unroll
        for (int s = 0; s < R; s++) c[s] = (double)x[s];
        c[R] = (double)nxt;
#pragma unroll
        for (int s = 0; s < R; s++) {
            const double v = (double)co[s] * (c[s] * (double)bm[s] - c[s + 1] * (double)bp[s]);
            f[s] = has[s] ? v : 0.0;
        }
        const double fprev = from_prev(f[R - 1]);   // also orders the neighbours' reads before the update
#pragma unroll
        for (int s = 0; s < R; s++) {
            const double fr = f[s], fl = s ? f[s ? s - 1 : 0] : fprev;
            double acc;
            if (kSafe) {
                const double vx = (double)(vf[s] * EXTRA_VOLUME_RATIO);
                acc = 0.0;
                if (s ? has[s ? s - 1 : 0] : hasL0) acc += fl / vx;
                if (has[s]) acc -= fr / vx;
            } else {
                acc = 4.0 * (over(fl, (double)vf[s], yv[s]) - over(fr, (double)vf[s], yv[s]));
            }
            x[s] = (float)(c[s] + acc);
        }
        row_put<R>(p.out[q], l, x);
    }
}

// Fick pass of a float field (diffusion_kernel.h:284-345).
template <int R, bool kGradStrict>
__device__ __forceinline__ void path_fick(const float (&ear)[R], const float (&edi)[R], const bool (&has)[R],
                                          const float (&vf)[R], float (&x)[R], float D, float thresh, float dt) {
    const float nxt = from_next(x[0]);
    float fl[R];
    bool on[R];
#pragma unroll
    for (int s = 0; s < R; s++) {
        const float dC = x[s] - (s < R - 1 ? x[s < R - 1 ? s + 1 : s] : nxt);
        on[s] = has[s] && (kGradStrict ? (dC > thresh || dC < -thresh) : !(dC < thresh && dC > -thresh));
        fl[s] = on[s] ? D * ear[s] * dC * dt / edi[s] : 0.0f;
    }
    const float fprev = from_prev(fl[R - 1]);
    const bool onprev = from_prev((int)on[R - 1]) != 0;
#pragma unroll
    for (int s = 0; s < R; s++) {
        float acc = 0.0f;
        if (s ? on[s ? s - 1 : 0] : onprev) acc += (s ? fl[s ? s - 1 : 0] : fprev) / vf[s];
        if (on[s]) acc -= fl[s] / vf[s];
        x[s] = x[s] + acc;
    }
}

// R slots per lane; NetDev::pt_* hold the slots.  kFew: the network leaves most of the
// chip idle, so a warp's latency counts: loops over ions and sweeps unrolled.
template <int R, bool kFew>
__global__ void __launch_bounds__(64, kFew ? 8 : R == 2 ? 12 : 6)
k_diffusion_path(NetDev d, float dt, unsigned long long tick) {
    constexpr int kUQ = kFew ? 7 : 1, kUV = kFew ? 5 : 1;
    __shared__ PathRows<R> rows[2];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= d.n_pt) return;
    if (d.clock) tick = d.clock[0];
    PathRows<R>& p = rows[threadIdx.x >> 5];
    const size_t N = d.n_seg;
    const size_t slot0 = ((size_t)w * 32 + lane) * R;
    const unsigned full = 0xFFFFFFFFu;

    // ---- load: state after step 1, stimuli, statics ----
    uint32_t g[R];
    bool on[R], right_first[R], has[R];
    float ear[R], edi[R], V[R], atp[R], vf[R];
    double itot[R];
    {
        float in[7][R], out[7][R];
#pragma unroll
        for (int s = 0; s < R; s++) {
            const uint32_t ps = d.pt_seg[slot0 + s];
            on[s] = ps != UINT32_MAX;
            right_first[s] = (ps >> 31) != 0;
            g[s] = ps & 0x7FFFFFFFu;
            ear[s] = d.pt_area[slot0 + s];
            edi[s] = d.pt_dist[slot0 + s];
            has[s] = ear[s] > 0.0f;
            V[s] = atp[s] = 0.0f;
            vf[s] = 1.0f;
            itot[s] = 0.0;
#pragma unroll
            for (int q = 0; q < 7; q++) in[q][s] = out[q][s] = 0.0f;
            if (on[s]) {
                const float4* r4 = reinterpret_cast<const float4*>(d.rec + g[s]);
                const float4 a = r4[0], b = r4[1], c = r4[2], e = r4[3];
                V[s] = a.x; in[0][s] = a.y; in[1][s] = a.z; in[2][s] = a.w;
                in[3][s] = b.x; in[4][s] = b.y; in[5][s] = b.z; in[6][s] = b.w;
                out[0][s] = c.x; out[1][s] = c.y; out[2][s] = c.z; out[3][s] = c.w;
                out[4][s] = e.x; out[5][s] = e.y; out[6][s] = e.z; atp[s] = e.w;
                vf[s] = (float)d.rec[g[s]].vol;
                if (vf[s] < 1e-6f) vf[s] = 1e-6f;
                itot[s] = stimulus_current(d, g[s], d.rec[g[s]].itot, dt, tick);
                d.ibuf[g[s]] = itot[s];
            }
        }
#pragma unroll
        for (int q = 0; q < 7; q++) {
            row_put<R>(p.in[q], lane, in[q]);
            row_put<R>(p.out[q], lane, out[q]);
        }
    }
    const bool hasL0 = from_prev((int)has[R - 1]) != 0;

    if (d.flags & NF_DIFFUSION) {
        const float dt_sub = dt / 5;
        const float ydts = 1.0f / dt_sub;
        bool sane = fabsf(dt_sub) >= 0x1p-32f && fabsf(dt_sub) <= 0x1p32f;

        // ---- phi_e (diffusion_kernel.h:41-104) ----
        double phi[R];
        {
            double sig[R], gr[R], diag[R], yd[R];
#pragma unroll
            for (int s = 0; s < R; s++) phi[s] = sig[s] = 0.0;
#pragma unroll kUQ
            for (int q = 0; q < 7; q++) {
                float x[R];
                row_get<R>(p.out[q], lane, x);
#pragma unroll
                for (int s = 0; s < R; s++) {
                    sig[s] += kZ2D[q] * (double)x[s];
                    if (q == 5) sane &= fabsf(x[s]) < 1e20f;
                }
            }
#pragma unroll
            for (int s = 0; s < R; s++) sig[s] = 3.612f * sig[s];
            const double nxt = from_next(sig[0]);
#pragma unroll
            for (int s = 0; s < R; s++) {
                const double v = 0.5 * (sig[s] + (s < R - 1 ? sig[s < R - 1 ? s + 1 : s] : nxt)) * ear[s] / edi[s];
                gr[s] = has[s] ? v : 0.0;
            }
            const double gl0 = from_prev(gr[R - 1]);
            bool live[R], dok[R], hl[R], hr[R];
#pragma unroll
            for (int s = 0; s < R; s++) {
                const double gl = s ? gr[s ? s - 1 : 0] : gl0;
                const float area = on[s] ? d.area[g[s]] : 1.0f;
                diag[s] = sig[s] * area / 1.0f;
                diag[s] = right_first[s] ? (diag[s] + gr[s]) + gl : (diag[s] + gl) + gr[s];
                live[s] = diag[s] > 1e-9;
                yd[s] = live[s] ? 1.0 / diag[s] : 1.0;
                dok[s] = diag[s] <= 0x1p500;
                hl[s] = gl > 0.0;
                hr[s] = gr[s] > 0.0;
            }
#pragma unroll 1
            for (int it = 0; it < 50; it++) {
                const double pprev = from_prev(phi[R - 1]), pnext = from_next(phi[0]);
                double nv[R];
                bool same = true;
#pragma unroll
                for (int s = 0; s < R; s++) {
                    const double gl = s ? gr[s ? s - 1 : 0] : gl0;
                    const double pl = s ? phi[s ? s - 1 : 0] : pprev, pr = s < R - 1 ? phi[s < R - 1 ? s + 1 : s] : pnext;
                    double pn = hl[s] ? 0.0 + gl * pl : 0.0;
                    pn = hr[s] ? pn + gr[s] * pr : pn;
                    const double a = pn - itot[s];
                    const double q0 = a * yd[s];
                    double v = __fma_rn(__fma_rn(-q0, diag[s], a), yd[s], q0);
                    // |q0| in [2^-500, 2^500) by its exponent field (and a zero dividend)
                    // make the corrected quotient exact
                    const uint32_t ex = ((uint32_t)__double2hiint(q0) & 0x7FFFFFFFu) - ((1023u - 500u) << 20);
                    if (!((ex < (1000u << 20) && dok[s]) || a == 0.0)) v = a / diag[s];
                    if (fabs(v) > 10.0) v = copysign(10.0, v);
                    if (!live[s]) v = 0.0;
                    nv[s] = v;
                    same &= __double_as_longlong(v) == __double_as_longlong(phi[s]);
                }
#pragma unroll
                for (int s = 0; s < R; s++) phi[s] = nv[s];
                if (__all_sync(full, same)) break;   // a fixed point: the other sweeps return it
            }
        }

        // Nernst-Planck flux coefficient of each connection and ion: kDiffC[q] * area *
        // dt_sub / dist, left to right, the same in every sub-step
        {
            float in5[R];
            row_get<R>(p.in[5], lane, in5);
#pragma unroll
            for (int s = 0; s < R; s++) sane &= vf[s] < 1e20f && fabsf(in5[s]) < 1e20f;
#pragma unroll 1
            for (int q = 0; q < 7; q++) {
                float co[R];
#pragma unroll
                for (int s = 0; s < R; s++) {
                    co[s] = kDiffC[q] * ear[s] * dt_sub / edi[s];
                    sane &= fabsf(co[s]) < 1e20f;
                }
                row_put<R>(p.coef[q], lane, co);
            }
        }
        sane = __all_sync(full, sane);

        // ---- intracellular Nernst-Planck, 5 sub-steps (diffusion_kernel.h:152-238) ----
        float cdt[R];
#pragma unroll
        for (int s = 0; s < R; s++) {
            const float cm = on[s] ? d.cm[g[s]] : 1.0f;
            cdt[s] = cm / dt_sub;
            if (cdt[s] < 1e-9f) cdt[s] = 1e-9f;
        }
#pragma unroll 1
        for (int sub = 0; sub < 5; sub++) {
            float gax[R], term[R];
            {
                float x[R], dve[R], sigma[R];
                {
                    double u[R];
#pragma unroll
                    for (int s = 0; s < R; s++) u[s] = (double)V[s] + phi[s];
                    const double unext = from_next(u[0]);
#pragma unroll
                    for (int s = 0; s < R; s++) {
                        dve[s] = (float)(u[s] - (s < R - 1 ? u[s < R - 1 ? s + 1 : s] : unext));
                        x[s] = has[s] ? 0.03742f * dve[s] : 0.0f;
                        sigma[s] = 0.0f;
                    }
                }
                bernoulli_four<R>(x, p, lane);
                __syncwarp();   // the neighbours' concentrations of the last sub-step
                // lo: twice the bits of the smallest nonzero |flux|, less one (zero wraps to
                // the largest; its quotients are exact zeros)
                uint32_t lo = 0xFFFFFFFFu;
                float hi = 0.0f;
#pragma unroll kUQ
                for (int q = 0; q < 7; q++) {
                    float c[R], co[R], f[R], bm[R], bp[R];
                    row_get<R>(p.in[q], lane, c);
                    row_get<R>(p.coef[q], lane, co);
                    row_get<R>(p.b[kBm[q]], lane, bm);
                    row_get<R>(p.b[kBp[q]], lane, bp);
                    const float cn = p.in[q][lane * R + R];
#pragma unroll
                    for (int s = 0; s < R; s++) {
                        const float Cb = s < R - 1 ? c[s < R - 1 ? s + 1 : s] : cn;
                        sigma[s] += kZ2D[q] * (0.5f * (c[s] + Cb));
                        const float v = co[s] * (c[s] * bm[s] - Cb * bp[s]);
                        f[s] = has[s] ? v : 0.0f;
                        if (q != 5) {
                            lo = min(lo, 2u * __float_as_uint(f[s]) - 1u);
                            hi = fmaxf(hi, fabsf(f[s]));
                        }
                    }
                    row_put<R>(p.f[q], lane, f);
                }
                // every flux far from under- and overflow, so the corrected quotients are exact
                bool ok = sane && lo >= 2u * 0x12800000u - 1u && hi <= 0x1p90f;   // 0x12800000: 2^-90
#pragma unroll
                for (int s = 0; s < R; s++) {
                    const float gv = 3.612f * sigma[s] * ear[s] / edi[s];
                    gax[s] = has[s] ? gv : 0.0f;
                    ok &= !has[s] || fabsf(dve[s]) < 1e18f;   // x times a concentration below 1e20 stays finite
                }
                ok = __all_sync(full, ok);
                __syncwarp();   // the neighbours' fluxes
                float ie[R];
                if (ok) path_apply_intra<R, false, kUQ>(p, lane, has, hasL0, vf, dt_sub, ydts, ie);
                else path_apply_intra<R, true, 1>(p, lane, has, hasL0, vf, dt_sub, ydts, ie);
#pragma unroll
                for (int s = 0; s < R; s++) term[s] = has[s] ? ie[s] - gax[s] * dve[s] : 0.0f;
            }
            // V_m: 50 Jacobi sweeps
            const float tprev = from_prev(term[R - 1]), gl0 = from_prev(gax[R - 1]);
            float rhs[R], den[R], yden[R];
            bool ok = true;
#pragma unroll
            for (int s = 0; s < R; s++) {
                const float gl = s ? gax[s ? s - 1 : 0] : gl0;
                float inp = 0.0f;
                inp += term[s];
                inp -= s ? term[s ? s - 1 : 0] : tprev;
                rhs[s] = cdt[s] * V[s] + inp;
                den[s] = cdt[s] + (gl + gax[s]);
                yden[s] = 1.0f / den[s];
                // Iterates stay within the largest |V_m| and |rhs| / C_dt (the diagonal
                // dominates), and rhs + off is 0 or above 2^-85: the quotients are exact.
                ok &= gl >= 0.0f && gax[s] >= 0.0f && den[s] >= 0x1p-32f && den[s] <= 0x1p32f &&
                      fabsf(V[s]) <= 0x1p60f && fabsf(rhs[s]) <= 0x1p60f && (fabsf(rhs[s]) >= 0x1p-60f || !on[s]);
            }
            if (__all_sync(full, ok)) {
                auto sweep = [&](const float (&v)[R], float (&nv)[R]) {
                    const float vprev = from_prev(v[R - 1]), vnext = from_next(v[0]);
#pragma unroll
                    for (int s = 0; s < R; s++) {
                        const float a = rhs[s] + ((s ? gax[s ? s - 1 : 0] : gl0) * (s ? v[s ? s - 1 : 0] : vprev) +
                                                  gax[s] * (s < R - 1 ? v[s < R - 1 ? s + 1 : s] : vnext));
                        const float q0 = a * yden[s];
                        nv[s] = __fmaf_rn(__fmaf_rn(-q0, den[s], a), yden[s], q0);
                    }
                };
#pragma unroll 1
                for (int it = 0; it < 50; it += 10) {
                    float nv[R];
#pragma unroll kUV
                    for (int k = 0; k < 5; k++) {
                        sweep(V, nv);
                        sweep(nv, V);
                    }
                    bool same = true;   // the last sweep returned its iterate: a fixed point
#pragma unroll
                    for (int s = 0; s < R; s++) same &= __float_as_uint(nv[s]) == __float_as_uint(V[s]);
                    if (__all_sync(full, same)) break;
                }
            } else {
#pragma unroll 1
                for (int it = 0; it < 50; it++) {
                    const float vprev = from_prev(V[R - 1]), vnext = from_next(V[0]);
                    float nv[R];
#pragma unroll
                    for (int s = 0; s < R; s++) {
                        float off = 0.0f;
                        if (s ? has[s ? s - 1 : 0] : hasL0)
                            off += (s ? gax[s ? s - 1 : 0] : gl0) * (s ? V[s ? s - 1 : 0] : vprev);
                        if (has[s]) off += gax[s] * (s < R - 1 ? V[s < R - 1 ? s + 1 : s] : vnext);
                        nv[s] = (rhs[s] + off) / den[s];
                    }
#pragma unroll
                    for (int s = 0; s < R; s++) V[s] = nv[s];
                }
            }
        }

        // ---- extracellular Nernst-Planck, 5 sub-steps (diffusion_kernel.h:244-281);
        // phi_e and so each connection's Bernoulli values are fixed for the tick ----
        {
            float x[R];
            double yv[R];
            const double pnext = from_next(phi[0]);
            bool fin = sane;
#pragma unroll
            for (int s = 0; s < R; s++) {
                const double dphi = phi[s] - (s < R - 1 ? phi[s < R - 1 ? s + 1 : s] : pnext);
                x[s] = has[s] ? (float)(0.03742f * dphi) : 0.0f;
                fin &= fabsf(x[s]) < 1e3f;
                yv[s] = 1.0 / (double)vf[s];
            }
            bernoulli_four<R>(x, p, lane);
#pragma unroll 1
            for (int sub = 0; sub < 5; sub++) {
                bool ok = fin;
#pragma unroll 1
                for (int q = 0; q < 7; q++) {
                    if (q == 5) continue;
                    float c[R];
                    row_get<R>(p.out[q], lane, c);
#pragma unroll
                    for (int s = 0; s < R; s++) ok &= !(fabsf(c[s]) >= 1e20f);
                }
                __syncwarp();
                if (__all_sync(full, ok)) path_extra<R, false, kUQ>(p, lane, has, hasL0, vf, yv);
                else path_extra<R, true, 1>(p, lane, has, hasL0, vf, yv);
            }
        }

        // ---- NT / ATP / heat / transcription (diffusion_kernel.h:284-363) ----
        auto field = [&](float* base, float D, float thresh, auto strict) {
            float x[R];
#pragma unroll
            for (int s = 0; s < R; s++) x[s] = on[s] ? base[g[s]] : 0.0f;
            path_fick<R, decltype(strict)::value>(ear, edi, has, vf, x, D, thresh, dt);
#pragma unroll
            for (int s = 0; s < R; s++)
                if (on[s]) base[g[s]] = x[s];
        };
        if (d.flags & NF_INTRA_NT)
            for (int nt = 0; nt < 15; nt++) field(d.intra_nt + nt * N, gNtD[nt], 1e-12f, std::false_type());
        if (d.flags & NF_NT_DIFFUSE_OUT)
            for (int nt = 0; nt < 15; nt++) field(d.nt + nt * N, gNtD[nt], 1e-12f, std::false_type());
        path_fick<R, true>(ear, edi, has, vf, atp, 0.14f, 1e-12f, dt);
        if (d.flags & NF_TEMP) field(d.temp, 0.0014f, 0.001f, std::true_type());
        if (d.flags & NF_TXN) field(d.txn, 0.01f, 1e-9f, std::true_type());
    }

    // ---- bath relaxation and clamp, write back ----
    const bool bath = (d.flags & NF_DIFFUSION) != 0;
#pragma unroll 1
    for (int q = 0; q < 7; q++) {
        float x[R], y[R];
        row_get<R>(p.in[q], lane, x);
        row_get<R>(p.out[q], lane, y);
#pragma unroll
        for (int s = 0; s < R; s++) {
            if (bath) {
                double e = (double)y[s];
                e += (kBathIon[q] - e) * dt / 1.0f;
                if (e < 1e-9) e = 1e-9;
                if (e > 1000.0) e = 1000.0;
                y[s] = (float)e;
            }
            if (on[s]) {
                d.ion_in[q * N + g[s]] = x[s];
                d.ion_out[q * N + g[s]] = y[s];
            }
        }
        row_put<R>(p.out[q], lane, y);
    }
#pragma unroll
    for (int s = 0; s < R; s++) {
        if (!on[s]) continue;
        const size_t k = g[s];
        const uint32_t o = lane * R + s;
        d.V[k] = V[s];
        d.atp[k] = atp[s];
        const float2 c21 = d.c21_cur[k];
        d.pre_rec[k] = make_float4(V[s], p.out[2][o], c21.x, c21.y);
        if (d.flags & NF_PRE_EXT) {
            d.pre_ext[k] = make_float4(p.in[0][o], p.in[1][o], p.in[2][o], p.out[0][o]);
            d.pre_ext2[k] = p.out[1][o];
        }
    }
}

static cudaError_t launch_diffusion_path(const NetDev& dev, uint32_t slots, float dt, unsigned long long tick,
                                         cudaStream_t stream) {
    const uint32_t blocks = (dev.n_pt + 1) / 2;   // two warps per CTA
    const bool few = dev.n_pt <= kPathFewWarps;
    if (slots == 1) k_diffusion_path<1, true><<<blocks, 64, 0, stream>>>(dev, dt, tick);
    else if (slots == 2 && few) k_diffusion_path<2, true><<<blocks, 64, 0, stream>>>(dev, dt, tick);
    else if (slots == 2) k_diffusion_path<2, false><<<blocks, 64, 0, stream>>>(dev, dt, tick);
    else k_diffusion_path<4, false><<<blocks, 64, 0, stream>>>(dev, dt, tick);
    return cudaGetLastError();
}

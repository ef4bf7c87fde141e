// diffuse_tree.cuh -- step 2.5 for networks whose components are trees of at most 2,048
// segments (branched dendrites), with the electrodiffusion options; included by diffuse.cu.
//
// One CTA per tile of whole components, two slots per thread (slots t and t + threads), so
// that the largest component needs no cluster: a sweep ends with a CTA barrier, where the
// 2-CTA cluster of k_diffusion<2> pays a cluster barrier, a copy of the ghosts through
// distributed shared memory and a second barrier (about 3,000 cycles a sweep).  Every
// connection belongs to its child's slot.  88 bytes of shared memory per slot: the two
// phi_e and V_m iterates, one ion side at a time (the other waits in the step-1 record or
// has been written back), the connections' fluxes.
//
// What bounds it: instruction issue of the one CTA an SM holds (57% of issue slots at
// 1,024 threads and 64 registers, with and without the options).  Step 2.5 per tick, against k_diffusion<2>: 74 trees of
// 2,047 segments 239 us against 456 (373 with one list of connections unpacked per use,
// 287 with the rows' addresses folded); 160 trees with the residual-controlled solves and
// the ledger 1,032 against 2,000.  Smaller trees with these options, few enough for one wave
// of the tile kernel, run that (options_on_tiles).
//
// The arithmetic is k_diffusion's: a connection runs from child to parent (with its ends
// exchanged, potential differences and fluxes change sign exactly), every sum keeps
// connection order; the remarks of diffuse_path.cuh on fixed points, corrected quotients
// and ion 5 hold here too.

// The rows of a tile of C slots in shared memory.  The connection rows have one more
// entry, kept zero: what a segment with fewer connections than the network's most reads
// in the missing ones' place.
template <int C>
struct __align__(16) TreeRows {
    double phiA[C], phiB[C];
    union {
        double fd[4][C + 2];      // FP64 connection fluxes
        struct {
            float f[7][C + 2];    // connection fluxes of the intracellular side
            float gax[C + 2], term[C + 2];
        };
    };
    float VA[C], VB[C];
    float c[7][C];                // the ions of one side
};

// sg_bernoulli at -x, x, -2x, 2x by the cheapest form that serves the warp (see
// bernoulli_four).
__device__ __forceinline__ void bernoulli_lane(float x, float (&b)[4]) {
    const float m2 = x == x ? 2.0f * fabsf(x) : 1e30f;
    const bool lin = __all_sync(0xFFFFFFFFu, m2 < 1e-3f), small = __all_sync(0xFFFFFFFFu, m2 < 0.34f),
               mid = __all_sync(0xFFFFFFFFu, m2 < 50.0f);
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float v = k ? 2.0f * x : x;
        float bm = 1.0f - 0.5f * -v, bp = 1.0f - 0.5f * v;
        if (small) {
            if (!lin) {
                bm = bernoulli_of(-v, dm_exp_taylor((double)-v), bm);
                bp = bernoulli_of(v, dm_exp_taylor((double)v), bp);
            }
        } else if (mid) {
            bm = bernoulli_of(-v, dm_exp_mid((double)-v), bm);
            bp = bernoulli_of(v, dm_exp_mid((double)v), bp);
        } else {
            bm = path_bernoulli_any(-v);
            bp = path_bernoulli_any(v);
        }
        b[2 * k] = bm;
        b[2 * k + 1] = bp;
    }
}

// One of a thread's two slots.  kInc: connections of a segment, at most.
template <int kInc>
struct TreeSlot {
    bool on, has;             // holds a segment; that segment has a connection to a parent
    uint32_t x, g, par;       // slot, device segment, the parent's slot (its own without one)
    // its connections in connection order: the other end (its own slot where there is
    // none) and the slot that owns the connection (this one for the connection to the
    // parent, the zero entry where there is none)
    uint32_t o[kInc], w[kInc];
    float vf, cdt, V;
};

// Runs one residual-controlled solve (see residual_solve) from wa; update(slot, w) returns a
// slot's new value.  Returns the buffer holding the result.
template <int kInc, typename F>
__device__ __forceinline__ const double* tree_residual(const NetDev& d, const TreeSlot<kInc> (&sl)[2], double* wa, double* wb,
                                                       unsigned* bits, F&& update, int slot) {
    const int tid = threadIdx.x, nth = blockDim.x;
    for (int k = tid; k < 128; k += nth) bits[k] = 0u;
    uint32_t grp[2];
    bool leader[2], done[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const uint32_t gw = sl[r].on ? d.tr_grp[sl[r].g] : 0u;
        grp[r] = gw & 0x7FFFu;
        leader[r] = (gw & 0x8000u) != 0u;
        done[r] = !sl[r].on;
    }
    uint32_t it = 0;
    __syncthreads();
    while (it < d.jac_max) {
        unsigned* cur = bits + (it & 1u) * 64;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            if (!sl[r].on) continue;
            double nv = wa[sl[r].x];
            if (!done[r]) {
                const double old = nv;
                nv = update(r, static_cast<const double*>(wa));
                if (fabs(nv - old) > d.jac_tol) atomicOr(&cur[grp[r] >> 5], 1u << (grp[r] & 31u));
            }
            wb[sl[r].x] = nv;
        }
        __syncthreads();
        bool more = false;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            if (done[r]) continue;
            if ((cur[grp[r] >> 5] >> (grp[r] & 31u)) & 1u) more = true;
            else done[r] = true;
        }
        for (int k = tid; k < 64; k += nth) bits[((it + 1) & 1u) * 64 + k] = 0u;
        it++;
        const bool any = __syncthreads_or(more) != 0;
        double* tmp = wa; wa = wb; wb = tmp;
        if (!any) break;
    }
#pragma unroll
    for (int r = 0; r < 2; r++)
        if (sl[r].on && leader[r] && !done[r]) atomicAdd(&d.jac_stats[2 + slot], 1u);
    if (tid == 0) atomicMax(&d.jac_stats[slot], it);
    return wa;
}

// Fick pass of a float field (diffusion_kernel.h:284-345); v: the field at the two slots.
template <int C, int kInc, bool kGradStrict>
__device__ __forceinline__ void tree_fick(const NetDev& d, TreeRows<C>& t, const TreeSlot<kInc> (&sl)[2], float (&v)[2],
                                          float D, float thresh, float dt) {
    __syncthreads();   // the last pass's readers
#pragma unroll
    for (int r = 0; r < 2; r++)
        if (sl[r].on) t.VA[sl[r].x] = v[r];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; r++) {
        if (!sl[r].has) continue;
        const float dC = v[r] - t.VA[sl[r].par];
        const bool on = kGradStrict ? (dC > thresh || dC < -thresh) : !(dC < thresh && dC > -thresh);
        t.f[0][sl[r].x] = on ? D * d.tr_area[sl[r].g] * dC * dt / d.tr_dist[sl[r].g] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; r++) {
        if (!sl[r].on) continue;
        float acc = 0.0f;
#pragma unroll
        for (int k = 0; k < kInc; k++) {
            const uint32_t w = sl[r].w[k];
            if (w == (uint32_t)C) continue;
            const float q = t.f[0][w] / sl[r].vf;
            if (w == sl[r].x) acc -= q; else acc += q;
        }
        v[r] = v[r] + acc;
    }
}

// kOpt: the options of NetDev::diff_mode compiled in.
template <int C, int kInc, bool kOpt>
__global__ void __launch_bounds__(C / 2, 2048 / C)
k_diffusion_tree(NetDev d, float dt, unsigned long long tick) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double sh_ledger[14];
    __shared__ unsigned sh_bits[128];
    if (threadIdx.x < 14) sh_ledger[threadIdx.x] = 0.0;
    TreeRows<C>& t = *reinterpret_cast<TreeRows<C>*>(smem);
    constexpr uint32_t nth = C / 2;
    const uint32_t tid = threadIdx.x;
    const size_t N = d.n_seg;
    const uint32_t s0 = d.tr_beg[blockIdx.x], ns = d.tr_beg[blockIdx.x + 1] - s0;
    if (d.clock) tick = d.clock[0];
    const float dt_sub = dt / 5;
    const float ydts = 1.0f / dt_sub;
    constexpr int kUQ = kOpt ? 1 : 7;
    const bool ledger = kOpt && (d.diff_mode & 2u) != 0u;

    // ---- load: state after step 1, stimuli, statics ----
    TreeSlot<kInc> sl[2];
    double itot[2];
    bool sane = fabsf(dt_sub) >= 0x1p-32f && fabsf(dt_sub) <= 0x1p32f;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        TreeSlot<kInc>& s = sl[r];
        s.x = tid + r * nth;
        s.on = s.x < ns;
        s.g = s0 + s.x;
        s.par = s.x;
        s.has = false;
#pragma unroll
        for (int k = 0; k < kInc; k++) { s.o[k] = s.on ? s.x : 0u; s.w[k] = C; }
        s.vf = s.cdt = 1.0f;
        s.V = 0.0f;
        itot[r] = 0.0;
        if (s.on) {
            const uint32_t pp = d.tr_par[s.g];
            s.has = pp != 0xFFFFu;
            if (s.has) s.par = pp;
            const uint2 oth = d.tr_oth[s.g];
#pragma unroll
            for (int k = 0; k < kInc; k++) {
                const uint32_t o = ((k < 2 ? oth.x : oth.y) >> (16 * (k & 1))) & 0xFFFFu;
                if (o == 0xFFFFu) continue;
                s.o[k] = o;
                s.w[k] = s.has && o == s.par ? s.x : o;
            }
            const SegRec* rec = d.rec + s.g;
            const float4* r4 = reinterpret_cast<const float4*>(rec);
            const float4 a = r4[0], b = r4[1];
            s.V = a.x;
            t.c[0][s.x] = a.y; t.c[1][s.x] = a.z; t.c[2][s.x] = a.w;
            t.c[3][s.x] = b.x; t.c[4][s.x] = b.y; t.c[5][s.x] = b.z; t.c[6][s.x] = b.w;
            s.vf = (float)rec->vol;
            if (s.vf < 1e-6f) s.vf = 1e-6f;
            const float cm = d.cm[s.g];
            s.cdt = cm / dt_sub;
            if (s.cdt < 1e-9f) s.cdt = 1e-9f;
            itot[r] = stimulus_current(d, s.g, rec->itot, dt, tick);
            d.ibuf[s.g] = itot[r];
            sane &= s.vf < 1e20f && fabsf(b.z) < 1e20f && fabsf(rec->out[5]) < 1e20f;
        }
    }

    if (tid < 4) t.fd[tid][C] = 0.0;   // the zero entries

    // ---- phi_e (diffusion_kernel.h:41-104) ----
    double* phi = t.phiA;
    {
        double* sig = t.phiB;
        double sg[2], yd[2], diag[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            double sacc = 0.0;
            if (sl[r].on) {
                const SegRec* rec = d.rec + sl[r].g;
#pragma unroll
                for (int q = 0; q < 7; q++) sacc += kZ2D[q] * (double)rec->out[q];
            }
            sg[r] = 3.612f * sacc;
            if (sl[r].on) sig[sl[r].x] = sg[r];
        }
        __syncthreads();
        double* ed = t.fd[0];
#pragma unroll
        for (int r = 0; r < 2; r++)
            if (sl[r].has) ed[sl[r].x] = 0.5 * (sg[r] + sig[sl[r].par]) * d.tr_area[sl[r].g] / d.tr_dist[sl[r].g];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 2; r++) {
            diag[r] = 0.0;
            yd[r] = 1.0;
            if (!sl[r].on) continue;
            diag[r] = sg[r] * d.area[sl[r].g] / 1.0f;
#pragma unroll
            for (int k = 0; k < kInc; k++) diag[r] += ed[sl[r].w[k]];
            if (diag[r] > 1e-9) yd[r] = 1.0 / diag[r];
            t.phiA[sl[r].x] = 0.0;
        }
        __syncthreads();
        auto update = [&](int r, const double* w) {
            double pn = 0.0;
#pragma unroll
            for (int k = 0; k < kInc; k++) {
                const double g = ed[sl[r].w[k]];
                const double p = pn + g * w[sl[r].o[k]];
                pn = g > 0.0 ? p : pn;
            }
            double v = diag[r] > 1e-9 ? div_rn_d(pn - itot[r], diag[r], yd[r]) : 0.0;
            if (v > 10.0) v = 10.0;
            if (v < -10.0) v = -10.0;
            return v;
        };
        if (kOpt && (d.diff_mode & 1u)) {
            phi = const_cast<double*>(tree_residual(d, sl, t.phiA, t.phiB, sh_bits, update, 1));
        } else {
            double* pn = t.phiB;
            for (int it = 0; it < 50; it++) {
                bool same = true;
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    if (!sl[r].on) continue;
                    const double v = update(r, phi);
                    same &= __double_as_longlong(v) == __double_as_longlong(phi[sl[r].x]);
                    pn[sl[r].x] = v;
                }
                const bool fixed = __syncthreads_and(same) != 0;
                double* tmp = phi; phi = pn; pn = tmp;
                if (fixed) break;   // the other sweeps return the same iterate
            }
        }
    }

    // ---- intracellular Nernst-Planck, 5 sub-steps (diffusion_kernel.h:152-238) ----
#pragma unroll
    for (int r = 0; r < 2; r++)
        if (sl[r].on) t.VA[sl[r].x] = sl[r].V;   // VA holds V_m as a sub-step begins
    if (tid < 9) (tid < 7 ? t.f[tid] : tid == 7 ? t.gax : t.term)[C] = 0.0f;
    __syncthreads();
#pragma unroll 1
    for (int sub = 0; sub < 5; sub++) {
        bool ok = sane;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const TreeSlot<kInc>& s = sl[r];
            const float area = s.has ? d.tr_area[s.g] : 0.0f, dist = s.has ? d.tr_dist[s.g] : 1.0f, rdist = 1.0f / dist;
            float dve = 0.0f;
            if (s.has) dve = (float)(((double)s.V + phi[s.x]) - ((double)t.VA[s.par] + phi[s.par]));
            float b[4];
            bernoulli_lane(0.03742f * dve, b);
            if (s.has) {
                float sigma = 0.0f, hi = 0.0f;
                uint32_t lo = 0xFFFFFFFFu;
#pragma unroll
                for (int q = 0; q < 7; q++) {
                    const int gq = q == 2 || q == 4 ? 2 : 0;
                    const bool neg = q == 3 || q == 5;
                    const float ca = t.c[q][s.x], cb = t.c[q][s.par];
                    sigma += kZ2D[q] * (0.5f * (ca + cb));
                    const float coef = div_rn_f(kDiffC[q] * area * dt_sub, dist, rdist);
                    const float f = coef * (ca * (neg ? b[1] : b[gq]) - cb * (neg ? b[0] : b[gq + 1]));
                    t.f[q][s.x] = f;
                    if (q != 5) {
                        lo = min(lo, 2u * __float_as_uint(f) - 1u);
                        hi = fmaxf(hi, fabsf(f));
                        ok &= fabsf(coef) < 1e20f;
                    }
                }
                t.gax[s.x] = div_rn_f(3.612f * sigma * area, dist, rdist);
                t.term[s.x] = dve;   // for now
                ok &= lo >= 2u * 0x12800000u - 1u && hi <= 0x1p90f && fabsf(dve) < 1e18f;   // 0x12800000: 2^-90
            }
        }
        const bool fast = __syncthreads_and(ok) != 0;
        // each connection's current: its own thread, from its own fluxes
#pragma unroll
        for (int r = 0; r < 2; r++) {
            if (!sl[r].has) continue;
            float ie = 0.0f;
#pragma unroll
            for (int q = 0; q < 7; q++) {
                if (fast && q == 5) continue;
                const float a = kZF[q] * t.f[q][sl[r].x];
                if (fast) {
                    const float q0 = a * ydts;
                    ie += __fmaf_rn(__fmaf_rn(-q0, dt_sub, a), ydts, q0);
                } else {
                    ie += a / dt_sub;
                }
            }
            t.term[sl[r].x] = ie - t.gax[sl[r].x] * t.term[sl[r].x];
        }
        // the ions (each reads the fluxes and its own concentrations: in place)
        float gd[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const TreeSlot<kInc>& s = sl[r];
            const double vf = (double)s.vf, yv = 1.0 / vf;
#pragma unroll kUQ
            for (int q = 0; q < 7; q++) {
                if (fast && q == 5 && !ledger) continue;
                double lost = 0.0;
                if (s.on) {
                    double acc = 0.0;
#pragma unroll
                    for (int k = 0; k < kInc; k++) {
                        const uint32_t w = s.w[k];
                        const double fl = (double)t.f[q][w];
                        const double dq = fast ? over(fl, vf, yv) : (w == (uint32_t)C ? 0.0 : fl / vf);
                        acc += w == s.x ? -dq : dq;
                    }
                    const float old = t.c[q][s.x];
                    const float upd = old + (float)acc;
                    t.c[q][s.x] = upd;
                    if (kOpt) lost = ((double)upd - (double)old - acc) * vf;
                }
                if (ledger) ledger_add(sh_ledger, q, lost);
            }
        }
        __syncthreads();   // term
        float rhs[2], den[2], yden[2], gx[2][kInc], inp[2];
        bool vok = true;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            gd[r] = inp[r] = 0.0f;
            bool pos = true;
#pragma unroll
            for (int k = 0; k < kInc; k++) {
                const uint32_t w = sl[r].w[k];
                gx[r][k] = t.gax[w];
                gd[r] += gx[r][k];
                inp[r] += w == sl[r].x ? t.term[w] : -t.term[w];
                pos &= gx[r][k] >= 0.0f;
            }
            rhs[r] = sl[r].cdt * sl[r].V + inp[r];
            den[r] = sl[r].cdt + gd[r];
            yden[r] = 1.0f / den[r];
            // the conditions of k_diffusion_path's solve
            vok &= !sl[r].on || (pos && den[r] >= 0x1p-32f && den[r] <= 0x1p32f && fabsf(sl[r].V) <= 0x1p60f &&
                                 fabsf(rhs[r]) <= 0x1p60f && fabsf(rhs[r]) >= 0x1p-60f);
        }
        if (kOpt && (d.diff_mode & 1u)) {
            // residual-controlled FP64 Jacobi; the iterates take the fluxes' rows
            __syncthreads();
            double *wa = t.fd[0], *wb = t.fd[1];
#pragma unroll
            for (int r = 0; r < 2; r++)
                if (sl[r].on) wa[sl[r].x] = (double)sl[r].V;
            double rd[2], dd[2], yd[2];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                rd[r] = (double)sl[r].cdt * (double)sl[r].V + (double)inp[r];
                dd[r] = (double)sl[r].cdt + (double)gd[r];
                yd[r] = 1.0 / dd[r];
            }
            const double* res = tree_residual(d, sl, wa, wb, sh_bits, [&](int r, const double* w) {
                double off = 0.0;
#pragma unroll
                for (int k = 0; k < kInc; k++)
                    if (sl[r].w[k] != (uint32_t)C) off += (double)gx[r][k] * w[sl[r].o[k]];
                return div_rn_d(rd[r] + off, dd[r], yd[r]);
            }, 0);
#pragma unroll
            for (int r = 0; r < 2; r++)
                if (sl[r].on) { sl[r].V = (float)res[sl[r].x]; t.VA[sl[r].x] = sl[r].V; }
            __syncthreads();
            if (tid < 7) t.f[tid][C] = 0.0f;   // the iterates ran over them
            continue;
        }
        if (__syncthreads_and(vok)) {
            // no connection: 0 x this slot's own value.  Sweeps in pairs, so that the
            // iterates' rows are fixed; the last of ten is compared with the one before.
            bool same = true;
            auto sweep = [&](const float* from, float* to, auto compare) {
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    float sum = gx[r][0] * from[sl[r].o[0]];
#pragma unroll
                    for (int k = 1; k < kInc; k++) sum += gx[r][k] * from[sl[r].o[k]];
                    const float a = rhs[r] + sum;
                    const float q0 = a * yden[r];
                    const float v = __fmaf_rn(__fmaf_rn(-q0, den[r], a), yden[r], q0);
                    if (!sl[r].on) continue;
                    if (decltype(compare)::value) same &= __float_as_uint(v) == __float_as_uint(from[sl[r].x]);
                    to[sl[r].x] = v;
                }
            };
            for (int it = 0; it < 50; it += 10) {
#pragma unroll 1
                for (int k = 0; k < 4; k++) {
                    sweep(t.VA, t.VB, std::false_type());
                    __syncthreads();
                    sweep(t.VB, t.VA, std::false_type());
                    __syncthreads();
                }
                sweep(t.VA, t.VB, std::false_type());
                __syncthreads();
                same = true;
                sweep(t.VB, t.VA, std::true_type());
                if (__syncthreads_and(same)) break;   // a fixed point
            }
#pragma unroll
            for (int r = 0; r < 2; r++)
                if (sl[r].on) sl[r].V = t.VA[sl[r].x];
        } else {
            float *va = t.VA, *vb = t.VB;
            for (int it = 0; it < 50; it++) {   // an even number: VA holds the result
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    if (!sl[r].on) continue;
                    float off = 0.0f;
#pragma unroll
                    for (int k = 0; k < kInc; k++)
                        if (sl[r].w[k] != (uint32_t)C) off += gx[r][k] * va[sl[r].o[k]];
                    sl[r].V = (rhs[r] + off) / den[r];
                    vb[sl[r].x] = sl[r].V;
                }
                float* tmp = va; va = vb; vb = tmp;
                __syncthreads();
            }
        }
    }

    // ---- the intracellular side is done; the extracellular one takes its rows ----
    __syncthreads();
    if (tid < 4) t.fd[tid][C] = 0.0;
    float fin_x[2];
    bool fin = sane;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        fin_x[r] = 0.0f;
        if (sl[r].has) fin_x[r] = (float)(0.03742f * (phi[sl[r].x] - phi[sl[r].par]));
        fin &= fabsf(fin_x[r]) < 1e3f;
        if (!sl[r].on) continue;
        const SegRec* rec = d.rec + sl[r].g;
        if (d.flags & NF_PRE_EXT)
            d.pre_ext[sl[r].g] = make_float4(t.c[0][sl[r].x], t.c[1][sl[r].x], t.c[2][sl[r].x], 0.0f);
#pragma unroll
        for (int q = 0; q < 7; q++) {
            d.ion_in[q * N + sl[r].g] = t.c[q][sl[r].x];
            t.c[q][sl[r].x] = rec->out[q];
        }
        d.V[sl[r].g] = sl[r].V;
    }
    // ---- extracellular Nernst-Planck, 5 sub-steps (diffusion_kernel.h:244-281), the ions in
    // pairs through two halves of the flux rows: one barrier per pair ----
    {
        float b[2][4];
        bernoulli_lane(fin_x[0], b[0]);
        bernoulli_lane(fin_x[1], b[1]);
        double yv[2];
#pragma unroll
        for (int r = 0; r < 2; r++) yv[r] = 1.0 / (double)sl[r].vf;
        const int np = 4;   // ions (0, 1), (2, 3), (4, 6) and, where its fluxes count, 5
        int half = 0;
#pragma unroll 1
        for (int sub = 0; sub < 5; sub++) {
            bool ok = fin;
#pragma unroll
            for (int r = 0; r < 2; r++)
                if (sl[r].on)
#pragma unroll
                    for (int q = 0; q < 7; q++) ok &= !(fabsf(t.c[q][sl[r].x]) >= 1e20f) || q == 5;
            const bool fast = __syncthreads_and(ok) != 0;
#pragma unroll 1
            for (int pr = 0; pr < np; pr++) {
                if (pr == 3 && fast && !ledger) break;
                double(*const fr)[C + 2] = t.fd + 2 * half;
                half ^= 1;
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    if (pr == 3 && j == 1) break;
                    const int q = pr == 3 ? 5 : (pr == 2 && j == 1 ? 6 : 2 * pr + j);
                    const int gq = q == 2 || q == 4 ? 2 : 0;
                    const bool neg = q == 3 || q == 5;
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        if (!sl[r].has) continue;
                        const float coef = kDiffC[q] * d.tr_area[sl[r].g] * dt_sub / d.tr_dist[sl[r].g];
                        const double Ca = t.c[q][sl[r].x], Cb = t.c[q][sl[r].par];
                        const float bm = neg ? b[r][1] : (gq ? b[r][2] : b[r][0]);
                        const float bp = neg ? b[r][0] : (gq ? b[r][3] : b[r][1]);
                        fr[j][sl[r].x] = coef * (Ca * bm - Cb * bp);
                    }
                }
                __syncthreads();
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    if (pr == 3 && j == 1) break;
                    const int q = pr == 3 ? 5 : (pr == 2 && j == 1 ? 6 : 2 * pr + j);
                    double lost = 0.0;
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        if (!sl[r].on) continue;
                        const float vx = sl[r].vf * EXTRA_VOLUME_RATIO;
                        double acc = 0.0;
#pragma unroll
                        for (int k = 0; k < kInc; k++) {
                            const uint32_t w = sl[r].w[k];
                            const double fl = fr[j][w];
                            const double dq = fast ? 4.0 * over(fl, (double)sl[r].vf, yv[r])
                                                   : (w == (uint32_t)C ? 0.0 : fl / (double)vx);
                            acc += w == sl[r].x ? -dq : dq;
                        }
                        const float old = t.c[q][sl[r].x];
                        const float upd = (float)((double)old + acc);
                        t.c[q][sl[r].x] = upd;
                        if (kOpt) lost += ((double)upd - (double)old - acc) * (double)vx;
                    }
                    if (ledger) ledger_add(sh_ledger, q, lost);
                }
            }
        }
    }
    // ---- NT / ATP / heat / transcription (diffusion_kernel.h:284-363) ----
    auto field = [&](float* base, float D, float thresh, auto strict) {
        float v[2];
#pragma unroll
        for (int r = 0; r < 2; r++) v[r] = sl[r].on ? base[sl[r].g] : 0.0f;
        tree_fick<C, kInc, decltype(strict)::value>(d, t, sl, v, D, thresh, dt);
#pragma unroll
        for (int r = 0; r < 2; r++)
            if (sl[r].on) base[sl[r].g] = v[r];
    };
    if (d.flags & NF_INTRA_NT)
        for (int nt = 0; nt < 15; nt++) field(d.intra_nt + nt * N, gNtD[nt], 1e-12f, std::false_type());
    if (d.flags & NF_NT_DIFFUSE_OUT)
        for (int nt = 0; nt < 15; nt++) field(d.nt + nt * N, gNtD[nt], 1e-12f, std::false_type());
    {
        float v[2];
#pragma unroll
        for (int r = 0; r < 2; r++) v[r] = sl[r].on ? d.rec[sl[r].g].atp : 0.0f;
        tree_fick<C, kInc, true>(d, t, sl, v, 0.14f, 1e-12f, dt);
#pragma unroll
        for (int r = 0; r < 2; r++)
            if (sl[r].on) d.atp[sl[r].g] = v[r];
    }
    if (d.flags & NF_TEMP) field(d.temp, 0.0014f, 0.001f, std::true_type());
    if (d.flags & NF_TXN) field(d.txn, 0.01f, 1e-9f, std::true_type());

    // ---- bath relaxation and clamp, write back (each slot its own values) ----
#pragma unroll 1
    for (int q = 0; q < 7; q++) {
        double x = 0.0;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            if (!sl[r].on) continue;
            const float old = t.c[q][sl[r].x];
            double e = (double)old;
            e += (kBathIon[q] - e) * dt / 1.0f;
            if (e < 1e-9) e = 1e-9;
            if (e > 1000.0) e = 1000.0;
            t.c[q][sl[r].x] = (float)e;
            d.ion_out[q * N + sl[r].g] = (float)e;
            if (kOpt) x += ((double)(float)e - (double)old) * (double)(sl[r].vf * EXTRA_VOLUME_RATIO);
        }
        if (ledger) ledger_add(sh_ledger, 7 + q, x);
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        if (!sl[r].on) continue;
        const uint32_t g = sl[r].g;
        const float2 c21 = d.c21_cur[g];
        d.pre_rec[g] = make_float4(sl[r].V, t.c[2][sl[r].x], c21.x, c21.y);
        if (d.flags & NF_PRE_EXT) {
            d.pre_ext[g].w = t.c[0][sl[r].x];
            d.pre_ext2[g] = t.c[1][sl[r].x];
        }
    }
    if (ledger) {
        __syncthreads();
        if (tid < 14) atomicAdd(&d.ledger[tid], sh_ledger[tid]);
    }
}

template <int C, int kInc>
static cudaError_t launch_tree(const NetDev& dev, float dt, unsigned long long tick, cudaStream_t stream) {
    if (dev.diff_mode) k_diffusion_tree<C, kInc, true><<<dev.n_tr, C / 2, sizeof(TreeRows<C>), stream>>>(dev, dt, tick);
    else k_diffusion_tree<C, kInc, false><<<dev.n_tr, C / 2, sizeof(TreeRows<C>), stream>>>(dev, dt, tick);
    return cudaGetLastError();
}
template <int C>
static cudaError_t launch_tree(const NetDev& dev, uint32_t inc, float dt, unsigned long long tick, cudaStream_t stream) {
    return inc <= 3 ? launch_tree<C, 3>(dev, dt, tick, stream) : launch_tree<C, 4>(dev, dt, tick, stream);
}
static cudaError_t launch_diffusion_tree(const NetDev& dev, uint32_t slots, uint32_t inc, float dt,
                                         unsigned long long tick, cudaStream_t stream) {
    return slots == 512 ? launch_tree<512>(dev, inc, dt, tick, stream)
                        : (slots == 1024 ? launch_tree<1024>(dev, inc, dt, tick, stream)
                                         : launch_tree<2048>(dev, inc, dt, tick, stream));
}
template <int C>
static cudaError_t prepare_tree() {
    const void* k[] = {(const void*)k_diffusion_tree<C, 3, false>, (const void*)k_diffusion_tree<C, 3, true>,
                       (const void*)k_diffusion_tree<C, 4, false>, (const void*)k_diffusion_tree<C, 4, true>};
    for (const void* f : k) {
        const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TreeRows<C>));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

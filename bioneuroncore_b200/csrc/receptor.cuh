// receptor.cuh -- the ionotropic receptor model shared by the synapse kernel and the
// adjoint's replay: constants of AMPA, NMDA, GABA-A and glycine, the device table of
// their permeabilities, and the current (modifier_helpers.h:1213-1279).  Each
// translation unit that includes it holds its own table and initialises it with
// k_init_receptors once per device.
#pragma once
#include "physics.cuh"

namespace bnc {

namespace {

// Ionotropic receptor constants (receptors_biological.cpp:42-82 through
// modifier_helpers.h:1213-1279): AMPA, NMDA, GABA-A, glycine.  The permeabilities at
// the default conductance are computed once on the device with the same helpers the
// models use, so they equal the constants a per-type specialisation folds.
struct RecKind {
    float gamma_ps, EC50, tau_rise, tau_decay, P_Na_ratio, P_K_ratio, P_Ca_ratio, tau_desens, K_desens;
    int is_anion, nmda;
    double P_Na, P_K, P_Ca, P_Cl;
};

__device__ RecKind gRec[4];

__global__ void k_init_receptors() {
    const float c[4][9] = {{8.0f, 0.5f, 0.5f, 3.0f, 0.5f, 0.5f, 0.0f, 3.0f, 0.0f},
                           {50.0f, 1.0f, 5.0f, 50.0f, 0.08f, 0.08f, 0.84f, 0.0f, 0.0f},
                           {28.0f, 1.0f, 1.0f, 5.0f, 0.0f, 0.0f, 0.0f, 2000.0f, 0.0f},
                           {60.0f, 0.5f, 0.3f, 5.0f, 0.0f, 0.0f, 0.0f, 2000.0f, 0.0f}};
    for (int k = 0; k < 4; k++) {
        RecKind& r = gRec[k];
        r.gamma_ps = c[k][0]; r.EC50 = c[k][1]; r.tau_rise = c[k][2]; r.tau_decay = c[k][3];
        r.P_Na_ratio = c[k][4]; r.P_K_ratio = c[k][5]; r.P_Ca_ratio = c[k][6];
        r.tau_desens = c[k][7]; r.K_desens = c[k][8];
        r.is_anion = k >= 2;
        r.nmda = k == 1;
        dp_partial_P(r.gamma_ps, r.P_Na_ratio, r.P_K_ratio, r.P_Ca_ratio, &r.P_Na, &r.P_K, &r.P_Ca);
        r.P_Cl = dp_ghk_P(r.gamma_ps, 1.0f, GHK_CBAR_CL_MM);
    }
}

__device__ __forceinline__ int receptor_kind(uint8_t type) {
    return type == 8 ? 0 : (type == 9 ? 1 : (type == 11 ? 2 : 3));
}

// modifier_helpers.h:1213-1279 (ionotropic_ghk_current) with the receptor's constants
// as data; NMDA adds the Mg2+ block and CDI/co-agonist factor (receptors_biological.cpp:48-70).
__device__ __forceinline__ double receptor_current(const RecKind& K, DMod& m, DSeg& s, float dt, float nt,
                                                  float mod_scale) {
    float area = m.area;
    double V = ((double)s.V);
    double vol = s.vol;
    double cpm = FARADAY_CONST * vol / 1000.0;
    const bool custom = m.av != 0;   // conductance override through active_vars
    float p_gamma_ps = K.gamma_ps;
    if (custom) {
        float stav = (m.av == 7) ? m.area : (m.av == 1 ? m.st[1] : (m.av == 2 ? m.st[2] : 0.0f));
        p_gamma_ps = (m.av > 0 && m.av < 8 && ((double)stav) > 0.0f) ? (float)((double)stav) : K.gamma_ps;
    }
    float r_inf = nt / (nt + K.EC50);
    float r = m.st[0];
    float tau = (r_inf > r) ? K.tau_rise : K.tau_decay;
    m.st[0] = (float)(((double)m.st[0]) + (r_inf - r) * dt / tau);
    if (((double)m.st[0]) < 0.0f) m.st[0] = 0.0f;
    if (((double)m.st[0]) > 1.0f) m.st[0] = 1.0f;
    float open_prob = m.st[0];
    if (K.tau_desens > 0.0f) {
        float kd = (K.K_desens > 0.0f) ? K.K_desens : K.EC50;
        float dd = m.st[1];
        float d_inf = nt / (nt + kd);
        dd += (d_inf - dd) * dt / K.tau_desens;
        if (dd < 0.0f) dd = 0.0f;
        if (dd > 1.0f) dd = 1.0f;
        m.st[1] = dd;
        open_prob *= (1.0f - dd);
    }
    double N = ((double)m.den) * area;
    double I;
    if (K.is_anion) {
        double P_Cl = custom ? dp_ghk_P(p_gamma_ps, 1.0f, GHK_CBAR_CL_MM) : K.P_Cl;
        double flux_Cl = dp_ghk_anion_c(s.gc, V, ((double)s.in[3]), ((double)s.out[3]));
        double I_Cl = P_Cl * flux_Cl * N * open_prob * mod_scale * A_TO_PA;
        s.in[3] = (float)(((double)s.in[3]) + (I_Cl * dt) / cpm);
        dp_clamp_ions(s.in);
        I = -I_Cl;
    } else {
        double P_Na = K.P_Na, P_K = K.P_K, P_Ca = K.P_Ca;
        if (custom) dp_partial_P(p_gamma_ps, K.P_Na_ratio, K.P_K_ratio, K.P_Ca_ratio, &P_Na, &P_K, &P_Ca);
        double I_Na = P_Na * dp_ghk_mono_c(s.gc, V, ((double)s.in[0]), ((double)s.out[0])) * N * open_prob * mod_scale * A_TO_PA;
        double I_K = P_K * dp_ghk_mono_c(s.gc, V, ((double)s.in[1]), ((double)s.out[1])) * N * open_prob * mod_scale * A_TO_PA;
        double I_total = I_Na + I_K;
        s.in[0] = (float)(((double)s.in[0]) - (I_Na * dt) / cpm);
        s.in[1] = (float)(((double)s.in[1]) - (I_K * dt) / cpm);
        if (K.P_Ca_ratio > 0.0f) {
            double I_Ca = P_Ca * dp_ghk_div_c(s.gc, V, ((double)s.in[2]), ((double)s.out[2])) * N * open_prob * mod_scale * A_TO_PA;
            I_total += I_Ca;
            s.in[2] = (float)(((double)s.in[2]) - (I_Ca * dt) / (2.0f * cpm));
        }
        dp_clamp_ions(s.in);
        I = -I_total;
    }
    if (K.nmda) {
        float mg_block = (float)(1.0f / (1.0f + (1.0f / 3.57f) * dm_exp(-0.062f * ((double)s.V))));
        double c = dp_nmda_cdi_coagonist(m, s, dt);
        I = I * mg_block * c;
    }
    return I;
}

// What the receptor currents of one segment share through step 3 (V_m, the extracellular
// ions and the volume are constant there): the GHK factors with their reciprocals, the
// products of the constant side, NMDA's Mg2+ block.  A receptor's current depends on the
// intracellular ions the receptor before it left, so a segment's receptors are one serial
// chain, and its latency bounds the synapse step of any network that does not fill the
// chip many times over.  With the reciprocals a receptor is about 16 dependent FP64
// operations (9 cycles each) in place of three full divisions (112 cycles each) among 25,
// and rec_gates, rec_flux and rec_tail run all four receptor kinds without divergence.
struct RecSeg {
    double A1, D1, y1, e1, o0, o1, o3;   // monovalent: out Na and K times e1, out Cl
    double A2, D2, y2, o2;               // divalent: out Ca times e2
    double cpm, yc;
    float mg;
    bool ok;                             // the fast form holds for this segment
};

__device__ __forceinline__ void rec_seg_fill(RecSeg& f, const DSeg& s, float dt) {
    f.A1 = s.gc.A1; f.D1 = s.gc.D1; f.e1 = s.gc.e1;
    f.A2 = s.gc.A2; f.D2 = s.gc.D2;
    f.y1 = 1.0 / f.D1;
    f.y2 = 1.0 / f.D2;
    f.o0 = (double)s.out[0] * s.gc.e1;
    f.o1 = (double)s.out[1] * s.gc.e1;
    f.o2 = (double)s.out[2] * s.gc.e2;
    f.o3 = (double)s.out[3];
    f.cpm = FARADAY_CONST * s.vol / 1000.0;
    f.yc = 1.0 / f.cpm;
    f.mg = (float)(1.0f / (1.0f + (1.0f / 3.57f) * dm_exp(-0.062f * ((double)s.V))));
    f.ok = s.gc.m1 == 0 && s.gc.m2 == 0 && fabs(f.cpm) >= 0x1p-100 && fabs(f.cpm) <= 0x1p100 && dt >= 1e-12f &&
           dt <= 1e12f;
}

// A kind's constants as the step reads them (shared memory): permeabilities of its first
// ion (Na, or Cl), K and Ca; time constants with their reciprocals rounded to nearest.
struct RecK {
    double P0, P1, P2, unused;
    double rise, y_rise, decay, y_decay, des, y_des;
};
__device__ __forceinline__ void rec_k_fill(RecK& k, const RecKind& K) {
    k.P0 = K.is_anion ? K.P_Cl : K.P_Na;
    k.P1 = K.is_anion ? 0.0 : K.P_K;
    k.P2 = K.nmda ? K.P_Ca : 0.0;
    k.unused = 0.0;
    k.rise = (double)K.tau_rise; k.y_rise = 1.0 / k.rise;
    k.decay = (double)K.tau_decay; k.y_decay = 1.0 / k.decay;
    k.des = K.tau_desens > 0.0f ? (double)K.tau_desens : 1.0; k.y_des = 1.0 / k.des;
}

// a / b rounded to nearest by Markstein's correction, given y = 1 / b rounded to nearest;
// for a zero (whose sign may be lost) or away from under- and overflow (the callers see to
// that).
__device__ __forceinline__ double rec_div(double a, double b, double y) {
    const double q0 = a * y;
    return __fma_rn(__fma_rn(-q0, b, a), y, q0);
}
// Zero, or of a magnitude in about [1e-200, 1e200], by the exponent field.
__device__ __forceinline__ bool rec_in_range(double x) {
    const uint32_t h = ((uint32_t)__double2hiint(x) & 0x7FFFFFFFu) - 0x16700000u;
    return (h < 0x53000000u) | (x == 0.0);
}
// x + (to - x) dt / tau in float, clamped to [0, 1].  The float quotient is the binary64
// one rounded again: that rounds twice to the same value (53 >= 2 x 24 + 2 bits), for
// subnormal quotients of a decayed gate too.
__device__ __forceinline__ float rec_relax(float x, float to, float dt, double tau, double ytau, bool& ok) {
    const float a = (to - x) * dt;
    ok &= fabsf(a) < 1e30f;
    const float v = x + (float)rec_div((double)a, tau, ytau);
    return v < 0.0f ? 0.0f : (v > 1.0f ? 1.0f : v);
}
__device__ __forceinline__ float rec_clamp(float x) { return x < 1e-9f ? 1e-9f : x; }

// receptor_current for a default-conductance receptor of a segment whose RecSeg is ok, the
// same operations in the same order, in three stages of which only the second is part of
// the segment's chain.  Every lane of the warp takes part, so that lanes with different
// kinds run one instruction stream.
//
// The gates.  r_inf: nt / (nt + EC50), also the desensitisation gate's target (K_desens is
// 0 for all kinds).  w: the desensitisation gate, relaxed; for NMDA the inactivation gate,
// left to rec_tail.  Returns whether the corrected quotients are the IEEE ones here.
__device__ __forceinline__ bool rec_gates(const RecK& K, int kind, float r, float& w, float dt, float r_inf, float& rn,
                                          float& open) {
    const bool nmda = kind == 1;
    const bool up = r_inf > r;
    bool ok = !nmda | (fabsf(w) < 1e30f);
    rn = rec_relax(r, r_inf, dt, up ? K.rise : K.decay, up ? K.y_rise : K.y_decay, ok);
    const float wn = rec_relax(w, r_inf, dt, K.des, K.y_des, ok);
    open = nmda ? rn : rn * (1.0f - wn);
    w = nmda ? w : wn;
    return ok;
}
// The currents: the sum of inward ones (It, without NMDA's block) and the segment's ions;
// ca: the intracellular Ca2+ it leaves.  Returns `ok` as long as the fast form holds;
// nothing is changed in a lane where it does not (a value out of the range in which the
// corrected quotients are the IEEE ones, or not finite).  kInline: the Ca2+ current in line
// with the others, which shortens the chain; else only where some lane has an NMDA receptor.
template <bool kInline>
__device__ __forceinline__ bool rec_flux(const RecSeg& f, const RecK& K, int kind, bool ok, float den, float area,
                                         float open, float (&in)[7], float dt, float mod_scale, double& It, float& ca) {
    const bool an = kind >= 2, nmda = kind == 1;
    const double N = (double)den * area;
    const double n0 = an ? f.o3 - (double)in[3] * f.e1 : (double)in[0] - f.o0;
    const double f0 = rec_div(f.A1 * n0, f.D1, f.y1);
    const double f1 = rec_div(f.A1 * ((double)in[1] - f.o1), f.D1, f.y1);
    const double I0 = K.P0 * f0 * N * open * mod_scale * A_TO_PA;
    const double I1 = K.P1 * f1 * N * open * mod_scale * A_TO_PA;
    const double q0 = rec_div(I0 * dt, f.cpm, f.yc);
    const float c0 = rec_clamp((float)((double)(an ? in[3] : in[0]) - (an ? -q0 : q0)));
    const float c1 = rec_clamp((float)((double)in[1] - rec_div(I1 * dt, f.cpm, f.yc)));
    It = an ? I0 : I0 + I1;
    float c2 = rec_clamp(in[2]);
    const bool any = kInline || __any_sync(0xFFFFFFFFu, ok & nmda);
    ok &= rec_in_range(I0) & (an | rec_in_range(I1));
    if (any) {
        const double f2 = rec_div(f.A2 * ((double)in[2] - f.o2), f.D2, f.y2);
        const double I2 = K.P2 * f2 * N * open * mod_scale * A_TO_PA;
        const float n2 = rec_clamp((float)((double)in[2] - 0.5 * rec_div(I2 * dt, f.cpm, f.yc)));
        c2 = nmda ? n2 : c2;
        It = nmda ? It + I2 : It;
        ok &= !nmda | (rec_in_range(I2) & (n2 < 1e30f));
    }
    ca = c2;
    if (ok) {   // with the clamp of the ions the receptor leaves alone
        in[0] = an ? rec_clamp(in[0]) : c0;
        in[1] = an ? rec_clamp(in[1]) : c1;
        in[2] = c2;
        in[3] = an ? c0 : rec_clamp(in[3]);
    }
    return ok;
}
// 0.8f c / (c + 1.0f) for NMDA's inactivation, c a float concentration from 1e-9 to 1e30
// times 1000: two steps of Newton's iteration for y = 1 / b, then Markstein's correction.
// Before its last rounding y is within 2^-80 of 1 / b, so it can miss the nearest double
// (6 of the 1,086,358,124 concentrations do) and Markstein's theorem does not cover it; the
// quotient is the IEEE one at every one of them, by exhaustion on the device.  In line and
// without the general division's branch, so that it overlaps the next receptor's chain.
__device__ __forceinline__ double rec_quot(double a, double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
#pragma unroll
    for (int k = 0; k < 2; k++) y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
    return rec_div(a, b, y);
}
// NMDA's Mg2+ block and inactivation (dp_nmda_cdi_coagonist) of the current It.
__device__ __forceinline__ void rec_tail(const RecSeg& f, float ca, float& w, float dt, double& It) {
    const double Ca_uM = (double)ca * MM_TO_UM;
    const double cdi_inf = 1.0 - rec_quot(0.8f * Ca_uM, Ca_uM + 1.0f);
    const bool fast = cdi_inf < (double)w;
    const float wn = (float)((double)w + rec_div((cdi_inf - (double)w) * dt, fast ? 500.0 : 9000.0, fast ? 1.0 / 500.0 : 1.0 / 9000.0));
    w = wn < 0.0f ? 0.0f : (wn > 1.0f ? 1.0f : wn);
    It = It * f.mg * ((double)w * (10.0f / (10.0f + 1.0f)));
}
// receptor_current out of line, for the receptors the fast form does not hold for.
struct RecSlow {
    DMod m;
    DSeg s;
    double I;
};
__device__ __noinline__ void receptor_slow(RecSlow* x, int kind, float dt, float nt, float mod_scale) {
    x->I = receptor_current(gRec[kind], x->m, x->s, dt, nt, mod_scale);
}

}  // namespace

}  // namespace bnc

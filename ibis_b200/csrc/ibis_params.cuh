// Device copy of the parameter record, converted once on the host to the
// kernel's arithmetic type, plus constants derived from it in double.
#pragma once
#include "../../include/ibis_layout.h"

namespace ibis {

// Two floats as one 64-bit word
struct ParPair {
    unsigned long long v;
};

template <typename R>
struct DevParams {
#define IBIS_S(name) R name;
#define IBIS_A(name, n) R name[n];
    IBIS_PARAM_LIST(IBIS_S, IBIS_A)
#undef IBIS_S
#undef IBIS_A
    unsigned int flags;
    // ---- derived in double on the host (kept in the same precision the reference forms them)
    R tfac;            // 1 / 0.999**cappa (canopy_exchange.py:206)
    R vonk2;           // vonk**2
    R cdmax;           // 300 / (2 dtime)
    R zweight;         // exp(-1 / (10 * 86400 / dtime)) (stomata.py:486)
    R wliqmin, wsnomin;  // interception.py:292-293
    R znorm;           // 1 - exp(stressfac) (stomata.py:545)
    R rdt;             // 1 / dtime
    R zir;             // 4 * 0.95 * stef (loops.py:170; canopy_exchange.py:566)
    // soil-water solve geometry in double (soil_physics.py:238-330)
    double sw_hm[6];   // interface k (1..5): 0.5 * (h[k-1] + h[k])
    double sw_wp[6];   // 0.5 * h[k] / sw_hm[k]
    double sw_wm[6];   // 1 - sw_wp[k]
    double sw_hb[6];   // row k: max(0.5 h[0] | 0.5 h[k-1] + 0.5 h[k], 1e-30)
    double sw_hp[6];   // row k < 5: max(0.5 * (h[k] + h[k+1]), 1e-30)
    double rdt64;      // 1 / dtime in double
    R rwood_s[12], rroot_s[12], keep[12];  // float32-formed respiration rates (loops_gswp3.py:185-190)
    R ch4_w;           // float32(dtime / 86400)
    R rh_conv;         // float32(12e-3 * 86400)
    R ch4_wtop[6];     // thickness weights of the wetland water-table average (methane.py:266-270)
    R ch4_wtot;        // their sum, floored at 1e-12
    R hsoi_top[6], hsoi_bot[6];  // layer tops/bottoms (cumsum of hsoi)
    // per-PFT capacity increment per unit cropland share (loops.py:218-231): the C4
    // (PFT 10) and C3 (PFT 11) vmax scales less one, formed in float32 as the
    // reference forms them on float32 masks; zero for the other PFTs
    R crop_inc[12];
    // index of the launch's first column in the caller's numbering: a launch
    // over a group of columns (ibis_step_host_f32) reports status[1] in it
    int cell0;
    // what the FP32 step multiplies by (formed in double on the host)
    R rtheta3, rbeta3, rtheta4, rbeta4;
    R ksu, kss, ksl;         // boundary-layer conductances of leaves, stems and lower canopy over rhoa sqrt(u)
    R hs_below5, hs_above5;  // h[5] and h[4] over h[4] + h[5]
    R bed_res[3];            // bedrock layer: half its thermal resistance
    R bed_con[3];            // conductance to the layer below
    R bed_rw[3];             // dtime over the heat capacity
    // and the pairs of floats its packed arithmetic takes, each a 64-bit word (ParPair)
    // so that one constant load fills a register pair
    ParPair h2[3], rhb2[3], rhp2[3], c12[3], c32[3], c52[3], c62[3];   // soil layers (0,1), (2,3), (4,5): thickness,
                             // 1/sw_hb, 1/sw_hp, 0.5 h[k]/sw_hb, 0.5 h[k+1]/sw_hp, 0.5 h[k-1]/sw_hb, 0.5 h[k]/sw_hp
    ParPair iwp2[3], iwm2[3], irh2[3];   // interfaces (1,2), (3,4), (5,bottom): sw_wp, sw_wm, 1/sw_hm
    ParPair hsb2[2], hsa2[2];            // interfaces (1,2), (3,4): h[k] and h[k-1] over h[k-1] + h[k]
    ParPair top2[3], bot2[3];            // layer tops and bottoms
    ParPair fr2[6], frl2[3], fru2[3];    // root profile: (lower, upper) of a layer; lower, upper of a pair of layers
    ParPair rho2[2], tau2[2], osno2;     // (visible, near infrared) of the lower and upper story; snow's scattering
    ParPair drip2[3], kdrip2[3];         // (1 / drip time, 1 / blow-off time), 1 - dtime / time: upper leaves, stems, lower
    ParPair water2, ralai2, chus2;       // (ch2o, cice), 1 / (alaiml, alaimu), (chu, chs)
    ParPair gam2[2], b02[2], gmin2[2];   // dark respiration, Ball-Berry intercept and least conductance of the
                                         // C3 big leaves: broadleaf and conifer; shrub and C3 grass
    ParPair cm2[2], vml2;                // their slopes; nominal vmax of the lower two
    ParPair rroot2[6], rwood2[5], keep2[6];   // respiration rates of PFTs (0,1), (2,3) ...
    // per-band thickness weights of the wetland water-table average and their
    // sums (IBIS_FLAG_CH4_BANDS: from ch4b_z_wt_ref as ch4_wtop from z_wt_ref)
    R ch4b_wtop[3][6];
    R ch4b_wtot[3];
};

// The parameters a calibration ensemble varies per run (the 31-parameter
// vector: vmax per plant type, Ball-Berry slopes, soil-stress shape,
// soil-evaporation exponent, interception capacities, wet fraction cap,
// wetland-CH4 parameters, maintenance/growth respiration), and the values
// derived from them.  The physics reads them through one of two sources:
// UniformQ (one parameter record for every cell) or RunQ (one run's values,
// 33 words: an odd stride, so a warp reading one field of its 32 runs' records
// in shared memory touches 32 different banks).
//
// ``x3`` marks the sources of the kernels compiled with the IBIS 3.0 extensions
// of the step (IBIS_FLAGS_X3): the F77 kernels carry none of their code.
template <typename R>
struct UniformQ {
    static constexpr bool x3 = false;
    const DevParams<R>& P;
    __device__ __forceinline__ R vmax(int j) const { return P.vmax_pft[j]; }
    __device__ __forceinline__ R coefm(int g) const { return P.coefm[g]; }
    __device__ __forceinline__ R stressfac() const { return P.stressfac; }
    __device__ __forceinline__ R znorm() const { return P.znorm; }
    __device__ __forceinline__ R beta_power() const { return P.soil_beta_power; }
    __device__ __forceinline__ R wliqumax() const { return P.wliqumax; }
    __device__ __forceinline__ R wliqsmax() const { return P.wliqsmax; }
    __device__ __forceinline__ R wliqlmax() const { return P.wliqlmax; }
    __device__ __forceinline__ R fmax() const { return P.fmax; }
    __device__ __forceinline__ R wliqmin() const { return P.wliqmin; }
    __device__ __forceinline__ R r_ch4() const { return P.r_ch4; }
    __device__ __forceinline__ R q10p() const { return P.q10p; }
    __device__ __forceinline__ R z_tau() const { return P.z_tau; }
    __device__ __forceinline__ R tau_oxid() const { return P.tau_oxid; }
    __device__ __forceinline__ R z_wt_max() const { return P.z_wt_max; }
    __device__ __forceinline__ R rwood(int j) const { return P.rwood_s[j]; }
    __device__ __forceinline__ R rroot(int j) const { return P.rroot_s[j]; }
    __device__ __forceinline__ R keep(int j) const { return P.keep[j]; }
    // the pairs of the FP32 step: st 0 upper, 1 lower; j an even PFT
    __device__ __forceinline__ ParPair coefm2(int st) const { return P.cm2[st]; }
    __device__ __forceinline__ ParPair vmaxl2() const { return P.vml2; }
    __device__ __forceinline__ ParPair rroot2(int j) const { return P.rroot2[j / 2]; }
    __device__ __forceinline__ ParPair rwood2(int j) const { return P.rwood2[j / 2]; }
    __device__ __forceinline__ ParPair keep2(int j) const { return P.keep2[j / 2]; }
};

// One parameter record for every cell, in the kernels that carry the IBIS 3.0
// extensions.
template <typename R>
struct UniformQ3 : UniformQ<R> {
    static constexpr bool x3 = true;
};

template <typename R>
struct RunQ {
    static constexpr bool x3 = false;
    R vmax_[12], coefm_[5], stressfac_, znorm_, beta_, wliqumax_, wliqsmax_, wliqlmax_, fmax_, wliqmin_;
    R r_ch4_, q10p_, z_tau_, tau_oxid_, z_wt_max_, rwood_, rroot_, keep_;
    __device__ __forceinline__ R vmax(int j) const { return vmax_[j]; }
    __device__ __forceinline__ R coefm(int g) const { return coefm_[g]; }
    __device__ __forceinline__ R stressfac() const { return stressfac_; }
    __device__ __forceinline__ R znorm() const { return znorm_; }
    __device__ __forceinline__ R beta_power() const { return beta_; }
    __device__ __forceinline__ R wliqumax() const { return wliqumax_; }
    __device__ __forceinline__ R wliqsmax() const { return wliqsmax_; }
    __device__ __forceinline__ R wliqlmax() const { return wliqlmax_; }
    __device__ __forceinline__ R fmax() const { return fmax_; }
    __device__ __forceinline__ R wliqmin() const { return wliqmin_; }
    __device__ __forceinline__ R r_ch4() const { return r_ch4_; }
    __device__ __forceinline__ R q10p() const { return q10p_; }
    __device__ __forceinline__ R z_tau() const { return z_tau_; }
    __device__ __forceinline__ R tau_oxid() const { return tau_oxid_; }
    __device__ __forceinline__ R z_wt_max() const { return z_wt_max_; }
    __device__ __forceinline__ R rwood(int) const { return rwood_; }
    __device__ __forceinline__ R rroot(int) const { return rroot_; }
    __device__ __forceinline__ R keep(int) const { return keep_; }
    static __device__ __forceinline__ ParPair pair(float a, float b) {
        ParPair p;
        asm("mov.b64 %0, {%1, %2};" : "=l"(p.v) : "f"(a), "f"(b));
        return p;
    }
    __device__ __forceinline__ ParPair coefm2(int st) const {
        return st ? pair(coefm_[2], coefm_[4]) : pair(coefm_[0], coefm_[1]);
    }
    __device__ __forceinline__ ParPair vmaxl2() const { return pair(vmax_[8], vmax_[11]); }
    __device__ __forceinline__ ParPair rroot2(int) const { return pair(rroot_, rroot_); }
    __device__ __forceinline__ ParPair rwood2(int) const { return pair(rwood_, rwood_); }
    __device__ __forceinline__ ParPair keep2(int) const { return pair(keep_, keep_); }
};

// One run's parameters in the kernels that carry the IBIS 3.0 extensions (the
// same record; the extensions' own tables come from the parameter record).
template <typename R>
struct RunQ3 : RunQ<R> {
    static constexpr bool x3 = true;
};
static_assert(sizeof(RunQ3<float>) == sizeof(RunQ<float>), "the run record's shared-memory size is one");

}  // namespace ibis

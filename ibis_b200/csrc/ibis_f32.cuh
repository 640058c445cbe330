// The hourly step of the FP32 kernels: the physics of ibis_column.cuh,
// ibis_canopy.cuh and ibis_ground.cuh (whose templates are the float64 kernels'
// operation-for-operation form), rewritten for what bounds these kernels on
// sm_100a: instruction fetch.  A warp-hour is one long body with almost no loops,
// and the instruction caches hold 128 KB (8,192 instructions): measured with
// straight-line code, a warp gets an instruction every 1.1 cycles from a 32 KB
// body, every 2.6 from a 128 KB body and every 5.8 from a larger one, which comes
// from L2.  So the same physics is written for fewer instructions:
//   * pairs of leaves, bands, stories and soil layers in packed float arithmetic
//     (ibis_pair.cuh);
//   * what the three canopy passes share formed once before them;
//   * the 9x9 canopy system (still in double) reduced to its 4x4 canopy-air block;
//   * one reciprocal where the formulas divide several times by one quantity;
//   * constants as register pairs, the passes' shared values in shared memory, the
//     statics' addresses not carried through the hour.
// Against the templates' operations in float the fused kernel went from 13,472 to 8,488
// instructions (about 7,600 of them in the hour, by the size of the kernel without the
// step; the caches hold 8,192) and six hours of 95,333 columns from 0.92 to 0.40 ms (0.26
// to 0.10 at 12,007; 24 hours of 356 columns 0.93 to 0.32-0.38, by the box; B200, 1965 MHz).
// Against the float64 kernels the error of a state or accumulator field is 0.85 times what
// it was (geometric mean of 106 fields, 1 and 6 hours, 8,001 columns, six seasons; 15
// fields' grew, none by more than a fifth: profiles/fp32_step_error_8001x6h.md).
// Sums and products are regrouped, nothing else: every value keeps the precision it
// had (the canopy island double, the rest float).
#pragma once
#include "ibis_phase.cuh"

namespace ibis {

using Par32 = DevParams<float>;
using Col32 = Col<float>;
using Forc32 = Forc<float>;
using Stat32 = Stat<float>;

__device__ __forceinline__ F2 stat2(const Stat32& S, int p, int k) { return F2(S(p, k), S(p, k + 1)); }

// ===========================================================================
// radiation: both bands of a story at once (physics/radiation.py)
// ===========================================================================

struct TwoStr2 {
    F2 abvegd, abvegi, refld, refli, fbelid, fbelii;
    float fbeldd;
    float term[5], h;   // of the visible band
    float om;           // of the visible band
};

__device__ __forceinline__ F2 tiny30_2(const F2& v) { return F2(tiny30(v.lo()), tiny30(v.hi())); }

// twoset (radiation.py:75-177) and twostr (radiation.py:180-313) of one story by
// day; y: its wet fraction less the liquid, os: that fraction times the snow's
// scattering weight; st: 0 lower, 1 upper.
template <int st>
__device__ __forceinline__ TwoStr2 two_stream2(float cosz, float k, float xai, const F2& asd, const F2& asi, float y,
                                               float o, float eps, const Par32& P) {
    const float ov = P.oriev[st], oh = P.orieh[st], orand = 1.0f - ov - oh;
    const float ztab = 0.5f - cosz * (1.0f / 3.0f);
    const F2 rho(P.rho2[st]), tau(P.tau2[st]);
    const float dry = 1.0f - y, ah = 0.5f * ov + oh;
    const F2 ys = F2(P.osno2) * (y * o);
    const F2 om = mx2((rho + tau) * dry + ys, 1e-12f);
    const F2 rdry = dry * rcp2(om), ysh = ys * 0.5f * rcp2(om);
    const F2 betad = (rho * (ah + orand * (1.0f - ztab)) + tau * (0.5f * ov + orand * ztab)) * rdry + ysh;
    const F2 betai = (rho * (ah + orand * float(2.0 / 3.0)) + tau * (0.5f * ov + orand * float(1.0 / 3.0))) * rdry + ysh;
    const F2 c = om * betai, b = 1.0f - om + c;
    const F2 t0 = (1.0f - om) * (b + c);
    const F2 q = sq2(mx2(t0, 0.0f));
    F2 p(k);
    {
        const float ql = q.lo(), qh = q.hi(), near = 0.001f * k;
        p = F2(ab(k - ql) < near ? (k >= ql ? 1.001f : 0.999f) * k : k,
               ab(k - qh) < near ? (k >= qh ? 1.001f : 0.999f) * k : k);
    }
    const F2 c0 = om * p, d = c0 * betad, f = c0 - d;
    const F2 rs = rcp2(tiny30_2(p * p - t0));
    const F2 ud1 = b - c * rcp2(mx2(asd, 1e-12f)), ui1 = b - c * rcp2(mx2(asi, 1e-12f));
    const F2 ud2 = b - c * asd, ui2 = b - c * asi, ud3 = f + c * asd;
    const F2 s1 = ex2(q * (-xai));
    const float s2 = ex(-k * xai);
    const F2 rw = rcp2(mx2(s1, 1e-30f));
    const F2 p1 = b + q, p2 = b - q, p3 = b + p;
    const F2 dm = (ud1 - q) * rw, dp = (ud1 + q) * s1;
    const F2 im = (ui1 - q) * rw, ip = (ui1 + q) * s1;
    const F2 em = (ud2 - q) * s1, ep = (ud2 + q) * rw;
    const F2 gm = (ui2 - q) * s1, gp = (ui2 + q) * rw;
    const F2 rdd1 = rcp2(tiny30_2(p1 * dm - p2 * dp)), rdi1 = rcp2(tiny30_2(p1 * im - p2 * ip));
    const F2 rdd2 = rcp2(tiny30_2(ep - em)), rdi2 = rcp2(tiny30_2(gp - gm));
    const F2 h1s = (d * (p - b) - c * f) * rs;
    const F2 rw2 = (d - c - h1s * (ud1 + p)) * s2;
    const F2 t = d - h1s * p3;
    const F2 h2 = (t * dm - p2 * rw2) * rdd1, h3 = (p1 * rw2 - t * dp) * rdd1;
    const F2 h4s = (f * p3 + c * d) * rs;    // -h4 / sigma
    const F2 rw3 = (ud3 + h4s * (ud2 - p)) * s2;
    const F2 h5 = (h4s * ep - rw3) * rdd2, h6 = (rw3 - h4s * em) * rdd2;
    const F2 h7 = c * im * rdi1, h8 = c * ip * rdi1;                // h8: -h8
    const F2 h9 = gp * rdi2, h10 = gm * rdi2;                       // h10: -h10
    TwoStr2 r;
    r.fbeldd = s2;
    r.fbelid = h5 * s1 + h6 * rw - h4s * s2;
    r.fbelii = h9 * s1 - h10 * rw;
    r.refld = h1s + h2 + h3;
    r.refli = h7 - h8;
    const bool bare = xai < eps;
    const F2 zero(0.0f);
    r.abvegd = sel2(bare, zero, mx2(1.0f - r.refld - ((1.0f - asd) * s2 + (1.0f - asi) * r.fbelid), 0.0f));
    r.abvegi = sel2(bare, zero, mx2(1.0f - r.refli - (1.0f - asi) * r.fbelii, 0.0f));
    r.om = om.lo();
    r.h = q.lo();
    r.term[0] = k * (1.0f - (h4s.lo() + h1s.lo()));
    r.term[1] = r.h * (h5.lo() - h2.lo());
    r.term[2] = r.h * (h9.lo() - h7.lo());
    r.term[3] = r.h * (h3.lo() - h6.lo());
    r.term[4] = r.h * (h10.lo() - h8.lo());
    return r;
}

// The direct-beam extinction of one story (the gdir of twoset over cos z)
template <int st>
__device__ __forceinline__ float beam_k(float cosz, const Par32& P) {
    const float ov = P.oriev[st], oh = P.orieh[st];
    const float gdir = ov * float(2.0 / 3.1415927) * sq(mx(0.0f, 1.0f - cosz * cosz)) + oh * cosz +
                       (1.0f - ov - oh) * 0.5f;
    return gdir / mx(cosz, 0.01f);
}

// solsur + solalb + solarf, then irrad (radiation.py:316-761).  With the sun down
// the two-stream solution is the trivial one (no scattering, no beam): nothing is
// absorbed and the scaling coefficients keep only the diffuse term.
__device__ __forceinline__ void radiation(Rad<float>& out, const Col32& c, const Forc32& F, const Stat32& S,
                                          float fwetu, float fwets, float fwetl, float rliqu, float rliqs,
                                          float rliql, const Par32& P) {
    const float eps = P.epsilon;
    const float lai0 = S(IBIS_STAT_LAI, 0), lai1 = S(IBIS_STAT_LAI, 1);
    const float sai0 = S(IBIS_STAT_SAI, 0), sai1 = S(IBIS_STAT_SAI, 1);
    const float fu = S(IBIS_STAT_FU), fl = S(IBIS_STAT_FL), fi = c.fi;
    const float gl = lai0 / mx(lai0 + sai0, eps), gu = lai1 / mx(lai1 + sai1, eps);
    if (F.cosz > 0.0f) {
        const float xu = lai1 / mx(lai1 + sai1, 1e-7f), xl0 = mx(lai0 + sai0, eps), xl1 = mx(lai1 + sai1, eps);
        const float zw = c.wsoi[0] * (1.0f - c.wisoi[0]);
        const float dinc = 1.0f + clip(1.0f - zw * 2.0f, 0.0f, 1.0f);
        const F2 albso = mn2(F2(S(IBIS_STAT_ALBSAV), S(IBIS_STAT_ALBSAN)) * dinc, 0.80f);
        const float us = clip((c.tsno[0] - (P.tmelt - 15.0f)) * float(1.0 / 15.0), 0.0f, 1.0f);
        const F2 x = F2(0.90f, 0.60f) - 0.2f * us;
        const float zfac = mx(0.0f, 1.5f / (1.0f + 4.0f * F.cosz) - 0.5f);
        const F2 albsnd = mn2(x + (1.0f - x) * zfac, 0.99f);
        // lower story over soil and snow
        const float yl = fwetl * (1.0f - rliql);
        const float ol = 0.6f + 0.4f * clip(P.tmelt - c.tl, 0.0f, 1.0f);
        const float kl = beam_k<0>(F.cosz, P), ku = beam_k<1>(F.cosz, P);
        const TwoStr2 lo = two_stream2<0>(F.cosz, kl, xl0, albso, albso, yl, ol, eps, P);
        const float fv = fl * (1.0f - fi), fb = (1.0f - fl) * (1.0f - fi);
        const F2 soil = albso * fb;
        const F2 asd = lo.refld * fv + soil + albsnd * fi, asi = lo.refli * fv + soil + x * fi;
        // upper story over both
        const float yu = xu * (fwetu * (1.0f - rliqu)) + (1.0f - xu) * (fwets * (1.0f - rliqs));
        const float ou = xu * clip((P.tmelt - c.tu) * 10.0f, 0.6f, 1.0f) +
                         (1.0f - xu) * clip((P.tmelt - c.ts) * 10.0f, 0.6f, 1.0f);
        const TwoStr2 up = two_stream2<1>(F.cosz, ku, xl1, asd, asi, yu, ou, eps, P);
        const F2 rd = up.refld * fu + (1.0f - fu) * asd, ri = up.refli * fu + (1.0f - fu) * asi;
        out.asurd[0] = rd.lo(); out.asurd[1] = rd.hi();
        out.asuri[0] = ri.lo(); out.asuri[1] = ri.hi();
        // solarf (radiation.py:450-540)
        const F2 sd(F.sd[0], F.sd[1]), si(F.si[0], F.si[1]);
        const F2 xx = sd * up.abvegd + si * up.abvegi;
        const F2 s3d = sd * (fu * up.fbeldd + (1.0f - fu));
        const F2 s3i = (sd * up.fbelid + si * up.fbelii) * fu + si * (1.0f - fu);
        const F2 xd = s3d * (fl * lo.fbeldd + 1.0f - fl);
        const F2 xi = (s3d * lo.fbelid + s3i * lo.fbelii) * fl + s3i * (1.0f - fl);
        const float xs = xx.sum();
        out.solu = xs * gu;
        out.sols = xs * (1.0f - gu);
        out.soll = (s3d * lo.abvegd + s3i * lo.abvegi).sum();
        out.solg = ((1.0f - albso) * (xd + xi)).sum();
        out.soli = ((1.0f - albsnd) * s3d + (1.0f - x) * s3i).sum();
        const float sdv = sd.lo(), siv = si.lo(), tdv = s3d.lo(), tiv = s3i.lo();
        float c0 = up.term[0] * sdv, c1 = up.term[1] * sdv + up.term[2] * siv, c2 = up.term[3] * sdv + up.term[4] * siv;
        float c3 = c0 + c1 + c2;
        out.scu[0] = c0; out.scu[1] = c1; out.scu[2] = c2; out.scu[3] = c3;
        out.topparu = c3 * gu;
        out.dbeamu = (1.0f - up.om) * ku * sdv;
        c0 = lo.term[0] * tdv;
        c1 = lo.term[1] * tdv + lo.term[2] * tiv;
        c2 = lo.term[3] * tdv + lo.term[4] * tiv;
        c3 = c0 + c1 + c2;
        out.scl[0] = c0; out.scl[1] = c1; out.scl[2] = c2; out.scl[3] = c3;
        out.topparl = c3 * gl;
        out.dbeaml = (1.0f - lo.om) * kl * tdv;
        out.termu6 = ku; out.termu7 = up.h;
        out.terml6 = kl; out.terml7 = lo.h;
    } else {
        out.solu = out.sols = out.soll = out.solg = out.soli = 0.0f;
        out.asurd[0] = out.asurd[1] = out.asuri[0] = out.asuri[1] = 0.0f;
        // no beam and no scattering: light times zero, which still shows a value that is
        // not finite to the leaves' sums
        const float none = 0.0f * F.sd[0] + 0.0f * F.si[0];
        const float su = F.si[0] + none, sl = (1.0f - fu) * F.si[0] + none;
        out.scu[0] = out.scu[2] = out.scl[0] = out.scl[2] = none;
        out.scu[1] = out.scu[3] = su;
        out.scl[1] = out.scl[3] = sl;
        out.topparu = su * gu;
        out.topparl = sl * gl;
        out.dbeamu = out.dbeaml = 0.0f;
        out.termu6 = out.terml6 = 0.0f;
        out.termu7 = out.terml7 = 1.0f;
    }
    // irrad (radiation.py:543-641)
    const F2 eus = ex2(F2(-lai1, -sai1));                       // 1 - emu, 1 - ems
    const float ku1 = eus.lo(), ks1 = eus.hi(), kl1 = ex(-(lai0 + sai0));
    const float emu = 1.0f - ku1, ems = 1.0f - ks1, eml = 1.0f - kl1;
    const float emg = 0.95f;
    F2 ts2(c.tu, c.ts), tg2(c.tg, c.ti);
    ts2 = ts2 * ts2; tg2 = tg2 * tg2;
    ts2 = ts2 * ts2 * P.stef; tg2 = tg2 * tg2 * (emg * P.stef);
    const float tu4 = ts2.lo(), ts4 = ts2.hi(), tl4 = P.stef * quart(c.tl), tg4 = tg2.lo(), ti4 = tg2.hi();
    const float fira = F.fira;
    const float fdown = (1.0f - fu) * fira + fu * (ku1 * ks1 * fira + emu * ks1 * tu4 + ems * ts4);
    const float fdowng = kl1 * fdown + eml * tl4;
    const float fupg = (1.0f - emg) * fdowng + tg4;
    const float fupgb = (1.0f - emg) * fdown + tg4;
    const float fupi = (1.0f - emg) * fdown + ti4;
    const float fup = (1.0f - fi) * (fl * (eml * tl4 + kl1 * fupg) + (1.0f - fl) * fupgb) + fi * fupi;
    out.firb = (1.0f - fu) * fup + fu * (ku1 * ks1 * fup + emu * tu4 + ems * ku1 * ts4);
    out.firu = emu * (ems * ts4 + ks1 * fup + fira - 2.0f * tu4);
    out.firs = ems * (emu * tu4 + fup + ku1 * fira - 2.0f * ts4);
    out.firl = eml * (fdown + fupg - 2.0f * tl4);
    out.firg = fl * (fdowng - fupg) + (1.0f - fl) * (fdown - fupgb);
    out.firi = fdown - fupi;
}

// ===========================================================================
// interception (physics/interception.py): liquid water in the low half, snow in
// the high half of each pair
// ===========================================================================

struct Surf2 {
    F2 w, pr, tp;   // water held, precipitation below and its temperature
    float pflux;
};

// mix of two precipitation streams (the reference's third carries no water here; what its
// temperature, not finite, gives the mix is left_over's)
__device__ __forceinline__ void mix_2(F2& xm, F2& tm, const F2& x1, const F2& t1, const F2& x2, const F2& t2,
                                      float eps) {
    const F2 s = x1 + x2;
    const bool a = ab(s.lo()) >= eps, b = ab(s.hi()) >= eps;
    const F2 zero(0.0f);
    tm = sel2(a, b, (t1 * x1 + t2 * x2) * rcp2(s), zero);
    xm = sel2(a, b, s, zero);
}

// A stream of no water from the canopy air: zero, or not a number from an infinite temperature
__device__ __forceinline__ F2 left_over(float tair, const Par32& P) {
    return 0.0f * F2(mx(tair, P.tmelt), mn(tair, P.tmelt));
}

// steph2o (interception.py:174-260) of one story (st: 0 upper leaves, 1 upper stems, 2 lower)
template <int st>
__device__ __forceinline__ Surf2 intercept2(float tveg, F2 w, float xai, const F2& pr0, const F2& tp, float wliqmax,
                                            float wsnomax, float wliqmin, const Par32& P) {
    const float dt = P.dtime, eps = P.epsilon;
    const float fint = xai >= eps ? (1.0f - ex(-0.5f * xai)) / xai : 0.5f;
    const float xr = xai * P.rdt;
    F2 drip = w * F2(P.drip2[st]) * xai;
    const F2 pf = pr0 * fint;
    w = w * F2(P.kdrip2[st]) + pf * dt;
    Surf2 s;
    s.pflux = (pf * (tveg - tp) * F2(P.water2)).sum();
    const F2 pr = pr0 * (1.0f - xai * fint);
    const F2 m = mn2(w, F2(wliqmax, wsnomax));
    const F2 kept = sel2(m.lo() < wliqmin, m.hi() < P.wsnomin, F2(0.0f), m);
    drip = drip + (w - kept) * xr;
    // freezing of the liquid below, melting of the snow above the melting point
    const float wl = kept.lo(), ws = kept.hi();
    const float mv = tveg < P.tmelt - 1.0e-9f ? wl : (tveg > P.tmelt + 1.0e-9f ? -ws : 0.0f);
    s.pflux = s.pflux + mv * ((P.ch2o - P.cice) * (P.tmelt - tveg) - P.hfus) * P.rdt;
    s.w = F2(wl - mv, ws + mv);
    mix_2(s.pr, s.tp, pr, tp, drip, F2(tveg), eps);
    return s;
}

// twet3 (interception.py:126-171)
__device__ __forceinline__ float wet_bulb32(float tak, float q, float p, const Par32& P) {
    const float ta = tak - P.tmelt;
    float twk = ta * q / mx(qsat(esat(tak), p), 1e-12f) + P.tmelt;
    const float rc = 1.0f / P.cair, h0 = P.hvap + P.cvap * ta;
#pragma unroll 1
    for (int it = 0; it < 20; ++it) {
        const float old = twk - P.tmelt;
        const float hv = h0 - P.ch2o * old;
        const float twb = ta - (hv * rc) * (qsat(esat(twk), p) - q);
        const float nxt = old + 0.2f * (twb - old) + P.tmelt;
        const bool conv = ab(nxt - P.tmelt - old) < 0.02f;
        twk = nxt;
        if (conv) break;
    }
    return twk;
}

// cascade (interception.py:263-357)
template <typename Q>
__device__ __forceinline__ void cascade32(Casc<float>& o, const Col32& c, const Forc32& F, const Stat32& S,
                                          const Par32& P, const Q& q) {
    const float eps = P.epsilon;
    const float fu = S(IBIS_STAT_FU), fl = S(IBIS_STAT_FL);
    const bool rains = ab(F.rain) >= eps, snows = ab(F.snow) >= eps;
    float tw = P.tmelt;
    // the wet-bulb temperature is only the rain's
    if (rains && F.ta > P.tmelt + 1.0e-9f) tw = wet_bulb32(F.ta, F.qa, F.ps, P);
    const F2 zero(0.0f);
    const F2 pr = sel2(rains, snows, F2(F.rain, F.snow), zero);
    const F2 tp = sel2(rains, snows, F2(mx(tw, P.tmelt), mn(F.ta, P.tmelt)) + left_over(c.t12, P), zero);
    const Surf2 u = intercept2<0>(c.tu, F2(c.wliqu, c.wsnou), 2.0f * S(IBIS_STAT_LAI, 1), pr, tp, q.wliqumax(),
                                  P.wsnoumax, q.wliqmin(), P);
    const Surf2 s = intercept2<1>(c.ts, F2(c.wliqs, c.wsnos), 2.0f * S(IBIS_STAT_SAI, 1), u.pr, u.tp, q.wliqsmax(),
                                  P.wsnosmax, q.wliqmin(), P);
    F2 pl, tl, pg, tg;
    mix_2(pl, tl, s.pr * fu, s.tp, pr * (1.0f - fu), tp + left_over(c.t34, P), eps);
    const Surf2 l = intercept2<2>(c.tl, F2(c.wliql, c.wsnol), 2.0f * (S(IBIS_STAT_LAI, 0) + S(IBIS_STAT_SAI, 0)), pl,
                                  tl, q.wliqlmax(), P.wsnolmax, q.wliqmin(), P);
    mix_2(pg, tg, l.pr * fl, l.tp, pl * (1.0f - fl), tl, eps);
    o.rainl = pl.lo(); o.snowl = pl.hi(); o.trainl = tl.lo(); o.tsnowl = tl.hi();
    o.raing = pg.lo(); o.snowg = pg.hi(); o.traing = tg.lo(); o.tsnowg = tg.hi();
    o.wliqu = u.w.lo(); o.wliqs = s.w.lo(); o.wliql = l.w.lo();
    o.wsnou = u.w.hi(); o.wsnos = s.w.hi(); o.wsnol = l.w.hi();
    o.pfluxu = u.pflux; o.pfluxs = s.pflux; o.pfluxl = l.pflux;
}

// ===========================================================================
// aerodynamics (physics/canopy_exchange.py:192-426): the lower story in the low
// half, the upper in the high half of each pair
// ===========================================================================

// What the three passes of turcof share.
//
// The exponential wind profile inside one canopy story (canopy_exchange.py:365-392)
// is in closed form.  With E = exp(h) the reference forms
// y = ((x+1)E + (x-1)/E) / ((x+1)E - (x-1)/E) and then the profile coefficients from
// y + 1 and y - 1.  In float32, y rounds to 1 once E passes ~3e3 (a dense canopy), so
// (y - 1) keeps no correct digit and the wind at the story's bottom, proportional to
// (y - 1) E, comes out wrong by O(1).  With D = 2x sinh h + 2 cosh h (the reference's
// denominator) the same quantities are
//   y = (x cosh h + sinh h) / (x sinh h + cosh h),
//   a = k (x+1) E,  b = k (x-1)/E,  k = tau / (D bd),
//   a + b = 2k (x cosh h + sinh h),  a/E^.5 + b E^.5 = 2k (x cosh h/2 + sinh h/2),
//   a/E + b E = 2k x,  bd (a/E - b E) = 2 tau / D.
// The lower story's profile depends on nothing a pass changes, so all of it is formed
// here; of the upper story's, x changes with the stability of the layer below.
struct alignas(8) Aero32 {
    F2 gdz;          // 2 g dz of the two layers the stability corrections act on
    F2 alt;          // log heights of their tops (lower layer: alog2, upper: aloga)
    F2 c3;           // lower profile: (u3, u34)**2 over taul
    float c4;        // u4**2 over taul
    float kca, kb, kd, ke;            // conductance factors: to the air, upper, between the stories, lower
    float rhoa, ua, ht;               // ht: ta tfac (1 + 0.622 qa)
    float alogl, alog1;               // alogl after the first pass
    float xu0, rbdu, sh, ch, sh2, ch2;   // upper profile: x sm, 1/bd, sinh and cosh of h and h/2
};

// What a pass of turcof carries to the next
struct Turc {
    F2 sm, sh;        // stability corrections of the lower and upper layer
    F2 alb;           // log heights of the bottoms: alogl, alogu
    float u2;
};

__device__ __forceinline__ void aero_geometry32(Aero32& A, Turc& tc, float& cp, const Forc32& F, const Stat32& S, float fi,
                                                const Par32& P) {
    const F2 ztop = stat2(S, IBIS_STAT_ZTOP, 0), zbot = stat2(S, IBIS_STAT_ZBOT, 0);
    const float fu = S(IBIS_STAT_FU), fl = S(IBIS_STAT_FL), z0soi = S(IBIS_STAT_Z0SOI);
    const float pa = F.ps * 0.999f;
    const float rhoa = pa / (P.rair * F.ta * (1.0f + float((double)P.rvap / (double)P.rair - 1.0) * F.qa));
    A.rhoa = rhoa;
    cp = P.cair * (1.0f + float((double)P.cvap / (double)P.cair - 1.0) * F.qa);
    const float za = mx((F.ps - pa) / (rhoa * P.grav), ztop.hi() + 1.0f);
    const F2 leaf = (stat2(S, IBIS_STAT_LAI, 0) + stat2(S, IBIS_STAT_SAI, 0)) * 2.0f * F2(fl * (1.0f - fi), fu);
    const F2 x = mn2(leaf * F2(P.ralai2), 3.0f);
    const F2 x1 = mn2(x, 1.0f);
    const F2 rw = mx2(ztop - zbot, 0.01f), rrw = rcp2(rw);
    const F2 cveg = mx2(x, 1e-5f) * 0.4f * rrw;
    const F2 rdveg = mx2(mx2(x, x * x), 1e-5f) * 10.0f * rrw;     // 1 / dveg
    const F2 bveg = sq2(cveg * 2.0f * rdveg);
    const F2 bd = bveg * 0.5f * rcp2(rdveg);
    // heights: lower story top and bottom z3, z4, upper z1, z2
    const float r3 = (1.0f - x1.lo()) * (mx(z0soi, P.z0sno) + 0.01f);
    const float z3 = x1.lo() * ztop.lo() + r3, z4 = x1.lo() * zbot.lo() + r3;
    const float r1 = (1.0f - x1.hi()) * (z3 + 0.01f);
    const float z1 = x1.hi() * ztop.hi() + r1, z2 = x1.hi() * zbot.hi() + r1;
    const float displ = x1.lo() * 0.7f * z3;
    const float dispu = x1.hi() * 0.7f * z1 + (1.0f - x1.hi()) * displ;
    const F2 dz(z3 - z4, z1 - z2);
    const F2 h = bveg * dz;
    const float alogav = (1.0f - fi) * lg(z0soi) + fi * lg(P.z0sno);
    const float alog4 = lg(mx(z4, mx(1.1f * z0soi, 1.1f * P.z0sno)));
    const F2 l32 = lg2(F2(z3 - displ, z2 - displ)), l1a = lg2(F2(z1 - dispu, za - dispu));
    const float alog3 = l32.lo(), alog2 = l32.hi(), alog1 = l1a.lo(), aloga = l1a.hi();
    A.alog1 = alog1;
    A.alt = F2(alog2, aloga);
    tc.alb = lg2(mx2(dz * 0.1f, 0.01f));
    tc.sm = tc.sh = F2(1.0f);
    A.gdz = mx2(F2(z2 - z3, za - z1), 0.0f) * (2.0f * P.grav);
    tc.u2 = F.ua * ex(-0.5f * h.hi());
    A.ua = F.ua;
    A.ht = F.ta * P.tfac * (1.0f + 0.622f * F.qa);
    // sinh and cosh of h/2 from expm1, of h by doubling (no cancellation)
    const F2 e = F2(em1(0.5f * h.lo()), em1(0.5f * h.hi()));
    const F2 em = e * rcp2(1.0f + e);                    // 1 - exp(-h/2)
    const F2 sh2 = (e + em) * 0.5f, ch2 = 1.0f + e * em * 0.5f;
    const F2 sh = sh2 * ch2 * 2.0f, ch = 1.0f + sh2 * sh2 * 2.0f;
    // lower profile: the same in every pass
    const float rvk = 1.0f / P.vonk;
    float v = (alog4 - alogav) * rvk;
    const float bdl = bd.lo(), rbdl = 1.0f / bdl, xl = (v * v) * bdl;
    const float nl = xl * ch.lo() + sh.lo(), dl = xl * sh.lo() + ch.lo(), rdl = 1.0f / dl;
    const float alogl = alog3 - P.vonk * sq(nl * rdl * rbdl);
    A.alogl = alogl;
    const float kl = 0.5f * rdl * rbdl;
    A.c3 = F2(nl, xl * ch2.lo() + sh2.lo()) * (2.0f * kl);
    A.c4 = 2.0f * kl * xl;
    v = (alog2 - alogl) * rvk;
    A.xu0 = (v * v) * bd.hi();
    A.sh = sh.hi(); A.ch = ch.hi(); A.sh2 = sh2.hi(); A.ch2 = ch2.hi();
    A.rbdu = 1.0f / bd.hi();
    const float rr = 1.0f / rhoa;
    A.kca = F.ua * P.vonk2 * rhoa / (aloga - alog1);
    // the layers' mid heights are halfway: z1 - z12 = z12 - z2 = (z1 - z2) / 2
    A.kb = rdveg.hi() * (z1 - z2) * rr;
    A.ke = rdveg.lo() * (z3 - z4) * rr;
    A.kd = (alog2 - alogl) * (alog2 - alog3) * rr / P.vonk2;
}

// fstrat (canopy_exchange.py:287-326) of both layers and turcof (:333-426)
__device__ __forceinline__ void transfer32(Trans<float>& T, Turc& c, const Aero32& A, float t12, float t34, float q12,
                                           float q34, bool first, const Par32& P) {
    const float h12 = t12 * (1.0f + 0.622f * q12), h34 = t34 * (1.0f + 0.622f * q34);
    const F2 zht(h12, A.ht), zhb(h34, h12);
    const F2 u(c.u2, A.ua);
    const F2 rich = clip2(A.gdz * (zht - zhb) * rcp2((zht + zhb) * (u * u)), -2.0f, 1.0f);
    // unstable (rich <= 0): 1 - 10 rich/E, 1 - 15 rich/E with E = 1 + 75 (vonk/xm)^2 e^(xm/2) sqrt(-rich);
    // stable: 1/(1 + 10 rich/r), 1/(1 + 15 rich r) with r = sqrt(1 + 5 rich)
    const bool a0 = rich.lo() <= 0.0f, a1 = rich.hi() <= 0.0f;
    const F2 a = abs2(rich);
    const F2 r = sq2(sel2(a0, a1, a, 1.0f + a * 5.0f));
    const F2 xm = mx2(A.alt - c.alb, 0.5f);
    const F2 vx = P.vonk * rcp2(xm);
    const F2 E = 1.0f + (vx * vx) * ex2(xm * 0.5f) * r * 75.0f;
    const F2 dm = sel2(a0, a1, E, r + a * 10.0f), dh = sel2(a0, a1, E, 1.0f + a * r * 15.0f);
    const F2 smn = sel2(a0, a1, E + a * 10.0f, r) * rcp2(dm), shn = sel2(a0, a1, E + a * 15.0f, F2(1.0f)) * rcp2(dh);
    c.sm = sel2(first, smn, (smn + c.sm) * 0.5f);
    c.sh = sel2(first, shn, (shn + c.sh) * 0.5f);
    // upper wind profile
    const float xu = A.xu0 / c.sm.lo();
    const float nu = xu * A.ch + A.sh, rd = 1.0f / (xu * A.sh + A.ch);
    const float alogu = A.alog1 - P.vonk * sq(nu * rd * A.rbdu);
    const float aloga = A.alt.hi();
    const float v = A.ua * P.vonk / (aloga - alogu);
    const float taul = (v * v) * c.sm.hi() * rd;                 // tauu / D
    const float ku = taul * A.rbdu;
    const F2 u1 = mx2(sq2(mx2(F2(nu, xu * A.ch2 + A.sh2) * ku, 0.0f)), 0.01f);
    const F2 u3 = mx2(sq2(mx2(A.c3 * taul, 0.0f)), 0.01f);
    const F2 ue = mx2(sq2(mx2(F2(ku * xu, taul * A.c4), 0.0f)), 0.01f);   // u2, u4
    const float u12 = u1.hi(), nu2 = ue.lo(), u34 = u3.hi(), u4 = ue.hi();
    const float ca = mn(P.cdmax * A.rhoa, A.kca * c.sh.hi() / (aloga - alogu));
    const float ub = u1.lo() + u12;
    T.cu = ca * ub / (ub + A.kb * ca);
    T.cl = 1.0f / (A.kb / (u12 + nu2) + A.kd / (nu2 * c.sh.lo()) + A.ke / (u3.lo() + u34));
    const float q1 = A.rhoa * sq(u12);
    T.su = q1 * P.ksu;
    T.ss = q1 * P.kss;
    T.sl = A.rhoa * sq(u34) * P.ksl;
    const F2 s0 = A.rhoa * (F2(0.004f, 0.003f) + F2(0.012f, 0.010f) * u4);
    const float uf = u34 + u4;
    const F2 sg = s0 * uf * rcp2(uf + A.ke * s0);
    T.sg = sg.lo();
    T.si = sg.hi();
    c.u2 = nu2;
    c.alb = F2(A.alogl, alogu);
}

// impexp (canopy_exchange.py:433-450) of two surfaces
__device__ __forceinline__ F2 weight_veg2(const F2& t, const F2& ch, const F2& wliq, const F2& wsno, const F2& prev,
                                          const Par32& P) {
    const F2 h = ch * (t - P.tmelt);
    const F2 z = abs2(h);
    const float lim = P.epsilon + 1.0e-8f;
    const F2 nw = 1.0f - mn2(sel2(h.lo() > 0.0f, h.hi() > 0.0f, wsno, wliq) * P.hfus * rcp2(mx2(z, P.epsilon)), 1.0f);
    return (prev + sel2(z.lo() > lim, z.hi() > lim, nw, F2(1.0f))) * 0.5f;
}

// ===========================================================================
// stomata (physics/stomata.py:198-1080): the leaves of a story in pairs
// ===========================================================================

// farquhar's smoothed minimum of two rates (quadratic with curvature theta); `least` is
// the reference's 1e-15 beside the root, in the rates' own units
constexpr float kLeast = 1.0e-15f;
__device__ __forceinline__ F2 colimit2(const F2& j1, const F2& j2, float theta, float rtheta, float least) {
    const F2 b = j1 + j2, c = j1 * j2;
    const F2 q = (b + sq2(mx2(b * b - c * (4.0f * theta), 0.0f))) * 0.5f + least;
    return mn2(q * rtheta, c * rcp2(q));
}

__device__ __forceinline__ float colimit1(float j1, float j2, float theta, float rtheta, float least) {
    const float b = j1 + j2, c = j1 * j2;
    const float q = 0.5f * (b + sq(mx(b * b - c * (4.0f * theta), 0.0f))) + least;
    return mn(q * rtheta, c / q);
}

// gross C3 rate from the light-, enzyme- and export-limited rates
__device__ __forceinline__ F2 c3_gross(const F2& je, const F2& jc, const F2& js, const Par32& P, float least = kLeast) {
    return colimit2(colimit2(je, jc, P.theta3, P.rtheta3, least), js, P.beta3, P.rbeta3, least);
}
__device__ __forceinline__ float c4_gross(float je, float jc, float ji, const Par32& P, float least = kLeast) {
    return colimit1(colimit1(je, jc, P.theta4, P.rtheta4, least), ji, P.beta4, P.rbeta4, least);
}

// Temperature functions of the two canopies' leaves (upper low half, lower high half)
struct Kin2 { F2 gst, kco, vm3; float vm4; };

__device__ __forceinline__ Kin2 kinetics2(const F2& tleaf, const Par32& P) {
    const F2 rw = 3.47e-03f - rcp2(tleaf);
    const F2 e45 = ex2(rw * 4500.0f);
    Kin2 k;
    k.gst = e45 * (P.o2conc * 0.5f / P.tau15);                    // o2 / (2 tau)
    k.kco = ex2(rw * 6000.0f) * P.kc15 + e45 * (P.kc15 * P.o2conc / P.ko15);   // kc (1 + o2 / ko)
    const F2 tc = tleaf - 273.16f;
    const F2 base = ex2(rw * 3500.0f), hot = 1.0f + ex2((tc - 50.0f) * 0.40f);
    const F2 cold = ex2((5.0f - tc) * 0.40f);
    k.vm3 = base * rcp2((1.0f + cold) * hot);
    k.vm4 = base.hi() / ((1.0f + cold.hi() * 7.38905609893065f) * hot.hi());   // e^(0.4 (10 - 5))
    return k;
}

// One story's constants of a pass (scale: the light scaling or, with the sunlit/shaded
// split, the smallest rate of the canopy's in units per leaf area)
struct Story {
    float gmn, rgb, rh, stress, scale, s, par, fw;
};

// Ball-Berry update of two leaves' (cs, gs, ci)
__device__ __forceinline__ void ball_berry2(F2& cs, F2& gs, F2& ci, const F2& an, const Story& t, const F2& m,
                                            const F2& b0, const F2& gmin, const Par32& P) {
    const F2 b0s = b0 * t.stress;
    const F2 csn = mx2((cs + P.co2conc - an * t.rgb) * 0.5f, t.gmn);
    F2 gsn = (gs + m * an * t.rh * rcp2(csn) + b0s) * 0.5f;
    gsn = mx2(gsn, mx2(gmin, b0s));
    ci = clip2((ci + csn - an * 1.6f * rcp2(gsn)) * 0.5f, t.gmn, P.cimax);
    cs = csn;
    gs = gsn;
}

// total conductance to water vapour of two leaves from the scaled net rate
__device__ __forceinline__ F2 leaf_conductance2(const F2& anc, const Story& t, const F2& m, const F2& b0,
                                                const F2& gmin, const Par32& P) {
    const F2 b0s = b0 * t.stress;
    const F2 csc = mx2(P.co2conc - anc * t.rgb, t.gmn);
    const F2 gsc = mx2(mx2(gmin, b0s), m * anc * t.rh * rcp2(csc) + b0s);
    return gsc * t.s * rcp2(gsc + t.s * float(1.0 / 0.029));      // 1 / (1/s + (1/0.029)/g)
}

// The light and capacity of a story's sunlit and shaded leaves (sunshade_canopy), per
// leaf area: (sunlit, shaded) pairs
struct Sun4 { F2 p, v; };

// Two C3 leaves of a story: rates, Ball-Berry, scaled rates and conductance.
// vn, cm: nominal vmax and slope; jf, cap, fcap: the IBIS 3.0 factors.
template <bool SUN, bool X3>
__device__ __forceinline__ F2 c3_pair(F2& cs, F2& gs, F2& ci_, F2& ag_o, F2& an_o, const Story& t, float gst,
                                      float kco, float vm3, const F2& vn, const F2& cm, const F2& gamma, const F2& b0,
                                      const F2& gmin, const Sun4& ss, const F2& jf, bool cap, float fcap,
                                      const Par32& P) {
    const F2 ci = clip2(ci_, t.gmn, P.cimax);
    const F2 vmax = vn * (vm3 * t.stress);
    const F2 rd = gamma * vn * vm3;
    const F2 X = (ci - gst) * rcp2(ci + 2.0f * gst) * (4.59e-06f * P.alpha3);
    const F2 Y = vmax * ((ci - gst) * rcp2(ci + kco)), Z = vmax * float(1.0 / 2.2);
    F2 Xf = X;
    if constexpr (X3) Xf = X * jf;
    F2 ag, an;
    if constexpr (SUN) {
        ag = c3_gross(Xf * ss.p.lo(), Y * ss.v.lo(), Z * ss.v.lo(), P, t.scale) +
             c3_gross(Xf * ss.p.hi(), Y * ss.v.hi(), Z * ss.v.hi(), P, t.scale);
        an = ag - rd * ss.v.sum();
    } else {
        ag = c3_gross(Xf * t.par, Y, Z, P);
        an = ag - rd;
    }
    ci_ = ci;
    ball_berry2(cs, gs, ci_, an, t, cm, b0, gmin, P);
    if constexpr (!SUN) {
        if (X3 && cap) {
            ag = c3_gross(Xf * (t.par * t.scale), Y * fcap, Z * fcap, P);
            an = ag - rd * fcap;
        } else {
            ag = ag * t.scale;
            an = an * t.scale;
        }
    }
    ag_o = ag * (1.0f - t.fw);
    an_o = an * (1.0f - t.fw);
    return leaf_conductance2(an, t, cm, b0, gmin, P);
}

// canopy_scaling (stomata.py:442-512) of both stories.  Nothing it reads changes
// between the hour's passes except its own carried means, and those only by day, when
// it does not read them: so it is formed once, and the means advanced once per pass.
__device__ __forceinline__ F2 light_scaling2(const Rad<float>& Rd, const F2& lai, const F2& sai, Col32& c,
                                             bool leaf_only, const Par32& P) {
    const F2 toppar(Rd.topparu, Rd.topparl), k(Rd.termu6, Rd.terml6), h(Rd.termu7, Rd.terml7);
    const F2 sc0(Rd.scu[0], Rd.scl[0]), sc12(Rd.scu[1] - Rd.scu[2], Rd.scl[1] - Rd.scl[2]), sc3(Rd.scu[3], Rd.scl[3]);
    const F2 ext = clip2((k * sc0 + h * sc12) * rcp2(mx2(sc3, P.epsilon)), 0.1f, 10.0f);
    const F2 pxai = ext * (lai + sai), plai = ext * lai;
    const F2 sday = (1.0f - ex2(pxai * -1.0f)) * rcp2(mx2(leaf_only ? pxai : plai, P.epsilon));
    F2 as(c.a10su, c.a10sl), ad(c.a10du, c.a10dl);
    const F2 snight = as * rcp2(mx2(ad, P.epsilon));
    const float z = P.zweight;
    const F2 tz = toppar * (1.0f - z), ts = sday * tz;
#pragma unroll
    for (int it = 0; it < 3; ++it) {
        as = as * z + ts;
        ad = ad * z + tz;
    }
    const bool hu = plai.lo() > 0.0f, hl = plai.hi() > 0.0f, du = toppar.lo() > 10.0f, dl = toppar.hi() > 10.0f;
    if (hu && du) { c.a10su = as.lo(); c.a10du = ad.lo(); }
    if (hl && dl) { c.a10sl = as.hi(); c.a10dl = ad.hi(); }
    return sel2(hu, hl, sel2(du, dl, sday, snight), F2(0.0f));
}

// ===========================================================================
// What the three canopy passes share, kept in shared memory for the hour
//
// The passes read some eighty values that none of them changes.  In registers they
// cannot stay (the double canopy solve needs the file), and spilled they miss: eight
// warps' local frames are three times what L1 has left, and two of three local loads
// went to L2, the largest stall of the kernel.  Here they are read in 64-bit words at
// shared-memory latency.  A record is an odd number of 64-bit words, so a warp's
// loads of one word touch every bank once per half-warp.
// ===========================================================================

template <bool SUN, bool X3>
struct HourExtra {};
template <>
struct alignas(8) HourExtra<true, false> { Sun4 su, sl; };
// with the IBIS 3.0 switches also the big leaves' nominal vmax, slopes and light
// factors (C4 grass last), the capacity integrals (upper, lower) and the upper and shrub
// leaves' area per capacity (negative: shares by area)
struct alignas(8) Leaves3 { F2 vnl, cmu, cml, jfu, jfl, cap; float vn4, cm4, jf4, rcap[3]; };
template <>
struct alignas(8) HourExtra<false, true> : Leaves3 {};
template <>
struct alignas(8) HourExtra<true, true> : Leaves3 { Sun4 su, sl; };

// Pairs: (upper leaves, upper stems) `_us`, (lower canopy, ground) `_lg`, (ground, snow) `_gi`
struct alignas(8) TvHour {
    F2 x_us, ch_us, ch_lg, wl_us, ws_us, wl_lg, ws_lg, rl_us, fw_us, frad_us, pf_us;
    F2 hv_gi, sol_gi, fir_gi, zir_gi;
    F2 stress, toppar, scale;       // (upper, lower)
    F2 vnu;                         // nominal vmax of the upper big leaves
    float xl, rliql, fwetl, fradl, pfluxl, psig, cp, firb, qa, ps, fi, fr3, fr4, unused;
    double betaw;                   // soil-surface wetness factor
    double fb, fc, fs, rlai;        // leaf-area shares of the big leaves; lai0 / (lai0 + sai0)
    double pg0, bg0, pi0, bi0;      // what the ground's and snow's rows have besides the air: pivot, right-hand side
    double hv0, hs0, tap;           // latent heats at 0 K extrapolated; ta tfac
};

template <bool SUN, bool X3>
struct alignas(8) HourWords : HourExtra<SUN, X3> {
    Aero32 A;
    TvHour X;
};

template <bool EVEN>
struct WordPad {};
template <>
struct WordPad<true> { unsigned long long pad; };
template <bool SUN, bool X3>
struct HourScratch : HourWords<SUN, X3>, WordPad<(sizeof(HourWords<SUN, X3>) / 8) % 2 == 0> {};

// One pass of stomata over the five big leaves (see the template in ibis_canopy.cuh)
template <bool SUN_U, bool SUN_L, typename Y, typename Q>
__device__ __forceinline__ void stomata32(Stom<float>& o, Col32& c, float tu, float tl, const F2& qair,
                                          const F2& qs_air, float su, float sl, const Y& y, const Par32& P,
                                          const Q& q) {
    constexpr bool X3 = Q::x3;
    const TvHour& X = y.X;
    const Kin2 K = kinetics2(F2(tu, tl), P);
    const F2 rh = mx2(qair * rcp2(mx2(qs_air, P.epsilon)), 0.30f);
    const F2 rgb = rcp2(clip2(F2(su, sl) * 25.5f, 0.1f, 10.0f));
    const F2 stress = X.stress, toppar = X.toppar, scale = X.scale;
    const bool cap = X3 && (P.flags & IBIS_FLAG_CAP_SCALE_L) != 0 && !SUN_L;
    // ---------------- upper canopy: broadleaf and conifer
    {
        const Story t{1.05f * K.gst.lo(), rgb.lo(), rh.lo(), stress.lo(), scale.lo(), su, toppar.lo(), X.fw_us.lo()};
        F2 cs(c.cs_u[0], c.cs_u[1]), gs(c.gs_u[0], c.gs_u[1]), ci(c.ci_u[0], c.ci_u[1]), ag, an, cm, jf(1.0f);
        Sun4 ss{};
        float fcap = 0.0f;
        bool capu = false;
        if constexpr (X3) {
            cm = y.cmu;
            jf = y.jfu;
            fcap = y.cap.lo();
            capu = !SUN_U && (P.flags & IBIS_FLAG_CAP_SCALE_U) != 0;
        } else {
            cm = F2(q.coefm2(0));
        }
        if constexpr (SUN_U) ss = y.su;
        const F2 tc = c3_pair<SUN_U, X3>(cs, gs, ci, ag, an, t, K.gst.lo(), K.kco.lo(), K.vm3.lo(), X.vnu, cm,
                                         F2(P.gam2[0]), F2(P.b02[0]), F2(P.gmin2[0]), ss, jf, capu, fcap, P);
        c.cs_u[0] = cs.lo(); c.cs_u[1] = cs.hi(); c.gs_u[0] = gs.lo(); c.gs_u[1] = gs.hi();
        c.ci_u[0] = ci.lo(); c.ci_u[1] = ci.hi();
        o.ag_u[0] = ag.lo(); o.ag_u[1] = ag.hi(); o.an_u[0] = an.lo(); o.an_u[1] = an.hi();
        o.tcub = tc.lo();
        o.tcuc = tc.hi();
    }
    // ---------------- lower canopy: shrub (group 2) and C3 grass (group 4), then C4 grass (group 3)
    {
        const Story t{1.05f * K.gst.hi(), rgb.hi(), rh.hi(), stress.hi(), scale.hi(), sl, toppar.hi(), X.fwetl};
        F2 cs(c.cs_l[0], c.cs_l[1]), gs(c.gs_l[0], c.gs_l[1]), ci(c.ci_l[0], c.ci_l[1]), ag, an, vn, cm, jf(1.0f);
        float vn4, cm4, jf4 = 1.0f, fcap = 0.0f;
        Sun4 ss{};
        if constexpr (X3) {
            vn = y.vnl; cm = y.cml; jf = y.jfl;
            vn4 = y.vn4; cm4 = y.cm4; jf4 = y.jf4;
            fcap = y.cap.hi();
        } else {
            vn = F2(q.vmaxl2()); cm = F2(q.coefm2(1));
            vn4 = q.vmax(10); cm4 = q.coefm(3);
        }
        if constexpr (SUN_L) ss = y.sl;
        const F2 tc = c3_pair<SUN_L, X3>(cs, gs, ci, ag, an, t, K.gst.hi(), K.kco.hi(), K.vm3.hi(), vn, cm,
                                         F2(P.gam2[1]), F2(P.b02[1]), F2(P.gmin2[1]), ss, jf, cap, fcap, P);
        c.cs_l[0] = cs.lo(); c.cs_l[1] = cs.hi(); c.gs_l[0] = gs.lo(); c.gs_l[1] = gs.hi();
        c.ci_l[0] = ci.lo(); c.ci_l[1] = ci.hi();
        o.ag_l[0] = ag.lo(); o.ag_l[1] = ag.hi(); o.an_l[0] = an.lo(); o.an_l[1] = an.hi();
        o.tcls = tc.lo();
        o.tcl3 = tc.hi();
        // C4 grass
        const float c4 = clip(c.ci_l[2], 0.0f, P.cimax);
        const float vmax = vn4 * K.vm4 * t.stress, rd = P.gamma[3] * vn4 * K.vm4;
        const float xe = 4.59e-06f * P.alpha4 * jf4, ji = 18.0e3f * vmax * c4;
        float ag4, an4;
        if constexpr (SUN_L) {
            ag4 = c4_gross(xe * ss.p.lo(), vmax * ss.v.lo(), ji * ss.v.lo(), P, t.scale) +
                  c4_gross(xe * ss.p.hi(), vmax * ss.v.hi(), ji * ss.v.hi(), P, t.scale);
            an4 = ag4 - rd * ss.v.sum();
        } else {
            ag4 = c4_gross(xe * t.par, vmax, ji, P);
            an4 = ag4 - rd;
        }
        const float b0s = P.coefb[3] * t.stress, gm = mx(P.gsmin[3], b0s), mr = cm4 * t.rh;
        const float csn = mx(1.0e-8f, 0.5f * (c.cs_l[2] + P.co2conc - an4 * t.rgb));
        const float gsn = mx(0.5f * (c.gs_l[2] + mr * an4 / csn + b0s), gm);
        c.ci_l[2] = clip(0.5f * (c4 + csn - 1.6f * an4 / gsn), 0.0f, P.cimax);
        c.cs_l[2] = csn;
        c.gs_l[2] = gsn;
        if constexpr (!SUN_L) {
            if (cap) {
                ag4 = c4_gross(xe * (t.par * t.scale), vmax * fcap, ji * fcap, P);
                an4 = ag4 - rd * fcap;
            } else {
                ag4 = ag4 * t.scale;
                an4 = an4 * t.scale;
            }
        }
        const float csc = mx(1.0e-8f, P.co2conc - an4 * t.rgb);
        const float gsc = mx(gm, mr * an4 / csc + b0s);
        o.tcl4 = gsc * t.s / (gsc + t.s * float(1.0 / 0.029));
        o.ag_l[2] = ag4 * (1.0f - t.fw);
        o.an_l[2] = an4 * (1.0f - t.fw);
    }
}

// ===========================================================================
// turvap: the 9x9 implicit canopy / air / ground / snow system
// (canopy_exchange.py:470-811), in double
// ===========================================================================

struct TvResult {
    float fsena, fsenu, fsens, fsenl, fseng, fseni;
    float fvapuw, fvaput, fvaps, fvaplw, fvaplt, fvapg, fvapi;
    float firg, firi, firb, ginvap, gsuvap, gtrans;
};

// One pass.  Five of the nine unknowns (the three canopy temperatures, ground and
// snow) appear only with the canopy air they touch: x = beta + rho T + sigma Q.
// Eliminating them leaves the 4x4 system of the two air layers' temperature and
// humidity, solved by 2x2 blocks (the layers couple through -cl I).  The full
// elimination it replaces filled 45 entries and divided by nine pivots.
__device__ __forceinline__ void turvap32(double (&W)[9], TvResult& o, const Col32& c, const Trans<float>& T,
                                         const F2& wus, const F2& wlg, float wif, const TvHour& X,
                                         const Stom<float>& st, const Stat32& S, float r34, float q34s, bool last,
                                         const Par32& P) {
    const double eps = (double)P.epsilon, dt = (double)P.dtime;
    const double wu = wus.lo(), ws = wus.hi(), wl = wlg.lo(), wg = wlg.hi(), wi = wif;
    // the temperatures at the hour's start (the column's are not advanced until the passes end)
    const double old[5] = {c.tu, c.ts, c.tl, c.tg, c.ti};
    const double tu = fma(wu, W[0] - old[0], old[0]), ts = fma(ws, W[1] - old[1], old[1]);
    const double tl = fma(wl, W[2] - old[2], old[2]), tg = fma(wg, W[7] - old[3], old[3]);
    const double ti = fma(wi, W[8] - old[4], old[4]);
    const double t34 = W[4], q12 = W[5], q34 = W[6];
    // saturation humidities and their capped derivatives in float, two at a time
    double qu, qs, ql, qg, qi, dqu, dqs, dql, dqg, dqi, dqs1;
    {
        const float ps = X.ps;
        const F2 ta((float)tu, (float)ts), tb((float)tl, (float)tg), tc((float)ti, (float)t34);
        const F2 ea = esat2(ta), eb = esat2(tb);
        const float ei = esat(tc.lo()), ri = 0.622f / mx(ps - ei * float(1.0 - 0.622), ei * 0.622f);
        const F2 ra = sat_quotient2(ea, ps), rb = sat_quotient2(eb, ps), rc(ri, r34);
        const F2 qa_ = ea * ra, qb = eb * rb, qc(ei * ri, q34s);
        const F2 da = mn2(sat_derivative2(ta, qa_, ra), qa_ * 0.1f), db = mn2(sat_derivative2(tb, qb, rb), qb * 0.1f);
        const F2 dc = sat_derivative2(tc, qc, rc);
        qu = qa_.lo(); qs = qa_.hi(); ql = qb.lo(); qg = qb.hi(); qi = qc.lo();
        dqu = da.lo(); dqs = da.hi(); dql = db.lo(); dqg = db.hi(); dqi = mn(dc.lo(), qc.lo() * 0.1f);
        dqs1 = dc.hi();
    }
    const double su = T.su, ss = T.ss, sl = T.sl, sg = T.sg, si = T.si, cu = T.cu, cl = T.cl, cp = X.cp;
    const double qeps = 1.0e-10, hvap = (double)P.hvap;
    // soil-surface humidity factor (canopy_exchange.py:532-572)
    const double hfac = (double)ex(X.psig / (P.rvap * (float)tg));
    const double xd = fma(cp, sg, (double)P.zir * cube(t34));
    const double betas = X.betaw * xd * rcp_nr(fma(hvap * dqs1 * sg, 1.0 - X.betaw, xd));
    const double hfac2 = q34 * rcp_nr(dmax(qg, eps));
    double qgfac = betas > 0.0 ? fma(betas, hfac - hfac2, hfac2) : hfac2;
    if (q34 > qg + qeps) qgfac = 1.0;
    // vapour conductances (canopy_exchange.py:587-618)
    const F2 wet_us = X.wl_us + X.ws_us;
    const double fwux = (q12 > qu + qeps) ? 1.0 : X.fw_us.lo();
    const double fwsx = (q12 > qs + qeps) ? 1.0 : X.fw_us.hi();
    const double fwlx = (q34 > ql + qeps) ? 1.0 : X.fwetl;
    const double suw = dmin(fwux * su, 0.8 * wet_us.lo() * rcp_nr(dmax(dt * (qu - q12), eps)));
    const double ssw = dmin(fwsx * ss, 0.8 * wet_us.hi() * rcp_nr(dmax(dt * (qs - q12), eps)));
    const double slw = dmin(fwlx * sl, 0.8 * (X.wl_lg.lo() + X.ws_lg.lo()) * rcp_nr(dmax(dt * (ql - q34), eps)));
    const double sut = dmax((0.5 - 0.5 * fwux) * (st.tcub * X.fb + st.tcuc * X.fc), 0.0);
    const double slt0 = dmax((0.5 - 0.5 * fwlx) * (st.tcls * X.fs + (double)st.tcl4 * X.fr4 +
                                                    (double)st.tcl3 * X.fr3), 0.0);
    const double slt = slt0 * X.rlai;
    const double hv0 = X.hv0, hs0 = X.hs0;
    const double hvu = fma(-(double)P.ch2o, tu, hv0), hvl = fma(-(double)P.ch2o, tl, hv0), hvs = fma(-(double)P.ch2o, ts, hv0);
    const double hsu = fma(-(double)P.cice, tu, hs0), hsl = fma(-(double)P.cice, tl, hs0), hss = fma(-(double)P.cice, ts, hs0);
    const double suh = fma(suw, fma((double)X.rl_us.lo(), hvu - hsu, hsu), sut * hvu);
    const double ssh = ssw * fma((double)X.rl_us.hi(), hvs - hss, hss);
    const double slh = fma(slw, fma((double)X.rliql, hvl - hsl, hsl), slt * hvl);

    // the five local rows: x = b + r T + s Q (canopy_exchange.py:620-682)
    const double rdt = P.rdt64, fi = X.fi, gi = 1.0 - fi;
    double bu, ru, au, bs, rs, as, bl, rl, al, bg, rg, ag, bi, ri, ai;
    auto leaf = [&](double old0, float chx, double w, double sc, double sh, double qx, double dq, double t, double rad,
                    double& b, double& r, double& a) {
        const double cap = chx * rdt, r2 = sc * cp;
        const double inv = rcp_nr(fma(w, fma(sh, dq, r2), cap));
        b = (fma(old0, cap, rad) - (r2 - w * r2) * t - sh * fma(-w * dq, t, qx)) * inv;
        r = r2 * inv;
        a = sh * inv;
    };
    leaf(old[0], X.ch_us.lo(), wu, su, suh, qu, dqu, tu, (double)X.frad_us.lo() - X.pf_us.lo(), bu, ru, au);
    leaf(old[1], X.ch_us.hi(), ws, ss, ssh, qs, dqs, ts, (double)X.frad_us.hi() - X.pf_us.hi(), bs, rs, as);
    leaf(old[2], X.ch_lg.lo(), wl, sl, slh, ql, dql, tl, (double)X.fradl - X.pfluxl, bl, rl, al);
    const bool bare = (X.x_us.lo() + X.x_us.hi() + X.xl) < P.epsilon;
    {
        const double r1 = sg * cp, r2 = sg * X.hv_gi.lo(), g = r2 * qgfac;
        const double inv = rcp_nr(r1 + fma(g, dqg, X.pg0));
        double b = fma(-g, fma(-dqg, tg, qg), X.bg0);
        // a bare cell's canopy heat goes to the ground (canopy_exchange.py:684-732)
        if (bare)
            b = b + (((double)X.frad_us.lo() - X.pf_us.lo()) * X.x_us.lo() + ((double)X.frad_us.hi() - X.pf_us.hi()) * X.x_us.hi() +
                     ((double)X.fradl - X.pfluxl) * X.xl);
        bg = b * inv; rg = r1 * inv; ag = r2 * inv;
    }
    {
        const double r1 = si * cp, r2 = si * X.hv_gi.hi();
        const double inv = rcp_nr(r1 + fma(r2, dqi, X.pi0));
        bi = fma(-r2, fma(-dqi, ti, qi), X.bi0) * inv;
        ri = r1 * inv; ai = r2 * inv;
    }
    // the 4x4 system of (t12, q12 | t34, q34)
    const double tap = X.tap, qa64 = X.qa;
    double n12, nq12, n34, nq34;
    {
        const double cc = cu + cl;
        double kt = X.x_us.lo() * su, kq = X.x_us.lo() * (suw + sut);
        double mt = wu * kt, mq = wu * kq * dqu;
        double u11 = cc + kt - mt * ru, u12 = -mt * au, f1 = fma(cu, tap, fma(kt - mt, tu, mt * bu));
        double u21 = -mq * ru, u22 = cc + kq - mq * au, f2 = fma(cu, qa64, fma(kq, qu, mq * (bu - tu)));
        kt = X.x_us.hi() * ss; kq = X.x_us.hi() * ssw;
        mt = ws * kt; mq = ws * kq * dqs;
        u11 += kt - mt * rs; u12 -= mt * as; f1 += fma(kt - mt, ts, mt * bs);
        u21 -= mq * rs; u22 += kq - mq * as; f2 += fma(kq, qs, mq * (bs - ts));
        kt = X.xl * sl; kq = X.xl * (slw + slt);
        mt = wl * kt; mq = wl * kq * dql;
        double l11 = cl + kt - mt * rl, l12 = -mt * al, g1 = fma(kt - mt, tl, mt * bl);
        double l21 = -mq * rl, l22 = cl + kq - mq * al, g2 = fma(kq, ql, mq * (bl - tl));
        kt = gi * sg; kq = kt;
        mt = wg * kt; mq = mt * qgfac * dqg;
        l11 += kt - mt * rg; l12 -= mt * ag; g1 += fma(kt - mt, tg, mt * bg);
        l21 -= mq * rg; l22 += kq - mq * ag; g2 += fma(kq * qgfac, qg, mq * (bg - tg));
        kt = fi * si; kq = kt;
        mt = wi * kt; mq = mt * dqi;
        l11 += kt - mt * ri; l12 -= mt * ai; g1 += fma(kt - mt, ti, mt * bi);
        l21 -= mq * ri; l22 += kq - mq * ai; g2 += fma(kq, qi, mq * (bi - ti));
        const double iu = rcp_nr(u11 * u22 - u12 * u21);
        const double h1 = (u22 * f1 - u12 * f2) * iu, h2 = (u11 * f2 - u21 * f1) * iu;
        const double ci = cl * iu, c2 = cl * ci;
        const double s11 = l11 - c2 * u22, s12 = l12 + c2 * u12, s21 = l21 + c2 * u21, s22 = l22 - c2 * u11;
        const double y1 = fma(cl, h1, g1), y2 = fma(cl, h2, g2);
        const double is = rcp_nr(s11 * s22 - s12 * s21);
        n34 = (s22 * y1 - s12 * y2) * is;
        nq34 = (s11 * y2 - s21 * y1) * is;
        n12 = fma(ci, u22 * n34 - u12 * nq34, h1);
        nq12 = fma(ci, u11 * nq34 - u21 * n34, h2);
    }
    if (bare) { n12 = n34 = tap; nq12 = nq34 = qa64; }
    double nu = fma(ru, n12, fma(au, nq12, bu)), ns = fma(rs, n12, fma(as, nq12, bs));
    double nl = fma(rl, n34, fma(al, nq34, bl));
    if (bare) nu = ns = nl = tap;
    const double ng = fma(rg, n34, fma(ag, nq34, bg)), ni = fma(ri, n34, fma(ai, nq34, bi));
    W[0] = nu; W[1] = ns; W[2] = nl; W[3] = n12; W[4] = n34; W[5] = nq12; W[6] = nq34; W[7] = ng; W[8] = ni;

    // flux diagnostics (canopy_exchange.py:746-795), of the last pass only
    if (last) {
        o.fsena = (float)(cp * cu * (tap - n12));
        const double vu = fma(wu, nu - tu, tu), vs = fma(ws, ns - ts, ts), vl = fma(wl, nl - tl, tl);
        const double vg = fma(wg, ng - tg, tg), vi = fma(wi, ni - ti, ti);
        o.fsenu = (float)(cp * su * (vu - n12));
        o.fsens = (float)(cp * ss * (vs - n12));
        o.fsenl = (float)(cp * sl * (vl - n12));
        o.fseng = (float)(cp * sg * (vg - n34));
        o.fseni = (float)(cp * si * (vi - n34));
        const double eu = fma(wu * dqu, nu - tu, qu) - nq12, el = fma(wl * dql, nl - tl, ql) - nq34;
        const double fvapuw = suw * eu, fvaput = dmax(sut * eu, 0.0);
        const double fvaps = ssw * (fma(ws * dqs, ns - ts, qs) - nq12);
        const double fvaplw = slw * el, fvaplt = dmax(slt0 * el, 0.0);
        const double fvapg = sg * (qgfac * fma(wg * dqg, ng - tg, qg) - nq34);
        const double fvapi = si * (fma(wi * dqi, ni - ti, qi) - nq34);
        const double dg = wg * X.zir_gi.lo() * (ng - old[3]), di = wi * X.zir_gi.hi() * (ni - old[4]);
        o.firg = (float)(X.fir_gi.lo() - dg);
        o.firi = (float)(X.fir_gi.hi() - di);
        o.firb = (float)(X.firb + gi * dg + fi * di);
        o.fvapuw = (float)fvapuw; o.fvaput = (float)fvaput; o.fvaps = (float)fvaps;
        o.fvaplw = (float)fvaplw; o.fvaplt = (float)fvaplt; o.fvapg = (float)fvapg; o.fvapi = (float)fvapi;
        o.ginvap = (float)(fvapuw * X.x_us.lo() + fvaps * X.x_us.hi() + fvaplw * X.xl);
        o.gsuvap = (float)(fvapg * gi + fvapi * fi);
        o.gtrans = (float)(fvaput * 2.0 * S(IBIS_STAT_LAI, 1) * S(IBIS_STAT_FU) +
                           fvaplt * 2.0 * S(IBIS_STAT_LAI, 0) * S(IBIS_STAT_FL) * gi);
    }
}

// What the surface phase forms of the soil that the ground phase reads again (the
// soil is not advanced in between): evaporation source fractions, top-layer
// conductivity, and the stress of every layer before the root profile's weights.
struct SoilHour {
    float q1, q2, q3, q4, consoi0, zw[NL], stresstu, stresstl;
    const float* rcap;   // Leaves3 (IBIS 3.0 kernels)
};

// The leaves' area per capacity of Leaves3, with gpp_split_by_capacity
template <typename Q>
__device__ __forceinline__ void area_per_capacity(float (&rcap)[3], const Stat32& S, const Q& q) {
    float twm, tfs;
    bool on;
    capacity_group(kBroadleafPfts, S, q, twm, tfs, on);
    rcap[0] = on ? tfs / twm : -1.0f;
    capacity_group(kConiferPfts, S, q, twm, tfs, on);
    rcap[1] = on ? tfs / twm : -1.0f;
    capacity_group(kShrubPfts, S, q, twm, tfs, on);
    rcap[2] = on ? tfs / twm : -1.0f;
}

// setsoi's conductivity of layer k (soil_physics.py:37-140): the dry solids'
// times 56^liquid 224^ice, one power of two
template <bool X3>
__device__ __forceinline__ float conductivity32(const Stat32& S, const Par32& P, int k, float por, float w, float i) {
    float dry = 0.265f + 0.01f * (0.035f * S(IBIS_STAT_SAND, k) - 0.015f * S(IBIS_STAT_CLAY, k));
    if constexpr (X3) {
        if (P.flags & IBIS_FLAG_FORGANIC) {
            const float fo = S(IBIS_STAT_FORGANIC, k);
            dry = (1.0f - fo) * dry + fo * 0.05f;
        }
    }
    return dry * exp2f(por * (w * (1.0f - i) * 5.807354922057604f + i * 7.807354922057604f));   // log2 of 56 and 224
}

// drystress (stomata.py:515-562)
template <typename Q>
__device__ __forceinline__ void soil_stress32(SoilHour& G, const Col32& c, const Stat32& S, const Par32& P, const Q& q) {
    const float rz = 1.0f / q.znorm(), sf = q.stressfac() * 1.4426950408889634f;
    F2 tot(0.0f);   // lower, upper
#pragma unroll
    for (int k = 0; k < NL; k += 2) {
        const F2 sw = stat2(S, IBIS_STAT_SWILT, k);
        const F2 w = F2(c.wsoi[k], c.wsoi[k + 1]) * (1.0f - F2(c.wisoi[k], c.wisoi[k + 1]));
        const F2 awc = clip2((w - sw) * rcp2(mx2(stat2(S, IBIS_STAT_SFIELD, k) - sw, 1e-10f)), 0.0f, 1.0f);
        const F2 z = clip2((1.0f - exp2_2(awc * sf)) * rz, 0.0f, 1.0f);
        G.zw[k] = z.lo();
        G.zw[k + 1] = z.hi();
        tot = tot + F2(P.fr2[k]) * z.lo();
        tot = tot + F2(P.fr2[k + 1]) * z.hi();
    }
    G.stresstl = tot.lo();
    G.stresstu = tot.hi();
}

// What the record of the hour holds of the parameters and the static planes alone: the
// big leaves' nominal capacities with the IBIS 3.0 switches (stomata.py:592-660).  No hour
// changes them, so a launch forms them once, before its hours: 33,001
// columns x 6 hours of the release formulation 231 -> 184 us.  The F77 step
// has too little of the kind (the same of its leaf-area shares made it 4% slower).
template <typename Y, typename Q>
__device__ __forceinline__ void column_begin32(Y& y, const Stat32& S, const Par32& P, const Q& q) {
    if constexpr (Q::x3) {
        float vu[2], ju[2], mu[2], vl[3], jl[3], ml[3];
        bool jon = false;
        big_leaves<float, false>(vu, ju, mu, jon, S, P, q);
        big_leaves<float, true>(vl, jl, ml, jon, S, P, q);
        y.X.vnu = F2(vu[0], vu[1]); y.cmu = F2(mu[0], mu[1]); y.jfu = F2(ju[0], ju[1]);
        y.vnl = F2(vl[0], vl[1]); y.cml = F2(ml[0], ml[1]); y.jfl = F2(jl[0], jl[1]);
        y.vn4 = vl[2]; y.cm4 = ml[2]; y.jf4 = jl[2];
        y.cap = F2(capacity_integral(S(IBIS_STAT_LAI, 1), P.cap_kn), capacity_integral(S(IBIS_STAT_LAI, 0), P.cap_kn));
        if (P.flags & IBIS_FLAG_GPP_CAPACITY) area_per_capacity(y.rcap, S, q);
    }
}

// Steps 1-9 of timestep_body (see surface_phase, ibis_step.cuh); y: the hour's record,
// begun by column_begin32,
// in shared memory
template <bool SUN_U, bool SUN_L, typename Y, typename Q, typename D32>
__device__ __forceinline__ void surface_phase32(Col32& c, Y& y, const Forc32& F, const Stat32& S, const D32& D,
                                                const Par32& P, const Q& q, Mid<float>& M, SoilHour& G) {
    const float eps = P.epsilon;
    const float fi = c.fi;
    TvHour& X = y.X;
    Casc<float> C;
    Turc tc;
    {
        const float lai0 = S(IBIS_STAT_LAI, 0), lai1 = S(IBIS_STAT_LAI, 1);
        const float sai0 = S(IBIS_STAT_SAI, 0), sai1 = S(IBIS_STAT_SAI, 1);
        const float fu = S(IBIS_STAT_FU), fl = S(IBIS_STAT_FL);
        float hvasug, hvasui;
        evap_sources(c, F, P, G.q1, G.q2, G.q3, G.q4, hvasug, hvasui);
        G.consoi0 = conductivity32<Q::x3>(S, P, 0, S(IBIS_STAT_POROS, 0), c.wsoi[0], c.wisoi[0]);
        X.hv_gi = F2(hvasug, hvasui);

        // ---- 2-3. wet fractions and radiation (loops.py:331-354)
        Rad<float> Rd;
        {
            float fwu, fws, fwl, rlu, rls, rll;
            wet_fraction(c.tu, c.wliqu, c.wsnou, q.wliqumax(), P.wsnoumax, q.fmax(), P, fwu, rlu);
            wet_fraction(c.ts, c.wliqs, c.wsnos, q.wliqsmax(), P.wsnosmax, q.fmax(), P, fws, rls);
            wet_fraction(c.tl, c.wliql, c.wsnol, q.wliqlmax(), P.wsnolmax, q.fmax(), P, fwl, rll);
            radiation(Rd, c, F, S, fwu, fws, fwl, rlu, rls, rll, P);
        }
        X.sol_gi = F2(Rd.solg, Rd.soli);
        X.fir_gi = F2(Rd.firg, Rd.firi);
        X.firb = Rd.firb;
        X.frad_us = F2(lai1 > eps ? (Rd.solu + Rd.firu) / (2.0f * lai1) : 0.0f,
                       sai1 > eps ? (Rd.sols + Rd.firs) / (2.0f * sai1) : 0.0f);
        X.fradl = (lai0 + sai0) > eps ? (Rd.soll + Rd.firl) / (2.0f * (lai0 + sai0)) : 0.0f;
        X.toppar = F2(Rd.topparu, Rd.topparl);
        F2 scale = light_scaling2(Rd, F2(lai1, lai0), F2(sai1, sai0), c,
                                  Q::x3 && (P.flags & IBIS_FLAG_LEAF_ONLY) != 0, P);
        if constexpr (SUN_U) {
            const SunShade<float> ss = sunshade(Rd.scu, Rd.dbeamu, Rd.termu6, Rd.termu7, lai1, sai1, P);
            const float r = lai1 > 0.0f ? 1.0f / mx(lai1, 1.0e-6f) : 0.0f;    // rates per leaf area
            y.su = Sun4{F2(ss.psun, ss.psha) * r, F2(ss.vsun, ss.vsha) * r};
            scale = F2(kLeast * mx(r, 1.0f), scale.hi());
        }
        if constexpr (SUN_L) {
            const SunShade<float> ss = sunshade(Rd.scl, Rd.dbeaml, Rd.terml6, Rd.terml7, lai0, sai0, P);
            const float r = lai0 > 0.0f ? 1.0f / mx(lai0, 1.0e-6f) : 0.0f;
            y.sl = Sun4{F2(ss.psun, ss.psha) * r, F2(ss.vsun, ss.vsha) * r};
            scale = F2(scale.lo(), kLeast * mx(r, 1.0f));
        }
        X.scale = scale;
        if constexpr (!Q::x3)
            X.vnu = F2(S(IBIS_STAT_EXIST, 0) > 0.5f ? q.vmax(0) : (S(IBIS_STAT_EXIST, 2) > 0.5f ? q.vmax(2) : q.vmax(4)),
                       S(IBIS_STAT_EXIST, 3) > 0.5f ? q.vmax(3) : q.vmax(5));
        if (D.on()) radiation_diagnostics(D, Rd);

        // ---- 4-5. precipitation cascade and wet fractions after it (loops.py:359-389)
        cascade32(C, c, F, S, P, q);
        float fwu, fws, rlu, rls;
        wet_fraction(c.tu, C.wliqu, C.wsnou, q.wliqumax(), P.wsnoumax, q.fmax(), P, fwu, rlu);
        wet_fraction(c.ts, C.wliqs, C.wsnos, q.wliqsmax(), P.wsnosmax, q.fmax(), P, fws, rls);
        wet_fraction(c.tl, C.wliql, C.wsnol, q.wliqlmax(), P.wsnolmax, q.fmax(), P, X.fwetl, X.rliql);
        X.fw_us = F2(fwu, fws);
        X.rl_us = F2(rlu, rls);
        X.pf_us = F2(C.pfluxu, C.pfluxs);
        X.pfluxl = C.pfluxl;

        // ---- 6. canopy exchange (loops.py:396-611)
        float cp;
        aero_geometry32(y.A, tc, cp, F, S, fi, P);
        soil_stress32(G, c, S, P, q);
        X.stress = F2(G.stresstu, G.stresstl);
        const float cs = S(IBIS_STAT_CSOI, 0), rs = S(IBIS_STAT_RHOSOI, 0);
        const float csoi0 = cs > 0.0f ? cs : P.csoi_mineral_val, rhosoi0 = rs > 0.0f ? rs : P.rhosoi_val;
        X.cp = cp;
        X.qa = F.qa; X.ps = F.ps; X.fi = fi;
        X.x_us = F2(lai1, sai1) * (2.0f * fu);
        X.xl = 2.0f * (lai0 + sai0) * fl * (1.0f - fi);
        const F2 tgi(c.tg, c.ti);
        const F2 zir = tgi * (tgi * tgi) * P.zir;
        X.zir_gi = zir;
        {
            const float cog = G.consoi0 / mx(0.5f * P.hsoi[0], eps);
            const float coi = P.consno / mx(0.5f * mx(c.hsno[0], P.hsnotop), eps);
            const double zg = zir.lo(), zi = zir.hi();
            X.pg0 = cog + zg;
            X.pi0 = coi + zi;
            X.bg0 = fma(zg, (double)c.tg, fma((double)cog, (double)c.tsoi[0], (double)X.sol_gi.lo() + (double)X.fir_gi.lo()));
            X.bi0 = fma(zi, (double)c.ti, fma((double)coi, (double)c.tsno[0], (double)X.sol_gi.hi() + (double)X.fir_gi.hi()));
            const double tmelt = P.tmelt, cvt = (double)P.cvap * ((double)F.ta - tmelt);
            X.hv0 = fma((double)P.ch2o, tmelt, (double)P.hvap + cvt);
            X.hs0 = fma((double)P.cice, tmelt, (double)P.hsub + cvt);
            X.tap = (double)F.ta * (double)P.tfac;
        }
        const float p0 = S(IBIS_STAT_POROS, 0), w0 = c.wsoi[0], i0 = c.wisoi[0];
        const float rwp = p0 * P.rhow, liq = rwp * (1.0f - i0) * w0, ice = rwp * i0;
        const float chg = P.ch2o * c.wpud + P.cice * c.wipud +
                          ((1.0f - p0) * csoi0 * rhosoi0 + liq * P.ch2o + ice * P.cice) * P.hsoi[0];
        X.wl_us = F2(C.wliqu, C.wliqs);
        X.ws_us = F2(C.wsnou, C.wsnos);
        X.wl_lg = F2(C.wliql, c.wpud + liq * P.hsoi[0]);
        X.ws_lg = F2(C.wsnol, c.wipud + ice * P.hsoi[0]);
        X.ch_us = F2(P.chus2) + X.wl_us * P.ch2o + X.ws_us * P.cice;
        X.ch_lg = F2(P.chl + P.ch2o * C.wliql + P.cice * C.wsnol, chg);
        const float zwp = clip(0.5f * (c.wpud + c.wipud) / mx(P.wpudmax, eps), 0.0f, 0.5f);
        const float zws = (1.0f - i0) * w0 + i0;
        const float zwtot = zwp + (1.0f - zwp) * zws;
        X.psig = -P.grav * S(IBIS_STAT_SUCTION, 0) * pw(zwtot, -S(IBIS_STAT_BEX, 0));
        const double sw0 = S(IBIS_STAT_SWILT, 0);
        double betaw = clip(((double)zwtot - sw0) * rcp_nr(fmax(1.0 - sw0, (double)eps)), 0.0, 1.0);
        if (q.beta_power() != 1.0f) betaw = (double)pw((float)betaw, q.beta_power());
        X.betaw = betaw;
        auto fr = [&](int j) { return (double)S(IBIS_STAT_FRAC, j); };
        X.fb = fr(0) + fr(1) + fr(2) + fr(4) + fr(6) + fr(7);
        X.fc = fr(3) + fr(5);
        X.fs = fr(8) + fr(9);
        X.fr4 = S(IBIS_STAT_FRAC, 10);
        X.fr3 = S(IBIS_STAT_FRAC, 11);
        X.rlai = (double)lai0 * rcp_nr(fmax((double)(lai0 + sai0), (double)eps));
    }
    double Wv[9] = {(double)c.tu, (double)c.ts, (double)c.tl, (double)c.t12, (double)c.t34,
                    (double)c.q12, (double)c.q34, (double)c.tg, (double)c.ti};
    F2 wus(1.0f), wlg(1.0f);      // implicit weights of the canopy's and of the lower canopy's and ground's temperatures
    float wi = 1.0f;
    Stom<float> st;
    TvResult tv;
#pragma unroll 1
    for (int it = 0; it < 3; ++it) {
        asm volatile("" ::: "memory");     // read the hour's record again in each pass instead of keeping it in registers
        const bool first = (it == 0);
        const float tu = (float)Wv[0], ts = (float)Wv[1], tl = (float)Wv[2];
        const F2 tair((float)Wv[3], (float)Wv[4]), qair((float)Wv[5], (float)Wv[6]);
        Trans<float> T;
        transfer32(T, tc, y.A, tair.lo(), tair.hi(), qair.lo(), qair.hi(), first, P);
        const F2 eair = esat2(tair), rair = sat_quotient2(eair, X.ps), qsair = eair * rair;
        stomata32<SUN_U, SUN_L>(st, c, tu, tl, qair, qsair, T.su, T.sl, y, P, q);
        if (!first) {
            const float tg = (float)Wv[7], ti = (float)Wv[8];
            wus = weight_veg2(F2(tu, ts), X.ch_us, X.wl_us, X.ws_us, wus, P);
            wlg = weight_veg2(F2(tl, tg), X.ch_lg, X.wl_lg, X.ws_lg, wlg, P);
            wi = weight_snow(ti, c.ti, wi, false, P);
        }
        turvap32(Wv, tv, c, T, wus, wlg, wi, X, st, S, rair.hi(), qsair.hi(), it == 2, P);
    }
    const float ti_new = mn((float)Wv[8], P.tmelt);
    const float tg_w = (float)Wv[7];

    // ---- 7-8. evaporation of intercepted water, bare-story reset (loops.py:616-640)
    float tu = (float)Wv[0], ts = (float)Wv[1], tl = (float)Wv[2];
    float wliqu = X.wl_us.lo(), wliqs = X.wl_us.hi(), wliql = X.wl_lg.lo();
    float wsnou = X.ws_us.lo(), wsnos = X.ws_us.hi(), wsnol = X.ws_lg.lo();
    evap_intercepted(tu, wliqu, wsnou, X.rl_us.lo(), tv.fvapuw, P.chu, P);
    evap_intercepted(ts, wliqs, wsnos, X.rl_us.hi(), tv.fvaps, P.chs, P);
    evap_intercepted(tl, wliql, wsnol, X.rliql, tv.fvaplw, P.chl, P);
    {
        const float tav = (1.0f - fi) * tg_w + fi * ti_new;
        const F2 x_us = X.x_us;
        if (x_us.lo() == 0.0f) { tu = tav; wliqu = 0.0f; wsnou = 0.0f; }
        if (x_us.hi() == 0.0f) { ts = tav; wliqs = 0.0f; wsnos = 0.0f; }
        if (2.0f * (S(IBIS_STAT_LAI, 0) + S(IBIS_STAT_SAI, 0)) == 0.0f || S(IBIS_STAT_FL) * (1.0f - fi) == 0.0f) {
            tl = tav;
            wliql = 0.0f;
            wsnol = 0.0f;
        }
    }

    // ---- 9. surface fluxes into soil and snow (loops.py:665-674)
    const float fm = P.flux_max;
    M.fvapg = tv.fvapg;
    M.fvapi = tv.fvapi;
    M.heatg = X.sol_gi.lo() + clip(tv.firg, -fm, fm) - clip(tv.fseng, -fm, fm) - X.hv_gi.lo() * M.fvapg;
    M.heati = X.sol_gi.hi() + clip(tv.firi, -fm, fm) - clip(tv.fseni, -fm, fm) - X.hv_gi.hi() * M.fvapi;
    M.fvaput = tv.fvaput;
    M.fvaplt = tv.fvaplt;
    M.ginvap = tv.ginvap;
    M.gsuvap = tv.gsuvap;
    M.gtrans = tv.gtrans;
    M.fsena = tv.fsena;
    M.raing = C.raing; M.traing = C.traing; M.snowg = C.snowg; M.tsnowg = C.tsnowg;
    M.rainl = C.rainl; M.trainl = C.trainl; M.snowl = C.snowl; M.tsnowl = C.tsnowl;
#pragma unroll
    for (int j = 0; j < 2; ++j) { M.an_u[j] = st.an_u[j]; M.ag_u[j] = st.ag_u[j]; }
#pragma unroll
    for (int j = 0; j < 3; ++j) { M.an_l[j] = st.an_l[j]; M.ag_l[j] = st.ag_l[j]; }

    // canopy state left for the ground phase (tu/ts/tl/tg unclamped)
    c.tu = tu; c.ts = ts; c.tl = tl; c.tg = tg_w; c.ti = ti_new;
    c.t12 = (float)Wv[3]; c.t34 = (float)Wv[4]; c.q12 = (float)Wv[5]; c.q34 = (float)Wv[6];
    c.wliqu = wliqu; c.wliqs = wliqs; c.wliql = wliql;
    c.wsnou = wsnou; c.wsnos = wsnos; c.wsnol = wsnol;

    // ---- diagnostics of the surface phase (loops.py:1158-1241)
    if (D.on()) {
        surface_diagnostics(D, st, X.fw_us.lo(), X.fw_us.hi(), X.fwetl, X.rl_us.lo(), X.rl_us.hi(), X.rliql, tv.firg,
                            tv.firi, tv.firb, tv.fsenu, tv.fsens, tv.fsenl, tv.fseng, tv.fseni, M, y.A.rhoa,
                            X.hv_gi.lo(), X.hv_gi.hi(), G.q1, G.q2, G.q3, G.q4);
    }
}

// The same, formed by the ground kernel of the two-kernel form
template <typename Q>
__device__ __forceinline__ void soil_hour32(SoilHour& G, const Col32& c, const Forc32& F, const Stat32& S,
                                            const Par32& P, const Q& q) {
    float hvasug, hvasui;
    evap_sources(c, F, P, G.q1, G.q2, G.q3, G.q4, hvasug, hvasui);
    G.consoi0 = conductivity32<Q::x3>(S, P, 0, S(IBIS_STAT_POROS, 0), c.wsoi[0], c.wisoi[0]);
    soil_stress32(G, c, S, P, q);
}

// ===========================================================================
// snow, soil water and heat (physics/snow_physics.py, soil_physics.py, bedrock.py):
// the soil layers in pairs (0,1), (2,3), (4,5)
// ===========================================================================

constexpr int NP = NL / 2;   // pairs of soil layers
static_assert(NL == 6, "three pairs of soil layers");

__device__ __forceinline__ F2 load2(const float (&a)[NL], int j) { return F2(a[2 * j], a[2 * j + 1]); }
__device__ __forceinline__ F2 stat_pair(const Stat32& S, int p, int j) { return stat2(S, p, 2 * j); }

// soilh2o (soil_physics.py:196-373): the implicit system in float, solved for the
// hour's increments delta = w_new - w; w, wpud advanced, wflo the fluxes.  Its
// right-hand side holds the flux divergence and the implicit terms applied to the
// current profile, so float32 rounds relative to the hour's change where a layer
// changes slowly, and relative to w where the implicit terms dominate (wet, conductive
// layers), as the float32 state's own storage does.  The saturation bound and the
// upward excess flux work on the increments too.  The five interfaces and the drainage boundary are handled as the three pairs
// (1,2), (3,4), (5,bottom); w**(2n+3) comes from w**(n+1), so one power serves each.
__device__ __forceinline__ void soil_water32(F2 (&w2)[NP], float& wpud, float (&wflo)[NL + 1], const F2 (&wi2)[NP],
                                             const F2 (&por)[NP], const F2 (&pflo)[NP], const Stat32& S, float fwtop,
                                             float fwpud, const Par32& P) {
    const float dmin = 1e-9f;
    const bool consistent = (P.flags & IBIS_FLAG_H2O_CONSISTENT) != 0;
    F2 e[NP], f[NP], g[NP];      // of interfaces (1,2), (3,4), (5,bottom)
    {
        float w[NL + 1], wi[NL + 1], hyd[NL + 1], hs[NL + 1], bex[NL + 1];
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            w[k] = k & 1 ? w2[k / 2].hi() : w2[k / 2].lo();
            wi[k] = k & 1 ? wi2[k / 2].hi() : wi2[k / 2].lo();
            hyd[k] = S(IBIS_STAT_HYDRAUL, k);
            bex[k] = S(IBIS_STAT_BEX, k);
            hs[k] = hyd[k] * S(IBIS_STAT_SUCTION, k) * bex[k];
        }
        // below the last layer: the same soil and water, so the boundary's own terms
        // come out of the interface formulas with equal weights of one layer
        w[NL] = w[NL - 1]; wi[NL] = wi[NL - 1]; hyd[NL] = hyd[NL - 1]; hs[NL] = hs[NL - 1]; bex[NL] = bex[NL - 1];
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const int k = 2 * j + 1;
            const F2 wp(P.iwp2[j]), wm(P.iwm2[j]), rhm(P.irh2[j]);
            const F2 a = wm * F2(hyd[k - 1], hyd[k]) + wp * F2(hyd[k], hyd[k + 1]);
            const F2 b = wm * F2(hs[k - 1], hs[k]) + wp * F2(hs[k], hs[k + 1]);
            // rounded to a whole exponent: from the difference, so that layers of one soil give its
            // own exponent whatever the weights' rounding (half-integer ones lie on the tie)
            const F2 b0(bex[k - 1], bex[k]);
            const F2 zb = b0 + wp * (F2(bex[k], bex[k + 1]) - b0) + 0.5f;
            const float n0 = floorf(zb.lo()), n1 = floorf(zb.hi());
            const F2 wa0(w[k - 1], w[k]), wa1(w[k], w[k + 1]);
            const F2 ws = consistent ? wp * wa0 + wm * wa1 : wm * wa0 + wp * wa1;
            const F2 wa = mn2(ws, 1.0f);
            const F2 pw1 = ipow2(wa, (int)n0 + 1, (int)n1 + 1);
            const F2 wam1 = pw1 * pw1;                            // wa**(m-1), m = 2 n + 3
            F2 bwn1 = b * pw1;
            const F2 bwn = bwn1 * wa;
            bwn1 = sel2(bwn.lo() < dmin, bwn.hi() < dmin, F2(0.0f), bwn1);
            const F2 n(n0, n1), nd = (n + 2.0f) * bwn1 * ((wa1 - wa0) * rhm), m1 = n * 2.0f + 2.0f, aw = a * wam1;
            const F2 zi0 = mx2(1.0f - mx2(F2(wi[k - 1], wi[k]), F2(wi[k], wi[k + 1])), 0.0f);
            const F2 zi = zi0 * zi0;
            e[j] = zi * (wa * (m1 * aw - nd));
            f[j] = zi * (nd - (m1 + 1.0f) * aw);
            g[j] = zi * mx2(bwn, dmin);
            if (j == NP - 1) {
                // free drainage: -K (w**m) bperm out of the bottom, no diffusion
                e[j] = F2(e[j].lo(), -(zi.hi() * aw.hi() * wa.hi()) * P.bperm);
                f[j] = F2(f[j].lo(), 0.0f);
                g[j] = F2(g[j].lo(), 0.0f);
            }
        }
    }
    float lo[NL], di[NL], up[NL], r[NL], dl[NL];
    {
        const float src = (fwtop + fwpud) / P.rhow;
        F2 ep(0.0f, e[0].lo()), fp(0.0f, f[0].lo()), gp(0.0f, g[0].lo());   // upper interfaces of the pair
        F2 wp(0.0f, w2[0].lo());
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const F2 dt = P.dtime * rcp2(mx2(pflo[j] * F2(P.h2[j]), 1e-30f));
            const F2 rhb = F2(P.rhb2[j]), gb = gp * rhb, gn = g[j] * F2(P.rhp2[j]);
            const F2 d1 = dt * (fp * F2(P.c12[j]) - gb);
            const F2 d3 = dt * (F2(0.0f) - f[j] * F2(P.c62[j]) - gn);
            const F2 d2m = dt * (fp * F2(P.c52[j]) - f[j] * F2(P.c32[j]) + gn + gb);
            const F2 wn(w2[j].hi(), j + 1 < NP ? w2[j + 1].lo() : 0.0f);
            F2 rk = e[j] - ep;
            if (j == 0) rk = rk + F2(src, 0.0f);
            rk = dt * rk - d2m * w2[j] - d1 * wp - d3 * wn;
            const F2 dd = 1.0f + d2m;
            lo[2 * j] = d1.lo(); lo[2 * j + 1] = d1.hi();
            di[2 * j] = dd.lo(); di[2 * j + 1] = dd.hi();
            up[2 * j] = d3.lo(); up[2 * j + 1] = d3.hi();
            r[2 * j] = rk.lo(); r[2 * j + 1] = rk.hi();
            if (j + 1 < NP) {
                ep = F2(e[j].hi(), e[j + 1].lo());
                fp = F2(f[j].hi(), f[j + 1].lo());
                gp = F2(g[j].hi(), g[j + 1].lo());
                wp = F2(w2[j].hi(), w2[j + 1].lo());
            }
        }
    }
    thomas(lo, di, up, r, dl);
    wflo[NL] = -P.rhow * e[NP - 1].hi();
    float over_kg = 0.0f;      // saturation excess passed up, kg m-2
#pragma unroll
    for (int j = NP - 1; j >= 0; --j) {
        const F2 zz2 = P.rhow * F2(P.h2[j]) * por[j] * mx2(1.0f - wi2[j], P.epsilon);
        const F2 rz2 = rcp2(zz2);
        float wn[2];
#pragma unroll
        for (int q = 1; q >= 0; --q) {
            const int k = 2 * j + q;
            const float zz = q ? zz2.hi() : zz2.lo(), rz = q ? rz2.hi() : rz2.lo(), w = q ? w2[j].hi() : w2[j].lo();
            float dw = dl[k] + over_kg * rz;                // w_new - w before the saturation bound
            const float over = (w - 1.0f) + dw;             // w_new - 1
            over_kg = mx(over, 0.0f) * zz;
            if (over > 0.0f) dw = 1.0f - w;
            wflo[k] = wflo[k + 1] + dw * zz * P.rdt;
            wn[q] = over > 0.0f ? 1.0f : w + dw;
        }
        w2[j] = F2(wn[0], wn[1]);
    }
    wpud = mx(wpud + (over_kg - fwpud * P.dtime), 0.0f);
    wflo[0] = wflo[0] + over_kg * P.rdt - fwpud;
}

// soilheat (soil_physics.py:385-490) or soilheat_with_bedrock (bedrock.py:88-153): the
// system in float for delta = T_new - t, whose right-hand side holds only small terms
// -- the heat-capacity change times t, the transpired water's heat, the flux
// divergence, and the conduction of the current temperature differences -- so float32
// rounds relative to the hour's change, not to the temperature.  On absolute
// temperatures (~280 K, one ulp 3e-5 K) it would round each hour by a sizeable part of
// a deep layer's change (~1e-4 K), and the residue repeats while a layer changes
// slowly: over a year that cooled the deep column of every cell by 0.03-0.09 K and
// drifted runoff, ET and CH4 by up to 4e-4.  The layers start from t + dtp (dtp: the
// heat of the transpired water), kept apart because in float32 an increment below half
// an ulp of the temperature would be dropped.  Bedrock carries no water, so its rows
// are the launch's constants (DevParams::bed_*).
template <int NT, bool HFLO>
__device__ __forceinline__ void soil_heat32(F2 (&t)[NP], float (&tb)[NB], float (&hflo)[NL + 1], const F2 (&dtp)[NP],
                                            const F2 (&ow)[NP], const F2 (&w)[NP], const F2 (&wi)[NP],
                                            const F2 (&por)[NP], const F2 (&cons)[NP], const F2 (&rsol)[NP],
                                            float c0pud0, float c1pud0, float fhtop, const float (&wflo)[NL + 1],
                                            const Par32& P) {
    constexpr int NBED = NT - NL;
    const float chr = P.ch2o * P.rhow, cir = P.cice * P.rhow;
    F2 res[NP], ts[NP], rc1[NP], c0[NP], dc[NP], c1[NP];
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        const F2 h = F2(P.h2[j]);
        res[j] = h * 0.5f * rcp2(mx2(cons[j], 1e-12f));
        ts[j] = t[j] + dtp[j];                            // starting temperatures, for the advected heat
        const F2 r2 = por[j] * (1.0f - wi[j]) * chr, r13 = rsol[j] + por[j] * wi[j] * cir;
        c0[j] = (r13 + r2 * ow[j]) * h;
        c1[j] = (r13 + r2 * w[j]) * h;
        dc[j] = r2 * (ow[j] - w[j]) * h;                  // c0 - c1
        if (j == 0) {
            c0[0] = c0[0] + F2(c0pud0, 0.0f);
            c1[0] = c1[0] + F2(c1pud0, 0.0f);
            dc[0] = dc[0] + F2(c0pud0 - c1pud0, 0.0f);
        }
        rc1[j] = rcp2(c1[j]);
    }
    // conductances and advected heat at the interfaces below each layer of a pair
    F2 con[NP], whf[NP];
    const float drain = wflo[NL] * P.ch2o * ts[NP - 1].hi();
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        const int k = 2 * j + 1;
        if (j + 1 < NP) {
            con[j] = rcp2(res[j] + F2(res[j].hi(), res[j + 1].lo()));
            const F2 up_(ts[j].lo(), ts[j].hi()), dn(ts[j].hi(), ts[j + 1].lo());
            whf[j] = F2(wflo[k], wflo[k + 1]) * P.ch2o *
                     (F2(P.hsb2[j]) * up_ + F2(P.hsa2[j]) * dn);
        } else {
            const float c5 = 1.0f / (res[j].lo() + res[j].hi());
            const float c6 = NBED > 0 ? 1.0f / (res[j].hi() + P.bed_res[0]) : 0.0f;
            con[j] = F2(c5, c6);
            whf[j] = F2(wflo[k] * P.ch2o * (P.hs_below5 * ts[j].lo() + P.hs_above5 * ts[j].hi()), drain);
        }
    }
    // res holds half the layer's resistance with itself: con = 1 / (r[k-1] + r[k])
    float lo[NT], di[NT], up[NT], r[NT], dl[NT];
    {
        F2 conu(0.0f, con[0].lo()), whu(wflo[0] * P.ch2o * ts[0].lo() + fhtop, whf[0].lo());
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const float tnext = j + 1 < NP ? t[j + 1].lo() : (NBED > 0 ? tb[0] : t[j].hi());
            const F2 tprev(j > 0 ? t[j - 1].hi() : t[0].lo(), t[j].lo());
            const F2 rw = rc1[j] * P.dtime;
            const F2 cond = conu * (t[j] - tprev) + con[j] * (t[j] - F2(t[j].hi(), tnext));
            const F2 l = rw * conu, u = rw * con[j], d = 1.0f + l + u;
            const F2 rr = dc[j] * rc1[j] * t[j] + c0[j] * rc1[j] * dtp[j] + rw * (whu - whf[j] - cond);
            lo[2 * j] = -l.lo(); lo[2 * j + 1] = -l.hi();
            up[2 * j] = -u.lo(); up[2 * j + 1] = -u.hi();
            di[2 * j] = d.lo(); di[2 * j + 1] = d.hi();
            r[2 * j] = rr.lo(); r[2 * j + 1] = rr.hi();
            if (j + 1 < NP) {
                conu = F2(con[j].hi(), con[j + 1].lo());
                whu = F2(whf[j].hi(), whf[j + 1].lo());
            }
        }
        if constexpr (NBED > 0) {
            float cu = con[NP - 1].hi(), tp = t[NP - 1].hi();
#pragma unroll
            for (int b = 0; b < NBED; ++b) {
                const float cd = b + 1 < NBED ? P.bed_con[b] : 0.0f, rw = P.bed_rw[b];
                const float tn = b + 1 < NBED ? tb[b + 1] : tb[b];
                lo[NL + b] = -rw * cu;
                up[NL + b] = -rw * cd;
                di[NL + b] = 1.0f + rw * cu + rw * cd;
                r[NL + b] = -rw * (cu * (tb[b] - tp) + cd * (tb[b] - tn));
                cu = cd;
                tp = tb[b];
            }
        }
    }
    thomas(lo, di, up, r, dl);
    if constexpr (HFLO) {
        float s = fhtop;
        hflo[0] = s;
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            const int j = k / 2;
            auto at = [&](const F2& v) { return k & 1 ? v.hi() : v.lo(); };
            s = s - (at(c1[j]) * dl[k] - at(dc[j]) * at(t[j]) - at(c0[j]) * at(dtp[j])) * P.rdt;
            hflo[k + 1] = s;
        }
    }
#pragma unroll
    for (int j = 0; j < NP; ++j) t[j] = t[j] + F2(dl[2 * j], dl[2 * j + 1]);
    if constexpr (NBED > 0) {
#pragma unroll
        for (int b = 0; b < NBED; ++b) tb[b] = tb[b] + dl[NL + b];
    }
}

// wadjust (soil_physics.py:147-189); with GADJ returns the mass adjustment rate
template <bool GADJ>
__device__ __forceinline__ float water_bounds32(F2 (&w)[NP], F2 (&i)[NP], const F2 (&por)[NP], const Par32& P) {
    const float eps = P.epsilon;
    float tot = 0.0f;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        const F2 z = F2(P.h2[j]) * por[j] * P.rhow;
        const F2 zero(0.0f);
        F2 ww = mn2(sel2(w[j].lo() < eps, w[j].hi() < eps, zero, w[j]), 1.0f);
        const F2 ii = mn2(sel2(i[j].lo() < eps, i[j].hi() < eps, zero, i[j]), 1.0f);
        ww = sel2(ii.lo() >= 1.0f - eps, ii.hi() >= 1.0f - eps, zero, ww);
        if constexpr (GADJ)
            tot = tot + (z * ((1.0f - ii) * ww + ii) - z * ((1.0f - i[j]) * w[j] + i[j])).sum();
        w[j] = ww;
        i[j] = ii;
    }
    return GADJ ? tot * P.rdt : 0.0f;
}

// freeze_thaw (soil_physics.py:497-564).  The heat left after freezing is the
// surplus the thaw sees, so the intermediate temperature is not formed.
__device__ __forceinline__ void phase_change32(F2 (&t)[NP], F2 (&w)[NP], F2 (&i)[NP], const F2 (&por)[NP],
                                               const F2 (&rsol)[NP], float c1pud0, const Par32& P) {
    const float eps = P.epsilon, rhw = 1.0f / P.rhow, rfus = 1.0f / P.hfus;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        const F2 zp = mx2(por[j], eps), rz = rcp2(zp);
        F2 rw = rsol[j] * rhw;
        if (j == 0) rw = rw + F2(c1pud0 * rhw / P.hsoi[0], 0.0f);
        const F2 zl = zp * P.ch2o, zi = zp * P.cice;
        F2 chav = rw + zl * (1.0f - i[j]) * w[j] + zi * i[j];
        const F2 zw = mn2(w[j], 1.0f);
        F2 dh = chav * (P.tmelt - t[j]);
        F2 dw = mn2(zp * (1.0f - i[j]) * zw, mx2(dh * rfus, 0.0f));
        F2 d = dw * rz;
        F2 ik = i[j] + d;
        F2 wk = w[j] - d * (1.0f - zw) * rcp2(mx2(1.0f - ik, eps));
        dh = dw * P.hfus - dh;
        dw = mn2(zp * ik, mx2(dh * rfus, 0.0f));
        d = dw * rz;
        ik = ik - d;
        wk = wk + d * (1.0f - wk) * rcp2(mx2(1.0f - ik, eps));
        chav = rw + zl * (1.0f - ik) * wk + zi * ik;
        t[j] = P.tmelt + (dh - dw * P.hfus) * rcp2(chav);
        w[j] = wk;
        i[j] = ik;
    }
}

// puddle_freeze_thaw (soil_physics.py:567-615)
__device__ __forceinline__ void puddle_phase32(float& t0, float& wpud, float& wipud, float por0, float w0, float i0,
                                               float rsol0, const Par32& P) {
    const float rw = (rsol0 + por0 * P.rhow * ((1.0f - i0) * w0 * P.ch2o + i0 * P.cice)) * P.hsoi[0];
    const float rfus = 1.0f / P.hfus;
    float dh = (P.ch2o * wpud + P.cice * wipud + rw) * (P.tmelt - t0);
    float dw = mn(wpud, mx(0.0f, dh * rfus));
    wipud = wipud + dw;
    wpud = wpud - dw;
    dh = P.hfus * dw - dh;
    dw = mn(wipud, mx(0.0f, dh * rfus));
    wipud = wipud - dw;
    wpud = wpud + dw;
    t0 = P.tmelt + (dh - P.hfus * dw) / (P.ch2o * wpud + P.cice * wipud + rw);
    wpud = mx(wpud, 0.0f);
    wipud = mx(wipud, 0.0f);
}

// methane_flux (methane.py:233-383; see the template in ibis_ground.cuh)
__device__ __forceinline__ float methane32(float f_inund, float rh, const F2 (&t)[NP], const F2 (&w)[NP],
                                           const F2 (&i)[NP], float zwt_obs, const Ch4Par<float>& m, const Par32& P) {
    F2 acc(0.0f);
#pragma unroll
    for (int j = 0; j < NP; ++j) acc = acc + clip2(w[j] * (1.0f - i[j]) + i[j], 0.0f, 1.0f) * load2(m.wtop, j);
    const float wet = clip(acc.sum() / (m.wtot * mx(m.sat_crit, 1e-6f)), 0.0f, 1.0f);
    float zwt = m.z_wt_max * (1.0f - wet);
    if (isfinite(zwt_obs)) zwt = clip(zwt_obs, 0.0f, m.z_max);
    F2 tt(0.0f), tw(0.0f);
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        const F2 an = mn2(mx2(F2(P.bot2[j]) - mx2(F2(P.top2[j]), zwt), 0.0f), F2(P.h2[j]));
        const F2 th = sel2(t[j].lo() >= 273.15f, t[j].hi() >= 273.15f, an, F2(0.0f));
        tt = tt + th;
        tw = tw + th * t[j];
    }
    const float ts = tt.sum();
    const float tth = ts > 1e-12f ? tw.sum() / mx(ts, 1e-12f) : t[0].lo();
    const float zp = mx(zwt, 0.0f);
    const float decay = ex(-zp / mx(m.z_tau, 1e-6f) - zp / mx(m.tau_oxid, 1e-6f));
    const float q10 = pw(m.q10p, (tth - m.t_ref) * 0.1f);
    const float prod = mx(rh, 0.0f) * decay * m.r_ch4 * q10;
    return tth < 273.15f ? 0.0f : clip(f_inund, 0.0f, 1.0f) * prod;    // a temperature that is not a number shows
}

// Steps 10-12 of timestep_body, the fire counters and the day-loop accumulators
// (see ground_phase, ibis_step.cuh)
template <int NT, typename Q, typename D32, int SLD>
__device__ __forceinline__ void ground_phase32(Col32& c, const Forc32& F, Stat32& S, const D32& D,
                                               const Acc<float, SLD>& Ac, const Par32& P, const Q& q,
                                               const Mid<float>& M, const SoilHour& G) {
    constexpr bool DIAG = D32::enabled;
    const float eps = P.epsilon, dt = P.dtime;
    const float fi = c.fi;
    // The view is renewed here and before the carbon sums: the compiler forms a plane's
    // address from another's, and chains of them through the whole hour took
    // registers (380 bytes of spills a thread with one view an hour, 200 with three;
    // 95,333 columns x 6 hours 0.393 -> 0.364 ms, 200 x 24 hours 0.349 -> 0.310).
    S.renew();
    const float lai0 = S(IBIS_STAT_LAI, 0), lai1 = S(IBIS_STAT_LAI, 1);
    const float fu = S(IBIS_STAT_FU), fl = S(IBIS_STAT_FL);
    const float tu = c.tu, tl = c.tl;

    // ---- 10. snow (loops.py:676-848)
    float smelt = 0.0f, zheat = 0.0f, sflo_bot = 0.0f, fhtop_snow = 0.0f;
    // Bare of snow and none falling on it: the block's result is known (cover below
    // fimin melts to none, layers at the melting point), and a warp of such columns
    // skips it.  Not where a layer's or the buried canopy's temperature is no finite number:
    // the block would carry that into the soil, and the skip would heal it unnoticed.
    // Launches with diagnostics report the block's fluxes too.
    const bool snowy = DIAG || !(fi == 0.0f && M.snowg == 0.0f && c.hsno[0] == 0.0f && c.hsno[1] == 0.0f &&
                                 c.hsno[2] == 0.0f && P.fimin > 0.0f &&
                                 finite((c.tsno[0] + c.tsno[1]) + (c.tsno[2] + c.tlsub)));
    if (!snowy) {
        c.tsno[0] = c.tsno[1] = c.tsno[2] = P.tmelt;
        c.tlsub = tl;
    } else {
        float wliql = c.wliql, wsnol = c.wsnol;
        fhtop_snow = M.heati + M.rainl * (P.ch2o * (M.trainl - P.tmelt) + P.hfus + P.cice * (P.tmelt - c.tsno[0])) +
                     M.snowl * P.cice * (M.tsnowl - c.tsno[0]);
        const float xlb = fl * 2.0f * (lai0 + S(IBIS_STAT_SAI, 0));
        const float rrhos = 1.0f / P.rhos;
        float hp[NS], tsh[NS];
#pragma unroll
        for (int k = 0; k < NS; ++k) { hp[k] = c.hsno[k]; tsh[k] = c.tsno[k]; }
        if (fi > 0.0f) hp[0] = hp[0] + (M.rainl + M.snowl - M.fvapi) * (dt * rrhos);
        float tlsub_h = c.tlsub;
        snow_heat(tsh, tlsub_h, sflo_bot, fhtop_snow, xlb, fi, hp, P.hsoi[0], G.consoi0, c.tsoi[0], P);
        const float ht = hp[0] + hp[1] + hp[2];
        const float hts = ht > 0.0f ? ht : P.hsnomin;
        float dfi = (1.0f - fi) * dt * M.snowg / (P.rhos * hts);
        dfi = mn(dfi, 1.0f - fi);
        const float fi1 = fi + dfi, rfi1 = 1.0f / mx(fi1, eps);
        float tm[NS], hm[NS];
        const bool fresh = (fi < eps) && (dfi > 0.0f);
        float htc = 0.0f;
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            tm[k] = fi1 > 0.0f ? (tsh[k] * fi + M.tsnowg * dfi) * rfi1 : tsh[k];
            const float hinit = k == 0 ? P.hsnotop : (P.hsnomin - P.hsnotop) * float(1.0 / (NS - 1));
            hm[k] = fresh ? hinit : hp[k];
            // snow_melt (snow_physics.py:236-260)
            const float ms = P.rhos * hm[k], xh = ms * P.cice * mx(tm[k] - P.tmelt, 0.0f);
            const float xm = mn(ms, xh * (1.0f / P.hfus));
            hm[k] = hm[k] - xm * rrhos;
            tm[k] = mn(tm[k], P.tmelt);
            smelt = smelt + fi1 * xm;
            zheat = zheat + fi1 * (xh - P.hfus * xm);
            htc = htc + hm[k];
        }
        // snow_coverage (snow_physics.py:263-290)
        const float ruf = mn(0.70f, mx(P.hsnomin + 0.05f, fl * S(IBIS_STAT_ZTOP, 0)));
        if (htc < 1e-10f) htc = P.hsnomin;
        const float zhh = 0.5f * P.hsnomin;
        const float zdh = mx(ruf - P.hsnomin, eps);
        float fic = clip((sq(zhh * zhh + zdh * fi1 * htc) - zhh) / zdh, 0.0f, P.fimax);
        const float scl = fi1 / mx(fic, eps);
#pragma unroll
        for (int k = 0; k < NS; ++k) hm[k] = hm[k] * scl;
        readapt_layers(hm, tm, P.hsnotop, eps);
        // fimin melt-all (loops.py:763-777)
        if (fic < P.fimin) {
            float hsum = 0.0f, heat = 0.0f;
#pragma unroll
            for (int k = 0; k < NS; ++k) {
                hsum = hsum + hm[k];
                heat = heat + P.rhos * hm[k] * fic * (P.cice * (P.tmelt - tm[k]) + P.hfus);
                hm[k] = 0.0f;
                tm[k] = P.tmelt;
            }
            smelt = smelt + P.rhos * hsum * fic;
            zheat = zheat - heat;
            fic = 0.0f;
        }
        // buried vegetation (loops.py:781-830)
        const float dfc = fic - fi;
        float tlsub = tlsub_h;
        if (dfc > 0.0f) {
            const float rf = 1.0f / mx(fic, eps);
            tlsub = (tlsub_h * fi + tl * dfc) * rf;
            zheat = zheat + dfc * xlb * (wliql * (P.ch2o * (tl - P.tmelt) + P.hfus + P.cice * (P.tmelt - tm[NS - 1])) +
                                         wsnol * P.cice * (tl - tm[NS - 1]));
            hm[NS - 1] = hm[NS - 1] + dfc * xlb * (wliql + wsnol) * (rf * rrhos);
        }
        if (dfc < 0.0f) {
            zheat = zheat - dfc * xlb * P.chl * (tlsub_h - tl);
            const float rdec = (1.0f - fi) / mx(1.0f - fic, eps);
            wliql = wliql * rdec;
            wsnol = wsnol * rdec;
        }
        if (!(fic > 0.0f)) tlsub = tl;
        c.fi = fic;
#pragma unroll
        for (int k = 0; k < NS; ++k) { c.hsno[k] = hm[k]; c.tsno[k] = tm[k]; }
        c.tlsub = tlsub;
        c.wliql = wliql;
        c.wsnol = wsnol;
    }
    const float heatg_avg = (1.0f - fi) * M.heatg + fi * sflo_bot + zheat * P.rdt;
    const float fvapg_avg = clip((1.0f - fi) * M.fvapg, -1.0e-3f, 1.0e-3f);
    const float raing_nf = (1.0f - fi) * M.raing;
    const float smr = smelt * P.rdt;
    const float rsum = raing_nf + smr;
    const bool rzero = rsum < eps;
    const float raing_avg = rzero ? 0.0f : rsum;
    const float traing_avg = rzero ? 0.0f : (raing_nf * M.traing + smr * P.tmelt) / rsum;

    // ---- 11. soil (loops.py:896-1125)
    F2 por[NP], rsol[NP], cons[NP], wsw[NP], wisw[NP], pflo[NP], t[NP];
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        por[j] = stat_pair(S, IBIS_STAT_POROS, j);
        const F2 cs = stat_pair(S, IBIS_STAT_CSOI, j), rs = stat_pair(S, IBIS_STAT_RHOSOI, j);
        rsol[j] = (1.0f - por[j]) * sel2(cs.lo() > 0.0f, cs.hi() > 0.0f, cs, F2(P.csoi_mineral_val)) *
                  sel2(rs.lo() > 0.0f, rs.hi() > 0.0f, rs, F2(P.rhosoi_val));
        wsw[j] = load2(c.wsoi, j);
        wisw[j] = load2(c.wisoi, j);
        t[j] = load2(c.tsoi, j);
        const float k0 = j == 0 ? G.consoi0
                                : conductivity32<Q::x3>(S, P, 2 * j, por[j].lo(), wsw[j].lo(), wisw[j].lo());
        cons[j] = F2(k0, conductivity32<Q::x3>(S, P, 2 * j + 1, por[j].hi(), wsw[j].hi(), wisw[j].hi()));
    }
    float grunof = mn(c.wpud, mx(0.0f, c.wpud + c.wipud - P.wpudmax)) * P.rdt;
    float wpw = c.wpud - grunof * dt;
    const float zfrez = clip((t[0].lo() - P.tmelt + 0.5f) * 2.0f, 0.0f, 1.0f);
    const float zrunf = zfrez * clip((wpw + c.wipud) / P.wpudmax, 0.0f, 1.0f);
    wpw = wpw + (1.0f - zrunf) * raing_avg * dt;
    grunof = grunof + zrunf * raing_avg;
    const bool evap = fvapg_avg >= 0.0f;
    const float edt = fvapg_avg * dt;
    const float fwtop = evap ? -G.q1 * fvapg_avg : 0.0f;
    wpw = wpw - (evap ? G.q3 : G.q1 + G.q3) * edt;
    float wiw = c.wipud - (evap ? G.q4 : G.q2 + G.q4) * edt;
    if (evap) {
        const float w0 = wsw[0].lo(), i0 = wisw[0].lo();
        const float isub = G.q2 * edt / mx(P.rhow * por[0].lo() * P.hsoi[0], eps);
        const float i0n = mx(0.0f, i0 - isub);
        wsw[0] = F2((1.0f - i0n) > eps ? w0 * (1.0f - i0) / (1.0f - i0n) : w0, wsw[0].hi());
        wisw[0] = F2(i0n, wisw[0].hi());
    }
    wpw = mx(wpw, 0.0f);
    wiw = mx(wiw, 0.0f);
    const float z1w = mx(1.0f - (evap ? wisw[0].lo() : mx(0.0f, c.wisoi[0])), 0.0f);
    const float zdpud = P.rhow * dt * (z1w * z1w) * S(IBIS_STAT_HYDRAUL, 0);
    const float fwpud = mx(0.0f, mn(wpw, zdpud)) * P.rdt;
    const float c0pud0 = P.ch2o * wpw + P.cice * wiw;
    const float gtransu = M.fvaput * 2.0f * lai1 * fu;
    const float gtransl = M.fvaplt * 2.0f * lai0 * fl * (1.0f - fi);
    F2 dtp[NP];
    {
        // root uptake: by the layers' stress, or by the root profile where nothing is stressed
        const bool fullu = G.stresstu >= 1.0f, fulll = G.stresstl >= 1.0f;
        const float gu = fullu ? gtransu : gtransu / mx(G.stresstu, eps);
        const float gl = fulll ? gtransl : gtransl / mx(G.stresstl, eps);
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const F2 frl(P.frl2[j]), fru(P.fru2[j]);
            const F2 z(G.zw[2 * j], G.zw[2 * j + 1]);
            const F2 uu = fru * gu * (fullu ? F2(1.0f) : z), ul = frl * gl * (fulll ? F2(1.0f) : z);
            const F2 h = F2(P.h2[j]);
            pflo[j] = mx2(por[j] * mx2(1.0f - wisw[j], eps), eps);
            wsw[j] = mx2(wsw[j] - (uu + ul) * (dt / P.rhow) * rcp2(pflo[j] * h), 0.0f);
            F2 cx = (rsol[j] + por[j] * P.rhow * ((1.0f - wisw[j]) * wsw[j] * P.ch2o + wisw[j] * P.cice)) * h;
            if (j == 0) cx = cx + F2(c0pud0, 0.0f);
            dtp[j] = (uu * (tu - t[j]) + ul * (tl - t[j])) * (-dt * P.ch2o) * rcp2(mx2(cx, eps));
        }
    }
    const float tpt0 = t[0].lo() + dtp[0].lo();
    const float fhtop_soil = heatg_avg + raing_avg * P.ch2o * (traing_avg - tpt0) -
                             grunof * P.ch2o * mx(P.tmelt - tpt0, 0.0f);
    F2 wnew[NP];
#pragma unroll
    for (int j = 0; j < NP; ++j) wnew[j] = wsw[j];
    float wflo[NL + 1], wpud = wpw;
    soil_water32(wnew, wpud, wflo, wisw, por, pflo, S, fwtop, fwpud, P);
    const float c1pud0 = P.ch2o * wpud + P.cice * wiw;
    float hflo[NL + 1], tb[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) tb[k] = c.tsoi_deep[k];
    soil_heat32<NT, DIAG>(t, tb, hflo, dtp, wsw, wnew, wisw, por, cons, rsol, c0pud0, c1pud0, fhtop_soil, wflo, P);
    float gadj = water_bounds32<DIAG>(wnew, wisw, por, P);
    phase_change32(t, wnew, wisw, por, rsol, c1pud0, P);
    float pflo_ft[NL];
    if constexpr (DIAG) {
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const F2 p = por[j] * mx2(1.0f - wisw[j], eps);
            pflo_ft[2 * j] = p.lo();
            pflo_ft[2 * j + 1] = p.hi();
        }
    }
    {
        float t0 = t[0].lo();
        puddle_phase32(t0, wpud, wiw, por[0].lo(), wnew[0].lo(), wisw[0].lo(), rsol[0].lo(), P);
        t[0] = F2(t0, t[0].hi());
    }
    gadj = gadj + water_bounds32<DIAG>(wnew, wisw, por, P);
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        c.tsoi[2 * j] = t[j].lo(); c.tsoi[2 * j + 1] = t[j].hi();
        c.wsoi[2 * j] = wnew[j].lo(); c.wsoi[2 * j + 1] = wnew[j].hi();
        c.wisoi[2 * j] = wisw[j].lo(); c.wisoi[2 * j + 1] = wisw[j].hi();
    }
    if constexpr (NT > NL) {
#pragma unroll
        for (int k = 0; k < NB; ++k) c.tsoi_deep[k] = tb[k];
    }
    c.wpud = wpud;
    c.wipud = wiw;

    // ---- 12. surface temperature bound (loops.py:1143-1151)
    const float lo_ = F.ta - P.t_max_dev, hi_ = F.ta + P.t_max_dev;
    c.tu = clip(c.tu, lo_, hi_);
    c.ts = clip(c.ts, lo_, hi_);
    c.tl = clip(c.tl, lo_, hi_);
    c.tg = clip(c.tg, lo_, hi_);
    fire_counters(c, S(IBIS_STAT_SWILT, 0), F, P);

    if (D.on()) {
        float consoi[NL], stressu[NL], stressl[NL];
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            consoi[k] = k & 1 ? cons[k / 2].hi() : cons[k / 2].lo();
            stressl[k] = G.zw[k] * P.froot[2 * k];
            stressu[k] = G.zw[k] * P.froot[2 * k + 1];
        }
        ground_diagnostics(D, consoi, stressu, stressl, pflo_ft, hflo, heatg_avg, G.stresstu, G.stresstl, gtransu,
                           gtransl, grunof, wflo[NL], gadj, raing_avg, traing_avg, fhtop_soil, sflo_bot, fhtop_snow);
    }

    // ---- accumulators of the day loop (loops_gswp3.py:161-318)
    if (!Ac.base) return;
    if (P.flags & IBIS_FLAG_ACC) {
        const float smask = 1.0f - c.fi;
        F2 rt(0.0f);
#pragma unroll
        for (int j = 0; j < NP; ++j)
            rt = rt + t[j] * (F2(P.frl2[j]) + F2(P.fru2[j]));
        const F2 tr = mx2(F2(c.ts, 0.5f * rt.sum()), 200.0f);
        const F2 fun = ex2((float(1.0 / 288.16) - rcp2(tr)) * 3500.0f);
        const float funca = fun.lo(), funcb = fun.hi();
        S.renew();
        const float cf = 12.0e-3f * dt;
        const float covu = lai1 * fu, covl = lai0 * fl * smask, wsu = funca * S(IBIS_STAT_SAPFRAC);
        // with gpp_split_by_capacity (X3), each big leaf's GPP is divided among its
        // PFTs by leaf area x vmax, re-normalised to the leaf-area sum
        // (capacity_shares, stomata.py:566-577; loops_gswp3.py:197-205)
        float rcap[3] = {0.0f, 0.0f, 0.0f};
        bool by_cap[3] = {false, false, false};
        if constexpr (Q::x3) {
            if (P.flags & IBIS_FLAG_GPP_CAPACITY) {
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    by_cap[g] = G.rcap[g] >= 0.0f;
                    rcap[g] = G.rcap[g];
                }
            }
        }
        F2 npp(0.0f);
#pragma unroll
        for (int j = 0; j < 12; j += 2) {
            // PFTs 3, 5, 7 are conifers, the other trees broadleaf; 8, 9 shrubs; 10 C4, 11 C3 grass
            const F2 an = j == 0   ? F2(M.an_u[0], M.an_u[0])
                          : j < 8  ? F2(M.an_u[0], M.an_u[1])
                          : j == 8 ? F2(M.an_l[0], M.an_l[0])
                                   : F2(M.an_l[2], M.an_l[1]);
            F2 share = stat2(S, IBIS_STAT_FRAC, j);
            if constexpr (Q::x3) {
                if (j < 10) {
                    const int g0 = j < 8 ? 0 : 2, g1 = j == 0 ? 0 : (j < 8 ? 1 : 2);
                    share = sel2(by_cap[g0], by_cap[g1], share * F2(q.vmax(j), q.vmax(j + 1)) * F2(rcap[g0], rcap[g1]),
                                 share);
                }
            }
            F2 r = F2(q.rroot2(j)) * stat2(S, IBIS_STAT_CBIOR, j) * funcb;
            if (j < 10) r = r + F2(q.rwood2(j)) * stat2(S, IBIS_STAT_CBIOW, j) * (j < 8 ? wsu : funca);
            const F2 inc = F2(q.keep2(j)) * (an * share * (j < 8 ? covu : covl) - r) * cf;
            const F2 grew = Ac.add2(IBIS_ACC_AYNPP + j, IBIS_ACC_AYNPP + j + 1, inc);
            npp = npp + (Ac.kahan ? inc : grew);
        }
        auto fr = [&](int j) { return S(IBIS_STAT_FRAC, j); };
        const float gu = (M.ag_u[0] * (fr(0) + fr(1) + fr(2) + fr(4) + fr(6)) + M.ag_u[1] * (fr(3) + fr(5) + fr(7))) * covu;
        const float gl = (M.ag_l[0] * (fr(8) + fr(9)) + M.ag_l[2] * fr(10) + M.ag_l[1] * fr(11)) * covl;
        const float nppt = npp.sum();
        Ac.add2(IBIS_ACC_ADRAIN, IBIS_ACC_ADSNOW, F2(F.rain, F.snow) * dt);
        Ac.add2(IBIS_ACC_ADAET, IBIS_ACC_AFSENA, F2(M.ginvap + M.gsuvap + M.gtrans, M.fsena) * dt);
        Ac.add2(IBIS_ACC_A10ANCUB, IBIS_ACC_A10ANCLS, F2(M.an_u[0], M.an_l[0]) * dt);
        Ac.add2(IBIS_ACC_A10ANCL3, IBIS_ACC_A10ANCL4, F2(M.an_l[1], M.an_l[2]) * dt);
        Ac.add2(IBIS_ACC_AYNPPTOT, IBIS_ACC_AYGPPTOT, F2(nppt, (gu + gl) * cf));
        Ac.add2(IBIS_ACC_AYTRUNOF, IBIS_ACC_AYTDRAIN, F2(grunof, wflo[NL]) * dt);
        // the optional ET components (loops_gswp3.py:263-272): the fluxes summed into
        // adaet, kept apart, sublimation from the snow cover taken out of soil evaporation
        if (P.flags & IBIS_FLAG_ETPARTS) {
            const float snowsub = M.fvapi * c.fi * dt;
            Ac.add(IBIS_ACC_ET_TRANS, M.gtrans * dt);
            Ac.add(IBIS_ACC_ET_INTERC, M.ginvap * dt);
            Ac.add(IBIS_ACC_ET_SOILEV, M.gsuvap * dt - snowsub);
            Ac.add(IBIS_ACC_ET_SNOWSUB, snowsub);
        }
        // the optional day/night NEE (loops_gswp3.py:274-281): the day's Rh rate spread
        // evenly over the steps less this step's NPP, booked to the night when the sun is
        // below the horizon
        if (P.flags & IBIS_FLAG_NEEPARTS) {
            const float nee = S(IBIS_STAT_TCO2MIC) * cf - nppt;
            Ac.add(F.cosz <= 0.0f ? IBIS_ACC_NEE_NIGHT : IBIS_ACC_NEE_DAY, nee);
        }
        if (Ac.last && Ac.live) {
            Ac.at(IBIS_ACC_STRESSTU_LAST) = G.stresstu;
            Ac.at(IBIS_ACC_STRESSTL_LAST) = G.stresstl;
        }
    }
    if (P.flags & IBIS_FLAG_CH4) {
        const float rh = S(IBIS_STAT_TCO2MIC) * P.rh_conv;
        const float zo = (P.flags & IBIS_FLAG_ZWT_OBS) ? S(IBIS_STAT_ZWT_OBS) : NAN;
        const Ch4Par<float> m = ch4_params((P.flags & IBIS_FLAG_CH4_BANDS) ? S(IBIS_STAT_CH4_BAND) : 0.0f, P, q);
        const float flux = methane32(S(IBIS_STAT_F_INUND), rh, t, wnew, wisw, zo, m, P);
        Ac.add2(IBIS_ACC_CH4, -1, F2(flux * P.ch4_w, 0.0f));
    }
    if (P.flags & IBIS_FLAG_SOIL_MEANS) {
#pragma unroll 1
        for (int k = 0; k < NL; ++k) {
            Ac.add(IBIS_ACC_TSOI_MEAN + k, c.tsoi[k] * P.ch4_w);
            Ac.add(IBIS_ACC_WSOI_MEAN + k, c.wsoi[k] * P.ch4_w);
            Ac.add(IBIS_ACC_WISOI_MEAN + k, c.wisoi[k] * P.ch4_w);
        }
        Ac.add(IBIS_ACC_TG_MEAN, c.tg * P.ch4_w);
    }
}

}  // namespace ibis

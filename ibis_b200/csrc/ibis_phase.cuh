// What the two phases of an hour share between the float64 kernels' templates
// (ibis_step.cuh) and the FP32 kernels' form (ibis_f32.cuh): the accumulator view,
// the values the surface phase hands to the ground phase, the diagnostics writers.
#pragma once
#include "ibis_canopy.cuh"
#include "ibis_ground.cuh"
#include "ibis_pair.cuh"

namespace ibis {

// ---- accumulators kept on chip
//
// A kernel that holds a launch's accumulators in shared memory holds the sums every
// day loop keeps (kAccSlots of them, two to a 64-bit word so that a pair is one
// load, one packed Kahan step and one store); the others -- the day means of the
// soil state, the last hour's stress and the optional ET and NEE components, all
// written only under their own flags or once a launch -- stay in the global buffer:
// two blocks of 128 fill an SM's shared memory without them (231 of 233 KB).  With the
// 19 day means, 95,333 columns x 24 hours take 1.66 against 1.37 ms, x 6 hours 0.50
// against 0.40, 356 x 24 hours 0.52 against 0.35.
constexpr int kAccSlots = 25;
constexpr int kAccPairs = (kAccSlots + 1) / 2;

__host__ __device__ constexpr int acc_slot_plane(int s) {
    return s < 3    ? IBIS_ACC_ADRAIN + s
           : s == 3 ? IBIS_ACC_AFSENA
           : s < 8  ? IBIS_ACC_A10ANCUB + (s - 4)
           : s < 20 ? IBIS_ACC_AYNPP + (s - 8)
           : s < 24 ? IBIS_ACC_AYNPPTOT + (s - 20)
                    : IBIS_ACC_CH4;
}
static_assert(IBIS_ACC_ADAET == IBIS_ACC_ADRAIN + 2 && IBIS_ACC_A10ANCL4 == IBIS_ACC_A10ANCUB + 3 &&
                  IBIS_ACC_AYNPPTOT == IBIS_ACC_AYNPP + 12 && IBIS_ACC_AYTDRAIN == IBIS_ACC_AYNPPTOT + 3,
              "acc_slot_plane walks the layout's runs of planes");

__host__ __device__ constexpr int acc_slot(int plane) {
    int r = -1;
    for (int s = 0; s < kAccSlots; ++s)
        if (acc_slot_plane(s) == plane) r = s;
    return r;
}

// Accumulator view of one cell.  In the global form (SLD = 0) ``base`` addresses
// every plane with leading dimension ``ld`` and the compensation term of plane p is
// plane p + IBIS_ACC_COUNT.  In the on-chip form (SLD = the distance of a thread's
// words) chip[j * SLD] holds pair j of the slots above and its two compensation
// terms, zero without compensation, one 128-bit access each way; ``base`` is still the
// global buffer, for the planes that have no slot.  ``live`` is false for a lane that repeats another's cell.
template <typename R, int SLD = 0>
struct Acc {
    R* __restrict__ base;  // nullptr: no accumulators
    int ld;
    bool kahan;
    bool last = true;      // the launch's last hour for this cell: keep the end-of-hour values
    float4* __restrict__ chip = nullptr;
    bool live = true;
    float keep = 0.0f;     // on chip: 1 with compensation, 0 without
    __device__ __forceinline__ void on_chip(float4* p) { chip = p; keep = kahan ? 1.0f : 0.0f; }
    __device__ __forceinline__ R& at(int plane) const { return base[(size_t)plane * ld]; }
    __device__ __forceinline__ R& comp(int plane) const { return base[(size_t)(plane + IBIS_ACC_COUNT) * ld]; }
    __device__ __forceinline__ void add(int plane, R x) const {
        if (!live) return;
        R& v = at(plane);
        if (kahan) {
            R& cmp = comp(plane);
            R s = v, cc = cmp;
            R y = x - cc;
            R t = s + y;
            cmp = (t - s) - y;
            v = t;
        } else {
            v = v + x;
        }
    }
    __device__ __forceinline__ R get(int plane) const { return at(plane); }
    // Two planes at once (FP32 kernels); returns what their sums grew by.  With
    // slots, p0 is an even one and p1 the next (p1 < 0: p0 alone).
    __device__ __forceinline__ F2 add2(int p0, int p1, const F2& x) const {
        if constexpr (SLD == 0) {
            if (!live) return x;     // the planes are the repeated cell's to read, too
        }
        F2 s, cc(0.0f);
        if constexpr (SLD > 0) {
            const float4 v = chip[(acc_slot(p0) >> 1) * SLD];
            s = F2(v.x, v.y);
            cc = F2(v.z, v.w);
        } else {
            s = F2(at(p0), p1 < 0 ? 0.0f : at(p1));
            if (kahan) cc = F2(comp(p0), p1 < 0 ? 0.0f : comp(p1));
        }
        const F2 y = x - cc;
        const F2 t = s + y;
        const F2 d = t - s;
        const F2 cn = d - y;
        if constexpr (SLD > 0) {
            const F2 ck = cn * keep;
            chip[(acc_slot(p0) >> 1) * SLD] = make_float4(t.lo(), t.hi(), ck.lo(), ck.hi());
        } else {
            at(p0) = t.lo();
            if (p1 >= 0) at(p1) = t.hi();
            if (kahan) {
                comp(p0) = cn.lo();
                if (p1 >= 0) comp(p1) = cn.hi();
            }
        }
        return d;
    }
};

// Values the surface phase (steps 1-9 of timestep_body) hands to the ground
// phase (steps 10-12 and the accumulators).  In the fused kernel they stay in
// registers; the two-kernel form passes them through a scratch buffer of
// IBIS_MID_COUNT planes.
template <typename R>
struct Mid {
    R heatg, heati, fvapg, fvapi, fvaput, fvaplt, ginvap, gsuvap, gtrans;
    R raing, traing, snowg, tsnowg, rainl, trainl, snowl, tsnowl;
    R an_u[2], ag_u[2], an_l[3], ag_l[3];
    R fsena;
};
constexpr int kMidCount = 28;

template <typename R>
__device__ __forceinline__ void mid_store(const Mid<R>& m, R* __restrict__ p, int ld) {
    const R v[kMidCount] = {m.heatg, m.heati, m.fvapg, m.fvapi, m.fvaput, m.fvaplt, m.ginvap, m.gsuvap, m.gtrans,
                            m.raing, m.traing, m.snowg, m.tsnowg, m.rainl, m.trainl, m.snowl, m.tsnowl,
                            m.an_u[0], m.an_u[1], m.ag_u[0], m.ag_u[1], m.an_l[0], m.an_l[1], m.an_l[2],
                            m.ag_l[0], m.ag_l[1], m.ag_l[2], m.fsena};
#pragma unroll
    for (int q = 0; q < kMidCount; ++q) p[(size_t)q * ld] = v[q];
}

template <typename R>
__device__ __forceinline__ void mid_load(Mid<R>& m, const R* __restrict__ p, int ld) {
    R v[kMidCount];
#pragma unroll
    for (int q = 0; q < kMidCount; ++q) v[q] = p[(size_t)q * ld];
    m.heatg = v[0]; m.heati = v[1]; m.fvapg = v[2]; m.fvapi = v[3]; m.fvaput = v[4]; m.fvaplt = v[5];
    m.ginvap = v[6]; m.gsuvap = v[7]; m.gtrans = v[8];
    m.raing = v[9]; m.traing = v[10]; m.snowg = v[11]; m.tsnowg = v[12];
    m.rainl = v[13]; m.trainl = v[14]; m.snowl = v[15]; m.tsnowl = v[16];
    m.an_u[0] = v[17]; m.an_u[1] = v[18]; m.ag_u[0] = v[19]; m.ag_u[1] = v[20];
    m.an_l[0] = v[21]; m.an_l[1] = v[22]; m.an_l[2] = v[23];
    m.ag_l[0] = v[24]; m.ag_l[1] = v[25]; m.ag_l[2] = v[26];
    m.fsena = v[27];
}

// setsoi (soil_physics.py:37-140): evaporation source fractions and latent heats
template <typename R>
__device__ __forceinline__ void evap_sources(const Col<R>& c, const Forc<R>& F, const DevParams<R>& P, R& q1, R& q2,
                                             R& q3, R& q4, R& hvasug, R& hvasui) {
    const R eps = P.epsilon;
    {
        R pud = c.wpud + c.wipud;
        R zwpud = clip(P.zwpmax * pud / mx(P.wpudmax, eps), R(0.0), P.zwpmax);
        R w0 = c.wsoi[0], i0 = c.wisoi[0];
        R zwsoi = (R(1.0) - i0) * w0 + i0;
        bool soilw = zwsoi >= eps, haspud = zwpud >= eps;
        R r1 = R(1.0) / mx(zwsoi, eps);
        R r2 = R(1.0) / mx(pud, eps);
        q1 = soilw ? (haspud ? (R(1.0) - zwpud) * (R(1.0) - i0) * w0 * r1 : (R(1.0) - i0) * w0 * r1) : R(0.0);
        q2 = soilw ? (haspud ? (R(1.0) - zwpud) * i0 * r1 : i0 * r1) : R(0.0);
        bool warm = c.tsoi[0] >= P.tmelt - R(1.0e-9);
        q3 = haspud ? zwpud * c.wpud * r2 : (soilw ? R(0.0) : (warm ? R(1.0) : R(0.0)));
        q4 = haspud ? zwpud * c.wipud * r2 : (soilw ? R(0.0) : (warm ? R(0.0) : R(1.0)));
        R zvap = P.hvap + P.cvap * (F.ta - P.tmelt) - P.ch2o * (c.tsoi[0] - P.tmelt);
        R zsub = P.hsub + P.cvap * (F.ta - P.tmelt) - P.cice * (c.tsoi[0] - P.tmelt);
        hvasug = (q1 + q3) * zvap + (q2 + q4) * zsub;
        hvasui = P.hsub + P.cvap * (F.ta - P.tmelt) - P.cice * (c.tsno[0] - P.tmelt);
    }
}

// capacity_shares (stomata.py:566-577) of one big leaf: the capacity-weighted
// leaf area (floored at 1e-12), the leaf area, and whether the capacity shares apply
template <typename R, int N, typename Q>
__device__ __forceinline__ void capacity_group(const int (&idx)[N], const Stat<R>& S, const Q& q, R& twm, R& tf,
                                               bool& on) {
    R tw = R(0.0);
    tf = R(0.0);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const R f = S(IBIS_STAT_FRAC, idx[i]);
        tw = tw + f * q.vmax(idx[i]);
        tf = tf + f;
    }
    on = tw > R(1.0e-12);
    twm = mx(tw, R(1.0e-12));
}

// ---- diagnostics of the radiation (loops.py:1158-1241)
template <typename R, typename DD>
__device__ __forceinline__ void radiation_diagnostics(const DD& to, const Rad<R>& Rd) {
    const DD D = to.renewed();
            D.put(IBIS_DIAG_SOLU, Rd.solu); D.put(IBIS_DIAG_SOLS, Rd.sols); D.put(IBIS_DIAG_SOLL, Rd.soll);
            D.put(IBIS_DIAG_SOLG, Rd.solg); D.put(IBIS_DIAG_SOLI, Rd.soli);
            D.put(IBIS_DIAG_FIRU, Rd.firu); D.put(IBIS_DIAG_FIRS, Rd.firs); D.put(IBIS_DIAG_FIRL, Rd.firl);
    #pragma unroll
            for (int b = 0; b < 2; ++b) { D.put(IBIS_DIAG_ASURD, b, Rd.asurd[b]); D.put(IBIS_DIAG_ASURI, b, Rd.asuri[b]); }
            D.put(IBIS_DIAG_TOPPARU, Rd.topparu); D.put(IBIS_DIAG_TOPPARL, Rd.topparl);
    #pragma unroll
            for (int j = 0; j < 4; ++j) { D.put(IBIS_DIAG_SCALCOEFU, j, Rd.scu[j]); D.put(IBIS_DIAG_SCALCOEFL, j, Rd.scl[j]); }
}

// ---- diagnostics of the surface phase (loops.py:1158-1241)
template <typename R, typename DD>
__device__ __forceinline__ void surface_diagnostics(const DD& to, const Stom<R>& st, R fwetu, R fwets, R fwetl, R rliqu,
                                                    R rliqs, R rliql, R firg, R firi, R firb,
                                                    R fsenu, R fsens, R fsenl, R fseng, R fseni, const Mid<R>& M,
                                                    R rhoa, R hvasug, R hvasui, R q1, R q2, R q3, R q4) {
    const DD D = to.renewed();
    #pragma unroll
            for (int j = 0; j < 2; ++j) { D.put(IBIS_DIAG_AN_UPPER, j, st.an_u[j]); D.put(IBIS_DIAG_AG_UPPER, j, st.ag_u[j]); }
    #pragma unroll
            for (int j = 0; j < 3; ++j) { D.put(IBIS_DIAG_AN_LOWER, j, st.an_l[j]); D.put(IBIS_DIAG_AG_LOWER, j, st.ag_l[j]); }
            D.put(IBIS_DIAG_FWETU, fwetu); D.put(IBIS_DIAG_FWETS, fwets); D.put(IBIS_DIAG_FWETL, fwetl);
            D.put(IBIS_DIAG_RLIQU, rliqu); D.put(IBIS_DIAG_RLIQS, rliqs); D.put(IBIS_DIAG_RLIQL, rliql);
            D.put(IBIS_DIAG_FIRG, firg); D.put(IBIS_DIAG_FIRI, firi); D.put(IBIS_DIAG_FIRB, firb);
            D.put(IBIS_DIAG_FSENU, fsenu); D.put(IBIS_DIAG_FSENS, fsens); D.put(IBIS_DIAG_FSENL, fsenl);
            D.put(IBIS_DIAG_FSENG, fseng); D.put(IBIS_DIAG_FSENI, fseni);
            D.put(IBIS_DIAG_FVAPG, M.fvapg); D.put(IBIS_DIAG_FVAPI, M.fvapi);
            D.put(IBIS_DIAG_RAING, M.raing); D.put(IBIS_DIAG_SNOWG, M.snowg); D.put(IBIS_DIAG_RHOA, rhoa);
            D.put(IBIS_DIAG_HVASUG, hvasug); D.put(IBIS_DIAG_HVASUI, hvasui);
            D.put(IBIS_DIAG_QGLIF, 0, q1); D.put(IBIS_DIAG_QGLIF, 1, q2); D.put(IBIS_DIAG_QGLIF, 2, q3); D.put(IBIS_DIAG_QGLIF, 3, q4);
            D.put(IBIS_DIAG_HEATI, M.heati);
            D.put(IBIS_DIAG_GINVAP, M.ginvap); D.put(IBIS_DIAG_GSUVAP, M.gsuvap); D.put(IBIS_DIAG_GTRANS, M.gtrans);
            D.put(IBIS_DIAG_RAINL, M.rainl); D.put(IBIS_DIAG_SNOWL, M.snowl);
            D.put(IBIS_DIAG_TRAINL, M.trainl); D.put(IBIS_DIAG_TSNOWL, M.tsnowl);
            D.put(IBIS_DIAG_FSENA, M.fsena);
}

// ---- diagnostics of the ground phase (loops.py:1158-1241)
template <typename R, typename DD>
__device__ __forceinline__ void ground_diagnostics(const DD& to, const R (&consoi)[NL], const R (&stressu)[NL],
                                                   const R (&stressl)[NL], const R (&pflo_ft)[NL],
                                                   const R (&hflo)[NL + 1], R heatg_avg, R stresstu, R stresstl,
                                                   R gtransu, R gtransl, R grunof, R gdrain, R gadj, R raing_avg,
                                                   R traing_avg, R fhtop_soil, R sflo_bot, R fhtop_snow) {
    const DD D = to.renewed();
    #pragma unroll
            for (int k = 0; k < NL; ++k) {
                D.put(IBIS_DIAG_CONSOI, k, consoi[k]);
                D.put(IBIS_DIAG_STRESSU, k, stressu[k]);
                D.put(IBIS_DIAG_STRESSL, k, stressl[k]);
                D.put(IBIS_DIAG_POROSFLO, k, pflo_ft[k]);
            }
    #pragma unroll
            for (int k = 0; k <= NL; ++k) D.put(IBIS_DIAG_HFLO, k, hflo[k]);
            D.put(IBIS_DIAG_HEATG, heatg_avg);
            D.put(IBIS_DIAG_STRESSTU, stresstu); D.put(IBIS_DIAG_STRESSTL, stresstl);
            D.put(IBIS_DIAG_GTRANSU, gtransu); D.put(IBIS_DIAG_GTRANSL, gtransl); D.put(IBIS_DIAG_GRUNOF, grunof);
            D.put(IBIS_DIAG_GDRAIN, gdrain); D.put(IBIS_DIAG_GADJUST, gadj); D.put(IBIS_DIAG_WTOT, R(0.0));
            D.put(IBIS_DIAG_RAING_AVG, raing_avg); D.put(IBIS_DIAG_TRAING_AVG, traing_avg);
            D.put(IBIS_DIAG_FHTOP_SOIL, fhtop_soil);
            D.put(IBIS_DIAG_SFLO_BOT, sflo_bot); D.put(IBIS_DIAG_FHTOP_SNOW, fhtop_snow);
}

}  // namespace ibis

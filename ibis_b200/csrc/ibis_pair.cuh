// Two floats in one 64-bit register pair, worked on by the packed single-precision
// instructions of sm_100 (add, sub, mul, fma .f32x2): one instruction does the
// arithmetic of two leaves, two radiation bands, two canopy stories or two soil
// layers.  The hourly step is bound by how fast its instructions can be fetched and
// issued, not by any arithmetic pipe, so halving them is what these pairs are for.
// A product and the sum or difference it feeds are contracted to one fma, as in scalar
// code: measured, a * b + c, a * b - c and c - a * b of 4,096 operand triples chosen so that
// the two roundings differ give the fused result in every one.  The code does not rely on
// it; where one rounding is meant it says fma2.
// Rounding is that of the scalar operations (round to nearest, denormals flushed
// as -use_fast_math does).
#pragma once
#include "ibis_math.cuh"
#include "ibis_params.cuh"

namespace ibis {

struct F2 {
    unsigned long long v;
    __device__ __forceinline__ F2() {}
    __device__ __forceinline__ F2(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
    __device__ __forceinline__ F2(float s) : F2(s, s) {}
    __device__ __forceinline__ F2(const ParPair& p) : v(p.v) {}
    __device__ __forceinline__ float lo() const {
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
        return a;
    }
    __device__ __forceinline__ float hi() const {
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
        return b;
    }
    __device__ __forceinline__ float sum() const { return lo() + hi(); }
};

#define IBIS_F2_OP(op, name)                                                                                \
    __device__ __forceinline__ F2 operator op(const F2& a, const F2& b) {                                   \
        F2 r;                                                                                               \
        asm(name ".rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));                             \
        return r;                                                                                           \
    }                                                                                                       \
    __device__ __forceinline__ F2 operator op(const F2& a, float b) { return a op F2(b); }                  \
    __device__ __forceinline__ F2 operator op(float a, const F2& b) { return F2(a) op b; }
IBIS_F2_OP(+, "add")
IBIS_F2_OP(-, "sub")
IBIS_F2_OP(*, "mul")
#undef IBIS_F2_OP

// a * b + c in one rounding
__device__ __forceinline__ F2 fma2(const F2& a, const F2& b, const F2& c) {
    F2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

__device__ __forceinline__ F2 mx2(const F2& a, const F2& b) { return F2(fmaxf(a.lo(), b.lo()), fmaxf(a.hi(), b.hi())); }
__device__ __forceinline__ F2 mn2(const F2& a, const F2& b) { return F2(fminf(a.lo(), b.lo()), fminf(a.hi(), b.hi())); }
__device__ __forceinline__ F2 clip2(const F2& x, float lo, float hi) { return mn2(mx2(x, lo), hi); }
__device__ __forceinline__ F2 abs2(const F2& a) { return F2(fabsf(a.lo()), fabsf(a.hi())); }
__device__ __forceinline__ F2 rcp2(const F2& a) { return F2(1.0f / a.lo(), 1.0f / a.hi()); }
__device__ __forceinline__ F2 sq2(const F2& a) { return F2(sqrtf(a.lo()), sqrtf(a.hi())); }
__device__ __forceinline__ F2 exp2_2(const F2& a) { return F2(exp2f(a.lo()), exp2f(a.hi())); }
// e**a = 2**(a log2 e)
__device__ __forceinline__ F2 ex2(const F2& a) { return exp2_2(a * 1.4426950408889634f); }
__device__ __forceinline__ F2 lg2(const F2& a) { return F2(logf(a.lo()), logf(a.hi())); }
__device__ __forceinline__ F2 sel2(bool a, bool b, const F2& x, const F2& y) {
    return F2(a ? x.lo() : y.lo(), b ? x.hi() : y.hi());
}
__device__ __forceinline__ F2 sel2(bool a, const F2& x, const F2& y) { return sel2(a, a, x, y); }

// x**n per half for 0 <= n < 64, by repeated squaring.  Exponents of 16 and more
// (a soil's Clapp-Hornberger exponent above 14) take the branch.
__device__ __forceinline__ F2 ipow2(F2 x, int n0, int n1) {
    float r0 = 1.0f, r1 = 1.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (n0 & (1 << k)) r0 = r0 * x.lo();
        if (n1 & (1 << k)) r1 = r1 * x.hi();
        if (k < 3) x = x * x;
    }
    if ((n0 | n1) >> 4) {
#pragma unroll
        for (int k = 4; k < 6; ++k) {
            x = x * x;
            if (n0 & (1 << k)) r0 = r0 * x.lo();
            if (n1 & (1 << k)) r1 = r1 * x.hi();
        }
    }
    return F2(r0, r1);
}

// The larger or smaller of two doubles by one comparison (the second where the first
// is not a number, as fmax and fmin with an ordinary second)
__device__ __forceinline__ double dmax(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double dmin(double a, double b) { return a < b ? a : b; }

// Lowe (1977) saturation vapour pressure and its derivative (as esat and desat in
// ibis_math.cuh: both branches on offsets clamped to their range) at two
// temperatures: a coefficient is the same for both halves, so each packed fma
// carries it as an immediate.
#define IBIS_LOWE2(t, L0, L1, L2, L3, L4, L5, L6, I0, I1, I2, I3, I4, I5, I6)                                   \
    do {                                                                                                        \
        const F2 d_ = (t) - 273.16f;                                                                            \
        const F2 l_ = clip2(d_, 0.0f, 100.0f), i_ = clip2(d_, -60.0f, 0.0f);                                    \
        const F2 base_((t).lo() >= 273.16f ? float(L0) : float(I0), (t).hi() >= 273.16f ? float(L0) : float(I0)); \
        F2 p_ = fma2(l_, F2(float(L6)), F2(float(L5)));                                                         \
        F2 q_ = fma2(i_, F2(float(I6)), F2(float(I5)));                                                         \
        p_ = fma2(l_, p_, F2(float(L4))); q_ = fma2(i_, q_, F2(float(I4)));                                     \
        p_ = fma2(l_, p_, F2(float(L3))); q_ = fma2(i_, q_, F2(float(I3)));                                     \
        p_ = fma2(l_, p_, F2(float(L2))); q_ = fma2(i_, q_, F2(float(I2)));                                     \
        p_ = fma2(l_, p_, F2(float(L1))); q_ = fma2(i_, q_, F2(float(I1)));                                     \
        return fma2(i_, q_, fma2(l_, p_, base_)) * 100.0f;                                                      \
    } while (0)

__device__ __forceinline__ F2 esat2(const F2& t) {
    IBIS_LOWE2(t, 6.1078000, 4.4365185e-1, 1.4289458e-2, 2.6506485e-4, 3.0312404e-6, 2.0340809e-8, 6.1368209e-11,
               6.1091780, 5.0346990e-1, 1.8860134e-2, 4.1762237e-4, 5.8247203e-6, 4.8388032e-8, 1.8388269e-10);
}
__device__ __forceinline__ F2 desat2(const F2& t) {
    IBIS_LOWE2(t, 4.4381000e-1, 2.8570026e-2, 7.9380540e-4, 1.2152151e-5, 1.0365614e-7, 3.5324218e-10,
               -7.0902448e-13, 5.0303052e-1, 3.7732550e-2, 1.2679954e-3, 2.4775631e-5, 3.0056931e-7, 2.1585425e-9,
               7.1310977e-12);
}
#undef IBIS_LOWE2

// Specific humidity at saturation, q = 0.622 e / max(p - 0.378 e, 0.622 e), and its
// derivative desat q (1 + q (1/0.622 - 1)) / e, whose q / e is the same quotient.
__device__ __forceinline__ F2 sat_quotient2(const F2& e, float p) {
    return 0.622f * rcp2(mx2(p - e * float(1.0 - 0.622), e * 0.622f));
}
__device__ __forceinline__ F2 sat_derivative2(const F2& t, const F2& q, const F2& qe) {
    return desat2(t) * qe * (1.0f + q * float(1.0 / 0.622 - 1.0));
}

// Reciprocal of a finite, non-zero double by two Newton-Raphson steps
// y <- y + y (1 - x y) from the hardware's approximation (rcp.approx.ftz.f64, 20 bits):
// the error squares, to 2**-40 and 2**-80, so the last step's one rounding is what is left and
// the result is the correctly rounded reciprocal or its neighbour.  Five dependent
// operations and no special-case path.  Used inside the canopy island of the FP32
// kernels, whose denominators are bounded away from zero.
__device__ __forceinline__ double rcp_nr(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    y = fma(y, fma(-x, y, 1.0), y);
    return fma(y, fma(-x, y, 1.0), y);
}

}  // namespace ibis

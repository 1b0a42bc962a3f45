// Exact arithmetic without data-dependent branches (sm_100a).
//
// The exact policy returns what IEEE float32 arithmetic returns, operation by
// operation.  The compiler's correctly rounded division and square root test
// their operands and branch to a slow path outside a range (a zero numerator is
// outside it), and a step takes about 25 divisions and 5 roots per cell: with them
// the 2048^2 urban step executes 41.9 warp instructions per cell with 21.5 of 32
// lanes active, waits for instruction fetches and branches in 2.8 of 6.9 cycles
// between issues and takes 303 us; with the form below 75.5 us.  QuickExact computes
// the same values from the published sequences for a machine with fused multiply-add (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34(1), 1990):
//
//   reciprocal  y = y0 + y0 (1 - b y0), y0 approximate;
//   quotient    q = a y, then q + (a - b q) y;
//   root        s = x r, then s + (x - s^2)(r / 2), r approximate 1/sqrt(x).
//
// The first and the last are correctly rounded for every mantissa (compared
// with __frcp_rn and __fsqrt_rn over all 2^23 and 2^24 of them), which makes the
// quotient correctly rounded as long as its remainder a - b q is a float: no
// operand so large or small that something over- or underflows (6e9 random and
// adversarial pairs equal __fdiv_rn).  Small operands are kept
// clear of that by scaling: numerators and wave speeds carry a factor
// kUp = 2^32 (a power of two changes no rounding), so a result can differ only
// where the IEEE one is vanishing (a friction divisor above 2^94 makes a momentum
// zero: below 2^-60 in a step that the CFL rule allows; elsewhere below 2^-94), or in
// the sign of a zero.  Large, infinite and NaN operands are caught per row: the march keeps the largest depth
// and speed of the cells of a row; where it is not below kQuickLimit on every lane of
// the warp (a NaN is not) the row takes the IEEE operations, and where only its new
// values leave the range it is computed again with them (two warp-uniform votes per
// row of 64 cells).
//
// Both cells of a lane share each instruction (f32x2).  A packed multiply whose
// result is only added would be contracted with the addition by the assembler,
// whatever its rounding qualifier (measured), so additions are written as
// fma(a, 1, b) with a 1 the compiler cannot see (Consts::one).
#pragma once

#include "swe_pair.cuh"

namespace swe {

constexpr float kUp = 4294967296.0f;            // 2^32
constexpr float kDown = 2.3283064365386963e-10f;  // 2^-32
// Depths (m) and speeds (m/s) from which on a row is computed with the IEEE operations:
// beyond any water on Earth, and with them below it (and gravity up to 2^6, cells from
// 2^-10) no term leaves the float range.  The largest are the HLL numerators, 2^32 x
// speed x momentum flux < 2^49 2^50, and an update's scaled divergence, 2^32 2^52 2^10;
// a momentum that friction multiplies out of the range gives a NaN, which the row's
// largest value shows.  (At 1024, a grid 2000 m deep took the IEEE operations
// everywhere: 2048^2 302 us a step instead of 79.)
constexpr float kQuickLimit = 65536.0f;

// The exact policy's branch-free form (a tag: the operations are PairOps).
struct QuickExact {};

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// Run-time constants of the separately rounded operations of a pair.
struct PairOps {
    float2 one, minus_one;
    __device__ __forceinline__ float2 add(float2 a, float2 b) const { return fma2(a, one, b); }
    __device__ __forceinline__ float2 sub(float2 a, float2 b) const { return fma2(b, minus_one, a); }
    __device__ __forceinline__ float2 mul(float2 a, float2 b) const { return __fmul2_rn(a, b); }
    __device__ __forceinline__ float2 fma(float2 a, float2 b, float2 c) const { return fma2(a, b, c); }
    __device__ __forceinline__ float2 minus(float2 a) const { return {-a.x, -a.y}; }
    __device__ __forceinline__ float2 splat(float a) const { return make_float2(a, a); }
    __device__ __forceinline__ float2 rcp_approx(float2 a) const { return {swe::rcp_approx(a.x), swe::rcp_approx(a.y)}; }
    __device__ __forceinline__ float2 rsqrt_approx(float2 a) const {
        return {swe::rsqrt_approx(a.x), swe::rsqrt_approx(a.y)};
    }
};

// Correctly rounded reciprocal of b (b normal, 1/b normal).
template <class O, class T>
__device__ __forceinline__ T quick_rcp(const O& o, T b) {
    const T y = o.rcp_approx(b);
    return o.fma(y, o.fma(o.minus(b), y, o.splat(1.0f)), y);
}

// Correctly rounded a / b from y = quick_rcp(b).
template <class O, class T>
__device__ __forceinline__ T quick_div(const O& o, T a, T b, T y) {
    const T q = o.mul(a, y);
    return o.fma(o.fma(o.minus(b), q, a), y, q);
}

// a / b, rounded once, for any a and b: the quotient above where no operand comes
// near the ends of the float range (its remainder is then a float) and for a
// zero numerator, which keeps its sign; the IEEE division otherwise.
__device__ __forceinline__ float ranged_div(float a, float b) {
    constexpr float lo = 0x1p-60f, hi = 0x1p60f;
    const float m = fabsf(a);
    if (!(b > lo && b < hi && (m == 0.f || (m > lo && m < hi)))) return __fdiv_rn(a, b);
    float y = rcp_approx(b);
    y = __fmaf_rn(y, __fmaf_rn(-b, y, 1.f), y);
    const float q = __fmul_rn(a, y);
    return m == 0.f ? q : __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

// Correctly rounded square root of x >= 0; `xr` is x, or any positive value where x is zero.
template <class O, class T>
__device__ __forceinline__ T quick_sqrt(const O& o, T x, T xr) {
    const T r = o.rsqrt_approx(xr);
    const T s = o.mul(x, r);
    return o.fma(o.fma(o.minus(s), s, x), o.mul(r, o.splat(0.5f)), s);
}

// hypot as ExactMath::hypot: the correctly rounded double root of s = a^2 + b^2 (the
// squares of floats are exact doubles), rounded once more to float.  The approximate
// reciprocal root y (relative error e at most 2^-20.03, measured over every value of
// the 20 mantissa bits it reads) gives r = s y and h = y / 2; a joint Newton step
// takes both to 1.5 e^2, and the step after it takes r to 3.4 e^4 < 2^-78.3 below the
// root, before its one rounding.  A different double matters only where one of the two
// candidates is a midpoint m of two floats: then s is the double next to m^2, and for
// m in [1, 2) the root lies (m - 1) / 2m or (2 - m) / 2m units from the tie between
// them, 2^-77 relative or more near 1 (m - 1 is at least 2^-24) and 2^-77.4 near 2 but for
// m = 2 - 2^-24, whose neighbouring s is the sum of no two float squares (all
// were tried).  Two steps with the first h reach 1.5 e^3 only and miss one in seventeen
// of the pairs whose sum lies next to such an m^2.  The tiny term keeps the reciprocal
// root finite for a = b = 0; a sum of two float squares that is not zero is at least
// 2e-90, which it does not change.
__device__ __forceinline__ float quick_hypot(float a, float b) {
    const double da = a, db = b;
    const double s = __fma_rn(da, da, __fma_rn(db, db, 1.0e-290));
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
    double h = __dmul_rn(0.5, y);
    double r = __dmul_rn(s, y);
    const double t = __fma_rn(-r, h, 0.5);
    r = __fma_rn(r, t, r);
    h = __fma_rn(h, t, h);
    r = __fma_rn(__fma_rn(-r, r, s), h, r);
    return __double2float_rn(r);
}
__device__ __forceinline__ float2 quick_hypot(float2 a, float2 b) {
    return {quick_hypot(a.x, b.x), quick_hypot(a.y, b.y)};
}

// x ** float32(7/3) (pow73_value) of a pair, from rx = quick_rcp(x).
__device__ __forceinline__ float2 quick_pow73(const PairOps& o, float2 x, float2 rx) {
    const float2 lg = {lg2_approx(x.x), lg2_approx(x.y)};
    const float2 e = o.mul(lg, o.splat(kThird));
    const float2 c = {ex2_approx(e.x), ex2_approx(e.y)};
    return pow73_value(o, x, rx, lg, c);
}

// Maximum that keeps a NaN.
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// ---------------------------------------------------------------------------
// Cells and faces
// ---------------------------------------------------------------------------
// set_vel_t of the exact policy.
template <class O, class T, class KP>
__device__ __forceinline__ void quick_vel(const O& o, CellT<T>& c, const KP& kp) {
    const auto wet = gt(c.h, kp.dry);
    const T y = quick_rcp(o, c.h), up = o.splat(kUp), down = o.splat(kDown);
    c.u = sel(wet, o.mul(quick_div(o, o.mul(c.hu, up), c.h, y), down), kp.zero);
    c.v = sel(wet, o.mul(quick_div(o, o.mul(c.hv, up), c.h, y), down), kp.zero);
}

// kUp * sqrt(g h), from g_up = kUp^2 g.
template <class O, class T>
__device__ __forceinline__ T quick_celerity_up(const O& o, T h, T g_up) {
    return quick_sqrt(o, o.mul(g_up, h), o.fma(g_up, h, o.splat(1.0e-27f)));
}

// face_t of the exact policy: the same operations in the same order, the normal
// velocities, the wave speeds and the numerators and denominator of the HLL
// middle state carrying the factor kUp.
template <int AXIS, bool MASKED, class O, class T, class KP>
__device__ __forceinline__ FaceT<T> quick_face(const O& o, const CellT<T>& lo, const CellT<T>& hi, const KP& kp) {
    T hL = lo.h, zL = lo.z, hR = hi.h, zR = hi.z;
    T uL = lo.u, vL = lo.v, uR = hi.u, vR = hi.v;
    auto relevant = all_true<T>();
    if constexpr (MASKED) {
        const auto a_lo = act_of(lo.nm), a_hi = act_of(hi.nm);
        relevant = a_lo | a_hi;
        const auto hi_wall = a_lo & !a_hi;
        const auto lo_wall = !a_lo & a_hi;
        hL = sel(lo_wall, hi.h, lo.h);
        zL = sel(lo_wall, hi.z, lo.z);
        hR = sel(hi_wall, lo.h, hi.h);
        zR = sel(hi_wall, lo.z, hi.z);
        if constexpr (AXIS == 1) {
            uL = sel(lo_wall, neg(hi.u), lo.u);
            vL = sel(lo_wall, hi.v, lo.v);
            uR = sel(hi_wall, neg(lo.u), hi.u);
            vR = sel(hi_wall, lo.v, hi.v);
        } else {
            uL = sel(lo_wall, hi.u, lo.u);
            vL = sel(lo_wall, neg(hi.v), lo.v);
            uR = sel(hi_wall, lo.u, hi.u);
            vR = sel(hi_wall, neg(lo.v), hi.v);
        }
    }
    const T up = o.splat(kUp), down = o.splat(kDown);
    const T zf = vmax(zL, zR);
    const T HL = vmax(o.sub(o.add(hL, zL), zf), kp.zero);
    const T HR = vmax(o.sub(o.add(hR, zR), zf), kp.zero);
    const T XL = o.mul(HL, uL), YL = o.mul(HL, vL);
    const T XR = o.mul(HR, uR), YR = o.mul(HR, vR);
    const auto wL = gt(HL, kp.dry), wR = gt(HR, kp.dry);
    const T yL = quick_rcp(o, HL), yR = quick_rcp(o, HR);
    // Velocities of the reconstructed momenta (n: normal, t: tangential), times kUp.
    const T nL_up = sel(wL, quick_div(o, o.mul(AXIS == 1 ? XL : YL, up), HL, yL), kp.zero);
    const T nR_up = sel(wR, quick_div(o, o.mul(AXIS == 1 ? XR : YR, up), HR, yR), kp.zero);
    const T unL = o.mul(nL_up, down), unR = o.mul(nR_up, down);
    const T cL = quick_celerity_up(o, HL, kp.g_up), cR = quick_celerity_up(o, HR, kp.g_up);
    const T HHL = o.mul(HL, HL), HHR = o.mul(HR, HR);
    const T pL = o.mul(kp.half_g, HHL), pR = o.mul(kp.half_g, HHR);
    T fL0, fL1, fL2, fR0, fR1, fR2;
    if constexpr (AXIS == 1) {
        const T tL = sel(wL, o.mul(quick_div(o, o.mul(YL, up), HL, yL), down), kp.zero);
        const T tR = sel(wR, o.mul(quick_div(o, o.mul(YR, up), HR, yR), down), kp.zero);
        fL0 = XL;
        fR0 = XR;
        fL1 = o.add(o.mul(XL, unL), pL);
        fR1 = o.add(o.mul(XR, unR), pR);
        fL2 = o.mul(XL, tL);
        fR2 = o.mul(XR, tR);
    } else {
        fL0 = YL;
        fR0 = YR;
        fL1 = o.mul(XL, unL);
        fR1 = o.mul(XR, unR);
        fL2 = o.add(o.mul(YL, unL), pL);
        fR2 = o.add(o.mul(YR, unR), pR);
    }
    const T sL = vmin(o.sub(nL_up, cL), o.sub(nR_up, cR));
    const T sR = vmax(o.add(nL_up, cL), o.add(nR_up, cR));
    const T spread = o.sub(sR, sL);
    const T den = sel(gt(spread, kp.eps_up), spread, up);
    const T yd = quick_rcp(o, den);
    const T s01 = o.mul(sL, o.mul(sR, down));
    const T m0 = quick_div(o, o.add(o.sub(o.mul(sR, fL0), o.mul(sL, fR0)), o.mul(s01, o.sub(HR, HL))), den, yd);
    const T m1 = quick_div(o, o.add(o.sub(o.mul(sR, fL1), o.mul(sL, fR1)), o.mul(s01, o.sub(XR, XL))), den, yd);
    const T m2 = quick_div(o, o.add(o.sub(o.mul(sR, fL2), o.mul(sL, fR2)), o.mul(s01, o.sub(YR, YL))), den, yd);
    const auto take_l = ge(sL, kp.zero), take_r = le(sR, kp.zero);
    FaceT<T> f;
    f.f0 = sel(take_l, fL0, sel(take_r, fR0, m0));
    f.f1 = sel(take_l, fL1, sel(take_r, fR1, m1));
    f.f2 = sel(take_l, fL2, sel(take_r, fR2, m2));
    f.corr_lo = o.mul(kp.half_g, o.sub(o.mul(hL, hL), HHL));
    f.corr_hi = o.mul(kp.half_g, o.sub(o.mul(hR, hR), HHR));
    if constexpr (MASKED) {
        f.f0 = sel(relevant, f.f0, kp.zero);
        f.f1 = sel(relevant, f.f1, kp.zero);
        f.f2 = sel(relevant, f.f2, kp.zero);
        f.corr_lo = sel(relevant, f.corr_lo, kp.zero);
        f.corr_hi = sel(relevant, f.corr_hi, kp.zero);
    }
    return f;
}

}  // namespace swe

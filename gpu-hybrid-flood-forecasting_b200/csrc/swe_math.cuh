// Arithmetic policies for the shallow-water step kernels (sm_100a).
//
// ExactMath rounds every operation on its own, in the order the reference
// NumPy solver performs it (src/hybrid_flood/numpy_solver/shallow_water_2d.py):
// explicit __fadd_rn/__fmul_rn/__fdiv_rn/__fsqrt_rn intrinsics, which the
// compiler never contracts into FMA whatever the -fmad setting.  Its only
// deliberate difference from the reference is the power in the friction term
// (pow73_exact: within 0.50003 ulp of the exact power over the depths of a
// flood, where NumPy's and CUDA's powf reach 0.9 ulp; powf elsewhere).
// hypot is evaluated as glibc's hypotf does (double products, one double sqrt,
// one rounding to float), which NumPy's float32 hypot reproduces.
//
// FastMath keeps the same algorithm but lets the compiler fuse multiply-adds,
// uses the hardware approximate reciprocal / square root / log2 / exp2
// (MUFU), divides the three HLL middle-state components by one reciprocal,
// and uses the identity (H*u)/H == u for the reconstructed velocities.  Its
// results are checked against the oracle with the tolerance the tests state.
#pragma once

#include <cuda_runtime.h>

namespace swe {

__device__ __forceinline__ float rcp_approx(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ float rsqrt_approx(float a) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ float lg2_approx(float a) {
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ float ex2_approx(float a) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// Depths for which pow73_value is used: far beyond a flood's on both sides.
constexpr float kPowLo = 9.3132257e-10f, kPowHi = 1048576.0f;  // 2^-30, 2^20

constexpr float kThird = 0.333333343f;
constexpr float kPow73Ke = (float)(((double)(float)(7.0 / 3.0) - 7.0 / 3.0) * 0.69314718055994530942);

// x ** float32(7/3) = x^2 * cbrt(x) * (1 + d ln x), d = float32(7/3) - 7/3: the
// cube root c from the approximate 2^(log2(x)/3), its relative error
// (c^3 - x) / (3 x) and the products x^2 and x^2 c from error-free products
// (Dekker; the low parts by fma), one rounding at the end.  `rx` is 1/x.
// Measured against the float64 power on every seventh float of [2^-30, 2^13]: at
// most 0.50003 ulp off and not the nearest float for 263 of 51.5 M arguments
// (powf: 0.899 ulp, 3.2 M).  `lg` is the approximate log2(x), `c` 2^(lg/3).
template <class O, class T>
__device__ __forceinline__ T pow73_value(const O& o, T x, T rx, T lg, T c) {
    const T c2h = o.mul(c, c), c2l = o.fma(c, c, o.minus(c2h));
    const T c3h = o.mul(c2h, c), c3l = o.fma(c2l, c, o.fma(c2h, c, o.minus(c3h)));
    const T d = o.add(o.sub(c3h, x), c3l);
    const T kap = o.fma(o.splat(kPow73Ke), lg, o.mul(o.mul(d, rx), o.splat(-kThird)));
    const T x2h = o.mul(x, x), x2l = o.fma(x, x, o.minus(x2h));
    const T ph = o.mul(x2h, c), pl = o.fma(x2l, c, o.fma(x2h, c, o.minus(ph)));
    return o.add(ph, o.fma(ph, kap, pl));
}

// Separately rounded operations on one value (on a pair: PairOps, swe_exact.cuh).
struct SoloOps {
    __device__ __forceinline__ float add(float a, float b) const { return __fadd_rn(a, b); }
    __device__ __forceinline__ float sub(float a, float b) const { return __fsub_rn(a, b); }
    __device__ __forceinline__ float mul(float a, float b) const { return __fmul_rn(a, b); }
    __device__ __forceinline__ float fma(float a, float b, float c) const { return __fmaf_rn(a, b, c); }
    __device__ __forceinline__ float minus(float a) const { return -a; }
    __device__ __forceinline__ float splat(float a) const { return a; }
    __device__ __forceinline__ float rcp_approx(float a) const { return swe::rcp_approx(a); }
    __device__ __forceinline__ float rsqrt_approx(float a) const { return swe::rsqrt_approx(a); }
};

__device__ __forceinline__ float pow73_exact(float x, float expo) {
    if (!(x >= kPowLo && x <= kPowHi)) return powf(x, expo);
    const SoloOps o;
    const float y0 = rcp_approx(x);
    const float rx = __fmaf_rn(y0, __fmaf_rn(-x, y0, 1.0f), y0);
    const float lg = lg2_approx(x);
    return pow73_value(o, x, rx, lg, ex2_approx(__fmul_rn(lg, kThird)));
}

struct ExactMath {
    static constexpr bool kExact = true;
    __device__ static __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    __device__ static __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    __device__ static __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    __device__ static __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
    __device__ static __forceinline__ float sqrt(float a) { return __fsqrt_rn(a); }
    // Reciprocal of the HLL denominator; exact mode divides each component instead.
    __device__ static __forceinline__ float recip(float a) { return a; }
    __device__ static __forceinline__ float over(float num, float den_or_recip) {
        return __fdiv_rn(num, den_or_recip);
    }
    // m / max(h, dry) where h > dry, else 0 (shallow_water_2d.py:60-63).
    __device__ static __forceinline__ float vel(float m, float h, float dry) {
        return h > dry ? __fdiv_rn(m, h) : 0.0f;
    }
    // Both velocities of a cell from one depth.
    __device__ static __forceinline__ void vel2(float mx, float my, float h, float dry, float& u,
                                                float& v) {
        const bool wet = h > dry;
        u = wet ? __fdiv_rn(mx, h) : 0.0f;
        v = wet ? __fdiv_rn(my, h) : 0.0f;
    }
    // Velocity recomputed from a reconstructed momentum H*u (shallow_water_2d.py:76-79).
    __device__ static __forceinline__ float recon_vel(float m, float H, float dry, float /*u*/) {
        return H > dry ? __fdiv_rn(m, H) : 0.0f;
    }
    __device__ static __forceinline__ float hypot(float a, float b) {
        const double da = (double)a, db = (double)b;
        return __double2float_rn(__dsqrt_rn(__dadd_rn(__dmul_rn(da, da), __dmul_rn(db, db))));
    }
    // max(h, dry) ** (7/3) with the exponent rounded to float as NumPy does.
    __device__ static __forceinline__ float pow73(float x, float expo) { return pow73_exact(x, expo); }
};

// ExactMath with the IEEE operations throughout: the paired march of domains whose
// controls lie outside the range of the branch-free form (swe_exact.cuh).
struct IeeeMath : ExactMath {};

struct FastMath {
    static constexpr bool kExact = false;
    __device__ static __forceinline__ float add(float a, float b) { return a + b; }
    __device__ static __forceinline__ float sub(float a, float b) { return a - b; }
    __device__ static __forceinline__ float mul(float a, float b) { return a * b; }
    __device__ static __forceinline__ float rcp(float a) {
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
        return r;
    }
    __device__ static __forceinline__ float div(float a, float b) { return a * rcp(b); }
    __device__ static __forceinline__ float sqrt(float a) {
        float r;
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
        return r;
    }
    __device__ static __forceinline__ float recip(float a) { return rcp(a); }
    __device__ static __forceinline__ float over(float num, float recip_den) { return num * recip_den; }
    __device__ static __forceinline__ float vel(float m, float h, float dry) {
        return h > dry ? m * rcp(h) : 0.0f;
    }
    __device__ static __forceinline__ void vel2(float mx, float my, float h, float dry, float& u,
                                                float& v) {
        const float r = h > dry ? rcp(h) : 0.0f;
        u = mx * r;
        v = my * r;
    }
    __device__ static __forceinline__ float recon_vel(float /*m*/, float H, float dry, float u) {
        return H > dry ? u : 0.0f;
    }
    __device__ static __forceinline__ float hypot(float a, float b) { return sqrt(a * a + b * b); }
    __device__ static __forceinline__ float pow73(float x, float expo) {
        float l, r;
        asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(x));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(l * expo));
        return r;
    }
};

}  // namespace swe

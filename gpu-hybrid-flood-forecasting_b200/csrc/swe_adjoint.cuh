// Hand-written reverse mode (adjoint) of the shallow-water step (sm_100a).
//
// The reference has no adjoint: it never differentiates its solver (the only
// gradients in it are of the U-Net, src/hybrid_flood/ml/train.py:181).  This is
// the vector-Jacobian product of one step of
// src/hybrid_flood/numpy_solver/shallow_water_2d.py:277-327 with dt held fixed
// (a stop-gradient, as jax.grad of a fixed-dt scan would treat it):
//
//   given lambda' = dL/dU_{k+1}, returns lambda = dL/dU_k and accumulates
//   dL/d(n^2) per cell and dL/d(rain scale).
//
// Non-smooth points use these conventions (zero where the forward is flat or
// undefined): max(x, 0) passes the gradient only for x > 0; velocities m/h
// only for h > dry; sqrt(g H) only for H > 0; the friction term's max(h, dry)
// only for h > dry; hypot only for a non-zero norm; HLL speed min/max route to
// the selected argument; the flux select follows the taken branch.
//
// One kernel per reverse step: adj_march_kernel where U_{k+1} is known (a rollout's
// reverse), adj_march_faces_kernel where it is not (a single step); or two, where
// lam_out aliases lam:
//   adj_cell_kernel  recomputes the cell's forward update (its four faces) and
//                    reverses the pointwise part (rain, clip, friction, masks):
//                    lambda_upd = dL/d(upd) per cell, plus the n^2 and rain
//                    scale gradients;
//   adj_face_tile_kernel  evaluates each face's flux VJP once per tile (each
//                    face's flux depends on the states of its two cells through
//                    reconstruction and HLL) and gathers, for each cell, its four
//                    faces' contributions into lambda = lambda_upd + their sum.
#pragma once

#include "swe_pair.cuh"
#include "swe_step.cuh"

namespace swe {

// Plain arithmetic on one value and on a pair of cells (packed f32x2; the
// compiler fuses multiply-adds of both).  The reverse needs no rounding order.
struct V2 {
    float2 v;
};
__device__ __forceinline__ V2 operator+(V2 a, V2 b) { return {__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ V2 operator-(V2 a) { return {{-a.v.x, -a.v.y}}; }
__device__ __forceinline__ V2 operator-(V2 a, V2 b) { return a + (-b); }
__device__ __forceinline__ V2 operator*(V2 a, V2 b) { return {__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ V2 operator*(float a, V2 b) { return V2{splat(a)} * b; }
__device__ __forceinline__ V2 sel(B2 p, V2 a, V2 b) { return {sel(p, a.v, b.v)}; }
__device__ __forceinline__ B2 gt(V2 a, float b) { return {a.v.x > b, a.v.y > b}; }
__device__ __forceinline__ B2 ge(V2 a, V2 b) { return {a.v.x >= b.v.x, a.v.y >= b.v.y}; }
__device__ __forceinline__ V2 vmax(V2 a, V2 b) { return {vmax(a.v, b.v)}; }
__device__ __forceinline__ V2 vmin(V2 a, V2 b) { return {vmin(a.v, b.v)}; }
__device__ __forceinline__ V2 vabs(V2 a) { return {vabs(a.v)}; }
template <class T>
__device__ __forceinline__ T lit(float a);
template <>
__device__ __forceinline__ float lit<float>(float a) { return a; }
template <>
__device__ __forceinline__ V2 lit<V2>(float a) { return {splat(a)}; }
// A flag per cell of T.
template <class T>
struct FlagOf {
    using type = bool;
};
template <>
struct FlagOf<V2> {
    using type = B2;
};
template <class T>
using Flag = typename FlagOf<T>::type;

struct AdjConsts {
    float g, half_g, dry, dx, dy;
};

// The reverse step needs derivative values to float accuracy, not the forward's
// rounding: approximate division, square root and power (a few ulp) keep it cheap.
// A reciprocal is formed once per divisor and multiplied.
__device__ __forceinline__ float arcp(float a) { return rcp_approx(a); }
__device__ __forceinline__ V2 arcp(V2 a) { return {{rcp_approx(a.v.x), rcp_approx(a.v.y)}}; }
__device__ __forceinline__ float asqrt(float a) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ V2 asqrt(V2 a) { return {{asqrt(a.v.x), asqrt(a.v.y)}}; }
__device__ __forceinline__ float apow(float x, float e) {  // x > 0
    float l, r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(l * e));
    return r;
}
__device__ __forceinline__ V2 apow(V2 x, float e) { return {{apow(x.v.x, e), apow(x.v.y, e)}}; }

// One side of a face: the cell's depth and bed, its velocities (m/h where h >
// dry, else 0) and 1/h, computed once per cell and shared by its four faces, and
// whether it is active.
template <class T>
struct FaceInT {
    T h, z, u, v, rh;
    Flag<T> act;
};
using FaceIn = FaceInT<float>;

__device__ __forceinline__ FaceIn face_in(float h, float hu, float hv, float z, bool act, float dry) {
    const bool wet = h > dry;
    const float rh = arcp(h);
    return {h, z, wet ? hu * rh : 0.f, wet ? hv * rh : 0.f, rh, act};
}

__device__ __forceinline__ FaceIn face_in(const Cell& c, float dry) {
    return face_in(c.h, c.hu, c.hv, c.z, active(c.nm), dry);
}

// The mirrored copy of a cell across a wall: the normal velocity changes sign.
template <int AXIS>
__device__ __forceinline__ FaceIn mirror(FaceIn c) {
    if (AXIS == 1) c.u = -c.u;
    else c.v = -c.v;
    return c;
}

// Forward flux of one face (plain float32 arithmetic; the adjoint needs the
// values, not the reference's bit pattern).
template <int AXIS>
__device__ void adj_face_fwd(FaceIn lo, FaceIn hi, const AdjConsts& k, float F[3], float& clo, float& chi) {
    F[0] = F[1] = F[2] = 0.f;
    clo = chi = 0.f;
    if (!(lo.act || hi.act)) return;
    FaceIn L = lo, R = hi;
    if (lo.act && !hi.act) {
        R = mirror<AXIS>(lo);
    } else if (!lo.act && hi.act) {
        L = mirror<AXIS>(hi);
    }
    const float zf = fmaxf(L.z, R.z);
    const float HL = fmaxf(L.h + L.z - zf, 0.f), HR = fmaxf(R.h + R.z - zf, 0.f);
    const float uL = L.u, vL = L.v, uR = R.u, vR = R.v;
    const float XL = HL * uL, YL = HL * vL, XR = HR * uR, YR = HR * vR;
    const float nL = AXIS == 1 ? XL : YL, nR = AXIS == 1 ? XR : YR;
    const float rHL = arcp(HL), rHR = arcp(HR);
    const float unL = HL > k.dry ? nL * rHL : 0.f, unR = HR > k.dry ? nR * rHR : 0.f;
    const float tL = HL > k.dry ? YL * rHL : 0.f, tR = HR > k.dry ? YR * rHR : 0.f;
    const float cL = asqrt(k.g * HL), cR = asqrt(k.g * HR);
    const float sL = fminf(unL - cL, unR - cR), sR = fmaxf(unL + cL, unR + cR);
    const float pL = k.half_g * HL * HL, pR = k.half_g * HR * HR;
    float fL[3], fR[3];
    if (AXIS == 1) {
        fL[0] = XL; fL[1] = XL * unL + pL; fL[2] = XL * tL;
        fR[0] = XR; fR[1] = XR * unR + pR; fR[2] = XR * tR;
    } else {
        fL[0] = YL; fL[1] = XL * unL; fL[2] = YL * unL + pL;
        fR[0] = YR; fR[1] = XR * unR; fR[2] = YR * unR + pR;
    }
    const float UL[3] = {HL, XL, YL}, UR[3] = {HR, XR, YR};
    const float spread = sR - sL;
    const float rden = arcp(spread > kHllEps ? spread : 1.f);
    for (int q = 0; q < 3; ++q) {
        const float m = (sR * fL[q] - sL * fR[q] + sL * sR * (UR[q] - UL[q])) * rden;
        F[q] = sL >= 0.f ? fL[q] : (sR <= 0.f ? fR[q] : m);
    }
    clo = k.half_g * (L.h * L.h - HL * HL);
    chi = k.half_g * (R.h * R.h - HR * HR);
}

// One side of a face in the reverse: given the weights of its flux (a0 mass, an
// normal, at tangential momentum), of its reconstructed state (uH, uN, uT), of its
// normal velocity and celerity in the wave speeds (lun, lc) and of its pressure
// correction, dL/d(h, normal momentum, tangential momentum) of the cell.
//
// With N = H n and T = H t the momenta of the reconstructed depth H, the flux is
// (N, N un + g H^2/2, N tt), where un and tt are the cell's velocities n and t
// where H > dry and zero elsewhere (the forward recomputes them as N/H and T/H).
// Reversed through (H, n, t) no term is divided by H.
template <class T>
struct AdjSide {
    T h, n, t, rh;     // the cell: depth, normal and tangential velocity, 1/h
    T H, un, tt, N, c; // reconstructed depth, velocities in the flux, N, celerity
    Flag<T> up, wet, deep;  // H > 0, H > dry, h > dry
};

template <class T>
__device__ __forceinline__ void adj_side(const AdjConsts& k, const AdjSide<T>& s, T a0, T an, T at, T uH, T uN, T uT,
                                         T lun, T lc, T lcorr, T out[3]) {
    const T zero = lit<T>(0.f);
    const T lN = a0 + s.un * an + s.tt * at + uN;
    const T ln = s.H * lN + sel(s.wet, s.N * an + lun, zero);
    const T lt = s.H * uT + sel(s.wet, s.N * at, zero);
    const T lH = uH + s.n * lN + s.t * uT + k.g * (s.H * (an - lcorr)) +
                 sel(gt(s.c, 0.f), 0.5f * k.g * (arcp(s.c) * lc), zero);
    const T lh = k.g * (s.h * lcorr) + sel(s.up, lH, zero);  // the bed is held fixed
    out[1] = sel(s.deep, ln * s.rh, zero);
    out[2] = sel(s.deep, lt * s.rh, zero);
    out[0] = lh - (s.n * out[1] + s.t * out[2]);
}

// VJP of one face (or of a pair of faces): given dL/dF (3), dL/dcorr_lo, dL/dcorr_hi,
// return dL/d(h, hu, hv) of the lo cell and of the hi cell (after undoing the
// wall mirroring).  No branch: a supercritical face's weights are those of the
// flux it takes, selected per cell.
template <int AXIS, bool MASKED, class T>
__device__ __forceinline__ void adj_face_vjp(const FaceInT<T>& lo, const FaceInT<T>& hi, const AdjConsts& k,
                                             const T lF[3], T lclo, T lchi, T dlo[3], T dhi[3]) {
    constexpr int in = AXIS == 1 ? 1 : 2, it = 3 - in;  // normal and tangential momentum component
    const T zero = lit<T>(0.f), one = lit<T>(1.f);
    const Flag<T> hi_wall = lo.act & !hi.act, lo_wall = !lo.act & hi.act, relevant = lo.act | hi.act;
    auto side = [&](const FaceInT<T>& f, const FaceInT<T>& across, const Flag<T>& wall, T zf) {
        AdjSide<T> s;
        s.h = f.h;
        s.n = AXIS == 1 ? f.u : f.v;
        s.t = AXIS == 1 ? f.v : f.u;
        s.rh = f.rh;
        T z = f.z;
        if constexpr (MASKED) {  // the mirrored copy of the cell across a wall
            s.h = sel(wall, across.h, s.h);
            s.n = sel(wall, -(AXIS == 1 ? across.u : across.v), s.n);
            s.t = sel(wall, AXIS == 1 ? across.v : across.u, s.t);
            s.rh = sel(wall, across.rh, s.rh);
            z = sel(wall, across.z, z);
        }
        const T a = s.h + z - zf;
        s.H = vmax(a, zero);
        s.up = gt(a, 0.f);
        s.wet = gt(s.H, k.dry);
        s.deep = gt(s.h, k.dry);
        s.un = sel(s.wet, s.n, zero);
        s.tt = sel(s.wet, s.t, zero);
        s.N = s.H * s.n;
        s.c = asqrt(k.g * s.H);
        return s;
    };
    T zf = vmax(lo.z, hi.z);
    if constexpr (MASKED) zf = vmax(sel(lo_wall, hi.z, lo.z), sel(hi_wall, lo.z, hi.z));
    const AdjSide<T> L = side(lo, hi, lo_wall, zf), R = side(hi, lo, hi_wall, zf);
    const T aminL = L.un - L.c, aminR = R.un - R.c, amaxL = L.un + L.c, amaxR = R.un + R.c;
    const T sL = vmin(aminL, aminR), sR = vmax(amaxL, amaxR);
    const T spread = sR - sL;
    const Flag<T> use_spread = gt(spread, kHllEps);
    const T rden = arcp(sel(use_spread, spread, one));
    const T s01 = sL * sR;
    const Flag<T> take_l = ge(sL, zero), take_r = !take_l & ge(zero, sR), middle = !(take_l | take_r);
    // Weights of the two sides' fluxes and of the state jump in the face's flux.
    const T wl = sel(middle, sR * rden, sel(take_l, one, zero));
    const T wr = sel(middle, -(sL * rden), sel(take_l, zero, sel(take_r, one, zero)));
    const T wu = sel(middle, s01 * rden, zero);
    const T f[3] = {lF[0], lF[in], lF[it]};
    const T fL[3] = {L.N, L.N * L.un + k.half_g * (L.H * L.H), L.N * L.tt};
    const T fR[3] = {R.N, R.N * R.un + k.half_g * (R.H * R.H), R.N * R.tt};
    const T dU[3] = {R.H - L.H, R.N - L.N, R.H * R.t - L.H * L.t};
    T lsL = zero, lsR = zero, lden = zero;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        lden = lden + (wl * fL[q] + wr * fR[q] + wu * dU[q]) * f[q];
        lsR = lsR + (fL[q] + sL * dU[q]) * f[q];
        lsL = lsL + (sR * dU[q] - fR[q]) * f[q];
    }
    lden = sel(use_spread, lden, zero);
    const T live = sel(middle, rden, zero);
    lsR = (lsR - lden) * live;
    lsL = (lsL + lden) * live;
    // Wave speeds: min/max route to the selected argument.
    const Flag<T> minL = ge(aminR, aminL), maxL = ge(amaxL, amaxR);
    const T lsLL = sel(minL, lsL, zero), lsLR = sel(minL, zero, lsL);
    const T lsRL = sel(maxL, lsR, zero), lsRR = sel(maxL, zero, lsR);
    T gL[3], gR[3];
    adj_side(k, L, wl * f[0], wl * f[1], wl * f[2], -(wu * f[0]), -(wu * f[1]), -(wu * f[2]), lsLL + lsRL, lsRL - lsLL,
             lclo, gL);
    adj_side(k, R, wr * f[0], wr * f[1], wr * f[2], wu * f[0], wu * f[1], wu * f[2], lsLR + lsRR, lsRR - lsLR, lchi, gR);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const int comp = q == 0 ? 0 : (q == 1 ? in : it);
        if constexpr (MASKED) {
            // The mirrored side's gradient belongs to the active cell.
            const T mR = q == 1 ? -gR[q] : gR[q], mL = q == 1 ? -gL[q] : gL[q];
            dlo[comp] = sel(relevant, sel(lo_wall, zero, gL[q] + sel(hi_wall, mR, zero)), zero);
            dhi[comp] = sel(relevant, sel(hi_wall, zero, gR[q] + sel(lo_wall, mL, zero)), zero);
        } else {
            dlo[comp] = gL[q];
            dhi[comp] = gR[q];
        }
    }
}

// What the reverse of a cell knows of its update before the pointwise part: nothing (it is
// rebuilt from the cell's four faces), the step's own output U_{k+1}, or the update
// without the rain.
enum class AdjSource { kNothing, kNext, kUpdate };

// Forward flux of a face (or a pair of faces), mass, normal and tangential momentum, and
// the pressure corrections of its two sides: adj_face_fwd without branches.
template <class T>
struct AdjFlux {
    T m, n, t, lo, hi;
};

template <int AXIS, bool MASKED, class T>
__device__ __forceinline__ AdjFlux<T> adj_flux(const FaceInT<T>& lo, const FaceInT<T>& hi, const AdjConsts& k) {
    const T zero = lit<T>(0.f), one = lit<T>(1.f);
    const Flag<T> hi_wall = lo.act & !hi.act, lo_wall = !lo.act & hi.act;
    auto side = [&](const FaceInT<T>& f, const FaceInT<T>& across, const Flag<T>& wall) {
        FaceInT<T> s = f;
        if (AXIS == 0) {
            s.u = f.v;
            s.v = f.u;
        }
        if constexpr (MASKED) {  // the mirrored copy of the cell across a wall
            s.h = sel(wall, across.h, s.h);
            s.z = sel(wall, across.z, s.z);
            s.u = sel(wall, -(AXIS == 1 ? across.u : across.v), s.u);
            s.v = sel(wall, AXIS == 1 ? across.v : across.u, s.v);
        }
        return s;
    };
    const FaceInT<T> L = side(lo, hi, lo_wall), R = side(hi, lo, hi_wall);  // u: normal, v: tangential
    const T zf = vmax(L.z, R.z);
    const T HL = vmax(L.h + L.z - zf, zero), HR = vmax(R.h + R.z - zf, zero);
    const Flag<T> wL = gt(HL, k.dry), wR = gt(HR, k.dry);
    const T nL = sel(wL, L.u, zero), nR = sel(wR, R.u, zero), tL = sel(wL, L.v, zero), tR = sel(wR, R.v, zero);
    const T cL = asqrt(k.g * HL), cR = asqrt(k.g * HR);
    const T sL = vmin(nL - cL, nR - cR), sR = vmax(nL + cL, nR + cR);
    const T spread = sR - sL;
    const T rden = arcp(sel(gt(spread, kHllEps), spread, one)), s01 = sL * sR;
    const Flag<T> take_l = ge(sL, zero), take_r = ge(zero, sR);
    const T NL = HL * L.u, NR = HR * R.u;
    auto hll = [&](T fl, T fr, T jump) {
        return sel(take_l, fl, sel(take_r, fr, (sR * fl - sL * fr + s01 * jump) * rden));
    };
    AdjFlux<T> f;
    f.m = hll(NL, NR, HR - HL);
    f.n = hll(NL * nL + k.half_g * (HL * HL), NR * nR + k.half_g * (HR * HR), NR - NL);
    f.t = hll(NL * tL, NR * tR, HR * R.v - HL * L.v);
    f.lo = k.half_g * (L.h * L.h - HL * HL);
    f.hi = k.half_g * (R.h * R.h - HR * HR);
    if constexpr (MASKED) {
        const Flag<T> relevant = lo.act | hi.act;
        f = {sel(relevant, f.m, zero), sel(relevant, f.n, zero), sel(relevant, f.t, zero), sel(relevant, f.lo, zero),
             sel(relevant, f.hi, zero)};
    }
    return f;
}

struct AdjLaunch {
    DomainDev d;
    StateView in;        // U_k
    StateView next;      // U_{k+1} when known (h == nullptr otherwise)
    StateView lam;       // dL/dU_{k+1}
    StateOut lam_out;    // dL/dU_k
    float* lupd[3];      // scratch: dL/d(upd) planes, pitch lpitch
    int64_t lpitch;
    float* grad_n2;      // rows x cols, accumulated
    double* grad_rain;   // device scalar, accumulated
    StepScalars s;       // float32 dt, dt*rate (scaled), dt*g
    float dt_rate;       // float32 dt * rate(t) before the rain scale
    AdjConsts k;
    float rdx, rdy;      // 1/dx, 1/dy
};

__device__ __forceinline__ Cell adj_load(const DomainDev& d, const StateView& s, int r, int c) {
    Cell t[1];
    load_cells<1>(d, s, r, c, t);
    return t[0];
}

// The forward update of cell (r, c) from its four faces: upd (3) before the
// pointwise part.
struct AdjUpd {
    float u0, u1, u2;
};
__device__ __noinline__ inline AdjUpd adj_cell_update(const AdjLaunch& p, int r, int c) {
    const DomainDev& d = p.d;
    const float dry = p.k.dry;
    const FaceIn C = face_in(adj_load(d, p.in, r, c), dry);
    const FaceIn W = face_in(adj_load(d, p.in, r, c - 1), dry), E = face_in(adj_load(d, p.in, r, c + 1), dry);
    const FaceIn S = face_in(adj_load(d, p.in, r - 1, c), dry), N = face_in(adj_load(d, p.in, r + 1, c), dry);
    float Fl[3], Fr[3], Fb[3], Ft[3], cl_lo, cl_hi, cr_lo, cr_hi, cb_lo, cb_hi, ct_lo, ct_hi;
    adj_face_fwd<1>(W, C, p.k, Fl, cl_lo, cl_hi);
    adj_face_fwd<1>(C, E, p.k, Fr, cr_lo, cr_hi);
    adj_face_fwd<0>(S, C, p.k, Fb, cb_lo, cb_hi);
    adj_face_fwd<0>(C, N, p.k, Ft, ct_lo, ct_hi);
    const Cell own = adj_load(d, p.in, r, c);
    const float U[3] = {own.h, own.hu, own.hv};
    float upd[3];
    for (int q = 0; q < 3; ++q) {
        const float xl = Fr[q] + (q == 1 ? cr_lo : 0.f);
        const float xr = Fl[q] + (q == 1 ? cl_hi : 0.f);
        const float yb = Ft[q] + (q == 2 ? ct_lo : 0.f);
        const float yt = Fb[q] + (q == 2 ? cb_hi : 0.f);
        upd[q] = U[q] - p.s.dt * ((xl - xr) * p.rdx + (yb - yt) * p.rdy);
    }
    return {upd[0], upd[1], upd[2]};
}

// Reverse of the pointwise part of an active cell (rain, clip, friction, masks):
// lu = dL/d(upd); when `owned`, also adds the cell's dL/d(n^2) to grad_n2 and its
// rain-scale term to *rain_acc.
//
// With kNext the cell update before the pointwise part is rebuilt from the step's
// own output U_{k+1} = (h1, q1, q2) instead of from the cell's four faces.  The
// momenta invert the semi-implicit friction: with a = dt g n^2 max(h,dry)^(-7/3),
// q = upd/(1 + a|upd|) gives upd = q/(1 - a|q|).  Where that inversion loses
// precision (a|q| > 0.999, i.e. friction dividing the momentum by more than 1000)
// the update is rebuilt from the faces.  For dry or clipped cells only the depth
// part is needed: the momentum outputs are zero and carry no gradient.
template <AdjSource SRC, bool MASKED>
__device__ __forceinline__ void adj_pointwise(const AdjLaunch& p, int r, int c, V2 nm, const V2 lam[3], const V2 known[3],
                                              B2 live, B2 owned, double* rain_acc, V2 lu[3]) {
    const DomainDev& d = p.d;
    const V2 zero = lit<V2>(0.f), n2 = MASKED ? vabs(nm) : nm;
    V2 mult = lit<V2>(1.f);
    if (d.mult) {
        if (live.x) mult.v.x = d.mult[(int64_t)r * d.spitch + c];
        if (live.y) mult.v.y = d.mult[(int64_t)r * d.spitch + c + 1];
    }
    V2 u0 = zero, u1 = zero, u2 = zero;  // u0: the depth after the rain (before the clip)
    B2 rebuild = live;
    if constexpr (SRC == AdjSource::kUpdate) {
        u0 = known[0] + p.s.dt_rain * mult;
        u1 = known[1];
        u2 = known[2];
    }
    if constexpr (SRC == AdjSource::kNext) {
        u0 = known[0];
        const B2 wet = gt(u0, p.k.dry);
        const V2 pw = apow(vmax(u0, lit<V2>(p.k.dry)), -7.0f / 3.0f);
        const V2 aq = p.s.dt_g * n2 * pw * asqrt(known[1] * known[1] + known[2] * known[2]);
        const V2 den = arcp(lit<V2>(1.f) - aq);
        u1 = sel(wet, known[1] * den, zero);
        u2 = sel(wet, known[2] * den, zero);
        rebuild = live & wet & B2{!(aq.v.x <= 0.999f), !(aq.v.y <= 0.999f)};
    }
    if constexpr (SRC != AdjSource::kUpdate) {
        if (rebuild.x) {
            const AdjUpd t = adj_cell_update(p, r, c);
            u0.v.x = t.u0 + p.s.dt_rain * mult.v.x;
            u1.v.x = t.u1;
            u2.v.x = t.u2;
        }
        if (rebuild.y) {
            const AdjUpd t = adj_cell_update(p, r, c + 1);
            u0.v.y = t.u0 + p.s.dt_rain * mult.v.y;
            u1.v.y = t.u1;
            u2.v.y = t.u2;
        }
    }
    const V2 h = vmax(u0, zero);
    const V2 pw = apow(vmax(h, lit<V2>(p.k.dry)), -7.0f / 3.0f);
    const V2 norm = asqrt(u1 * u1 + u2 * u2);
    const V2 a = p.s.dt_g * n2 * pw;
    const V2 fr = a * norm;
    const V2 rden = arcp(lit<V2>(1.f) + fr);
    const V2 qx = u1 * rden, qy = u2 * rden;
    const B2 wet = gt(h, p.k.dry);
    const V2 lqx = sel(wet, lam[1], zero), lqy = sel(wet, lam[2], zero);
    const V2 lden = -((lqx * qx + lqy * qy) * rden);
    const V2 ln = sel(gt(norm, 0.f), lden * a * arcp(norm), zero);
    const V2 lh = lam[0] + sel(wet, (-7.0f / 3.0f) * (lden * fr * arcp(h)), zero);
    lu[0] = sel(live & gt(u0, 0.f), lh, zero);
    lu[1] = sel(live, lqx * rden + ln * u1, zero);
    lu[2] = sel(live, lqy * rden + ln * u2, zero);
    const B2 add = owned & live;
    const V2 gn = p.s.dt_g * (lden * norm * pw);
    float* g = p.grad_n2 + (int64_t)r * d.cols + c;
    if (add.x) {
        g[0] += gn.v.x;
        *rain_acc += (double)lu[0].v.x * (double)p.dt_rate * (double)mult.v.x;
    }
    if (add.y) {
        g[1] += gn.v.y;
        *rain_acc += (double)lu[0].v.y * (double)p.dt_rate * (double)mult.v.y;
    }
}

// Adds a CTA's rain-scale gradient to the device scalar (one atomic per CTA).
template <int THREADS>
__device__ __forceinline__ void adj_flush_rain(const AdjLaunch& p, double rain_acc) {
    rain_acc = warp_sum(rain_acc);
    __shared__ double s_r[THREADS / kWarp];
    if ((threadIdx.x & 31) == 0) s_r[threadIdx.x >> 5] = rain_acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < THREADS / kWarp; ++w) t += s_r[w];
        if (t != 0.0) atomicAdd(p.grad_rain, t);
    }
}

template <int THREADS, bool NEXT>
__global__ void __launch_bounds__(THREADS) adj_cell_kernel(const __grid_constant__ AdjLaunch p) {
    const DomainDev& d = p.d;
    const int64_t n = (int64_t)d.rows * d.cols;
    double rain_acc = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * THREADS) {
        const int r = (int)(i / d.cols), c = (int)(i - (int64_t)r * d.cols);
        const int64_t li = (int64_t)r * p.lam.pitch + c, no = (int64_t)r * p.next.pitch + c;
        auto one = [](float x) { return V2{{x, x}}; };
        const float nm = d.nm[(int64_t)r * d.spitch + c];
        const V2 lam[3] = {one(p.lam.h[li]), one(p.lam.hu[li]), one(p.lam.hv[li])};
        V2 next[3] = {}, lu[3];
        if constexpr (NEXT) {
            next[0] = one(p.next.h[no]);
            next[1] = one(p.next.hu[no]);
            next[2] = one(p.next.hv[no]);
        }
        adj_pointwise<NEXT ? AdjSource::kNext : AdjSource::kNothing, true>(p, r, c, one(nm), lam, next, B2{active(nm), false}, B2{true, false}, &rain_acc, lu);
        const int64_t lo = (int64_t)r * p.lpitch + c;
        p.lupd[0][lo] = lu[0].v.x;
        p.lupd[1][lo] = lu[1].v.x;
        p.lupd[2][lo] = lu[2].v.x;
    }
    adj_flush_rain<THREADS>(p, rain_acc);
}

// dL/d(upd) of cell (r, c); zero outside the grid (ghost cells are not updated).
__device__ __forceinline__ void lupd_at(const AdjLaunch& p, int r, int c, float l[3]) {
    if (r < 0 || r >= p.d.rows || c < 0 || c >= p.d.cols) {
        l[0] = l[1] = l[2] = 0.f;
        return;
    }
    const int64_t o = (int64_t)r * p.lpitch + c;
    l[0] = p.lupd[0][o];
    l[1] = p.lupd[1][o];
    l[2] = p.lupd[2][o];
}

// VJP of the face between the lo cell (rl, cl) and the hi cell (rh, ch) (ghost
// cells allowed: they carry no dL/d(upd)), given a = dt/dx or dt/dy; the
// normal-momentum component is hu for x-faces and hv for y-faces.
template <int AXIS>
__device__ __forceinline__ void adj_face_at(const AdjLaunch& p, int rl, int cl, int rh, int ch, float a,
                                            float* dlo, float* dhi) {
    const FaceIn L = face_in(adj_load(p.d, p.in, rl, cl), p.k.dry), H = face_in(adj_load(p.d, p.in, rh, ch), p.k.dry);
    float ll[3], lh[3], lF[3];
    lupd_at(p, rl, cl, ll);
    lupd_at(p, rh, ch, lh);
#pragma unroll
    for (int q = 0; q < 3; ++q) lF[q] = -a * ll[q] + a * lh[q];
    constexpr int nq = AXIS == 1 ? 1 : 2;
    float lo[3], hi[3];
    adj_face_vjp<AXIS, true, float>(L, H, p.k, lF, -a * ll[nq], a * lh[nq], lo, hi);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        dlo[q] = lo[q];
        dhi[q] = hi[q];
    }
}

// The face gather with every face evaluated once.  A CTA of 256 threads takes
// a tile of 32 x 8 cells: each thread evaluates the x-face left of its cell and
// the y-face below it (round 1), warp 0 the y-faces above the tile's top row
// and 8 lanes of warp 1 the x-faces right of its last column (round 2), all
// into shared memory; then each cell adds the four faces' VJPs for its side
// (round 3).  Tile-edge faces are evaluated by both neighbouring tiles, about
// 2.25 face VJPs per cell instead of the 4 of a per-cell gather.
constexpr int kAdjTW = 32, kAdjTH = 8;

__global__ void __launch_bounds__(kAdjTW * kAdjTH) adj_face_tile_kernel(const AdjLaunch p) {
    __shared__ float s_x[kAdjTH][kAdjTW + 1][6];  // face left of tile column c: dlo (0..2), dhi (3..5)
    __shared__ float s_y[kAdjTH + 1][kAdjTW][6];  // face below tile row r
    const DomainDev& d = p.d;
    const int tiles_x = (d.cols + kAdjTW - 1) / kAdjTW, tiles_y = (d.rows + kAdjTH - 1) / kAdjTH;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const float ax = p.s.dt * p.rdx, ay = p.s.dt * p.rdy;
    for (int tile = blockIdx.x; tile < tiles_x * tiles_y; tile += gridDim.x) {
        const int c0 = (tile % tiles_x) * kAdjTW, r0 = (tile / tiles_x) * kAdjTH;
        const int r = r0 + ty, c = c0 + tx;
        // x-faces exist for rows [0, rows) and columns [0, cols] (left of column c);
        // y-faces for columns [0, cols) and rows [0, rows] (below row r).
        if (r < d.rows && c <= d.cols) adj_face_at<1>(p, r, c - 1, r, c, ax, &s_x[ty][tx][0], &s_x[ty][tx][3]);
        if (c < d.cols && r <= d.rows) adj_face_at<0>(p, r - 1, c, r, c, ay, &s_y[ty][tx][0], &s_y[ty][tx][3]);
        if (ty == 0) {
            const int rt = r0 + kAdjTH;
            if (c < d.cols && rt <= d.rows) adj_face_at<0>(p, rt - 1, c, rt, c, ay, &s_y[kAdjTH][tx][0], &s_y[kAdjTH][tx][3]);
        } else if (ty == 1 && tx < kAdjTH) {
            const int rr = r0 + tx, cr = c0 + kAdjTW;
            if (rr < d.rows && cr <= d.cols) adj_face_at<1>(p, rr, cr - 1, rr, cr, ax, &s_x[tx][kAdjTW][0], &s_x[tx][kAdjTW][3]);
        }
        __syncthreads();
        if (r < d.rows && c < d.cols) {
            float g[3];
            lupd_at(p, r, c, g);  // upd_q = U_q - ... : direct term
            const float* fl = s_x[ty][tx];       // left face: this cell is its hi side
            const float* fr = s_x[ty][tx + 1];   // right face: lo side
            const float* fb = s_y[ty][tx];       // bottom face: hi side
            const float* ft = s_y[ty + 1][tx];   // top face: lo side
#pragma unroll
            for (int q = 0; q < 3; ++q) g[q] += fl[3 + q] + fr[q] + fb[3 + q] + ft[q];
            // Ghost cells are mirrored copies of their boundary cell: their side of a
            // boundary face belongs to that cell (normal momentum sign-flipped on reflective edges).
            if (c == 0) {
                const float s = d.bnd[0] == 0 ? -1.f : 1.f;
                g[0] += fl[0]; g[1] += s * fl[1]; g[2] += fl[2];
            }
            if (c == d.cols - 1) {
                const float s = d.bnd[1] == 0 ? -1.f : 1.f;
                g[0] += fr[3]; g[1] += s * fr[4]; g[2] += fr[5];
            }
            if (r == 0) {
                const float s = d.bnd[2] == 0 ? -1.f : 1.f;
                g[0] += fb[0]; g[1] += fb[1]; g[2] += s * fb[2];
            }
            if (r == d.rows - 1) {
                const float s = d.bnd[3] == 0 ? -1.f : 1.f;
                g[0] += ft[3]; g[1] += ft[4]; g[2] += s * ft[5];
            }
            const int64_t o = (int64_t)r * p.lam_out.pitch + c;
            p.lam_out.h[o] = g[0];
            p.lam_out.hu[o] = g[1];
            p.lam_out.hv[o] = g[2];
        }
        __syncthreads();  // the next tile reuses the shared faces
    }
}

// ---------------------------------------------------------------------------
// The whole reverse step in one kernel, for lam_out not aliasing lam
// ---------------------------------------------------------------------------
// A warp owns 60 columns and marches up a chunk of rows, two cells per lane
// evaluated together (packed f32x2); lanes 0 and 31 hold the columns either side,
// so that every face of the strip lies within the warp.  A row's cells are reversed pointwise once
// (dL/d(upd) in registers), its x-faces are evaluated between neighbouring lanes
// and their two sides moved by shuffle, and the y-face above it is evaluated once,
// its upper side carried to the next row.  Only the rows below and above the chunk
// and the two outer columns are reversed twice; lam is read in a neighbour's rows
// while that warp writes lam_out, which is why the two must not alias.
//
// The step is bound by instructions and their latency, not by memory (56 bytes
// a cell): 18 warp instructions a cell, issued at 47 % by the 12 warps of an SM.
// A CTA of 32 x 16 cells staged in shared memory, with a barrier between its three
// phases and the face loop's last round mostly idle, took 9.9 us on 128^2, 17.2 on
// 512^2 and 54 on 1024^2; this march takes 4.4, 11.4 and 33.7 us.
constexpr int kMarchCols = 2 * kWarp - 4;

// What the faces of a pair of cells read of it, and its dL/d(upd).
struct AdjCells {
    FaceInT<V2> f;
    V2 l[3];
};

// The values a row's cells are built from, loaded one row ahead of their use.
struct AdjRaw {
    V2 h, hu, hv, z, nm;
    V2 h1, q1, q2;  // U_{k+1}
    V2 l0, l1, l2;  // dL/dU_{k+1}
};

// Two neighbouring elements of a plane: one 8-byte load where VEC (even column,
// even pitch, 8-byte aligned plane), else two loads at the clamped columns.
// FINISHED: a plane that no kernel writes while this one runs (non-coherent loads;
// see pdl_enter).
template <bool VEC, bool FINISHED>
__device__ __forceinline__ V2 load2(const float* p, uint32_t row, int c0, int c1) {
    auto get = [](const auto* q) {
        if constexpr (FINISHED) return __ldg(q);
        else return state_load(q);
    };
    if constexpr (VEC) return {get(reinterpret_cast<const float2*>(p + row + c0))};
    return {{get(p + row + c0), get(p + row + c1)}};
}

// 32-bit element offsets: planes hold fewer than 2^31 elements (checked on the host).
__device__ __forceinline__ uint32_t adj_row(const DomainDev& d, int r) { return (uint32_t)min(max(r, 0), d.rows - 1); }

template <bool NEXT, bool VEC>
__device__ __forceinline__ void load_states(const AdjLaunch& p, int r, int c0, int c1, AdjRaw& a) {
    const uint32_t rr = adj_row(p.d, r), so = rr * (uint32_t)p.in.pitch, zo = rr * (uint32_t)p.d.spitch;
    a.h = load2<VEC, true>(p.in.h, so, c0, c1);
    a.hu = load2<VEC, true>(p.in.hu, so, c0, c1);
    a.hv = load2<VEC, true>(p.in.hv, so, c0, c1);
    a.z = load2<VEC, true>(p.d.bed, zo, c0, c1);
    a.nm = load2<VEC, true>(p.d.nm, zo, c0, c1);
    if constexpr (NEXT) {
        const uint32_t no = rr * (uint32_t)p.next.pitch;
        a.h1 = load2<VEC, true>(p.next.h, no, c0, c1);
        a.q1 = load2<VEC, true>(p.next.hu, no, c0, c1);
        a.q2 = load2<VEC, true>(p.next.hv, no, c0, c1);
    }
}

// dL/dU_{k+1}: written by the reverse step before, which may still be running when this kernel starts.
template <bool VEC>
__device__ __forceinline__ void load_lam(const AdjLaunch& p, int r, int c0, int c1, AdjRaw& a) {
    const uint32_t lo = adj_row(p.d, r) * (uint32_t)p.lam.pitch;
    a.l0 = load2<VEC, false>(p.lam.h, lo, c0, c1);
    a.l1 = load2<VEC, false>(p.lam.hu, lo, c0, c1);
    a.l2 = load2<VEC, false>(p.lam.hv, lo, c0, c1);
}

template <bool VEC>
__device__ __forceinline__ AdjRaw adj_raw(const AdjLaunch& p, int r, int c0, int c1) {
    AdjRaw a;
    load_states<true, VEC>(p, r, c0, c1, a);
    load_lam<VEC>(p, r, c0, c1, a);
    return a;
}

// The momenta that a cell's faces see: those of the ghost ring are mirrored.
struct AdjMomenta {
    V2 hu, hv;
};

// Cells (r, c) and (r, c + 1) from their loaded values: velocities, no dL/d(upd) yet.
template <bool MASKED, bool VEC>
__device__ __forceinline__ AdjCells adj_velocities(const AdjLaunch& p, AdjRaw& a, int r, int c, AdjMomenta& m) {
    const DomainDev& d = p.d;
    if (VEC && (c < 0 || c >= d.cols)) {
        auto edge = [&](V2& x) { c < 0 ? x.v.y = x.v.x : x.v.x = x.v.y; };
        edge(a.h);
        edge(a.hu);
        edge(a.hv);
        edge(a.z);
        edge(a.nm);
    }
    V2 hu = a.hu, hv = a.hv;
    // Ghost columns and rows (the loads are clamped to the grid): reflective edges mirror the normal momentum.
    if (d.bnd[0] == 0) hu = {{c < 0 ? -hu.v.x : hu.v.x, c + 1 < 0 ? -hu.v.y : hu.v.y}};
    if (d.bnd[1] == 0) hu = {{c >= d.cols ? -hu.v.x : hu.v.x, c + 1 >= d.cols ? -hu.v.y : hu.v.y}};
    if ((r < 0 && d.bnd[2] == 0) || (r >= d.rows && d.bnd[3] == 0)) hv = -hv;
    m = {hu, hv};
    const V2 zero = lit<V2>(0.f);
    AdjCells k;
    k.f.h = a.h;
    k.f.z = a.z;
    k.f.act = MASKED ? act_of(a.nm.v) : B2{true, true};
    k.f.rh = arcp(a.h);
    const B2 deep = gt(a.h, p.k.dry);
    k.f.u = sel(deep, hu * k.f.rh, zero);
    k.f.v = sel(deep, hv * k.f.rh, zero);
    k.l[0] = k.l[1] = k.l[2] = zero;
    return k;
}

// The same with the pointwise reverse (rain, clip, friction, masks) of the cells inside
// the grid (flags `in`) from U_{k+1}; the others carry no dL/d(upd).  Owned cells add
// their n^2 and rain-scale gradients.
template <bool MASKED, bool VEC>
__device__ __forceinline__ AdjCells adj_cells(const AdjLaunch& p, AdjRaw a, int r, int c, B2 in, B2 owned,
                                              double* rain_acc) {
    AdjMomenta m;
    AdjCells k = adj_velocities<MASKED, VEC>(p, a, r, c, m);
    if (r >= 0 && r < p.d.rows) {
        const B2 live = in & k.f.act;
        const V2 lam[3] = {a.l0, a.l1, a.l2}, next[3] = {a.h1, a.q1, a.q2};
        adj_pointwise<AdjSource::kNext, MASKED>(p, r, c, a.nm, lam, next, live, owned, rain_acc, k.l);
    }
    return k;
}

// The cells one column to the right of a lane's: its own second cell and the
// first cell of the next lane.
template <bool MASKED>
__device__ __forceinline__ AdjCells right_of(const AdjCells& a) {
    auto next = [](V2 x) { return V2{{x.v.y, __shfl_down_sync(0xffffffffu, x.v.x, 1)}}; };
    AdjCells b;
    b.f = {next(a.f.h), next(a.f.z), next(a.f.u), next(a.f.v), next(a.f.rh), {true, true}};
    if (MASKED) b.f.act = {a.f.act.y, __shfl_down_sync(0xffffffffu, a.f.act.x ? 1 : 0, 1) != 0};
#pragma unroll
    for (int q = 0; q < 3; ++q) b.l[q] = next(a.l[q]);
    return b;
}

// VJP of the faces between two pairs of cells for their dL/d(upd) (s = dt/dx or dt/dy).
template <int AXIS, bool MASKED>
__device__ __forceinline__ void adj_faces(const AdjConsts& k, const AdjCells& lo, const AdjCells& hi, float s, V2 dlo[3],
                                          V2 dhi[3]) {
    constexpr int nq = AXIS == 1 ? 1 : 2;
    V2 lF[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) lF[q] = s * (hi.l[q] - lo.l[q]);
    adj_face_vjp<AXIS, MASKED, V2>(lo.f, hi.f, k, lF, -(s * lo.l[nq]), s * hi.l[nq], dlo, dhi);
}

// dL/dU_k of row r into lam_out: the faces left, right, below (their upper side, carried in
// `below`) and above of the row's cells.
template <bool MASKED, bool VEC>
__device__ __forceinline__ void adj_gather(const AdjLaunch& p, const AdjCells& cur, const AdjCells& nxt, int r, int c, B2 mine,
                                           float ax, float ay, V2 below[3]) {
    const DomainDev& d = p.d;
    V2 lo[3], hi[3], g[3];
    adj_faces<0, MASKED>(p.k, cur, nxt, ay, lo, hi);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        g[q] = cur.l[q] + below[q] + lo[q];
        below[q] = hi[q];
    }
    if (r == d.rows - 1) {
        g[0] = g[0] + hi[0];
        g[1] = g[1] + hi[1];
        g[2] = g[2] + (d.bnd[3] == 0 ? -hi[2] : hi[2]);
    }
    adj_faces<1, MASKED>(p.k, cur, right_of<MASKED>(cur), ax, lo, hi);
    const float sw = d.bnd[0] == 0 ? -1.f : 1.f, se = d.bnd[1] == 0 ? -1.f : 1.f;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        // hi.x is this lane's second cell's left side, hi.y the next lane's first cell's.
        const float from_left = __shfl_up_sync(0xffffffffu, hi[q].v.y, 1);
        g[q] = g[q] + lo[q] + V2{{from_left, hi[q].v.x}};
        const float west = __shfl_up_sync(0xffffffffu, lo[q].v.y, 1);  // the ghost left of column 0
        if (c == 0) g[q].v.x += (q == 1 ? sw : 1.f) * west;
        if (c == d.cols - 1) g[q].v.x += (q == 1 ? se : 1.f) * hi[q].v.x;
        if (c + 1 == d.cols - 1) g[q].v.y += (q == 1 ? se : 1.f) * hi[q].v.y;
    }
    const uint32_t o = (uint32_t)r * (uint32_t)p.lam_out.pitch + (uint32_t)c;
    if (VEC && mine.y) {
        *reinterpret_cast<float2*>(p.lam_out.h + o) = g[0].v;
        *reinterpret_cast<float2*>(p.lam_out.hu + o) = g[1].v;
        *reinterpret_cast<float2*>(p.lam_out.hv + o) = g[2].v;
    } else {
        if (mine.x) {
            p.lam_out.h[o] = g[0].v.x;
            p.lam_out.hu[o] = g[1].v.x;
            p.lam_out.hv[o] = g[2].v.x;
        }
        if (mine.y) {
            p.lam_out.h[o + 1] = g[0].v.y;
            p.lam_out.hu[o + 1] = g[1].v.y;
            p.lam_out.hv[o + 1] = g[2].v.y;
        }
    }
}

// The upper side of the face between a chunk's first row and the row below it.
template <bool MASKED>
__device__ __forceinline__ void adj_first_face(const AdjLaunch& p, const AdjCells& cur, const AdjCells& nxt, int r0, float ay,
                                               V2 below[3]) {
    V2 blo[3];
    adj_faces<0, MASKED>(p.k, cur, nxt, ay, blo, below);
    // Ghost cells are mirrored copies of their boundary cell: their side of a
    // boundary face belongs to that cell (normal momentum sign-flipped on reflective edges).
    if (r0 == 0) {
        below[0] = below[0] + blo[0];
        below[1] = below[1] + blo[1];
        below[2] = below[2] + (p.d.bnd[2] == 0 ? -blo[2] : blo[2]);
    }
}

template <int THREADS, bool MASKED, bool VEC>
__global__ void __launch_bounds__(THREADS) adj_march_kernel(const __grid_constant__ AdjLaunch p, int nstrips,
                                                            int rows_per_warp) {
    const DomainDev& d = p.d;
    const int lane = threadIdx.x & 31;
    const int gw = blockIdx.x * (THREADS / kWarp) + (threadIdx.x >> 5);
    const int r0 = (gw / nstrips) * rows_per_warp, r1 = min(r0 + rows_per_warp, d.rows);
    const int c = (gw % nstrips) * kMarchCols - 2 + 2 * lane;
    // Columns clamped to the grid.  With VEC (an even number of columns) a pair
    // outside the grid loads the nearest pair and keeps the value of its edge column.
    const int c0 = min(max(c, 0), VEC ? d.cols - 2 : d.cols - 1), c1 = min(max(c + 1, 0), d.cols - 1);
    const B2 in{c >= 0 && c < d.cols, c + 1 >= 0 && c + 1 < d.cols};
    const bool strip = lane >= 1 && lane <= kWarp - 2;
    const B2 mine{strip && in.x, strip && in.y};  // cells this warp writes
    const float ax = p.s.dt * p.rdx, ay = p.s.dt * p.rdy;
    const V2 zero = lit<V2>(0.f);
    double rain_acc = 0.0;
    if (r0 >= d.rows) pdl_enter();
    if (r0 < d.rows) {
        // The states are those of a finished forward pass; only lam (and the gradients)
        // come from the reverse step before, which is waited for once they are loading.
        AdjRaw raw, ahead;
        load_states<true, VEC>(p, r0 - 1, c0, c1, raw);
        load_states<true, VEC>(p, r0, c0, c1, ahead);
        pdl_enter();
        load_lam<VEC>(p, r0 - 1, c0, c1, raw);
        load_lam<VEC>(p, r0, c0, c1, ahead);
        AdjCells cur = adj_cells<MASKED, VEC>(p, raw, r0 - 1, c, in, B2{false, false}, &rain_acc);
        raw = ahead;
        ahead = adj_raw<VEC>(p, r0 + 1, c0, c1);
        AdjCells nxt = adj_cells<MASKED, VEC>(p, raw, r0, c, in, mine, &rain_acc);
        V2 below[3];  // the upper side of the y-face below the row
        adj_first_face<MASKED>(p, cur, nxt, r0, ay, below);
        for (int r = r0; r < r1; ++r) {
            cur = nxt;
            raw = ahead;
            if (r + 2 <= r1) ahead = adj_raw<VEC>(p, r + 2, c0, c1);
            nxt = adj_cells<MASKED, VEC>(p, raw, r + 1, c, in, r + 1 < r1 ? mine : B2{false, false}, &rain_acc);
            adj_gather<MASKED, VEC>(p, cur, nxt, r, c, mine, ax, ay, below);
        }
    }
    adj_flush_rain<THREADS>(p, rain_acc);
}

// The same without U_{k+1}: the updates are rebuilt from the faces' forward fluxes, each
// evaluated once within the warp, one row ahead of the reverse (the rows and columns
// outside the strip once more).  us a call at 257 x 333 masked, 512^2, 700^2, 1024^2,
// 2048^2 and masked 3000 x 3001: 22 (the host), 22, 23, 54, 208 and 458; with each
// cell's update rebuilt apart from its four faces and their cells' loads 25, 36, 49, 116,
// 370 and 796, in a tile of 32 x 16 cells 22, 31, 46, 102, 399 and 874.
template <int THREADS, bool MASKED, bool VEC>
__global__ void __launch_bounds__(THREADS, 3) adj_march_faces_kernel(const __grid_constant__ AdjLaunch p, int nstrips,
                                                                  int rows_per_warp) {
    const DomainDev& d = p.d;
    const int lane = threadIdx.x & 31;
    const int gw = blockIdx.x * (THREADS / kWarp) + (threadIdx.x >> 5);
    const int r0 = (gw / nstrips) * rows_per_warp, r1 = min(r0 + rows_per_warp, d.rows);
    const int c = (gw % nstrips) * kMarchCols - 2 + 2 * lane;
    const int c0 = min(max(c, 0), VEC ? d.cols - 2 : d.cols - 1), c1 = min(max(c + 1, 0), d.cols - 1);
    const B2 in{c >= 0 && c < d.cols, c + 1 >= 0 && c + 1 < d.cols};
    const bool strip = lane >= 1 && lane <= kWarp - 2;
    const B2 mine{strip && in.x, strip && in.y}, none{false, false};
    const float ax = p.s.dt * p.rdx, ay = p.s.dt * p.rdy;
    double rain_acc = 0.0;
    if (r0 < d.rows) {
        struct Row {
            AdjCells k;
            AdjMomenta m;
            V2 nm;
        };
        struct Flux {
            V2 m, n, t;  // mass, normal (with the side's pressure correction) and tangential momentum
        };
        auto row = [&](int r) -> Row {
            AdjRaw a;
            load_states<false, VEC>(p, r, c0, c1, a);
            Row w;
            w.k = adj_velocities<MASKED, VEC>(p, a, r, c, w.m);
            w.nm = a.nm;
            return w;
        };
        Flux low;  // the upper side of the face below the row
        auto face_above = [&](const Row& w, const Row& above) -> Flux {
            const AdjFlux<V2> f = adj_flux<0, MASKED, V2>(w.k.f, above.k.f, p.k);
            low = {f.m, f.n + f.hi, f.t};
            return {f.m, f.n + f.lo, f.t};
        };
        // dL/d(upd) of row r of cells w from its faces.
        auto reverse = [&](Row& w, const Row& above, int r, B2 owned) {
            const Flux yb = low, yt = face_above(w, above);
            const AdjFlux<V2> f = adj_flux<1, MASKED, V2>(w.k.f, right_of<MASKED>(w.k).f, p.k);
            // f.x is the face between a lane's cells, f.y the one to the next lane's first cell.
            auto left = [](V2 x) { return V2{{__shfl_up_sync(0xffffffffu, x.v.y, 1), x.v.x}}; };
            const V2 xm = f.m - left(f.m), xn = f.n + f.lo - left(f.n + f.hi), xt = f.t - left(f.t);
            if (r < 0 || r >= d.rows) return;
            const V2 upd[3] = {w.k.f.h - (ax * xm + ay * (yt.m - yb.m)), w.m.hu - (ax * xn + ay * (yt.t - yb.t)),
                               w.m.hv - (ax * xt + ay * (yt.n - yb.n))};
            AdjRaw a;
            load_lam<VEC>(p, r, c0, c1, a);
            const V2 lam[3] = {a.l0, a.l1, a.l2};
            adj_pointwise<AdjSource::kUpdate, MASKED>(p, r, c, w.nm, lam, upd, in & w.k.f.act, owned, &rain_acc, w.k.l);
        };
        Row cur = row(r0 - 1), nxt = row(r0), ahead = row(r0 + 1);
        face_above(row(r0 - 2), cur);
        reverse(cur, nxt, r0 - 1, none);
        reverse(nxt, ahead, r0, mine);
        V2 below[3];
        adj_first_face<MASKED>(p, cur.k, nxt.k, r0, ay, below);
        for (int r = r0; r < r1; ++r) {
            cur = nxt;
            nxt = ahead;
            ahead = row(r + 2);
            reverse(nxt, ahead, r + 1, r + 1 < r1 ? mine : none);
            adj_gather<MASKED, VEC>(p, cur.k, nxt.k, r, c, mine, ax, ay, below);
        }
    }
    adj_flush_rain<THREADS>(p, rain_acc);
}

}  // namespace swe

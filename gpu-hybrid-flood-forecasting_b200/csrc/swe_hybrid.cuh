// Physics-AI coupling kernels (sm_100a): network features and the
// volume-preserving residual correction of the hybrid rollout
// (src/hybrid_flood/hybrid/coupled_forecast.py:49-120).
#pragma once

#include <cuda_bf16.h>

#include "swe_exact.cuh"
#include "swe_step.cuh"

namespace swe {

// Feature layouts.
//   kFeatRef6   the reference's six channels (coupled_forecast.py:53-79):
//               (h, u, v) standardised by mean/std and zeroed off-mask, the rain
//               rate in mm/h over its scale, standardised terrain, roughness.
//   kFeatState5 (h, hu, hv, z, rain rate in mm/h), each standardised by
//               mean/std, off-mask cells zero.
constexpr int kFeatRef6 = 0;
constexpr int kFeatState5 = 1;

struct FeatureArgs {
    int rows, cols;
    StateView s;
    const float* nm;    // n^2 with the mask in the sign bit (pitch spitch)
    const float* bed;   // pitch spitch
    int64_t spitch;
    const float* terrain;    // rows*cols (kFeatRef6), may be null
    const float* roughness;  // rows*cols (kFeatRef6), may be null
    float mean[5], stdv[5];
    float rain_feature;      // the rain channel's value for this call
    float dry;
    void* out;               // [rows][cols][channels] (channels-last), bfloat16 or float32
};

// Warps of these kernels take pieces of kPiece columns of a row, a lane the
// columns lane + 32 k of it: a lane's loads of a piece are independent and issued
// together, and coalesced at every pitch and alignment.  All of them are bound
// by memory; with one cell at a time a warp had too few bytes in flight.  us at
// 2048^2 on a cold cache, one cell and four: features (float32, six channels)
// 56 and 33, output fields 33.5 and 21.9, the two correction passes 61 and 55 with a
// plane less in memory; the calls together 159 and 117.
constexpr int kCells = 4;  // cells a lane takes at a time
constexpr int kPiece = kCells * kWarp;
constexpr int kPieceWarps = 8;  // per CTA

// body(r, c0) for the warp's pieces (grid.x over pieces, grid.y over groups of rows, piece_grid on the host).
template <class F>
__device__ __forceinline__ void for_pieces(int rows, int cols, F&& body) {
    for (int r = (int)(blockIdx.y * kPieceWarps + (threadIdx.x >> 5)); r < rows; r += (int)gridDim.y * kPieceWarps)
        for (int c0 = (int)blockIdx.x * kPiece; c0 < cols; c0 += (int)gridDim.x * kPiece) body(r, c0);
}

// v[k] = f(column) for the lane's columns of the piece, 0 past the row's end.
template <class F>
__device__ __forceinline__ void piece_load(float (&v)[kCells], int c0, int cols, F&& f) {
#pragma unroll
    for (int k = 0; k < kCells; ++k) {
        const int c = c0 + k * kWarp + (int)(threadIdx.x & 31);
        v[k] = c < cols ? f(c) : 0.f;
    }
}

// Copies n elements of a warp's shared row to out (an element boundary) in the widest words its address allows.
template <class T>
__device__ __forceinline__ void warp_copy_out(T* out, const T* row, int n) {
    const int lane = threadIdx.x & 31;
    int done = 0;
    auto words = [&](auto w) {
        using W = decltype(w);
        if (sizeof(W) <= sizeof(T) || reinterpret_cast<uintptr_t>(out) % sizeof(W) != 0 || done != 0) return;
        constexpr int per = (int)(sizeof(W) / sizeof(T));
        const int m = n / (per > 0 ? per : 1);
        for (int i = lane; i < m; i += kWarp) reinterpret_cast<W*>(out)[i] = reinterpret_cast<const W*>(row)[i];
        done = m * per;
    };
    words(uint4{});
    words(uint2{});
    words(unsigned{});
    for (int i = done + lane; i < n; i += kWarp) out[i] = row[i];
}

// The channels of a cell are adjacent: a lane that stores them one by one touches
// a 32-byte sector per lane with each store, so they are laid out in shared
// memory and leave as whole lines.
template <int LAYOUT, class T>
__global__ void __launch_bounds__(kPieceWarps* kWarp) features_kernel(const FeatureArgs a) {
    constexpr int CH = LAYOUT == kFeatRef6 ? 6 : 5;
    __shared__ alignas(16) T s_row[kPieceWarps][kPiece * CH];
    T* row = s_row[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    auto put = [&](int cell, int q, float x) {
        if constexpr (sizeof(T) == 2)
            row[cell * CH + q] = __float2bfloat16_rn(x);
        else
            row[cell * CH + q] = x;
    };
    for_pieces(a.rows, a.cols, [&](int r, int c0) {
        const float* ph = a.s.h + (int64_t)r * a.s.pitch;
        const float* phu = a.s.hu + (int64_t)r * a.s.pitch;
        const float* phv = a.s.hv + (int64_t)r * a.s.pitch;
        const float* pnm = a.nm + (int64_t)r * a.spitch;
        float h[kCells], hu[kCells], hv[kCells], nm[kCells], e[kCells], f[kCells];
        piece_load(h, c0, a.cols, [&](int c) { return ph[c]; });
        piece_load(hu, c0, a.cols, [&](int c) { return phu[c]; });
        piece_load(hv, c0, a.cols, [&](int c) { return phv[c]; });
        piece_load(nm, c0, a.cols, [&](int c) { return pnm[c]; });
        if constexpr (LAYOUT == kFeatRef6) {
            const int64_t i = (int64_t)r * a.cols;
            piece_load(e, c0, a.cols, [&](int c) { return a.terrain ? a.terrain[i + c] : 0.f; });
            piece_load(f, c0, a.cols, [&](int c) { return a.roughness ? a.roughness[i + c] : 0.f; });
        } else {
            const float* pz = a.bed + (int64_t)r * a.spitch;
            piece_load(e, c0, a.cols, [&](int c) { return pz[c]; });
        }
        __syncwarp();  // the previous piece has left
#pragma unroll
        for (int k = 0; k < kCells; ++k) {
            const int cell = k * kWarp + lane;
            const bool act = active(nm[k]);
            auto standard = [&](int q, float x) {
                put(cell, q, act ? ranged_div(__fsub_rn(x, a.mean[q]), a.stdv[q]) : 0.f);
            };
            if constexpr (LAYOUT == kFeatRef6) {
                const bool wet = h[k] > a.dry;
                standard(0, h[k]);
                standard(1, wet ? ranged_div(hu[k], fmaxf(h[k], a.dry)) : 0.f);
                standard(2, wet ? ranged_div(hv[k], fmaxf(h[k], a.dry)) : 0.f);
                put(cell, 3, a.rain_feature);
                put(cell, 4, e[k]);
                put(cell, 5, f[k]);
            } else {
                standard(0, h[k]);
                standard(1, hu[k]);
                standard(2, hv[k]);
                standard(3, e[k]);
                standard(4, a.rain_feature);
            }
        }
        __syncwarp();
        warp_copy_out(static_cast<T*>(a.out) + ((int64_t)r * a.cols + c0) * CH, row, min(kPiece, a.cols - c0) * CH);
    });
}

struct CorrectionArgs {
    int rows, cols;
    StateView s;          // predicted state (physics result)
    StateOut out;         // corrected state (may alias s)
    const float* nm;
    int64_t spitch;
    const void* res;      // residual, element (r, c, ch) at res[r*rs_r + c*rs_c + ch*rs_ch]
    int64_t rs_r, rs_c, rs_ch;
    int res_channels;     // 1 (depth only) or 3 (depth, u, v)
    int res_bf16;         // 1: bfloat16 residual, 0: float32
    float lim[3];         // clip limits per channel (+inf: none), coupled_forecast.py:199-200
    float relax, dry, eps;
    double* sums;         // [2] device: sum of masked predicted h, sum of provisional h
};

// Residual channel ch of the lane's cells, clipped to [-lim, lim] with NaN kept (jnp.clip).
__device__ __forceinline__ void residual_load(float (&v)[kCells], const CorrectionArgs& a, int r, int c0, int ch) {
    const int64_t o = (int64_t)r * a.rs_r + (int64_t)ch * a.rs_ch;
    if (a.res_bf16)
        piece_load(v, c0, a.cols, [&](int c) {
            return __bfloat162float(static_cast<const __nv_bfloat16*>(a.res)[o + (int64_t)c * a.rs_c]);
        });
    else
        piece_load(v, c0, a.cols, [&](int c) { return static_cast<const float*>(a.res)[o + (int64_t)c * a.rs_c]; });
    const float l = a.lim[ch];
#pragma unroll
    for (int k = 0; k < kCells; ++k) v[k] = v[k] < -l ? -l : (v[k] > l ? l : v[k]);
}

// Provisional depth max(h + r*res_h, 0) of an active cell.  Both passes evaluate
// it: the residual's first channel is in the sectors that pass 2 reads for the
// others, and is no larger than a plane of it would be (33 MB at 2048^2).
__device__ __forceinline__ float provisional_depth(const CorrectionArgs& a, float nm, float h, float rh) {
    return active(nm) ? fmaxf(__fadd_rn(h, __fmul_rn(a.relax, rh)), 0.f) : 0.f;
}

// Pass 1: the two volume sums in float64 (coupled_forecast.py:98-104).
__global__ void __launch_bounds__(kPieceWarps* kWarp) correction_sums_kernel(const CorrectionArgs a) {
    double t = 0.0, p = 0.0;
    for_pieces(a.rows, a.cols, [&](int r, int c0) {
        const float* ph = a.s.h + (int64_t)r * a.s.pitch;
        const float* pnm = a.nm + (int64_t)r * a.spitch;
        float h[kCells], nm[kCells], rh[kCells];
        piece_load(h, c0, a.cols, [&](int c) { return ph[c]; });
        piece_load(nm, c0, a.cols, [&](int c) { return pnm[c]; });
        residual_load(rh, a, r, c0, 0);
#pragma unroll
        for (int k = 0; k < kCells; ++k) {
            if (c0 + k * kWarp + (int)(threadIdx.x & 31) >= a.cols) continue;
            if (active(nm[k])) t += (double)h[k];
            p += (double)provisional_depth(a, nm[k], h[k], rh[k]);
        }
    });
    t = warp_sum(t);
    p = warp_sum(p);
    __shared__ double s_t[32], s_p[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        s_t[w] = t;
        s_p[w] = p;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double tt = 0.0, pp = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            tt += s_t[k];
            pp += s_p[k];
        }
        atomicAdd(&a.sums[0], tt);
        atomicAdd(&a.sums[1], pp);
    }
}

// Pass 2: project onto the physics volume and rebuild the momenta
// (coupled_forecast.py:105-120).  Reads the predicted momenta before writing.
__global__ void __launch_bounds__(kPieceWarps* kWarp) correction_apply_kernel(const CorrectionArgs a) {
    const double target = a.sums[0], provisional = a.sums[1];
    const float scale = provisional > (double)a.eps ? (float)(target / provisional) : 1.f;
    const bool keep = !(target > (double)a.eps);
    for_pieces(a.rows, a.cols, [&](int r, int c0) {
        const float* ph = a.s.h + (int64_t)r * a.s.pitch;
        const float* phu = a.s.hu + (int64_t)r * a.s.pitch;
        const float* phv = a.s.hv + (int64_t)r * a.s.pitch;
        const float* pnm = a.nm + (int64_t)r * a.spitch;
        float h[kCells], hu[kCells], hv[kCells], nm[kCells], rh[kCells], ru[kCells], rv[kCells];
        piece_load(h, c0, a.cols, [&](int c) { return ph[c]; });
        piece_load(hu, c0, a.cols, [&](int c) { return phu[c]; });
        piece_load(hv, c0, a.cols, [&](int c) { return phv[c]; });
        piece_load(nm, c0, a.cols, [&](int c) { return pnm[c]; });
        residual_load(rh, a, r, c0, 0);
        if (a.res_channels >= 3) {
            residual_load(ru, a, r, c0, 1);
            residual_load(rv, a, r, c0, 2);
        }
#pragma unroll
        for (int k = 0; k < kCells; ++k) {
            const int c = c0 + k * kWarp + (int)(threadIdx.x & 31);
            if (c >= a.cols) continue;
            const int64_t oo = (int64_t)r * a.out.pitch + c;
            const bool wet0 = h[k] > a.dry;
            float u = wet0 ? ranged_div(hu[k], fmaxf(h[k], a.dry)) : 0.f;
            float v = wet0 ? ranged_div(hv[k], fmaxf(h[k], a.dry)) : 0.f;
            const float ch = keep ? h[k] : __fmul_rn(provisional_depth(a, nm[k], h[k], rh[k]), scale);
            if (a.res_channels >= 3) {
                u = __fadd_rn(u, __fmul_rn(a.relax, ru[k]));
                v = __fadd_rn(v, __fmul_rn(a.relax, rv[k]));
            }
            const bool wet = active(nm[k]) && ch > a.dry;
            a.out.h[oo] = ch;
            a.out.hu[oo] = wet ? __fmul_rn(ch, u) : 0.f;
            a.out.hv[oo] = wet ? __fmul_rn(ch, v) : 0.f;
        }
    });
}

// Output schema of a state (conserved_to_xarray, structured_io.py:160-209):
// depth, x/y velocity (momentum / depth where depth > dry, else 0) and speed
// (hypot, evaluated in double and rounded once as float32 hypot is), each NaN
// off the domain mask.  IEEE division, so the fields equal NumPy's bit for bit.
struct SchemaArgs {
    int rows, cols;
    StateView s;
    const float* nm;
    int64_t spitch;
    float dry;
    float *depth, *u, *v, *speed;
    int64_t out_pitch;
};

// ExactMath::hypot, by the root without branches where it is defined.
__device__ __forceinline__ float field_hypot(float u, float v) {
    const float m = fmaxf(fabsf(u), fabsf(v));
    return m < 3.0e38f && u == u && v == v ? quick_hypot(u, v) : ExactMath::hypot(u, v);
}

__global__ void __launch_bounds__(kPieceWarps* kWarp) schema_kernel(const SchemaArgs a) {
    const float nan = __int_as_float(0x7fc00000);
    for_pieces(a.rows, a.cols, [&](int r, int c0) {
        const float* ph = a.s.h + (int64_t)r * a.s.pitch;
        const float* phu = a.s.hu + (int64_t)r * a.s.pitch;
        const float* phv = a.s.hv + (int64_t)r * a.s.pitch;
        const float* pnm = a.nm + (int64_t)r * a.spitch;
        float h[kCells], hu[kCells], hv[kCells], nm[kCells];
        piece_load(h, c0, a.cols, [&](int c) { return ph[c]; });
        piece_load(hu, c0, a.cols, [&](int c) { return phu[c]; });
        piece_load(hv, c0, a.cols, [&](int c) { return phv[c]; });
        piece_load(nm, c0, a.cols, [&](int c) { return pnm[c]; });
#pragma unroll
        for (int k = 0; k < kCells; ++k) {
            const int c = c0 + k * kWarp + (int)(threadIdx.x & 31);
            if (c >= a.cols) continue;
            const int64_t oo = (int64_t)r * a.out_pitch + c;
            const bool act = active(nm[k]), wet = h[k] > a.dry;
            const float u = wet ? ranged_div(hu[k], h[k]) : 0.f;
            const float v = wet ? ranged_div(hv[k], h[k]) : 0.f;
            a.depth[oo] = act ? h[k] : nan;
            a.u[oo] = act ? u : nan;
            a.v[oo] = act ? v : nan;
            a.speed[oo] = act ? field_hypot(u, v) : nan;
        }
    });
}

}  // namespace swe

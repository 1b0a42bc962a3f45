// Start and end of runs (sm_100a): the control block, the initial state with its
// CFL maximum and volume, and the results, each as ONE launch for any number of
// domains.
//
// The state is read once: each cell goes into the run's first ping-pong buffer (and
// into output 0 and the strip-edge array) and into the reduction in the same pass,
// and the domains of a batch are parts of one grid, their arguments in the launch
// parameters.  What the calls around the steps cost is launches: 24 ensemble members
// start and end 50 steps in 0.9 of 9.0 ms with four of them (2.4 of 10.5 ms with a
// dozen operations a member), and compute_cfl_dt and a step of 96 x 130 take 48 us
// together (74 us with a clear, a reduction with IEEE divisions and a copy).
#pragma once

#include "swe_exact.cuh"
#include "swe_step.cuh"
#include "swe_step_pair.cuh"

namespace swe {

constexpr int kBatchDomains = 32;  // domains per launch (their arguments fit the 32 KB of launch parameters)

// ---------------------------------------------------------------------------
// Control blocks
// ---------------------------------------------------------------------------
// A run's control block written from launch parameters: the head as the host
// built it, the stripe maxima zeroed and the target times.  Parameters are
// captured when the launch is queued, so the host needs no staging buffer, and
// the queue never waits for the stream as a copy from pageable host memory may.
struct ControlHeadImage {
    unsigned long long w[kControlHead / 8];
};
static_assert(kControlHead % 8 == 0 && sizeof(ControlHeadImage) <= 2048, "control head must fit the launch parameters");

// NT output times carried in the launch parameters.
template <int NT>
struct InitDomain {
    Control* ctl;
    ControlHeadImage head;
    int n;              // entries of t (and of t64, at most 2, when times64 is set) written
    float t[NT];
    double t64[2];
    float* times;       // device arrays receiving them (times64 may be null)
    double* times64;
};

template <int ND, int NT>
struct InitBatch {
    InitDomain<NT> d[ND];
};
static_assert(sizeof(InitBatch<kBatchDomains, 2>) <= 32764, "a batch of control blocks must fit the launch parameters");

template <int ND, int NT>
__global__ void control_init_kernel(const __grid_constant__ InitBatch<ND, NT> b) {
    const InitDomain<NT>& q = b.d[blockIdx.x];
    auto* dst = reinterpret_cast<unsigned long long*>(q.ctl);
    for (int i = threadIdx.x; i < (int)(kControlHead / 8); i += blockDim.x) dst[i] = q.head.w[i];
    unsigned long long* mk = &q.ctl->maxk[0][0];
    for (int i = threadIdx.x; i < 2 * kMaxStripes * kStripeWords; i += blockDim.x) mk[i] = 0ull;
    for (int i = threadIdx.x; i < q.n; i += blockDim.x) q.times[i] = q.t[i];
    if (q.times64 && (int)threadIdx.x < min(q.n, 2)) q.times64[threadIdx.x] = q.t64[threadIdx.x];
}

// ---------------------------------------------------------------------------
// Initial state
// ---------------------------------------------------------------------------
// A CTA's share of the start reduction.
struct StartPartial {
    double vol;
    float maxinv;
};

// One domain of a load (swe_max_inverse_dt reduces a state without loading it:
// out.h, edge and slots null).
struct LoadDomain {
    int rows, cols, upd_lo, upd_hi;  // the rows [upd_lo, upd_hi) are reduced
    int gx, gy, cta0;                // its CTAs: gx over the columns, gy over the rows, from cta0 on
    int edge_rows, nslots;
    Consts k;
    double area;
    const float* nm;
    int64_t spitch;
    StateView in;
    StateOut out;       // ping-pong buffer 0, or null
    float* snap[3];     // output 0 (rows x cols contiguous), or null
    float* edge;        // strip-edge array of buffer 0 (DomainDev::edge), or null
    LedgerSlot* slots;  // cleared, or null
    Control* ctl;
    StartPartial* parts;  // gx * gy
    float* host_max;      // host memory receiving the maximum, or null
};

template <int ND>
struct LoadBatch {
    int n;
    LoadDomain d[ND];
};
static_assert(sizeof(LoadBatch<kBatchDomains>) <= 32764, "a batch of loads must fit the launch parameters");

// (|u| + c)/dx + (|v| + c)/dy of a cell (shallow_water_2d.py:269-273).
__device__ __noinline__ inline float ieee_inverse_dt(float h, float hu, float hv, float g, float dry, float dx, float dy) {
    float u, v;
    ExactMath::vel2(hu, hv, h, dry, u, v);
    const float w = ExactMath::sqrt(ExactMath::mul(g, fmaxf(h, 0.0f)));
    return ExactMath::add(ExactMath::div(ExactMath::add(fabsf(u), w), dx), ExactMath::div(ExactMath::add(fabsf(v), w), dy));
}

template <class M>
__device__ __forceinline__ float inverse_dt(const Consts& k, float rdx, float rdy, float h, float hu, float hv) {
    if constexpr (M::kExact) {
        if (!(k.forms & kFormQuick)) return ieee_inverse_dt(h, hu, hv, k.g, k.dry, k.dx, k.dy);
        // The branch-free form, and the IEEE operations for a cell outside its range.
        // (A velocity too small for it does not reach the sum: the celerity of a wet cell is
        // 2^-18 at least, from the smallest gravity and dry tolerance of kFormQuick, and
        // only quotients below 2^-94 can differ.)
        const SoloOps o;
        const bool wet = h > k.dry;
        const float rh = quick_rcp(o, h);
        const float u = wet ? quick_div(o, hu, h, rh) : 0.f, v = wet ? quick_div(o, hv, h, rh) : 0.f;
        const float w = o.mul(quick_celerity_up(o, fmaxf(h, 0.f), k.g * 1.8446744073709552e19f), kDown);
        const float inv = o.add(quick_div(o, o.add(fabsf(u), w), k.dx, rdx), quick_div(o, o.add(fabsf(v), w), k.dy, rdy));
        if (max3_nan(h, fabsf(u), fabsf(v)) < kQuickLimit) return inv;
        return ieee_inverse_dt(h, hu, hv, k.g, k.dry, k.dx, k.dy);
    } else {
        float u, v;
        M::vel2(hu, hv, h, k.dry, u, v);
        const float w = M::sqrt(M::mul(k.g, fmaxf(h, 0.0f)));
        return M::add(M::div(M::add(fabsf(u), w), k.dx), M::div(M::add(fabsf(v), w), k.dy));
    }
}

// CTA-wide maximum and sum (fixed order), valid on thread 0.  The maximum is of
// non-negative values or NaN, whose bit patterns compare as integers.
template <int THREADS>
__device__ __forceinline__ StartPartial start_reduce(float maxinv, double vol) {
    constexpr int W = THREADS / kWarp;
    __shared__ unsigned s_max[W];
    __shared__ double s_vol[W];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(maxinv) & 0x7fffffffu);
    vol = warp_sum(vol);
    if (lane == 0) {
        s_max[warp] = m;
        s_vol[warp] = vol;
    }
    __syncthreads();
    StartPartial p{};
    if (threadIdx.x == 0) {
        unsigned mm = s_max[0];
        p.vol = s_vol[0];
        for (int w = 1; w < W; ++w) {
            mm = max(mm, s_max[w]);
            p.vol += s_vol[w];
        }
        p.maxinv = __uint_as_float(mm);
    }
    __syncthreads();  // s_max / s_vol are free again
    return p;
}

// End of a load: the CTA partials are folded by the domain's last CTA to arrive,
// in a fixed order, into the initial volume and CFL maximum, and the run's first
// position is set: clock at t_start, output 0 taken as the initial state, the
// first target loaded, the maximum stored for step 0 (step count 0 in the high
// word of stripe 0).
template <int THREADS>
__device__ void finish_start(const LoadDomain& q, int cta, float maxinv, double vol) {
    const int nparts = q.gx * q.gy;
    Control* ctl = q.ctl;
    __shared__ bool s_last;
    const StartPartial p = start_reduce<THREADS>(maxinv, vol);
    if (threadIdx.x == 0) {
        q.parts[cta] = p;
        __threadfence();
        s_last = atomicAdd(&ctl->counter, 1u) == (unsigned)nparts - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // Thread t folds partials t, t+T, ...; the loads bypass the L1 (the other CTAs'
    // writes are visible in the L2 after the fence).
    float m = 0.f;
    double v = 0.0;
    for (int b = threadIdx.x; b < nparts; b += THREADS) {
        const float bm = __ldcg(&q.parts[b].maxinv);
        m = nan_max(m, bm);
        v += __ldcg(&q.parts[b].vol);
    }
    const StartPartial t = start_reduce<THREADS>(m, v);
    if (threadIdx.x != 0) return;
    float mx = t.maxinv;
    // A NaN volume means a non-finite state somewhere: report it as a NaN CFL
    // maximum, the form plan_step tests.
    if (!(t.vol == t.vol)) mx = __int_as_float(0x7fffffff);
    const int n_out = ctl->n_out;
    RunPos p0;
    p0.t = ctl->t_start;
    p0.target = n_out > 1 ? output_time(ctl, 1) : 0.0;
    p0.rain = RainSeg{0.0, 0.0, 0.0, 0.0, 0.0, -1};
    p0.steps = 0;
    p0.idx = 1;
    p0.done = (1 >= n_out || ctl->max_steps <= 0) ? 1 : 0;
    p0.status = 0;
    ctl->pos[0] = p0;
    ctl->t = p0.t;
    ctl->dt = 0.0;
    ctl->idx = 1;
    ctl->steps = 0;
    ctl->done = p0.done;
    ctl->status = 0;
    ctl->ledger[0] = t.vol * q.area;
    ctl->ledger[1] = t.vol * q.area;
    ctl->ledger[2] = ctl->ledger[3] = ctl->ledger[4] = ctl->ledger[5] = 0.0;
    // A row strip plans from the maximum across strips: NaN is kept as +inf
    // there, so that a maximum carries it.
    const float shown = (ctl->defer_plan && !(mx == mx)) ? INFINITY : mx;
    ctl->maxinv = shown;
    ctl->maxk[0][0] = (unsigned long long)(__float_as_uint(mx) & 0x7fffffffu);
    ctl->counter = 0;
    if (q.host_max) *q.host_max = shown;
    __threadfence_system();
}

// Max inverse CFL dt and stored volume of the states (the reduction of
// compute_cfl_dt, shallow_water_2d.py:269-273), the states copied into the runs'
// buffers on the way.  A thread has four rows' loads in flight.
template <class M, int THREADS, int ND>
__global__ void __launch_bounds__(THREADS) load_kernel(const __grid_constant__ LoadBatch<ND> b) {
    int m = 0;
    while (m + 1 < b.n && (int)blockIdx.x >= b.d[m + 1].cta0) ++m;
    const LoadDomain& q = b.d[m];
    const int cta = (int)blockIdx.x - q.cta0, bx = cta % q.gx, by = cta / q.gx;
    const Consts& k = q.k;
    const float rdx = __frcp_rn(k.dx), rdy = __frcp_rn(k.dy);
    if (q.slots) {
        double* s = reinterpret_cast<double*>(q.slots);
        const int n = q.nslots * (int)(sizeof(LedgerSlot) / sizeof(double));
        for (int i = cta * THREADS + (int)threadIdx.x; i < n; i += q.gx * q.gy * THREADS) s[i] = 0.0;
    }
    float maxinv = 0.f;
    double vol = 0.0;
    constexpr int kRows = 4;
    for (int c = bx * THREADS + (int)threadIdx.x; c < q.cols; c += q.gx * THREADS) {
        // The strip-edge run of this column: right cell of the boundary at a strip's
        // first column, left cell of the next boundary at its last.
        const int in_strip = c % kEdgeStrip, bd = c / kEdgeStrip;
        float* edge = nullptr;
        if (q.edge && in_strip == 0) edge = q.edge + ((int64_t)bd * 6 + 3) * q.edge_rows;
        if (q.edge && in_strip == kEdgeStrip - 1) edge = q.edge + (int64_t)(bd + 1) * 6 * q.edge_rows;
        for (int r0 = by; r0 < q.rows; r0 += kRows * q.gy) {
            float h[kRows], hu[kRows], hv[kRows], nm[kRows];
#pragma unroll
            for (int j = 0; j < kRows; ++j) {
                const int r = min(r0 + j * q.gy, q.rows - 1);
                const int64_t so = (int64_t)r * q.in.pitch + c;
                h[j] = q.in.h[so];
                hu[j] = q.in.hu[so];
                hv[j] = q.in.hv[so];
                nm[j] = q.nm[(int64_t)r * q.spitch + c];
            }
#pragma unroll
            for (int j = 0; j < kRows; ++j) {
                const int r = r0 + j * q.gy;
                if (r >= q.rows) break;
                if (q.out.h) {
                    const int64_t oo = (int64_t)r * q.out.pitch + c;
                    q.out.h[oo] = h[j];
                    q.out.hu[oo] = hu[j];
                    q.out.hv[oo] = hv[j];
                }
                if (q.snap[0]) {
                    const int64_t oo = (int64_t)r * q.cols + c;
                    q.snap[0][oo] = h[j];
                    q.snap[1][oo] = hu[j];
                    q.snap[2][oo] = hv[j];
                }
                if (edge) {
                    edge[r] = h[j];
                    edge[r + q.edge_rows] = hu[j];
                    edge[r + 2 * q.edge_rows] = hv[j];
                }
                if (r >= q.upd_lo && r < q.upd_hi && active(nm[j])) {
                    maxinv = nan_max(maxinv, inverse_dt<M>(k, rdx, rdy, h[j], hu[j], hv[j]));
                    vol += (double)h[j];
                }
            }
        }
    }
    finish_start<THREADS>(q, cta, maxinv, vol);
}

// ---------------------------------------------------------------------------
// Results
// ---------------------------------------------------------------------------
// What the host reads of a finished run, written to its (page-locked) memory by
// the fold.
struct RunSummary {
    double t;
    double ledger[6];
    int idx, steps, done, status;
};

struct FoldDomain {
    double area;
    Control* ctl;
    const LedgerSlot* slots;
    int nslots;
    RunSummary* host;
};

template <int ND>
struct FoldBatch {
    FoldDomain d[ND];
};

// The runs' ledgers from the warps' slots (one CTA per domain, fixed order): the
// stored volume of the last step and the rain, outflow, clip and mask terms summed
// over the run.  With no step taken the volume stays the initial one.
template <int THREADS, int ND>
__global__ void __launch_bounds__(THREADS) ledger_fold_kernel(const __grid_constant__ FoldBatch<ND> b) {
    const FoldDomain& q = b.d[blockIdx.x];
    Accum a;
    a.zero();
    for (int i = threadIdx.x; i < q.nslots; i += THREADS) {
        a.vol += q.slots[i].vol; a.rain += q.slots[i].rain; a.outflow += q.slots[i].outflow;
        a.clip += q.slots[i].clip; a.mask += q.slots[i].mask;
    }
    const Partial t = cta_reduce<THREADS>(a);
    if (threadIdx.x != 0) return;
    Control* c = q.ctl;
    c->ledger[1] = c->steps > 0 ? t.vol * q.area : c->ledger[0];
    c->ledger[2] = t.rain * q.area;
    c->ledger[3] = t.outflow;
    c->ledger[4] = t.clip * q.area;
    c->ledger[5] = t.mask * q.area;
    RunSummary s;
    s.t = c->t;
    for (int i = 0; i < 6; ++i) s.ledger[i] = c->ledger[i];
    s.idx = c->idx;
    s.steps = c->steps;
    s.done = c->done;
    s.status = c->status;
    *q.host = s;
    __threadfence_system();
}

// The runs' final states into the callers' planes: the ping-pong buffer is the
// parity of the steps taken, read from the control block.
struct StoreDomain {
    int rows, cols, gx, gy, cta0;
    const float* src[2][3];
    int64_t spitch;
    float* dst[3];
    int64_t dpitch;
    const Control* ctl;
    int unless_failed;  // 1: a run that stopped with an error status leaves dst as it was
};

template <int ND>
struct StoreBatch {
    int n;
    StoreDomain d[ND];
};
static_assert(sizeof(StoreBatch<kBatchDomains>) <= 32764, "a batch of stores must fit the launch parameters");

template <int THREADS, int ND>
__global__ void __launch_bounds__(THREADS) store_kernel(const __grid_constant__ StoreBatch<ND> b) {
    int m = 0;
    while (m + 1 < b.n && (int)blockIdx.x >= b.d[m + 1].cta0) ++m;
    const StoreDomain& q = b.d[m];
    if (q.unless_failed && q.ctl->status) return;
    const int cta = (int)blockIdx.x - q.cta0, bx = cta % q.gx, by = cta / q.gx;
    const int par = q.ctl->steps & 1;
    const float* h = q.src[par][0];
    const float* hu = q.src[par][1];
    const float* hv = q.src[par][2];
    constexpr int kRows = 4;
    for (int c = bx * THREADS + (int)threadIdx.x; c < q.cols; c += q.gx * THREADS)
        for (int r0 = by; r0 < q.rows; r0 += kRows * q.gy) {
            float x[kRows][3];
#pragma unroll
            for (int j = 0; j < kRows; ++j) {
                const int64_t so = (int64_t)min(r0 + j * q.gy, q.rows - 1) * q.spitch + c;
                x[j][0] = h[so];
                x[j][1] = hu[so];
                x[j][2] = hv[so];
            }
#pragma unroll
            for (int j = 0; j < kRows; ++j) {
                const int r = r0 + j * q.gy;
                if (r >= q.rows) break;
                const int64_t o = (int64_t)r * q.dpitch + c;
                q.dst[0][o] = x[j][0];
                q.dst[1][o] = x[j][1];
                q.dst[2][o] = x[j][2];
            }
        }
}

// A run's position, in host memory.  Written by a kernel and not copied: a copy of
// a few words waits behind the outputs on their way to the host (0.9 ms for a
// 2048^2 state), and the steps queued behind it with it.
struct RunProgress {
    double t, dt;
    int idx, steps, done;
};

__global__ void run_progress_kernel(const Control* c, RunProgress* host) {
    if (threadIdx.x) return;
    *host = RunProgress{c->t, c->dt, c->idx, c->steps, c->done};
    __threadfence_system();
}

// How far an ensemble's advance to a target time has come, in host memory: the
// members that are done and the largest number of steps one is expected to take
// (the time left at its current dt).
struct EnsProgress {
    int done;
    long long expected;
};

__global__ void ens_progress_kernel(const MemberDev* members, int n, double target, EnsProgress* host) {
    __shared__ int s_done, s_expected;
    if (threadIdx.x == 0) s_done = s_expected = 0;
    __syncthreads();
    for (int m = threadIdx.x; m < n; m += blockDim.x) {
        const Control* c = members[m].ctl;
        if (c->done) {
            atomicAdd(&s_done, 1);
            continue;
        }
        const double left = c->dt > 0.0 ? fmin(fmax(ceil((target - c->t) / c->dt), 1.0), 1.0e9) : 1.0;
        atomicMax(&s_expected, c->steps + (int)left);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        host->done = s_done;
        host->expected = s_expected;
        __threadfence_system();
    }
}

}  // namespace swe

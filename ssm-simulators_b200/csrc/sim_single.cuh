// What the single-accumulator simulators share: the per-trial rows, the launch
// parameters, the boundaries, and how a walk is found, started and finished.
// sim_single.cu steps one walk per lane (throughput), sim_wide.cu one walk per
// group of lanes (latency).
#pragma once

#include "common.cuh"

namespace ssm {

// M_SDV: ddm_sdv (drift v + sv N(0,1) per trajectory); M_FULL: full_ddm (and
// start point + U(-sz, sz), non-decision time + U(-st, st)); M_OU:
// ornstein_uhlenbeck (drift v - g y); M_DFLEX: ddm_flex (drift v(t) from a
// per-trial table the host evaluates from the drift function).
enum Model { M_FLEX = 0, M_LEGACY = 1, M_LEVY = 2, M_SDV = 3, M_FULL = 4, M_OU = 5, M_DFLEX = 6 };

struct alignas(16) TrialRow {
    float drift;     // v * dt ; SDV/FULL: v
    float scale;     // sqrt(dt) * s ;  Levy: s * dt^(1/alpha)
    float y0;        // start point
    float dl_tmp;    // min(max_t, deadline - t): the walk runs while t <= dl_tmp
    float t;         // non-decision time
    float deadline;  // rt >= deadline (or deadline <= 0) -> omission
    float a;         // boundary height (legacy DDM: upper bound)
    float p1;        // LINEAR: slope ; WEIBULL: shape alpha
    float p2;        // WEIBULL: scale beta
    float dtp1;      // dt * p1 (linear boundary per step, fast path)
    float inv_beta;  // 1 / beta
    float alpha;     // Levy: stability index ; SDV/FULL: sv ; OU: v
    float inv_alpha; // Levy: 1 / alpha ; FULL: sz ; OU: g
    float expo;      // Levy: (1 - alpha) / alpha ; FULL: st ; OU: 1 - g dt
    float capf;      // hard limit on Euler steps: a walk reaching it raises SSM_ERR_DEVICE
    float c2;        // -2 ln(2) * scale^2: folds the noise scale into Box-Muller's radius
};
static_assert(sizeof(TrialRow) == 64, "TrialRow is one 64-byte line");

// A walk that the one-lane kernel leaves to the lanes-per-walk kernel: where it
// stands, at a step that is a whole number of blocks.
struct alignas(16) LeftWalk {
    int64_t w;
    uint32_t k, n;
    float y, tp, ixf, dinc;
    uint32_t pad[4];
};
static_assert(sizeof(LeftWalk) == 48, "three 16-byte rows");
// A warp leaves its walks once the queue is empty and this many or fewer are
// still running (see k_single).  Measured (ms; 0 = walks stay, 4, 16): 256 angle
// sets 1.91, 1.67, 1.65; 64 sets 1.48, 1.03, 0.75; 64 Levy sets 4.78, 2.98, 2.62;
// 512 Ornstein sets 8.84, 8.80, 8.45; 24 measured as 16.
constexpr int LEAVE_MAX = 16;

struct SingleParams {
    PhiloxKeys key;
    const TrialRow *rows;
    const int64_t *offsets;  // ragged prefix sums (n_trials + 1) or nullptr
    const int32_t *order;    // ragged only: trial simulated j-th (nullptr = index order)
    const int64_t *qoff;     // prefix sums of the sample counts in that order
    int64_t n_trials;
    int64_t total;           // number of trajectories; -1 = offsets[n_trials] - offsets[0]
    uint32_t k_base;         // random-stream index of trial 0 (trial windows of a larger batch)
    int ustride;             // injected uniforms per trajectory (3 for full_ddm: u_t, u_y, u_smooth)
    float dt;
    int smooth;
    int chunk;
    int refill_min;          // ended walks a warp collects before it restarts lanes
    const float *table;
    int64_t tstride, tlen;
    const float *dtable;     // DFLEX: drift v(t_ix) per trial, row stride dstride, dlen entries
    int64_t dstride, dlen;
    int dvec;                // rows 16-byte aligned: a block's drifts are float4 loads
    const float *noise;      // injected increments: row w holds nlen floats
    int64_t nlen;
    const float *nunif;      // injected jitter uniforms, one per trajectory
    float *rts;
    int32_t *choices;
    int32_t *steps;
    WorkspaceHeader *hdr;
    LeftWalk *left;          // walks left to the lanes-per-walk kernel (hdr->aux[0] of them), or nullptr
    float *traj;             // trajectory recorder (record kernel only)
    int64_t traj_len;
};

__device__ __forceinline__ int64_t ragged_find(const int64_t *off, int64_t K, int64_t w,
                                               int64_t hint) {
    int64_t k = hint;
    if (k < 0 || k >= K || __ldg(off + k) > w) k = 0;
    int64_t step = 1;
    while (k + step < K && __ldg(off + k + step) <= w) {
        k += step;
        step <<= 1;
    }
    int64_t hi = (k + step < K) ? k + step : K;
    while (hi - k > 1) {
        const int64_t mid = (k + hi) >> 1;
        if (__ldg(off + mid) <= w) k = mid; else hi = mid;
    }
    return k;
}

template <int BOUND, bool EXACT>
__device__ __forceinline__ float bound_at(const TrialRow &r, float ixf, int ix,
                                          const SingleParams &p, int64_t k) {
    if (BOUND == SSM_BOUND_CONSTANT) {
        return r.a;
    } else if (BOUND == SSM_BOUND_LINEAR) {
        // table value a + f32(ix*dt) * p1 (boundary_functions.py:57-72 on t_s)
        if (EXACT) return __fadd_rn(r.a, __fmul_rn(__fmul_rn(ixf, p.dt), r.p1));
        return fmaf(ixf, r.dtp1, r.a);
    } else if (BOUND == SSM_BOUND_WEIBULL) {
        // a * exp(-(t/beta)^alpha) (boundary_functions.py:103-122)
        const float x = ixf * p.dt * r.inv_beta;
        const float pw = (x > 0.f) ? exp2f(r.p1 * __log2f(x)) : 0.f;
        return r.a * __expf(-pw);
    } else {
        const int64_t i = (ix < p.tlen) ? ix : p.tlen - 1;
        return __ldg(p.table + k * p.tstride + i);
    }
}

// sin x and cos x on [0, pi/2] from their Taylor series through x^11 and x^12
// (truncation errors below 6e-8 and 7e-9 there): short branch-free code for
// the stable sampler, whose angles are always reduced to that interval.
__device__ __forceinline__ float sin_q(float x) {
    const float t = x * x;
    float p = fmaf(t, -2.5052108e-08f, 2.7557319e-06f);  // -1/11!, 1/9!
    p = fmaf(t, p, -1.9841270e-04f);                     // -1/7!
    p = fmaf(t, p, 8.3333333e-03f);                      // 1/5!
    p = fmaf(t, p, -1.6666667e-01f);                     // -1/3!
    p = fmaf(t, p, 1.0f);
    return x * p;
}
__device__ __forceinline__ float cos_q(float x) {
    const float t = x * x;
    float p = fmaf(t, 2.0876757e-09f, -2.7557319e-07f);  // 1/12!, -1/10!
    p = fmaf(t, p, 2.4801587e-05f);                      // 1/8!
    p = fmaf(t, p, -1.3888889e-03f);                     // -1/6!
    p = fmaf(t, p, 4.1666667e-02f);                      // 1/4!
    p = fmaf(t, p, -0.5f);
    return fmaf(t, p, 1.0f);
}

// Symmetric alpha-stable variate by Chambers-Mallows-Stuck (Chambers, Mallows
// & Stuck, JASA 71, 1976) with the reference's guards (_utils.pyx:426-472):
// U ~ U(-pi/2 + 1e-7, pi/2 - 1e-7), W ~ Exp(1) floored at 1e-10, output
// clipped to +-1e10 and NaN -> 0.
//   X = sin(alpha U) / cos(U)^(1/alpha) * (cos((1 - alpha) U) / W)^((1 - alpha) / alpha)
// (tan U for alpha = 1).  U = pi (u - 1/2) with u on a 2^-23 grid; the sampler
// works with |U| and its complement V = pi/2 - |U| = pi min(u, 1 - u), which
// carries one rounding only, so cos U = sin V keeps its relative precision as
// |U| -> pi/2, where the heavy tail comes from.  Both powers are taken as one
// power of two.
__device__ __forceinline__ float cms_stable(uint32_t bu, uint32_t bw, const TrialRow &r) {
    const float u01 = bits_to_1_2(bu) - 1.0f;
    const float m = fmaxf(0.5f - fabsf(u01 - 0.5f), 3.1830988e-08f);  // V >= 1e-7 (the U clamp)
    const float V = 3.14159265f * m;
    const float aU = 1.57079633f - V;  // |U|
    const float W = fmaxf(-0.69314718f * lg2_ftz(uniform_open(bw)), 1e-10f);
    float X;
    if (r.alpha == 1.0f) {
        X = cos_q(V) / sin_q(V);  // |tan U|
    } else {
        const float cu = sin_q(V);                                             // cos U > 0
        // cos((1 - alpha) U) = cos(c |U|), c = |1 - alpha| <= 1, evaluated as
        // sin(pi/2 - c |U|) = sin(pi/2 (1 - c) + c V): two non-negative terms,
        // so the argument does not cancel, and one polynomial serves every c |U|
        const float c = fabsf(1.0f - r.alpha);
        const float cua = fmaxf(sin_q(fmaf(c, V, 1.57079633f * (1.0f - c))), 1e-10f);
        // alpha |U| in [0, pi); past pi/2 use pi - alpha |U| = pi (1 - alpha/2) + alpha V,
        // which does not cancel as alpha -> 2
        float A = r.alpha * aU;
        if (A > 1.57079633f) A = fmaf(r.alpha, V, 3.14159265f * fmaf(-0.5f, r.alpha, 1.0f));
        const float e = fmaf(r.expo, lg2_ftz(cua) - lg2_ftz(W), -r.inv_alpha * lg2_ftz(cu));
        float p2;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p2) : "f"(e));
        X = sin_q(A) * p2;  // |sin(alpha U)| ...
    }
    X = (u01 < 0.5f) ? -X : X;  // ... times sign(U): every factor but sin(alpha U) is even in U
    if (X != X) X = 0.f;
    return fminf(fmaxf(X, -1e10f), 1e10f);
}

// Two stable variates at once, the arithmetic of cms_stable two lanes to an
// instruction (the SFU's functions, minima and selects stay scalar): the same
// values.  512 Levy sets of 10 000: 18.3 -> 16.1 ms.
__device__ __forceinline__ uint64_t dup_f2(float x) { return pack_f2(x, x); }
__device__ __forceinline__ uint64_t sin_q2(uint64_t x) {
    const uint64_t t = mul_f2(x, x);
    uint64_t p = fma_f2(t, dup_f2(-2.5052108e-08f), dup_f2(2.7557319e-06f));
    p = fma_f2(t, p, dup_f2(-1.9841270e-04f));
    p = fma_f2(t, p, dup_f2(8.3333333e-03f));
    p = fma_f2(t, p, dup_f2(-1.6666667e-01f));
    p = fma_f2(t, p, dup_f2(1.0f));
    return mul_f2(x, p);
}
__device__ __forceinline__ void cms_stable2(uint4 b, const TrialRow &r, float &x0, float &x1) {
    if (r.alpha == 1.0f) {
        x0 = cms_stable(b.x, b.y, r);
        x1 = cms_stable(b.z, b.w, r);
        return;
    }
    const float2 u01 = unpack_f2(add_f2(pack_f2(bits_to_1_2(b.x), bits_to_1_2(b.z)), dup_f2(-1.0f)));
    const float2 h = unpack_f2(add_f2(pack_f2(u01.x, u01.y), dup_f2(-0.5f)));
    const float2 d = unpack_f2(add_f2(dup_f2(0.5f), pack_f2(-fabsf(h.x), -fabsf(h.y))));
    const uint64_t m = pack_f2(fmaxf(d.x, 3.1830988e-08f), fmaxf(d.y, 3.1830988e-08f));  // V >= 1e-7
    const uint64_t V = mul_f2(dup_f2(3.14159265f), m);
    const uint64_t aU = fma_f2(V, dup_f2(-1.0f), dup_f2(1.57079633f));  // pi/2 - V of the rounded V, as in cms_stable
    const float2 uw = unpack_f2(add_f2(pack_f2(bits_to_1_2(b.y), bits_to_1_2(b.w)), dup_f2(-0.99999994f)));
    const float2 lw = unpack_f2(mul_f2(dup_f2(-0.69314718f), pack_f2(lg2_ftz(uw.x), lg2_ftz(uw.y))));
    const float W0 = fmaxf(lw.x, 1e-10f), W1 = fmaxf(lw.y, 1e-10f);
    const float2 cu = unpack_f2(sin_q2(V));
    const float c = fabsf(1.0f - r.alpha);
    const float2 sc = unpack_f2(sin_q2(fma_f2(dup_f2(c), V, dup_f2(1.57079633f * (1.0f - c)))));
    const float cua0 = fmaxf(sc.x, 1e-10f), cua1 = fmaxf(sc.y, 1e-10f);
    const uint64_t al = dup_f2(r.alpha);
    const float2 A = unpack_f2(mul_f2(al, aU));
    const float2 B = unpack_f2(fma_f2(al, V, dup_f2(3.14159265f * fmaf(-0.5f, r.alpha, 1.0f))));
    const float A0 = (A.x > 1.57079633f) ? B.x : A.x, A1 = (A.y > 1.57079633f) ? B.y : A.y;
    const uint64_t dl = add_f2(pack_f2(lg2_ftz(cua0), lg2_ftz(cua1)), pack_f2(-lg2_ftz(W0), -lg2_ftz(W1)));
    const float2 e = unpack_f2(fma_f2(dup_f2(r.expo), dl,
                                      mul_f2(dup_f2(-r.inv_alpha), pack_f2(lg2_ftz(cu.x), lg2_ftz(cu.y)))));
    float p0, p1;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p0) : "f"(e.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(p1) : "f"(e.y));
    const float2 X = unpack_f2(mul_f2(sin_q2(pack_f2(A0, A1)), pack_f2(p0, p1)));
    x0 = (u01.x < 0.5f) ? -X.x : X.x;
    x1 = (u01.y < 0.5f) ? -X.y : X.y;
    if (x0 != x0) x0 = 0.f;
    if (x1 != x1) x1 = 0.f;
    x0 = fminf(fmaxf(x0, -1e10f), 1e10f);
    x1 = fminf(fmaxf(x1, -1e10f), 1e10f);
}

struct Lane {
    int64_t w;
    uint32_t k, n, blk;
    int ix;           // steps taken (maintained where an integer index is needed)
    float y, tp, ixf; // position, float32 time accumulator, steps taken as float (see step_block)
    float tpb;        // time accumulator at the start of the current block
    float dinc;       // SDV/FULL: this trajectory's drift increment (v + sv g) dt
};

// models whose drift is drawn once per trajectory
template <int MODEL> struct DrawnDrift { static constexpr bool value = (MODEL == M_SDV || MODEL == M_FULL); };

// Models and boundaries that a caller may run with several lanes per walk.
template <int MODEL, bool NOISE, int BOUND> struct WideOk {
    static constexpr bool value =
        !NOISE && MODEL != M_LEVY && MODEL != M_DFLEX && BOUND != SSM_BOUND_TABLE;
};
// The rt of a walk of trial k, sample n that ended at time tp (output index w):
// time + non-decision time + jitter, omitted past the deadline.
template <int MODEL, bool NOISE>
__device__ __forceinline__ float finish_rt(const SingleParams &p, uint32_t k, uint32_t n, int64_t w, float tp) {
    // fields needed only here are re-read instead of being held across the walk
    const TrialRow *row = p.rows + k;
    const float t = __ldg(&row->t), deadline = __ldg(&row->deadline), dl = __ldg(&row->dl_tmp);
    float u;
    if (NOISE) u = __ldg(p.nunif + w * p.ustride + (p.ustride - 1));
    else u = uniform_co(philox10(make_uint4(0u, n, k + p.k_base, 1u), p.key).x);
    float tt = t;
    if (MODEL == M_FULL) {
        // t + 2 (u - 0.5) st in double (ddm_models.pyx:2253); the same uniform as at the start
        float ut;
        if (NOISE) ut = __ldg(p.nunif + w * p.ustride);
        else ut = uniform_co(philox10(make_uint4(0u, n, k + p.k_base, 3u), p.key).z);
        tt = __double2float_rn((double)t + (2.0 * ((double)ut - 0.5)) * (double)__ldg(&row->expo));
    }
    // compute_smooth_unif (_utils.pyx:668-695): double arithmetic, float result
    float sm = 0.f;
    if (p.smooth) {
        if (tp == 0.f) sm = __double2float_rn(((double)u * 0.5) * (double)p.dt);
        else if (tp < dl) sm = __double2float_rn((0.5 - (double)u) * (double)p.dt);
    }
    const float rt = __fadd_rn(__fadd_rn(tp, tt), sm);
    return (rt >= deadline || deadline <= 0.f) ? -999.f : rt;  // enforce_deadline
}

// The trial that queue index w belongs to: queue indices [lo, hi) are its
// samples 0, 1, ... and sample n is output out0 + n.
struct Span {
    int64_t lo, hi, out0;
    uint32_t k;
};

// Find the span of queue index w (ragged layout; hint: the search's last
// position); false (and the error word set) if a caller-given processing order
// does not cover that index.
__device__ __forceinline__ bool find_span(const SingleParams &p, int64_t w, int64_t &hint, Span &s) {
    int64_t k;
    if (p.order != nullptr) {
        // queue index -> position j in the processing order -> trial k; the
        // output index stays offsets[k] + n, so results do not depend on the order
        const int64_t j = ragged_find(p.qoff, p.n_trials, w, hint);
        hint = j;
        k = __ldg(p.order + j);
        s.lo = __ldg(p.qoff + j);
        s.hi = __ldg(p.qoff + j + 1);
        const int64_t n = w - s.lo;
        if (k < 0 || k >= p.n_trials || n < 0 || n >= __ldg(p.offsets + k + 1) - __ldg(p.offsets + k)) {
            raise_error(p.hdr, SSM_ERR_ARG, (int)j);
            return false;
        }
        // a span never reaches past its trial's outputs
        s.hi = min(s.hi, s.lo + __ldg(p.offsets + k + 1) - __ldg(p.offsets + k));
        s.out0 = __ldg(p.offsets + k);
    } else {
        const int64_t w0 = __ldg(p.offsets);  // global output index (trial windows start past 0)
        k = ragged_find(p.offsets, p.n_trials, w + w0, hint);
        hint = k;
        s.out0 = __ldg(p.offsets + k);
        s.lo = s.out0 - w0;
        s.hi = __ldg(p.offsets + k + 1) - w0;
    }
    s.k = (uint32_t)k;
    return true;
}

// Start lane L on sample n of trial k (output index w).  A fresh lane has L.k =
// NO_TRIAL.
constexpr uint32_t NO_TRIAL = 0xffffffffu;
template <int MODEL, bool NOISE>
__device__ __forceinline__ void lane_start(const SingleParams &p, Lane &L, TrialRow &r, int64_t w, uint32_t k,
                                           uint32_t n) {
    if (L.k != k) {  // else the lane's last walk was of this trial
        const float4 *src = reinterpret_cast<const float4 *>(p.rows + k);
        float4 *dst = reinterpret_cast<float4 *>(&r);
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = __ldg(src + i);
    }
    L.w = w;
    L.k = k;
    L.n = n;
    L.blk = 0;
    L.ix = 0;
    L.ixf = 0.f;
    L.tp = 0.f;
    L.y = r.y0;
    if (DrawnDrift<MODEL>::value) {
        // per-trajectory drift normal and (full_ddm) start-point uniform
        // (ddm_models.pyx:2249-2266): injected, or drawn from the trajectory's stream
        float g0, uy = 0.5f;
        if (NOISE) {
            g0 = __ldg(p.noise + L.w * p.nlen);
            if (MODEL == M_FULL) uy = __ldg(p.nunif + L.w * p.ustride + 1);
        } else {
            const uint4 b = philox10(make_uint4(0u, L.n, L.k + p.k_base, 3u), p.key);
            g0 = box_muller(b.x, b.y).x;
            uy = uniform_co(b.w);
        }
        L.dinc = __fmul_rn(__fadd_rn(r.drift, __fmul_rn(r.alpha, g0)), p.dt);
        if (MODEL == M_FULL)
            L.y = __double2float_rn((double)L.y + (2.0 * ((double)uy - 0.5)) * (double)r.inv_alpha);
    }
}

// Trial and sample of queue index w in the reference layout (output w = n
// n_trials + k); one trial, and 32-bit division where it reaches.
__device__ __forceinline__ void layout_trial(const SingleParams &p, int64_t w, uint32_t &k, uint32_t &n) {
    if (p.n_trials == 1) {
        k = 0u;
        n = (uint32_t)w;
    } else if (((w | p.n_trials) >> 32) == 0) {
        n = (uint32_t)w / (uint32_t)p.n_trials;
        k = (uint32_t)w - n * (uint32_t)p.n_trials;
    } else {
        k = (uint32_t)(w % p.n_trials);
        n = (uint32_t)(w / p.n_trials);
    }
}

// Lanes-per-walk launches (sim_wide.cu): the whole call with W = 8, 16 or 32
// lanes per walk (with p.traj one more CTA records trial 0 / sample 0's path
// beside the walks), or the walks that k_single left in p.left.
int wide_launch(int model, int bound, int W, const SingleParams &p, const ssm_launch *opt, cudaStream_t st);
int wide_finish(int model, int bound, const SingleParams &p, cudaStream_t st);

}  // namespace ssm

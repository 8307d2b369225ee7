// Single-accumulator Euler-Maruyama simulators for sm_100a: the flexible-bound
// DDM (cssm.ddm_flexbound), the legacy [0, a] DDM (cssm.ddm) and the Levy
// flight DDM (cssm.levy_flexbound).
//
// Design (one thread per trajectory, persistent grid):
//  * A per-trial prologue (k_prep) turns the reference's per-trial arrays into
//    a 64-byte TrialRow with every derived float computed once, in the same
//    IEEE operation order the reference uses (src/cssm/ddm_models.pyx:700-744).
//  * The main kernel runs one grid of resident CTAs.  Each warp claims
//    trajectories from a global work counter in chunks; once refill_min of
//    its lanes have ended their walks (ballot), it writes their results and
//    hands them the next trajectories of its chunk (popc rank) in one
//    divergent pass, so that pass is paid once per several trajectories and
//    an ended lane idles for a few blocks at most.
//  * Steps run in blocks of 36 (24 for ddm_flex with a Weibull or table
//    bound, 16 for Levy): six independent Philox4x32-10 calls yield 24 words =
//    18 Box-Muller pairs = the block's increments, already scaled to drift +
//    s sqrt(dt) N(0,1), drawn two calls at a time in the step loop just before
//    the twelve steps that use them, with two pairs to an FP32 instruction; the
//    steps themselves are predicated (no per-step branch), and a warp whose walks
//    cannot reach their time limit within the block skips the time test.
//  * What bounds it: the issue of integer and SFU work of the draws.  A step
//    of the angle batch takes 26 cycles of a warp scheduler; its SFU operations alone
//    (two per increment, eight cycles each) 16.  Occupancy does not matter from 8
//    warps per SM up.  4 096 angle sets, 43 M walks: 27.4 -> 24.3 ms (packed pairs,
//    the rts turned from times into results by k_finish, restarts that stay in
//    their trial without a search); 509 Levy sets of 9 973: 19.1 -> 14.5 ms (packed
//    transform, 16-step blocks).
//  * A launch lasts as long as its longest walk.  When the queue is empty and a
//    warp has at most LEAVE_MAX walks left, it hands them (LeftWalk) to k_wide
//    (sim_wide.cu), which gives each of them eight lanes; a launch with fewer walks
//    than the grid has lanes may go there as a whole, on 8, 16 or 32 lanes a walk
//    (effective_lanes).  Outputs are bit-identical to one lane per walk.
//  * Boundaries are evaluated in registers (constant / linear collapse /
//    Weibull) or read from a caller-evaluated table for arbitrary shapes.
//  * Noise injection replaces the generator by caller rows and switches every
//    float operation to explicit round-to-nearest intrinsics, giving results
//    bit-identical to the sequential CPU restatement.
#include <cuda.h>  // CUcontext / CUresult types of the driver entry points below

#include <algorithm>
#include <mutex>

#include "sim_single.cuh"

namespace ssm {

struct PrepArgs {
    const float *v, *a, *z, *t, *deadline, *s, *alpha, *p1, *p2, *maxt_k, *table;
    const float *sv, *sz, *st, *g;  // variability (SDV/FULL) and leak (OU) parameters
    int64_t n_trials, tstride;
    float dt, sqrt_dt, max_t;
    int model, bound;
    TrialRow *rows;
};

// ------------------------------------------------------------------ prologue
__global__ void k_prep(const PrepArgs A) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= A.n_trials) return;
    TrialRow r;
    const float dt = A.dt;
    r.drift = __fmul_rn(A.v[k], dt);
    r.t = A.t[k];
    r.deadline = A.deadline[k];
    const float maxt = A.maxt_k ? A.maxt_k[k] : A.max_t;
    const float dl = __fsub_rn(r.deadline, r.t);
    r.dl_tmp = (dl < maxt) ? dl : maxt;  // src/cssm/_utils.pyx:712-718
    r.a = A.a ? A.a[k] : 0.f;
    r.p1 = A.p1 ? A.p1[k] : 0.f;
    r.p2 = A.p2 ? A.p2[k] : 1.f;
    r.dtp1 = dt * r.p1;
    r.inv_beta = 1.0f / r.p2;
    r.alpha = A.alpha ? A.alpha[k] : 2.f;
    r.inv_alpha = (float)(1.0 / (double)r.alpha);
    r.expo = (float)((1.0 - (double)r.alpha) / (double)r.alpha);
    if (A.model == M_SDV || A.model == M_FULL) {
        r.drift = A.v[k];  // the drift increment (v + sv g) dt is drawn per trajectory
        r.alpha = A.sv[k];
        r.inv_alpha = (A.model == M_FULL) ? A.sz[k] : 0.f;
        r.expo = (A.model == M_FULL) ? A.st[k] : 0.f;
    } else if (A.model == M_OU) {
        r.alpha = A.v[k];
        r.inv_alpha = A.g[k];
        r.expo = 1.0f - A.g[k] * dt;
    }
    // The walk stops once the float32 time passes dl_tmp, i.e. after about
    // dl_tmp/dt steps; twice that plus slack bounds every legal walk.  A stalled
    // accumulator (dt below half an ulp of t) or an infinite horizon hits the cap.
    const double nsteps = (double)r.dl_tmp / (double)dt;
    if (!(nsteps > 0.0)) r.capf = 64.f;                   // NaN or <= 0: at most one step
    else if (nsteps <= 8388608.0) r.capf = (float)(int)(2.0 * nsteps + 64.0);
    else r.capf = 0.f;                                    // unsupported horizon: flagged
    if (A.model == M_LEVY) {
        // delta_t_alpha = s * pow(delta_t, 1.0 / alpha) in double (levy_models.pyx:166)
        r.scale = __double2float_rn((double)A.s[k] * pow((double)dt, 1.0 / (double)r.alpha));
    } else {
        r.scale = __fmul_rn(A.sqrt_dt, A.s[k]);  // ddm_models.pyx:705
    }
    r.c2 = -1.3862944f * r.scale * r.scale;
    if (A.model == M_LEGACY) {
        r.y0 = __fmul_rn(A.z[k], r.a);  // ddm_models.pyx:451
    } else if (A.model == M_OU || A.model == M_DFLEX) {
        // (-1) * b0 + z * 2 * b0 with integer literals: float arithmetic
        // (ornstein_models.pyx:167, ddm_models.pyx:1014)
        const float b0 = (A.bound == SSM_BOUND_TABLE) ? A.table[k * A.tstride] : r.a;
        r.y0 = __fadd_rn(-b0, __fmul_rn(__fmul_rn(A.z[k], 2.0f), b0));
    } else {
        const float b0 = (A.bound == SSM_BOUND_TABLE) ? A.table[k * A.tstride] : r.a;
        // -b0 + z*2*b0, evaluated in double as the generated C does (ddm_models.pyx:709)
        const double bd = (double)b0;
        r.y0 = __double2float_rn(__dadd_rn(-bd, __dmul_rn(__dmul_rn((double)A.z[k], 2.0), bd)));
    }
    reinterpret_cast<TrialRow *>(A.rows)[k] = r;
}

// Euler steps per block.  The Gaussian models draw six increments per
// Philox4x32-10 call (three Box-Muller pairs, see bm6_increment), so a
// 36-step block makes six independent Philox calls whose latencies overlap.
// Measured on the 4096-set angle batch on one B200 (ms per launch): six per
// call with 24-step blocks 27.8, 36 steps 26.8, 48 steps 27.0 (all 80
// registers, 3 CTAs per SM; 4 CTAs per SM at 64 registers 27.3 for 24 and 36
// steps); four per call with 32-step blocks 31.2.  With the re-tuned launch
// (128 threads, claims of 256): 30 steps 26.95, 36 steps 26.54, 42 steps
// 26.39, but on 1024 sets 42 steps is the slower (8.02 against 7.92 ms).
// ddm_flex holds a block's table drifts in registers as well: with the
// increments drawn a block at a time, 24 steps (four Philox calls, six float4
// drift loads) took 14.46 ms on the 1 024 conflict_ds sets against 15.73 for
// 12 steps and 16.51 for 16-step blocks of four increments per call (36 steps
// spilled).  With the draws fused into the steps (step_block FUSE) 36 steps
// fit for the constant and linear bounds (11.42 -> 11.00 ms against 24); the
// Weibull and table bounds keep 24 (at 36 the Weibull bound spills 294 bytes).
// The Levy model takes 16-step blocks: 512 sets of 10 000, 15.4 ms against 15.8
// for 8 steps, 16.3 for 24 and 17.1 for 32 (which spill).
// Call h of block b uses counter (BLK/6) b + h, so a stream does not depend
// on the block length.
template <int MODEL, int BOUND = SSM_BOUND_CONSTANT> struct Blk {
    static constexpr int value =
        (MODEL == M_LEVY) ? 16
                          : ((MODEL == M_DFLEX && BOUND != SSM_BOUND_CONSTANT && BOUND != SSM_BOUND_LINEAR) ? 24 : 36);
};
// Device-RNG Gaussian models draw their increments inside the step loop
// (step_block FUSE).  Outputs are bit-identical to drawing the block first;
// measured on one B200 (ms per launch): 4 096-set angle batch 26.43 -> 26.33
// (80 -> 64 registers), 1 024 conflict_ds sets 12.29 -> 11.42 (its 52-62 bytes
// of spills gone), Ornstein 20.70 -> 20.41.
template <int MODEL, bool NOISE> struct FuseOk {
    static constexpr bool value = !NOISE && MODEL != M_LEVY;
};
// Increments drawn together: two Philox calls' twelve, whose Box-Muller pairs
// share packed instructions (4 096-set angle batch 25.4 -> 24.4 ms against one
// call's six at a time); one call's six for a Weibull bound, whose own arithmetic
// needs the registers (256 sets: 4.41 ms against 4.67 with twelve).
template <int BOUND> struct DrawN { static constexpr int value = (BOUND == SSM_BOUND_WEIBULL) ? 6 : 12; };

// Increments DrawN h .. DrawN (h + 1) - 1 of the lane's current block from the
// device RNG (Gaussian models): Philox calls (BLK/6) blk + ... of the
// trajectory's stream, six increments each.
template <int MODEL, int BOUND>
__device__ __forceinline__ void draw_calls(const SingleParams &p, const Lane &L, const TrialRow &r, int h,
                                           float *g) {
    constexpr int BLK = Blk<MODEL, BOUND>::value, C = DrawN<BOUND>::value / 6;
    // ddm_flex: drift 0 here, v(t_ix) dt from the table in the step
    const float drift = (MODEL == M_DFLEX) ? 0.f : (DrawnDrift<MODEL>::value ? L.dinc : r.drift);
    const uint32_t ctr = (uint32_t)(BLK / 6) * L.blk + (uint32_t)(C * h);
    const uint4 b0 = philox10(make_uint4(ctr, L.n, L.k + p.k_base, 0u), p.key);
    if constexpr (C == 1) {
        bm6_increment(b0, r.c2, drift, g);
    } else {
        const uint4 b1 = philox10(make_uint4(ctr + 1u, L.n, L.k + p.k_base, 0u), p.key);
        bm12_increment(b0, b1, r.c2, drift, g);
    }
}

// The block's increments.  Noise injection returns the raw caller draws (the
// step applies drift and scale with explicit rounding); the device RNG returns
// finished increments drift + scale * X.
template <int MODEL, int BOUND, bool NOISE>
__device__ __forceinline__ void draw_block(const SingleParams &p, const Lane &L, const TrialRow &r,
                                           float g[Blk<MODEL, BOUND>::value]) {
    constexpr int BLK = Blk<MODEL, BOUND>::value;
    if (NOISE) {
        // SDV/FULL rows start with the trajectory's drift normal
        constexpr int OFF = DrawnDrift<MODEL>::value ? 1 : 0;
        const float *row = p.noise + L.w * p.nlen + OFF;
#pragma unroll
        for (int q = 0; q < BLK; ++q) g[q] = (L.ix + OFF + q < p.nlen) ? __ldg(row + L.ix + q) : 0.f;
    } else if (MODEL == M_LEVY) {
        // two variates per call; calls count in groups of four (eight steps), whatever the block length
#pragma unroll
        for (int h = 0; h < BLK / 2; ++h) {
            const uint4 b = philox10(make_uint4((uint32_t)(BLK / 8) * L.blk + (uint32_t)(h / 4), L.n, L.k + p.k_base,
                                                2u + (uint32_t)(h % 4)), p.key);
            float x0, x1;
            cms_stable2(b, r, x0, x1);
            g[2 * h] = fmaf(r.scale, x0, r.drift);
            g[2 * h + 1] = fmaf(r.scale, x1, r.drift);
        }
    } else {
        constexpr int DN = DrawN<BOUND>::value;
        static_assert(MODEL == M_LEVY || BLK % DN == 0, "whole draws per block");
#pragma unroll
        for (int h = 0; h < BLK / DN; ++h) draw_calls<MODEL, BOUND>(p, L, r, h, g + DN * h);
    }
}

// Advance one lane by up to BLK Euler steps.  Every step first tests the
// reference's `while` condition (ddm_models.pyx:719; legacy DDM :451); once it
// fails the remaining steps of the block are predicated off.  Returns whether
// the walk is still running.  With FUSE (device RNG, Gaussian models) the
// increments are drawn inside the step loop, six per Philox call (g unused):
// the same values as draw_block, with each call's draws in the same straight-
// line code as the steps, so their independent work fills the latency of the
// dependent step chain and only six increments are live at a time.
template <int MODEL, int BOUND, bool NOISE, bool RECORD, bool TCHK = true, bool FUSE = false>
__device__ __forceinline__ bool step_block(const SingleParams &p, Lane &L, const TrialRow &r,
                                           const float *g) {
    constexpr int BLK = Blk<MODEL, BOUND>::value;
    static_assert(!FUSE || (!NOISE && MODEL != M_LEVY), "fused draws: device RNG, Gaussian models");
    constexpr int DN = DrawN<BOUND>::value;
    float gd[DN];
    if (L.ixf >= r.capf) {
        raise_error(p.hdr, SSM_ERR_DEVICE, (int)L.w);
        return false;
    }
    constexpr bool INT_IX = NOISE || RECORD || BOUND == SSM_BOUND_TABLE;
    // Without an integer index (device RNG, in-register bounds) step q of the
    // block sits at step ixf0 + q: the step count advances once per block,
    // the linear bound is a + ixf0 slope dt plus q slope dt, and finalize()
    // recovers the steps of the last block from the time accumulator.
    const float ixf0 = L.ixf;
    // (Levy: bases every eight steps)
    constexpr int BB = (MODEL == M_LEVY) ? 8 : BLK;
    float base[BLK / BB];
#pragma unroll
    for (int u = 0; u < BLK / BB; ++u)
        base[u] = (!INT_IX && BOUND == SSM_BOUND_LINEAR) ? fmaf(ixf0 + (float)(BB * u), r.dtp1, r.a) : 0.f;
    if (!INT_IX) L.tpb = L.tp;
    const float *drow = (MODEL == M_DFLEX) ? p.dtable + (int64_t)L.k * p.dstride : nullptr;
    // device RNG: the block's drifts v(t_ix .. t_ix+BLK-1) are read before
    // the steps, off the dependency chain (a live walk starts every block at
    // a multiple of BLK steps); past the table's end the last entry repeats
    float dvq[BLK];
    if (MODEL == M_DFLEX && !NOISE) {
        const int ix0 = INT_IX ? L.ix : (int)ixf0;  // the block's first step
        if (p.dvec && (ix0 & 3) == 0 && ix0 + BLK <= p.dlen) {
            const float4 *d4 = reinterpret_cast<const float4 *>(drow + ix0);
#pragma unroll
            for (int h = 0; h < BLK / 4; ++h) {
                const float4 a = __ldg(d4 + h);
                dvq[4 * h] = a.x; dvq[4 * h + 1] = a.y; dvq[4 * h + 2] = a.z; dvq[4 * h + 3] = a.w;
            }
        } else {
#pragma unroll
            for (int q = 0; q < BLK; ++q) dvq[q] = __ldg(drow + ((ix0 + q < p.dlen) ? ix0 + q : p.dlen - 1));
        }
    }
    bool live = true;
#pragma unroll
    for (int q = 0; q < BLK; ++q) {
        if (FUSE && q % DN == 0) draw_calls<MODEL, BOUND>(p, L, r, q / DN, gd);
        const float gq = FUSE ? gd[q % DN] : g[q];
        bool inside;
        // the time test; a block whose every step is known to pass it skips it (TCHK false)
        const bool in_time = !TCHK || (L.tp <= r.dl_tmp);
        if (MODEL == M_LEGACY) {
            inside = live && (L.y <= r.a) && (L.y >= 0.f) && in_time;
        } else {
            float b;
            if (INT_IX) b = bound_at<BOUND, NOISE>(r, L.ixf, L.ix, p, L.k);
            else if (BOUND == SSM_BOUND_LINEAR) b = (q % BB == 0) ? base[q / BB] : fmaf((float)(q % BB), r.dtp1, base[q / BB]);
            else b = bound_at<BOUND, NOISE>(r, ixf0 + (float)q, 0, p, L.k);
            inside = live && (fabsf(L.y) <= b) && in_time;
        }
        if (NOISE && inside && L.ix + (DrawnDrift<MODEL>::value ? 1 : 0) >= p.nlen) {
            raise_error(p.hdr, SSM_ERR_NOISE_RANGE, (int)L.w);
            inside = false;
        }
        if (inside) {
            if (NOISE) {
                if (MODEL == M_OU) {
                    // (y + (v - g y) dt) + scale*g (ornstein_models.pyx:177)
                    const float lk = __fmul_rn(__fsub_rn(r.alpha, __fmul_rn(r.inv_alpha, L.y)), p.dt);
                    L.y = __fadd_rn(__fadd_rn(L.y, lk), __fmul_rn(r.scale, gq));
                } else if (MODEL == M_DFLEX) {
                    // (y + v(t_ix) dt) + scale*g (ddm_models.pyx:1025)
                    const float dv = __ldg(drow + ((L.ix < p.dlen) ? L.ix : p.dlen - 1));
                    L.y = __fadd_rn(__fadd_rn(L.y, __fmul_rn(dv, p.dt)), __fmul_rn(r.scale, gq));
                } else {
                    // (y + v*dt) + scale*g: the association the reference build uses
                    const float dr = DrawnDrift<MODEL>::value ? L.dinc : r.drift;
                    L.y = __fadd_rn(__fadd_rn(L.y, dr), __fmul_rn(r.scale, gq));
                }
                L.tp = __fadd_rn(L.tp, p.dt);
            } else {
                if (MODEL == M_OU) L.y = fmaf(L.y, r.expo, gq);  // y (1 - g dt) + v dt + noise
                else if (MODEL == M_DFLEX)                          // y + v(t_ix) dt + noise
                    L.y += fmaf(dvq[q], p.dt, gq);
                else L.y += gq;
                L.tp += p.dt;
            }
            if (INT_IX) {
                L.ixf += 1.0f;
                L.ix += 1;
            }
            if (RECORD && L.ix < p.traj_len) p.traj[L.ix] = L.y;
        }
        live = inside;
    }
    if (!INT_IX) L.ixf = ixf0 + (float)BLK;
    return live;
}

// True when all BLK time tests of the lane's next block are known to pass
// (device RNG, in-register bounds only).  Step q of the block tests the float
// accumulator after q more additions of dt, at most t + (BLK-1) dt plus the
// additions' rounding; below 65536 dt an ulp of t is at most dt/64, so that
// rounding stays under dt/4, and t + (BLK+1) dt <= dl_tmp, evaluated in float,
// leaves more than that margin.
template <int MODEL, int BOUND, bool NOISE>
__device__ __forceinline__ bool block_in_time(const SingleParams &p, const Lane &L, const TrialRow &r) {
    constexpr bool INT_IX = NOISE || BOUND == SSM_BOUND_TABLE;
    if (INT_IX) return false;
    constexpr float SPAN = (float)(Blk<MODEL, BOUND>::value + 1);
    return (L.tp < p.dt * 65536.f) && (fmaf(SPAN, p.dt, L.tp) <= r.dl_tmp);
}

// Steps taken by a walk that has ended.  Without an integer index L.ixf
// counts whole blocks; the steps of the last block are those that took the
// time accumulator from L.tpb to L.tp (the same float additions replayed).
template <int MODEL, int BOUND, bool NOISE>
__device__ __forceinline__ int steps_taken(const SingleParams &p, const Lane &L) {
    constexpr int BLK = Blk<MODEL, BOUND>::value;
    constexpr bool INT_IX = NOISE || BOUND == SSM_BOUND_TABLE;
    if (INT_IX) return (int)L.ixf;
    float tt = L.tpb;
    int c = 0;
    while (c < BLK && tt != L.tp) {
        tt += p.dt;
        ++c;
    }
    return (int)L.ixf - BLK + c;
}

// Write an ended walk's outputs.  With LATE the time is written as it is and
// k_finish turns the whole array into rts: a warp finishes few walks at a time,
// so the jitter's Philox call and the rest of finish_rt would run here with
// most lanes idle (about 100 instructions per pass, 5 % of the launch).
template <int MODEL, int BOUND, bool NOISE, bool LATE>
__device__ __forceinline__ void finalize(const SingleParams &p, const Lane &L) {
    p.rts[L.w] = LATE ? L.tp : finish_rt<MODEL, NOISE>(p, L.k, L.n, L.w, L.tp);
    p.choices[L.w] = (L.y > 0.f) - (L.y < 0.f);  // sign(y)
    if (p.steps) p.steps[L.w] = steps_taken<MODEL, BOUND, NOISE>(p, L);
}

// ------------------------------------------------------------------ main kernel
// One lane per walk.  80 registers: three 256-thread CTAs per SM; more resident
// warps measured no faster (24.4 ms with 24 to 32 warps per SM).
template <int MODEL, int BOUND, bool NOISE>
__global__ void __launch_bounds__(256, 3) k_single(const __grid_constant__ SingleParams p) {
    constexpr int BLK = Blk<MODEL, BOUND>::value;
    static_assert(BLK % 2 == 0, "walks are handed over at even steps (TimeSteps, sim_wide.cu)");
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    const int64_t total = (p.total >= 0) ? p.total : __ldg(p.offsets + p.n_trials) - __ldg(p.offsets);
    const int64_t chunk = warp_chunk(p.chunk, total);

    Lane L;
    TrialRow r = {};
    L.w = 0; L.k = NO_TRIAL; L.n = L.blk = 0; L.ix = 0; L.y = L.tp = L.ixf = L.dinc = L.tpb = 0.f;
    bool active = false;
    bool pending = false;  // walk ended, result not yet written
    bool exhausted = false;
    int64_t q_next = 0, q_end = 0, hint = 0;
    // The last trial this warp looked up (the same in every lane).  A claim is
    // consecutive queue indices, so most restarts stay in it: the next `left` of
    // them are its samples n_next, n_next + 1, ... with outputs from w_next, and need
    // neither the queue nor a search (q_next is brought up to date by left0 -
    // left when they run out).
    Span sp = {0, 0, 0, 0u};
    if (p.offsets == nullptr && p.n_trials == 1) sp.hi = total;
    int64_t w_next = 0;
    uint32_t n_next = 0u;
    int left = 0, left0 = 0;
    constexpr bool LATE = !NOISE;  // rts by k_finish (see finalize)

    for (;;) {
        // Lanes whose walk ended wait (predicated off) until refill_min of
        // them have: finishing and restarting lanes runs divergently, with the
        // rest of the warp idle, so it is done for several lanes in one pass.
        // Once the queue is empty, pending results are written at once.
        const unsigned need = __ballot_sync(FULL, !active);
        const int cnt = __popc(need);
        if (need != 0u && (exhausted || cnt >= p.refill_min)) {
            if (pending) {
                finalize<MODEL, BOUND, NOISE, LATE>(p, L);
                pending = false;
            }
            const int rank = __popc(need & lt_mask);
            if (cnt <= left) {
                if (!active) {
                    lane_start<MODEL, NOISE>(p, L, r, w_next + rank, sp.k, n_next + (uint32_t)rank);
                    active = true;
                }
                w_next += cnt;
                n_next += (uint32_t)cnt;
                left -= cnt;
            } else if (!exhausted) {
                q_next += left0 - left;
                const int64_t avail = q_end - q_next;
                int64_t base = 0;
                if (avail < cnt) {
                    unsigned long long b = 0ull;
                    if (lane == 0) b = atomicAdd(&p.hdr->counter, (unsigned long long)chunk);
                    base = (int64_t)__shfl_sync(FULL, b, 0);
                    if ((uint64_t)base >= (uint64_t)total) exhausted = true;
                }
                const int64_t w = (rank < avail) ? q_next + rank : base + (rank - avail);
                const bool start = !active && w < total;
                if (p.offsets == nullptr) {
                    if (start) {
                        uint32_t k, n;
                        layout_trial(p, w, k, n);
                        lane_start<MODEL, NOISE>(p, L, r, w, k, n);
                        active = true;
                    }
                } else {
                    // the last restart's trial, searched by the whole warp, is the
                    // next ones' most likely one; a restart of another trial
                    // searches on its own
                    const unsigned misses = __ballot_sync(FULL, start && !(w >= sp.lo && w < sp.hi));
                    if (misses != 0u) {
                        const int64_t last = __shfl_sync(FULL, w, 31 - __clz(misses));
                        if (!find_span(p, last, hint, sp)) sp.lo = sp.hi = 0;
                    }
                    if (start) {
                        Span mine = sp;
                        int64_t from = hint;
                        if ((w >= sp.lo && w < sp.hi) || find_span(p, w, from, mine)) {
                            const int64_t n = w - mine.lo;
                            lane_start<MODEL, NOISE>(p, L, r, mine.out0 + n, mine.k, (uint32_t)n);
                            active = true;
                        }
                    }
                    __syncwarp();
                }
                if (avail >= cnt) {
                    q_next += cnt;
                } else {
                    q_next = base + (cnt - avail);
                    q_end = base + chunk;
                }
                const int64_t in_span = (q_next >= sp.lo) ? sp.hi - q_next : 0;
                left = left0 = exhausted ? 0 : (int)max(min(min(q_end, total) - q_next, in_span), (int64_t)0);
                w_next = sp.out0 + (q_next - sp.lo);
                n_next = (uint32_t)(q_next - sp.lo);
            }
        }
        // The queue is empty and few of the warp's walks still run: a walk here
        // takes the time of a whole warp's steps, a walk with eight lanes of its
        // own a tenth of it, so they are left to the lanes-per-walk kernel.
        if (p.left != nullptr && exhausted) {
            const unsigned on = __ballot_sync(FULL, active);
            if (__popc(on) <= LEAVE_MAX) {
                unsigned long long b = 0ull;
                if (lane == 0) b = atomicAdd(&p.hdr->aux[0], (unsigned long long)__popc(on));
                b = __shfl_sync(FULL, b, 0);
                if (active) {
                    LeftWalk &o = p.left[b + __popc(on & lt_mask)];
                    o.w = L.w; o.k = L.k; o.n = L.n;
                    o.y = L.y; o.tp = L.tp; o.ixf = L.ixf; o.dinc = L.dinc;
                    active = false;
                }
            }
        }
        if (__ballot_sync(FULL, active) == 0u) break;
        // warp-uniform: skip the per-step time test when no active lane can reach its limit in this block
        const bool skip_time = __all_sync(FULL, !active || block_in_time<MODEL, BOUND, NOISE>(p, L, r));
        bool live = false;
        if (active) {
            if constexpr (FuseOk<MODEL, NOISE>::value) {
                live = skip_time ? step_block<MODEL, BOUND, NOISE, false, false, true>(p, L, r, nullptr)
                                 : step_block<MODEL, BOUND, NOISE, false, true, true>(p, L, r, nullptr);
            } else {
                float g[BLK];
                draw_block<MODEL, BOUND, NOISE>(p, L, r, g);
                live = skip_time ? step_block<MODEL, BOUND, NOISE, false, false>(p, L, r, g)
                                 : step_block<MODEL, BOUND, NOISE, false, true>(p, L, r, g);
            }
        }
        if (active) {
            L.blk += 1;
            if (!live) {
                active = false;
                pending = true;
            }
        }
    }
}

// The rts of a launch whose walks wrote their bare times (finalize LATE): one
// thread per output, full warps.  Each CTA takes runs of FINISH_RUN consecutive
// outputs, so one search places the run and the threads walk on from there.
constexpr int FINISH_RUN = 2048;
template <int MODEL>
__global__ void __launch_bounds__(256) k_finish(const __grid_constant__ SingleParams p) {
    const int64_t w0 = p.offsets ? __ldg(p.offsets) : 0;
    const int64_t total = (p.total >= 0) ? p.total : __ldg(p.offsets + p.n_trials) - w0;
    for (int64_t b = (int64_t)blockIdx.x * FINISH_RUN; b < total; b += (int64_t)gridDim.x * FINISH_RUN) {
        int64_t hint = 0;
#pragma unroll 2
        for (int64_t i = b + threadIdx.x; i < min(b + FINISH_RUN, total); i += 256) {
            uint32_t k, n;
            if (p.offsets == nullptr) {
                layout_trial(p, i, k, n);
            } else {
                hint = ragged_find(p.offsets, p.n_trials, w0 + i, hint);
                k = (uint32_t)hint;
                n = (uint32_t)(w0 + i - __ldg(p.offsets + hint));
            }
            const float tp = p.rts[w0 + i];
            p.rts[w0 + i] = finish_rt<MODEL, false>(p, k, n, w0 + i, tp);
        }
    }
}

// Re-simulates trial 0 / sample 0 with the same stream and writes its path
// (metadata['trajectory'], -999 padded: ddm_models.pyx:714-728).
template <int MODEL, int BOUND, bool NOISE>
__global__ void k_record(const __grid_constant__ SingleParams p) {
    for (int64_t i = threadIdx.x; i < p.traj_len; i += blockDim.x) p.traj[i] = -999.f;
    __syncthreads();
    if (threadIdx.x != 0) return;
    Lane L;
    TrialRow r;
    // sample 0 of the first trial that has one
    L.k = NO_TRIAL;
    int64_t k0 = 0;
    if (p.offsets != nullptr) k0 = ragged_find(p.offsets, p.n_trials, __ldg(p.offsets), 0);
    lane_start<MODEL, NOISE>(p, L, r, p.offsets ? __ldg(p.offsets + k0) : 0, (uint32_t)k0, 0u);
    if (p.traj_len > 0) p.traj[0] = L.y;
    for (;;) {
        float g[Blk<MODEL, BOUND>::value];
        draw_block<MODEL, BOUND, NOISE>(p, L, r, g);
        const bool live = step_block<MODEL, BOUND, NOISE, true>(p, L, r, g);
        L.blk += 1;
        if (!live) break;
    }
}

// ------------------------------------------------------------------ host side
// What the caller's 0 stands for, by how short of walks the launch is: several
// lanes per walk pay where it holds fewer than the grid has lanes (the walks'
// latency sets the time) and cost throughput beyond.  effective_lanes turns the
// class into lanes.
int auto_lanes_per_walk(int64_t n_walks) {
    if (n_walks <= 0) return 1;
    const double per_lane = (double)n_walks / ((double)sm_count() * 768.0);  // 24 resident warps per SM
    if (per_lane <= 0.25) return 8;
    if (per_lane <= 1.5) return 4;
    if (per_lane <= 4.0) return 2;
    return 1;
}

// The lanes a launch really takes.  Asked for 8, a launch of known size takes 32 or
// 16 as long as the GPU holds all its walks that way.  Asked for 2, it runs one lane
// per walk and hands its last walks over if it has the room for them (left).
// Asked for 4, it does so from 24 walks per resident warp on (85 248 on 148 SMs), where
// both cost the same, and in the ragged layout, whose total the host does not know
// here; below, and without that room, it takes 8 lanes.  Plain DDM, one parameter set, us for 1 / 4 / 8 / 16 / 32 lanes
// (one lane without and with handing over): 1 000 walks 266, 160 / 120 / 78 / 57 /
// 47; 10 000 385, 215 / 175 / 120 / 92 / 106; 30 000 407, 256 / 219 / 161 / 170 /
// 243; 100 000 613, 353 / 360 / 351 / 445 / 721; 300 000 778, 549 / 749 / 904.
static int effective_lanes(int W, int64_t total, bool left) {
    const int64_t warps = (int64_t)sm_count() * 24;
    if (total >= 0) {
        if (W < 8) return (W == 4 && (!left || total <= 24 * warps)) ? 8 : 1;
        return (total <= warps) ? 32 : (total <= 4 * warps) ? 16 : 8;
    }
    return (W == 8 || (W == 4 && !left)) ? 8 : 1;
}

struct Launcher {
    template <int MODEL, int BOUND, bool NOISE>
    static int run(const SingleParams &call, const ssm_launch *opt, cudaStream_t st) {
        int threads = (opt && opt->block_threads > 0) ? opt->block_threads : 256;
        if (threads > 256 || threads % 32) {
            set_error("block_threads must be a multiple of 32 and at most 256");
            return SSM_ERR_ARG;
        }
        constexpr bool WIDE = WideOk<MODEL, NOISE, BOUND>::value;
        int W = (opt && opt->lanes_per_walk > 0) ? opt->lanes_per_walk : 1;
        if (W != 1 && W != 2 && W != 4 && W != 8) {
            set_error("lanes_per_walk must be 0 (automatic), 1, 2, 4 or 8");
            return SSM_ERR_ARG;
        }
        if (W > 1 && !WIDE) {
            set_error("lanes_per_walk > 1 needs the device RNG and a constant, linear or Weibull boundary");
            return SSM_ERR_ARG;
        }
        if (WIDE && call.total >= 0 && !(opt && opt->lanes_per_walk > 0)) W = auto_lanes_per_walk(call.total);
        if (WIDE && W > 1) W = effective_lanes(W, call.total, call.left != nullptr);
        if (W > 1) return wide_launch(MODEL, BOUND, W, call, opt, st);
        SingleParams p = call;
        if (NOISE || BOUND == SSM_BOUND_TABLE) p.left = nullptr;
        auto kern = k_single<MODEL, BOUND, NOISE>;
        int per_sm = 0;
        SSM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, 0));
        if (opt && opt->blocks_per_sm > 0 && opt->blocks_per_sm < per_sm) per_sm = opt->blocks_per_sm;
        if (per_sm < 1) per_sm = 1;
        kern<<<sm_count() * per_sm, threads, 0, st>>>(p);
        SSM_CUDA(cudaGetLastError());
        if (p.left != nullptr) {
            const int rc = wide_finish(MODEL, BOUND, p, st);
            if (rc != SSM_OK) return rc;
        }
        if (!NOISE) {
            // up to 8 CTAs per SM; a known total needs no more than its runs
            int64_t grid = (int64_t)sm_count() * 8;
            if (p.total >= 0) grid = std::min(grid, (p.total + FINISH_RUN - 1) / FINISH_RUN);
            k_finish<MODEL><<<(unsigned)grid, 256, 0, st>>>(p);
            SSM_CUDA(cudaGetLastError());
        }
        if (p.traj && p.traj_len > 0) {
            SingleParams pr = p;  // trial 0 / sample 0, whatever the processing order
            pr.order = nullptr;
            pr.qoff = nullptr;
            k_record<MODEL, BOUND, NOISE><<<1, 128, 0, st>>>(pr);
            SSM_CUDA(cudaGetLastError());
        }
        return SSM_OK;
    }

    template <int MODEL>
    static int dispatch(int bound, bool noise, const SingleParams &p, const ssm_launch *opt,
                        cudaStream_t st) {
        if (MODEL == M_LEGACY) {
            return noise ? run<MODEL, SSM_BOUND_CONSTANT, true>(p, opt, st)
                         : run<MODEL, SSM_BOUND_CONSTANT, false>(p, opt, st);
        }
        switch (bound) {
            case SSM_BOUND_TABLE:
                return noise ? run<MODEL, SSM_BOUND_TABLE, true>(p, opt, st)
                             : run<MODEL, SSM_BOUND_TABLE, false>(p, opt, st);
            case SSM_BOUND_CONSTANT:
                return noise ? run<MODEL, SSM_BOUND_CONSTANT, true>(p, opt, st)
                             : run<MODEL, SSM_BOUND_CONSTANT, false>(p, opt, st);
            case SSM_BOUND_LINEAR:
                return noise ? run<MODEL, SSM_BOUND_LINEAR, true>(p, opt, st)
                             : run<MODEL, SSM_BOUND_LINEAR, false>(p, opt, st);
            case SSM_BOUND_WEIBULL:
                return noise ? run<MODEL, SSM_BOUND_WEIBULL, true>(p, opt, st)
                             : run<MODEL, SSM_BOUND_WEIBULL, false>(p, opt, st);
            default:
                set_error("unknown boundary kind %d", bound);
                return SSM_ERR_ARG;
        }
    }
};

// The header and the rows are needed; with the room for the walks that the
// one-lane kernel leaves (LEAVE_MAX for each of an SM's 64 warps) behind them the
// launch hands its last walks over.
static size_t single_ws_bytes(int64_t n_trials) {
    size_t b = sizeof(WorkspaceHeader) + (size_t)(n_trials > 0 ? n_trials : 0) * sizeof(TrialRow);
    return (b + 255) & ~(size_t)255;
}
static size_t left_bytes() { return (size_t)sm_count() * 64 * LEAVE_MAX * sizeof(LeftWalk); }

struct SingleCall {
    int model;
    const float *v, *a, *z, *alpha, *t, *deadline, *s;
    const float *sv, *sz, *st, *g;
    const float *dtable;
    int64_t dstride, dlen;
    int64_t n_trials, n_samples;
    const int64_t *offsets;
    float max_t;
    const float *maxt_k;
    float dt;
    int bound;
    const float *p1, *p2, *table;
    int64_t tstride, tlen;
    uint64_t seed;
    int smooth;
    const float *noise;
    int64_t nlen;
    const float *nunif;
    float *rts;
    int32_t *choices, *steps;
    float *traj;
    int64_t traj_len;
    const ssm_launch *launch;
    void *ws;
    size_t ws_bytes;
    void *stream;
};

static int run_single(const SingleCall &c) {
    SSM_REQUIRE(c.n_trials >= 0 && c.n_samples >= 0, "n_trials and n_samples must be >= 0");
    SSM_REQUIRE(c.dt > 0.f && isfinite(c.dt), "delta_t must be finite and > 0");
    SSM_REQUIRE(c.maxt_k || (isfinite(c.max_t) && (double)c.max_t / (double)c.dt <= 8388608.0),
                "max_t must be finite with max_t / delta_t <= 2^23");
    SSM_REQUIRE(c.v && c.z && c.t && c.deadline && c.s && c.a, "v, a, z, t, deadline, s are required");
    SSM_REQUIRE((c.rts && c.choices) || (!c.offsets && c.n_trials * c.n_samples == 0),
                "rts and choices outputs are required");
    SSM_REQUIRE(c.model != M_LEVY || c.alpha, "alpha is required for the Levy model");
    SSM_REQUIRE((c.model != M_SDV && c.model != M_FULL) || c.sv, "sv is required");
    SSM_REQUIRE(c.model != M_FULL || (c.sz && c.st), "sz and st are required");
    SSM_REQUIRE(c.model != M_OU || c.g, "g is required for the Ornstein-Uhlenbeck model");
    SSM_REQUIRE(c.model != M_DFLEX || (c.dtable && c.dlen >= 1 && c.dstride >= c.dlen),
                "ddm_flex needs drift_table with drift_stride >= drift_len >= 1");
    if (c.model != M_LEGACY) {
        SSM_REQUIRE(c.bound >= SSM_BOUND_TABLE && c.bound <= SSM_BOUND_WEIBULL, "unknown boundary kind %d", c.bound);
        SSM_REQUIRE(c.bound != SSM_BOUND_LINEAR || c.p1, "linear boundary needs bound_p1");
        SSM_REQUIRE(c.bound != SSM_BOUND_WEIBULL || (c.p1 && c.p2), "weibull boundary needs bound_p1 and bound_p2");
        SSM_REQUIRE(c.bound != SSM_BOUND_TABLE || (c.table && c.tlen >= 1 && c.tstride >= c.tlen),
                    "table boundary needs bound_table with table_stride >= table_len >= 1");
    }
    SSM_REQUIRE(!c.noise || (c.nlen > 0 && c.nunif), "noise_rows needs noise_row_len > 0 and noise_unif");
    SSM_REQUIRE(!c.traj || c.traj_len >= 1, "traj needs traj_len >= 1");
    SSM_REQUIRE(!c.launch || (!c.launch->trial_order == !c.launch->order_offsets),
                "trial_order and order_offsets go together");
    SSM_REQUIRE(!c.launch || !c.launch->trial_order || c.offsets,
                "a trial order needs the ragged layout (sample_offsets)");
    const size_t need = single_ws_bytes(c.n_trials);
    if (!c.ws || c.ws_bytes < need || ((uintptr_t)c.ws & 255u)) {
        set_error("workspace must be 256-byte aligned and hold %zu bytes", need);
        return SSM_ERR_WORKSPACE;
    }
    cudaStream_t st = (cudaStream_t)c.stream;
    WorkspaceHeader *hdr = (WorkspaceHeader *)c.ws;
    TrialRow *rows = (TrialRow *)((char *)c.ws + sizeof(WorkspaceHeader));
    SSM_CUDA(cudaMemsetAsync(hdr, 0, sizeof(WorkspaceHeader), st));
    if (c.n_trials == 0) return SSM_OK;

    PrepArgs A;
    A.v = c.v; A.a = c.a; A.z = c.z; A.t = c.t; A.deadline = c.deadline; A.s = c.s;
    A.alpha = c.alpha; A.p1 = c.p1; A.p2 = c.p2; A.maxt_k = c.maxt_k; A.table = c.table;
    A.sv = c.sv; A.sz = c.sz; A.st = c.st; A.g = c.g;
    A.n_trials = c.n_trials; A.tstride = c.tstride; A.dt = c.dt;
    A.sqrt_dt = (float)sqrt((double)c.dt);  // setup_simulation: sqrt(delta_t) -> float
    A.max_t = c.max_t; A.model = c.model; A.bound = c.bound; A.rows = rows;
    k_prep<<<(unsigned)((c.n_trials + 127) / 128), 128, 0, st>>>(A);
    SSM_CUDA(cudaGetLastError());

    SingleParams p;
    p.key = philox_keys(c.seed);
    p.rows = rows;
    p.offsets = c.offsets;
    p.order = c.offsets && c.launch ? c.launch->trial_order : nullptr;
    p.qoff = p.order ? c.launch->order_offsets : nullptr;
    p.n_trials = c.n_trials;
    p.total = c.offsets ? -1 : c.n_trials * c.n_samples;
    p.k_base = (uint32_t)((c.launch && c.launch->first_trial > 0) ? c.launch->first_trial : 0);
    p.ustride = (c.model == M_FULL) ? 3 : 1;
    p.dtable = c.dtable; p.dstride = c.dstride; p.dlen = c.dlen;
    p.dvec = (c.dtable && ((uintptr_t)c.dtable & 15u) == 0 && (c.dstride & 3) == 0) ? 1 : 0;
    p.dt = c.dt;
    p.smooth = c.smooth ? 1 : 0;
    p.chunk = (c.launch && c.launch->chunk >= 32) ? c.launch->chunk : 64;
    p.refill_min = (c.launch && c.launch->refill_min > 0) ? min(c.launch->refill_min, 32) : SSM_REFILL_MIN;
    p.table = c.table; p.tstride = c.tstride; p.tlen = c.tlen;
    p.noise = c.noise; p.nlen = c.nlen; p.nunif = c.nunif;
    p.rts = c.rts; p.choices = c.choices; p.steps = c.steps;
    p.hdr = hdr;
    p.left = (c.ws_bytes >= need + left_bytes()) ? (LeftWalk *)((char *)c.ws + need) : nullptr;
    p.traj = c.traj; p.traj_len = c.traj_len;
    if (p.total == 0) {
        if (c.traj) {  // nothing simulated: trajectory metadata is all padding
            p.traj_len = c.traj_len;
        }
        return SSM_OK;
    }
    const bool noise = c.noise != nullptr;
    switch (c.model) {
        case M_FLEX: return Launcher::dispatch<M_FLEX>(c.bound, noise, p, c.launch, st);
        case M_LEGACY: return Launcher::dispatch<M_LEGACY>(c.bound, noise, p, c.launch, st);
        case M_SDV: return Launcher::dispatch<M_SDV>(c.bound, noise, p, c.launch, st);
        case M_FULL: return Launcher::dispatch<M_FULL>(c.bound, noise, p, c.launch, st);
        case M_OU: return Launcher::dispatch<M_OU>(c.bound, noise, p, c.launch, st);
        case M_DFLEX: return Launcher::dispatch<M_DFLEX>(c.bound, noise, p, c.launch, st);
        default: return Launcher::dispatch<M_LEVY>(c.bound, noise, p, c.launch, st);
    }
}

}  // namespace ssm

extern "C" {

size_t ssm_ddm_workspace_bytes(int64_t n_trials) { return ssm::single_ws_bytes(n_trials) + ssm::left_bytes(); }
int ssm_auto_lanes_per_walk(int64_t n_walks) { return ssm::auto_lanes_per_walk(n_walks); }

int ssm_ddm_flexbound(const float *v, const float *a, const float *z, const float *t,
                      const float *deadline, const float *s, int64_t n_trials, int64_t n_samples,
                      const int64_t *sample_offsets, float max_t, const float *max_t_per_trial,
                      float delta_t, int bound_kind, const float *bound_p1, const float *bound_p2,
                      const float *bound_table, int64_t table_stride, int64_t table_len,
                      uint64_t seed, int smooth_unif, const float *noise_rows,
                      int64_t noise_row_len, const float *noise_unif, float *rts,
                      int32_t *choices, int32_t *steps, float *traj, int64_t traj_len,
                      const ssm_launch *launch, void *workspace, size_t workspace_bytes,
                      void *stream) {
    ssm::SingleCall c{ssm::M_FLEX, v, a, z, nullptr, t, deadline, s, nullptr, nullptr, nullptr, nullptr, nullptr, 0, 0,
                      n_trials, n_samples,
                      sample_offsets, max_t, max_t_per_trial, delta_t, bound_kind, bound_p1,
                      bound_p2, bound_table, table_stride, table_len, seed, smooth_unif,
                      noise_rows, noise_row_len, noise_unif, rts, choices, steps, traj,
                      traj_len, launch, workspace, workspace_bytes, stream};
    return ssm::run_single(c);
}

int ssm_ddm(const float *v, const float *a, const float *z, const float *t, const float *deadline,
            const float *s, int64_t n_trials, int64_t n_samples, const int64_t *sample_offsets,
            float max_t, float delta_t,
            uint64_t seed, int smooth_unif, const float *noise_rows, int64_t noise_row_len,
            const float *noise_unif, float *rts, int32_t *choices, int32_t *steps, float *traj,
            int64_t traj_len, const ssm_launch *launch, void *workspace, size_t workspace_bytes,
            void *stream) {
    ssm::SingleCall c{ssm::M_LEGACY, v, a, z, nullptr, t, deadline, s, nullptr, nullptr, nullptr, nullptr, nullptr, 0, 0,
                      n_trials, n_samples,
                      sample_offsets, max_t, nullptr, delta_t, SSM_BOUND_CONSTANT, nullptr, nullptr,
                      nullptr, 0, 0, seed, smooth_unif, noise_rows, noise_row_len, noise_unif,
                      rts, choices, steps, traj, traj_len, launch, workspace, workspace_bytes,
                      stream};
    return ssm::run_single(c);
}

int ssm_levy_flexbound(const float *v, const float *a, const float *z, const float *alpha,
                       const float *t, const float *deadline, const float *s, int64_t n_trials,
                       int64_t n_samples, const int64_t *sample_offsets, float max_t,
                       float delta_t, int bound_kind, const float *bound_p1, const float *bound_p2,
                       const float *bound_table, int64_t table_stride, int64_t table_len,
                       uint64_t seed, int smooth_unif, const float *noise_rows,
                       int64_t noise_row_len, const float *noise_unif, float *rts,
                       int32_t *choices, int32_t *steps, float *traj, int64_t traj_len,
                       const ssm_launch *launch, void *workspace, size_t workspace_bytes,
                       void *stream) {
    ssm::SingleCall c{ssm::M_LEVY, v, a, z, alpha, t, deadline, s, nullptr, nullptr, nullptr, nullptr, nullptr, 0, 0,
                      n_trials, n_samples,
                      sample_offsets, max_t, nullptr, delta_t, bound_kind, bound_p1, bound_p2,
                      bound_table, table_stride, table_len, seed, smooth_unif, noise_rows,
                      noise_row_len, noise_unif, rts, choices, steps, traj, traj_len, launch,
                      workspace, workspace_bytes, stream};
    return ssm::run_single(c);
}

int ssm_ddm_sdv(const float *v, const float *a, const float *z, const float *t, const float *sv,
                const float *deadline, const float *s, int64_t n_trials, int64_t n_samples,
                const int64_t *sample_offsets, float max_t, float delta_t, int bound_kind,
                const float *bound_p1, const float *bound_p2, const float *bound_table,
                int64_t table_stride, int64_t table_len, uint64_t seed, int smooth_unif,
                const float *noise_rows, int64_t noise_row_len, const float *noise_unif, float *rts,
                int32_t *choices, int32_t *steps, float *traj, int64_t traj_len,
                const ssm_launch *launch, void *workspace, size_t workspace_bytes, void *stream) {
    ssm::SingleCall c{ssm::M_SDV, v, a, z, nullptr, t, deadline, s, sv, nullptr, nullptr, nullptr, nullptr, 0, 0,
                      n_trials, n_samples, sample_offsets, max_t, nullptr, delta_t, bound_kind,
                      bound_p1, bound_p2, bound_table, table_stride, table_len, seed, smooth_unif,
                      noise_rows, noise_row_len, noise_unif, rts, choices, steps, traj, traj_len,
                      launch, workspace, workspace_bytes, stream};
    return ssm::run_single(c);
}

int ssm_full_ddm(const float *v, const float *a, const float *z, const float *t, const float *sz,
                 const float *sv, const float *st, const float *deadline, const float *s,
                 int64_t n_trials, int64_t n_samples, const int64_t *sample_offsets, float max_t,
                 float delta_t, int bound_kind, const float *bound_p1, const float *bound_p2,
                 const float *bound_table, int64_t table_stride, int64_t table_len, uint64_t seed,
                 int smooth_unif, const float *noise_rows, int64_t noise_row_len,
                 const float *noise_unif, float *rts, int32_t *choices, int32_t *steps, float *traj,
                 int64_t traj_len, const ssm_launch *launch, void *workspace,
                 size_t workspace_bytes, void *stream) {
    ssm::SingleCall c{ssm::M_FULL, v, a, z, nullptr, t, deadline, s, sv, sz, st, nullptr, nullptr, 0, 0,
                      n_trials, n_samples, sample_offsets, max_t, nullptr, delta_t, bound_kind,
                      bound_p1, bound_p2, bound_table, table_stride, table_len, seed, smooth_unif,
                      noise_rows, noise_row_len, noise_unif, rts, choices, steps, traj, traj_len,
                      launch, workspace, workspace_bytes, stream};
    return ssm::run_single(c);
}

int ssm_ornstein_uhlenbeck(const float *v, const float *a, const float *z, const float *g,
                           const float *t, const float *deadline, const float *s, int64_t n_trials,
                           int64_t n_samples, const int64_t *sample_offsets, float max_t,
                           float delta_t, int bound_kind, const float *bound_p1,
                           const float *bound_p2, const float *bound_table, int64_t table_stride,
                           int64_t table_len, uint64_t seed, int smooth_unif,
                           const float *noise_rows, int64_t noise_row_len, const float *noise_unif,
                           float *rts, int32_t *choices, int32_t *steps, float *traj,
                           int64_t traj_len, const ssm_launch *launch, void *workspace,
                           size_t workspace_bytes, void *stream) {
    ssm::SingleCall c{ssm::M_OU, v, a, z, nullptr, t, deadline, s, nullptr, nullptr, nullptr, g, nullptr, 0, 0,
                      n_trials, n_samples, sample_offsets, max_t, nullptr, delta_t, bound_kind,
                      bound_p1, bound_p2, bound_table, table_stride, table_len, seed, smooth_unif,
                      noise_rows, noise_row_len, noise_unif, rts, choices, steps, traj, traj_len,
                      launch, workspace, workspace_bytes, stream};
    return ssm::run_single(c);
}

int ssm_ddm_flex(const float *v, const float *a, const float *z, const float *t, const float *deadline,
                 const float *s, int64_t n_trials, int64_t n_samples, const int64_t *sample_offsets,
                 float max_t, float delta_t, int bound_kind, const float *bound_p1,
                 const float *bound_p2, const float *bound_table, int64_t table_stride,
                 int64_t table_len, const float *drift_table, int64_t drift_stride, int64_t drift_len,
                 uint64_t seed, int smooth_unif, const float *noise_rows, int64_t noise_row_len,
                 const float *noise_unif, float *rts, int32_t *choices, int32_t *steps, float *traj,
                 int64_t traj_len, const ssm_launch *launch, void *workspace,
                 size_t workspace_bytes, void *stream) {
    ssm::SingleCall c{ssm::M_DFLEX, v, a, z, nullptr, t, deadline, s, nullptr, nullptr, nullptr, nullptr,
                      drift_table, drift_stride, drift_len, n_trials, n_samples, sample_offsets, max_t,
                      nullptr, delta_t, bound_kind, bound_p1, bound_p2, bound_table, table_stride,
                      table_len, seed, smooth_unif, noise_rows, noise_row_len, noise_unif, rts, choices,
                      steps, traj, traj_len, launch, workspace, workspace_bytes, stream};
    return ssm::run_single(c);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free variant.  Its scratch is this file-scope device array; host
// code must not hand the symbol itself to a kernel (in host code it names a
// host-side stand-in), so the device address is looked up with the device
// current and cached per device together with the unique id of the CUDA
// context it was looked up in.  A call under another context of that device
// (after cudaDeviceReset, or a primary-context reset) looks the address up
// again instead of reusing one from a context that no longer exists.
namespace ssm {
static __device__ __align__(256) unsigned char g_static_ws[SSM_STATIC_WS_BYTES];
static std::mutex g_static_mu;
struct StaticSlot {
    unsigned long long ctx_id;  // 0: not looked up yet
    void *ptr;
};
static StaticSlot g_static_slot[64] = {};

using PfnCtxGetCurrent = CUresult (*)(CUcontext *);
using PfnCtxGetId = CUresult (*)(CUcontext, unsigned long long *);

// Unique id of the calling thread's current CUDA context (cuCtxGetId, CUDA
// 12.0+, reached through the runtime's driver entry points); 0 when no context
// is current or the driver does not offer the query.  Called under g_static_mu.
static unsigned long long current_context_id() {
    static bool resolved = false;
    static PfnCtxGetCurrent get_current = nullptr;
    static PfnCtxGetId get_id = nullptr;
    if (!resolved) {
        resolved = true;
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) ==
                cudaSuccess && q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<PfnCtxGetCurrent>(f);
        f = nullptr;
        q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<PfnCtxGetId>(f);
    }
    if (get_current == nullptr || get_id == nullptr) return 0;
    CUcontext ctx = nullptr;
    if (get_current(&ctx) != CUDA_SUCCESS || ctx == nullptr) return 0;
    unsigned long long id = 0;
    return get_id(ctx, &id) == CUDA_SUCCESS ? id : 0;
}

static int static_workspace(void **out) {
    int dev = 0;
    SSM_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_error("device ordinal %d out of range for the static workspace", dev);
        return SSM_ERR_ARG;
    }
    std::lock_guard<std::mutex> lock(g_static_mu);
    StaticSlot &slot = g_static_slot[dev];
    const unsigned long long id = current_context_id();
    if (slot.ctx_id == 0 || id != slot.ctx_id) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_static_ws);  // makes the device's context current
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_static_ws)");
        slot.ptr = p;
        slot.ctx_id = current_context_id();
    }
    *out = slot.ptr;
    return SSM_OK;
}
}  // namespace ssm

extern "C" int ssm_ddm_flexbound_static(
    const float *v, const float *a, const float *z, const float *t, const float *deadline,
    const float *s, int64_t n_trials, int64_t n_samples, const int64_t *sample_offsets,
    float max_t, const float *max_t_per_trial, float delta_t, int bound_kind,
    const float *bound_p1, const float *bound_p2, const float *bound_table, int64_t table_stride,
    int64_t table_len, uint64_t seed, int smooth_unif, const float *noise_rows,
    int64_t noise_row_len, const float *noise_unif, float *rts, int32_t *choices, int32_t *steps,
    float *traj, int64_t traj_len, const ssm_launch *launch, void *stream) {
    if (n_trials > SSM_STATIC_MAX_TRIALS) {
        ssm::set_error("ssm_ddm_flexbound_static supports at most %d trials (got %lld); "
                       "use ssm_ddm_flexbound with a caller workspace",
                       SSM_STATIC_MAX_TRIALS, (long long)n_trials);
        return SSM_ERR_ARG;
    }
    void *ws = nullptr;
    const int st = ssm::static_workspace(&ws);
    if (st != SSM_OK) return st;
    return ssm_ddm_flexbound(v, a, z, t, deadline, s, n_trials, n_samples, sample_offsets, max_t,
                             max_t_per_trial, delta_t, bound_kind, bound_p1, bound_p2,
                             bound_table, table_stride, table_len, seed, smooth_unif, noise_rows,
                             noise_row_len, noise_unif, rts, choices, steps, traj, traj_len,
                             launch, ws, SSM_STATIC_WS_BYTES, stream);
}

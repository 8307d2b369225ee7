// Single-accumulator simulators with W = 8, 16 or 32 lanes per walk, for launches
// with fewer walks than the GPU has lanes, and for the last walks of larger ones:
// they last as long as their longest walk, so what counts is the time of one
// walk's step.
//
// A walk's floating-point sum has to be taken in order (results are those of one
// lane per walk, bit for bit), so a step costs at least one dependent addition,
// four cycles.  Everything else is kept off that chain.  A block is 18 W steps
// in W segments of 18:
//  * lane s of the group draws segment s's increments (three Philox calls with
//    the counters the one-lane mode uses for those steps) and leaves them in
//    shared memory, for the block after the one being stepped, so the
//    draws fill the chain's idle issue slots;
//  * every lane adds up all 18 W increments, untested, and keeps the sum at the
//    start of its own segment;
//  * every lane then tests the 18 steps of its own segment, all segments at once.
//    The walk ends in the first segment with a failed test; that lane's count
//    and position are the walk's.
// The time needs no sum: inside one binade of the float accumulator every
// addition of dt adds the same amount (see TimeSteps).  A warp whose walks reach
// a time limit or a binade's end within the block sums the time, too.
//
// The version before this one stepped and tested in order on every lane, each
// increment broadcast by a shuffle.  Plain DDM, one parameter set, us before (8
// lanes) and now: 100 walks 82 -> 35 (32 lanes), 1 000 113 -> 47 (32), 10 000 187 -> 92
// (16), 30 000 239 -> 161 (8); 500 angle parameter sets, one walk each, 157 -> 57 (32).
#include <algorithm>

#include "sim_single.cuh"

namespace ssm {
namespace {

// Steps per segment: three Philox calls of six increments, or (Levy) eight calls
// of two.
template <int MODEL> struct Seg { static constexpr int value = (MODEL == M_LEVY) ? 16 : 18; };
constexpr int SEG_STRIDE = 20;  // floats between segments in shared memory: 16-byte rows, no bank conflicts
constexpr int WIDE_WARPS = 8;

// The float32 time accumulator t = dt + dt + ... (an even number of additions) after n
// more of them.  Inside one binade, of ulp u, an addition moves it by dt rounded to a
// multiple of u, the same every time unless dt is an odd multiple of u / 2: then
// each addition is a tie with an even result, so the amount is the same from an
// even accumulator on.  next = RN(t + dt) is even in that case: if t lies in the same
// binade, it is such a result; if t lies below, all additions so far were exact (dt
// is a multiple of every smaller ulp), t + dt = (k + 1) dt after k of them, and with
// k even this is an odd multiple of u / 2, a tie again.  (With k odd it could be exact
// and odd, and the additions after the first would differ: k = 1 049, dt =
// 15979 / 2^24.)  So next and inc = RN(next + dt) - next are exact values, and after
// n >= 1 additions the accumulator is next + (n - 1) inc exactly, as long as that
// stays in next's binade.  Walks start at step 0, are handed over after whole blocks of
// the one-lane mode and advance by whole blocks here: all even (asserted).
struct TimeSteps {
    float t, next, inc;
    __device__ __forceinline__ TimeSteps(float t0, float dt) : t(t0) {
        next = __fadd_rn(t0, dt);
        inc = __fsub_rn(__fadd_rn(next, dt), next);
    }
    __device__ __forceinline__ float after(int n) const { return n == 0 ? t : fmaf((float)(n - 1), inc, next); }
    __device__ __forceinline__ bool uniform(int n) const {  // n additions stay in one binade
        return (__float_as_uint(next) >> 23) == (__float_as_uint(after(n)) >> 23);
    }
};

// Increments of the segment that starts at step ix0 (whole segments from a block's
// start, which is a multiple of the one-lane mode's block).
template <int MODEL>
__device__ __forceinline__ void draw_segment(const SingleParams &p, const Lane &L, const TrialRow &r, uint32_t ix0,
                                             float (&g)[Seg<MODEL>::value]) {
    const uint32_t k = L.k + p.k_base;
    if constexpr (MODEL == M_LEVY) {
#pragma unroll
        for (int h = 0; h < 8; ++h) {  // calls count in groups of four (eight steps)
            const uint4 b = philox10(make_uint4(ix0 / 8u + (uint32_t)(h / 4), L.n, k, 2u + (uint32_t)(h % 4)), p.key);
            float x0, x1;
            cms_stable2(b, r, x0, x1);
            g[2 * h] = fmaf(r.scale, x0, r.drift);
            g[2 * h + 1] = fmaf(r.scale, x1, r.drift);
        }
    } else {
        const float drift = (MODEL == M_DFLEX) ? 0.f : (DrawnDrift<MODEL>::value ? L.dinc : r.drift);
        const uint32_t ctr = ix0 / 6u;
        const uint4 b0 = philox10(make_uint4(ctr, L.n, k, 0u), p.key);
        const uint4 b1 = philox10(make_uint4(ctr + 1u, L.n, k, 0u), p.key);
        const uint4 b2 = philox10(make_uint4(ctr + 2u, L.n, k, 0u), p.key);
        bm12_increment(b0, b1, r.c2, drift, g);
        bm6_increment(b2, r.c2, drift, g + 12);
        if constexpr (MODEL == M_DFLEX) {  // + v(t_ix) dt; past the table's end the last entry repeats
            const float *row = p.dtable + (int64_t)(L.k == NO_TRIAL ? 0u : L.k) * p.dstride;
#pragma unroll
            for (int j = 0; j < 18; ++j) {
                const int64_t ix = min((int64_t)ix0 + j, p.dlen - 1);
                g[j] = fmaf(__ldg(row + ix), p.dt, g[j]);
            }
        }
    }
}

template <int N>
__device__ __forceinline__ void store_segment(float *own, const float (&g)[N]) {
#pragma unroll
    for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4 *>(own + j) = make_float4(g[j], g[j + 1], g[j + 2], g[j + 3]);
    if constexpr (N == 18) *reinterpret_cast<float2 *>(own + 16) = make_float2(g[16], g[17]);
}
template <int N>
__device__ __forceinline__ void load_segment(const float *seg, float (&g)[N]) {
#pragma unroll
    for (int j = 0; j < 16; j += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(seg + j);
        g[j] = v.x; g[j + 1] = v.y; g[j + 2] = v.z; g[j + 3] = v.w;
    }
    if constexpr (N == 18) {
        const float2 v = *reinterpret_cast<const float2 *>(seg + 16);
        g[16] = v.x; g[17] = v.y;
    }
}

template <int MODEL>
__device__ __forceinline__ float step_y(float y, float g, const TrialRow &r) {
    return (MODEL == M_OU) ? fmaf(y, r.expo, g) : y + g;  // y (1 - g dt) + v dt + noise
}
template <int MODEL>
__device__ __forceinline__ bool holds(float y, float b) {
    return (MODEL == M_LEGACY) ? (y <= b && y >= 0.f) : (fabsf(y) <= b);
}

// Bounds of a segment's steps from step ix0 on, as the one-lane mode evaluates
// them: a linear bound from its bases every 36 steps (two segments; odd: the
// second), Levy's every eight.
template <int MODEL, int BOUND>
__device__ __forceinline__ void segment_bounds(const SingleParams &p, const TrialRow &r, float ix0, bool odd,
                                               float (&b)[Seg<MODEL>::value]) {
    constexpr int SEG = Seg<MODEL>::value;
    const float off = (MODEL != M_LEVY && odd) ? 18.f : 0.f;
    float base = 0.f;
#pragma unroll
    for (int j = 0; j < SEG; ++j) {
        const int q = (MODEL == M_LEVY) ? j % 8 : j;
        if (BOUND == SSM_BOUND_LINEAR && q == 0) base = fmaf(ix0 + (float)j - off, r.dtp1, r.a);
        if (MODEL == M_LEGACY || BOUND == SSM_BOUND_CONSTANT) b[j] = r.a;
        else if (BOUND == SSM_BOUND_LINEAR) b[j] = (q == 0 && off == 0.f) ? base : fmaf(off + (float)q, r.dtp1, base);
        else b[j] = bound_at<BOUND, false>(r, ix0 + (float)j, 0, p, 0);
    }
}

// y (and with TIME the accumulator) over a whole block of the group at `seg`:
// the sums at its end and at the start of the lane's own segment.
template <int MODEL, int W, bool TIME>
__device__ __forceinline__ void sum_block(const float *seg, const TrialRow &r, float dt, int sub, float y0, float t0,
                                          float &y_end, float &t_end, float &y_own, float &t_own) {
    constexpr int SEG = Seg<MODEL>::value;
    float y = y0, t = t0;
    y_own = y0;
    t_own = t0;
#pragma unroll 4
    for (int s = 0; s < W; ++s) {
        if (s > 0) {
            y_own = (sub == s) ? y : y_own;
            if (TIME) t_own = (sub == s) ? t : t_own;
        }
        float g[SEG];
        load_segment(seg + s * SEG_STRIDE, g);
#pragma unroll
        for (int j = 0; j < SEG; ++j) {
            y = step_y<MODEL>(y, g[j], r);
            if (TIME) t = __fadd_rn(t, dt);
        }
    }
    y_end = y;
    t_end = t;
}

// Trial 0 / sample 0's path (metadata['trajectory'], -999 padded:
// ddm_models.pyx:714-728) by one CTA, its first warp stepping the walk.
template <int MODEL, int BOUND>
__device__ void record_path(const SingleParams &p, float *buf) {
    constexpr int W = 32, SEG = Seg<MODEL>::value;
    constexpr unsigned FULL = 0xffffffffu;
    for (int64_t i = threadIdx.x; i < p.traj_len; i += blockDim.x) p.traj[i] = -999.f;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int sub = threadIdx.x;
    Lane L;
    TrialRow r = {};
    L.k = NO_TRIAL;
    L.dinc = 0.f;
    int64_t k0 = 0;
    if (p.offsets != nullptr) k0 = ragged_find(p.offsets, p.n_trials, __ldg(p.offsets), 0);
    lane_start<MODEL, false>(p, L, r, p.offsets ? __ldg(p.offsets + k0) : 0, (uint32_t)k0, 0u);
    if (sub == 0) p.traj[0] = L.y;
    for (uint32_t blk = 0;; ++blk) {
        if (L.ixf >= r.capf) {
            if (sub == 0) raise_error(p.hdr, SSM_ERR_DEVICE, (int)L.w);
            break;
        }
        float g[SEG];
        draw_segment<MODEL>(p, L, r, blk * (uint32_t)(SEG * W) + (uint32_t)(SEG * sub), g);
        __syncwarp();
        store_segment(buf + sub * SEG_STRIDE, g);
        __syncwarp();
        float y_end, t_end, y, t;
        sum_block<MODEL, W, true>(buf, r, p.dt, sub, L.y, L.tp, y_end, t_end, y, t);
        const int64_t ix0 = (int64_t)blk * (SEG * W) + SEG * sub;
        const float y_own = y;
        int c = 0;
        bool live = true;
#pragma unroll
        for (int j = 0; j < SEG; ++j) {
            // the recorder's bound at a step, not the block-based one
            const float b = (MODEL == M_LEGACY) ? r.a : bound_at<BOUND, false>(r, (float)(ix0 + j), 0, p, L.k);
            live = live && holds<MODEL>(y, b) && (t <= r.dl_tmp);
            if (live) {
                y = step_y<MODEL>(y, g[j], r);
                t = __fadd_rn(t, p.dt);
                c += 1;
            }
        }
        const unsigned ended = __ballot_sync(FULL, !live);
        const int first = ended ? __ffs(ended) - 1 : W;
        const int mine = (sub < first) ? SEG : (sub == first) ? c : 0;
        y = y_own;
#pragma unroll
        for (int j = 0; j < SEG; ++j) {
            y = step_y<MODEL>(y, g[j], r);
            if (j < mine && ix0 + j + 1 < p.traj_len) p.traj[ix0 + j + 1] = y;
        }
        if (ended) break;
        L.y = y_end;
        L.tp = t_end;
        L.ixf += (float)(SEG * W);
    }
}

template <int MODEL, int BOUND, int W>
__global__ void __launch_bounds__(32 * WIDE_WARPS, 2) k_wide(const __grid_constant__ SingleParams p) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int SEG = Seg<MODEL>::value, BLK = SEG * W;
    static_assert(BLK % 2 == 0, "TimeSteps: a block starts at an even step");
    __shared__ __align__(16) float shared[WIDE_WARPS][32 * SEG_STRIDE];
    if constexpr (WideOk<MODEL, false, BOUND>::value) {
        if (p.traj != nullptr && blockIdx.x == gridDim.x - 1) {
            record_path<MODEL, BOUND>(p, shared[0]);
            return;
        }
    }
    const int lane = threadIdx.x & 31;
    const int sub = lane & (W - 1);              // place in the group
    const int src0 = lane - sub;                 // the group's first lane
    const unsigned lt_mask = (1u << src0) - 1u;  // lanes of the groups before this one
    const unsigned group = (W == 32) ? FULL : ((1u << (W & 31)) - 1u) << src0;
    float *buf = shared[threadIdx.x >> 5];
    float *own = buf + lane * SEG_STRIDE;
    const float *seg = buf + src0 * SEG_STRIDE;
    const bool left = (p.left != nullptr);  // continue the walks that k_single left
    unsigned long long *counter = left ? &p.hdr->aux[1] : &p.hdr->counter;
    const int64_t total = left           ? (int64_t)p.hdr->aux[0]
                          : p.total >= 0 ? p.total
                                         : __ldg(p.offsets + p.n_trials) - __ldg(p.offsets);

    Lane L;
    TrialRow r = {};
    L.w = 0; L.k = NO_TRIAL; L.n = 0; L.blk = 0; L.ix = 0; L.y = L.tp = L.ixf = L.dinc = L.tpb = 0.f;
    bool active = false;
    bool primed = false;   // the group's segments hold the walk's next block
    bool pending = false;  // walk ended, result not yet written
    bool exhausted = false;
    int64_t hint = 0;
    for (;;) {
        // a group restarts as soon as its walk has ended (or refill_min of them have)
        const unsigned need = __ballot_sync(FULL, !active);
        const int cnt = __popc(need) / W;
        const bool pass = exhausted ? (__ballot_sync(FULL, pending) != 0u) : (cnt >= p.refill_min);
        if (pass && pending) {
            // a left walk's rt is k_finish's, as those of the launch that left it
            const float rt = left ? L.tp : finish_rt<MODEL, false>(p, L.k, L.n, L.w, L.tp);
            if (sub == 0) {
                p.rts[L.w] = rt;
                p.choices[L.w] = (L.y > 0.f) - (L.y < 0.f);  // sign(y)
                if (p.steps) p.steps[L.w] = (int)L.ixf;
            }
            pending = false;
        }
        if (pass && !exhausted) {
            unsigned long long b = 0ull;
            if (lane == 0) b = atomicAdd(counter, (unsigned long long)cnt);
            const int64_t base = (int64_t)__shfl_sync(FULL, b, 0);
            if ((uint64_t)(base + cnt) >= (uint64_t)total) exhausted = true;
            const int64_t w = base + __popc(need & lt_mask) / W;
            if (!active && w < total) {
                if (left) {
                    const LeftWalk o = p.left[w];
                    lane_start<MODEL, false>(p, L, r, o.w, o.k, o.n);
                    L.y = o.y; L.tp = o.tp; L.ixf = o.ixf; L.dinc = o.dinc;
                    active = true;
                } else if (p.offsets == nullptr) {
                    uint32_t k, n;
                    layout_trial(p, w, k, n);
                    lane_start<MODEL, false>(p, L, r, w, k, n);
                    active = true;
                } else {
                    Span sp;
                    if (find_span(p, w, hint, sp)) {
                        const int64_t n = w - sp.lo;
                        lane_start<MODEL, false>(p, L, r, sp.out0 + n, sp.k, (uint32_t)n);
                        active = true;
                    }
                }
                primed = false;
            }
        }
        if (__ballot_sync(FULL, active) == 0u) break;

        // next block's increments, independent of the sums below
        float g[SEG];
        draw_segment<MODEL>(p, L, r, (uint32_t)L.ixf + (uint32_t)((primed ? BLK : 0) + SEG * sub), g);

        bool go = active && primed;
        bool ended = false;
        if (go && L.ixf >= r.capf) {
            raise_error(p.hdr, SSM_ERR_DEVICE, (int)L.w);
            go = false;
            ended = true;
        }
        const TimeSteps ts(L.tp, p.dt);
        // no step of the block can pass the time limit: dl lies past the block's end
        // with room for the accumulator's rounding (2 dt per 64 steps below 65536 dt)
        constexpr float SPAN = (float)(BLK + 1 + 2 * (BLK / 64));
        const bool plain = (L.tp < p.dt * 65536.f) && (fmaf(SPAN, p.dt, L.tp) <= r.dl_tmp) && ts.uniform(BLK);
        const bool fast = __all_sync(FULL, !go || plain);
        float y_end, t_end, y_own, t_own;
        if (fast) sum_block<MODEL, W, false>(seg, r, p.dt, sub, L.y, L.tp, y_end, t_end, y_own, t_own);
        else sum_block<MODEL, W, true>(seg, r, p.dt, sub, L.y, L.tp, y_end, t_end, y_own, t_own);
        if (fast) t_end = ts.after(BLK);

        // this lane's segment, tested
        float e[SEG], bnd[SEG];
        load_segment(own, e);
        segment_bounds<MODEL, BOUND>(p, r, L.ixf + (float)(SEG * sub), sub & 1, bnd);
        bool ok = true;
        {
            float y = y_own, t = t_own;
#pragma unroll
            for (int j = 0; j < SEG; ++j) {
                ok = ok && holds<MODEL>(y, bnd[j]);
                y = step_y<MODEL>(y, e[j], r);
                if (!fast) {
                    ok = ok && (t <= r.dl_tmp);
                    t = __fadd_rn(t, p.dt);
                }
            }
        }
        const unsigned failed = __ballot_sync(FULL, go && !ok);
        if (failed != 0u) {  // once per walk: where in the segment
            float y = y_own, t = t_own;
            int c = 0;
            bool live = true;
#pragma unroll
            for (int j = 0; j < SEG; ++j) {
                live = live && holds<MODEL>(y, bnd[j]) && (fast || t <= r.dl_tmp);
                if (live) {
                    y = step_y<MODEL>(y, e[j], r);
                    t = __fadd_rn(t, p.dt);
                    c += 1;
                }
            }
            const unsigned mine = failed & group;
            const int src = mine ? __ffs(mine) - 1 : lane;
            const float y_x = __shfl_sync(FULL, y, src), t_x = __shfl_sync(FULL, t, src);
            const int c_x = __shfl_sync(FULL, c, src);
            if (mine) {
                const int n = SEG * (src - src0) + c_x;
                y_end = y_x;
                t_end = fast ? ts.after(n) : t_x;
                L.ixf += (float)n;
                ended = true;
            }
        }
        __syncwarp();
        store_segment(own, g);
        __syncwarp();
        if (active) {
            if (go) {
                L.y = y_end;
                L.tp = t_end;
                if (!ended) L.ixf += (float)BLK;
            }
            primed = true;
            if (ended) {
                active = false;
                pending = true;
            }
        }
    }
}

template <int MODEL, int BOUND, int W>
int launch(const SingleParams &p, const ssm_launch *opt, cudaStream_t st) {
    auto kern = k_wide<MODEL, BOUND, W>;
    const int threads = (opt && opt->block_threads > 0) ? opt->block_threads : 256;
    int per_sm = 0;
    SSM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, 0));
    if (opt && opt->blocks_per_sm > 0 && opt->blocks_per_sm < per_sm) per_sm = opt->blocks_per_sm;
    if (per_sm < 1) per_sm = 1;
    SingleParams q = p;
    q.refill_min = (opt && opt->refill_min > 0) ? std::min(opt->refill_min, 32 / W) : 1;
    int64_t grid = (int64_t)sm_count() * per_sm;
    if (p.total >= 0) {  // no more CTAs than walks need, spread over the SMs first
        const int64_t per_cta = (int64_t)(threads / 32) * (32 / W);
        grid = std::min(grid, std::max<int64_t>(1, (p.total + per_cta - 1) / per_cta));
    }
    const bool record = p.traj != nullptr && p.traj_len > 0;
    if (!record) q.traj = nullptr;
    kern<<<(unsigned)(grid + (record ? 1 : 0)), threads, 0, st>>>(q);
    SSM_CUDA(cudaGetLastError());
    return SSM_OK;
}

// The left walks, eight lanes each: at most LEAVE_MAX of each warp's 32, which is
// half of k_single's lanes and six times the groups of this grid; groups that are
// done take the next ones from the queue.
template <int MODEL, int BOUND>
int finish(const SingleParams &p, cudaStream_t st) {
    auto kern = k_wide<MODEL, BOUND, 8>;
    SingleParams q = p;
    q.refill_min = 1;
    q.traj = nullptr;
    kern<<<(unsigned)(sm_count() * 2), 32 * WIDE_WARPS, 0, st>>>(q);
    SSM_CUDA(cudaGetLastError());
    return SSM_OK;
}

template <int MODEL, int BOUND>
int pick_width(int W, const SingleParams &p, const ssm_launch *opt, cudaStream_t st) {
    if (W == 0) return finish<MODEL, BOUND>(p, st);
    if constexpr (WideOk<MODEL, false, BOUND>::value) {
        switch (W) {
            case 8: return launch<MODEL, BOUND, 8>(p, opt, st);
            case 16: return launch<MODEL, BOUND, 16>(p, opt, st);
            default: return launch<MODEL, BOUND, 32>(p, opt, st);
        }
    }
    set_error("no lanes-per-walk kernel for this model");
    return SSM_ERR_ARG;
}

template <int MODEL>
int pick_bound(int bound, int W, const SingleParams &p, const ssm_launch *opt, cudaStream_t st) {
    if constexpr (MODEL == M_LEGACY) {
        return pick_width<MODEL, SSM_BOUND_CONSTANT>(W, p, opt, st);
    } else {
        switch (bound) {
            case SSM_BOUND_CONSTANT: return pick_width<MODEL, SSM_BOUND_CONSTANT>(W, p, opt, st);
            case SSM_BOUND_LINEAR: return pick_width<MODEL, SSM_BOUND_LINEAR>(W, p, opt, st);
            default: return pick_width<MODEL, SSM_BOUND_WEIBULL>(W, p, opt, st);
        }
    }
}

int pick_model(int model, int bound, int W, const SingleParams &p, const ssm_launch *opt, cudaStream_t st) {
    switch (model) {
        case M_LEGACY: return pick_bound<M_LEGACY>(bound, W, p, opt, st);
        case M_SDV: return pick_bound<M_SDV>(bound, W, p, opt, st);
        case M_FULL: return pick_bound<M_FULL>(bound, W, p, opt, st);
        case M_OU: return pick_bound<M_OU>(bound, W, p, opt, st);
        case M_DFLEX: return pick_bound<M_DFLEX>(bound, W, p, opt, st);
        case M_LEVY: return pick_bound<M_LEVY>(bound, W, p, opt, st);
        default: return pick_bound<M_FLEX>(bound, W, p, opt, st);
    }
}

}  // namespace

int wide_launch(int model, int bound, int W, const SingleParams &p, const ssm_launch *opt, cudaStream_t st) {
    SingleParams q = p;
    q.left = nullptr;
    return pick_model(model, bound, W, q, opt, st);
}

int wide_finish(int model, int bound, const SingleParams &p, cudaStream_t st) {
    return pick_model(model, bound, 0, p, nullptr, st);
}

}  // namespace ssm

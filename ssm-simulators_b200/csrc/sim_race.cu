// Multi-accumulator Euler-Maruyama simulators for sm_100a: the race model
// (cssm.race_model, src/cssm/race_models.pyx:356-506) and the leaky competing
// accumulator (cssm.lca, race_models.pyx:757-920).
//
// One thread per trajectory, persistent grid, warps refill finished lanes from a
// global work counter.  The NP accumulators of a trajectory live in registers.
// Each step tests the reference's loop condition (no accumulator above b(t) and
// t <= min(max_t, deadline - t_nd)), then updates every accumulator with its
// own N(0,1) increment and clips it at 0.  Choices are argmax (first maximum).
// Noise injection reads caller rows (draw index step * NP + j) and evaluates
// every float operation with explicit rounding in the reference's order.
//
// With the device RNG and up to four accumulators (k_race_window) a walk goes
// through windows of 24 increments, four Philox calls.  A window costs about 440
// instructions, 430 of them the draws and the bare steps: 24 of them would be
// needed for each accumulator's tests, so a window runs without tests and is
// taken again, step by step, only by the walks that may end in it (one window in
// 120 on the LCA sets).  Time per window and scheduler is 680 cycles, of which
// the SFU is busy 390.  Measured per launch, ms, 512 sets of 10 000 walks with
// tests in every step, before and now: LCA (4 accumulators) 22.8 -> 15.3, racing
// diffusion (3) 12.8 -> 9.8, race with a collapsing bound (4; 190 steps a walk, so
// half of a warp's windows have a walk that ends) 5.6 -> 5.4.
#include "common.cuh"

namespace ssm {

constexpr int RACE_MAX_NP = 16;

// Simulator families sharing this kernel: the race model, the LCA and the
// racing diffusion model (racing_diffusion_model, race_models.pyx:1150-1266:
// starts U(0, A), no lower barrier, the first accumulator at or above b wins
// and the step that reaches it does not advance the time).
enum RaceFamily { FAM_RACE = 0, FAM_LCA = 1, FAM_RDM = 2 };

// Per-trial header (64 B) followed by v[np], sq[np] (= sqrt(dt)*s), z[np]
// padded to a multiple of 4 floats.
struct alignas(16) RaceHead {
    float t, deadline, dl_tmp, a;
    float p1, dtp1, inv_beta, capf;
    float g, b, y0scale, pad0;   // y0scale = b(0): start p_j = z_j * b(0)
    float pad[4];
};
static_assert(sizeof(RaceHead) == 64, "RaceHead is one 64-byte line");

__host__ __device__ inline int64_t race_row_floats(int np) {
    return 16 + ((3 * (int64_t)np + 3) / 4) * 4;
}

struct RaceParams {
    PhiloxKeys key;
    const float *rows;
    int64_t row_floats;
    const int64_t *offsets;
    const int32_t *order;     // ragged only: trial simulated j-th (nullptr = index order)
    const int64_t *qoff;      // prefix sums of the sample counts in that order
    int64_t n_trials, total;  // total -1: offsets[n_trials] - offsets[0]
    uint32_t k_base;          // random-stream index of trial 0 (trial windows of a larger batch)
    int np;
    float dt;
    int smooth, chunk;
    int refill_min;           // ended walks a warp collects before it restarts lanes
    const float *table;
    int64_t tstride, tlen;
    const float *noise;
    int64_t nlen;
    const float *nunif;
    float *rts;
    int32_t *choices, *steps;
    WorkspaceHeader *hdr;
    float *traj;
    int64_t traj_len;
};

struct RacePrep {
    const float *v, *z, *t, *s, *deadline, *a, *p1, *p2, *g, *b, *table;
    int per_trial_zs;  // rdm: z (the start range A) and s hold one value per trial
    int64_t n_trials, tstride, row_floats;
    int np, bound;
    float dt, sqrt_dt, max_t;
    float *rows;
};

__global__ void k_race_prep(const RacePrep A) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= A.n_trials) return;
    float *row = A.rows + k * A.row_floats;
    RaceHead h;
    const float dt = A.dt;
    h.t = A.t[k];
    h.deadline = A.deadline[k];
    const float dl = __fsub_rn(h.deadline, h.t);
    h.dl_tmp = (dl < A.max_t) ? dl : A.max_t;  // compute_deadline_tmp (_utils.pyx:712-718)
    h.a = A.a ? A.a[k] : 0.f;
    h.p1 = A.p1 ? A.p1[k] : 0.f;
    h.dtp1 = dt * h.p1;
    h.inv_beta = 1.0f / (A.p2 ? A.p2[k] : 1.f);
    const double nsteps = (double)h.dl_tmp / (double)dt;
    if (!(nsteps > 0.0)) h.capf = 64.f;
    else if (nsteps <= 8388608.0) h.capf = (float)(int)(2.0 * nsteps + 64.0);
    else h.capf = 0.f;
    h.g = A.g ? A.g[k] : 0.f;
    h.b = A.b ? A.b[k] : 0.f;
    h.y0scale = (A.bound == SSM_BOUND_TABLE) ? A.table[k * A.tstride] : h.a;
    h.pad0 = 0.f;
    for (int i = 0; i < 4; ++i) h.pad[i] = 0.f;
    *reinterpret_cast<RaceHead *>(row) = h;
    float *v = row + 16, *sq = v + A.np, *z = sq + A.np;
    for (int j = 0; j < A.np; ++j) {
        v[j] = A.v[k * A.np + j];
        const int64_t i = A.per_trial_zs ? k : k * A.np + j;
        sq[j] = __fmul_rn(A.sqrt_dt, A.s[i]);  // delta_t_sqrt * s (race_models.pyx:385)
        z[j] = A.z[i];
    }
}

template <int BOUND, bool EXACT>
__device__ __forceinline__ float race_bound(const RaceHead &h, float ixf, int ix,
                                            const RaceParams &p, int64_t k) {
    if (BOUND == SSM_BOUND_CONSTANT) {
        return h.a;
    } else if (BOUND == SSM_BOUND_LINEAR) {
        if (EXACT) return __fadd_rn(h.a, __fmul_rn(__fmul_rn(ixf, p.dt), h.p1));
        return fmaf(ixf, h.dtp1, h.a);
    } else if (BOUND == SSM_BOUND_WEIBULL) {
        const float x = ixf * p.dt * h.inv_beta;
        const float pw = (x > 0.f) ? exp2f(h.p1 * __log2f(x)) : 0.f;
        return h.a * __expf(-pw);
    } else {
        const int64_t i = (ix < p.tlen) ? ix : p.tlen - 1;
        return __ldg(p.table + k * p.tstride + i);
    }
}

__device__ __forceinline__ float2 std_normal_pair(uint32_t a, uint32_t b) {
    return box_muller(a, b);
}

// Models with at most 4 accumulators draw a window of WIN steps' increments at
// once, six per Philox4x32-10 call, WIN * NP a multiple of six: 2 accumulators
// 12 steps, 3 accumulators 8, 4 accumulators 6 -- four independent calls per
// window, whose latencies overlap.
template <int NP> struct RaceWin { static constexpr int value = NP == 2 ? 12 : (NP == 3 ? 8 : 6); };

template <int NP>
struct RaceLane {
    int64_t w;
    uint32_t k, n;
    float ixf, tp;  // steps taken (as float); race: float32 time accumulator
    double tpd;     // lca: double time accumulator (Cython infers double, race_models.pyx:838)
    int win;        // rdm: index of the winning accumulator (-1 while racing)
    float x[NP];
};

// Two accumulators' constants per increment: radius constant c2 = -2 ln(2) sq^2
// and drift v dt of the steps' increments v dt + sq N(0,1).
template <int NP> struct RaceScale { float c2[NP], d[NP]; };

// The radius and phase bits of pair i of a call (bm6_increment_pairs' layout).
__device__ __forceinline__ uint32_t rad_bits(uint4 b, int i) { return i == 0 ? b.x : (i == 1 ? b.y : b.z); }
__device__ __forceinline__ uint32_t phase_bits(uint4 b, int i) {
    return i == 0 ? (b.w & 0x007fffffu) : (i == 1 ? phase18(b.w, b.x) : phase18(b.y, b.z));
}

// The next window's increments, six per Philox call (calls ctr .. ctr + 3),
// accumulator-major: pre[j * WIN + s] is accumulator j's increment
// v_j dt + sq_j N(0,1) at step s of the window.  WIN is even, so every
// Box-Muller pair belongs to one accumulator, whose scale and drift fold into
// the pair.  Two pairs share the FP32 instructions: those of accumulators j and
// j + 1 at the same steps, so that a step takes both in one packed operation (an
// odd last accumulator's pairs go two by two).
template <int NP>
__device__ __forceinline__ void draw_window(const RaceParams &p, const RaceLane<NP> &L, const RaceScale<NP> &S,
                                            uint32_t ctr, float *pre) {
    constexpr int WIN = RaceWin<NP>::value, H = WIN / 2;
    static_assert(WIN % 2 == 0 && WIN * NP == 24, "pairs within one accumulator, four calls");
    uint4 r[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) r[c] = philox10(make_uint4(ctr + (uint32_t)c, L.n, L.k + p.k_base, 0u), p.key);
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        // packed operation q works on Box-Muller pairs i0 and i1 of the window's twelve
        const bool odd = q >= (NP / 2) * H;  // the last of an odd number of accumulators
        const int j0 = odd ? NP - 1 : 2 * (q / H), j1 = odd ? NP - 1 : j0 + 1;
        const int i0 = odd ? j0 * H + 2 * (q - (NP / 2) * H) : j0 * H + q % H;
        const int i1 = odd ? i0 + 1 : j1 * H + q % H;
        uint64_t cs, sn;
        bm_pair2(rad_bits(r[i0 / 3], i0 % 3), rad_bits(r[i1 / 3], i1 % 3), phase_bits(r[i0 / 3], i0 % 3),
                 phase_bits(r[i1 / 3], i1 % 3), pack_f2(S.c2[j0], S.c2[j1]), pack_f2(S.d[j0], S.d[j1]), cs, sn);
        const float2 c = unpack_f2(cs), t = unpack_f2(sn);
        pre[2 * i0] = c.x;
        pre[2 * i0 + 1] = t.x;
        pre[2 * i1] = c.y;
        pre[2 * i1 + 1] = t.y;
    }
}

// True when none of the lane's next `win` steps can reach the step cap or the
// time limit: the float32 accumulator after (win - 1) more additions of dt is
// at most t + (win - 1) dt plus their roundings (under dt/4 below 65536 dt),
// so t + (win + 1) dt <= dl_tmp leaves margin.  LCA's time is exactly steps dt;
// the margin of 2^-22 covers the two roundings here.
template <int NP, int FAM>
__device__ __forceinline__ bool window_clear(const RaceParams &p, const RaceLane<NP> &L, const RaceHead &h,
                                             int win) {
    if (L.ixf + (float)win > h.capf) return false;
    const float span = (float)(win + 1);
    if (FAM == FAM_LCA) return p.dt >= 1e-30f && (L.ixf + span) * (p.dt * 1.00000024f) <= h.dl_tmp;
    return (L.tp < p.dt * 65536.f) && (fmaf(span, p.dt, L.tp) <= h.dl_tmp);
}

// One Euler step of every accumulator.  Returns false when the loop condition
// failed before the step (the walk is over).  With PRE the step's increments
// v_j dt + sq_j N(0,1) come from pre[j * PSTRIDE] (draw_window); ctr still
// counts the steps.
template <int NP, int FAM, int BOUND, bool NOISE, bool RECORD, bool PRE = false, int PSTRIDE = 1>
__device__ __forceinline__ bool race_step(const RaceParams &p, RaceLane<NP> &L, const RaceHead &h,
                                          const float *v, const float *sq, int np, uint32_t &ctr,
                                          const float *pre = nullptr) {
    if (L.ixf >= h.capf) {
        raise_error(p.hdr, SSM_ERR_DEVICE, (int)L.w);
        return false;
    }
    const float bnd = race_bound<BOUND, NOISE>(h, L.ixf, (int)L.ixf, p, L.k);
    bool finished = false;
    if (FAM != FAM_RDM) {  // race / LCA test the bound before the step; RDM after each update
#pragma unroll
        for (int j = 0; j < NP; ++j)
            if (j < np) finished |= (L.x[j] > bnd);
    }
    constexpr bool LCA = (FAM == FAM_LCA);
    const bool in_time = LCA ? (L.tpd <= (double)h.dl_tmp) : (L.tp <= h.dl_tmp);
    if (finished || !in_time) return false;
    float gsn[NP];
    if (NOISE) {
        const int64_t base = (int64_t)L.ixf * np;
        if (base + np > p.nlen) {
            raise_error(p.hdr, SSM_ERR_NOISE_RANGE, (int)L.w);
            return false;
        }
        const float *row = p.noise + L.w * p.nlen + base;
#pragma unroll
        for (int j = 0; j < NP; ++j) gsn[j] = (j < np) ? __ldg(row + j) : 0.f;
    } else if (PRE) {
#pragma unroll
        for (int j = 0; j < NP; ++j) gsn[j] = pre[j * PSTRIDE];
        ctr += 1;
    } else {
#pragma unroll
        for (int j0 = 0; j0 < NP; j0 += 4) {
            if (j0 < np) {
                const uint4 r = philox10(make_uint4(ctr, L.n, L.k + p.k_base, 0u), p.key);
                ctr += 1;
                const float2 a = std_normal_pair(r.x, r.y);
                const float2 b = std_normal_pair(r.z, r.w);
                if (j0 + 0 < NP) gsn[j0 + 0] = a.x;
                if (j0 + 1 < NP) gsn[j0 + 1] = a.y;
                if (j0 + 2 < NP) gsn[j0 + 2] = b.x;
                if (j0 + 3 < NP) gsn[j0 + 3] = b.y;
            }
        }
    }
    if (LCA) {
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < NP; ++j)
            if (j < np) sum = NOISE ? __fadd_rn(sum, L.x[j]) : sum + L.x[j];
        // with PRE the increments carry v dt + sq N: x (1 - g dt + b dt) - b dt sum + increment
        const float c1 = fmaf(h.b - h.g, p.dt, 1.f), c2 = -h.b * p.dt;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            if (j < np) {
                float xj = L.x[j];
                if (PRE && !NOISE) {
                    xj = fmaf(xj, c1, fmaf(sum, c2, gsn[j]));
                } else if (NOISE) {
                    // race_models.pyx:849-857 with the reference build's association
                    const float red = __double2float_rn(__dadd_rn(-(double)xj, (double)sum));
                    const float A = __fsub_rn(__fsub_rn(v[j], __fmul_rn(h.g, xj)), __fmul_rn(h.b, red));
                    xj = __fadd_rn(__fadd_rn(xj, __fmul_rn(A, p.dt)), __fmul_rn(sq[j], gsn[j]));
                } else {
                    const float red = sum - xj;
                    const float A = v[j] - h.g * xj - h.b * red;
                    xj = fmaf(sq[j], gsn[j], fmaf(A, p.dt, xj));
                }
                L.x[j] = fmaxf(0.f, xj);
            }
        }
        L.tpd = NOISE ? __dadd_rn(L.tpd, (double)p.dt) : L.tpd + (double)p.dt;
    } else if (FAM == FAM_RDM) {
        // no lower barrier; the first accumulator (in index order) at or above b
        // wins and its step does not advance the time (race_models.pyx:1227-1244)
        bool hit = false;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            if (j < np) {
                float xj;
                if (NOISE) xj = __fadd_rn(__fadd_rn(L.x[j], __fmul_rn(v[j], p.dt)), __fmul_rn(sq[j], gsn[j]));
                else if (PRE) xj = L.x[j] + gsn[j];
                else xj = fmaf(sq[j], gsn[j], L.x[j] + v[j] * p.dt);
                L.x[j] = xj;
                hit |= (xj >= bnd);
            }
        }
        if (hit) {  // once per walk: the winner is the first accumulator at or above b
            int win = 0;
#pragma unroll
            for (int j = NP - 1; j >= 0; --j)
                if (j < np && L.x[j] >= bnd) win = j;
            L.win = win;
            return false;
        }
        L.tp = NOISE ? __fadd_rn(L.tp, p.dt) : L.tp + p.dt;
    } else {
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            if (j < np) {
                float xj;
                if (NOISE) xj = __fadd_rn(__fadd_rn(L.x[j], __fmul_rn(v[j], p.dt)), __fmul_rn(sq[j], gsn[j]));
                else if (PRE) xj = L.x[j] + gsn[j];
                else xj = fmaf(sq[j], gsn[j], L.x[j] + v[j] * p.dt);
                L.x[j] = fmaxf(0.f, xj);
            }
        }
        L.tp = NOISE ? __fadd_rn(L.tp, p.dt) : L.tp + p.dt;
    }
    L.ixf += 1.0f;  // steps taken, exact in float32 below 2^24
    if (RECORD) {
        const int64_t ix = (int64_t)L.ixf;
        if ((ix + 1) * np <= p.traj_len)
            for (int j = 0; j < np && j < NP; ++j) p.traj[ix * np + j] = L.x[j];
    }
    return true;
}

__device__ __forceinline__ float max3(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }

// Advance a walk by a window of steps whose increments are in pre (draw_window).
// Returns whether it is still running.  The steps run without a test each: the
// largest accumulator seen is compared once with the lowest bound of the window
// (constant and linear bounds; the others compare each step), and only a walk that may
// have ended, or may reach its time limit, takes the window again step by step.
template <int NP, int FAM, int BOUND>
__device__ __forceinline__ bool advance_window(const RaceParams &p, RaceLane<NP> &L, const RaceHead &h,
                                               const float *pre) {
    constexpr int WIN = RaceWin<NP>::value;
    constexpr bool LCA = (FAM == FAM_LCA), ONE_TEST = (BOUND == SSM_BOUND_CONSTANT || BOUND == SSM_BOUND_LINEAR);
    // (a walk of the other families ends above its bound, which is what the test of
    // each step for the other bounds looks for)
    static_assert(FAM != FAM_RDM || BOUND == SSM_BOUND_CONSTANT, "racing diffusion ends at or above a constant bound");
    if (window_clear<NP, FAM>(p, L, h, WIN)) {
        // accumulators 0 and 1 in x01, 2 and 3 in x23 (2 alone: its upper half is idle)
        uint64_t xp[(NP + 1) / 2];
#pragma unroll
        for (int j = 0; j < NP; j += 2) xp[j / 2] = pack_f2(L.x[j], (j + 1 < NP) ? L.x[j + 1] : 0.f);
        float tp = L.tp, m = 0.f;
        bool first = true, below = true;
        const float c1 = fmaf(h.b - h.g, p.dt, 1.f), c2 = -h.b * p.dt;
        const uint64_t c1p = pack_f2(c1, c1), c2p = pack_f2(c2, c2);
#pragma unroll
        for (int s = 0; s < WIN; ++s) {
            float x[NP + 1];
            auto read = [&]() {
#pragma unroll
                for (int j = 0; j < NP; j += 2) {
                    const float2 v = unpack_f2(xp[j / 2]);
                    x[j] = v.x;
                    x[j + 1] = v.y;
                }
            };
            auto see = [&]() {
                if (!ONE_TEST || first) m = fmaxf(x[0], x[1]);
                else m = max3(m, x[0], x[1]);
                if (NP == 3) m = fmaxf(m, x[2]);
                if (NP == 4) m = max3(m, x[2], x[NP - 1]);
                first = false;
                if (!ONE_TEST) below &= m <= race_bound<BOUND, false>(h, L.ixf + (float)s, (int)(L.ixf) + s, p, L.k);
            };
            read();
            if (FAM != FAM_RDM) see();
            if (LCA) {
                float sum = x[0] + x[1];
                if (NP >= 3) sum += x[2];
                if (NP == 4) sum += x[NP - 1];
                const uint64_t sp = pack_f2(sum, sum);
#pragma unroll
                for (int j = 0; j < NP; j += 2) {
                    if (j + 1 < NP) {
                        const uint64_t g = pack_f2(pre[j * WIN + s], pre[(j + 1) * WIN + s]);
                        xp[j / 2] = fma_f2(xp[j / 2], c1p, fma_f2(sp, c2p, g));
                    } else {
                        xp[j / 2] = pack_f2(fmaf(x[j], c1, fmaf(sum, c2, pre[j * WIN + s])), 0.f);
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < NP; j += 2) {
                    if (j + 1 < NP) xp[j / 2] = add_f2(xp[j / 2], pack_f2(pre[j * WIN + s], pre[(j + 1) * WIN + s]));
                    else xp[j / 2] = pack_f2(x[j] + pre[j * WIN + s], 0.f);
                }
                tp += p.dt;
            }
            if (FAM != FAM_RDM) {
#pragma unroll
                for (int j = 0; j < NP; j += 2) {
                    const float2 v = unpack_f2(xp[j / 2]);
                    xp[j / 2] = pack_f2(fmaxf(0.f, v.x), (j + 1 < NP) ? fmaxf(0.f, v.y) : 0.f);
                }
            } else {
                read();
                see();
            }
        }
        if (ONE_TEST) {
            float lo = race_bound<BOUND, false>(h, L.ixf, 0, p, L.k);
            if (BOUND == SSM_BOUND_LINEAR)  // rounded monotonically: lowest at one of the ends
                lo = fminf(lo, race_bound<BOUND, false>(h, L.ixf + (float)(WIN - 1), 0, p, L.k));
            below = (FAM == FAM_RDM) ? m < lo : m <= lo;
        }
        if (below) {
#pragma unroll
            for (int j = 0; j < NP; j += 2) {
                const float2 v = unpack_f2(xp[j / 2]);
                L.x[j] = v.x;
                if (j + 1 < NP) L.x[j + 1] = v.y;
            }
            L.tp = tp;
            L.ixf += (float)WIN;
            return true;
        }
    }
    if (LCA) L.tpd = (double)L.ixf * (double)p.dt;  // exact: 24-bit dt, fewer than 2^29 steps
    bool live = true;
    uint32_t unused = 0;
#pragma unroll
    for (int s = 0; s < WIN; ++s)
        if (live) live = race_step<NP, FAM, BOUND, false, false, true, WIN>(p, L, h, nullptr, nullptr, NP, unused, pre + s);
    return live;
}

template <int NP, int FAM, bool NOISE>
__device__ __forceinline__ void race_finalize(const RaceParams &p, const RaceLane<NP> &L,
                                              const RaceHead &h, int np) {
    float u;
    if (NOISE) u = __ldg(p.nunif + ((FAM == FAM_RDM) ? L.w * (np + 1) + np : L.w));
    else u = uniform_co(philox10(make_uint4(0xFFFFFFFFu, L.n, L.k + p.k_base, 1u), p.key).x);
    // compute_smooth_unif receives the time as a C float (_utils.pyx:668-695)
    constexpr bool LCA = (FAM == FAM_LCA);
    const float tpf = LCA ? __double2float_rn(L.tpd) : L.tp;
    float sm = 0.f;
    if (p.smooth) {
        if (tpf == 0.f) sm = __double2float_rn(((double)u * 0.5) * (double)p.dt);
        else if (tpf < h.dl_tmp) sm = __double2float_rn((0.5 - (double)u) * (double)p.dt);
    }
    float rt;
    if (LCA) rt = __double2float_rn(__dadd_rn(__dadd_rn(L.tpd, (double)h.t), (double)sm));
    else rt = __fadd_rn(__fadd_rn(L.tp, h.t), sm);
    if (rt >= h.deadline || h.deadline <= 0.f) rt = -999.f;  // enforce_deadline
    if (FAM == FAM_RDM) {  // no decision or an omission: rt -999, choice -1
        const bool omit = (rt == -999.f) || (L.win < 0);
        p.rts[L.w] = omit ? -999.f : rt;
        p.choices[L.w] = omit ? -1 : L.win;
        if (p.steps) p.steps[L.w] = (int)L.ixf;
        return;
    }
    int best = 0;
    float bv = L.x[0];
#pragma unroll
    for (int j = 1; j < NP; ++j)
        if (j < np && L.x[j] > bv) {
            bv = L.x[j];
            best = j;
        }
    p.rts[L.w] = rt;
    p.choices[L.w] = best;
    if (p.steps) p.steps[L.w] = (int)L.ixf;
}

__device__ __forceinline__ int64_t race_find(const int64_t *off, int64_t K, int64_t w, int64_t hint) {
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

template <int NP, int FAM, bool NOISE>
__device__ __forceinline__ bool race_init(const RaceParams &p, RaceLane<NP> &L, RaceHead &h,
                                          int64_t w, int64_t &hint, int np) {
    int64_t k, n;
    if (p.offsets == nullptr) {
        k = w % p.n_trials;
        n = w / p.n_trials;
    } else if (p.order != nullptr) {
        // queue index -> position j in the processing order -> trial k (outputs
        // stay at offsets[k] + n); an entry that does not fit is reported
        const int64_t j = race_find(p.qoff, p.n_trials, w, hint);
        hint = j;
        k = __ldg(p.order + j);
        n = w - __ldg(p.qoff + j);
        if (k < 0 || k >= p.n_trials || n < 0 || n >= __ldg(p.offsets + k + 1) - __ldg(p.offsets + k)) {
            raise_error(p.hdr, SSM_ERR_ARG, (int)j);
            return false;
        }
        w = __ldg(p.offsets + k) + n;
    } else {
        w += __ldg(p.offsets);  // global output index (trial windows start past 0)
        k = race_find(p.offsets, p.n_trials, w, hint);
        n = w - __ldg(p.offsets + k);
        hint = k;
    }
    const float *row = p.rows + k * p.row_floats;
    const float4 *src = reinterpret_cast<const float4 *>(row);
    float4 *dst = reinterpret_cast<float4 *>(&h);
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[i] = __ldg(src + i);
    const float *z = row + 16 + 2 * np;
    L.w = w;
    L.k = (uint32_t)k;
    L.n = (uint32_t)n;
    L.win = -1;
    if (FAM == FAM_RDM) {
        // starts U(0, A): z holds A; injected uniforms, or the trajectory's own stream
#pragma unroll
        for (int j0 = 0; j0 < NP; j0 += 4) {
            uint4 r = make_uint4(0u, 0u, 0u, 0u);
            if (!NOISE && j0 < np) r = philox10(make_uint4(0xFFFFFFFEu, L.n, L.k + p.k_base, 2u + (uint32_t)j0), p.key);
            const uint32_t wd[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = j0 + q;
                if (j < NP) {
                    const float u = NOISE ? ((j < np) ? __ldg(p.nunif + L.w * (np + 1) + j) : 0.f) : uniform_co(wd[q]);
                    L.x[j] = (j < np) ? __fmul_rn(u, __ldg(z + j)) : 0.f;
                }
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < NP; ++j) L.x[j] = (j < np) ? __fmul_rn(__ldg(z + j), h.y0scale) : 0.f;
    }
    L.ixf = 0.f;
    L.tp = 0.f;
    L.tpd = 0.0;
    return true;
}

// A trial's RaceScale from its row.
template <int NP>
__device__ __forceinline__ void race_scale(const RaceParams &p, const float *row, RaceScale<NP> &S) {
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        const float sq = __ldg(row + 16 + NP + j);
        S.c2[j] = -1.3862944f * sq * sq;
        S.d[j] = __ldg(row + 16 + j) * p.dt;
    }
}

// Walks a warp still runs when the queue is empty for its lanes to share their
// draws (four lanes each at least: a window has four calls).
constexpr int RACE_SHARE_MAX = 8;

template <int NP, int FAM, int BOUND>
__global__ void __launch_bounds__(256) k_race_window(const __grid_constant__ RaceParams p) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    const int64_t total = (p.total >= 0) ? p.total : __ldg(p.offsets + p.n_trials) - __ldg(p.offsets);
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    // A launch of at most four walks per warp is spread over all warps, each
    // taking its walks in one claim: the lanes then share their draws from the start.
    const int64_t per_warp = (total + warps - 1) / warps;
    const bool spread = per_warp <= 4;
    constexpr int np = NP, WIN = RaceWin<NP>::value;
    __shared__ float drawn[8][32 * 6];  // the last walks' increments, a call of each lane
    RaceLane<NP> L;
    RaceHead h;
    RaceScale<NP> S;
    L.w = 0; L.k = L.n = 0; L.ixf = L.tp = 0.f; L.tpd = 0.0; L.win = -1;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        L.x[j] = 0.f;
        S.c2[j] = S.d[j] = 0.f;
    }
    uint32_t ctr = 0;
    bool active = false, pending = false, exhausted = false;
    int64_t q_next = 0, q_end = 0, hint = 0;
    for (;;) {
        // ended walks are written and their lanes restarted refill_min at a
        // time (one divergent pass for several lanes); all at once when the
        // queue is empty
        const unsigned need = __ballot_sync(FULL, !active && (!spread || lane < per_warp));
        const bool pass = exhausted ? (__ballot_sync(FULL, pending) != 0u) : (spread || __popc(need) >= p.refill_min);
        if (pass && pending) {
            race_finalize<NP, FAM, false>(p, L, h, np);
            pending = false;
        }
        if (pass && !exhausted) {
            const int cnt = __popc(need);
            const int64_t avail = q_end - q_next;
            int64_t base = 0, claim = 0;
            if (avail < cnt) {
                // claims shrink with what is left of the queue, down to the walks
                // needed now.  Small claims matter here: the longest walks come
                // first, and a warp with two rounds of them is the launch's end (256
                // LCA sets: claims of 64 9.6 ms, 32 6.5 ms).
                claim = max((int64_t)cnt, min((int64_t)p.chunk, (total - q_end) / (2 * warps)));
                unsigned long long bb = 0ull;
                if (lane == 0) bb = atomicAdd(&p.hdr->counter, (unsigned long long)claim);
                base = (int64_t)__shfl_sync(FULL, bb, 0);
                if (base >= total || spread) exhausted = true;
            }
            if (need >> lane & 1u) {
                const int rank = __popc(need & lt_mask);
                const int64_t w = (rank < avail) ? q_next + rank : base + (rank - avail);
                if (w < total && race_init<NP, FAM, false>(p, L, h, w, hint, np)) {
                    race_scale<NP>(p, p.rows + (int64_t)L.k * p.row_floats, S);
                    ctr = 0;
                    active = true;
                }
            }
            if (avail >= cnt) {
                q_next += cnt;
            } else {
                q_next = base + (cnt - avail);
                q_end = base + claim;
            }
        }
        const unsigned running = __ballot_sync(FULL, active);
        if (running == 0u || (exhausted && __popc(running) <= RACE_SHARE_MAX)) break;
        if (active) {
            float pre[WIN * NP];
            draw_window<NP>(p, L, S, ctr, pre);
            ctr += 4;
            if (!advance_window<NP, FAM, BOUND>(p, L, h, pre)) {
                active = false;
                pending = true;
            }
        }
    }
    // The queue is empty and few of the warp's walks still run: G lanes draw for
    // each, a Philox call per lane (G / 4 windows), and the walk's own lane takes the
    // steps.  A walk's lane alone would wait for its four calls one after the other.
    unsigned running = __ballot_sync(FULL, active);
    while (running != 0u) {
        const int m = __popc(running);
        int G = 4;
        while (2 * G * m <= 32) G *= 2;
        const int g = lane / G, call = lane & 3;
        const int src = (g < m) ? (int)__fns(running, 0u, g + 1) : lane;
        RaceLane<NP> D;
        D.n = __shfl_sync(FULL, L.n, src);
        D.k = __shfl_sync(FULL, L.k, src);
        uint32_t c = __shfl_sync(FULL, ctr, src) + (uint32_t)(lane & (G - 1));
        float c2[3] = {0.f, 0.f, 0.f}, d[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            const float cj = __shfl_sync(FULL, S.c2[j], src), dj = __shfl_sync(FULL, S.d[j], src);
#pragma unroll
            for (int e = 0; e < 3; ++e)
                if ((6 * call + 2 * e) / WIN == j) {
                    c2[e] = cj;
                    d[e] = dj;
                }
        }
        float *mine = drawn[threadIdx.x >> 5] + lane * 6;
        const float *walk = drawn[threadIdx.x >> 5] + __popc(running & lt_mask) * G * 6;
        unsigned now;
        do {
            if (g < m) {
                float x[6];
                bm6_increment_pairs(philox10(make_uint4(c, D.n, D.k + p.k_base, 0u), p.key), c2, d, x);
#pragma unroll
                for (int e = 0; e < 6; ++e) mine[e] = x[e];
            }
            c += (uint32_t)G;
            __syncwarp();
            if (active) {
                bool live = true;
#pragma unroll 1
                for (int u = 0; u < G / 4 && live; ++u) {
                    float pre[WIN * NP];
#pragma unroll
                    for (int e = 0; e < WIN * NP; ++e) pre[e] = walk[24 * u + e];
                    live = advance_window<NP, FAM, BOUND>(p, L, h, pre);
                }
                ctr += (uint32_t)G;
                if (!live) {
                    race_finalize<NP, FAM, false>(p, L, h, np);
                    active = false;
                }
            }
            __syncwarp();
            now = __ballot_sync(FULL, active);
        } while (now == running);
        running = now;
    }
}

template <int NP, int FAM, int BOUND, bool NOISE>
__global__ void __launch_bounds__(256) k_race(const __grid_constant__ RaceParams p) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    const int64_t total = (p.total >= 0) ? p.total : __ldg(p.offsets + p.n_trials) - __ldg(p.offsets);
    const int64_t chunk = warp_chunk(p.chunk, total);
    const int np = (NP == RACE_MAX_NP) ? p.np : NP;
    RaceLane<NP> L;
    RaceHead h;
    L.w = 0; L.k = L.n = 0; L.ixf = L.tp = 0.f; L.tpd = 0.0; L.win = -1;
#pragma unroll
    for (int j = 0; j < NP; ++j) L.x[j] = 0.f;
    uint32_t ctr = 0;
    bool active = false, pending = false, exhausted = false;
    int64_t q_next = 0, q_end = 0, hint = 0;
    for (;;) {
        // ended walks are written and their lanes restarted refill_min at a
        // time (one divergent pass for several lanes); all at once when the
        // queue is empty
        const unsigned need = __ballot_sync(FULL, !active);
        const bool pass = exhausted ? (__ballot_sync(FULL, pending) != 0u) : (__popc(need) >= p.refill_min);
        if (pass && pending) {
            race_finalize<NP, FAM, NOISE>(p, L, h, np);
            pending = false;
        }
        if (pass && !exhausted) {
            const int cnt = __popc(need);
            const int64_t avail = q_end - q_next;
            int64_t base = 0;
            if (avail < cnt) {
                unsigned long long bb = 0ull;
                if (lane == 0) bb = atomicAdd(&p.hdr->counter, (unsigned long long)chunk);
                base = (int64_t)__shfl_sync(FULL, bb, 0);
                if (base >= total) exhausted = true;
            }
            if (!active) {
                const int rank = __popc(need & lt_mask);
                const int64_t w = (rank < avail) ? q_next + rank : base + (rank - avail);
                if (w < total && race_init<NP, FAM, NOISE>(p, L, h, w, hint, np)) {
                    ctr = 0;
                    active = true;
                }
            }
            if (avail >= cnt) {
                q_next += cnt;
            } else {
                q_next = base + (cnt - avail);
                q_end = base + chunk;
            }
        }
        if (__ballot_sync(FULL, active) == 0u) break;
        if (active) {
            const float *row = p.rows + (int64_t)L.k * p.row_floats;
            const float *v = row + 16;
            const float *sq = v + np;
            float vr[NP], sr[NP];
#pragma unroll
            for (int j = 0; j < NP; ++j) {
                vr[j] = (j < np) ? __ldg(v + j) : 0.f;
                sr[j] = (j < np) ? __ldg(sq + j) : 0.f;
            }
            bool live = true;
#pragma unroll 1
            for (int s = 0; s < 4 && live; ++s)
                live = race_step<NP, FAM, BOUND, NOISE, false>(p, L, h, vr, sr, np, ctr);
            if (!live) {
                active = false;
                pending = true;
            }
        }
    }
}

template <int NP, int FAM, int BOUND, bool NOISE>
__global__ void k_race_record(const __grid_constant__ RaceParams p) {
    const int np = (NP == RACE_MAX_NP) ? p.np : NP;
    for (int64_t i = threadIdx.x; i < p.traj_len; i += blockDim.x) p.traj[i] = -999.f;
    __syncthreads();
    if (threadIdx.x != 0) return;
    RaceLane<NP> L;
    RaceHead h;
    int64_t hint = 0;
    race_init<NP, FAM, NOISE>(p, L, h, 0, hint, np);
    for (int j = 0; j < np && j < NP && j < p.traj_len; ++j) p.traj[j] = L.x[j];
    const float *row = p.rows + (int64_t)L.k * p.row_floats;
    float vr[NP], sr[NP];
    for (int j = 0; j < NP; ++j) {
        vr[j] = (j < np) ? row[16 + j] : 0.f;
        sr[j] = (j < np) ? row[16 + np + j] : 0.f;
    }
    uint32_t ctr = 0;
    if constexpr (!NOISE && NP <= 4) {
        // the main kernel's windows: the same normals in the same order
        constexpr int WIN = RaceWin<NP>::value;
        RaceScale<NP> S;
        race_scale<NP>(p, row, S);
        bool live = true;
        while (live) {
            float nrm[WIN * NP];
            draw_window<NP>(p, L, S, ctr, nrm);
            ctr += 4;
            uint32_t unused = 0;
            for (int s = 0; s < WIN && live; ++s)
                live = race_step<NP, FAM, BOUND, NOISE, true, true, WIN>(p, L, h, vr, sr, np, unused, nrm + s);
        }
    } else {
        while (race_step<NP, FAM, BOUND, NOISE, true>(p, L, h, vr, sr, np, ctr)) {
        }
    }
}

template <int NP, int FAM, int BOUND, bool NOISE>
static auto race_kernel() -> void (*)(const RaceParams) {
    if constexpr (!NOISE && NP <= 4) return k_race_window<NP, FAM, BOUND>;
    else return k_race<NP, FAM, BOUND, NOISE>;
}

template <int NP, int FAM, int BOUND, bool NOISE>
static int race_launch(const RaceParams &p, const ssm_launch *opt, cudaStream_t st) {
    auto kern = race_kernel<NP, FAM, BOUND, NOISE>();
    int threads = (opt && opt->block_threads > 0) ? opt->block_threads : 256;
    if (threads > 256 || threads % 32) {
        set_error("block_threads must be a multiple of 32 and at most 256");
        return SSM_ERR_ARG;
    }
    int per_sm = 0;
    SSM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, 0));
    if (opt && opt->blocks_per_sm > 0 && opt->blocks_per_sm < per_sm) per_sm = opt->blocks_per_sm;
    if (per_sm < 1) per_sm = 1;
    kern<<<sm_count() * per_sm, threads, 0, st>>>(p);
    SSM_CUDA(cudaGetLastError());
    if (p.traj && p.traj_len > 0) {
        RaceParams pr = p;  // trial 0 / sample 0, whatever the processing order
        pr.order = nullptr;
        pr.qoff = nullptr;
        k_race_record<NP, FAM, BOUND, NOISE><<<1, 128, 0, st>>>(pr);
        SSM_CUDA(cudaGetLastError());
    }
    return SSM_OK;
}

// Racing diffusion has a constant bound (ssm_racing_diffusion takes no other); the
// kernels of its other forms are not built.
template <int NP, int FAM>
static int race_dispatch_bound(int bound, bool noise, const RaceParams &p, const ssm_launch *opt,
                               cudaStream_t st) {
    if constexpr (FAM == FAM_RDM) {
        SSM_REQUIRE(bound == SSM_BOUND_CONSTANT, "racing diffusion has a constant boundary");
        return noise ? race_launch<NP, FAM, SSM_BOUND_CONSTANT, true>(p, opt, st)
                     : race_launch<NP, FAM, SSM_BOUND_CONSTANT, false>(p, opt, st);
    } else if (noise) {  // exact mode: any boundary shape arrives as a host table or in closed form
        switch (bound) {
            case SSM_BOUND_TABLE: return race_launch<NP, FAM, SSM_BOUND_TABLE, true>(p, opt, st);
            case SSM_BOUND_CONSTANT: return race_launch<NP, FAM, SSM_BOUND_CONSTANT, true>(p, opt, st);
            case SSM_BOUND_LINEAR: return race_launch<NP, FAM, SSM_BOUND_LINEAR, true>(p, opt, st);
            default: break;
        }
        set_error("noise injection supports table, constant and linear boundaries");
        return SSM_ERR_ARG;
    } else {
        switch (bound) {
            case SSM_BOUND_TABLE: return race_launch<NP, FAM, SSM_BOUND_TABLE, false>(p, opt, st);
            case SSM_BOUND_CONSTANT: return race_launch<NP, FAM, SSM_BOUND_CONSTANT, false>(p, opt, st);
            case SSM_BOUND_LINEAR: return race_launch<NP, FAM, SSM_BOUND_LINEAR, false>(p, opt, st);
            case SSM_BOUND_WEIBULL: return race_launch<NP, FAM, SSM_BOUND_WEIBULL, false>(p, opt, st);
            default: break;
        }
        set_error("unknown boundary kind %d", bound);
        return SSM_ERR_ARG;
    }
}

template <int FAM>
static int race_dispatch(int np, int bound, bool noise, const RaceParams &p, const ssm_launch *opt,
                         cudaStream_t st) {
    switch (np) {
        case 2: return race_dispatch_bound<2, FAM>(bound, noise, p, opt, st);
        case 3: return race_dispatch_bound<3, FAM>(bound, noise, p, opt, st);
        case 4: return race_dispatch_bound<4, FAM>(bound, noise, p, opt, st);
        default: return race_dispatch_bound<RACE_MAX_NP, FAM>(bound, noise, p, opt, st);
    }
}

static size_t race_ws_bytes(int64_t n_trials, int np) {
    if (n_trials < 0) n_trials = 0;
    size_t b = sizeof(WorkspaceHeader) + (size_t)n_trials * race_row_floats(np) * sizeof(float);
    return (b + 255) & ~(size_t)255;
}

static int run_race(int fam, const float *v, const float *z, const float *t, const float *s,
                    const float *deadline, const float *g, const float *b, int64_t n_trials,
                    int64_t n_samples, int np, const int64_t *offsets, float max_t, float dt,
                    int bound, const float *a, const float *p1, const float *p2,
                    const float *table, int64_t tstride, int64_t tlen, uint64_t seed, int smooth,
                    const float *noise, int64_t nlen, const float *nunif, float *rts,
                    int32_t *choices, int32_t *steps, float *traj, int64_t traj_len,
                    const ssm_launch *launch, void *ws, size_t ws_bytes, void *stream) {
    SSM_REQUIRE(n_trials >= 0 && n_samples >= 0, "n_trials and n_samples must be >= 0");
    SSM_REQUIRE(np >= 1 && np <= RACE_MAX_NP, "n_particles must be in [1, %d]", RACE_MAX_NP);
    SSM_REQUIRE(dt > 0.f && isfinite(dt), "delta_t must be finite and > 0");
    SSM_REQUIRE(isfinite(max_t) && (double)max_t / (double)dt <= 8388608.0,
                "max_t must be finite with max_t / delta_t <= 2^23");
    SSM_REQUIRE(n_trials == 0 || (v && z && t && s && deadline), "v, z, t, s, deadline are required");
    SSM_REQUIRE(fam != FAM_LCA || n_trials == 0 || (g && b), "lca needs g and b");
    SSM_REQUIRE(!launch || (!launch->trial_order == !launch->order_offsets),
                "trial_order and order_offsets go together");
    SSM_REQUIRE(!launch || !launch->trial_order || offsets, "a trial order needs the ragged layout (sample_offsets)");
    SSM_REQUIRE((rts && choices) || (!offsets && n_trials * n_samples == 0), "rts and choices outputs are required");
    SSM_REQUIRE(bound >= SSM_BOUND_TABLE && bound <= SSM_BOUND_WEIBULL, "unknown boundary kind %d", bound);
    SSM_REQUIRE(bound == SSM_BOUND_TABLE || n_trials == 0 || a, "boundary height a is required");
    SSM_REQUIRE(bound != SSM_BOUND_LINEAR || n_trials == 0 || p1, "linear boundary needs bound_p1");
    SSM_REQUIRE(bound != SSM_BOUND_WEIBULL || n_trials == 0 || (p1 && p2), "weibull boundary needs bound_p1 and bound_p2");
    SSM_REQUIRE(bound != SSM_BOUND_TABLE || (table && tlen >= 1 && tstride >= tlen),
                "table boundary needs bound_table with table_stride >= table_len >= 1");
    SSM_REQUIRE(!noise || (nlen > 0 && nunif), "noise_rows needs noise_row_len > 0 and noise_unif");
    const size_t need = race_ws_bytes(n_trials, np);
    if (!ws || ws_bytes < need || ((uintptr_t)ws & 255u)) {
        set_error("workspace must be 256-byte aligned and hold %zu bytes", need);
        return SSM_ERR_WORKSPACE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    WorkspaceHeader *hdr = (WorkspaceHeader *)ws;
    float *rows = (float *)((char *)ws + sizeof(WorkspaceHeader));
    SSM_CUDA(cudaMemsetAsync(hdr, 0, sizeof(WorkspaceHeader), st));
    const int64_t total = offsets ? -1 : n_trials * n_samples;
    if (n_trials == 0 || total == 0) return SSM_OK;
    RacePrep A;
    A.v = v; A.z = z; A.t = t; A.s = s; A.deadline = deadline; A.a = a; A.p1 = p1; A.p2 = p2;
    A.g = g; A.b = b; A.table = table; A.n_trials = n_trials; A.tstride = tstride;
    A.row_floats = race_row_floats(np); A.np = np; A.bound = bound; A.dt = dt;
    A.sqrt_dt = (float)sqrt((double)dt); A.max_t = max_t; A.rows = rows;
    A.per_trial_zs = (fam == FAM_RDM) ? 1 : 0;
    k_race_prep<<<(unsigned)((n_trials + 127) / 128), 128, 0, st>>>(A);
    SSM_CUDA(cudaGetLastError());
    RaceParams p;
    p.key = philox_keys(seed);
    p.rows = rows; p.row_floats = race_row_floats(np); p.offsets = offsets;
    p.order = (offsets && launch) ? launch->trial_order : nullptr;
    p.qoff = p.order ? launch->order_offsets : nullptr;
    p.n_trials = n_trials; p.total = total; p.np = np; p.dt = dt; p.smooth = smooth ? 1 : 0;
    p.k_base = (uint32_t)((launch && launch->first_trial > 0) ? launch->first_trial : 0);
    p.chunk = (launch && launch->chunk >= 32) ? launch->chunk : 32;
    p.refill_min = (launch && launch->refill_min > 0) ? min(launch->refill_min, 32) : SSM_REFILL_MIN_RACE;
    p.table = table; p.tstride = tstride; p.tlen = tlen;
    p.noise = noise; p.nlen = nlen; p.nunif = nunif;
    p.rts = rts; p.choices = choices; p.steps = steps; p.hdr = hdr;
    p.traj = traj; p.traj_len = traj_len;
    switch (fam) {
        case FAM_LCA: return race_dispatch<FAM_LCA>(np, bound, noise != nullptr, p, launch, st);
        case FAM_RDM: return race_dispatch<FAM_RDM>(np, bound, noise != nullptr, p, launch, st);
        default: return race_dispatch<FAM_RACE>(np, bound, noise != nullptr, p, launch, st);
    }
}

}  // namespace ssm

extern "C" {

size_t ssm_race_workspace_bytes(int64_t n_trials, int n_particles) {
    return ssm::race_ws_bytes(n_trials, n_particles);
}

int ssm_race_model(const float *v, const float *z, const float *t, const float *s,
                   const float *deadline, int64_t n_trials, int64_t n_samples, int n_particles,
                   const int64_t *sample_offsets, float max_t, float delta_t, int bound_kind,
                   const float *a, const float *bound_p1, const float *bound_p2,
                   const float *bound_table, int64_t table_stride, int64_t table_len,
                   uint64_t seed, int smooth_unif, const float *noise_rows, int64_t noise_row_len,
                   const float *noise_unif, float *rts, int32_t *choices, int32_t *steps,
                   float *traj, int64_t traj_len, const ssm_launch *launch, void *workspace,
                   size_t workspace_bytes, void *stream) {
    return ssm::run_race(ssm::FAM_RACE, v, z, t, s, deadline, nullptr, nullptr, n_trials, n_samples,
                         n_particles, sample_offsets, max_t, delta_t, bound_kind, a, bound_p1,
                         bound_p2, bound_table, table_stride, table_len, seed, smooth_unif,
                         noise_rows, noise_row_len, noise_unif, rts, choices, steps, traj,
                         traj_len, launch, workspace, workspace_bytes, stream);
}

int ssm_lca(const float *v, const float *z, const float *g, const float *b, const float *t,
            const float *s, const float *deadline, int64_t n_trials, int64_t n_samples,
            int n_particles, const int64_t *sample_offsets, float max_t, float delta_t,
            int bound_kind, const float *a, const float *bound_p1, const float *bound_p2,
            const float *bound_table, int64_t table_stride, int64_t table_len, uint64_t seed,
            int smooth_unif, const float *noise_rows, int64_t noise_row_len,
            const float *noise_unif, float *rts, int32_t *choices, int32_t *steps, float *traj,
            int64_t traj_len, const ssm_launch *launch, void *workspace, size_t workspace_bytes,
            void *stream) {
    return ssm::run_race(ssm::FAM_LCA, v, z, t, s, deadline, g, b, n_trials, n_samples, n_particles,
                         sample_offsets, max_t, delta_t, bound_kind, a, bound_p1, bound_p2,
                         bound_table, table_stride, table_len, seed, smooth_unif, noise_rows,
                         noise_row_len, noise_unif, rts, choices, steps, traj, traj_len, launch,
                         workspace, workspace_bytes, stream);
}

int ssm_racing_diffusion(const float *v, const float *b, const float *A, const float *t, const float *s,
                         const float *deadline, int64_t n_trials, int64_t n_samples, int n_particles,
                         const int64_t *sample_offsets, float max_t, float delta_t, uint64_t seed,
                         int smooth_unif, const float *noise_rows, int64_t noise_row_len,
                         const float *noise_unif, float *rts, int32_t *choices, int32_t *steps,
                         float *traj, int64_t traj_len, const ssm_launch *launch, void *workspace,
                         size_t workspace_bytes, void *stream) {
    SSM_REQUIRE(n_trials == 0 || (b && A), "b and A are required");
    return ssm::run_race(ssm::FAM_RDM, v, A, t, s, deadline, nullptr, nullptr, n_trials, n_samples,
                         n_particles, sample_offsets, max_t, delta_t, SSM_BOUND_CONSTANT, b, nullptr,
                         nullptr, nullptr, 0, 0, seed, smooth_unif, noise_rows, noise_row_len,
                         noise_unif, rts, choices, steps, traj, traj_len, launch, workspace,
                         workspace_bytes, stream);
}

}  // extern "C"

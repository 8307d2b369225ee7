// Batched log-rt Gaussian KDE for sm_100a: the reference's LogKDE
// (ssms/support_utils/kde_class.py) and the record layout of its
// ResampleMixtureStrategy (ssms/dataset_generators/strategies/
// resample_mixture_strategy.py:64-214), for many parameter sets at once.
//
// Layout.  Simulated data of set s occupies [soff[s], soff[s+1]) of rts /
// choices.  Group g = s * nc + c holds the log-rts of set s with choice c
// (omissions dropped) at points[poff[g] .. poff[g+1]), in sample order.
//
// Evaluation.  For a query log-rt q of group g the reference evaluates
//   log p_c + log( 1/(n h sqrt(2 pi)) sum_j exp(-(q - x_j)^2 / (2 h^2)) ) - q
// exactly (scikit-learn with atol = rtol = 0).  k_kde_eval tiles the group's
// points through shared memory, keeps up to four queries per lane in registers
// (q split into float hi + lo parts so q - x_j keeps full precision), evaluates
// each kernel term as ex2(-(d s)^2) on the SFU and sums in float over 32 terms
// before adding into a float64 accumulator.  Groups differ in cost by orders
// of magnitude (queries x points), so the work is scheduled Stream-K style
// (Osama, Merrill, Cecka, Garland & Owens, PPoPP'23): the cost space (group,
// unit of up to 16 rows of 32 queries, point tile) is cut into equal contiguous
// ranges, one per CTA of a persistent grid; units cut between CTAs are finished
// by a fix-up kernel that adds the CTAs' partial sums in CTA order.
#include <cooperative_groups.h>


#include "common.cuh"

namespace ssm {

constexpr int KDE_MAX_CHOICES = 16;
constexpr int KDE_MAX_ROWS = 12288;  // records per set
constexpr double KDE_LOG_2PI = 1.8378770664093453;

struct KdeFit {
    const float *rts;
    const int32_t *choices;
    int64_t n_sets;
    const int64_t *soff;
    const int32_t *cvals;
    int nc;
    const double *shift; // per-set displacement (displace_t) or nullptr
    double *bwvals;      // [total] displaced-mode bandwidth inputs, or nullptr
    int64_t *count_all;  // [G] samples with choice c, omissions included
    int64_t *n_valid;    // [G] non-omitted samples
    int64_t *poff;       // [G + 1]
    float *points;       // [total valid]
    double *h;           // [G] bandwidth (-1: no data)
    double *lognorm;     // [G] log p_c - log n - log h - log(2 pi)/2
    double *prop;        // [G] choice proportion
};

// The choice values in registers; NC is the compiled capacity (2, 4 or 16),
// nc the number in use.
template <int NC> struct ChoiceSet {
    int32_t v[NC];
    int nc;
    __device__ __forceinline__ ChoiceSet(const int32_t *cvals, int n) : nc(n) {
#pragma unroll
        for (int c = 0; c < NC; ++c) v[c] = (c < n) ? __ldg(cvals + c) : 0;
    }
    __device__ __forceinline__ int index(int32_t ch) const {  // first match, -1: none
        int ci = -1;
#pragma unroll
        for (int c = NC - 1; c >= 0; --c)
            if (c < nc && v[c] == ch) ci = c;
        return ci;
    }
};

// The fit and the summary give every set a cluster of J CTAs (J = gridDim.x /
// n_sets), each taking one contiguous slice of the set's samples: a handful of
// sets still fills the GPU, and the slices' counts meet over distributed shared
// memory instead of in a workspace.
struct Slice {
    int64_t set, lo, hi;
    unsigned rank, J;
};
__device__ __forceinline__ Slice set_slice(const int64_t *soff, int64_t n_sets) {
    Slice s;
    s.J = (unsigned)(gridDim.x / n_sets);
    s.set = blockIdx.x / s.J;
    s.rank = (unsigned)(blockIdx.x - s.set * s.J);
    const int64_t a = soff[s.set], n = soff[s.set + 1] - a;
    s.lo = a + n * s.rank / s.J;
    s.hi = a + n * (s.rank + 1) / s.J;
    return s;
}

// A barrier of the set's CTAs.
__device__ __forceinline__ void sync_set(const Slice &s) {
    if (s.J > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();
}

// f(rt, choice) for the samples [lo, hi) in no particular order: 16-byte loads
// where both arrays allow them (same offset from a 16-byte boundary), scalar
// loads at the ragged ends and otherwise.
template <class F>
__device__ __forceinline__ void for_each_sample(const float *rts, const int32_t *choices, int64_t lo, int64_t hi,
                                                F f) {
    const bool vec = ((((uintptr_t)rts ^ (uintptr_t)choices) & 15u) == 0);
    int64_t v0 = hi, v1 = hi;
    if (vec) {
        v0 = min(hi, lo + (int64_t)((4 - (((uintptr_t)(rts + lo) >> 2) & 3)) & 3));
        v1 = v0 + ((hi - v0) & ~(int64_t)3);
    }
    for (int64_t i = lo + threadIdx.x; i < v0; i += blockDim.x) f(rts[i], choices[i]);
#pragma unroll 4
    for (int64_t i = v0 + 4 * (int64_t)threadIdx.x; i < v1; i += 4 * (int64_t)blockDim.x) {
        const float4 r = *reinterpret_cast<const float4 *>(rts + i);
        const int4 c = *reinterpret_cast<const int4 *>(choices + i);
        f(r.x, c.x);
        f(r.y, c.y);
        f(r.z, c.z);
        f(r.w, c.w);
    }
    for (int64_t i = v1 + threadIdx.x; i < hi; i += blockDim.x) f(rts[i], choices[i]);
}

// Samples per choice, with and without omissions.  Bound by reading 8 bytes a
// sample: the counts stay in registers (one compare-and-add per choice; 32 bits
// hold a warp's share of a slice of 2^35 samples, more than the memory does), are
// summed over the warp by one reduction each, and the cluster's CTAs meet in
// rank 0.  Two 64-bit shared counters per choice, which every lane hit, had
// serialised the whole pass: 128 sets of 20 000 samples 831 us, 256 of 50 000
// 2 500 us.
template <int NC>
__global__ void __launch_bounds__(256) k_kde_count(const KdeFit a) {
    namespace cg = cooperative_groups;
    __shared__ unsigned long long tot[2 * NC];
    const Slice sl = set_slice(a.soff, a.n_sets);
    const ChoiceSet<NC> cs(a.cvals, a.nc);
    if (threadIdx.x < 2 * NC) tot[threadIdx.x] = 0ull;
    __syncthreads();
    unsigned int all[NC], val[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) all[c] = val[c] = 0u;
    for_each_sample(a.rts, a.choices, sl.lo, sl.hi, [&](float rt, int32_t ch) {
        const int ci = cs.index(ch);
        const bool kept = (rt != -999.f);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            all[c] += (ci == c);
            val[c] += (ci == c && kept);
        }
    });
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const unsigned int x = __reduce_add_sync(0xffffffffu, all[c]), y = __reduce_add_sync(0xffffffffu, val[c]);
        if (lane == 0) {
            atomicAdd(&tot[c], (unsigned long long)x);
            atomicAdd(&tot[NC + c], (unsigned long long)y);
        }
    }
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    if (sl.rank == 0 && threadIdx.x < a.nc) {
        int64_t x = 0, y = 0;
        for (unsigned j = 0; j < sl.J; ++j) {
            const unsigned long long *t = cl.map_shared_rank(tot, j);
            x += (int64_t)t[threadIdx.x];
            y += (int64_t)t[NC + threadIdx.x];
        }
        a.count_all[sl.set * a.nc + threadIdx.x] = x;
        a.n_valid[sl.set * a.nc + threadIdx.x] = y;
    }
    cl.sync();  // the slices' shared counters stay until rank 0 has read them
}

// Exclusive prefix sum of n int64 values into out[0..n] (one CTA of 1024).
__global__ void k_scan_i64(const int64_t *in, int64_t n, int64_t *out) {
    __shared__ int64_t warp_sum[32];
    __shared__ int64_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t base = 0; base < n; base += blockDim.x) {
        const int64_t i = base + threadIdx.x;
        const int64_t v = (i < n) ? in[i] : 0;
        int64_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int64_t w = (lane < (int)(blockDim.x >> 5)) ? warp_sum[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            warp_sum[lane] = w;  // inclusive warp prefix
        }
        __syncthreads();
        const int64_t excl = carry + (warp > 0 ? warp_sum[warp - 1] : 0) + x - v;
        if (i < n) out[i] = excl;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = excl + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) out[n] = carry;
}

// Sums over the points of the set's groups by its whole cluster: f(c, x) over group
// c's points (or displaced bandwidth inputs), the total of choice c to out[c].  The
// points' rows of 32 go round KDE_PLACES places, and the cluster's warps share the
// places, K = KDE_PLACES / (8 J) to a warp with their loads in flight together.  A
// place's sum and the sum of the places are the same additions whatever J is, so
// a set's moments have the same bits in any call.
constexpr int KDE_PLACES = 64;  // the warps of the largest cluster
template <int NC, int K, class F>
__device__ __forceinline__ void sum_places(const KdeFit &a, const Slice &sl, double *place, F f) {
    constexpr int WARPS = KDE_PLACES / K;
    const int lane = threadIdx.x & 31, gw = (int)(sl.rank * 8 + (threadIdx.x >> 5));
    for (int c = 0; c < a.nc; ++c) {
        const int64_t g = sl.set * a.nc + c, lo = a.poff[g], n = a.poff[g + 1] - lo;
        const int first = (gw - c) & (WARPS - 1);  // small groups of different choices go to different warps
        if (32 * first >= n) continue;
        const double *bw = a.bwvals ? a.bwvals + lo : nullptr;
        const float *pt = a.points + lo;
        double t[K];
#pragma unroll
        for (int k = 0; k < K; ++k) t[k] = 0.0;
        for (int64_t i = 32 * first + lane; i < n; i += 32 * KDE_PLACES) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int64_t at = i + 32 * WARPS * k;
                if (at < n) t[k] += f(c, bw ? __ldcg(bw + at) : (double)__ldcg(pt + at));
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int k = 0; k < K; ++k) t[k] += __shfl_down_sync(0xffffffffu, t[k], o);
        }
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < K; ++k) place[c * KDE_PLACES + first + WARPS * k] = t[k];
        }
    }
}
// (place: NC * KDE_PLACES values of shared memory that no other CTA of the cluster
// still reads; ends with a barrier of the CTA alone)
template <int NC, class F>
__device__ __forceinline__ void sum_points(const KdeFit &a, const Slice &sl, double *place, double *out, F f) {
    switch (sl.J) {
        case 1: sum_places<NC, 8>(a, sl, place, f); break;
        case 2: sum_places<NC, 4>(a, sl, place, f); break;
        case 4: sum_places<NC, 2>(a, sl, place, f); break;
        default: sum_places<NC, 1>(a, sl, place, f); break;
    }
    sync_set(sl);
    const int lane = threadIdx.x & 31;
    for (int c = threadIdx.x >> 5; c < a.nc; c += 8) {
        const int64_t n = a.poff[sl.set * a.nc + c + 1] - a.poff[sl.set * a.nc + c];
        double t = 0.0;
#pragma unroll
        for (int v = lane; v < KDE_PLACES; v += 32)
            if (32 * v < n)
                t += cooperative_groups::this_cluster().map_shared_rank(
                    place, ((v + c) & (8 * sl.J - 1)) >> 3)[c * KDE_PLACES + v];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) out[c] = t;
    }
    __syncthreads();
}

// Stable per-choice compaction of log(rt - shift) into the group regions, then
// Silverman's bandwidth (kde_class.py:508-553) and the normaliser of each group.
//
// Each CTA of the set's cluster first counts its own slice (the samples are in
// L2 after k_kde_count), so its first position per choice follows from the
// lower ranks' counts; then it walks the slice in chunks of 1 024 samples, four
// consecutive ones per thread.  Ranks inside a chunk come from a warp scan of
// byte-packed counts (four choices in one word, at most 128 each) and the warps'
// totals, one barrier per chunk.  Mean and squared deviations are two passes over
// the group's points, still in L2, shared by the cluster (sum_points).  What
// remains is the float64 logarithm of every sample.  One CTA per set with a barrier
// pair per 256 samples and the moments in a kernel of their own had taken 87 + 13 us
// for 128 sets of 20 000 samples and 348 + 45 us for 256 of 50 000.  The whole fit, us,
// with the mean's sums taken on the way (in an order that followed the cluster's size)
// and now: those two 88 and 236, now 84 and 233; two million samples in one set 995,
// now 818; 1 000 sets of 100 000 1 328, now 1 405; 5 000 sets of 200 122, now 134; four
// choices 1 934, now 1 798, and 192, now 169.
template <int NC>
__global__ void __launch_bounds__(256, NC == 2 ? 6 : NC == 4 ? 5 : 3) k_kde_scatter(const KdeFit a) {
    namespace cg = cooperative_groups;
    constexpr int W = 8, NW = (NC + 3) / 4;
    __shared__ unsigned long long tot[NC];
    __shared__ __align__(16) unsigned int wtot[2][NW][W];
    __shared__ double place[2][NC * KDE_PLACES], mean[NC], dev[NC];
    cg::cluster_group cl = cg::this_cluster();
    const Slice sl = set_slice(a.soff, a.n_sets);
    const ChoiceSet<NC> cs(a.cvals, a.nc);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double sh = a.shift ? a.shift[sl.set] : 0.0;

    // this slice's counts, then the position of its first sample of each choice
    int64_t base[NC];
    {
        if (threadIdx.x < NC) tot[threadIdx.x] = 0ull;
        __syncthreads();
        if (sl.J > 1) {
            unsigned int val[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) val[c] = 0u;
            for_each_sample(a.rts, a.choices, sl.lo, sl.hi, [&](float rt, int32_t ch) {
                const int ci = (rt != -999.f) ? cs.index(ch) : -1;
#pragma unroll
                for (int c = 0; c < NC; ++c) val[c] += (ci == c);
            });
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const unsigned int y = __reduce_add_sync(0xffffffffu, val[c]);
                if (lane == 0) atomicAdd(&tot[c], (unsigned long long)y);
            }
        }
        cl.sync();
#pragma unroll
        for (int c = 0; c < NC; ++c) base[c] = (c < a.nc) ? a.poff[sl.set * a.nc + c] : 0;
        for (unsigned j = 0; j < sl.rank; ++j) {
            const unsigned long long *t = cl.map_shared_rank(tot, j);
#pragma unroll
            for (int c = 0; c < NC; ++c) base[c] += (int64_t)t[c];
        }
    }
    const bool vec = ((((uintptr_t)a.rts ^ (uintptr_t)a.choices) & 15u) == 0);
    const int64_t start = sl.lo - (int64_t)(((uintptr_t)(a.rts + sl.lo) >> 2) & 3);  // 16-byte boundary at or before lo
    int buf = 0;
    for (int64_t c0 = start; c0 < sl.hi; c0 += 1024, buf ^= 1) {
        const int64_t i0 = c0 + 4 * threadIdx.x;
        float rt[4];
        int ci[4];
        if (vec && i0 >= sl.lo && i0 + 4 <= sl.hi) {
            const float4 r = *reinterpret_cast<const float4 *>(a.rts + i0);
            const int4 h = *reinterpret_cast<const int4 *>(a.choices + i0);
            rt[0] = r.x; rt[1] = r.y; rt[2] = r.z; rt[3] = r.w;
            ci[0] = cs.index(h.x); ci[1] = cs.index(h.y); ci[2] = cs.index(h.z); ci[3] = cs.index(h.w);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool in = (i0 + q >= sl.lo) && (i0 + q < sl.hi);
                rt[q] = in ? a.rts[i0 + q] : -999.f;
                ci[q] = in ? cs.index(a.choices[i0 + q]) : -1;
            }
        }
        unsigned int own[NW], inc[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) own[w] = 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (rt[q] == -999.f) ci[q] = -1;
#pragma unroll
            for (int c = 0; c < NC; ++c) own[c / 4] += (ci[q] == c) ? (1u << (8 * (c % 4))) : 0u;
        }
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            inc[w] = own[w];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int y = __shfl_up_sync(0xffffffffu, inc[w], o);
                if (lane >= o) inc[w] += y;
            }
            if (lane == 31) wtot[buf][w][warp] = inc[w];
        }
        __syncthreads();  // the other buffer's readers are past it once everybody is here
        int64_t pos[NC];
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            // the eight warps' totals as 16-bit fields: choices 4w, 4w+2 and 4w+1, 4w+3
            unsigned int pe = 0, po = 0, te = 0, to = 0;
#pragma unroll
            for (int k = 0; k < W; ++k) {
                const unsigned int x = wtot[buf][w][k], e = x & 0x00ff00ffu, o = (x >> 8) & 0x00ff00ffu;
                te += e;
                to += o;
                pe += (k < warp) ? e : 0u;
                po += (k < warp) ? o : 0u;
            }
            const unsigned int ex = inc[w] - own[w];
            pe += ex & 0x00ff00ffu;
            po += (ex >> 8) & 0x00ff00ffu;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int c = 4 * w + q;
                if (c < NC) {
                    pos[c] = base[c] + (((q & 1) ? po : pe) >> (16 * (q / 2)) & 0xffffu);
                    base[c] += ((q & 1) ? to : te) >> (16 * (q / 2)) & 0xffffu;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (ci[q] < 0) continue;
            int64_t at = 0;
#pragma unroll
            for (int c = 0; c < NC; ++c)
                if (ci[q] == c) at = pos[c]++;
            // kernels sit on float32 log of the float32 (displaced) rt; with a
            // shift the rt is displaced in float64 and stored as float32, and the
            // bandwidth uses log(exp(float32 log rt) - shift) in float64
            // (kde_class.py:174-186, 478-493)
            const float r = a.shift ? __double2float_rn((double)rt[q] - sh) : rt[q];
            const float x = __double2float_rn(log((double)r));
            a.points[at] = x;
            if (a.bwvals) a.bwvals[at] = log(exp((double)__double2float_rn(log((double)rt[q]))) - sh);
        }
    }
    sync_set(sl);  // orders the cluster's point writes before the reads below
    sum_points<NC>(a, sl, place[0], mean, [](int, double x) { return x; });
    if ((int)threadIdx.x < a.nc) {
        const int64_t g = sl.set * a.nc + threadIdx.x, n = a.poff[g + 1] - a.poff[g];
        mean[threadIdx.x] /= (double)(n > 0 ? n : 1);
    }
    __syncthreads();
    sum_points<NC>(a, sl, place[1], dev, [&](int c, double x) {
        const double d = x - mean[c];
        return d * d;
    });
    if (sl.rank == 0 && threadIdx.x < a.nc) {
        const int c = threadIdx.x;
        const int64_t g = sl.set * a.nc + c, n = a.poff[g + 1] - a.poff[g];
        const int64_t N = a.soff[sl.set + 1] - a.soff[sl.set];
        const double ss = dev[c];
        const double var = ss / (double)(n > 0 ? n : 1);
        const double p = (N > 0) ? (double)a.count_all[g] / (double)N : 0.0;
        a.prop[g] = p;
        if (n == 0) {
            a.h[g] = -1.0;
            a.lognorm[g] = 0.0;
        } else {
            double sd = (n > 1) ? sqrt(var) : 10.0;
            if (n > 1 && sd < 1e-3) sd = 1e-3;
            const double h = pow(4.0 / (3.0 * (double)n), 0.2) * sd;
            a.h[g] = h;
            a.lognorm[g] = log(p) - log((double)n) - log(h) - 0.5 * KDE_LOG_2PI;
        }
    }
    sync_set(sl);  // the others have read this CTA's places
}

struct KdeEval {
    const float *points;
    const int64_t *poff;
    const double *h, *lognorm;
    const int64_t *qoff;  // [G + 1] queries sorted by group
    const double *q_rt;
    double *out;
    int nc;
    int64_t G;
    const int64_t *soff;
    const double *shift;
    double lb, eps, max_t;
    // Stream-K schedule (see k_kde_plan): units are (group, up to KDE_ROWS rows
    // of 32 queries); unit u's cost span is [ioff[u], ioff[u + 1]).
    int64_t *head;     // [3] number of units, total cost, CTAs that share it
    int64_t *ioff;     // [u_max + 1]
    int32_t *ugroup;   // [u_max] the unit's group
    int32_t *uidx;     // [u_max] its place among the group's units
    int32_t *tail;     // [P] unit whose first part CTA c holds (-1: none)
    int32_t *link;     // [P] what CTA c holds of the unit begun before it (SPLIT_*)
    int64_t u_max;     // capacity of the unit arrays
    double *slots;     // [P][2][KDE_QT] partial sums of units split between CTAs
    int64_t P;         // CTAs of the evaluation grid
};

constexpr int KDE_TILE = 512;     // points staged in shared memory at a time (a multiple of 32)
constexpr int KDE_THREADS = 128;
constexpr int KDE_ROWS = 16;      // rows of 32 queries per unit, four per warp at most
constexpr int KDE_QT = 32 * KDE_ROWS;
enum { SPLIT_PART = 1, SPLIT_LAST = 2, SPLIT_NONE = 3 };

__device__ __forceinline__ int64_t upper_index(const int64_t *off, int64_t n, int64_t x) {
    // largest i in [0, n) with off[i] <= x (off non-decreasing, off[0] <= x)
    int64_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (off[mid] <= x) lo = mid; else hi = mid;
    }
    return lo;
}

// Rows of 32 queries [r0, r1) of unit k of a group with m queries: the
// group's ceil(m / 32) rows spread evenly over its ceil(m / KDE_QT) units.
struct UnitRows {
    int64_t r0, r1;
};
__device__ __forceinline__ int64_t group_units(int64_t m) { return m > 0 ? (m + KDE_QT - 1) / KDE_QT : 0; }
__device__ __forceinline__ UnitRows unit_rows(int64_t m, int64_t k) {
    const int64_t rows = (m + 31) / 32, T = group_units(m);
    return {rows * k / T, rows * (k + 1) / T};
}
__device__ __forceinline__ int64_t point_tiles(int64_t n) { return n > 0 ? (n + KDE_TILE - 1) / KDE_TILE : 1; }

// The Stream-K schedule, by one CTA: a unit of R rows costs R + 1 per point
// tile (the 1 for staging the tile), a group's units R_group + T in all, so one
// two-value scan over the groups places every unit.  A thread writes its own
// group's units; one with more than KDE_OWN_UNITS shares them among its warp's
// lanes, since unit k begins tiles (rows before it + k) into the group's cost and
// needs no other.  (One thread for all of a group's units: a single group of 1 000
// points and 1 M queries, 1 954 units, 729 us for the whole evaluation; now 345.
// Dealing all units of all groups to all threads by search cost the usual call, 256
// groups of one unit, 5 us.)
constexpr int KDE_OWN_UNITS = 4;
__global__ void __launch_bounds__(1024) k_kde_plan(const KdeEval a) {
    __shared__ int64_t wu[32], wi[32];
    __shared__ int64_t wt[32];
    int64_t n_tiles = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t cu = 0, ci = 0;  // units and cost of the groups before this pass
    for (int64_t b = 0; b < a.G; b += blockDim.x) {
        const int64_t g = b + threadIdx.x;
        int64_t m = 0, T = 0, tiles = 0, cost = 0;
        if (g < a.G) {
            m = a.qoff[g + 1] - a.qoff[g];
            T = group_units(m);
            tiles = point_tiles(a.poff[g + 1] - a.poff[g]);
            cost = (m > 0) ? tiles * ((m + 31) / 32 + T) : 0;
            n_tiles += tiles * T;
        }
        int64_t x = T, y = cost;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t p = __shfl_up_sync(0xffffffffu, x, o), q = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) {
                x += p;
                y += q;
            }
        }
        __syncthreads();
        if (lane == 31) {
            wu[warp] = x;
            wi[warp] = y;
        }
        __syncthreads();
        if (warp == 0) {
            int64_t p = wu[lane], q = wi[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t pp = __shfl_up_sync(0xffffffffu, p, o), qq = __shfl_up_sync(0xffffffffu, q, o);
                if (lane >= o) {
                    p += pp;
                    q += qq;
                }
            }
            wu[lane] = p;
            wi[lane] = q;
        }
        __syncthreads();
        int64_t u = cu + (warp > 0 ? wu[warp - 1] : 0) + x - T;
        int64_t i = ci + (warp > 0 ? wi[warp - 1] : 0) + y - cost;
        unsigned many = __ballot_sync(0xffffffffu, T > KDE_OWN_UNITS);
        if (T <= KDE_OWN_UNITS) {
            for (int64_t k = 0; k < T && u < a.u_max; ++k, ++u) {
                const UnitRows r = unit_rows(m, k);
                a.ioff[u] = i;
                a.ugroup[u] = (int32_t)g;
                a.uidx[u] = (int32_t)k;
                i += tiles * (r.r1 - r.r0 + 1);
            }
        }
        for (; many != 0u; many &= many - 1u) {
            const int src = __ffs(many) - 1;
            const int64_t gm = __shfl_sync(0xffffffffu, m, src), gT = __shfl_sync(0xffffffffu, T, src);
            const int64_t gt = __shfl_sync(0xffffffffu, tiles, src), gi = __shfl_sync(0xffffffffu, i, src);
            const int64_t gu = __shfl_sync(0xffffffffu, u, src);
            for (int64_t k = lane; k < gT && gu + k < a.u_max; k += 32) {
                a.ioff[gu + k] = gi + gt * (unit_rows(gm, k).r0 + k);
                a.ugroup[gu + k] = (int32_t)(g - lane + src);
                a.uidx[gu + k] = (int32_t)k;
            }
        }
        cu += wu[31];
        ci += wi[31];
    }
    for (int o = 16; o > 0; o >>= 1) n_tiles += __shfl_down_sync(0xffffffffu, n_tiles, o);
    if (lane == 0) wt[warp] = n_tiles;
    __syncthreads();
    if (threadIdx.x == 0) {
        a.head[0] = min(cu, a.u_max);
        a.head[1] = ci;
        // no more CTAs than tiles: a unit cut between CTAs without a tile each
        // would only make the fix-up's chain longer (one set of
        // 20 000 points, 1 000 queries: fix-up 108 -> 12 us)
        n_tiles = 0;
        for (int w = 0; w < 32; ++w) n_tiles += wt[w];
        a.head[2] = min(a.P, n_tiles);
        a.ioff[min(cu, a.u_max)] = ci;
    }
}

// first cost index of CTA c: floor(c * I / P) (c <= P < 2^16 and I < 2^46, so
// the product fits in 64 bits)
__device__ __forceinline__ int64_t sk_begin(int64_t c, int64_t I, int64_t P) {
    return (c * I) / P;
}

// log-likelihood of one query from its kernel sum acc (kde_class.py:188-329)
__device__ __forceinline__ double kde_finalize(const KdeEval &a, int64_t g, int64_t n, double acc,
                                               double disp, double lq) {
    const int64_t s = g / a.nc;
    double ll;
    if (n == 0) {
        // choice without base data: log(1 / n_trials) + log(1 / max_t)
        ll = -log((double)(a.soff[s + 1] - a.soff[s]) * a.max_t);
    } else if (!(disp > 0.0)) {
        ll = a.lb;
    } else {
        ll = a.lognorm[g] + log(acc) - lq;
        if (!(ll > a.lb)) ll = a.lb;
    }
    return ll;
}

__device__ __forceinline__ float ex2_neg_sum(uint64_t e) {  // 2^-lo + 2^-hi
    float lo, hi, r0, r1;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(e));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(-lo));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(-hi));
    return r0 + r1;
}

// Kernel sums of NJ queries per lane over one staged tile of 32 * n32 points
// (padding points weigh exactly 0): float over 32 terms, then float64.
template <int NJ>
__device__ __forceinline__ void kde_tile(const float *tile, int n32, const float *qhi, const float *qlo, float sc,
                                         double *acc) {
    const uint64_t minus1 = pack_f2(-1.f, -1.f), sc2 = pack_f2(sc, sc);
    uint64_t h2[NJ], l2[NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        h2[j] = pack_f2(qhi[j], qhi[j]);
        l2[j] = pack_f2(qlo[j], qlo[j]);
    }
    const ulonglong2 *t4 = reinterpret_cast<const ulonglong2 *>(tile);
#pragma unroll 1
    for (int k0 = 0; k0 < n32; ++k0) {
        float part[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) part[j] = 0.f;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
            const ulonglong2 x = t4[8 * k0 + kk];
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const uint64_t a = mul_f2(add_f2(fma_f2(x.x, minus1, h2[j]), l2[j]), sc2);
                const uint64_t b = mul_f2(add_f2(fma_f2(x.y, minus1, h2[j]), l2[j]), sc2);
                part[j] += ex2_neg_sum(mul_f2(a, a)) + ex2_neg_sum(mul_f2(b, b));
            }
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[j] += (double)part[j];
    }
}

// Lanes hold queries (q split into float hi + lo parts so q - x_j keeps full
// precision), the group's points stream through shared memory one tile at a
// time, and each kernel term is ex2(-(d s)^2).  Bound by the SFU: one ex2 per
// term, 16 a clock and SM.  A unit's rows of 32 queries go round the CTA's four
// warps (up to four each, the first warp rotating with the unit), so a group
// pays for its queries to a multiple of 32 instead of 512, and the rest of a
// term -- subtract, add the low part, scale, square -- is packed two points to
// an instruction: 4 issue slots a term against the SFU's 8 clocks a warp (6 and
// the tail's selects before).  Measured, 256 groups of about 10 000 points
// and 500 queries each: 763 -> 476 us (XU pipe 83 % of the active cycles); 512 of
// 25 000 points and 450 queries: 3 530 -> 2 538 us.  7 CTAs per SM: 479 us, 6: 497,
// 8: 509.  Tiles of 2 048, 1 024, 512 and 256 points: 530, 479, 472 and 468 us,
// and on a single set of 20 000 points 49, 37, 22 and 20 us.
__global__ void __launch_bounds__(KDE_THREADS, 7) k_kde_eval(const KdeEval a) {
    __shared__ __align__(16) float tile[KDE_TILE];
    const int64_t U = a.head[0], I = a.head[1], P = a.head[2];
    const int64_t c = blockIdx.x;
    const int64_t i0 = (c < P) ? sk_begin(c, I, P) : I, i1 = (c < P) ? sk_begin(c + 1, I, P) : I;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int tail = -1;
    if (threadIdx.x == 0) a.link[c] = SPLIT_NONE;
    if (i0 < i1) {
        for (int64_t u = upper_index(a.ioff, U, i0); u < U; ++u) {
            const int64_t ubeg = a.ioff[u], uend = a.ioff[u + 1];
            if (ubeg >= i1) break;
            const int64_t g = a.ugroup[u], qa = a.qoff[g], q1 = a.qoff[g + 1];
            const UnitRows rows = unit_rows(q1 - qa, a.uidx[u]);
            const int R = (int)(rows.r1 - rows.r0);
            const int64_t p0 = a.poff[g], n = a.poff[g + 1] - p0, tiles = point_tiles(n);
            // this CTA computes the tiles whose first cost index is in [i0, i1)
            const int64_t t0 = (i0 > ubeg) ? (i0 - ubeg + R) / (R + 1) : 0;
            const int64_t t1 = (i1 < uend) ? min((i1 - ubeg + R) / (R + 1), tiles) : tiles;
            if (t0 >= t1) continue;
            if (i0 > ubeg && threadIdx.x == 0) a.link[c] = (t1 == tiles) ? SPLIT_LAST : SPLIT_PART;
            const int64_t q0 = qa + 32 * rows.r0;
            const int first = (warp - (int)u) & 3;                 // this warp's rows: first, first + 4, ...
            const int nj = (first < R) ? (R - first + 3) >> 2 : 0;
            const double sh = a.shift ? a.shift[g / a.nc] : 0.0;
            // 2^(-(d*sc)^2) = exp(-d^2 / (2 h^2))
            const float sc = (n > 0) ? (float)(0.8493218002880191 / a.h[g]) : 0.f;  // sqrt(log2(e)/2) / h
            float qhi[4], qlo[4];
            double acc[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int64_t qi = q0 + 32 * (first + 4 * j) + lane;
                const double lq = log(fmax((j < nj && qi < q1) ? a.q_rt[qi] - sh : 1.0, a.eps));
                qhi[j] = (float)lq;
                qlo[j] = (float)(lq - (double)qhi[j]);
                acc[j] = 0.0;
            }
            for (int64_t t = t0; t < t1 && n > 0; ++t) {
                const int64_t b0 = t * KDE_TILE;
                const int cnt = (int)min((int64_t)KDE_TILE, n - b0), n32 = (cnt + 31) >> 5;
                __syncthreads();
                for (int i = threadIdx.x; i < 32 * n32; i += KDE_THREADS)
                    tile[i] = (i < cnt) ? __ldg(a.points + p0 + b0 + i) : 1e30f;  // padding: zero weight
                __syncthreads();
                switch (nj) {
                    case 4: kde_tile<4>(tile, n32, qhi, qlo, sc, acc); break;
                    case 3: kde_tile<3>(tile, n32, qhi, qlo, sc, acc); break;
                    case 2: kde_tile<2>(tile, n32, qhi, qlo, sc, acc); break;
                    case 1: kde_tile<1>(tile, n32, qhi, qlo, sc, acc); break;
                    default: break;
                }
            }
            const bool whole = (t0 == 0 && t1 == tiles);
            // split unit: slot 0 if it began in an earlier CTA, else slot 1
            double *slot = a.slots + (c * 2 + (t0 > 0 ? 0 : 1)) * KDE_QT;
            if (!whole && t0 == 0) tail = (int)u;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j >= nj) continue;
                const int r = 32 * (first + 4 * j) + lane;
                const int64_t qi = q0 + r;
                if (!whole) {
                    slot[r] = acc[j];
                } else if (qi < q1) {
                    const double disp = a.q_rt[qi] - sh;
                    a.out[qi] = kde_finalize(a, g, n, acc[j], disp, log(fmax(disp, a.eps)));
                }
            }
        }
    }
    if (threadIdx.x == 0) a.tail[c] = tail;
}

// Units split between CTAs, one block per CTA that holds a first part: the
// partial sums are added in CTA order (a fixed order, so results do not
// depend on timing) and finalised.
__global__ void __launch_bounds__(KDE_THREADS) k_kde_fixup(const KdeEval a) {
    const int64_t c = blockIdx.x;
    const int u = a.tail[c];
    if (u < 0) return;
    const int64_t g = a.ugroup[u], qa = a.qoff[g], q1 = a.qoff[g + 1];
    const UnitRows rows = unit_rows(q1 - qa, a.uidx[u]);
    const int nq = 32 * (int)(rows.r1 - rows.r0);
    const int64_t q0 = qa + 32 * rows.r0, n = a.poff[g + 1] - a.poff[g];
    const double sh = a.shift ? a.shift[g / a.nc] : 0.0;
    for (int r = threadIdx.x; r < nq; r += KDE_THREADS) {
        const int64_t qi = q0 + r;
        if (qi >= q1) continue;
        double acc = a.slots[(c * 2 + 1) * KDE_QT + r];
        bool more = true;
        for (int64_t cc = c + 1; cc < a.P && more; cc += 4) {
            int l[4];
            double v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // four links and sums in flight
                l[k] = (cc + k < a.P) ? a.link[cc + k] : SPLIT_LAST;
                v[k] = (cc + k < a.P) ? a.slots[(cc + k) * 2 * KDE_QT + r] : 0.0;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (more && l[k] != SPLIT_NONE) acc += v[k];
                more = more && l[k] != SPLIT_LAST;
            }
        }
        const double disp = a.q_rt[qi] - sh;
        a.out[qi] = kde_finalize(a, g, n, acc, disp, log(fmax(disp, a.eps)));
    }
}

// Queries / samples per group: slots [o[g], o[g] + nk[g]) get KDE samples
// (point j ~ U{0..n-1}, log-rt + h N(0,1), exponentiated, plus the shift);
// the following nu[g] slots get U(ulo, uhi) rts.  Groups without data draw
// their KDE part from U(0, max_t) as the reference does.
struct KdeSample {
    PhiloxKeys key;
    const float *points;
    const int64_t *poff;
    const double *h;
    const int64_t *ooff;    // [G + 1] output slots per group
    const int64_t *nkde;    // [G] KDE samples at the start of each group's slots
    int64_t n_groups;
    const double *shift;
    int nc;
    double max_t, ulo, uhi;
    double *out_rt;
};

__device__ __forceinline__ double u53(uint32_t a, uint32_t b) {
    return ((double)(a >> 5) * 67108864.0 + (double)(b >> 6)) * (1.0 / 9007199254740992.0);
}

__global__ void k_kde_sample(const KdeSample a) {
    const int64_t total = a.ooff[a.n_groups];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t lo = 0, hi = a.n_groups;  // ooff[lo] <= i < ooff[hi]
        while (hi - lo > 1) {
            const int64_t mid = (lo + hi) >> 1;
            if (a.ooff[mid] <= i) lo = mid; else hi = mid;
        }
        const int64_t g = lo, j = i - a.ooff[g];
        const uint4 r = philox10(make_uint4((uint32_t)j, (uint32_t)g, (uint32_t)(g >> 32), 7u), a.key);
        const double sh = a.shift ? a.shift[g / a.nc] : 0.0;
        const int64_t n = a.poff[g + 1] - a.poff[g];
        double rt;
        if (j < a.nkde[g]) {
            if (n > 0) {
                int64_t idx = (int64_t)(u53(r.x, r.y) * (double)n);
                if (idx >= n) idx = n - 1;
                const float2 z = box_muller(r.z, r.w);
                rt = exp((double)a.points[a.poff[g] + idx] + a.h[g] * (double)z.x) + sh;
            } else {
                rt = u53(r.x, r.y) * a.max_t + sh;
            }
        } else {
            rt = a.ulo + u53(r.x, r.y) * (a.uhi - a.ulo);
        }
        a.out_rt[i] = rt;
    }
}

// Training records (ResampleMixtureStrategy layout): per set s, rows
// [theta_0..theta_{P-1}, rt, choice, loglik] as float32.  The evaluated
// queries of the set's groups come first, then n_down rows with
// rt ~ U(-1, 0.0001), a uniformly drawn choice and loglik = neg_ll; rows are
// shuffled within the set (Fisher-Yates driven by Philox).
struct KdeRecords {
    PhiloxKeys key;
    const float *theta;  // [S, P]
    int P;
    int64_t n_sets;
    const int64_t *qoff;  // [G + 1]
    const double *q_rt, *q_ll;
    const int32_t *cvals;
    int nc;
    int64_t n_down;  // per set
    int64_t rows_per_set;
    float neg_ll;
    float *out;      // [S * rows_per_set, P + 3]
};

// The Fisher-Yates shuffle "for i = M-1 .. 1: swap(perm[i], perm[j_i])" in
// parallel rounds with the result of the sequential loop (deterministic
// reservations: Shun, Gu, Blelloch, Fineman & Gibbons, SODA'15): every swap not
// yet done bids for its two places, the earliest swap (largest i) wins a place,
// and a swap that won both is done.  About log M rounds instead of M dependent
// swaps by one thread: 256 sets of 1 000 rows, 137 -> 27 us.
__global__ void __launch_bounds__(256) k_kde_records(const KdeRecords a) {
    extern __shared__ int bid[];  // [M] bids, then [M] 16-bit places and [M] 16-bit partners
    const int64_t s = blockIdx.x;
    const int M = (int)a.rows_per_set;
    uint16_t *perm = reinterpret_cast<uint16_t *>(bid + M), *other = perm + M;
    const int64_t qa = a.qoff[s * a.nc], qb = a.qoff[(s + 1) * a.nc];
    for (int i = threadIdx.x; i < M; i += blockDim.x) {
        const uint4 r = philox10(make_uint4((uint32_t)i, (uint32_t)s, (uint32_t)(s >> 32), 9u), a.key);
        const int j = (int)(u53(r.x, r.y) * (double)(i + 1));
        perm[i] = (uint16_t)i;
        other[i] = (uint16_t)(j <= i ? j : i);
        bid[i] = 0;
    }
    // this thread's swaps i = threadIdx.x + k blockDim.x not yet done, one bit each (i = 0 is none)
    static_assert(KDE_MAX_ROWS <= 64 * 256, "one bit per swap of a thread");
    unsigned long long open = 0ull;
    for (int i = threadIdx.x, k = 0; i < M; i += blockDim.x, ++k)
        if (i > 0) open |= 1ull << k;
    __syncthreads();
    for (int round = 1;; ++round) {
        // a later round's bids beat all earlier ones, so nothing is cleared (M < 2^14, rounds <= M)
        for (unsigned long long m = open; m; m &= m - 1) {
            const int i = threadIdx.x + (__ffsll((long long)m) - 1) * (int)blockDim.x;
            atomicMax(&bid[i], (round << 14) | i);
            atomicMax(&bid[other[i]], (round << 14) | i);
        }
        __syncthreads();
        for (unsigned long long m = open; m; m &= m - 1) {
            const int k = __ffsll((long long)m) - 1, i = threadIdx.x + k * (int)blockDim.x, j = other[i];
            const int mine = (round << 14) | i;
            if (bid[i] == mine && bid[j] == mine) {
                const uint16_t t = perm[i];
                perm[i] = perm[j];
                perm[j] = t;
                open &= ~(1ull << k);
            }
        }
        if (!__syncthreads_or(open != 0ull)) break;
    }
    const int W = a.P + 3;
    for (int i = threadIdx.x; i < M; i += blockDim.x) {
        float *row = a.out + (s * M + perm[i]) * W;
        for (int p = 0; p < a.P; ++p) row[p] = a.theta[s * a.P + p];
        float rt, ch, ll;
        const int64_t q = qa + i;
        if (q < qb) {
            int64_t c = 0;  // group of query q within this set
            while (c + 1 < a.nc && a.qoff[s * a.nc + c + 1] <= q) ++c;
            rt = (float)a.q_rt[q];
            ch = (float)a.cvals[c];
            ll = (float)a.q_ll[q];
        } else {
            const uint4 r = philox10(make_uint4((uint32_t)i, (uint32_t)s, (uint32_t)(s >> 32), 11u), a.key);
            rt = (float)(-1.0 + u53(r.x, r.y) * (0.0001 + 1.0));
            ch = (float)a.cvals[min((int)(u53(r.z, r.w) * a.nc), a.nc - 1)];
            ll = a.neg_ll;
        }
        row[a.P] = rt;
        row[a.P + 1] = ch;
        row[a.P + 2] = ll;
    }
}

// Per-set summaries for the auxiliary labels of the data pipeline
// (simulation_pipeline.py:262-351): choice counts, the pipeline's omission
// count (choices equal to -999), no-go count ((choice != max choice) or rt ==
// -999) and per-choice rt histograms over np.linspace(0, max_t, nb + 1) with
// numpy's index rules (right edge inclusive in the last bin, float64 edges,
// +-1 corrections at the edges), omissions excluded.
struct SetSummary {
    const float *rts;
    const int32_t *choices;
    int64_t n_sets;
    const int64_t *soff;
    const int32_t *cvals;
    int nc;
    double max_t;
    int64_t *counts, *nogo, *omit;
    int nb_a, nb_b;
    float *hist_a, *hist_b;
};

// numpy.histogram's bin of v over linspace(0, max_t, nb + 1) (step = max_t / nb
// in float64): the i with i step <= v < (i + 1) step, the last bin closed; -1
// outside.  A float32 guess, then moved to the bin whose float64 edges hold v.
__device__ __forceinline__ int np_hist_index(float rt, double max_t, double step, float inv_step, int nb) {
    const double v = (double)rt;
    if (!(v >= 0.0) || !(v <= max_t)) return -1;
    int i = max(min((int)(rt * inv_step), nb - 1), 0);
    while (i > 0 && v < (double)i * step) --i;
    while (i < nb - 1 && v >= (double)(i + 1) * step) ++i;
    return i;
}

// One pass over a set's samples by its cluster: counts in registers, the
// histograms as 32-bit shared counters per CTA (equal bins of a warp are added
// up by the hardware), added over the cluster at the end.  A slice of more than
// 2^31 samples is counted in parts, after each of which the counters' top bits move
// to a byte of their own (the memory holds less than 2^35 samples).  A histogram with half
// the bins of the other is its pairwise sum (its edges are every second one,
// exactly: the steps differ by a power of two).  64-bit shared counters hit by
// every lane and two float64 divisions per sample: 256 sets of 50 000 samples
// 2 176 -> 50 us.
template <int NC>
__global__ void __launch_bounds__(256) k_set_summary(const SetSummary a) {
    namespace cg = cooperative_groups;
    extern __shared__ unsigned int sh[];  // [nc * (nb_a + nb_b)] histogram counters, then a byte of 2^31s each
    __shared__ unsigned long long cnt[NC + 2];  // choices, no-go, omissions
    cg::cluster_group cl = cg::this_cluster();
    const Slice sl = set_slice(a.soff, a.n_sets);
    const ChoiceSet<NC> cs(a.cvals, a.nc);
    const int H = a.nc * (a.nb_a + a.nb_b);
    const bool pairs = (a.nb_b == 2 * a.nb_a);
    const double step_a = a.max_t / (double)a.nb_a, step_b = a.max_t / (double)a.nb_b;
    const float inv_a = (float)(1.0 / step_a), inv_b = (float)(1.0 / step_b);
    unsigned int *hb = sh + a.nc * a.nb_a;
    unsigned char *top = reinterpret_cast<unsigned char *>(sh + H);
    constexpr int64_t PART = (int64_t)1 << 31;
    const bool parts = sl.hi - sl.lo > PART;
    int32_t max_choice = cs.v[0];
#pragma unroll
    for (int c = 1; c < NC; ++c)
        if (c < a.nc) max_choice = max(max_choice, cs.v[c]);
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        sh[i] = 0u;
        top[i] = 0;
    }
    if (threadIdx.x < NC + 2) cnt[threadIdx.x] = 0ull;
    __syncthreads();
    unsigned int n[NC], nogo = 0u, omit = 0u;
#pragma unroll
    for (int c = 0; c < NC; ++c) n[c] = 0u;
    const auto sample = [&](float rt, int32_t ch) {
        const bool omitted = (rt == -999.f);
        omit += (ch == -999);
        nogo += (ch != max_choice || omitted);
        const int c = cs.index(ch);
#pragma unroll
        for (int k = 0; k < NC; ++k) n[k] += (c == k);
        if (c < 0 || omitted) return;
        const int ib = np_hist_index(rt, a.max_t, step_b, inv_b, a.nb_b);
        if (ib >= 0) atomicAdd(&hb[c * a.nb_b + ib], 1u);
        if (!pairs) {
            const int ia = np_hist_index(rt, a.max_t, step_a, inv_a, a.nb_a);
            if (ia >= 0) atomicAdd(&sh[c * a.nb_a + ia], 1u);
        }
    };
    for (int64_t lo = sl.lo; lo < sl.hi; lo += PART) {
        for_each_sample(a.rts, a.choices, lo, min(lo + PART, sl.hi), sample);
        if (parts) {
            __syncthreads();
            for (int i = threadIdx.x; i < H; i += blockDim.x) {
                top[i] += (unsigned char)(sh[i] >> 31);
                sh[i] &= 0x7fffffffu;
            }
            __syncthreads();
        }
    }
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const unsigned int x = __reduce_add_sync(0xffffffffu, n[c]);
        if (lane == 0 && c < a.nc) atomicAdd(&cnt[c], (unsigned long long)x);
    }
    nogo = __reduce_add_sync(0xffffffffu, nogo);
    omit = __reduce_add_sync(0xffffffffu, omit);
    if (lane == 0) {
        atomicAdd(&cnt[NC], (unsigned long long)nogo);
        atomicAdd(&cnt[NC + 1], (unsigned long long)omit);
    }
    if (pairs) {
        __syncthreads();
        for (int i = threadIdx.x; i < a.nc * a.nb_a; i += blockDim.x) {
            const int c = i / a.nb_a, k = i - c * a.nb_a, j = c * a.nb_b + 2 * k;
            sh[i] = hb[j] + hb[j + 1];  // both below 2^31
            top[i] = top[a.nc * a.nb_a + j] + top[a.nc * a.nb_a + j + 1];
        }
    }
    cl.sync();
    if (sl.rank == 0 && threadIdx.x < NC + 2) {
        int64_t x = 0;
        for (unsigned j = 0; j < sl.J; ++j) x += (int64_t)cl.map_shared_rank(cnt, j)[threadIdx.x];
        if ((int)threadIdx.x < a.nc) a.counts[sl.set * a.nc + threadIdx.x] = x;
        if (threadIdx.x == NC) a.nogo[sl.set] = x;
        if (threadIdx.x == NC + 1) a.omit[sl.set] = x;
    }
    // layout [S, nb, nc] like the pipeline's binned_128 / binned_256 arrays; the ranks share the bins
    for (int i = (int)sl.rank * (int)blockDim.x + threadIdx.x; i < H; i += (int)(sl.J * blockDim.x)) {
        int64_t x = 0;
        for (unsigned j = 0; j < sl.J; ++j)
            x += (int64_t)cl.map_shared_rank(sh, j)[i] + ((int64_t)cl.map_shared_rank(top, j)[i] << 31);
        if (i < a.nc * a.nb_a) {
            const int c = i / a.nb_a, b = i % a.nb_a;
            a.hist_a[(sl.set * a.nb_a + b) * a.nc + c] = (float)x;
        } else {
            const int k = i - a.nc * a.nb_a, c = k / a.nb_b, b = k % a.nb_b;
            a.hist_b[(sl.set * a.nb_b + b) * a.nc + c] = (float)x;
        }
    }
    cl.sync();  // the others' counters stay until they have been read
}

// CTAs per set of the per-set kernels (a cluster, at most the portable 8): the
// fewest that give every SM four 256-thread CTAs.
static unsigned ctas_per_set(int64_t n_sets) {
    unsigned J = 1;
    while (J < 8 && n_sets * J < (int64_t)sm_count() * 4) J *= 2;
    return J;
}

template <class K, class A>
static int launch_per_set(K kernel, const A &args, int64_t n_sets, size_t smem, cudaStream_t st) {
    const unsigned J = ctas_per_set(n_sets);
    SSM_REQUIRE(n_sets <= (int64_t)INT32_MAX / J, "too many sets for one launch");  // the grid's limit
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n_sets * J));
    cfg.blockDim = dim3(256);
    if (smem > 48 * 1024) SSM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = J;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    SSM_CUDA(cudaLaunchKernelEx(&cfg, kernel, args));
    return SSM_OK;
}

template <int NC>
static int kde_fit(const KdeFit &a, cudaStream_t st) {
    int rc = launch_per_set(k_kde_count<NC>, a, a.n_sets, 0, st);
    if (rc != SSM_OK) return rc;
    k_scan_i64<<<1, 1024, 0, st>>>(a.n_valid, a.n_sets * a.nc, a.poff);
    SSM_CUDA(cudaGetLastError());
    return launch_per_set(k_kde_scatter<NC>, a, a.n_sets, 0, st);
}

}  // namespace ssm

extern "C" {

int ssm_set_summary(const float *rts, const int32_t *choices, int64_t n_sets,
                    const int64_t *sample_offsets, const int32_t *choice_values, int n_choices,
                    double max_t, int64_t *choice_counts, int64_t *nogo_counts,
                    int64_t *omission_counts, int nbins_a, float *hist_a, int nbins_b,
                    float *hist_b, void *stream) {
    using namespace ssm;
    SSM_REQUIRE(n_sets >= 0 && n_choices >= 1 && n_choices <= KDE_MAX_CHOICES, "bad n_sets / n_choices");
    SSM_REQUIRE(nbins_a >= 1 && nbins_b >= 1 && (size_t)n_choices * (nbins_a + nbins_b) * 4 <= 48 * 1024,
                "histograms must fit in 48 KB of shared memory");
    if (n_sets == 0) return SSM_OK;
    SSM_REQUIRE(rts && choices && sample_offsets && choice_values && choice_counts && nogo_counts &&
                omission_counts && hist_a && hist_b, "all buffers are required");
    SetSummary a;
    a.n_sets = n_sets;
    a.rts = rts; a.choices = choices; a.soff = sample_offsets; a.cvals = choice_values;
    a.nc = n_choices; a.max_t = max_t; a.counts = choice_counts; a.nogo = nogo_counts;
    a.omit = omission_counts; a.nb_a = nbins_a; a.nb_b = nbins_b; a.hist_a = hist_a; a.hist_b = hist_b;
    const size_t smem = (size_t)n_choices * (nbins_a + nbins_b) * (sizeof(unsigned int) + 1);
    cudaStream_t st = (cudaStream_t)stream;
    if (n_choices <= 2) return launch_per_set(k_set_summary<2>, a, n_sets, smem, st);
    if (n_choices <= 4) return launch_per_set(k_set_summary<4>, a, n_sets, smem, st);
    return launch_per_set(k_set_summary<KDE_MAX_CHOICES>, a, n_sets, smem, st);
}

int ssm_kde_fit(const float *rts, const int32_t *choices, int64_t n_sets,
                const int64_t *sample_offsets, const int32_t *choice_values, int n_choices,
                const double *displace, double *displaced_logs, int64_t *count_all,
                int64_t *n_valid, int64_t *point_offsets, float *points, double *bandwidth,
                double *log_norm, double *proportion, void *stream) {
    using namespace ssm;
    SSM_REQUIRE(n_sets >= 0, "n_sets must be >= 0");
    SSM_REQUIRE(n_choices >= 1 && n_choices <= KDE_MAX_CHOICES, "n_choices must be in [1, %d]", KDE_MAX_CHOICES);
    SSM_REQUIRE(n_sets == 0 || (rts && choices && sample_offsets && choice_values && count_all &&
                                n_valid && point_offsets && points && bandwidth && log_norm && proportion),
                "all buffers are required");
    if (n_sets == 0) return SSM_OK;
    cudaStream_t st = (cudaStream_t)stream;
    SSM_REQUIRE(!displace || displaced_logs, "displace needs the displaced_logs buffer");
    KdeFit a{rts, choices, n_sets, sample_offsets, choice_values, n_choices, displace,
             displace ? displaced_logs : nullptr, count_all, n_valid, point_offsets, points,
             bandwidth, log_norm, proportion};
    if (n_choices <= 2) return kde_fit<2>(a, st);
    if (n_choices <= 4) return kde_fit<4>(a, st);
    return kde_fit<KDE_MAX_CHOICES>(a, st);
}

}  // extern "C"

namespace ssm {

// CTAs of the evaluation grid: every SM filled to the kernel's occupancy.
static int64_t kde_eval_ctas() {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_kde_eval, KDE_THREADS, 0) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    return (int64_t)per_sm * sm_count();
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct KdeEvalLayout {
    size_t head, ioff, ugroup, uidx, tail, link, slots, total;
    int64_t u_max, P;
};

static KdeEvalLayout kde_eval_layout(int64_t G, int64_t n_queries) {
    KdeEvalLayout L;
    L.P = kde_eval_ctas();
    L.u_max = n_queries / KDE_QT + G + 1;
    L.head = 0;
    L.ioff = L.head + 256;
    L.ugroup = L.ioff + align256((size_t)(L.u_max + 1) * 8);
    L.uidx = L.ugroup + align256((size_t)L.u_max * 4);
    L.tail = L.uidx + align256((size_t)L.u_max * 4);
    L.link = L.tail + align256((size_t)L.P * 4);
    L.slots = L.link + align256((size_t)L.P * 4);
    L.total = L.slots + (size_t)L.P * 2 * KDE_QT * sizeof(double);
    return L;
}

}  // namespace ssm

extern "C" {

size_t ssm_kde_eval_workspace_bytes(int64_t n_sets, int n_choices, int64_t n_queries) {
    if (n_sets < 0 || n_choices < 1 || n_queries < 0) return 0;
    return ssm::kde_eval_layout(n_sets * n_choices, n_queries).total;
}

int ssm_kde_eval(const float *points, const int64_t *point_offsets, const double *bandwidth,
                 const double *log_norm, int64_t n_sets, int n_choices,
                 const int64_t *sample_offsets, const double *displace,
                 const int64_t *query_offsets, const double *query_rt, int64_t n_queries, double lb,
                 double eps, double max_t, void *workspace, size_t workspace_bytes,
                 double *out_loglik, void *stream) {
    using namespace ssm;
    SSM_REQUIRE(n_sets >= 0 && n_choices >= 1 && n_choices <= KDE_MAX_CHOICES, "bad n_sets / n_choices");
    SSM_REQUIRE(n_queries >= 0, "n_queries must be >= 0");
    if (n_sets == 0 || n_queries == 0) return SSM_OK;
    SSM_REQUIRE(points && point_offsets && bandwidth && log_norm && sample_offsets && query_offsets &&
                query_rt && out_loglik && workspace, "all buffers are required");
    const int64_t G = n_sets * n_choices;
    const KdeEvalLayout L = kde_eval_layout(G, n_queries);
    SSM_REQUIRE(workspace_bytes >= L.total, "workspace too small: %zu bytes, need %zu (ssm_kde_eval_workspace_bytes)",
                workspace_bytes, L.total);
    SSM_REQUIRE(((uintptr_t)workspace & 255) == 0, "workspace must be 256-byte aligned");
    SSM_REQUIRE(L.u_max < (int64_t)1 << 31, "too many groups for one launch");
    uint8_t *ws = static_cast<uint8_t *>(workspace);
    KdeEval a;
    a.points = points; a.poff = point_offsets; a.h = bandwidth; a.lognorm = log_norm;
    a.qoff = query_offsets; a.q_rt = query_rt; a.out = out_loglik; a.nc = n_choices; a.G = G;
    a.soff = sample_offsets; a.shift = displace; a.lb = lb; a.eps = eps; a.max_t = max_t;
    a.head = reinterpret_cast<int64_t *>(ws + L.head);
    a.ioff = reinterpret_cast<int64_t *>(ws + L.ioff);
    a.ugroup = reinterpret_cast<int32_t *>(ws + L.ugroup);
    a.uidx = reinterpret_cast<int32_t *>(ws + L.uidx);
    a.tail = reinterpret_cast<int32_t *>(ws + L.tail);
    a.link = reinterpret_cast<int32_t *>(ws + L.link);
    a.u_max = L.u_max;
    a.slots = reinterpret_cast<double *>(ws + L.slots);
    a.P = L.P;
    cudaStream_t st = (cudaStream_t)stream;
    k_kde_plan<<<1, 1024, 0, st>>>(a);
    SSM_CUDA(cudaGetLastError());
    k_kde_eval<<<(unsigned)L.P, KDE_THREADS, 0, st>>>(a);
    SSM_CUDA(cudaGetLastError());
    k_kde_fixup<<<(unsigned)L.P, KDE_THREADS, 0, st>>>(a);
    SSM_CUDA(cudaGetLastError());
    return SSM_OK;
}

int ssm_kde_sample(const float *points, const int64_t *point_offsets, const double *bandwidth,
                   int64_t n_sets, int n_choices, const double *displace,
                   const int64_t *out_offsets, const int64_t *n_kde, uint64_t seed, double max_t,
                   double unif_lo, double unif_hi, double *out_rt, void *stream) {
    using namespace ssm;
    SSM_REQUIRE(n_sets >= 0 && n_choices >= 1 && n_choices <= KDE_MAX_CHOICES, "bad n_sets / n_choices");
    if (n_sets == 0) return SSM_OK;
    SSM_REQUIRE(points && point_offsets && bandwidth && out_offsets && n_kde && out_rt, "all buffers are required");
    KdeSample a;
    a.key = philox_keys(seed);
    a.points = points; a.poff = point_offsets; a.h = bandwidth; a.ooff = out_offsets; a.nkde = n_kde;
    a.n_groups = n_sets * n_choices; a.shift = displace; a.nc = n_choices; a.max_t = max_t;
    a.ulo = unif_lo; a.uhi = unif_hi; a.out_rt = out_rt;
    k_kde_sample<<<sm_count() * 8, 256, 0, (cudaStream_t)stream>>>(a);
    SSM_CUDA(cudaGetLastError());
    return SSM_OK;
}

int ssm_kde_records(const float *theta, int n_params, int64_t n_sets, int n_choices,
                    const int32_t *choice_values, const int64_t *query_offsets,
                    const double *query_rt, const double *query_loglik, int64_t n_down,
                    int64_t rows_per_set, float negative_rt_loglik, uint64_t seed, float *out,
                    void *stream) {
    using namespace ssm;
    SSM_REQUIRE(n_sets >= 0 && n_params >= 1 && n_choices >= 1 && n_choices <= KDE_MAX_CHOICES, "bad sizes");
    SSM_REQUIRE(rows_per_set >= 1 && rows_per_set <= KDE_MAX_ROWS, "rows_per_set must be in [1, %d]", KDE_MAX_ROWS);
    if (n_sets == 0) return SSM_OK;
    SSM_REQUIRE(theta && choice_values && query_offsets && query_rt && query_loglik && out, "all buffers are required");
    KdeRecords a;
    a.key = philox_keys(seed);
    a.theta = theta; a.P = n_params; a.n_sets = n_sets; a.qoff = query_offsets; a.q_rt = query_rt;
    a.q_ll = query_loglik; a.cvals = choice_values; a.nc = n_choices; a.n_down = n_down;
    a.rows_per_set = rows_per_set; a.neg_ll = negative_rt_loglik; a.out = out;
    const size_t smem = (size_t)rows_per_set * (sizeof(int) + 2 * sizeof(uint16_t));
    if (smem > 48 * 1024)
        SSM_CUDA(cudaFuncSetAttribute(k_kde_records, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_kde_records<<<(unsigned)n_sets, 256, smem, (cudaStream_t)stream>>>(a);
    SSM_CUDA(cudaGetLastError());
    return SSM_OK;
}

}  // extern "C"

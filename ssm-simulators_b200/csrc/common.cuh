// Shared device/host helpers for the sm_100a simulators: status handling,
// the counter-based Philox4x32-10 generator and normal/uniform transforms.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "ssm_b200.h"

namespace ssm {

// ---------------------------------------------------------------- host side
void set_error(const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *where);
int sm_count();

#define SSM_CUDA(call)                                         \
    do {                                                       \
        cudaError_t e_ = (call);                               \
        if (e_ != cudaSuccess) return ::ssm::cuda_fail(e_, #call); \
    } while (0)

#define SSM_REQUIRE(cond, ...)          \
    do {                                \
        if (!(cond)) {                  \
            ::ssm::set_error(__VA_ARGS__); \
            return SSM_ERR_ARG;         \
        }                               \
    } while (0)

// Trajectories a persistent simulator warp claims per queue access: the
// caller's chunk, cut to a twelfth of a warp's share of the launch (a multiple
// of the warp's 32 walks, at least one each), so that no warp is left with a large
// claim at the end, nor with a large one of the longest walks, which come first.
// Measured with claims of 256 / 64 (ms): 256 angle sets 2.62 / 1.67, 64 sets
// 1.48 / 0.84, 4 096 sets 23.8 / 24.1.
__device__ __forceinline__ int64_t warp_chunk(int chunk, int64_t total) {
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5) * 12;
    const int64_t fair = ((total + warps - 1) / warps + 31) / 32 * 32;
    return max((int64_t)32, min((int64_t)chunk, fair));
}

// Ended walks a persistent simulator warp collects before it writes their
// results and restarts those lanes (ssm_launch.refill_min = 0).  Batching
// pays where a step is cheap next to the restart.  Measured defaults: with restarts
// that stay in their trial two at a time are best on the single-accumulator
// batches (4 096 angle sets: 24.3 ms, four 24.5), four on the race family (racing
// diffusion 9.7 ms, two 9.9; LCA 15.1, 15.3).
#ifndef SSM_REFILL_MIN
#define SSM_REFILL_MIN 2
#endif
#ifndef SSM_REFILL_MIN_RACE
#define SSM_REFILL_MIN_RACE 4
#endif

// Workspace header shared by every persistent kernel: a work counter and an
// error word.  It sits at the start of the caller's workspace and is cleared
// by the launching entry point (cudaMemsetAsync) before each launch.
struct alignas(256) WorkspaceHeader {
    unsigned long long counter;  // next unclaimed trajectory index
    int err;                     // first error code raised on the device (0 = none)
    int err_detail;              // e.g. the trajectory that overran its noise row
    unsigned long long aux[4];
};
static_assert(sizeof(WorkspaceHeader) == 256, "header must stay 256 B");

// Philox4x32-10 round keys.  The key schedule depends only on the seed, so it
// is expanded once on the host and travels in the kernel parameter block
// (constant bank): each round's key XOR is then a free constant operand.
struct PhiloxKeys {
    uint32_t k0[10];
    uint32_t k1[10];
};

inline PhiloxKeys philox_keys(uint64_t seed) {
    PhiloxKeys k;
    uint32_t a = (uint32_t)seed, b = (uint32_t)(seed >> 32);
    for (int r = 0; r < 10; ++r) {
        k.k0[r] = a;
        k.k1[r] = b;
        a += 0x9E3779B9u;  // Weyl increments of the Philox key schedule
        b += 0xBB67AE85u;
    }
    return k;
}

// ---------------------------------------------------------------- device side
// Philox4x32 with 10 rounds (Salmon, Moraes, Dror & Shaw, "Parallel Random
// Numbers: As Easy as 1, 2, 3", SC'11).  One call maps a 128-bit counter to
// 128 random bits; we key it by the seed and count over (step block, sample,
// trial, stream) so every trajectory owns an independent stream.
__device__ __forceinline__ uint4 philox10(uint4 c, const PhiloxKeys &key) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        // one 32x32->64 multiply (IMAD.WIDE.U32) per product gives both halves
        const uint64_t p0 = (uint64_t)0xD2511F53u * c.x;
        const uint64_t p1 = (uint64_t)0xCD9E8D57u * c.z;
        c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ key.k0[r], (uint32_t)p1,
                       (uint32_t)(p0 >> 32) ^ c.w ^ key.k1[r], (uint32_t)p0);
    }
    return c;
}

// 23 random bits -> float in [1, 2) by exponent stuffing (two integer ops, no
// int->float conversion, which runs at quarter rate).
__device__ __forceinline__ float bits_to_1_2(uint32_t x) {
    return __uint_as_float(0x3f800000u | (x >> 9));
}
// Uniform on the open interval (0, 1): values j*2^-23 + 2^-24, j = 0..2^23-1.
__device__ __forceinline__ float uniform_open(uint32_t x) {
    return bits_to_1_2(x) - 0.99999994f;  // 1 - 2^-24; exact in float32
}
// Uniform on [0, 1) with 24-bit resolution (used once per trajectory).
__device__ __forceinline__ float uniform_co(uint32_t x) {
    return (float)(x >> 8) * 5.9604645e-08f;  // 2^-24
}

// SFU approximations in their flush-to-zero forms.  Every argument the
// generators pass is a normal float (uniforms are at least 2^-24, angles 0 or
// at least 2^-21), for which these give the same results as the non-ftz
// forms, without the extra instructions that rescale subnormal inputs.
__device__ __forceinline__ float lg2_ftz(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void sincos_ftz(float x, float &s, float &c) {
    asm("sin.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(x));
    asm("cos.approx.ftz.f32 %0, %1;" : "=f"(c) : "f"(x));
}

// Packed pairs of float32: two IEEE operations per instruction with the results
// of the scalar ones.  The simulators and the KDE are bound by issue slots or the
// SFU, not by the FP32 lanes, so a packed operation saves an issue slot.
__device__ __forceinline__ uint64_t pack_f2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack_f2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma_f2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add_f2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul_f2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Box-Muller transform of two 32-bit words into two N(0,1) variates
// (r = sqrt(-2 ln u1), phase 2 pi u2).  Uses the SFU approximations of log2,
// rsqrt, sin and cos: 4 MUFU operations per pair (u1 >= 2^-24 and the phase
// is 0 or at least 2 pi 2^-23: normal floats, so the ftz forms apply).
__device__ __forceinline__ float2 box_muller(uint32_t a, uint32_t b) {
    const float u1 = uniform_open(a);
    const float u2 = bits_to_1_2(b) - 1.0f;
    const float e = -1.3862944f * lg2_ftz(u1);  // -2 ln u1 > 0
    const float r = e * rsqrtf(e);
    float s, c;
    sincos_ftz(6.2831853f * u2, s, c);
    return make_float2(r * c, r * s);
}

// The top nine bits of hi and of lo as an 18-bit phase in the upper bits of a
// float mantissa (bits 22-14 and 13-5): one shift, one funnel shift and the mask
// (which joins the exponent's OR), where two shifts and two masks would be four.
// The ALU pipe takes two cycles an instruction and an added one cost the angle
// batch 1.6 ms per step; this is one instruction less per pair.
__device__ __forceinline__ uint32_t phase18(uint32_t hi, uint32_t lo) {
    return __funnelshift_r(lo, hi >> 23, 18) & 0x007fffe0u;
}

// Six increments from one Philox4x32-10 call (128 bits): three Box-Muller pairs whose
// radii take 23-bit uniforms from the low bits of x, y and z, and whose phases
// take the low 23 bits of w, and 18 bits each from the top nine bits of (w, x)
// and of (y, z).  The radius resolution is that of the four-per-call layout
// (uniforms on a 2^-23 grid, so |N| <= 5.6); an 18-bit phase puts the pair on
// one of 262 144 rays, far below what a one-dimensional increment can show.
// Compared with two pairs per call this takes a third less Philox work per
// increment.  c2 = -2 ln(2) scale^2 scales the radius, so each output is
// drift + scale * N(0,1) (scale 1, drift 0: standard normals).  Pair i (outputs
// 2i, 2i+1) takes its own c2[i] and drift[i] (bm6_increment: the same for all).
__device__ __forceinline__ void bm6_increment_pairs(uint4 b, const float (&c2)[3], const float (&drift)[3],
                                                    float *g) {
    const uint32_t rad[3] = {b.x, b.y, b.z};
    const uint32_t ph[3] = {b.w & 0x007fffffu, phase18(b.w, b.x), phase18(b.y, b.z)};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float u1 = __uint_as_float(0x3f800000u | (rad[i] & 0x007fffffu)) - 0.99999994f;  // (0, 1)
        const float ang = fmaf(__uint_as_float(0x3f800000u | ph[i]), 6.2831853f, -6.2831853f);
        const float e = c2[i] * lg2_ftz(u1);
        float r;
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(e));
        float sn, cs;
        sincos_ftz(ang, sn, cs);
        g[2 * i] = fmaf(r, cs, drift[i]);
        g[2 * i + 1] = fmaf(r, sn, drift[i]);
    }
}
__device__ __forceinline__ void bm6_increment(uint4 b, float c2, float drift, float *g) {
    const float c[3] = {c2, c2, c2}, d[3] = {drift, drift, drift};
    bm6_increment_pairs(b, c, d, g);
}

// Two Box-Muller pairs (bits ra, pa and rb, pb; radius constants c2, drifts d) with
// the FP32 operations packed: cs and sn hold pair a's output in the lower half,
// pair b's in the upper one, the values of bm6_increment_pairs.
__device__ __forceinline__ void bm_pair2(uint32_t ra, uint32_t rb, uint32_t pa, uint32_t pb, uint64_t c2,
                                         uint64_t d, uint64_t &cs, uint64_t &sn) {
    const float2 u = unpack_f2(add_f2(pack_f2(__uint_as_float(0x3f800000u | (ra & 0x007fffffu)),
                                              __uint_as_float(0x3f800000u | (rb & 0x007fffffu))),
                                      pack_f2(-0.99999994f, -0.99999994f)));
    const float2 ang = unpack_f2(fma_f2(pack_f2(__uint_as_float(0x3f800000u | pa), __uint_as_float(0x3f800000u | pb)),
                                        pack_f2(6.2831853f, 6.2831853f), pack_f2(-6.2831853f, -6.2831853f)));
    const float2 e = unpack_f2(mul_f2(c2, pack_f2(lg2_ftz(u.x), lg2_ftz(u.y))));
    float r0, r1, s0, s1, k0, k1;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(e.x));
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(e.y));
    sincos_ftz(ang.x, s0, k0);
    sincos_ftz(ang.y, s1, k1);
    const uint64_t r = pack_f2(r0, r1);
    cs = fma_f2(r, pack_f2(k0, k1), d);
    sn = fma_f2(r, pack_f2(s0, s1), d);
}

// Twelve increments from two calls, two Box-Muller pairs to an instruction
// wherever the arithmetic is FP32 (7.5 issue slots fewer per six increments than
// bm6_increment_pairs, the same values): pairs (0, 1), (2, 3), (4, 5) of the six
// share the packed operations, the SFU ones stay scalar.
__device__ __forceinline__ void bm12_increment(uint4 b0, uint4 b1, float c2, float drift, float *g) {
    const uint32_t rad[6] = {b0.x, b0.y, b0.z, b1.x, b1.y, b1.z};
    const uint32_t ph[6] = {b0.w & 0x007fffffu, phase18(b0.w, b0.x), phase18(b0.y, b0.z),
                            b1.w & 0x007fffffu, phase18(b1.w, b1.x), phase18(b1.y, b1.z)};
    const uint64_t c = pack_f2(c2, c2), d = pack_f2(drift, drift);
#pragma unroll
    for (int i = 0; i < 6; i += 2) {
        uint64_t cs, sn;
        bm_pair2(rad[i], rad[i + 1], ph[i], ph[i + 1], c, d, cs, sn);
        const float2 k = unpack_f2(cs), s = unpack_f2(sn);
        g[2 * i] = k.x;
        g[2 * i + 1] = s.x;
        g[2 * i + 2] = k.y;
        g[2 * i + 3] = s.y;
    }
}

__device__ __forceinline__ void raise_error(WorkspaceHeader *h, int code, int detail) {
    if (atomicCAS(&h->err, 0, code) == 0) h->err_detail = detail;
}

}  // namespace ssm

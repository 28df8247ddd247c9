// The storage quantisers on float32 rows: the midrise quantiser with one scale per group of channels
// [reference memlm_sh.py:221-229] and fp8-e4m3 with one scale per row.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include "slotscan.h"
#include "slotscan_common.cuh"

namespace slotscan {

__device__ __forceinline__ float round_to(float v, float) { return v; }
__device__ __forceinline__ float round_to(float v, __nv_bfloat16) { return __bfloat162float(__float2bfloat16_rn(v)); }

// fq of one group member, in the arithmetic of the reference: s = max(a / half, 1e-30),
// q = (clamp(floor(x / s), -half, half - 1) + 0.5) * s, zero for an all-zero group, returned in the straight-through
// form x + (q - x) evaluated in the input dtype (memlm_sh.py:229).
// The IEEE division x / s is what costs: it is replaced by x * (1 / s) wherever that provably has the same floor (the
// product is off by a few ulp of a quotient that is at most 128 in size, so any result further than 1e-3 from an
// integer floors alike), by the known answer for the group's own extreme (x = +-a gives exactly +-half), and kept for
// the rare rest.  s, 1 / s are per group.
struct FqScale { float a, half, s, rs; bool plain; };
__device__ __forceinline__ FqScale fq_scale(float a, float half) {
    FqScale g;
    g.a = a; g.half = half;
    g.s = fmaxf(__fdiv_rn(a, half), 1e-30f);
    g.rs = __frcp_rn(g.s);
    g.plain = a > 1e-20f;                    // s = a / half exactly: not clamped, not denormal
    return g;
}
template <typename Tin>
__device__ __forceinline__ float fq_one(float x, const FqScale& g) {
    float f;
    const float qt = x * g.rs, fl = floorf(qt), fr = qt - fl;
    if (g.plain && fabsf(x) == g.a) f = x > 0.f ? g.half : -g.half;
    else if (g.plain && fr > 1e-3f && fr < 0.999f) f = fl;
    else f = floorf(__fdiv_rn(x, g.s));
    f = fminf(fmaxf(f, -g.half), g.half - 1.f);
    const float q = (g.a > 0.f) ? __fmul_rn(__fadd_rn(f, 0.5f), g.s) : 0.f;
    const float qd = round_to(q, Tin());
    const float diff = round_to(__fsub_rn(qd, x), Tin());
    return round_to(__fadd_rn(x, diff), Tin());
}

// fp8-e4m3 with scale sc of a row whose largest magnitude is a
__device__ __forceinline__ float e4m3_scale(float a) { return fmaxf(__fdiv_rn(a, 448.f), 1e-30f); }
__device__ __forceinline__ float e4m3_one(float x, float a, float sc) {
    const __nv_fp8_storage_t b = __nv_cvt_float_to_fp8(__fdiv_rn(x, sc), __NV_SATFINITE, __NV_E4M3);
    const float f = __half2float(__half(__nv_cvt_fp8_to_halfraw(b, __NV_E4M3)));
    return a > 0.f ? __fmul_rn(f, sc) : 0.f;
}

// A row held by LPR neighbouring lanes, each with NPC pieces of 8 consecutive columns that lie LPR * 8 columns apart
// (piece q of lane c: columns q * LPR * 8 + c * 8 ..), quantised as the writer epilogue quantises it: bits 2..8 with
// groups of `group` channels, or SLOTSCAN_BITS_E4M3.  gmask: the row's lanes (the rows of a warp may be apart).
template <int LPR, int NPC>
__device__ __forceinline__ void quantise_lanes(float* y, const float* x, int bits, int group, unsigned gmask) {
    if (bits == SLOTSCAN_BITS_E4M3 || group > LPR * 8) {                 // one group over all pieces
        float a = 0.f;
#pragma unroll
        for (int j = 0; j < 8 * NPC; j++) a = fmaxf(a, fabsf(x[j]));
#pragma unroll
        for (int off = LPR / 2; off > 0; off >>= 1) a = fmaxf(a, __shfl_xor_sync(gmask, a, off));
        if (bits == SLOTSCAN_BITS_E4M3) {
            const float sc = e4m3_scale(a);
#pragma unroll
            for (int j = 0; j < 8 * NPC; j++) y[j] = e4m3_one(x[j], a, sc);
        } else {
            const FqScale g = fq_scale(a, (float)(1 << (bits - 1)));
#pragma unroll
            for (int j = 0; j < 8 * NPC; j++) y[j] = fq_one<float>(x[j], g);
        }
        return;
    }
    const float half = (float)(1 << (bits - 1));
#pragma unroll
    for (int q = 0; q < NPC; q++) {
        float a0 = 0.f, a1 = 0.f;
#pragma unroll
        for (int j = 0; j < 4; j++) { a0 = fmaxf(a0, fabsf(x[8 * q + j])); a1 = fmaxf(a1, fabsf(x[8 * q + 4 + j])); }
        if (group >= 8) {
            a0 = fmaxf(a0, a1);
            for (int off = 1; off < group / 8; off <<= 1) a0 = fmaxf(a0, __shfl_xor_sync(gmask, a0, off));
            a1 = a0;
        }
        const FqScale g0 = fq_scale(a0, half), g1 = group >= 8 ? g0 : fq_scale(a1, half);
#pragma unroll
        for (int j = 0; j < 4; j++) { y[8 * q + j] = fq_one<float>(x[8 * q + j], g0); y[8 * q + 4 + j] = fq_one<float>(x[8 * q + 4 + j], g1); }
    }
}

}  // namespace slotscan

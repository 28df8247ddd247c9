// Shared device helpers of the slot-scan kernels (sm_100a).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "slotscan.h"

namespace slotscan {

constexpr unsigned FULL = 0xffffffffu;
constexpr int BIGI = 0x7fffffff;

// ---- typed vector loads / stores: token streams and snapshots are f32 or bf16, arithmetic is always f32 ----
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ld4(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void st4(__nv_bfloat16* p, float4 v) {
    __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    uint2 u;
    u.x = *reinterpret_cast<unsigned*>(&a);
    u.y = *reinterpret_cast<unsigned*>(&b);
    *reinterpret_cast<uint2*>(p) = u;
}
__device__ __forceinline__ void ld8(float* d, const float* s) {
    const float4 a = ld4(s), b = ld4(s + 4);
    d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w; d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
}
__device__ __forceinline__ void ld8(float* d, const __nv_bfloat16* s) {
    const uint4 u = *reinterpret_cast<const uint4*>(s);
    const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
        d[2 * i] = f.x; d[2 * i + 1] = f.y;
    }
}
__device__ __forceinline__ void st8(float* d, const float* s) {
    st4(d, make_float4(s[0], s[1], s[2], s[3]));
    st4(d + 4, make_float4(s[4], s[5], s[6], s[7]));
}
__device__ __forceinline__ void st8(__nv_bfloat16* d, const float* s) {
    unsigned w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        __nv_bfloat162 h = __floats2bfloat162_rn(s[2 * i], s[2 * i + 1]);
        w[i] = *reinterpret_cast<unsigned*>(&h);
    }
    *reinterpret_cast<uint4*>(d) = make_uint4(w[0], w[1], w[2], w[3]);
}
// one element, float32 or bfloat16
__device__ __forceinline__ float ld1(const float* p) { return *p; }
__device__ __forceinline__ float ld1(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void st1(float* p, float v) { *p = v; }
__device__ __forceinline__ void st1(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(FULL, v, off);
    return v;
}
// sum over the LPR (power of two <= 32) adjacent lanes that share one row
template <int LPR>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) v += __shfl_xor_sync(FULL, v, off);
    return v;
}
// 1 / s in double for s and 1 / s normal, within one unit in the last place of the division's result: the softmax sums of the
// two soft scans, on whose token chains the division itself costs a tenth of the call (B = 4, T = 512, H = 12, 192 x (64 + 64):
// 1.97 -> 2.18 ms with it).  One step of Householder's iteration of order two for f(r) = 1/r - s from the hardware's approximation
// r, whose relative error is below 2^-19 (it reads the upper half of s and gives 20 bits): with t = 1 - s r,
// 1/s = r / (1 - t) = r (1 + t + t^2 + ...), and what is cut off is below |t|^3 < 2^-57.
__device__ __forceinline__ double rcp_normal(double s) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(s));
    const double t = fma(-s, r, 1.0);
    return fma(r, fma(t, t, t), r);
}
__device__ __forceinline__ float dot4(float4 a, float4 b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }

// ---- two float32 multiply-adds in one instruction (sm_100), each rounded as its own: half the instructions where a warp's
// instruction stream is what bounds (the pipe's rate per operation is about the same) ----
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
struct f32x4 { f32x2 a, b; };                             // x, y | z, w of a float4
__device__ __forceinline__ f32x4 ld4x2(const float* p) {
    const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(p);
    return {u.x, u.y};
}
__device__ __forceinline__ f32x4 pack4(float4 v) { return {pack2(v.x, v.y), pack2(v.z, v.w)}; }
__device__ __forceinline__ f32x4 ld4x2(const __nv_bfloat16* p) { return pack4(ld4(p)); }
__device__ __forceinline__ void fma4(f32x4& c, const f32x4& a, const f32x4& b) { c.a = fma2(a.a, b.a, c.a); c.b = fma2(a.b, b.b, c.b); }
// (x + y) + (z + w)
__device__ __forceinline__ float sum4(const f32x4& v) {
    const float2 p = unpack2(v.a), q = unpack2(v.b);
    return (p.x + p.y) + (q.x + q.y);
}

// The one write rule of the scan, state <- (1-g) state + g x, spelled identically in every kernel so that a row
// replayed by another kernel is bit-identical to the row the address kernel held.
__device__ __forceinline__ float blend(float old, float x, float g, float omw) {
    return __fmaf_rn(g, x, __fmul_rn(omw, old));
}

// occupied candidate (z, i): larger z wins, equal z -> smaller index (argmax returns the FIRST maximum)
__device__ __forceinline__ void best(float& z, int& i, float z2, int i2) {
    if (z2 > z || (z2 == z && i2 < i)) { z = z2; i = i2; }
}

__device__ __forceinline__ unsigned ord_key(float f) {    // monotone float -> unsigned
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float gate_eff(float g, int hard_gate) { return hard_gate ? (g > 0.5f ? 1.f : 0.f) : g; }

}  // namespace slotscan

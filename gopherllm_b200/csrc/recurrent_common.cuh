// Gates and decays of the mixers with per-sequence state, in 32-bit.
#pragma once

#include "common.cuh"

#define RC_THREADS 128

__device__ __forceinline__ float rc_sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float rc_silu(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float rc_log_sigmoid(float x) { return fminf(x, 0.0f) - log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float rc_softplus(float x) { return x > 20.0f ? x : log1pf(expf(x)); }
// e^x for a decay that is applied at every token: near one the factor comes from expm1f, which is
// rounded once; expf's last-bit errors near one do not average out over a thousand tokens of a slowly
// decaying state.
__device__ __forceinline__ float rc_decay(float x) {
    if (x > -0.5f && x <= 0.f) {
        // 1 + (e^x - 1) with e^x - 1 from its series to x^9/9! (below 2^-28 here), Horner in 32-bit
        float p = 2.755731922e-6f;
        p = fmaf(p, x, 2.48015873e-5f);
        p = fmaf(p, x, 1.984126984e-4f);
        p = fmaf(p, x, 1.388888889e-3f);
        p = fmaf(p, x, 8.333333333e-3f);
        p = fmaf(p, x, 4.166666667e-2f);
        p = fmaf(p, x, 1.666666667e-1f);
        p = fmaf(p, x, 0.5f);
        p = fmaf(p, x, 1.0f);
        return fmaf(p, x, 1.0f);
    }
    if (x > -0.5f) return 1.0f + expm1f(x);
    return expf(x);
}

// 16 bytes of a row (4 floats or 8 bfloat16) as floats; both addresses 16-byte aligned
__device__ __forceinline__ void mc_load16(const float* src, float* dst) {
    *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(src);
}
__device__ __forceinline__ void mc_load16(const __nv_bfloat16* src, float* dst) {
    const uint4 raw = *reinterpret_cast<const uint4*>(src);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
    const float2 f0 = __bfloat1622float2(h[0]), f1 = __bfloat1622float2(h[1]);
    const float2 f2 = __bfloat1622float2(h[2]), f3 = __bfloat1622float2(h[3]);
    reinterpret_cast<float4*>(dst)[0] = make_float4(f0.x, f0.y, f1.x, f1.y);
    reinterpret_cast<float4*>(dst)[1] = make_float4(f2.x, f2.y, f3.x, f3.y);
}

// 4 or 8 floats as 16 bytes of a row
__device__ __forceinline__ void mc_store16(float* dst, const float* v) {
    *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(v);
}
__device__ __forceinline__ void mc_store16(__nv_bfloat16* dst, const float* v) {
    uint4 raw;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
    h[0] = __floats2bfloat162_rn(v[0], v[1]);
    h[1] = __floats2bfloat162_rn(v[2], v[3]);
    h[2] = __floats2bfloat162_rn(v[4], v[5]);
    h[3] = __floats2bfloat162_rn(v[6], v[7]);
    *reinterpret_cast<uint4*>(dst) = raw;
}

// two 32-bit multiply-adds in one instruction (the pair's halves are independent and rounded like fmaf's)
__device__ __forceinline__ unsigned long long mc_pack(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ unsigned long long mc_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long mc_mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float2 mc_unpack(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

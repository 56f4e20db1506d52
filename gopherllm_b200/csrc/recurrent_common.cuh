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

// Divisions by cheaper instructions with the same results, for host and device.
#pragma once
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>

namespace xpbd {

// a / s with one division, for s in [2^-20, 2^63] (constraint counts; distances
// that are not too short for a direction) where no component overflows: the
// products with the rounded reciprocal and a residual step each, which rounds like
// three divisions (P. Markstein, 1990) for components that are 0 (a zero may lose
// its sign) or at least 2^-100 (below, where the residual leaves the number range,
// the last bit may differ).  The residual of an infinite component is not a
// number: fminf drops it, and the component stays infinite.
__host__ __device__ __forceinline__ float3 over(float3 a, float s) {
    const float r = 1.f / s;
    const float3 q = make_float3(a.x * r, a.y * r, a.z * r);
    return make_float3(fmaf(fminf(fmaf(-q.x, s, a.x), FLT_MAX), r, q.x),
                       fmaf(fminf(fmaf(-q.y, s, a.y), FLT_MAX), r, q.y),
                       fmaf(fminf(fmaf(-q.z, s, a.z), FLT_MAX), r, q.z));
}

// x / 6 in three instructions, one residual step on the product with the rounded
// reciprocal: the division's result for 2^-125 <= |x| < inf and for 0 (a zero may
// lose its sign); NaN for an infinite x.
__host__ __device__ __forceinline__ float sixth(float x) {
    const float q = x * (1.f / 6.f);
    return fmaf(fmaf(-6.f, q, x), 1.f / 6.f, q);
}

}  // namespace xpbd

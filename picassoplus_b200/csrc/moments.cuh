// Statistics of channels as (count, mean, sum of squared deviations) triples, merged pairwise, and the ReLU beside them.
#pragma once
#include "common.cuh"

namespace pb {
namespace norm {

// ReLU as torch has it: a NaN stays one, forward and backward
__device__ __forceinline__ float relu_of(float x) {
    float y;
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float relu_grad(float g, float act) { return act <= 0.f ? 0.f : g; }

struct Moments { float n, mean, m2; };
__device__ __forceinline__ void merge(Moments& a, const Moments& b) {
    const float n = a.n + b.n, d = b.mean - a.mean, f = b.n > 0.f ? __fdividef(b.n, n) : 0.f;      // no branch: loads run ahead
    a.mean = fmaf(d, f, a.mean);
    a.m2 += b.m2 + d * d * a.n * f;
    a.n = n;
}

// from n values and the sums of their differences (and squares) to `shift`, one of them
__device__ __forceinline__ Moments moments(float n, float shift, float s1, float s2) {
    Moments m{n, shift, 0.f};
    if (n > 0.f) { m.mean = shift + s1 / n; m.m2 = relu_of(s2 - s1 * s1 / n); }        // (a NaN stays one)
    return m;
}

}  // namespace norm
}  // namespace pb

// GELU (tanh form) and its derivative (kernels/fused_ops.cu:66-82, :96-103).
#pragma once

#include <cuda_runtime.h>

namespace mni {

// 0.5 (1 + tanh u) = s(2u) with s the logistic function, so gelu(v) = v s(2u) and, as 0.5 (1 - tanh^2 u) = 2 s (1 - s),
// gelu'(v) = s + 2 v s (1 - s) u', u = sqrt(2/pi) (v + 0.044715 v^3).  One exponential and one approximate reciprocal
// instead of tanhf: the passes over 2048 x 3072 were bound by that arithmetic.
// With e = exp(-|2u|) <= 1 neither s nor 1 - s is the difference of two close numbers, and nothing overflows.  s is kept as
// hi + lo: lo carries what the rounding of 1 + e and the approximate reciprocal left, so that each result is rounded once.
// Relative 2-norm error over normally distributed v against float64: gelu 2.9e-8 and gelu' 4.2e-8; with tanhf 3.8e-8 and
// 4.5e-8; without lo, a correctly rounded reciprocal and 1 - s as a difference 4.7e-8 and 7.3e-8.  For negative v the relative
// error of s is that of e, up to (4 + 3.2 |2u|) 2^-23 with the rounding of u, where 1 + tanhf had lost up to all digits.
// 2048 x 3072: forward 8.1 us, backward 14.7 (tanhf 11.1 and 16.9); 8192 x 4096: 43 and 75 (51 and 77).
struct GeluGate {
    float hi, lo, slope, du;       // s = hi + lo; s (1 - s); d(2u)/dv
};
__device__ __forceinline__ GeluGate gelu_gate(float v) {
    constexpr float kLinear = 1.5957691216057308f, kCubic = 0.07135481627260025f;        // 2u = v (linear + cubic v^2)
    const float w = v * v;
    const float e = __expf(-fabsf(v * fmaf(kCubic, w, kLinear)));
    const float n = 1.0f + e, lost = e - (n - 1.0f);            // 1 + e = n + lost exactly
    const float r = __fdividef(1.0f, n);
    const float top = v >= 0.0f ? 1.0f : e;
    GeluGate g;
    g.hi = top * r;
    g.lo = (fmaf(-g.hi, n, top) - g.hi * lost) * r;
    g.slope = e * r * r;
    g.du = fmaf(3.0f * kCubic, w, kLinear);
    return g;
}
__device__ __forceinline__ float gelu_tanh(float v) {
    const GeluGate g = gelu_gate(v);
    return fmaf(v, g.hi, fminf(v, 1e30f) * g.lo);               // the bound keeps gelu(inf) = inf, where lo = 0
}
__device__ __forceinline__ float gelu_tanh_grad(float v) {
    const GeluGate g = gelu_gate(v);
    return g.hi + fmaf(v * g.slope, g.du, g.lo);
}

}  // namespace mni

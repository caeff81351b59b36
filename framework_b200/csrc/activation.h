// GELU (tanh form) and its derivative (kernels/fused_ops.cu:66-82, :96-103).
#pragma once

#include <cuda_runtime.h>

namespace mni {

// 0.5 (1 + tanh u) = s(2u) with s the logistic function, so gelu(v) = v s(2u) and, as 0.5 (1 - tanh^2 u) = 2 s (1 - s),
// gelu'(v) = s + 2 v s (1 - s) u', u = sqrt(2/pi) (v + 0.044715 v^3).  One exponential and one reciprocal instead of tanhf:
// the passes over 2048 x 3072 were bound by this arithmetic (backward 22 us of 75 MB).  Large |v| end in s = 0 or 1.
// __expf is off by 2 + 1.2 |x| units in the last place, which 1 + exp divides by 1 + 1/exp: below one unit of s for
// positive v; for negative v the relative error of s stays below 1e-6, where 1 + tanh had lost up to all of its digits.
__device__ __forceinline__ float gelu_gate(float v) {
    const float u2 = 1.5957691216057308f * (v + 0.044715f * v * v * v);
    return __frcp_rn(1.0f + __expf(-u2));
}
__device__ __forceinline__ float gelu_tanh(float v) { return v * gelu_gate(v); }
__device__ __forceinline__ float gelu_tanh_grad(float v) {
    const float s = gelu_gate(v);
    return s + v * s * (1.0f - s) * (1.5957691216057308f * (1.0f + 0.134145f * v * v));
}

}  // namespace mni

// GELU (tanh form) and its derivative (kernels/fused_ops.cu:66-82, :96-103).
#pragma once

#include <cuda_runtime.h>

namespace mni {

// 0.5 (1 + tanh u) = s(2u) with s the logistic function, so gelu(v) = v s(2u) and, as 0.5 (1 - tanh^2 u) = 2 s (1 - s),
// gelu'(v) = s + 2 v s (1 - s) u', u = sqrt(2/pi) (v + 0.044715 v^3).  One exponential and one reciprocal instead of tanhf:
// the backward over 2048 x 3072 was bound by this arithmetic, 22 us of 75 MB.  Large |v| end in s = 0 or 1.
__device__ __forceinline__ float gelu_gate(float v) {
    const float u2 = 1.5957691216057308f * (v + 0.044715f * v * v * v);
    return __frcp_rn(1.0f + expf(-fminf(fmaxf(u2, -80.0f), 80.0f)));
}
__device__ __forceinline__ float gelu_tanh(float v) { return v * gelu_gate(v); }
__device__ __forceinline__ float gelu_tanh_grad(float v) {
    const float s = gelu_gate(v);
    return s + v * s * (1.0f - s) * (1.5957691216057308f * (1.0f + 0.134145f * v * v));
}

}  // namespace mni

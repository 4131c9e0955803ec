// silu and its gradient as every SwiGLU kernel computes them (solution/swiglu_recompute.py:36-79): in fp32,
// silu(g) = g / (1 + 2^(-g * log2 e)).
#pragma once

namespace soup {

__device__ __forceinline__ float silu_denom(float g) { return 1.0f + exp2f(g * -1.4426950408889634f); }
__device__ __forceinline__ float silu_of(float g) { return __fdividef(g, silu_denom(g)); }

// sig = 1 / denom; silu'(g) = sig * (1 + g * (1 - sig))
__device__ __forceinline__ float silu_slope(float g, float sig) { return sig * (1.0f + g * (1.0f - sig)); }

}  // namespace soup

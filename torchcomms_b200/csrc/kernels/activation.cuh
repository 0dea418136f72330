// The activation of a gated MLP and its gradients, for every kernel that makes them: the same bits whichever does.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

namespace b200c {

#ifdef __CUDACC__

// 1 / (1 + exp(-g)). The hardware's reciprocal, an ulp off, and one step of Newton's iteration by fused multiply-adds, which
// rounds it correctly but for a few last-bit ties (Markstein, IBM J. Res. Dev. 34, 1990): for every bf16 gate the bits of the
// division, whose branch a warp alone on its scheduler waits for (epilogue of 4096 x 14336 x 256: 350 us with the division). An
// infinite sum has no residual to step by.
__device__ __forceinline__ float sigmoid_of(float g) {
  const float d = 1.0f + __expf(-g);
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
  return d < INFINITY ? __fmaf_rn(r, __fmaf_rn(-d, r, 1.0f), r) : r;
}

__device__ __forceinline__ float gated(float gate, float up) { return gate * sigmoid_of(gate) * up; }

// The gradients of gate and up from `d`, that of gated(gate, up).
__device__ __forceinline__ void gated_gradient(float d, float gate, float up, float* dgate, float* dup) {
  const float sig = sigmoid_of(gate);
  const float silu = gate * sig;
  *dgate = d * up * (sig + silu * (1.0f - sig));
  *dup = d * silu;
}

#endif

} // namespace b200c

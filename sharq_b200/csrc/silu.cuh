// SiLU with the bf16 bits of ATen's, shared by the SwiGLU kernel and the GEMM epilogue that applies SwiGLU.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

namespace sharq {

__device__ __forceinline__ float exp2f_approx(float v) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

__device__ __forceinline__ float rcp_approx(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// A float that rounds to the bf16 value ATen's silu gives for the bf16-exact x: x / (1 + exp(-x)) in float, rounded.
// Formed with the approximate exp2 and reciprocal units, which is within 32 float ulps of the true value for |x| <= 16; a
// bf16 rounding boundary lies that close to the exact result for no bf16 input, which the test over all 65536 inputs
// (tests/test_swiglu_gemm_gpu.py) holds the kernels to.  The factor 1/4 on the divisor (exact, undone on x) keeps its
// reciprocal a normal number up to the largest finite exp(-x), where rcp.ftz would flush it.  An accurate
// evaluation with expf and an IEEE division behind a per-element boundary test came before; without it the linears of a
// 2048-token prefill layer (SwiGLU of 2048 x 14336 among them) take 438 instead of 446 us.
__device__ __forceinline__ float silu_f32(float x) {
  const float e = exp2f_approx(-1.4426950408889634f * x);
  return __fmul_rn(0.25f * x, rcp_approx(__fmaf_rn(e, 0.25f, 0.25f)));
}

}  // namespace sharq

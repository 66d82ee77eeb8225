// Shared helpers of the model kernels (bf16 activations, fp32 statistics).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace piccl_ops {

typedef __nv_bfloat16 bf16;

struct alignas(16) bf16x8 { __nv_bfloat162 v[4]; };

__device__ __forceinline__ void unpack8(const bf16x8& p, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; i++) { float2 t = __bfloat1622float2(p.v[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
__device__ __forceinline__ bf16x8 pack8(const float (&f)[8]) {
  bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; i++) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// GPT-2's tanh GELU and its derivative, through 0.5 (1 + tanh u) = 1 / (1 + exp(-2u)): two special-function instructions in place of
// the branches of tanhf, and no cancellation in 1 + tanh u for negative u.
__device__ __forceinline__ float gelu_sigmoid(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return __fdividef(1.f, 1.f + __expf(-2.f * k0 * x * (1.f + k1 * x * x)));      // exp may be inf: 1 / inf is the 0 that is wanted
}
__device__ __forceinline__ float gelu_f(float x) { return x * gelu_sigmoid(x); }
__device__ __forceinline__ float gelu_grad_f(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float s = gelu_sigmoid(x);
  return s + 2.f * x * s * (1.f - s) * (k0 + 3.f * k0 * k1 * x * x);
}

}  // namespace piccl_ops

#define PICCL_OPS_CHECK_LAUNCH() do { cudaError_t e_ = cudaGetLastError(); if (e_ != cudaSuccess) return (int)e_; } while (0)

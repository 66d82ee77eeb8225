// Shared helpers of the model kernels (bf16 activations, fp32 statistics).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace piccl_ops {

typedef __nv_bfloat16 bf16;

// Programmatic dependent launch: the grid may start while the kernel before it on the stream still runs; what it does before
// pdl_begin() overlaps that kernel's tail, everything after it sees the kernel before completed.  A step is hundreds of kernels of 2 to
// 50 us, so the launch latency between two of them (1 us and more) counts.  Every kernel launched by launch_pdl calls pdl_begin()
// before it touches global memory, reads as well as writes.
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Status word of the current device (status.cu); null if there is no device.
enum StatusKind { STATUS_GEMM, STATUS_ATTENTION, kStatusKinds };
int* status_word(StatusKind kind);
int read_status(StatusKind kind);         // synchronises

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
// GPT-2's tanh GELU and its derivative, through 0.5 (1 + tanh u) = 1 / (1 + exp(-2u)), u = k0 (x + k1 x^3): two special-function
// instructions in place of the branches of tanhf, and no cancellation in 1 + tanh u for negative u.  Two values at a time: the
// polynomial parts run as packed fp32 pairs, since the GEMM epilogues that call these are bound by instruction issue.
__device__ __forceinline__ float ex2_approx(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float rcp_approx(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ f32x2 both2(float a) { return pack2(a, a); }
__device__ __forceinline__ float sum2(f32x2 v) { float a, b; unpack2(v, a, b); return a + b; }
__device__ __forceinline__ void unpack8(const bf16x8& p, f32x2 (&f)[4]) {
#pragma unroll
  for (int i = 0; i < 4; i++) { const float2 t = __bfloat1622float2(p.v[i]); f[i] = pack2(t.x, t.y); }
}
__device__ __forceinline__ bf16x8 pack8(const f32x2 (&f)[4]) {
  bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; i++) { float a, b; unpack2(f[i], a, b); p.v[i] = __floats2bfloat162_rn(a, b); }
  return p;
}

__device__ __forceinline__ f32x2 gelu_sigmoid2(f32x2 x, f32x2 xx) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f, c = -2.f * k0 * 1.4426950408889634f;
  const f32x2 z = mul2(x, fma2(both2(c * k1), xx, both2(c)));
  float a, b; unpack2(z, a, b);
  unpack2(add2(pack2(ex2_approx(a), ex2_approx(b)), both2(1.f)), a, b);      // exp may be inf: 1 / inf is the 0 that is wanted
  return pack2(rcp_approx(a), rcp_approx(b));
}
__device__ __forceinline__ f32x2 gelu2(f32x2 x) { return mul2(x, gelu_sigmoid2(x, mul2(x, x))); }
__device__ __forceinline__ f32x2 gelu_grad2(f32x2 x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const f32x2 xx = mul2(x, x), s = gelu_sigmoid2(x, xx);
  const f32x2 t = fma2(mul2(s, both2(-1.f)), s, s);                          // s (1 - s)
  return fma2(t, mul2(x, fma2(both2(6.f * k0 * k1), xx, both2(2.f * k0))), s);
}
// arrays of an even number of values in registers
template <int N> __device__ __forceinline__ void gelu_n(float (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) unpack2(gelu2(pack2(v[i], v[i + 1])), v[i], v[i + 1]);
}
template <int N> __device__ __forceinline__ void mul_gelu_grad_n(float* v, const float (&x)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) unpack2(mul2(pack2(v[i], v[i + 1]), gelu_grad2(pack2(x[i], x[i + 1]))), v[i], v[i + 1]);
}

}  // namespace piccl_ops

#define PICCL_OPS_CHECK_LAUNCH() do { cudaError_t e_ = cudaGetLastError(); if (e_ != cudaSuccess) return (int)e_; } while (0)

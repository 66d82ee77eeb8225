// Fused element-wise model kernels: bias + GELU (forward / backward), bias
// gradient (column sums), softmax cross entropy with in-place gradient, and a
// flat AdamW step with fp32 master weights.
#include <cstring>
#include "ops_common.cuh"

namespace piccl_ops {

// The 8 warps of a block hold sums of columns [blockIdx.x * 256, + 256), 8 to a lane: their total is row blockIdx.y of part[][C].
__device__ __forceinline__ void block_colsum(const float (&acc)[8], float* __restrict__ part, int C) {
  __shared__ float sh[8][256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int e = 0; e < 8; e++) sh[warp][lane * 8 + e] = acc[e];
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < C) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; w++) s += sh[w][threadIdx.x];
    part[(size_t)blockIdx.y * C + c] = s;
  }
}

// g = gelu(h + bias); h_out = h + bias (kept for the backward pass); h may alias h_out
__global__ void __launch_bounds__(256) bias_gelu_fwd_kernel(const bf16* __restrict__ h, const bf16* __restrict__ bias, bf16* __restrict__ h_out,
                                                            bf16* __restrict__ g, size_t n8, int C8) {
  pdl_begin();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n8; i += (size_t)gridDim.x * blockDim.x) {
    float v[8], b[8];
    unpack8(reinterpret_cast<const bf16x8*>(h)[i], v);
    if (bias) { unpack8(reinterpret_cast<const bf16x8*>(bias)[i % C8], b);
#pragma unroll
      for (int e = 0; e < 8; e++) v[e] += b[e]; }
    if (h_out) { bf16x8 p = pack8(v); reinterpret_cast<bf16x8*>(h_out)[i] = p; unpack8(p, v); }
    gelu_n(v);
    reinterpret_cast<bf16x8*>(g)[i] = pack8(v);
  }
}

// dh = dg * gelu'(h)    (h includes the bias); dh may alias dg.  Block (bx, by): 256 columns, every gridDim.y-th group of 8 rows.
// part (optional): [gridDim.y][C] column sums of the dh written, the bias gradient of the layer, taken while the rows are in
// registers instead of by a second pass over dh.
constexpr int kColRows = 4;      // rows in flight per warp
__global__ void __launch_bounds__(256) gelu_bwd_kernel(const bf16* __restrict__ dg, const bf16* __restrict__ h, bf16* __restrict__ dh, float* __restrict__ part,
                                                       long long rows, int C) {
  pdl_begin();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c8 = blockIdx.x * 32 + lane, C8 = C / 8;
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; e++) acc[e] = 0.f;
  if (c8 < C8)
    for (long long r0 = (blockIdx.y * 8ll + warp) * kColRows; r0 < rows; r0 += gridDim.y * 8ll * kColRows) {
      bf16x8 pd[kColRows], ph[kColRows];
#pragma unroll
      for (int r = 0; r < kColRows; r++)
        if (r0 + r < rows) { const size_t i = (size_t)(r0 + r) * C8 + c8; pd[r] = reinterpret_cast<const bf16x8*>(dg)[i]; ph[r] = reinterpret_cast<const bf16x8*>(h)[i]; }
#pragma unroll
      for (int r = 0; r < kColRows; r++)
        if (r0 + r < rows) {
          float d[8], v[8];
          unpack8(pd[r], d); unpack8(ph[r], v);
          mul_gelu_grad_n(d, v);
          const bf16x8 p = pack8(d);
          reinterpret_cast<bf16x8*>(dh)[(size_t)(r0 + r) * C8 + c8] = p;
          unpack8(p, d);
#pragma unroll
          for (int e = 0; e < 8; e++) acc[e] += d[e];
        }
    }
  if (part) block_colsum(acc, part, C);
}

// dqkv[b * S + s, which * H * D + head * D + d] from the three gradients of the attention, which lie as [B, H, S, D] views with
// strides sb / sh / ss (elements) and contiguous rows of D; part: [gridDim.y][3 * H * D] column sums of what is written.
struct QkvGrads { const bf16* p[3]; long long sb[3], sh[3], ss[3]; };
__global__ void __launch_bounds__(256) qkv_grad_kernel(const QkvGrads q, bf16* __restrict__ dqkv, float* __restrict__ part, int rows, int S, int H, int D) {
  pdl_begin();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, C = H * D, C3 = 3 * C;
  const int c = (blockIdx.x * 32 + lane) * 8;
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; e++) acc[e] = 0.f;
  if (c < C3) {
    const int which = c / C, head = (c - which * C) / D, d = c - which * C - head * D;
    const bf16* src = (which == 0 ? q.p[0] : which == 1 ? q.p[1] : q.p[2]) + d + head * (which == 0 ? q.sh[0] : which == 1 ? q.sh[1] : q.sh[2]);
    const long long sb = which == 0 ? q.sb[0] : which == 1 ? q.sb[1] : q.sb[2], ss = which == 0 ? q.ss[0] : which == 1 ? q.ss[1] : q.ss[2];
    for (int r0 = (blockIdx.y * 8 + warp) * kColRows; r0 < rows; r0 += gridDim.y * 8 * kColRows) {
      bf16x8 v[kColRows];
#pragma unroll
      for (int r = 0; r < kColRows; r++)
        if (r0 + r < rows) { const int b = (r0 + r) / S, s = (r0 + r) - b * S; v[r] = *reinterpret_cast<const bf16x8*>(src + b * sb + s * ss); }
#pragma unroll
      for (int r = 0; r < kColRows; r++)
        if (r0 + r < rows) {
          *reinterpret_cast<bf16x8*>(dqkv + (size_t)(r0 + r) * C3 + c) = v[r];
          float f[8]; unpack8(v[r], f);
#pragma unroll
          for (int e = 0; e < 8; e++) acc[e] += f[e];
        }
    }
  }
  block_colsum(acc, part, C3);
}

// partial column sums: block (bx, by) sums rows [by*rpb, ...) of 8*32 = 256 columns starting at bx*256
__global__ void __launch_bounds__(256) colsum_kernel(const bf16* __restrict__ x, float* __restrict__ part, int rows, int C, int rows_per_block) {
  pdl_begin();
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int c8 = blockIdx.x * 32 + lane;                 // index of the 8-column group
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; e++) acc[e] = 0.f;
  int r0 = blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  if (c8 * 8 < C)
    for (int r = r0 + warp; r < r1; r += 8) {
      float v[8]; unpack8(reinterpret_cast<const bf16x8*>(x + (size_t)r * C)[c8], v);
#pragma unroll
      for (int e = 0; e < 8; e++) acc[e] += v[e];
    }
  block_colsum(acc, part, C);
}

// out[c] (+)= sum over parts of part[p][c] for several vectors in one launch (blockIdx.y: vector, blockIdx.x: 64 columns).
// Latency bound: the partial rows are spread over the 16 warps of the block, each with 10 loads of 8 bytes a lane in flight, so a vector of 296 partial
// rows takes two round trips to L2.  The eight vectors of a layer of GPT-2 medium (12 MB):
// 5.3 us with 32 columns a block and loads of 4 bytes, now 4.3; of 8 layers of 768 columns on 3 x 777 tokens 4.9 / 4.3.
struct FinishJob { const float* part; bf16* out; int nparts, C, accumulate, pad; };
constexpr int kMaxFinish = 16;
struct FinishJobs { FinishJob j[kMaxFinish]; };
__global__ void __launch_bounds__(512) finish_parts_kernel(const __grid_constant__ FinishJobs jobs) {
  pdl_begin();
  const FinishJob& j = jobs.j[blockIdx.y];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, C = j.C, n = j.nparts;
  const int c = blockIdx.x * 64 + 2 * lane;
  if (blockIdx.x * 64 >= C) return;
  float2 s = make_float2(0.f, 0.f);
  if (c < C) {
    const float* p = j.part + c;
    const bool pairs = ((C | (int)(reinterpret_cast<uintptr_t>(j.part) >> 2)) & 1) == 0;      // else a row's pair may straddle its word or its end
    constexpr int U = 10;
    for (int r = warp; r < n; r += 16 * U) {
      float2 v[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const float* q = p + (size_t)(r + u * 16) * C;
        v[u] = make_float2(0.f, 0.f);
        if (r + u * 16 < n) {
          if (pairs) v[u] = *reinterpret_cast<const float2*>(q);
          else { v[u].x = q[0]; if (c + 1 < C) v[u].y = q[1]; }
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) { s.x += v[u].x; s.y += v[u].y; }
    }
  }
  __shared__ float2 sh[16][32];
  sh[warp][lane] = s;
  __syncthreads();
  const int col = blockIdx.x * 64 + threadIdx.x;
  if (threadIdx.x < 64 && col < C) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 16; w++) t += reinterpret_cast<const float*>(sh[w])[threadIdx.x];
    if (j.accumulate) t += __bfloat162float(j.out[col]);
    j.out[col] = __float2bfloat16_rn(t);
  }
}

// One block per row: loss[row] = logsumexp(logits[:V]) - logits[target]; logits <- (softmax - onehot) * gscale
// (columns V..Vp-1 are padding: ignored in the sum, gradient zero).
__global__ void __launch_bounds__(512) ce_fwd_bwd_kernel(bf16* __restrict__ logits, const long long* __restrict__ targets, float* __restrict__ loss,
                                                         int V, int Vp, float gscale) {
  pdl_begin();
  int row = blockIdx.x, tid = threadIdx.x;
  bf16* lp = logits + (size_t)row * Vp;
  const int n8 = Vp / 8;
  float m = -INFINITY, s = 0.f;
  for (int i = tid; i < n8; i += blockDim.x) {
    float v[8]; unpack8(reinterpret_cast<const bf16x8*>(lp)[i], v);
    float lm = m;
#pragma unroll
    for (int e = 0; e < 8; e++) if (i * 8 + e < V) lm = fmaxf(lm, v[e]);
    float acc = 0.f;
#pragma unroll
    for (int e = 0; e < 8; e++) if (i * 8 + e < V) acc += __expf(v[e] - lm);
    s = s * __expf(m - lm) + acc; m = lm;
  }
  __shared__ float shm[16], shs[16];
  // combine (m, s) pairs: first in the warp, then across warps
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
    float mm = fmaxf(m, m2);
    s = (m == -INFINITY ? 0.f : s * __expf(m - mm)) + (m2 == -INFINITY ? 0.f : s2 * __expf(m2 - mm)); m = mm;
  }
  int warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  if (lane == 0) { shm[warp] = m; shs[warp] = s; }
  __syncthreads();
  float M = -INFINITY;
  for (int w = 0; w < nw; w++) M = fmaxf(M, shm[w]);
  float S = 0.f;
  for (int w = 0; w < nw; w++) if (shm[w] != -INFINITY) S += shs[w] * __expf(shm[w] - M);
  long long t = targets[row];
  float inv = 1.f / S;
  if (tid == 0) loss[row] = (t >= 0 && t < V) ? (logf(S) + M - __bfloat162float(lp[t])) : 0.f;
  __syncthreads();     // the target logit is read before anybody overwrites it
  const bool valid = t >= 0 && t < V;
  for (int i = tid; i < n8; i += blockDim.x) {
    float v[8], o[8]; unpack8(reinterpret_cast<const bf16x8*>(lp)[i], v);
#pragma unroll
    for (int e = 0; e < 8; e++) {
      int c = i * 8 + e;
      float p = (c < V && valid) ? __expf(v[e] - M) * inv : 0.f;
      if (c == t) p -= 1.f;
      o[e] = p * gscale;
    }
    reinterpret_cast<bf16x8*>(lp)[i] = pack8(o);
  }
}

// What a thread has seen of a row so far: maximum and sum of exp(x - maximum).  The maximum is taken off before the value is scaled to base 2:
// one fma of both would round maximum * log2(e), and the sum would be off by that (3e-5 at logits around 400).
struct OnlineSum {
  float m = -INFINITY, s = 0.f;
  static constexpr float kLog2e = 1.4426950408889634f;
  __device__ __forceinline__ void add(const f32x2 x2, float neg_m, f32x2& a) {
    float x, y; unpack2(mul2(add2(x2, both2(neg_m)), both2(kLog2e)), x, y);
    a = add2(a, pack2(ex2_approx(x), ex2_approx(y)));
  }
  template <int N> __device__ __forceinline__ void packs(const bf16x8 (&p)[N]) {
    __nv_bfloat162 q = p[0].v[0];
#pragma unroll
    for (int u = 0; u < N; u++)
#pragma unroll
      for (int e = 0; e < 4; e++) q = __hmax2(q, p[u].v[e]);
    const float top = fmaxf(__low2float(q), __high2float(q));
    if (top > m) { s *= ex2_approx((m - top) * kLog2e); m = top; }               // at first 0 * exp(-inf)
    const float neg_m = m == -INFINITY ? 0.f : -m;
    f32x2 a[2] = {both2(0.f), both2(0.f)};
#pragma unroll
    for (int u = 0; u < N; u++) {
      float v[8]; unpack8(p[u], v);
#pragma unroll
      for (int e = 0; e < 8; e += 2) add(pack2(v[e], v[e + 1]), neg_m, a[(e >> 1) & 1]);
    }
    float x, y; unpack2(add2(a[0], a[1]), x, y);
    s += x + y;
  }
  // all threads of a block of W warps: the whole row's m and s
  template <int W> __device__ __forceinline__ void block(float2 (&sh)[W]) {
    const float wm = warp_max(m);
    const float ws = warp_sum(wm == -INFINITY ? 0.f : s * ex2_approx((m - wm) * kLog2e));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = make_float2(wm, ws);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const float2 w = lane < W ? sh[lane] : make_float2(-INFINITY, 0.f);
    m = warp_max(w.x);
    s = warp_sum(w.x == -INFINITY ? 0.f : w.y * ex2_approx((w.x - m) * kLog2e));
  }
};
// columns from V on are padding
__device__ __forceinline__ bf16x8 mask_padding(bf16x8 p, int col, int V) {
  float v[8]; unpack8(p, v);
#pragma unroll
  for (int e = 0; e < 8; e++) if (col + e >= V) v[e] = -INFINITY;
  return pack8(v);
}
// exp(x - m) / s * gs of a pack; ls = -log2 s
__device__ __forceinline__ bf16x8 ce_gradient(const bf16x8& p, float neg_m, float ls, float gs) {
  float v[8]; unpack8(p, v);
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    float x, y; unpack2(fma2(add2(pack2(v[e], v[e + 1]), both2(neg_m)), both2(OnlineSum::kLog2e), both2(ls)), x, y);
    unpack2(mul2(pack2(ex2_approx(x), ex2_approx(y)), both2(gs)), v[e], v[e + 1]);
  }
  return pack8(v);
}
// the target's column has gs less
__device__ __forceinline__ bf16 ce_gradient_target(float x, float neg_m, float ls, float gs) { return __float2bfloat16_rn(ex2_approx(fmaf(x + neg_m, OnlineSum::kLog2e, ls)) * gs - gs); }

// The same in one pass over memory: the sum of exponentials is taken while the row comes in, relative to the thread's maximum so far, and
// the gradient needs the row once more, from shared memory.  GRAD = false leaves the logits as they are and keeps nothing.
// Two blocks share an SM: one loads while the other computes.  8192 x 50304: 364 us with the gradient, 183 without (372 and 193 from a cold L2; 386 and 219 with a pass
// of its own for the sum; the copy rate allows 252 and 126, the special-function units 183 and 92).  One block per SM with the next row
// on its way to a second buffer was slower, 492 us.
template <bool GRAD>
__global__ void __launch_bounds__(512, 2) ce_row_kernel(bf16* __restrict__ logits, const long long* __restrict__ targets, float* __restrict__ loss, int V, int Vp, float gscale) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char ce_smem[];
  bf16x8* const row_s = reinterpret_cast<bf16x8*>(ce_smem);
  __shared__ float2 sh[16];
  const int row = blockIdx.x, tid = threadIdx.x;
  bf16x8* lp = reinterpret_cast<bf16x8*>(logits + (size_t)row * Vp);
  const int n8 = Vp / 8, full8 = V / 8;               // packs [full8, n8) hold padding columns
  const long long t = targets[row];
  const bool valid = t >= 0 && t < V;
  const bool owner = valid ? (int)(t >> 3) % 512 == tid : tid == 0;      // has the target's pack
  const float xt = valid && owner ? __bfloat162float(reinterpret_cast<const bf16*>(lp)[t]) : 0.f;
  OnlineSum o;
  int i = tid;
  for (; i + 3 * 512 < full8; i += 4 * 512) {
    bf16x8 p[4];
#pragma unroll
    for (int u = 0; u < 4; u++) p[u] = lp[i + u * 512];
    if (GRAD) {
#pragma unroll
      for (int u = 0; u < 4; u++) row_s[i + u * 512] = p[u];
    }
    o.packs(p);
  }
  for (; i < n8; i += 512) {
    const bf16x8 p[1] = {i < full8 ? lp[i] : mask_padding(lp[i], i * 8, V)};
    if (GRAD) row_s[i] = p[0];
    o.packs(p);
  }
  o.block(sh);
  if (owner) loss[row] = valid ? logf(o.s) + (o.m - xt) : 0.f;
  if (!GRAD) return;
  const float ls = -log2f(o.s);
#pragma unroll 1       // stores in bursts of four cost a quarter of the time
  for (i = tid; i < n8; i += 512) lp[i] = ce_gradient(row_s[i], -o.m, ls, valid ? gscale : 0.f);
  if (valid && owner) reinterpret_cast<bf16*>(lp)[t] = ce_gradient_target(xt, -o.m, ls, gscale);
}

// out[0] = mean of x[0..n), one block; not a number where a word of `status` (optional) is set
__global__ void __launch_bounds__(1024) mean_kernel(const float* __restrict__ x, float* __restrict__ out, int n, const int* status) {
  pdl_begin();
  int failed = 0;
  if (status && threadIdx.x == 0) for (int i = 0; i < kStatusKinds; i++) failed |= status[i];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += 1024) s += x[i];
  __shared__ float sh[32];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = warp_sum(sh[threadIdx.x]);
    if (threadIdx.x == 0) out[0] = failed ? __int_as_float(0x7fffffff) : s / (float)n;
  }
}

// AdamW on flat buffers: bf16 gradient and parameter, fp32 master copy and moments.
__global__ void __launch_bounds__(256) adamw_kernel(bf16* __restrict__ p, float* __restrict__ master, float* __restrict__ m, float* __restrict__ v,
                                                    const bf16* __restrict__ g, size_t n8, float lr, float b1, float b2, float eps, float wd,
                                                    float bc1, float bc2, float gscale, const int* __restrict__ step_dev) {
  pdl_begin();
  if (step_dev) {   // step number kept on the device (the launch can then be replayed from a CUDA graph)
    const float st = (float)*step_dev;
    bc1 = 1.f - powf(b1, st); bc2 = 1.f - powf(b2, st);
  }
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n8; i += (size_t)gridDim.x * blockDim.x) {
    float gv[8]; unpack8(reinterpret_cast<const bf16x8*>(g)[i], gv);
    float4 w0 = reinterpret_cast<float4*>(master)[2 * i], w1 = reinterpret_cast<float4*>(master)[2 * i + 1];
    float4 m0 = reinterpret_cast<float4*>(m)[2 * i], m1 = reinterpret_cast<float4*>(m)[2 * i + 1];
    float4 v0 = reinterpret_cast<float4*>(v)[2 * i], v1 = reinterpret_cast<float4*>(v)[2 * i + 1];
    float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
    float mm[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
    float vv[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
    for (int e = 0; e < 8; e++) {
      float gr = gv[e] * gscale;
      mm[e] = b1 * mm[e] + (1.f - b1) * gr;
      vv[e] = b2 * vv[e] + (1.f - b2) * gr * gr;
      float upd = (mm[e] / bc1) / (sqrtf(vv[e] / bc2) + eps);
      w[e] = w[e] * (1.f - lr * wd) - lr * upd;
    }
    reinterpret_cast<float4*>(master)[2 * i] = make_float4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<float4*>(master)[2 * i + 1] = make_float4(w[4], w[5], w[6], w[7]);
    reinterpret_cast<float4*>(m)[2 * i] = make_float4(mm[0], mm[1], mm[2], mm[3]);
    reinterpret_cast<float4*>(m)[2 * i + 1] = make_float4(mm[4], mm[5], mm[6], mm[7]);
    reinterpret_cast<float4*>(v)[2 * i] = make_float4(vv[0], vv[1], vv[2], vv[3]);
    reinterpret_cast<float4*>(v)[2 * i + 1] = make_float4(vv[4], vv[5], vv[6], vv[7]);
    reinterpret_cast<bf16x8*>(p)[i] = pack8(w);
  }
}

// AdamW over all parameters in one launch: run g of the flat buffers ends before pack ends[g] (8 elements), runs of parity
// `decay_parity` decay.  The step number is the device's own (*step holds the steps done so far); the last block to finish advances it.
constexpr int kMaxRuns = 1024;
__global__ void __launch_bounds__(256) adamw_runs_kernel(bf16* __restrict__ p, float* __restrict__ master, float* __restrict__ m, float* __restrict__ v,
                                                         const bf16* __restrict__ g, const int* __restrict__ ends, int nruns, int decay_parity, size_t n8,
                                                         float lr, float b1, float b2, float eps, float wd, int* __restrict__ step, unsigned* __restrict__ ticket) {
  pdl_begin();
  __shared__ int s_end[kMaxRuns];
  for (int i = threadIdx.x; i < nruns; i += 256) s_end[i] = ends[i];
  const float st = (float)(*(volatile int*)step + 1);
  const float rbc1 = 1.f / (1.f - powf(b1, st)), rbc2 = 1.f / (1.f - powf(b2, st));
  __syncthreads();
  const size_t stride = (size_t)gridDim.x * 256;
  int run = 0;
  for (size_t i = blockIdx.x * 256ull + threadIdx.x; i < n8; i += stride) {
    const bf16x8 gp = reinterpret_cast<const bf16x8*>(g)[i];
    float4 wa[2], ma[2], va[2];
#pragma unroll
    for (int h = 0; h < 2; h++) { wa[h] = reinterpret_cast<float4*>(master)[2 * i + h]; ma[h] = reinterpret_cast<float4*>(m)[2 * i + h]; va[h] = reinterpret_cast<float4*>(v)[2 * i + h]; }
    while (run + 1 < nruns && i >= (size_t)s_end[run]) run++;
    const float keep = 1.f - lr * (((run & 1) == decay_parity) ? wd : 0.f);
    float gv[8]; unpack8(gp, gv);
    float* w = reinterpret_cast<float*>(wa); float* mm = reinterpret_cast<float*>(ma); float* vv = reinterpret_cast<float*>(va);
#pragma unroll
    for (int e = 0; e < 8; e++) {
      mm[e] = b1 * mm[e] + (1.f - b1) * gv[e];
      vv[e] = b2 * vv[e] + (1.f - b2) * gv[e] * gv[e];
      w[e] = w[e] * keep - lr * (mm[e] * rbc1) / (sqrtf(vv[e] * rbc2) + eps);
    }
#pragma unroll
    for (int h = 0; h < 2; h++) { reinterpret_cast<float4*>(master)[2 * i + h] = wa[h]; reinterpret_cast<float4*>(m)[2 * i + h] = ma[h]; reinterpret_cast<float4*>(v)[2 * i + h] = va[h]; }
    float o[8];
#pragma unroll
    for (int e = 0; e < 8; e++) o[e] = w[e];
    reinterpret_cast<bf16x8*>(p)[i] = pack8(o);
  }
  __syncthreads();                                    // every thread has read *step
  if (threadIdx.x == 0 && atomicAdd(ticket, 1u) == gridDim.x - 1) { *ticket = 0; atomicAdd(step, 1); }
}

// out[r, :] = wte[idx[r], :] + wpe[r % S, :]
__global__ void __launch_bounds__(128) embed_fwd_kernel(const long long* __restrict__ idx, const bf16* __restrict__ wte, const bf16* __restrict__ wpe,
                                                        bf16* __restrict__ out, int rows, int S, int C8) {
  pdl_begin();
  int row = blockIdx.x;
  long long t = idx[row];
  const bf16x8* a = reinterpret_cast<const bf16x8*>(wte) + (size_t)t * C8;
  const bf16x8* b = reinterpret_cast<const bf16x8*>(wpe) + (size_t)(row % S) * C8;
  for (int i = threadIdx.x; i < C8; i += blockDim.x) {
    float x[8], y[8]; unpack8(a[i], x); unpack8(b[i], y);
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] += y[e];
    reinterpret_cast<bf16x8*>(out)[(size_t)row * C8 + i] = pack8(x);
  }
}

// dwpe[s, :] (+)= sum over batch of dx[b*S + s, :]   (one block per row of the table; deterministic).  Positions from S on, which no token
// of this batch had, get the empty sum.
__global__ void __launch_bounds__(128) wpe_bwd_kernel(const bf16* __restrict__ dx, bf16* __restrict__ dwpe, int B, int S, int C8, int accumulate) {
  pdl_begin();
  int s = blockIdx.x;
  if (s >= S) B = 0;
  for (int i = threadIdx.x; i < C8; i += blockDim.x) {
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; e++) acc[e] = 0.f;
    for (int b = 0; b < B; b++) {
      float v[8]; unpack8(reinterpret_cast<const bf16x8*>(dx)[((size_t)b * S + s) * C8 + i], v);
#pragma unroll
      for (int e = 0; e < 8; e++) acc[e] += v[e];
    }
    if (accumulate) { float o[8]; unpack8(reinterpret_cast<const bf16x8*>(dwpe)[(size_t)s * C8 + i], o);
#pragma unroll
      for (int e = 0; e < 8; e++) acc[e] += o[e]; }
    reinterpret_cast<bf16x8*>(dwpe)[(size_t)s * C8 + i] = pack8(acc);
  }
}

// dwte[idx[r], :] += dx[r, :] in fp32 (atomics on an fp32 staging table), then folded into the bf16 gradient
__global__ void __launch_bounds__(128) wte_bwd_scatter_kernel(const long long* __restrict__ idx, const bf16* __restrict__ dx, float* __restrict__ stage, int C) {
  pdl_begin();
  int row = blockIdx.x; long long t = idx[row];
  for (int c = threadIdx.x; c < C; c += blockDim.x) atomicAdd(&stage[(size_t)t * C + c], __bfloat162float(dx[(size_t)row * C + c]));
}
__global__ void __launch_bounds__(256) add_f32_into_bf16_kernel(const float* __restrict__ src, bf16* __restrict__ dst, size_t n) {
  pdl_begin();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = __float2bfloat16_rn(__bfloat162float(dst[i]) + src[i]);
}

// dwte[v, :] += sum of dx[r, :] over the rows with idx[r] = v, touching only the rows of the table that occur.  stage (fp32 [V, C]) is
// all zero before and after; owner[v] names one of the rows that hold v: its block folds the sum and clears it again.
__global__ void __launch_bounds__(128) wte_scatter_rows_kernel(const long long* __restrict__ idx, const bf16* __restrict__ dx, float* __restrict__ stage, int* __restrict__ owner, int C8) {
  pdl_begin();
  const int row = blockIdx.x; const long long t = idx[row];
  if (threadIdx.x == 0) owner[t] = row;
  float4* dst = reinterpret_cast<float4*>(stage) + (size_t)t * C8 * 2;
  for (int i = threadIdx.x; i < C8; i += 128) {
    float v[8]; unpack8(reinterpret_cast<const bf16x8*>(dx)[(size_t)row * C8 + i], v);
#pragma unroll
    for (int h = 0; h < 2; h++)
      asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + 2 * i + h), "f"(v[4 * h]), "f"(v[4 * h + 1]), "f"(v[4 * h + 2]), "f"(v[4 * h + 3]) : "memory");
  }
}
__global__ void __launch_bounds__(128) wte_fold_rows_kernel(const long long* __restrict__ idx, float* __restrict__ stage, const int* __restrict__ owner, bf16* __restrict__ dwte, int C8) {
  pdl_begin();
  const int row = blockIdx.x; const long long t = idx[row];
  if (owner[t] != row) return;
  float4* src = reinterpret_cast<float4*>(stage) + (size_t)t * C8 * 2;
  bf16x8* dst = reinterpret_cast<bf16x8*>(dwte) + (size_t)t * C8;
  for (int i = threadIdx.x; i < C8; i += 128) {
    float v[8]; unpack8(dst[i], v);
    const float4 a = src[2 * i], b = src[2 * i + 1];
    v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w; v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
    dst[i] = pack8(v);
    src[2 * i] = make_float4(0.f, 0.f, 0.f, 0.f); src[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

}  // namespace piccl_ops

using namespace piccl_ops;

static int grid_for(size_t n, int block) { size_t g = (n + block - 1) / block; return (int)(g > 148 * 16 ? 148 * 16 : (g ? g : 1)); }

extern "C" {

int piccl_ops_bias_gelu_fwd(const void* h, const void* bias, void* h_out, void* g, long long rows, int C, void* stream) {
  if (C % 8) return -1;
  if ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(h_out) | reinterpret_cast<uintptr_t>(g)) & 15) return -2;      // 16-byte words
  size_t n8 = (size_t)rows * C / 8;
  launch_pdl(bias_gelu_fwd_kernel, grid_for(n8, 256), 256, 0, (cudaStream_t)stream, (const bf16*)h, (const bf16*)bias, (bf16*)h_out, (bf16*)g, n8, C / 8);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
// Row groups (partial rows) of the kernels that walk C columns of a [rows, C] matrix 256 at a time: four blocks per SM
int piccl_ops_col_parts(long long rows, int C) {
  const long long bx = (C + 255) / 256, most = (rows + 8 * kColRows - 1) / (8 * kColRows);
  const long long n = 148 * 4 / bx;
  return (int)(n < 1 ? 1 : n < most ? n : most > 0 ? most : 1);
}
// part: null, or piccl_ops_col_parts(rows, C) * C floats that receive partial column sums of dh
int piccl_ops_gelu_bwd(const void* dg, const void* h, void* dh, float* part, long long rows, int C, void* stream) {
  if (C % 8) return -1;
  launch_pdl(gelu_bwd_kernel, dim3((C + 255) / 256, piccl_ops_col_parts(rows, C)), 256, 0, (cudaStream_t)stream, (const bf16*)dg, (const bf16*)h, (bf16*)dh, part, rows, C);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
// g[3]: gradients of q, k, v; strides: {sb, sh, ss} of each in elements (multiples of 8, the rows 16-byte aligned);
// part: piccl_ops_col_parts(B * S, 3 * H * D) * 3 * H * D floats
int piccl_ops_qkv_grad(const void* const* g, const long long* strides, void* dqkv, float* part, int B, int S, int H, int D, void* stream) {
  if (D % 8) return -1;
  QkvGrads q;
  for (int i = 0; i < 3; i++) {
    q.p[i] = (const bf16*)g[i]; q.sb[i] = strides[3 * i]; q.sh[i] = strides[3 * i + 1]; q.ss[i] = strides[3 * i + 2];
    if ((q.sb[i] | q.sh[i] | q.ss[i]) % 8 || (uintptr_t)g[i] % 16) return -2;
  }
  const int C3 = 3 * H * D;
  launch_pdl(qkv_grad_kernel, dim3((C3 + 255) / 256, piccl_ops_col_parts((long long)B * S, C3)), 256, 0, (cudaStream_t)stream, q, (bf16*)dqkv, part, B * S, S, H, D);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
// Folds the partial rows of up to 16 vectors into their bf16 results in one launch.
int piccl_ops_finish_parts(const void* jobs, int n, void* stream) {
  if (n < 1 || n > kMaxFinish) return -1;
  FinishJobs a; memset(&a, 0, sizeof a); memcpy(&a, jobs, n * sizeof(FinishJob));
  int c = 0;
  for (int i = 0; i < n; i++) c = a.j[i].C > c ? a.j[i].C : c;
  launch_pdl(finish_parts_kernel, dim3((c + 63) / 64, n), 512, 0, (cudaStream_t)stream, a);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
// workspace: ceil(rows / rows_per_block) * C floats; out null: the partial rows are left there
int piccl_ops_colsum(const void* x, void* out, float* workspace, int rows, int C, int rows_per_block, int accumulate, void* stream) {
  if (C % 8) return -1;
  int nparts = (rows + rows_per_block - 1) / rows_per_block;
  launch_pdl(colsum_kernel, dim3((C + 255) / 256, nparts), 256, 0, (cudaStream_t)stream, (const bf16*)x, workspace, rows, C, rows_per_block);
  PICCL_OPS_CHECK_LAUNCH();
  if (!out) return 0;
  const FinishJob j{workspace, (bf16*)out, nparts, C, accumulate, 0};
  return piccl_ops_finish_parts(&j, 1, stream);
}
// grad = 0: losses only, the logits stay as they are.
int piccl_ops_ce(void* logits, const long long* targets, float* loss, int rows, int V, int Vp, float gscale, int grad, void* stream) {
  if (Vp % 8 || V > Vp) return -1;
  const int smem = Vp * 2, most = 220 * 1024;        // a row fits one SM (two up to 56 Ki columns); beyond, the gradient takes the two-pass kernel
  cudaStream_t s = (cudaStream_t)stream;
  if (!grad) launch_pdl(ce_row_kernel<false>, rows, 512, 0, s, (bf16*)logits, targets, loss, V, Vp, gscale);
  else if (smem <= most) {
    static bool ready[64] = {false};
    int dev = 0; cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !ready[dev]) {
      if (cudaFuncSetAttribute(ce_row_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess) return -4;
      ready[dev] = true;
    }
    launch_pdl(ce_row_kernel<true>, rows, 512, smem, s, (bf16*)logits, targets, loss, V, Vp, gscale);
  } else launch_pdl(ce_fwd_bwd_kernel, rows, 512, 0, s, (bf16*)logits, targets, loss, V, Vp, gscale);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
int piccl_ops_ce_fwd_bwd(void* logits, const long long* targets, float* loss, int rows, int V, int Vp, float gscale, void* stream) {
  return piccl_ops_ce(logits, targets, loss, rows, V, Vp, gscale, 1, stream);
}
int piccl_ops_mean(const float* x, float* out, int n, void* stream) {
  if (n < 1) return -1;
  launch_pdl(mean_kernel, 1, 1024, 0, (cudaStream_t)stream, x, out, n, nullptr);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
// The same at the end of a pass: not a number where a wait of a GEMM or attention kernel on this device ran out, in this pass or an earlier one (piccl_ops_status tells which).
int piccl_ops_pass_loss(const float* rows, float* loss, int n, void* stream) {
  if (n < 1) return -1;
  const int* status = status_word(STATUS_GEMM);
  if (!status) return -7;
  launch_pdl(mean_kernel, 1, 1024, 0, (cudaStream_t)stream, rows, loss, n, status);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
// One AdamW step over flat buffers of n elements that alternate between decaying and non-decaying runs: ends[i] (device) is the end of
// run i in packs of 8 elements, runs with (i & 1) == decay_parity decay.  step / ticket: device ints, the steps done so far and a zero.
int piccl_ops_adamw_runs(void* p, float* master, float* m, float* v, const void* g, long long n, const int* ends, int nruns, int decay_parity, float lr, float b1, float b2,
                         float eps, float wd, int* step, unsigned* ticket, void* stream) {
  if (n % 8 || nruns < 1 || nruns > kMaxRuns || n / 8 > 0x7fffffffll) return -1;
  const size_t n8 = (size_t)n / 8;
  launch_pdl(adamw_runs_kernel, grid_for(n8, 256), 256, 0, (cudaStream_t)stream, (bf16*)p, master, m, v, (const bf16*)g, ends, nruns, decay_parity, n8, lr, b1, b2, eps, wd, step, ticket);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
int piccl_ops_adamw(void* p, float* master, float* m, float* v, const void* g, long long n, float lr, float b1, float b2, float eps, float wd,
                    int step, float gscale, void* stream) {
  if (n % 8) return -1;
  float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  launch_pdl(adamw_kernel, grid_for(n / 8, 256), 256, 0, (cudaStream_t)stream, (bf16*)p, master, m, v, (const bf16*)g, (size_t)n / 8, lr, b1, b2, eps, wd, bc1, bc2, gscale, nullptr);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
// Same update with the step number read from device memory (`step_dev`, an int the caller advances on the device).
int piccl_ops_adamw_devstep(void* p, float* master, float* m, float* v, const void* g, long long n, float lr, float b1, float b2, float eps, float wd,
                            const int* step_dev, float gscale, void* stream) {
  if (n % 8 || !step_dev) return -1;
  launch_pdl(adamw_kernel, grid_for(n / 8, 256), 256, 0, (cudaStream_t)stream, (bf16*)p, master, m, v, (const bf16*)g, (size_t)n / 8, lr, b1, b2, eps, wd, 1.f, 1.f, gscale, step_dev);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
int piccl_ops_embed_fwd(const long long* idx, const void* wte, const void* wpe, void* out, int rows, int S, int C, void* stream) {
  if (C % 8) return -1;
  launch_pdl(embed_fwd_kernel, rows, 128, 0, (cudaStream_t)stream, idx, (const bf16*)wte, (const bf16*)wpe, (bf16*)out, rows, S, C / 8);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
// rows: rows of dwpe that are written, S or more
int piccl_ops_wpe_bwd(const void* dx, void* dwpe, int B, int S, int rows, int C, int accumulate, void* stream) {
  if (C % 8 || rows < S) return -1;
  launch_pdl(wpe_bwd_kernel, rows, 128, 0, (cudaStream_t)stream, (const bf16*)dx, (bf16*)dwpe, B, S, C / 8, accumulate);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}
// stage: fp32 [V, C], zeroed by the caller
int piccl_ops_wte_bwd(const long long* idx, const void* dx, float* stage, void* dwte, int rows, long long V, int C, void* stream) {
  launch_pdl(wte_bwd_scatter_kernel, rows, 128, 0, (cudaStream_t)stream, idx, (const bf16*)dx, stage, C);
  size_t n = (size_t)V * C;
  launch_pdl(add_f32_into_bf16_kernel, grid_for(n, 256), 256, 0, (cudaStream_t)stream, stage, (bf16*)dwte, n);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}

// stage: fp32 [V, C], all zero (and left so); owner: V ints, any content
int piccl_ops_wte_bwd_rows(const long long* idx, const void* dx, float* stage, int* owner, void* dwte, int rows, int C, void* stream) {
  if (C % 8) return -1;
  launch_pdl(wte_scatter_rows_kernel, rows, 128, 0, (cudaStream_t)stream, idx, (const bf16*)dx, stage, owner, C / 8);
  launch_pdl(wte_fold_rows_kernel, rows, 128, 0, (cudaStream_t)stream, idx, stage, owner, (bf16*)dwte, C / 8);
  PICCL_OPS_CHECK_LAUNCH(); return 0;
}

}  // extern "C"

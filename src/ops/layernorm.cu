// Fused residual-add + LayerNorm, forward and backward (bf16 data, fp32 statistics).
// One warp per row, rows of C = 8*32*V elements held in registers, a single pass
// over HBM in each direction.  The residual sum is produced by the same kernel,
// so the x + f(x) tensors of a transformer block are never a separate pass.
#include "ops_common.cuh"

namespace piccl_ops {

// y = LN(x + res) * gamma + beta ; sum_out = x + res (optional)
// Memory bound: up to 4 tensors of rows * C bf16.  The grid is what the chip holds at once; a warp loads its next row before it works on the
// one it has, so that 4 KiB per warp are always on their way at C = 1024 (16 to 20 warps an SM: more than the 44 KB that
// cover the latency).  8192 x 1024: 18.6 -> 17.3 us without the L2, 10.3 at the copy rate of a long copy.
constexpr int ln_fwd_blocks(int V) { return V == 1 ? 10 : V == 2 ? 6 : V <= 4 ? 5 : V <= 6 ? 4 : 3; }      // of 4 warps per SM
template <int V, bool RES>   // V 16-byte vectors per lane: C = 256 * V
__global__ void __launch_bounds__(128, ln_fwd_blocks(V)) ln_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res, const bf16* __restrict__ gamma,
                                                                       const bf16* __restrict__ beta, bf16* __restrict__ sum_out, bf16* __restrict__ y,
                                                                       float* __restrict__ mean, float* __restrict__ rstd, int rows, float eps) {
  pdl_begin();
  constexpr int C = 256 * V;
  const int lane = threadIdx.x & 31, step = gridDim.x * 4;
  int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) return;
  bf16x8 px[V], pr[V];
  auto load = [&](int r) {
#pragma unroll
    for (int i = 0; i < V; i++) {
      px[i] = reinterpret_cast<const bf16x8*>(x)[(size_t)r * (C / 8) + lane + 32 * i];
      if (RES) pr[i] = reinterpret_cast<const bf16x8*>(res)[(size_t)r * (C / 8) + lane + 32 * i];
    }
  };
  load(row);
  for (; row < rows; row += step) {
    float v[V][8];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < V; i++) {
      unpack8(px[i], v[i]);
      if (RES) {
        float r[8]; unpack8(pr[i], r);
#pragma unroll
        for (int e = 0; e < 8; e++) v[i][e] += r[e];
      }
      if (sum_out) {
        const bf16x8 p = pack8(v[i]);
        reinterpret_cast<bf16x8*>(sum_out)[(size_t)row * (C / 8) + lane + 32 * i] = p;
        unpack8(p, v[i]);          // normalise exactly what was stored
      }
#pragma unroll
      for (int e = 0; e < 8; e++) s += v[i][e];
    }
    if (row + step < rows) load(row + step);
    const float mu = warp_sum(s) / C;
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < V; i++)
#pragma unroll
      for (int e = 0; e < 8; e++) { const float d = v[i][e] - mu; q += d * d; }
    const float rs = rsqrtf(warp_sum(q) / C + eps);
    if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
#pragma unroll
    for (int i = 0; i < V; i++) {
      float g[8], b[8], o[8];
      unpack8(reinterpret_cast<const bf16x8*>(gamma)[lane + 32 * i], g);
      unpack8(reinterpret_cast<const bf16x8*>(beta)[lane + 32 * i], b);
#pragma unroll
      for (int e = 0; e < 8; e++) o[e] = (v[i][e] - mu) * rs * g[e] + b[e];
      reinterpret_cast<bf16x8*>(y)[(size_t)row * (C / 8) + lane + 32 * i] = pack8(o);
    }
  }
}

// dx = LN-backward(dy) + dres ; per-block partial column sums in fp32: part[0] = dgamma, part[1] = dbeta and, with_dsum, part[2] = sum
// of the dx written (dx is the gradient that enters the layer before, whose bias gradient is exactly that sum: the kernel that
// has the rows in registers adds them up, so nobody reads dx again for it).
// Memory bound: 4 tensors of rows * C bf16.  A row is spread over V warps (8 columns a thread), so the three accumulators cost 24
// registers instead of the 96 of a warp per row at C = 1024, and R rows are in flight per group; G groups of V warps make a
// block of about 8 warps.  The grid is what the chip holds at once: each block leaves one partial row per vector.  The next rows are loaded
// while those at hand wait for their sums (8192 x 1024: 19.7 -> 17.6 us without the L2, 10.3 at the copy rate of a long copy).
template <int V, int G, int R, bool RES>   // C = 256 * V
__global__ void __launch_bounds__(32 * V * G, 2) ln_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ xin, const bf16* __restrict__ gamma,
                                                               const float* __restrict__ mean, const float* __restrict__ rstd, const bf16* __restrict__ dres,
                                                               bf16* __restrict__ dx, float* __restrict__ part, int rows, int with_dsum) {
  pdl_begin();
  constexpr int C = 256 * V;
  __shared__ float red[2][G][V][2 * R];
  __shared__ float sh[G][C];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = warp / V, wv = warp % V;
  const int c8 = wv * 32 + lane;
  float ga[8], dg[8], db[8], ds[8];
  unpack8(reinterpret_cast<const bf16x8*>(gamma)[c8], ga);
#pragma unroll
  for (int e = 0; e < 8; e++) { dg[e] = 0.f; db[e] = 0.f; ds[e] = 0.f; }
  int buf = 0;
  bf16x8 ny[R], nx[R], nr[R];                          // the rows to come: loaded while those before them are worked on
  float nmu[R], nrs[R];
  auto load = [&](int r0) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int row = min(r0 + r, rows - 1);
      const size_t o = (size_t)row * (C / 8) + c8;
      ny[r] = reinterpret_cast<const bf16x8*>(dy)[o];
      nx[r] = reinterpret_cast<const bf16x8*>(xin)[o];
      if (RES) nr[r] = reinterpret_cast<const bf16x8*>(dres)[o];
      nmu[r] = mean[row]; nrs[r] = rstd[row];
    }
  };
  const int step = gridDim.x * G * R;
  int r0 = (blockIdx.x * G + g) * R;
  if (r0 < rows) load(r0);
  for (; r0 < rows; r0 += step, buf ^= 1) {
    bf16x8 py[R], px[R], pr[R];
    float mu[R], rs[R];
#pragma unroll
    for (int r = 0; r < R; r++) { py[r] = ny[r]; px[r] = nx[r]; if (RES) pr[r] = nr[r]; mu[r] = nmu[r]; rs[r] = nrs[r]; }
    if (r0 + step < rows) load(r0 + step);
    float s[2 * R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      s[2 * r] = 0.f; s[2 * r + 1] = 0.f;
      if (r0 + r < rows) {
        float x[8], y[8];
        unpack8(px[r], x); unpack8(py[r], y);
#pragma unroll
        for (int e = 0; e < 8; e++) {
          const float xh = (x[e] - mu[r]) * rs[r], t = y[e] * ga[e];
          dg[e] += y[e] * xh; db[e] += y[e];
          s[2 * r] += t; s[2 * r + 1] += t * xh;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2 * R; i++) s[i] = warp_sum(s[i]);
    if (V > 1) {
      if (lane == 0) {
#pragma unroll
        for (int i = 0; i < 2 * R; i++) red[buf][g][wv][i] = s[i];
      }
      asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(32 * V) : "memory");      // the other buffer is free: its readers have passed this barrier
#pragma unroll
      for (int i = 0; i < 2 * R; i++) {
        s[i] = 0.f;
#pragma unroll
        for (int w = 0; w < V; w++) s[i] += red[buf][g][w][i];
      }
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (r0 + r < rows) {
        const float s1 = s[2 * r] * (1.f / C), s2 = s[2 * r + 1] * (1.f / C);
        float x[8], y[8], o[8];
        unpack8(px[r], x); unpack8(py[r], y);
        if (RES) unpack8(pr[r], o);
        else {
#pragma unroll
          for (int e = 0; e < 8; e++) o[e] = 0.f;
        }
#pragma unroll
        for (int e = 0; e < 8; e++) o[e] += rs[r] * (y[e] * ga[e] - s1 - (x[e] - mu[r]) * rs[r] * s2);
        const bf16x8 p = pack8(o);
        reinterpret_cast<bf16x8*>(dx)[(size_t)(r0 + r) * (C / 8) + c8] = p;
        if (with_dsum) {
          unpack8(p, o);
#pragma unroll
          for (int e = 0; e < 8; e++) ds[e] += o[e];
        }
      }
    }
  }
  // one partial row per block and vector
#pragma unroll
  for (int vec = 0; vec < 3; vec++) {
    if (vec == 2 && !with_dsum) break;
#pragma unroll
    for (int e = 0; e < 8; e++) sh[g][c8 * 8 + e] = vec == 0 ? dg[e] : vec == 1 ? db[e] : ds[e];
    __syncthreads();
    float* dst = part + ((size_t)vec * gridDim.x + blockIdx.x) * C;
    for (int c = threadIdx.x; c < C; c += 32 * V * G) {
      float t = 0.f;
#pragma unroll
      for (int q = 0; q < G; q++) t += sh[q][c];
      dst[c] = t;
    }
    __syncthreads();
  }
}

}  // namespace piccl_ops

using namespace piccl_ops;

extern "C" {

// C must be 256, 512, 768, 1024, 1280, 1536 or 2048.  res / sum_out may be null.
int piccl_ops_ln_fwd(const void* x, const void* res, const void* gamma, const void* beta, void* sum_out, void* y, float* mean, float* rstd,
                     int rows, int C, float eps, void* stream) {
  const int need = (rows + 3) / 4;
  cudaStream_t s = (cudaStream_t)stream;
#define LN_CASE(V) case 256 * V: launch_pdl(res ? ln_fwd_kernel<V, true> : ln_fwd_kernel<V, false>, need < 148 * ln_fwd_blocks(V) ? need : 148 * ln_fwd_blocks(V), 128, 0, s, (const bf16*)x, (const bf16*)res, (const bf16*)gamma, (const bf16*)beta, (bf16*)sum_out, (bf16*)y, mean, rstd, rows, eps); break;
  switch (C) { LN_CASE(1) LN_CASE(2) LN_CASE(3) LN_CASE(4) LN_CASE(5) LN_CASE(6) LN_CASE(8) default: return -1; }
#undef LN_CASE
  PICCL_OPS_CHECK_LAUNCH();
  return 0;
}

// Blocks, that is partial rows per vector, that piccl_ops_ln_bwd leaves for `rows` rows of C columns (0: C is not supported).
int piccl_ops_ln_bwd_parts(int rows, int C) {
  int per = 0;                                       // rows a block has in flight
  switch (C) { case 256: per = 8 * 2; break; case 512: per = 4 * 2; break; case 768: case 1024: per = 2 * 2; break; default: return 0; }
  const int n = (rows + per - 1) / per;
  return n < 296 ? (n > 0 ? n : 1) : 296;            // two blocks on each of 148 SMs
}

// part: [2 or 3][piccl_ops_ln_bwd_parts(rows, C)][C] floats, see the kernel; piccl_ops_finish_parts folds them.
int piccl_ops_ln_bwd(const void* dy, const void* xin, const void* gamma, const float* mean, const float* rstd, const void* dres, void* dx,
                     float* part, int with_dsum, int rows, int C, void* stream) {
  const int nb = piccl_ops_ln_bwd_parts(rows, C);
  if (!nb) return -1;
  cudaStream_t s = (cudaStream_t)stream;
#define LN_CASE(V, G) case 256 * V: launch_pdl(dres ? ln_bwd_kernel<V, G, 2, true> : ln_bwd_kernel<V, G, 2, false>, nb, 32 * V * G, 0, s, (const bf16*)dy, (const bf16*)xin, (const bf16*)gamma, mean, rstd, (const bf16*)dres, (bf16*)dx, part, rows, with_dsum); break;
  switch (C) { LN_CASE(1, 8) LN_CASE(2, 4) LN_CASE(3, 2) LN_CASE(4, 2) default: return -1; }
#undef LN_CASE
  PICCL_OPS_CHECK_LAUNCH();
  return 0;
}

}  // extern "C"

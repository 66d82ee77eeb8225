// Fused residual-add + LayerNorm, forward and backward (bf16 data, fp32 statistics).
// One warp per row, rows of C = 8*32*V elements held in registers, a single pass
// over HBM in each direction.  The residual sum is produced by the same kernel,
// so the x + f(x) tensors of a transformer block are never a separate pass.
#include "ops_common.cuh"

namespace piccl_ops {

// y = LN(x + res) * gamma + beta ; sum_out = x + res (optional)
// Up to 4 tensors of rows * C bf16.  The grid is what the chip holds at once; a warp loads its next row before it works on the one it has, so
// that 4 KiB per warp are always on their way at C = 1024 (20 warps an SM: more than the 44 KB that cover the latency).  gamma and beta come
// from shared memory and the arithmetic runs on pairs: reading them from the L1 again for each row and with
// an instruction per element the kernel was bound by its load queue and by issue (32768 x 1024: 56.4 us, now 44.5, 41.1 at the copy rate;
// 8192 x 1024: 17.2 us, now 14.1 without the L2).
constexpr int ln_fwd_blocks(int V) { return V == 1 ? 10 : V == 2 ? 6 : V <= 4 ? 5 : V <= 6 ? 4 : 3; }      // of 4 warps per SM
template <int V, bool RES>   // V 16-byte vectors per lane: C = 256 * V
__global__ void __launch_bounds__(128, ln_fwd_blocks(V)) ln_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res, const bf16* __restrict__ gamma,
                                                                       const bf16* __restrict__ beta, bf16* __restrict__ sum_out, bf16* __restrict__ y,
                                                                       float* __restrict__ mean, float* __restrict__ rstd, int rows, float eps) {
  pdl_begin();
  constexpr int C = 256 * V;
  const int lane = threadIdx.x & 31, step = gridDim.x * 4;
  int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  __shared__ bf16x8 sg[V * 32], sb[V * 32];
  bf16x8 px[V], pr[V];
  auto load = [&](int r) {
#pragma unroll
    for (int i = 0; i < V; i++) {
      px[i] = reinterpret_cast<const bf16x8*>(x)[(size_t)r * (C / 8) + lane + 32 * i];
      if (RES) pr[i] = reinterpret_cast<const bf16x8*>(res)[(size_t)r * (C / 8) + lane + 32 * i];
    }
  };
  if (row < rows) load(row);
  for (int i = threadIdx.x; i < V * 32; i += 128) { sg[i] = reinterpret_cast<const bf16x8*>(gamma)[i]; sb[i] = reinterpret_cast<const bf16x8*>(beta)[i]; }
  __syncthreads();
  for (; row < rows; row += step) {
    f32x2 v[V][4];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < V; i++) {
      unpack8(px[i], v[i]);
      if (RES) {
        f32x2 r[4]; unpack8(pr[i], r);
#pragma unroll
        for (int e = 0; e < 4; e++) v[i][e] = add2(v[i][e], r[e]);
      }
      if (sum_out) {
        const bf16x8 p = pack8(v[i]);
        reinterpret_cast<bf16x8*>(sum_out)[(size_t)row * (C / 8) + lane + 32 * i] = p;
        unpack8(p, v[i]);          // normalise exactly what was stored
      }
#pragma unroll
      for (int e = 0; e < 4; e++) { float a, b; unpack2(v[i][e], a, b); s += a; s += b; }
    }
    if (row + step < rows) load(row + step);
    const float mu = warp_sum(s) / C;
    const f32x2 neg_mu = both2(-mu);
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < V; i++)
#pragma unroll
      for (int e = 0; e < 4; e++) { v[i][e] = add2(v[i][e], neg_mu); float a, b; unpack2(v[i][e], a, b); q = fmaf(a, a, q); q = fmaf(b, b, q); }
    const float rs = rsqrtf(warp_sum(q) / C + eps);
    const f32x2 rs2 = both2(rs);
    if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
#pragma unroll
    for (int i = 0; i < V; i++) {
      f32x2 g[4], b[4];
      unpack8(sg[lane + 32 * i], g); unpack8(sb[lane + 32 * i], b);
#pragma unroll
      for (int e = 0; e < 4; e++) v[i][e] = fma2(mul2(v[i][e], rs2), g[e], b[e]);
      reinterpret_cast<bf16x8*>(y)[(size_t)row * (C / 8) + lane + 32 * i] = pack8(v[i]);
    }
  }
}

// dx = LN-backward(dy) + dres ; per-block partial column sums in fp32: part[0] = dgamma, part[1] = dbeta and, with_dsum, part[2] = sum
// of the dx written (dx is the gradient that enters the layer before, whose bias gradient is exactly that sum: the kernel that
// has the rows in registers adds them up, so nobody reads dx again for it).
// 4 tensors of rows * C bf16.  A row is spread over V warps (8 columns a thread), so the three accumulators cost 24
// registers instead of the 96 of a warp per row at C = 1024, and R rows are in flight per group; G groups of V warps make a
// block of about 8 warps.  The grid is what the chip holds at once: each block leaves one partial row per vector.  The next rows are loaded
// while those at hand wait for their sums, the arithmetic runs on pairs and the four sums of two rows are reduced together: 2 instructions
// in 3 had been shuffles, conversions and single additions (32768 x 1024: 58.1 -> 55.4 us, 41.1 at the copy rate; 8192 x 1024: 16.7 us).
// What is left is the wait for the sums, with 16 warps an SM.
template <int V, int G, int R, bool RES>   // C = 256 * V
__global__ void __launch_bounds__(32 * V * G, 2) ln_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ xin, const bf16* __restrict__ gamma,
                                                               const float* __restrict__ mean, const float* __restrict__ rstd, const bf16* __restrict__ dres,
                                                               bf16* __restrict__ dx, float* __restrict__ part, int rows, int with_dsum) {
  pdl_begin();
  constexpr int C = 256 * V;
  static_assert(R == 2, "four sums are reduced together");
  __shared__ float4 red[2][G][V];
  __shared__ float sh[G][C];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = warp / V, wv = warp % V;
  const int c8 = wv * 32 + lane;
  f32x2 ga[4], dg[4], db[4], ds[4];
  unpack8(reinterpret_cast<const bf16x8*>(gamma)[c8], ga);
#pragma unroll
  for (int e = 0; e < 4; e++) { dg[e] = both2(0.f); db[e] = both2(0.f); ds[e] = both2(0.f); }
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
    f32x2 t[R][4], xh[R][4];                           // dy * gamma and the normalised input
    bf16x8 pr[R];
    float s[2 * R], rs[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      const bool in = r0 + r < rows;
      f32x2 y[4];
      unpack8(nx[r], xh[r]); unpack8(ny[r], y);
      if (RES) pr[r] = nr[r];
      rs[r] = nrs[r];
      const f32x2 neg_mu = both2(-nmu[r]), rs2 = both2(rs[r]);
      f32x2 s1 = both2(0.f), s2 = both2(0.f);
#pragma unroll
      for (int e = 0; e < 4; e++) {
        if (!in) y[e] = both2(0.f);                    // a row beyond the last one adds nothing
        xh[r][e] = mul2(add2(xh[r][e], neg_mu), rs2);
        t[r][e] = mul2(y[e], ga[e]);
        dg[e] = fma2(y[e], xh[r][e], dg[e]);
        db[e] = add2(db[e], y[e]);
        s1 = add2(s1, t[r][e]);
        s2 = fma2(t[r][e], xh[r][e], s2);
      }
      s[2 * r] = sum2(s1); s[2 * r + 1] = sum2(s2);
    }
    if (r0 + step < rows) load(r0 + step);
    // the four sums over the warp together: each exchange halves what a lane still has to add, lanes 8 i to 8 i + 7 end up with sum i
    const bool hi = lane & 16, odd = lane & 8;
    float a = hi ? s[2] : s[0], b = hi ? s[3] : s[1];
    a += __shfl_xor_sync(0xffffffffu, hi ? s[0] : s[2], 16);
    b += __shfl_xor_sync(0xffffffffu, hi ? s[1] : s[3], 16);
    float c = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (V > 1) {
      if ((lane & 7) == 0) reinterpret_cast<float*>(&red[buf][g][wv])[lane >> 3] = c;
      asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(32 * V) : "memory");      // the other buffer is free: its readers have passed this barrier
      float4 w = red[buf][g][0];
#pragma unroll
      for (int i = 1; i < V; i++) { const float4 u = red[buf][g][i]; w.x += u.x; w.y += u.y; w.z += u.z; w.w += u.w; }
      s[0] = w.x; s[1] = w.y; s[2] = w.z; s[3] = w.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++) s[i] = __shfl_sync(0xffffffffu, c, 8 * i);
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (r0 + r < rows) {
        const f32x2 neg_s1 = both2(s[2 * r] * (-1.f / C)), neg_s2 = both2(s[2 * r + 1] * (-1.f / C)), rs2 = both2(rs[r]);
        f32x2 o[4];
        if (RES) unpack8(pr[r], o);
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const f32x2 d = fma2(xh[r][e], neg_s2, add2(t[r][e], neg_s1));
          o[e] = RES ? fma2(d, rs2, o[e]) : mul2(d, rs2);
        }
        const bf16x8 p = pack8(o);
        reinterpret_cast<bf16x8*>(dx)[(size_t)(r0 + r) * (C / 8) + c8] = p;
        if (with_dsum) {
          unpack8(p, o);
#pragma unroll
          for (int e = 0; e < 4; e++) ds[e] = add2(ds[e], o[e]);
        }
      }
    }
  }
  // one partial row per block and vector
#pragma unroll
  for (int vec = 0; vec < 3; vec++) {
    if (vec == 2 && !with_dsum) break;
#pragma unroll
    for (int e = 0; e < 4; e++) unpack2(vec == 0 ? dg[e] : vec == 1 ? db[e] : ds[e], sh[g][c8 * 8 + 2 * e], sh[g][c8 * 8 + 2 * e + 1]);
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

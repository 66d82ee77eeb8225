// Causal attention of heads of 64 columns on the tensor cores of sm_100a, forward and backward, on the packed rows [q | k | v] that the
// product before it writes; the backward kernels write the packed gradient that the products after them read, and leave its partial column
// sums (the bias gradient) on the way.  Nothing is transposed, converted or summed by another kernel, and no sum depends on timing: two runs
// give the same bits.
//
// Three kernels of one build.  A CTA has a tile of 128 rows (queries; keys in the kernel of dK and dV) and walks the other side in steps of 64.
// Eight warps hold the tile's rows, one row per thread (TMEM lane = row) and each row twice; one warp brings the steps' tiles by TMA,
// one issues the MMAs.  The 128 x 64 scores of a step appear in TMEM, the threads turn them into bf16 probabilities (or score gradients) and
// put them back into TMEM, where they are the A operand of the next product: they never pass through shared memory.
//   forward   S = Q K^T            P = softmax     O  += P V
//   dQ        S, dP = dO V^T       dS = P (dP - d) dQ += dS K
//   dK, dV    S^T, dP^T            P^T, dS^T       dV += P^T dO, dK += dS^T Q
// (Two backward kernels compute S and dP twice, 7 products in place of 5; one kernel would have to add its dQ tiles up in memory, 32 KiB
// of fp32 atomics for each 128 x 128 scores, and to clear and convert them.)
// TMEM is 256 columns a CTA, so two CTAs share an SM: one computes exponentials while the other one's products run.  A step of 128 x 64 scores is
// 512 clocks of an SM's special-function units (16 results a clock) and 256 / 384 / 640 of its tensor cores (forward, dQ, dK and dV; the last
// reads K and V from shared memory for every step); what is measured is 1070 / 1100 / 1550, most of it the way from one product through
// the threads to the next and the start and end of a CTA.  (A third of the exponentials as polynomials on the fma units changed nothing.)
// 8 x 1024 tokens, 16 heads, within a training step of GPT-2 medium: backward 112 us, where cuDNN's kernel with the sum o * do, the conversion of dQ and the
// packing and column sums of the gradient took 123 in five launches; forward 41, cuDNN 40.  Back to back on a stream: 8 x 1024 tokens 35 and 95, 3 x 777 with 12 heads 13.7 and 36.3,
// 4 x 128 with 4 heads 4.5 and 9.9.
// Blocks are ordered by falling length of their walk.
#include <cstring>
#include <mutex>
#include "../include/sm100_gemm_pair.cuh"
#include "ops_common.cuh"

namespace piccl_ops {

using namespace sm100;

constexpr int AT_ROWS = 128, AT_STEP = 64, AT_D = 64, AT_STAGES = 4, AT_THREADS = 320, AT_TMEM = 256;
constexpr int AT_LOAD = 8, AT_MMA = 9;                   // warps: 0 to 7 hold rows, 4 to 7 the same ones as 0 to 3
constexpr int AT_TILE = AT_STEP * AT_D * 2;              // bytes of a step's tile: 64 rows of 128 bytes, 128-byte swizzle
constexpr unsigned long long kAttnWaitLimitNs = 4000000000ull;

struct AttnArgs {
  CUtensorMap qkv, out, dout, result;   // 64 rows of the packed rows, of the output and its gradient; 32 rows of the result
  const float* lse_in;                  // [B * H][S] logarithm of the row's sum of exponentials
  float *lse_out, *lse, *delta, *part;  // the same; [B * H][tiles * 128] minus that to base 2 (-inf beyond S), minus the sum of o * do; [B * tiles][3 H D]
  int B, S, H, tiles;
  int* status;
};
constexpr float kAttnScale = 0.125f, kAttnLog2 = 0.125f * 1.4426950408889634f;      // 1 / sqrt(64), and to base 2

struct AttnSmem {
  static constexpr int STAGE = 2 * AT_TILE, RING = AT_STAGES * STAGE;
  static constexpr int OWN = RING, OWN_BYTES = 2 * AT_ROWS * AT_D * 2;      // the tile's own operands (Q; Q and dO; K and V), its results on their way out
  static constexpr int ROWS = OWN + OWN_BYTES;                              // lse and delta of a step of queries; what the warps of a row exchange; column sums
  static constexpr int BARS = ROWS + AT_STAGES * 2 * AT_STEP * 4;
  static constexpr int DYNAMIC = BARS + 256 + 1024;                         // slack for the alignment of the tiles
};

// What every warp of a CTA knows.
struct AttnCtx {
  uint8_t* smem;
  uint64_t *full, *empty;                                // per stage of the ring
  uint64_t *ready, *s_full, *p_full, *acc_done;          // two each but the first: by step parity in the forward kernel, [0] alone elsewhere
  uint64_t *dp_full, *ds_full, *sums, *own;              // sums: two
  uint32_t tmem;
  volatile int* abort;
  __device__ bool wait(uint64_t* bar, uint32_t parity) const { return mbar_wait(bar, parity, abort, kAttnWaitLimitNs); }
};

// rows: warps that hold rows and arrive together; ready: arrivals that make the tile's own operands complete.  first(): the loads that need nothing but the
// barriers; the loading warp starts them while TMEM is allocated and the CTA assembles (a thousand clocks).
template <class F>
__device__ __forceinline__ void attn_begin(AttnCtx& c, uint8_t* raw, int* s_abort, uint32_t* s_tmem, int warp, int rows, int ready, const F& first) {
  c.smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  uint64_t* b = reinterpret_cast<uint64_t*>(c.smem + AttnSmem::BARS);
  c.full = b; c.empty = b + AT_STAGES; b += 2 * AT_STAGES;
  c.ready = b; c.s_full = b + 1; c.p_full = b + 3; c.acc_done = b + 5; c.dp_full = b + 7; c.ds_full = b + 8; c.sums = b + 9; c.own = b + 11;
  c.abort = s_abort;
  if (warp == AT_LOAD && elect_one()) {
    *s_abort = 0;
    for (int i = 0; i < AT_STAGES; i++) { mbar_init(&c.full[i], 1); mbar_init(&c.empty[i], 1); }
    for (int i = 0; i < 2; i++) { mbar_init(&c.s_full[i], 1); mbar_init(&c.p_full[i], rows); mbar_init(&c.acc_done[i], 1); mbar_init(&c.sums[i], 4); }
    mbar_init(c.ready, ready); mbar_init(c.dp_full, 1); mbar_init(c.ds_full, rows); mbar_init(c.own, 1);
    fence_barrier_init();
    pdl_begin();
    first(c);
  }
  if (warp == AT_MMA) tmem_alloc_cta(s_tmem, AT_TMEM);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  c.tmem = *s_tmem;
  pdl_begin();
}
__device__ __forceinline__ void attn_end(const AttnCtx& c, int warp, int lane) {
  if (warp < 8 && lane == 0) bulk_wait_read_all();
  tc_fence_before();
  __syncthreads();
  if (*c.abort) {                                        // copies in flight get time to land
    const unsigned long long t0 = gtime_ns();
    while (gtime_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == AT_MMA) { tc_fence_after(); tmem_dealloc_cta(c.tmem, AT_TMEM); }
}

// row r of a tile in shared memory -> 32 registers of pairs
__device__ __forceinline__ void load_row(const uint8_t* tile, int r, uint32_t (&x)[32]) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const uint4 v = *reinterpret_cast<const uint4*>(tile + r * 128 + ((i ^ (r & 7)) << 4));
    x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
  }
}
__device__ __forceinline__ float max3(float a, float b, float c) { float r; asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ void ex2_pair(f32x2 x, float& a, float& b) { unpack2(x, a, b); a = ex2_approx(a); b = ex2_approx(b); }
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) { const __nv_bfloat162 h = __floats2bfloat162_rn(a, b); return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {      // what the warp read from or wrote to TMEM comes before
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// 32 columns of a result's row -> half `half` of the warp's piece: 32 rows of 128 bytes in the layout of a swizzled store
__device__ __forceinline__ void stage_half(uint8_t* piece, int half, const float (&v)[32], int lane) {
#pragma unroll
  for (int j = 0; j < 4; j++) {
    uint4 o;
    o.x = pack_bf16(v[8 * j], v[8 * j + 1]); o.y = pack_bf16(v[8 * j + 2], v[8 * j + 3]); o.z = pack_bf16(v[8 * j + 4], v[8 * j + 5]); o.w = pack_bf16(v[8 * j + 6], v[8 * j + 7]);
    *reinterpret_cast<uint4*>(piece + lane * 128 + (((4 * half + j) ^ (lane & 7)) << 4)) = o;
  }
}
__device__ __forceinline__ void store_piece(const AttnArgs& a, const uint8_t* piece, int col, int row0, int b, int lane) {
  fence_proxy_async();
  __syncwarp();
  if (lane == 0 && row0 < a.S) { tma_store_3d(&a.result, piece, col, row0, b); bulk_commit(); }
}
// The four warps of a tile: 64 columns of an accumulator times f -> result, and the sums of its columns (rows beyond S are zero) -> part[0..63].
__device__ __forceinline__ bool store_gradient(const AttnCtx& c, const AttnArgs& a, uint32_t tmem, float f, uint8_t* piece, int col, int row0, int b, float* sums, uint64_t* bar, float* part,
                                               int warp, int lane) {
#pragma unroll
  for (int q = 0; q < 2; q++) {
    uint32_t r[32]; float v[32];
    tmem_ld_32x32(tmem + 32 * q, r);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]) * f;
    stage_half(piece, q, v, lane);
  }
  store_piece(a, piece, col, row0, b, lane);
  float s0 = 0.f, s1 = 0.f;
#pragma unroll
  for (int r = 0; r < 32; r++) {
    const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(piece + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4));
    s0 += x.x; s1 += x.y;
  }
  reinterpret_cast<float2*>(sums + warp * 64)[lane] = make_float2(s0, s1);
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
  if (warp >= 2) return true;
  if (!c.wait(bar, 0)) return false;
  const float* s = sums + warp * 32 + lane;
  part[warp * 32 + lane] = (s[0] + s[64]) + (s[128] + s[192]);
  return true;
}

// K = 64; a_step: columns between the second and the third 16 k of A (halves that two groups of warps wrote are 32 apart)
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t at, int a_step, uint64_t db, int b_step, uint32_t idesc, bool fresh) {
#pragma unroll
  for (int k = 0; k < 4; k++) umma_f16_ts(d, at + a_step * (k >> 1) + 8 * (k & 1), desc_advance(db, k * b_step), idesc, !fresh || k != 0);
}
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc) {
#pragma unroll
  for (int k = 0; k < 4; k++) umma_f16_ss(d, desc_advance(da, k * 32), desc_advance(db, k * 32), idesc, k != 0);
}

// The tiles of the steps, through a ring of STAGES: columns x0 of map 0 and x1 of map 1, rows 64 * (first + j), and those rows of r0 and r1.
struct AttnSteps {
  const CUtensorMap *m0, *m1;
  int x0, x1, first, steps, b;
  const float *r0, *r1;
  __device__ __forceinline__ void load(const AttnCtx& c, int j, int st) const {      // one thread
    uint8_t* s = c.smem + st * AttnSmem::STAGE;
    mbar_arrive_expect_tx(&c.full[st], AttnSmem::STAGE + (r0 ? 2 * AT_STEP * 4 : 0));
    tma_load_3d(s, m0, x0, (first + j) * AT_STEP, b, &c.full[st]);
    tma_load_3d(s + AT_TILE, m1, x1, (first + j) * AT_STEP, b, &c.full[st]);
    if (r0) {
      uint8_t* q = c.smem + AttnSmem::ROWS + st * 2 * AT_STEP * 4;
      bulk_load(q, r0 + (first + j) * AT_STEP, AT_STEP * 4, &c.full[st]);
      bulk_load(q + AT_STEP * 4, r1 + (first + j) * AT_STEP, AT_STEP * 4, &c.full[st]);
    }
  }
  template <int STAGES> __device__ __forceinline__ void begin(const AttnCtx& c) const { for (int j = 0; j < STAGES && j < steps; j++) load(c, j, j); }      // one thread
  template <int STAGES> __device__ __forceinline__ bool rest(const AttnCtx& c) const {
    const bool issuer = elect_one();
    for (int j = STAGES; j < steps; j++) {
      const int st = j % STAGES;
      if (!c.wait(&c.empty[st], ((j / STAGES) & 1) ^ 1)) return false;
      if (issuer) load(c, j, st);
      __syncwarp();
    }
    return true;
  }
};
// 128 rows of a matrix -> 16 KiB of shared memory
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* m, int x, int row0, int b, uint64_t* bar) {
  for (int i = 0; i < 2; i++) tma_load_3d(dst + i * AT_TILE, m, x, row0 + i * AT_STEP, b, bar);
}

constexpr uint32_t kIdescK = make_idesc_bf16_major(AT_ROWS, AT_STEP, false, false), kIdescMN = make_idesc_bf16_major(AT_ROWS, AT_D, false, true);

// ------------------------------------------------------------------ forward
// The two groups of four warps take the steps in turn, each with a maximum, a sum and an accumulator of its own; they are put together at the end.
// TMEM columns: O 0 and 64, S 128 and 192 (P of a step lies over its S).  A row's maximum is raised only when the new one is more than 2^8
// above it (the conditional rescaling of FlashAttention-4): until then the sums stay within range, and the accumulator is scaled a few times a row instead of at every step.
__global__ void __launch_bounds__(AT_THREADS, 2) attn_fwd_kernel(const __grid_constant__ AttnArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ int s_abort;
  __shared__ uint32_t s_tmem;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int heads = a.B * a.H, tile = a.tiles - 1 - blockIdx.x / heads, bh = blockIdx.x % heads, b = bh / a.H, h = bh % a.H, C = a.H * AT_D, q0 = tile * AT_ROWS;
  const int steps = (min(a.S, q0 + AT_ROWS) + AT_STEP - 1) / AT_STEP;
  constexpr uint32_t T_O = 0, T_S = 128;
  const AttnSteps keys{&a.qkv, &a.qkv, C + h * AT_D, 2 * C + h * AT_D, 0, steps, b, nullptr, nullptr};
  AttnCtx c;
  attn_begin(c, smem_raw, &s_abort, &s_tmem, warp, 4, 1, [&](const AttnCtx& c) {
    mbar_arrive_expect_tx(c.ready, 2 * AT_TILE);
    load_tile(c.smem + AttnSmem::OWN, &a.qkv, h * AT_D, q0, b, c.ready);
    keys.begin<AT_STAGES>(c);
  });
  bool ok = true;

  if (warp == AT_LOAD) ok = keys.rest<AT_STAGES>(c);
  else if (warp == AT_MMA) {
    const bool issuer = elect_one();
    const uint64_t dq = make_smem_desc_k128(c.smem + AttnSmem::OWN), dk0 = make_smem_desc_k128(c.smem), dv0 = make_smem_desc_mn128(c.smem + AT_TILE);
    auto scores = [&](int j) {
      const int st = j % AT_STAGES;
      if (!c.wait(&c.full[st], (j / AT_STAGES) & 1)) return false;
      tc_fence_after();
      if (issuer) { mma_ss(c.tmem + T_S + 64 * (j & 1), dq, desc_advance(dk0, st * AttnSmem::STAGE), kIdescK); umma_commit_cta(&c.s_full[j & 1]); }
      __syncwarp();
      return true;
    };
    ok = c.wait(c.ready, 0) && scores(0) && (steps < 2 || scores(1));
    for (int j = 0; ok && j < steps; j++) {
      if (!c.wait(&c.p_full[j & 1], (j >> 1) & 1)) { ok = false; break; }
      tc_fence_after();
      const int st = j % AT_STAGES;
      if (issuer) {
        mma_ts(c.tmem + T_O + 64 * (j & 1), c.tmem + T_S + 64 * (j & 1), 16, desc_advance(dv0, st * AttnSmem::STAGE), 2048, kIdescMN, j < 2);
        umma_commit_cta(&c.empty[st]);
        umma_commit_cta(&c.acc_done[j & 1]);
      }
      __syncwarp();
      if (j + 2 < steps && !scores(j + 2)) { ok = false; break; }
    }
  } else {
    const int g = warp >> 2, r = (warp & 3) * 32 + lane, row = q0 + r, turns = (steps - g + 1) / 2;
    const uint32_t lanes = c.tmem + ((uint32_t)((warp & 3) * 32) << 16), ts = lanes + T_S + 64 * g, to = lanes + T_O + 64 * g;
    float m = -INFINITY, l = 0.f;
    for (int i = 0; i < turns; i++) {
      const int k0 = (2 * i + g) * AT_STEP;
      if (!c.wait(&c.s_full[g], i & 1)) { ok = false; break; }
      tc_fence_after();
      uint32_t r0[32], r1[32];
      tmem_ld_32x32(ts, r0);
      tmem_ld_32x32(ts + 32, r1);
      tmem_ld_wait();
      const int last = row - k0;                         // the last key of the step that the row sees
      if (k0 + AT_STEP - 1 > q0 + (warp & 3) * 32) {
#pragma unroll
        for (int e = 0; e < 32; e++) { if (e > last) r0[e] = 0xff800000u; if (e + 32 > last) r1[e] = 0xff800000u; }
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int e = 0; e < 32; e++) mx[e & 3] = max3(mx[e & 3], __uint_as_float(r0[e]), __uint_as_float(r1[e]));
      const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      // Every warp sees every phase of its accumulator's barrier: the next product waits for the arrival below, so phase i - 1 is the one at hand.
      if (i > 0 && !c.wait(&c.acc_done[g], (i - 1) & 1)) { ok = false; break; }
      const bool raise = (top - m) * kAttnLog2 > 8.f;    // at first from -inf
      if (__any_sync(0xffffffffu, raise)) {
        const float f = raise ? ex2_approx((m - top) * kAttnLog2) : 1.f;
        if (raise) m = top;
        l *= f;
        if (i > 0) {
          tc_fence_after();
#pragma unroll
          for (int q = 0; q < 4; q++) {
            uint32_t o[16];
            tmem_ld_32x16(to + 16 * q, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; e++) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
            tmem_st_32x16(to + 16 * q, o);
          }
        }
      }
      // a row that has seen nothing yet (steps beyond its diagonal) keeps -inf
      const f32x2 c2 = both2(kAttnLog2), n2 = both2(m == -INFINITY ? 0.f : -m * kAttnLog2);
      f32x2 s2[2] = {both2(0.f), both2(0.f)};
#pragma unroll
      for (int e = 0; e < 32; e++) {
        float x, y;
        const uint32_t* s = e < 16 ? r0 + 2 * e : r1 + 2 * (e - 16);
        ex2_pair(fma2(pack2(__uint_as_float(s[0]), __uint_as_float(s[1])), c2, n2), x, y);
        s2[e & 1] = add2(s2[e & 1], pack2(x, y));
        r0[e] = pack_bf16(x, y);                         // (the words from 2 e on are still to be read: e <= 2 e)
      }
      tmem_st_32x32(ts, r0);
      tmem_st_wait();
      warp_arrive(&c.p_full[g], lane);
      l += sum2(add2(s2[0], s2[1]));
    }
    float2* const other = reinterpret_cast<float2*>(c.smem + AttnSmem::ROWS);
    if (ok && turns > 0) ok = c.wait(&c.acc_done[g], (turns - 1) & 1);
    if (ok && g == 1) {
      other[r] = make_float2(m, l);
      warp_arrive(c.sums, lane);
    } else if (ok && c.wait(c.sums, 0)) {
      tc_fence_after();
      const float2 w = other[r];
      const float top = fmaxf(m, w.x);                   // finite: key 0 is in a step of group 0
      const float f0 = ex2_approx((m - top) * kAttnLog2), f1 = w.x == -INFINITY ? 0.f : ex2_approx((w.x - top) * kAttnLog2), sum = l * f0 + w.y * f1, inv = 1.f / sum;
      if (a.lse_out && row < a.S) a.lse_out[(size_t)bh * a.S + row] = fmaf(top, kAttnScale, logf(sum));
      uint8_t* const piece = c.smem + AttnSmem::OWN + warp * 4096;      // Q has been read for the last time
#pragma unroll
      for (int q = 0; q < 2; q++) {
        uint32_t r0[32]; float v[32];
        tmem_ld_32x32(lanes + T_O + 32 * q, r0);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; e++) v[e] = __uint_as_float(r0[e]) * (f0 * inv);
        if (steps > 1) {
          tmem_ld_32x32(lanes + T_O + 64 + 32 * q, r0);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e++) v[e] = fmaf(__uint_as_float(r0[e]), f1 * inv, v[e]);
        }
        stage_half(piece, q, v, lane);
      }
      store_piece(a, piece, h * AT_D, q0 + warp * 32, b, lane);
    } else ok = false;
  }
  if (!ok) { *c.abort = 1; if (lane == 0) atomicExch(a.status, 10 + warp); }
  attn_end(c, warp, lane);
}

// ------------------------------------------------------------------ gradient of the queries
// Both groups of four warps work on every step, on 32 columns each.
// TMEM columns: Q 0, dO 32, dQ 64, S 128, dP 192 (dS lies over dP, so that the next step's S is computed while a step's dS is).
__global__ void __launch_bounds__(AT_THREADS, 2) attn_dq_kernel(const __grid_constant__ AttnArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ int s_abort;
  __shared__ uint32_t s_tmem;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int heads = a.B * a.H, tile = a.tiles - 1 - blockIdx.x / heads, bh = blockIdx.x % heads, b = bh / a.H, h = bh % a.H, C = a.H * AT_D, q0 = tile * AT_ROWS;
  const int steps = (min(a.S, q0 + AT_ROWS) + AT_STEP - 1) / AT_STEP;
  constexpr int STAGES = AT_STAGES - 1;                  // the last stage's place has the tile of the output
  constexpr uint32_t T_Q = 0, T_DO = 32, T_DQ = 64, T_S = 128, T_DP = 192;
  const AttnSteps keys{&a.qkv, &a.qkv, C + h * AT_D, 2 * C + h * AT_D, 0, steps, b, nullptr, nullptr};
  AttnCtx c;
  attn_begin(c, smem_raw, &s_abort, &s_tmem, warp, 8, 8, [&](const AttnCtx& c) {
    uint8_t* const t = c.smem + AttnSmem::OWN;
    mbar_arrive_expect_tx(c.own, 6 * AT_TILE);
    load_tile(t, &a.qkv, h * AT_D, q0, b, c.own); load_tile(t + 2 * AT_TILE, &a.dout, h * AT_D, q0, b, c.own); load_tile(c.smem + STAGES * AttnSmem::STAGE, &a.out, h * AT_D, q0, b, c.own);
    keys.begin<STAGES>(c);
  });
  uint8_t* const own = c.smem + AttnSmem::OWN;           // Q, then dO
  bool ok = true;

  if (warp == AT_LOAD) ok = keys.rest<STAGES>(c);
  else if (warp == AT_MMA) {
    const bool issuer = elect_one();
    const uint64_t dk0 = make_smem_desc_k128(c.smem), dv0 = make_smem_desc_k128(c.smem + AT_TILE), dkn0 = make_smem_desc_mn128(c.smem);
    auto scores = [&](int j) {
      const int st = j % STAGES;
      if (!c.wait(&c.full[st], (j / STAGES) & 1)) return false;
      tc_fence_after();
      if (issuer) { mma_ts(c.tmem + T_S, c.tmem + T_Q, 16, desc_advance(dk0, st * AttnSmem::STAGE), 32, kIdescK, true); umma_commit_cta(c.s_full); }
      __syncwarp();
      return true;
    };
    auto grads = [&](int j) {
      if (issuer) { mma_ts(c.tmem + T_DP, c.tmem + T_DO, 16, desc_advance(dv0, (j % STAGES) * AttnSmem::STAGE), 32, kIdescK, true); umma_commit_cta(c.dp_full); }
      __syncwarp();
    };
    ok = c.wait(c.ready, 0);
    tc_fence_after();
    ok = ok && scores(0);
    if (ok) grads(0);
    for (int j = 0; ok && j < steps; j++) {
      if (j + 1 < steps && !(c.wait(c.p_full, j & 1) && scores(j + 1))) { ok = false; break; }      // the threads have S of step j in registers
      if (!c.wait(c.ds_full, j & 1)) { ok = false; break; }
      tc_fence_after();
      const int st = j % STAGES;
      if (issuer) {
        mma_ts(c.tmem + T_DQ, c.tmem + T_DP, 32, desc_advance(dkn0, st * AttnSmem::STAGE), 2048, kIdescMN, j == 0);
        umma_commit_cta(&c.empty[st]);
      }
      __syncwarp();
      if (j + 1 < steps) grads(j + 1);
    }
    if (ok && issuer) umma_commit_cta(c.acc_done);
    __syncwarp();
  } else {
    const int g = warp >> 2, r = (warp & 3) * 32 + lane, row = q0 + r;
    const uint32_t lanes = c.tmem + ((uint32_t)((warp & 3) * 32) << 16), ts = lanes + T_S + 32 * g, tdp = lanes + T_DP + 32 * g;
    const size_t pad = (size_t)bh * a.tiles * AT_ROWS + row;
    const float minus_lse = row < a.S ? a.lse_in[(size_t)bh * a.S + row] * -1.4426950408889634f : -INFINITY;
    const f32x2 n2 = both2(minus_lse);
    float* const rows = reinterpret_cast<float*>(c.smem + AttnSmem::ROWS);
    ok = c.wait(c.own, 0);
    {
      uint32_t x[32];
      if (g == 0) {
        load_row(own, r, x);
        tmem_st_32x32(lanes + T_Q, x);
      } else {
        uint32_t o[32];
        load_row(own + 2 * AT_TILE, r, x);
        load_row(c.smem + STAGES * AttnSmem::STAGE, r, o);
        tmem_st_32x32(lanes + T_DO, x);
        float d = 0.f;
#pragma unroll
        for (int i = 0; i < 32; i++) {
          const float2 u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[i])), v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o[i]));
          d = fmaf(u.x, v.x, d); d = fmaf(u.y, v.y, d);
        }
        rows[r] = -d;
        a.delta[pad] = -d; a.lse[pad] = minus_lse;
      }
      tmem_st_wait();
      if (ok) warp_arrive(c.ready, lane);
    }
    const f32x2 c2 = both2(kAttnLog2);
    ok = ok && c.wait(c.ready, 0);
    const f32x2 d2 = both2(rows[r]);
    for (int j = 0; ok && j < steps; j++) {
      if (!c.wait(c.s_full, j & 1)) { ok = false; break; }
      tc_fence_after();
      uint32_t x[32];
      tmem_ld_32x32(ts, x);
      tmem_ld_wait();
      warp_arrive(c.p_full, lane);
      float p[32];
#pragma unroll
      for (int i = 0; i < 32; i += 2) ex2_pair(fma2(pack2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])), c2, n2), p[i], p[i + 1]);
      const int last = row - j * AT_STEP - 32 * g;
      if (j * AT_STEP + AT_STEP - 1 > q0 + (warp & 3) * 32) {
#pragma unroll
        for (int i = 0; i < 32; i++) if (i > last) p[i] = 0.f;
      }
      if (!c.wait(c.dp_full, j & 1)) { ok = false; break; }
      tc_fence_after();
      tmem_ld_32x32(tdp, x);
      tmem_ld_wait();
      uint32_t y[16];
#pragma unroll
      for (int i = 0; i < 16; i++) {
        float u, v;
        unpack2(mul2(add2(pack2(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1])), d2), pack2(p[2 * i], p[2 * i + 1])), u, v);
        y[i] = pack_bf16(u, v);
      }
      tmem_st_32x16(tdp, y);
      tmem_st_wait();
      warp_arrive(c.ds_full, lane);
    }
    if (ok) ok = c.wait(c.acc_done, 0);
    if (ok && g == 0) {
      tc_fence_after();
      ok = store_gradient(c, a, lanes + T_DQ, kAttnScale, own + warp * 4096, h * AT_D, q0 + warp * 32, b, rows + 128, c.sums, a.part + ((size_t)b * a.tiles + tile) * 3 * C + h * AT_D, warp, lane);
    }
  }
  if (!ok) { *c.abort = 1; if (lane == 0) atomicExch(a.status, 20 + warp); }
  attn_end(c, warp, lane);
}

// ------------------------------------------------------------------ gradients of the keys and values
// TMEM columns: dK 0, dV 64, S^T 128 (P^T over it), dP^T 192 (dS^T over it).  A thread has a key and 32 of a step's queries: their lse and delta
// come with the step.  K and V stay in shared memory.
__global__ void __launch_bounds__(AT_THREADS, 2) attn_dkv_kernel(const __grid_constant__ AttnArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ int s_abort;
  __shared__ uint32_t s_tmem;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int heads = a.B * a.H, tile = blockIdx.x / heads, bh = blockIdx.x % heads, b = bh / a.H, h = bh % a.H, C = a.H * AT_D, k0 = tile * AT_ROWS;
  const int first = k0 / AT_STEP, steps = (a.S + AT_STEP - 1) / AT_STEP - first;
  constexpr uint32_t T_DK = 0, T_DV = 64, T_S = 128, T_DP = 192;
  const size_t at = (size_t)bh * a.tiles * AT_ROWS;
  const AttnSteps queries{&a.qkv, &a.dout, h * AT_D, h * AT_D, first, steps, b, a.lse + at, a.delta + at};
  AttnCtx c;
  attn_begin(c, smem_raw, &s_abort, &s_tmem, warp, 8, 1, [&](const AttnCtx& c) {
    uint8_t* const t = c.smem + AttnSmem::OWN;
    mbar_arrive_expect_tx(c.ready, 4 * AT_TILE);
    load_tile(t, &a.qkv, C + h * AT_D, k0, b, c.ready); load_tile(t + 2 * AT_TILE, &a.qkv, 2 * C + h * AT_D, k0, b, c.ready);
    queries.begin<AT_STAGES>(c);
  });
  uint8_t* const own = c.smem + AttnSmem::OWN;           // K, then V: 128 rows each
  bool ok = true;

  if (warp == AT_LOAD) ok = queries.rest<AT_STAGES>(c);
  else if (warp == AT_MMA) {
    const bool issuer = elect_one();
    const uint64_t k_own = make_smem_desc_k128(own), v_own = make_smem_desc_k128(own + 2 * AT_TILE);
    const uint64_t dq0 = make_smem_desc_k128(c.smem), do0 = make_smem_desc_k128(c.smem + AT_TILE), dqn0 = make_smem_desc_mn128(c.smem), don0 = make_smem_desc_mn128(c.smem + AT_TILE);
    auto product = [&](uint32_t d, uint64_t da, uint64_t db, uint64_t* bar) {
      if (issuer) { mma_ss(c.tmem + d, da, db, kIdescK); umma_commit_cta(bar); }
      __syncwarp();
    };
    auto stage = [&](int j) { const bool in = c.wait(&c.full[j % AT_STAGES], (j / AT_STAGES) & 1); tc_fence_after(); return in; };
    ok = c.wait(c.ready, 0) && stage(0);
    if (ok) { product(T_S, k_own, dq0, c.s_full); product(T_DP, v_own, do0, c.dp_full); }
    for (int j = 0; ok && j < steps; j++) {
      const uint32_t at = (j % AT_STAGES) * AttnSmem::STAGE, next = ((j + 1) % AT_STAGES) * AttnSmem::STAGE;
      if (!c.wait(c.p_full, j & 1)) { ok = false; break; }
      tc_fence_after();
      if (issuer) mma_ts(c.tmem + T_DV, c.tmem + T_S, 32, desc_advance(don0, at), 2048, kIdescMN, j == 0);
      __syncwarp();
      if (j + 1 < steps) {
        if (!stage(j + 1)) { ok = false; break; }
        product(T_S, k_own, desc_advance(dq0, next), c.s_full);
      }
      if (!c.wait(c.ds_full, j & 1)) { ok = false; break; }
      tc_fence_after();
      if (issuer) { mma_ts(c.tmem + T_DK, c.tmem + T_DP, 32, desc_advance(dqn0, at), 2048, kIdescMN, j == 0); umma_commit_cta(&c.empty[j % AT_STAGES]); }
      __syncwarp();
      if (j + 1 < steps) product(T_DP, v_own, desc_advance(do0, next), c.dp_full);
    }
    if (ok && issuer) umma_commit_cta(c.acc_done);
    __syncwarp();
  } else {
    const int g = warp >> 2, w = warp & 3, row = k0 + w * 32 + lane;
    const uint32_t lanes = c.tmem + ((uint32_t)(w * 32) << 16), ts = lanes + T_S + 32 * g, tdp = lanes + T_DP + 32 * g;
    const f32x2 c2 = both2(kAttnLog2);
    for (int j = 0; j < steps; j++) {
      const int st = j % AT_STAGES;
      const ulonglong2* const lse = reinterpret_cast<const ulonglong2*>(c.smem + AttnSmem::ROWS + st * 2 * AT_STEP * 4) + 8 * g;
      const ulonglong2* const delta = lse + AT_STEP / 4;
      if (!c.wait(&c.full[st], (j / AT_STAGES) & 1) || !c.wait(c.s_full, j & 1)) { ok = false; break; }
      tc_fence_after();
      uint32_t x[32], y[16];
      tmem_ld_32x32(ts, x);
      tmem_ld_wait();
      float p[32];
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const ulonglong2 u = lse[i / 4];
        ex2_pair(fma2(pack2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])), c2, u.x), p[i], p[i + 1]);
        ex2_pair(fma2(pack2(__uint_as_float(x[i + 2]), __uint_as_float(x[i + 3])), c2, u.y), p[i + 2], p[i + 3]);
      }
      const int hidden = row - (first + j) * AT_STEP - 32 * g;      // of these queries, those that do not see this key
      if (k0 + w * 32 + 31 > (first + j) * AT_STEP) {
#pragma unroll
        for (int i = 0; i < 32; i++) if (i < hidden) p[i] = 0.f;
      }
#pragma unroll
      for (int i = 0; i < 16; i++) y[i] = pack_bf16(p[2 * i], p[2 * i + 1]);
      tmem_st_32x16(ts, y);
      tmem_st_wait();
      warp_arrive(c.p_full, lane);
      if (!c.wait(c.dp_full, j & 1)) { ok = false; break; }
      tc_fence_after();
      tmem_ld_32x32(tdp, x);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const ulonglong2 u = delta[i / 4];
        float d, e;
        unpack2(mul2(add2(u.x, pack2(__uint_as_float(x[i]), __uint_as_float(x[i + 1]))), pack2(p[i], p[i + 1])), d, e);
        y[i / 2] = pack_bf16(d, e);
        unpack2(mul2(add2(u.y, pack2(__uint_as_float(x[i + 2]), __uint_as_float(x[i + 3]))), pack2(p[i + 2], p[i + 3])), d, e);
        y[i / 2 + 1] = pack_bf16(d, e);
      }
      tmem_st_32x16(tdp, y);
      tmem_st_wait();
      warp_arrive(c.ds_full, lane);
    }
    if (ok && c.wait(c.acc_done, 0)) {                   // K and V have been read for the last time; one group has dK, the other one dV
      tc_fence_after();
      ok = store_gradient(c, a, lanes + (g ? T_DV : T_DK), g ? 1.f : kAttnScale, own + g * 2 * AT_TILE + w * 4096, (1 + g) * C + h * AT_D, k0 + w * 32, b,
                          reinterpret_cast<float*>(c.smem + AttnSmem::ROWS) + 256 * g, c.sums + g, a.part + ((size_t)b * a.tiles + tile) * 3 * C + (1 + g) * C + h * AT_D, w, lane);
    } else ok = false;
  }
  if (!ok) { *c.abort = 1; if (lane == 0) atomicExch(a.status, 30 + warp); }
  attn_end(c, warp, lane);
}

// (nothing but attributes: the first call may lie inside a stream capture)
static int attn_ready(int dev) {
  static std::mutex mu;
  static bool ready[64] = {false};
  std::lock_guard<std::mutex> l(mu);
  if (ready[dev]) return 0;
  for (const void* f : {(const void*)attn_fwd_kernel, (const void*)attn_dq_kernel, (const void*)attn_dkv_kernel})
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnSmem::DYNAMIC) != cudaSuccess) return -4;
  ready[dev] = true;
  return 0;
}
static int attn_args(AttnArgs& a, const void* qkv, int B, int S, int H) {
  if (B <= 0 || S <= 0 || H <= 0 || S > (1 << 24) || H > (1 << 20) || (long long)B * H * ((S + AT_ROWS - 1) / AT_ROWS) > 0x7fffffffll) return -1;
  int dev = 0; cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -6;
  const int rc = attn_ready(dev); if (rc) return rc;
  memset(&a, 0, sizeof a);
  a.B = B; a.S = S; a.H = H; a.tiles = (S + AT_ROWS - 1) / AT_ROWS; a.status = status_word(STATUS_ATTENTION);
  if (!a.status) return -7;
  return make_tmap_bf16_rows(&a.qkv, qkv, B, S, 3ull * H * AT_D, AT_STEP) ? 0 : -3;
}

}  // namespace piccl_ops

using namespace piccl_ops;

extern "C" {

// Causal attention of packed rows qkv [B * S, 3 * H * 64] -> out [B * S, H * 64], all bf16, contiguous, 16-byte aligned.
// lse (null: not wanted): B * H * S floats, the logarithm of the sum of exponentials of each row's scaled scores.
int piccl_ops_attn_rows(int S) { return (S + AT_ROWS - 1) / AT_ROWS * AT_ROWS; }
int piccl_ops_attn_fwd(const void* qkv, void* out, float* lse, int B, int S, int H, void* stream) {
  if (!qkv || !out || ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out)) & 15) || (reinterpret_cast<uintptr_t>(lse) & 3)) return -2;
  AttnArgs a;
  const int rc = attn_args(a, qkv, B, S, H); if (rc) return rc;
  if (!make_tmap_bf16_rows(&a.result, out, B, S, (uint64_t)H * AT_D, 32)) return -3;
  a.out = a.dout = a.qkv; a.lse_out = lse;
  return launch_pdl(attn_fwd_kernel, B * H * a.tiles, AT_THREADS, AttnSmem::DYNAMIC, (cudaStream_t)stream, a) == cudaSuccess ? 0 : -5;
}
// lse: as above, from whichever kernel computed out.  dqkv: gradient of qkv; part: [piccl_ops_attn_parts(B, S)][3 * H * 64] floats, its partial column sums; scratch: 2 * B * H *
// piccl_ops_attn_rows(S) floats, 16-byte aligned.
int piccl_ops_attn_parts(int B, int S) { return B * ((S + AT_ROWS - 1) / AT_ROWS); }
int piccl_ops_attn_bwd(const void* qkv, const void* out, const void* dout, const float* lse, float* scratch, void* dqkv, float* part, int B, int S, int H, void* stream) {
  for (const void* p : {qkv, out, dout, (const void*)dqkv, (const void*)scratch}) if (!p || (reinterpret_cast<uintptr_t>(p) & 15)) return -2;
  for (const void* p : {(const void*)lse, (const void*)part}) if (!p || (reinterpret_cast<uintptr_t>(p) & 3)) return -2;
  AttnArgs a;
  const int rc = attn_args(a, qkv, B, S, H); if (rc) return rc;
  if (!make_tmap_bf16_rows(&a.out, out, B, S, (uint64_t)H * AT_D, AT_STEP) || !make_tmap_bf16_rows(&a.dout, dout, B, S, (uint64_t)H * AT_D, AT_STEP) ||
      !make_tmap_bf16_rows(&a.result, dqkv, B, S, 3ull * H * AT_D, 32)) return -3;
  a.lse_in = lse; a.lse = scratch; a.delta = scratch + (size_t)B * H * a.tiles * AT_ROWS; a.part = part;
  const int grid = B * H * a.tiles;
  if (launch_pdl(attn_dq_kernel, grid, AT_THREADS, AttnSmem::DYNAMIC, (cudaStream_t)stream, a) != cudaSuccess) return -5;
  return launch_pdl(attn_dkv_kernel, grid, AT_THREADS, AttnSmem::DYNAMIC, (cudaStream_t)stream, a) == cudaSuccess ? 0 : -5;
}
// Is this kernel (backward: both) at least as fast as cuDNN's, with the packing and the column sums that come with that one?  Measured alone at 1 to 64 batch entries times heads, time of
// this against that in percent; n: tiles of 128 rows, of which a chip of 148 SMs holds 296 at once.  One tile's walk grows with S: where all tiles are resident together the longest walk
// is the whole time and cuDNN's shorter step wins, where they take turns the early ends of the short walks are filled.  cuDNN has no tail to mask where S is a multiple of 128.
//   backward  S 512 -3 to -31, 640 +2 to -22, 777 -5 to -37, 1000 +2 to -34 | 896 n 7 +9, 224 +11, 308 -10, 448 -23; 1024 n 32 +11, 224 +19, 320 -8, 384 -18;
//             1536 n 240 +33, 336 +3, 384 -9; 2048 n 256 +46, 384 0, 448 -8; 3072 n 288 +60, 432 0, 480 -4; 4096 n 256 +73, 512 +1, 1024 -2; 8192 n 256 +94, 1024 +6
//   forward   S 33 +1 to -5, 128 -13 to -29, 512 -9 to -31, 1024 -1 to -28 | 1536 n 144 -19, 288 +7, 384 -1, 768 -7; 1600 -2 to -29;
//             2048 n 192 -13, 288 +9, 1024 -1; 4096 n 128 -18, 384 +11, 1024 +4; 8192 n 128 -17, 512 +15
int piccl_ops_attn_pays(int backward, int B, int S, int H, int sms) {
  const long long n = (long long)B * H * ((S + AT_ROWS - 1) / AT_ROWS), slots = 2ll * sms;
  const bool ragged = S % AT_ROWS != 0;
  if (backward) return S <= 640 || (ragged && S < 1024) || (S <= 3584 && n >= slots + S / 20);
  return S <= 1024 || 3 * n <= 4ll * sms || (S <= 1600 && (ragged || n > slots + 16));
}
// Non-zero if an attention kernel on the current device gave up on a wait (10 / 20 / 30 + warp).  Synchronises.
int piccl_ops_attn_status(void) { return read_status(STATUS_ATTENTION); }

}  // extern "C"

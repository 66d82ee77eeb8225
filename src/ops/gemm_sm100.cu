// bf16 GEMM for sm_100a with fused epilogues, on the CTA-pair core of sm100_gemm_pair.cuh.
//
//   layout 0  C[M,N] = A[M,K] B[N,K]^T      (forward products)
//   layout 1  C[M,N] = A[M,K] B[K,N]        (input gradients)
//   layout 2  C[M,N] = A[K,M]^T B[K,N]      (weight gradients)
//
//   epilogue 0  C = acc + bias
//   epilogue 1  pre = acc + bias (optional), C = gelu(pre as stored)
//   epilogue 2  C = acc + bias + aux                     (residual stream)
//   epilogue 3  C = acc * gelu'(aux), part = partial column sums of C: the input gradient of the GELU's product and the bias
//               gradient below it, without a pass over C
// M, N and K need not be multiples of the tile: what a load finds beyond the extents is zero, what a store would put there is dropped.
#include <cuda_bf16.h>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include "../include/sm100_gemm_pair.cuh"
#include "ops_common.cuh"

namespace piccl_ops {

using namespace sm100;

enum Epi : int { EPI_BIAS = 0, EPI_GELU = 1, EPI_RESIDUAL = 2, EPI_GELU_GRAD = 3 };

struct GemmArgs {
  CUtensorMap ta, tb, tc, tpre;
  const bf16* bias; const bf16* aux; float* part;
  float4* split; unsigned* ticket;                     // split K: fp32 partial accumulators, arrivals per tile and warp (all zero between launches)
  int M, N, K, has_pre, slices;
  int* status;
};

template <int TN, int EPI, bool SPLIT>
struct PlainPolicy {
  const GemmArgs& a;
  int num_m, num_n;                                    // tiles of 256 rows, of TN columns
  __device__ PlainPolicy(const GemmArgs& g) : a(g), num_m((g.M + 2 * PAIR_BM - 1) / (2 * PAIR_BM)), num_n((g.N + TN - 1) / TN) {}
  __device__ void begin() const { pdl_begin(); }
  __device__ void report(int role) const { atomicExch(a.status, role); }
  __device__ int num_tiles() const { return num_m * num_n * a.slices; }
  // Bands of 16 row tiles, inside a band column tiles outer / row tiles inner: the pairs that run together share a band of A
  // (about 30 MB at K = 3584) that stays in L2 while B streams through once per band.
  // With K split, the slices of one tile follow each other, so they run at the same time on different pairs.
  __device__ void tile(int idx, int v, int& m_blk, int& n_blk) const {
    constexpr int GM = 16;
    idx /= a.slices;
    const int per_band = GM * num_n, band = idx / per_band, within = idx % per_band;
    const int rows = min(GM, num_m - band * GM);
    m_blk = 2 * (band * GM + within % rows) + v; n_blk = within / rows;
  }
  __device__ void k_range(int idx, int num_kb, int& kb0, int& kb1) const {
    const int sl = idx % a.slices;
    kb0 = (int)((long long)num_kb * sl / a.slices); kb1 = (int)((long long)num_kb * (sl + 1) / a.slices);
  }
  __device__ const CUtensorMap* a_map(int m_blk, int& row0) const { row0 = m_blk * PAIR_BM; return &a.ta; }
  __device__ const CUtensorMap* b_map() const { return &a.tb; }
  __device__ bool gate(int, volatile int*) const { return true; }

  static constexpr int EXTRA_BYTES = 0, NSTAGE = 1;
  __device__ void finish(const EpiCtx&) {}
  static constexpr bool AUX = EPI == EPI_RESIDUAL || EPI == EPI_GELU_GRAD;
  static constexpr int PIECES = TN / 64;               // 64-column pieces of the tile; the halves of the warps share them
  static constexpr int PER = PIECES >= 2 ? PIECES / 2 : 1;
  uint4 x[8];                                          // the piece of aux that comes next, in flight
  // Four rows of 128 bytes per instruction (a thread that loads its own row touches 32 lines at a time, more than the L1 that 225 KB of
  // shared memory leave can keep: 74 us instead of 61 for 8192 x 4096 x 1024).
  __device__ void load_aux(const EpiCtx& e, int m_blk, int n_blk, int pc) {
    const int row0 = m_blk * PAIR_BM + e.quarter * 32 + (e.lane >> 3), col = n_blk * TN + pc * 64 + (e.lane & 7) * 8;
#pragma unroll
    for (int i = 0; i < 8; i++)
      x[i] = (row0 + 4 * i < a.M && col < a.N) ? *reinterpret_cast<const uint4*>(a.aux + (size_t)(row0 + 4 * i) * a.N + col) : make_uint4(0, 0, 0, 0);
  }
  __device__ int first_piece(const EpiCtx& e) const { return PIECES >= 2 ? e.half * PER : e.half; }
  __device__ void prefetch(const EpiCtx& e, int m_blk, int n_blk) {
    if (AUX && (PIECES >= 2 || e.half == 0)) load_aux(e, m_blk, n_blk, first_piece(e));
  }

  // Split K: every slice leaves its accumulator in fp32; the warp whose slice arrives last (nobody waits) adds the slices in their
  // order and goes on to the epilogue.  Pieces are kept as the threads hold them, so all accesses are coalesced.
  __device__ float4* split_at(int tile, int slice, int v8, int piece) const { return a.split + ((((size_t)tile * a.slices + slice) * 16 + v8) * PER + piece) * 512; }
  __device__ bool last_slice(const EpiCtx& e, int idx, int m_blk, int p0) {
    const int tile = idx / a.slices, v8 = (m_blk & 1) * 8 + e.half * 4 + e.quarter;
    for (int pc = p0; pc < p0 + PER; pc++) {
      float v[64];
      epi_load64(e, pc * 64, v);
      float4* dst = split_at(tile, idx % a.slices, v8, pc - p0) + e.lane;
#pragma unroll
      for (int j = 0; j < 16; j++) dst[j * 32] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
    __threadfence();
    __syncwarp();
    unsigned n = 0;
    if (e.lane == 0) {
      n = atomicAdd(a.ticket + tile * 16 + v8, 1u);
      if (n == (unsigned)a.slices - 1) a.ticket[tile * 16 + v8] = 0;
    }
    n = __shfl_sync(0xffffffffu, n, 0);
    __threadfence();
    return n == (unsigned)a.slices - 1;
  }
  __device__ void add_slices(const EpiCtx& e, int idx, int m_blk, int piece, float (&v)[64]) const {
    const int tile = idx / a.slices, v8 = (m_blk & 1) * 8 + e.half * 4 + e.quarter;
#pragma unroll
    for (int i = 0; i < 64; i++) v[i] = 0.f;
#pragma unroll 1
    for (int sl = 0; sl < a.slices; sl++) {
      const float4* src = split_at(tile, sl, v8, piece) + e.lane;
#pragma unroll
      for (int j = 0; j < 16; j++) { const float4 f = __ldcg(src + j * 32); v[4 * j] += f.x; v[4 * j + 1] += f.y; v[4 * j + 2] += f.z; v[4 * j + 3] += f.w; }
    }
  }

  __device__ bool epilogue(const EpiCtx& e, int idx, int m_blk, int n_blk, volatile int*) {
    const int row0 = m_blk * PAIR_BM + e.quarter * 32;
    if (row0 >= a.M || (PIECES < 2 && e.half)) return true;
    const int p0 = first_piece(e), p1 = p0 + PER;
    if (SPLIT && !last_slice(e, idx, m_blk, p0)) return true;
#pragma unroll 1
    for (int pc = p0; pc < p1; pc++) {
      const int col = n_blk * TN + pc * 64;
      if (col >= a.N) break;
      uint4 y[8];                                      // this thread's row of aux
      epi_staging_free(e);
      if (AUX) {
#pragma unroll
        for (int i = 0; i < 8; i++) { const int r = 4 * i + (e.lane >> 3); *reinterpret_cast<uint4*>(e.staging + r * 128 + (((e.lane & 7) ^ (r & 7)) << 4)) = x[i]; }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; j++) y[j] = *reinterpret_cast<const uint4*>(e.staging + e.lane * 128 + ((j ^ (e.lane & 7)) << 4));
        __syncwarp();
        if (pc + 1 < p1) load_aux(e, m_blk, n_blk, pc + 1);
      }
      float v[64];
      if (SPLIT) add_slices(e, idx, m_blk, pc - p0, v); else epi_load64(e, pc * 64, v);
      if (EPI != EPI_GELU_GRAD && a.bias) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
          if (col + 8 * j < a.N) {
            float b[8]; unpack8(*reinterpret_cast<const bf16x8*>(a.bias + col + 8 * j), b);
#pragma unroll
            for (int q = 0; q < 8; q++) v[8 * j + q] += b[q];
          }
        }
      }
      if (EPI == EPI_RESIDUAL) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
          float b[8]; unpack8(*reinterpret_cast<const bf16x8*>(&y[j]), b);
#pragma unroll
          for (int q = 0; q < 8; q++) v[8 * j + q] += b[q];
        }
      }
      if (EPI == EPI_GELU_GRAD) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
          float b[8]; unpack8(*reinterpret_cast<const bf16x8*>(&y[j]), b);
          mul_gelu_grad_n(v + 8 * j, b);
        }
      }
      if (EPI == EPI_GELU) {
        if (a.has_pre) { epi_stage_row(e, v); epi_ship(e, &a.tpre, col, row0); }
        if (a.has_pre) {                               // of the value as stored, which the backward pass sees
#pragma unroll
          for (int i = 0; i < 64; i++) v[i] = __bfloat162float(__float2bfloat16_rn(v[i]));
        }
        gelu_n(v);
        if (a.has_pre) epi_staging_free(e);
      }
      epi_stage_row(e, v);
      epi_ship(e, &a.tc, col, row0);
      if (EPI == EPI_GELU_GRAD && a.part) {            // two columns a lane, down the 32 rows of the staging buffer (rows beyond M hold zeros)
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int r = 0; r < 32; r++) {
          const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(e.staging + r * 128 + (((e.lane >> 2) ^ (r & 7)) << 4) + (e.lane & 3) * 4));
          s0 += f.x; s1 += f.y;
        }
        if (col + 2 * e.lane < a.N) *reinterpret_cast<float2*>(a.part + (size_t)(m_blk * 4 + e.quarter) * a.N + col + 2 * e.lane) = make_float2(s0, s1);
      }
    }
    return true;
  }
};

template <int TN, int STAGES, bool A_MN, bool B_MN, int EPI, bool SPLIT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1) gemm_pair_kernel(const __grid_constant__ GemmArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ int s_abort;
  if (threadIdx.x == 0) { s_abort = 0; tma_prefetch_desc(&a.ta); tma_prefetch_desc(&a.tb); tma_prefetch_desc(&a.tc); }
  PlainPolicy<TN, EPI, SPLIT> pol(a);
  gemm_pair_persistent<TN, STAGES, A_MN, B_MN>(smem_raw, pol, a.K, blockIdx.x >> 1, gridDim.x >> 1, &s_abort);
}

// ------------------------------------------------------------------ host
struct MapKey {
  const void* p; long rows, cols; int box;
  bool operator<(const MapKey& o) const { return std::tie(p, rows, cols, box) < std::tie(o.p, o.rows, o.cols, o.box); }
};
static std::mutex g_mu;
static std::map<MapKey, CUtensorMap> g_maps;
static int g_pairs[64] = {0};

// box rows x 64 columns of a row-major [rows, cols] matrix
static bool get_map(const void* p, long rows, long cols, int box, CUtensorMap* out) {
  std::lock_guard<std::mutex> l(g_mu);
  const MapKey k{p, rows, cols, box};
  auto it = g_maps.find(k);
  if (it != g_maps.end()) { *out = it->second; return true; }
  CUtensorMap m;
  if (!make_tmap_bf16_k64(&m, p, (uint64_t)rows, (uint64_t)cols, (uint64_t)cols, (uint32_t)box)) return false;
  if (g_maps.size() > 4096) g_maps.clear();
  g_maps[k] = m; *out = m;
  return true;
}

typedef void (*GemmFn)(GemmArgs);
struct Variant { int tn, layout, epi, split; GemmFn fn; int smem; bool ready[64]; };
#define V_(TN, ST, L, E, SP) {TN, L, E, SP, gemm_pair_kernel<TN, ST, L == 2, L != 0, E, SP != 0>, PairSmem<TN, ST>::DYNAMIC, {false}}
static Variant g_variants[] = {
  V_(256, 6, 0, EPI_BIAS, 0), V_(128, 8, 0, EPI_BIAS, 0), V_(64, 9, 0, EPI_BIAS, 0), V_(256, 6, 0, EPI_BIAS, 1), V_(128, 8, 0, EPI_BIAS, 1),
  V_(256, 6, 0, EPI_GELU, 0), V_(128, 8, 0, EPI_GELU, 0), V_(64, 9, 0, EPI_GELU, 0),
  V_(256, 6, 0, EPI_RESIDUAL, 0), V_(128, 8, 0, EPI_RESIDUAL, 0), V_(64, 9, 0, EPI_RESIDUAL, 0),
  V_(256, 6, 1, EPI_BIAS, 0), V_(128, 8, 1, EPI_BIAS, 0), V_(256, 6, 1, EPI_BIAS, 1), V_(128, 8, 1, EPI_BIAS, 1),
  V_(256, 6, 1, EPI_GELU_GRAD, 0), V_(128, 8, 1, EPI_GELU_GRAD, 0),
  V_(256, 6, 2, EPI_BIAS, 0), V_(128, 8, 2, EPI_BIAS, 0), V_(256, 6, 2, EPI_BIAS, 1), V_(128, 8, 2, EPI_BIAS, 1),
};
#undef V_

// Prepares the device state; pairs that can be resident at once (a pair needs two SMs of one GPC): the persistent grid is never larger.
static int device_ready(int dev) {
  std::lock_guard<std::mutex> l(g_mu);
  if (!g_pairs[dev]) {
    Variant& v = g_variants[0];
    if (cudaFuncSetAttribute((const void*)v.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem) != cudaSuccess) return -4;
    int sms = 148; cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sms / 2 * 2); cfg.blockDim = dim3(PAIR_THREADS); cfg.dynamicSmemBytes = v.smem;
    cudaLaunchAttribute at; memset(&at, 0, sizeof at);
    at.id = cudaLaunchAttributeClusterDimension; at.val.clusterDim.x = 2; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at; cfg.numAttrs = 1;
    int active = 0, n = sms / 2;
    if (cudaOccupancyMaxActiveClusters(&active, v.fn, &cfg) == cudaSuccess && active > 0) n = active < n ? active : n;
    else cudaGetLastError();
    g_pairs[dev] = n;
  }
  return 0;
}

// Tile width and slices of K: waves of the persistent grid times the clocks of a tile.  A k-step of 16 takes 136 / 84 / 70 clocks at
// 256 / 128 / 64 columns: the MMA alone needs TN / 2, and with all pairs busy narrow tiles ask more of the L2 than it gives (8192 x 4096 x
// 1024: 50 / 67 / 98 us; alone on the chip 68 and 51 clocks).  Over 48 shapes of 128 to 8192 rows the width taken is 1 % behind the best
// of the three on average, 11 % at worst (3 % and 24 % when the rule had the clocks of a chip that is otherwise idle).
// K is split where the tiles of a deep product leave pairs idle (weight gradients, few rows): a slice then writes its accumulator and
// the last one reads the others' (about 30 clocks a column and slice: 1024 x 1024 x 8192 gains, 23.1 -> 18.7 us, 3072 x 1024 x 8192 does not).  A slice keeps at least 8 k-blocks.
constexpr size_t kTicketBytes = 64 * 1024;
static size_t split_bytes(long tiles, int slices, int tn) { return kTicketBytes + (size_t)tiles * slices * 256 * tn * 4; }
static Variant* choose(int layout, int epi, int M, int N, int K, int pairs, size_t ws_bytes, int* slices) {
  Variant* best = nullptr; double best_cost = 0;
  const int kb = (K + PAIR_BK - 1) / PAIR_BK;
  for (auto& v : g_variants) {
    if (v.layout != layout || v.epi != epi) continue;
    const long tiles = (long)((M + 255) / 256) * ((N + v.tn - 1) / v.tn);
    const double step = v.tn == 256 ? 136 : v.tn == 128 ? 84 : 70;
    for (int s = v.split ? 2 : 1; s <= (v.split ? 16 : 1) && (s == 1 || kb / s >= 8); s++) {
      if (s > 1 && (split_bytes(tiles, s, v.tn) > ws_bytes || tiles * 64 > (long)kTicketBytes)) break;
      const double cost = (double)((tiles * s + pairs - 1) / pairs) * (step * 4 * ((kb + s - 1) / s) + 10.0 * v.tn) + (s > 1 ? 30.0 * v.tn * (s + 1) : 0);
      if (!best || cost < best_cost) { best = &v; best_cost = cost; *slices = s; }
    }
  }
  return best;
}

}  // namespace piccl_ops

extern "C" {

// Row-major, contiguous bf16 operands, 16-byte aligned, rows a multiple of 16 bytes.  bias [N], aux / pre [M, N] or null as the epilogue
// says; part: [ceil(M / 32)][N] floats or null; ws: workspace of ws_bytes for splitting K, its first 64 KiB zero (and left so), used by
// one stream at a time, or null.  Returns 0 on launch, a negative code if the shape is unsupported or set-up failed.
int piccl_ops_gemm(int layout, int epi, const void* A, const void* B, void* C, void* pre, const void* bias, const void* aux, float* part, void* ws, size_t ws_bytes, int M, int N, int K,
                   void* stream) {
  using namespace piccl_ops;
  if (layout < 0 || layout > 2 || M <= 0 || N <= 0 || K <= 0 || N % 8 || (layout != 2 && K % 8) || (layout == 2 && M % 8)) return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(pre) |
       reinterpret_cast<uintptr_t>(aux) | reinterpret_cast<uintptr_t>(part)) & 15) return -2;
  if ((epi == EPI_RESIDUAL || epi == EPI_GELU_GRAD) && !aux) return -2;
  int dev = 0; cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -6;
  int rc = device_ready(dev); if (rc) return rc;
  int slices = 1;
  Variant* v = choose(layout, epi, M, N, K, g_pairs[dev], ws ? ws_bytes : 0, &slices);
  if (!v) return -1;
  if (!v->ready[dev]) {
    if (cudaFuncSetAttribute((const void*)v->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, v->smem) != cudaSuccess) return -4;
    v->ready[dev] = true;
  }
  GemmArgs a;
  const bool a_ok = layout == 2 ? get_map(A, K, M, 64, &a.ta) : get_map(A, M, K, PAIR_BM, &a.ta);
  const bool b_ok = layout == 0 ? get_map(B, N, K, v->tn / 2, &a.tb) : get_map(B, K, N, 64, &a.tb);
  if (!a_ok || !b_ok || !get_map(C, M, N, 32, &a.tc)) return -3;
  a.has_pre = pre != nullptr;
  if (pre) { if (!get_map(pre, M, N, 32, &a.tpre)) return -3; } else a.tpre = a.tc;
  a.bias = (const bf16*)bias; a.aux = (const bf16*)aux; a.part = part;
  a.slices = slices; a.ticket = (unsigned*)ws; a.split = (float4*)((char*)ws + kTicketBytes);
  a.M = M; a.N = N; a.K = K; a.status = status_word(STATUS_GEMM);
  if (!a.status) return -7;
  const long tiles = (long)((M + 255) / 256) * ((N + v->tn - 1) / v->tn) * slices;
  const int pairs = (int)(tiles < g_pairs[dev] ? tiles : g_pairs[dev]);
  return launch_pdl(v->fn, dim3(2 * pairs), dim3(PAIR_THREADS), v->smem, (cudaStream_t)stream, a) == cudaSuccess ? 0 : -5;
}

// C = act(A · B^T + bias).  A [M,K], B [N,K], C [M,N], all bf16 row-major and contiguous; bias [N] bf16 or null;
// c_pre (optional) receives the value before the activation.  Requires M % 128 == 0, N % 128 == 0, K % 64 == 0.
// Returns 0 on launch, a negative code if the shape is unsupported or set-up failed.
int piccl_ops_gemm_bf16_nt_ex(const void* A, const void* B, void* C, void* c_pre, const void* bias, int M, int N, int K, int gelu, void* stream) {
  using namespace piccl_ops;
  if (M <= 0 || N <= 0 || K <= 0 || M % 128 || N % 128 || K % 64) return -1;
  return piccl_ops_gemm(0, gelu ? EPI_GELU : EPI_BIAS, A, B, C, c_pre, bias, nullptr, nullptr, nullptr, 0, M, N, K, stream);
}
int piccl_ops_gemm_bf16_nt(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int gelu, void* stream) {
  return piccl_ops_gemm_bf16_nt_ex(A, B, C, nullptr, bias, M, N, K, gelu, stream);
}
// Non-zero if a GEMM on the current device gave up on a wait (1 producer, 2/3 MMA issuer, 4 epilogue).  Synchronises.
int piccl_ops_gemm_status(void) { return piccl_ops::read_status(piccl_ops::STATUS_GEMM); }

}  // extern "C"

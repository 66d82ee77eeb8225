// Persistent tcgen05 GEMM core on CTA PAIRS (two SMs of one cluster, `cta_group::2`), shared by the plain GEMM
// (src/ops/gemm_sm100.cu) and the fused tensor-parallel kernels (src/tp).  bf16 operands, fp32 accumulation in TMEM.
//
// A pair works on a tile of 2 x 128 rows and TN columns.  CTA v (0 = leader, 1 = follower) stages its own 128 rows of A and half
// of the tile's columns of B; the tensor cores of both SMs read both halves of B.  Per SM and k-block that is 32 KiB of operands
// at TN = 256 where a lone CTA with the same accumulator needs 48 KiB: the ring is 6 k-blocks deep instead of 4 and a third less
// comes out of L2.  (8192 x 8192 x 3584: 401 us with the one-CTA core, whose tensor pipe waited for operands.)
// The two row blocks of a tile are independent (a policy may pair any two), only the columns are common.
//
// Operand layouts: K-major (rows of 64 k, one 128-byte swizzled row each) or MN-major (the operand lies transposed: 64 k-rows of
// 64 elements each per box), so C = A B^T, C = A B and C = A^T B need no transposed copy.
//
// Roles inside a CTA of 320 threads (352 with a policy's extra warp):
//   warp 0     TMA producer; the bytes of both CTAs are counted on the LEADER's `full` barrier
//   warp 1     TMEM allocation; in the leader one lane issues the MMAs and commits to the barriers of both CTAs
//   warps 2-9  epilogue: warp w reads TMEM lanes of quarter w & 3, columns of half (w - 2) / 4, through 64-column pieces.
//              Eight warps, because an epilogue of a few dozen instructions per element has to fit under the main loop of the
//              next tile (4096 clocks at K = 1024).
//   warp 10    Policy::extra_warp, where the policy has one (EXTRA_BYTES > 0: shared memory it gets)
//
//   struct Policy {
//     void begin() const;                                           // every thread, after the set-up (barriers, TMEM) and before global memory is touched
//     void report(int role) const;                                  // status word: a wait of that role ran out
//     int  num_tiles() const;
//     void tile(int idx, int v, int& m_blk, int& n_blk);           // 128-row block of CTA v (< 0: none), block of TN columns; the calls below are about it
//     void k_range(int idx, int num_kb, int& kb0, int& kb1) const; // k-blocks that this entry of the tile order sums, not empty
//     const CUtensorMap* a_map(int m_blk, int& row0) const;        // tensor map and first row of A for it
//     const CUtensorMap* b_map() const;                            // tensor map of B
//     static constexpr bool K_RANKS = true; int kb_per_rank; const CUtensorMap* a_of(int p) const, *b_of(int p) const;      // optional: k-blocks [p, p + 1) * kb_per_rank come from
//                                                                   // these maps, each from its column 0 (a_map still gives the row)
//     bool gate(int m_blk, volatile int* abort) const;             // producer: wait until the row block may be loaded
//     void prefetch(const EpiCtx&, int m_blk, int n_blk);          // epilogue warps, before they wait for the accumulator
//     bool epilogue(const EpiCtx&, int idx, int m_blk, int n_blk, volatile int* abort);  // called by all eight warps; false: gave up
//     void finish(const EpiCtx&);                                   // epilogue warps, after their last tile
//     static constexpr int NSTAGE;                                  // staging buffers per epilogue warp
//     static constexpr int EXTRA_BYTES; void extra_warp(uint8_t* smem, int lane, volatile int* abort);           // all lanes of warp 10
//   };
// Every wait is bounded; a wait that runs out sets the status word (1 producer, 2 / 3 MMA issuer, 4 epilogue, 5 gate, 6 policy), every
// role leaves its loop, copies in flight get time to land, TMEM is released.
#pragma once
#include <cuda_bf16.h>
#include "sm100_ptx.cuh"

namespace sm100 {

constexpr int PAIR_BM = 128, PAIR_BK = 64, PAIR_THREADS = 320, PAIR_EPI_WARPS = 8;
constexpr int PAIR_STAGING = 4096;                                  // bytes of a staging buffer of an epilogue warp: 32 rows of 64 bf16
constexpr unsigned long long kPairWaitLimitNs = 4000000000ull;      // 4 s
constexpr uint32_t kLeaderMask = 0xFEFFFFFFu;      // clears the bit that tells the two CTAs of a pair apart in a shared::cluster address

// NSTAGE: staging buffers per epilogue warp
template <int TN, int STAGES, int EXTRA_BYTES = 0, int NSTAGE = 1>
struct PairSmem {
  static constexpr int A_BYTES = PAIR_BM * PAIR_BK * 2, B_BYTES = (TN / 2) * PAIR_BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGING_OFF = STAGES * STAGE_BYTES;
  static constexpr int BAR_OFF = STAGING_OFF + PAIR_EPI_WARPS * PAIR_STAGING * NSTAGE;
  static constexpr int EXTRA_OFF = (BAR_OFF + (2 * STAGES + 4) * 8 + 16 + 127) / 128 * 128;
  static constexpr int TOTAL = EXTRA_OFF + EXTRA_BYTES;
  static constexpr int DYNAMIC = TOTAL + 1024;                      // slack for the 1024-byte alignment of the tiles
  static_assert(DYNAMIC <= 232448, "more shared memory than a CTA can have");
};

__device__ __forceinline__ uint32_t cluster_ctarank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Tile load of a CTA pair: the bytes are counted on the mbarrier at the same offset in the LEADER's shared memory.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar) & kLeaderMask), "r"(x), "r"(y) : "memory");
}
// 2-D tile shared -> global; what lies beyond the tensor's extents is not written
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(smem_src)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {      // whole warp, in both CTAs, same warp index, same address
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D[tmem of both CTAs] (+)= A[both CTAs' smem] * B[both CTAs' smem]; issued by one thread of the leader
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
               ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// The mbarrier at this offset in BOTH CTAs gets one arrival once all MMAs issued so far have completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  const uint16_t both = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(both) : "memory");
}
// One arrival on the mbarrier at this offset in the LEADER's shared memory (from either CTA).
__device__ __forceinline__ void mbar_arrive_leader(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(smem_u32(bar) & kLeaderMask) : "memory");
}
// Operand lying MN-major: boxes of 64 k-rows x 64 elements (128 bytes, 128-byte swizzle).  Groups of 8 k-rows are 1024 bytes apart
// (stride offset), the next 64 elements along MN one box, 8192 bytes, further (leading offset).
__device__ __forceinline__ uint64_t make_smem_desc_mn128(const void* smem_tile) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_u32(smem_tile) & 0x3FFFFu) >> 4);
  d |= (uint64_t)(8192u >> 4) << 16;
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__host__ __device__ constexpr uint32_t make_idesc_bf16_major(uint32_t M, uint32_t N, bool a_mn, bool b_mn) {
  return make_idesc_bf16(M, N) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16);
}

// What an epilogue warp knows about itself and its accumulator.
struct EpiCtx {
  uint32_t tmem;         // this warp's lanes, first column of the accumulator
  uint8_t* staging;      // this warp's staging buffers
  int quarter, half, lane;
};
// 64 columns of this thread's row, starting at column col0 of the tile
__device__ __forceinline__ void epi_load64(const EpiCtx& e, int col0, float (&v)[64]) {
  uint32_t r0[32], r1[32];
  tmem_ld_32x32(e.tmem + col0, r0);
  tmem_ld_32x32(e.tmem + col0 + 32, r1);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; i++) { v[i] = __uint_as_float(r0[i]); v[32 + i] = __uint_as_float(r1[i]); }
}

// 64 bf16 of this thread's row -> the warp's staging buffer: 16-byte pieces XOR-ed with the row, conflict free and the layout that a
// store through a 128-byte swizzled map of 32 x 64 boxes expects
__device__ __forceinline__ void epi_stage_row(const EpiCtx& e, const float (&v)[64]) {
#pragma unroll
  for (int j = 0; j < 8; j++) {
    uint4 o; __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int q = 0; q < 4; q++) o2[q] = __floats2bfloat162_rn(v[8 * j + 2 * q], v[8 * j + 2 * q + 1]);
    *reinterpret_cast<uint4*>(e.staging + e.lane * 128 + ((j ^ (e.lane & 7)) << 4)) = o;
  }
  fence_proxy_async();                                 // these stores must be visible to the bulk-copy engine
  __syncwarp();
}
__device__ __forceinline__ void epi_ship(const EpiCtx& e, const CUtensorMap* map, int x, int y) {
  if (e.lane == 0) { tma_store_2d(map, e.staging, x, y); bulk_commit(); }
}
__device__ __forceinline__ void epi_staging_free(const EpiCtx& e) {
  if (e.lane == 0) bulk_wait_read_all();               // the last store has been read out of the staging buffer
  __syncwarp();
}

template <class P, class = void> struct k_over_ranks { static constexpr bool value = false; };
template <class P> struct k_over_ranks<P, decltype((void)P::K_RANKS)> { static constexpr bool value = P::K_RANKS; };

template <int TN, int STAGES, bool A_MN, bool B_MN, class Policy>
__device__ __forceinline__ void gemm_pair_persistent(uint8_t* smem_raw, Policy& pol, int K, int first_tile, int tile_stride, volatile int* s_abort) {
  typedef PairSmem<TN, STAGES, Policy::EXTRA_BYTES, Policy::NSTAGE> L;
  static_assert(!B_MN || TN >= 128, "an MN-major half of B is at least one box of 64 columns");
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* empty = full + STAGES;
  uint64_t* tmem_full = empty + STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  // The producer and the MMA warp run their loops with all lanes (only the issue itself is one lane's), from a warp index that the
  // compiler can see is uniform: barrier addresses and descriptors then live in uniform registers.  As one lane's divergent
  // loop a k-block took at least 545 clocks whatever the tile.
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int v = (int)cluster_ctarank();
  const int num_tiles = pol.num_tiles(), num_kb = (K + PAIR_BK - 1) / PAIR_BK;
  constexpr uint32_t TMEM_COLS = 2 * TN;                    // two accumulators; a power of two from 128 to 512

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; a++) { mbar_init(&tmem_full[a], 1); mbar_init(&tmem_empty[a], 2 * PAIR_EPI_WARPS); }
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc_pair(tmem_slot, TMEM_COLS); tmem_relinquish_pair(); }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                       // the partner's barriers exist before anything is signalled across
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pol.begin();                                              // nothing of global memory has been touched so far

  if (warp == 0) {
    const bool issuer = elect_one();
    int stage = 0; uint32_t phase = 0;
    for (int t = first_tile; t < num_tiles && !*s_abort; t += tile_stride) {
      int m_blk, n_blk; pol.tile(t, v, m_blk, n_blk);
      if (!pol.gate(m_blk, s_abort)) { *s_abort = 1; if (issuer) pol.report(5); break; }
      int row0; const CUtensorMap* ta = pol.a_map(m_blk, row0);
      const CUtensorMap* tb = pol.b_map();
      const int col0 = n_blk * TN + v * (TN / 2);
      int kb0, kb1; pol.k_range(t, num_kb, kb0, kb1);
      bool ok = true;
      for (int kb = kb0; kb < kb1; kb++) {
        if (!mbar_wait(&empty[stage], phase ^ 1, s_abort, kPairWaitLimitNs)) { if (issuer) pol.report(1); ok = false; break; }
        uint8_t* sa = smem + stage * L::STAGE_BYTES; uint8_t* sb = sa + L::A_BYTES;
        int k0 = kb * PAIR_BK;
        if constexpr (k_over_ranks<Policy>::value) { const int p = kb / pol.kb_per_rank; ta = pol.a_of(p); tb = pol.b_of(p); k0 = (kb - p * pol.kb_per_rank) * PAIR_BK; }
        if (issuer) {
          if (v == 0) mbar_arrive_expect_tx(&full[stage], 2 * L::STAGE_BYTES);      // the bytes of both CTAs land on the leader's barrier
          if (A_MN) {
#pragma unroll
            for (int i = 0; i < PAIR_BM / 64; i++) tma_load_2d_pair(sa + i * 8192, ta, row0 + i * 64, k0, &full[stage]);
          } else tma_load_2d_pair(sa, ta, k0, row0, &full[stage]);
          if (B_MN) {
#pragma unroll
            for (int i = 0; i < TN / 128; i++) tma_load_2d_pair(sb + i * 8192, tb, col0 + i * 64, k0, &full[stage]);
          } else tma_load_2d_pair(sb, tb, k0, col0, &full[stage]);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
    }
  } else if (warp == 1) {
    if (v == 0) {
      const bool issuer = elect_one();
      constexpr uint32_t idesc = make_idesc_bf16_major(2 * PAIR_BM, TN, A_MN, B_MN);
      const uint64_t da0 = A_MN ? make_smem_desc_mn128(smem) : make_smem_desc_k128(smem);
      const uint64_t db0 = B_MN ? make_smem_desc_mn128(smem + L::A_BYTES) : make_smem_desc_k128(smem + L::A_BYTES);
      int stage = 0; uint32_t phase = 0; int local = 0;
      for (int t = first_tile; t < num_tiles && !*s_abort; t += tile_stride, local++) {
        const int acc = local & 1; const uint32_t acc_phase = (local >> 1) & 1;
        if (!mbar_wait(&tmem_empty[acc], acc_phase ^ 1, s_abort, kPairWaitLimitNs)) { if (issuer) pol.report(2); break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * TN;
        int kb0, kb1; pol.k_range(t, num_kb, kb0, kb1);
        bool ok = true;
        for (int kb = kb0; kb < kb1; kb++) {
          if (!mbar_wait(&full[stage], phase, s_abort, kPairWaitLimitNs)) { if (issuer) pol.report(3); ok = false; break; }
          tc_fence_after();
          const uint64_t da = desc_advance(da0, stage * L::STAGE_BYTES), db = desc_advance(db0, stage * L::STAGE_BYTES);
          if (issuer) {
            // 16 k are 32 bytes of a K-major row, or 16 rows of 128 bytes of an MN-major box
#pragma unroll
            for (int k = 0; k < PAIR_BK / 16; k++)
              umma_f16_pair(d_tmem, desc_advance(da, k * (A_MN ? 2048 : 32)), desc_advance(db, k * (B_MN ? 2048 : 32)), idesc, kb != kb0 || k != 0);
            umma_commit_pair(&empty[stage]);
          }
          __syncwarp();
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (issuer) umma_commit_pair(&tmem_full[acc]);
        __syncwarp();
      }
    }
  } else if (Policy::EXTRA_BYTES > 0 && warp >= 2 + PAIR_EPI_WARPS) {
    if constexpr (Policy::EXTRA_BYTES > 0) pol.extra_warp(smem + L::EXTRA_OFF, lane, s_abort);
  } else {
    EpiCtx e;
    e.quarter = warp & 3; e.half = (warp - 2) >> 2; e.lane = lane;
    e.staging = smem + L::STAGING_OFF + (warp - 2) * PAIR_STAGING * Policy::NSTAGE;
    int local = 0;
    for (int t = first_tile; t < num_tiles; t += tile_stride, local++) {
      int m_blk, n_blk; pol.tile(t, v, m_blk, n_blk);
      const int acc = local & 1; const uint32_t acc_phase = (local >> 1) & 1;
      e.tmem = tmem_base + ((uint32_t)(e.quarter * 32) << 16) + acc * TN;
      pol.prefetch(e, m_blk, n_blk);
      if (!mbar_wait(&tmem_full[acc], acc_phase, s_abort, kPairWaitLimitNs)) { pol.report(4); break; }
      tc_fence_after();
      if (!pol.epilogue(e, t, m_blk, n_blk, s_abort)) { *s_abort = 1; pol.report(6); break; }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_leader(&tmem_empty[acc]);      // this warp's part of the accumulator may be overwritten
    }
    pol.finish(e);
  }
  // Neither CTA leaves while the other may still touch its shared memory or barriers, TMEM is freed after the last read of it.  The
  // arrival goes out before the wait for the stores' reads of the staging buffers, so the two latencies overlap.
  tc_fence_before();
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  if (warp >= 2 && lane == 0) bulk_wait_read_all();            // (the extra warp has waited for its own copies)
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (*s_abort) {
    unsigned long long t0 = gtime_ns();
    while (gtime_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) { tc_fence_after(); tmem_dealloc_pair(tmem_base, TMEM_COLS); }
}

}  // namespace sm100

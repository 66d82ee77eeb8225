// Fused tensor-parallel kernels: one launch does the tcgen05 GEMM AND the
// collective that follows or precedes it, tile by tile, over peer memory.
// Both run on the CTA-pair core of sm100_gemm_pair.cuh.
//
//  gemm_rs   C = A_r · B_r^T per rank, summed over ranks, row block r kept by rank r.
//            Row blocks owned by OTHER ranks come first: an epilogue warp ships each piece of 32 rows x 64
//            columns as bf16 with one 4 KiB bulk store into the owner's heap, the last of the tile's eight
//            warps raises a per-(source, tile) epoch flag.  The rank's OWN blocks come last: their epilogue
//            waits (bounded) for the n-1 partials of that tile, adds them in rank order to the accumulator it
//            just read from TMEM, and writes the final result.
//            No partial of an own tile ever goes to memory; transfer overlaps the remaining MMA work.
//  ag_gemm   A is row-sharded over ranks; C = concat(A_r) · B^T.  One more warp in EVERY CTA pushes parts of
//            this rank's shard into every peer's gathered buffer (the peer that needs them next first) with
//            bulk copies through a small ring in shared memory, and raises per-part flags; it takes neither an SM nor
//            issue slots from the products.  (24 CTAs set aside for it cost a sixth of the SMs for the whole call:
//            two ranks of 4096 x 2048 x 4096 166 us.)  The GEMM starts on the local shard and gates the TMA
//            loads of a remote row block on its flags.  TMA only ever reads LOCAL memory (the local
//            shard or the local gathered buffer), never a peer's.
//
// Buffers are double buffered by call parity, flags carry the call epoch, so nothing is reset
// between calls.  All waits are bounded; a wait that gives up is reported through
// piccl_tp_status().  The reference has no GEMM at all; the comparison is cuBLAS + NCCL.
#include <cuda_bf16.h>
#include <algorithm>
#include <cstring>
#include "../include/sm100_gemm_pair.cuh"
#include "../runtime/comm.h"

namespace piccl {

using namespace sm100;
typedef __nv_bfloat16 bf16;
constexpr int TP_BN = 256, RS_STAGES = 5, AG_STAGES = 5, TP_MAX_RANKS = 8;
constexpr int TP_BM = PAIR_BM, TP_BK = PAIR_BK;

// Flags, for ranks on several GPUs or (one_gpu) all of them in one launch.
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p, bool one_gpu) {
  unsigned v;
  if (one_gpu) asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  else asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v, bool one_gpu) {
  if (one_gpu) asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
  else asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Bounded wait until *flag == epoch.
__device__ __forceinline__ bool wait_flag(const unsigned* flag, unsigned epoch, bool one_gpu, volatile int* abort_flag) {
  unsigned long long t0 = 0;
  for (unsigned it = 1;; it++) {
    if (ld_acquire_u32(flag, one_gpu) == epoch) return true;
    if ((it & 63u) == 0) {
      if (*abort_flag) return false;
      unsigned long long now = gtime_ns();
      if (!t0) t0 = now; else if (now - t0 > kPairWaitLimitNs) return false;
    }
  }
}

// The flag area of a rank's heap: half of it for each kernel, half of that for each parity of the kernel's call count, whatever the shape.  A
// rank that is one call ahead, with another shape, then never writes a flag that a peer still waits for: waits look for
// equality, so a flag of the next call in its place would be waited out.
constexpr long long TP_FLAG_KERNEL = 512 << 10, TP_FLAG_CALL = TP_FLAG_KERNEL / 2;
// bytes from the start of a kernel's half: flag t of the `per_src` that source rank src raises
__host__ __device__ inline long long tp_flag_at(int parity, int src, long long per_src, long long t) { return parity * TP_FLAG_CALL + (src * per_src + t) * 4; }

struct TpRank {
  CUtensorMap ta;            // gemm_rs: A [M, K_local];   ag_gemm: local shard [M/n, K]
  CUtensorMap ta2;           // ag_gemm: gathered buffer [2*M, K] in this rank's heap
  CUtensorMap tb;
  CUtensorMap tc;            // this rank's output, boxes of 32 rows x 64 columns
  char* heap[TP_MAX_RANKS];  // all ranks' heaps as mapped here
  const bf16* a_shard;       // ag_gemm: the local shard (feeder source)
  bf16* out;
  int* status;
  int rank;
};
struct TpArgs {
  int n, M, N, K;            // gemm_rs: K = K_local, N full;  ag_gemm: N = N_local, K full
  int nv;                    // (virtual) ranks of this launch: every pair works for all of them, see the policies
  int n_part;                // ag_gemm: parts of a row block, each with a flag of its own
  unsigned epoch;
  int one_gpu;               // all ranks in this launch: flags need no scope beyond the GPU
  long long flag_off, data_off;
  TpRank r[TP_MAX_RANKS];    // one entry per virtual rank of the launch
};

// ------------------------------------------------------------------ GEMM -> reduce-scatter
// Several virtual ranks on one device: every pair of CTAs works for each of them in turn, so that at any time one rank's operands are in
// L2.  (With a ninth of the pairs for each of eight ranks, eight working sets of 12 MB per wave thrashed it: 3.4 GB read from memory for
// 0.6 GB of operands, and the power that took held the clocks down: 4.2 ms for 8192 x 8192 x 3584 in a steady loop.)
struct RsPolicy {
  const TpArgs& a; const TpRank* R = nullptr; unsigned* s_arrived;
  int n, rank = 0, mb_per_owner, num_n, parity, tiles_per_owner, rp_remote, rp_own;
  unsigned* pending = nullptr;       // flag of the remote tile whose stores this warp has issued but not waited for, and the tile's slot in s_arrived
  int pending_slot = 0, seq = 0;
  static constexpr int EXTRA_BYTES = 0, NSTAGE = 2;
  __device__ RsPolicy(const TpArgs& args, unsigned* arrived)
      : a(args), s_arrived(arrived), n(args.n), mb_per_owner(args.M / args.n / TP_BM), num_n(args.N / TP_BN), parity((int)(args.epoch & 1)), tiles_per_owner(mb_per_owner * num_n),
        rp_remote(((args.n - 1) * mb_per_owner + 1) / 2), rp_own((mb_per_owner + 1) / 2) {}
  __device__ void begin() const {}
  __device__ void report(int role) const { for (int i = 0; i < a.nv; i++) atomicExch(a.r[i].status, role); }
  __device__ int num_tiles() const { return a.nv * (rp_remote + rp_own) * num_n; }
  // Panels of 16 column blocks (one panel of B stays in L2); inside a panel first the row blocks of other owners, in the order rank+1,
  // rank+2, ..., for every rank of the launch, then the own ones; two blocks to a pair, bands of 16 pairs, inside a band rows fastest.
  // All ranks walk the panels in the same order, so the partials of my own tiles of a panel are on their way while I still compute
  // the other owners' tiles of that panel; and as a panel's own tiles come after all its remote ones, waits never form a cycle.
  __device__ void tile(int idx, int v, int& m_blk, int& n_blk) {
    constexpr int PN = 16, BAND = 16;
    const int per_panel = PN * a.nv * (rp_remote + rp_own), panel = idx / per_panel, cols = min(PN, num_n - panel * PN);      // the last panel may be narrower
    int w = idx % per_panel;
    const int remote = a.nv * rp_remote * cols;
    const bool own = w >= remote;
    if (own) w -= remote;
    const int rp = own ? rp_own : rp_remote, vr = w / (rp * cols);
    w %= rp * cols;
    R = &a.r[vr]; rank = R->rank;
    const int band = w / (BAND * cols), rows = min(BAND, rp - band * BAND);
    w %= BAND * cols;
    const int i = 2 * (band * BAND + w % rows) + v;
    n_blk = panel * PN + w / rows;
    if (own) m_blk = i < mb_per_owner ? rank * mb_per_owner + i : -1;
    else m_blk = i < (n - 1) * mb_per_owner ? (rank + 1 + i / mb_per_owner) % n * mb_per_owner + i % mb_per_owner : -1;
  }
  __device__ void k_range(int, int num_kb, int& kb0, int& kb1) const { kb0 = 0; kb1 = num_kb; }
  __device__ const CUtensorMap* a_map(int m_blk, int& row0) const { row0 = max(m_blk, 0) * TP_BM; return &R->ta; }
  __device__ const CUtensorMap* b_map() const { return &R->tb; }
  __device__ bool gate(int, volatile int*) const { return true; }
  __device__ int tile_id(int m_blk, int n_blk) const { return (m_blk % mb_per_owner) + n_blk * mb_per_owner; }
  __device__ unsigned* flag_ptr(int owner, int src, int t) const {
    return reinterpret_cast<unsigned*>(R->heap[owner] + a.flag_off + tp_flag_at(parity, src, tiles_per_owner, t));
  }
  // A tile travels as pieces of 32 rows x 64 columns: 4 KiB each, the 16-byte words of a row 512 bytes apart, so that both the
  // staging stores of the writer and the loads of the reader take consecutive words.  data_off: this call's half of the region.
  __device__ char* piece(int owner, int src, int t, const EpiCtx& e, int pc) const {
    return R->heap[owner] + a.data_off + ((size_t)src * tiles_per_owner + t) * (size_t)(TP_BM * TP_BN * 2) + (e.quarter * 4 + pc) * PAIR_STAGING;
  }
  __device__ void prefetch(const EpiCtx&, int, int) {}
  // Lane 0: this warp's stores for the pending tile have been performed (at most KEEP newer groups may be in flight); the last of the eight warps
  // of the tile tells the owner.
  template <int KEEP> __device__ void announce() {
    if (!pending) return;
    asm volatile("cp.async.bulk.wait_group %0;" ::"n"(KEEP) : "memory");
    asm volatile("fence.proxy.async;" ::: "memory");
    unsigned before;
    asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;" : "=r"(before) : "r"(smem_u32(&s_arrived[pending_slot])) : "memory");
    if (before == PAIR_EPI_WARPS - 1) {
      s_arrived[pending_slot] = 0;                       // used again four tiles on, when every warp has left this one
      st_release_u32(pending, a.epoch, a.one_gpu);
    }
    pending = nullptr;
  }
  __device__ void finish(const EpiCtx& e) { if (e.lane == 0) announce<0>(); }
  // Buffer p of the warp, free to be written: every tile with a result, own or remote, sends its first piece from buffer 0 and its second
  // from buffer 1, one group each, so the last store out of buffer p is two groups old whatever kind of tile came before.
  __device__ EpiCtx staging_turn(EpiCtx e, int p) const {
    if (e.lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
    __syncwarp();
    e.staging += p * PAIR_STAGING;
    return e;
  }
  __device__ bool epilogue(const EpiCtx& e, int, int m_blk, int n_blk, volatile int* abort_flag) {
    const int slot = seq++ & 3;
    const int owner = m_blk < 0 ? -1 : m_blk / mb_per_owner, t = m_blk < 0 ? 0 : tile_id(m_blk, n_blk);
    if (m_blk < 0 || owner == rank) {                    // nothing is held back where this warp may wait, or has nothing to store
      if (e.lane == 0) announce<0>();
      __syncwarp();
      if (m_blk < 0) return true;
    }
    if (owner != rank) {
      // The two pieces of this warp go out from a staging buffer each; the flag of a tile is raised in the epilogue of the next one, when its
      // stores have long been performed (waiting for them here made short K wait: 8192 x 8192 x 1024 among eight ranks 1.6 ms).
#pragma unroll
      for (int p = 0; p < 2; p++) {
        const int pc = e.half * 2 + p;
        float v[64];
        epi_load64(e, pc * 64, v);
        uint8_t* const st = staging_turn(e, p).staging;
#pragma unroll
        for (int j = 0; j < 8; j++) {
          uint4 o; __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
          for (int q = 0; q < 4; q++) o2[q] = __floats2bfloat162_rn(v[8 * j + 2 * q], v[8 * j + 2 * q + 1]);
          *reinterpret_cast<uint4*>(st + j * 512 + e.lane * 16) = o;
        }
        fence_proxy_async();                             // these stores must be visible to the bulk-copy engine
        __syncwarp();
        if (e.lane == 0) { bulk_store(piece(owner, rank, t, e, pc), st, PAIR_STAGING); bulk_commit(); }
      }
      if (e.lane == 0) { announce<2>(); pending = flag_ptr(owner, rank, t); pending_slot = slot; }
      __syncwarp();
      return true;
    }
    // own tile: all other ranks' partials of this tile must have landed
    const bool ok = e.lane >= n || e.lane == rank || wait_flag(flag_ptr(rank, e.lane, t), a.epoch, a.one_gpu, abort_flag);
    if (!__all_sync(0xffffffffu, ok)) return false;
#pragma unroll 1
    for (int p = 0; p < 2; p++) {
      const int pc = e.half * 2 + p;
      const EpiCtx b = staging_turn(e, p);
#pragma unroll 1
      for (int h = 0; h < 2; h++) {                      // 32 columns; the words of four partials are in flight at a time
        float sum[32];
#pragma unroll
        for (int i = 0; i < 32; i++) sum[i] = 0.f;
        auto add_own = [&]() {
          uint32_t r[32];
          tmem_ld_32x32(e.tmem + pc * 64 + h * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i++) sum[i] += __uint_as_float(r[i]);
        };
#pragma unroll
        for (int q0 = 0; q0 < TP_MAX_RANKS - 1; q0 += 4) {  // rank order: the same result whatever the arrival order
          uint4 w[4][4];
#pragma unroll
          for (int i = 0; i < 4; i++) {
            if (q0 + i < n - 1) {
              const char* p = piece(rank, q0 + i < rank ? q0 + i : q0 + i + 1, t, e, pc) + h * 2048 + e.lane * 16;
#pragma unroll
              for (int j = 0; j < 4; j++)
                asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[i][j].x), "=r"(w[i][j].y), "=r"(w[i][j].z), "=r"(w[i][j].w) : "l"(p + j * 512) : "memory");
            }
          }
#pragma unroll
          for (int i = 0; i < 4; i++) {
            if (q0 + i == rank) add_own();
            if (q0 + i < n - 1) {
#pragma unroll
              for (int j = 0; j < 4; j++) {
                const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&w[i][j]);
#pragma unroll
                for (int q = 0; q < 4; q++) { float2 f = __bfloat1622float2(b2[q]); sum[8 * j + 2 * q] += f.x; sum[8 * j + 2 * q + 1] += f.y; }
              }
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
          uint4 o; __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
          for (int q = 0; q < 4; q++) o2[q] = __floats2bfloat162_rn(sum[8 * j + 2 * q], sum[8 * j + 2 * q + 1]);
          *reinterpret_cast<uint4*>(b.staging + e.lane * 128 + (((h * 4 + j) ^ (e.lane & 7)) << 4)) = o;      // as epi_stage_row lays a row out
        }
      }
      fence_proxy_async();
      __syncwarp();
      epi_ship(b, &R->tc, n_blk * TP_BN + pc * 64, (m_blk % mb_per_owner) * TP_BM + e.quarter * 32);
    }
    return true;
  }
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1) gemm_rs_kernel(const __grid_constant__ TpArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ int s_abort;
  __shared__ unsigned s_arrived[4];
  if (threadIdx.x == 0) { s_abort = 0; for (int i = 0; i < 4; i++) s_arrived[i] = 0; }
  RsPolicy pol(a, s_arrived);
  gemm_pair_persistent<TP_BN, RS_STAGES, false, false>(smem_raw, pol, a.K, blockIdx.x >> 1, gridDim.x >> 1, &s_abort);
}

// ------------------------------------------------------------------ all-gather -> GEMM
constexpr int FEED_PIECE = 4096, FEED_STAGES = 8, FEED_AHEAD = 5;
struct AgPolicy {
  const TpArgs& a; const TpRank* R = nullptr; int rank = 0, mb_per_shard, num_n, parity;
  static constexpr int NSTAGE = 1, EXTRA_BYTES = FEED_STAGES * FEED_PIECE + FEED_STAGES * 8;
  __device__ AgPolicy(const TpArgs& args) : a(args), mb_per_shard(args.M / args.n / TP_BM), num_n(args.N / TP_BN), parity((int)(args.epoch & 1)) {}
  __device__ void begin() const {}
  __device__ void report(int role) const { for (int i = 0; i < a.nv; i++) atomicExch(a.r[i].status, role); }
  __device__ int num_tiles() const { return a.nv * ((a.M / TP_BM + 1) / 2) * num_n; }
  // Row blocks of the own shard first, then rank+1, ..., two to a pair; chunks of pairs, inside a chunk rows fastest (bands of 16).  The
  // first chunk is the own shard, of every rank of the launch; after that a chunk is about a shard, so that little has to have arrived before it
  // starts, or, with several ranks on the device, 16 pairs: their own shards gave the feeding time enough, and B is read less often.
  __device__ void tile(int idx, int v, int& m_blk, int& n_blk) {
    constexpr int BAND = 16;
    const int rp = (a.M / TP_BM + 1) / 2, own = (mb_per_shard + 1) / 2, chunk = a.nv > 1 ? BAND : own;
    int base = 0, rows = own, w = idx;
    const int first = a.nv * own * num_n;
    if (w >= first) {
      w -= first;
      const int c = w / (a.nv * chunk * num_n);
      w %= a.nv * chunk * num_n;
      base = own + c * chunk; rows = min(chunk, rp - base);
    }
    R = &a.r[w / (rows * num_n)]; rank = R->rank;
    w %= rows * num_n;
    const int band = w / (BAND * num_n), in_band = min(BAND, rows - band * BAND);
    w %= BAND * num_n;
    const int i = 2 * (base + band * BAND + w % in_band) + v;
    n_blk = w / in_band;
    m_blk = i < a.n * mb_per_shard ? (rank + i / mb_per_shard) % a.n * mb_per_shard + i % mb_per_shard : -1;
  }
  __device__ void k_range(int, int num_kb, int& kb0, int& kb1) const { kb0 = 0; kb1 = num_kb; }
  __device__ const CUtensorMap* a_map(int m_blk, int& row0) const {
    if (m_blk < 0) { row0 = 0; return &R->ta; }
    if (m_blk / mb_per_shard == rank) { row0 = (m_blk % mb_per_shard) * TP_BM; return &R->ta; }
    row0 = m_blk * TP_BM; return &R->ta2;               // ta2 covers this call's half of the region
  }
  __device__ const CUtensorMap* b_map() const { return &R->tb; }
  __device__ unsigned* flags(const TpRank* r, int dest, int src, int mb) const {
    return reinterpret_cast<unsigned*>(r->heap[dest] + a.flag_off + tp_flag_at(parity, src, (long long)mb_per_shard * a.n_part, (long long)mb * a.n_part));
  }
  __device__ bool gate(int m_blk, volatile int* abort_flag) const {
    if (m_blk < 0 || m_blk / mb_per_shard == rank) return true;
    const int lane = threadIdx.x & 31;
    const unsigned* f = flags(R, rank, m_blk / mb_per_shard, m_blk % mb_per_shard);
    const bool ok = lane >= a.n_part || wait_flag(f + lane, a.epoch, a.one_gpu, abort_flag);
    const bool all = __all_sync(0xffffffffu, ok);
    asm volatile("fence.proxy.async;" ::: "memory");    // the rows arrived before the flags; TMA reads them through the async proxy
    return all;
  }
  __device__ void prefetch(const EpiCtx&, int, int) {}
  __device__ void finish(const EpiCtx&) {}
  __device__ bool epilogue(const EpiCtx& e, int, int m_blk, int n_blk, volatile int*) {
    if (m_blk < 0) return true;
#pragma unroll 1
    for (int pc = e.half * 2; pc < e.half * 2 + 2; pc++) {
      float v[64];
      epi_load64(e, pc * 64, v);
      epi_staging_free(e);
      epi_stage_row(e, v);
      epi_ship(e, &R->tc, n_blk * TP_BN + pc * 64, m_blk * TP_BM + e.quarter * 32);
    }
    return true;
  }
  // The feeding warp: parts of the shard's row blocks to the peers, distance-major (the peer that needs my shard next comes first), spread over
  // all CTAs.  One lane streams a part through the ring, FEED_AHEAD loads in flight, and raises the part's flag when its stores have been performed.
  __device__ void extra_warp(uint8_t* smem, int lane, volatile int* abort_flag) {
    if (lane != 0) return;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + FEED_STAGES * FEED_PIECE);
    for (int i = 0; i < FEED_STAGES; i++) mbar_init(&bar[i], 1);
    fence_barrier_init();
    uint32_t phase = 0;                                  // bit s: the parity the next wait on stage s looks for
    const size_t block_bytes = (size_t)TP_BM * a.K * 2, part_bytes = block_bytes / a.n_part;
    const int per_dest = mb_per_shard * a.n_part, units = (a.n - 1) * a.nv * per_dest, np = (int)((part_bytes + FEED_PIECE - 1) / FEED_PIECE);
    bool ok = true;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const int step = u / per_dest, mb = u % per_dest / a.n_part, part = u % a.n_part;
      const TpRank* r = &a.r[step % a.nv];
      const int from = r->rank, dest = (from - 1 - step / a.nv + a.n) % a.n;
      const size_t off = (size_t)mb * block_bytes + (size_t)part * part_bytes;
      const char* src = reinterpret_cast<const char*>(r->a_shard) + off;
      char* dst = r->heap[dest] + a.data_off + (size_t)from * (a.M / a.n) * a.K * 2 + off;
      int issued = 0;
      for (int i = 0; i < np + FEED_AHEAD; i++) {
        if (i < np && ok) {
          issued = i + 1;
          const uint32_t bytes = (uint32_t)min((size_t)FEED_PIECE, part_bytes - (size_t)i * FEED_PIECE);
          const int st = i % FEED_STAGES;
          // the stage last held piece i - FEED_STAGES: all but the newest stores have been read out of shared memory
          if (i >= FEED_STAGES) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(FEED_STAGES - 1 - FEED_AHEAD) : "memory");
          mbar_arrive_expect_tx(&bar[st], bytes);
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem + st * FEED_PIECE)),
                       "l"(src + (size_t)i * FEED_PIECE), "r"(bytes), "r"(smem_u32(&bar[st])) : "memory");
        }
        const int j = i - FEED_AHEAD;
        if (j >= 0 && j < issued) {                      // every issued load is waited for, also after a failure
          const int st = j % FEED_STAGES;
          const bool landed = mbar_wait(&bar[st], (phase >> st) & 1u, abort_flag, kPairWaitLimitNs);
          phase ^= 1u << st;
          if (!landed) { ok = false; continue; }
          const uint32_t bytes = (uint32_t)min((size_t)FEED_PIECE, part_bytes - (size_t)j * FEED_PIECE);
          bulk_store(dst + (size_t)j * FEED_PIECE, smem + st * FEED_PIECE, bytes); bulk_commit();
        }
      }
      bulk_wait_all();                                   // the writes are performed; then tell the reader
      asm volatile("fence.proxy.async;" ::: "memory");
      if (ok) st_release_u32(flags(r, dest, from, mb) + part, a.epoch, a.one_gpu);
    }
    if (!ok) { *abort_flag = 1; report(7); }
  }
};

constexpr int AG_THREADS = PAIR_THREADS + 32;
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(AG_THREADS, 1) ag_gemm_kernel(const __grid_constant__ TpArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ int s_abort;
  if (threadIdx.x == 0) s_abort = 0;
  AgPolicy pol(a);
  gemm_pair_persistent<TP_BN, AG_STAGES, false, false>(smem_raw, pol, a.K, blockIdx.x >> 1, gridDim.x >> 1, &s_abort);
}

// ------------------------------------------------------------------ all ranks in one launch on one GPU
// There every rank's operands can be read where they are: nothing is pushed, flagged or waited for.  ag_gemm takes the rows of a shard from its owner; gemm_rs sums an owner's tile over
// all ranks' k in the accumulator, where the partial tiles otherwise go through memory as bf16.  Without waits between CTAs the launch need not be cooperative, overlaps the end of the kernel
// before, has no more CTAs than tiles, and takes narrow tiles where wide ones leave the chip idle.  Large products are bound by the power cap, small ones by the launch and one tile's k.
// us, exchanging through the workspace and this: ag_gemm 2 x 4096 x 2048 x 4096 120 / 109, 2 x 512 x 768 x 1024 16.4 / 7.7, 4 x 3584 x 1280 x 1728 86.7 / 52.5, 8 x 8192 x 8192 x 4096 3439 / 3179;
// gemm_rs 8 x 8192 x 8192 x 3584 3021 / 2931, 4 x 512 x 1280 x 384 18.5 / 9.5, 2 x 8192 x 8192 x 256 159 / 66, 8 x 8192 x 1024 x 4096 473 / 449.
template <int TN, bool RS>
struct LocalPolicy {
  const TpArgs& a; const TpRank* R = nullptr; int rank = 0, mb_per_shard, blocks, rp, num_n, kb_per_rank;
  static constexpr int EXTRA_BYTES = 0, NSTAGE = 1;
  static constexpr bool K_RANKS = RS;
  __device__ LocalPolicy(const TpArgs& args)
      : a(args), mb_per_shard(args.M / args.n / TP_BM), blocks(args.M / TP_BM), rp((blocks + 1) / 2), num_n(args.N / TN), kb_per_rank(args.K / TP_BK) {}
  __device__ void begin() const {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }
  __device__ void report(int role) const { for (int i = 0; i < a.nv; i++) atomicExch(a.r[i].status, role); }
  __device__ int num_tiles() const { return (RS ? 1 : a.nv) * rp * num_n; }
  // ag_gemm: one rank after the other; bands of 16 pairs of row blocks, inside a band rows fastest.  gemm_rs: bands of 8 pairs across owners, so that a wave of the grid is about as many
  // rows as columns: each wave reads all ranks' k of them.  A pair of CTAs may work for two owners: with one row block to each of eight ranks half of the CTAs would multiply for nothing.
  __device__ void tile(int idx, int v, int& m_blk, int& n_blk) {
    if (RS) {
      constexpr int BAND = 8;
      const int band = idx / (BAND * num_n), in_band = min(BAND, rp - band * BAND), w = idx % (BAND * num_n), i = 2 * (band * BAND + w % in_band) + v;
      n_blk = w / in_band;
      rank = min(i, blocks - 1) / mb_per_shard;
      R = &a.r[rank];
      m_blk = i < blocks ? i % mb_per_shard : -1;
      return;
    }
    constexpr int BAND = 16;
    rank = idx / (rp * num_n);
    R = &a.r[rank];
    int w = idx % (rp * num_n);
    const int band = w / (BAND * num_n), in_band = min(BAND, rp - band * BAND);
    w %= BAND * num_n;
    const int i = 2 * (band * BAND + w % in_band) + v;
    n_blk = w / in_band;
    m_blk = i < blocks ? i : -1;
  }
  __device__ void k_range(int, int num_kb, int& kb0, int& kb1) const { kb0 = 0; kb1 = num_kb; }
  __device__ const CUtensorMap* a_map(int m_blk, int& row0) const {
    const int m = max(m_blk, 0);
    if (RS) { row0 = (rank * mb_per_shard + m) * TP_BM; return &R->ta; }
    row0 = m % mb_per_shard * TP_BM; return &a.r[m / mb_per_shard].ta;
  }
  __device__ const CUtensorMap* b_map() const { return &R->tb; }
  __device__ const CUtensorMap* a_of(int p) const { return &a.r[p].ta; }
  __device__ const CUtensorMap* b_of(int p) const { return &a.r[p].tb; }
  __device__ bool gate(int, volatile int*) const { return true; }
  __device__ void prefetch(const EpiCtx&, int, int) {}
  __device__ void finish(const EpiCtx&) {}
  __device__ bool epilogue(const EpiCtx& e, int, int m_blk, int n_blk, volatile int*) {
    constexpr int PIECES = TN / 128 > 0 ? TN / 128 : 1;      // of 64 columns, to each half of the warps; a tile of 64 columns is the first half's
    if (m_blk < 0 || e.half * PIECES * 64 >= TN) return true;
#pragma unroll 1
    for (int pc = e.half * PIECES; pc < (e.half + 1) * PIECES; pc++) {
      float v[64];
      epi_load64(e, pc * 64, v);
      epi_staging_free(e);
      epi_stage_row(e, v);
      epi_ship(e, &R->tc, n_blk * TN + pc * 64, m_blk * TP_BM + e.quarter * 32);
    }
    return true;
  }
};
template <int TN, int STAGES, bool RS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1) tp_local_kernel(const __grid_constant__ TpArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ int s_abort;
  if (threadIdx.x == 0) s_abort = 0;
  LocalPolicy<TN, RS> pol(a);
  gemm_pair_persistent<TN, STAGES, false, false>(smem_raw, pol, RS ? a.n * a.K : a.K, blockIdx.x >> 1, gridDim.x >> 1, &s_abort);
}
struct LocalVariant { void (*fn)(TpArgs); int tn, smem; };
static const LocalVariant kLocal[2][3] = {
    {{tp_local_kernel<256, 6, true>, 256, PairSmem<256, 6>::DYNAMIC}, {tp_local_kernel<128, 8, true>, 128, PairSmem<128, 8>::DYNAMIC}, {tp_local_kernel<64, 9, true>, 64, PairSmem<64, 9>::DYNAMIC}},
    {{tp_local_kernel<256, 6, false>, 256, PairSmem<256, 6>::DYNAMIC}, {tp_local_kernel<128, 8, false>, 128, PairSmem<128, 8>::DYNAMIC}, {tp_local_kernel<64, 9, false>, 64, PairSmem<64, 9>::DYNAMIC}}};

// ------------------------------------------------------------------ host
// The workspace is used in four quarters: [kernel: gemm_rs, ag_gemm][parity of that kernel's call count].
static long long tp_quarter(long long tp_bytes) { return tp_bytes / 4 / 1024 * 1024; }
static long long tp_need_per_call(int which, int nranks, int M, int N, int K) {
  if (which == 0) return (long long)nranks * ((long long)M / nranks / TP_BM) * (N / TP_BN) * (TP_BM * TP_BN * 2);     // [src][tile] bf16 tiles
  return (long long)M * K * 2;                                                                                              // [M][K] bf16
}

// Flags per row block: 16 parts of 8 K bytes spread a block over as many CTAs (a power of two; fewer where the flag area would not hold them).
static int ag_parts(int M) {
  int p = 16;
  while (p > 1 && (M / TP_BM) * 4LL * p > TP_FLAG_CALL) p /= 2;
  return p;
}
static long long tp_flags_per_src(int which, int nranks, int M, int N) {
  const long long blocks = M / nranks / TP_BM;
  return which == 0 ? blocks * (N / TP_BN) : blocks * ag_parts(M);
}

static int tp_common_checks(piccl_comm** cs, int n, int M, int N, int K, int which) {
  if (n < 1 || n > TP_MAX_RANKS) return fail(PICCL_INVALID_ARGUMENT, "1..%d communicators per launch", TP_MAX_RANKS);
  piccl_comm* c = cs[0];
  if (c->nranks > TP_MAX_RANKS) return fail(PICCL_UNSUPPORTED, "fused tensor-parallel kernels support up to %d ranks", TP_MAX_RANKS);
  for (int i = 0; i < n; i++) if (!cs[i]->connected || cs[i]->broken) return fail(PICCL_INVALID_USAGE, "communicator not usable");
  if (M <= 0 || M % (TP_BM * c->nranks) || N % TP_BN || K % TP_BK || N <= 0 || K <= 0) return fail(PICCL_INVALID_ARGUMENT, "shape: M %% (128*ranks), N %% 256, K %% 64 must be 0");
  if (c->nranks * tp_flags_per_src(which, c->nranks, M, N) * 4 > TP_FLAG_CALL) return fail(PICCL_UNSUPPORTED, "too many tiles for the flag area");
  long long need = piccl_tp_workspace_bytes(which, c->nranks, M, N, K);
  if (tp_quarter(c->h_ctx.tp_bytes) < tp_need_per_call(which, c->nranks, M, N, K)) return fail(PICCL_INVALID_USAGE, "tensor-parallel workspace too small: %lld bytes needed, %lld configured (tp_bytes / PICCL_TP_MB)", need, c->h_ctx.tp_bytes);
  return PICCL_OK;
}

// All ranks in this launch on one GPU, and no result over an operand?
static bool tp_local(piccl_comm** cs, int n, const void* const* A, const void* const* B, void* const* out, int M, int N, int K, int which) {
  if (n < 2 || n != cs[0]->nranks) return false;
  const long long rows = M / n, a_bytes = (which ? rows : M) * 2LL * K, b_bytes = 2LL * N * K, o_bytes = (which ? M : rows) * 2LL * N;
  auto meet = [](const void* x, long long nx, const void* y, long long ny) { return (const char*)x < (const char*)y + ny && (const char*)y < (const char*)x + nx; };
  for (int i = 0; i < n; i++) {
    if (cs[i]->rank != i || cs[i]->device != cs[0]->device || cs[i]->slots_only) return false;
    for (int j = 0; j < n; j++) if (meet(out[i], o_bytes, A[j], a_bytes) || meet(out[i], o_bytes, B[j], b_bytes) || (i < j && meet(out[i], o_bytes, out[j], o_bytes))) return false;
  }
  return true;
}
static long long tp_local_tiles(int n, int M, int N, int which, int tn) { return (long long)(which ? n : 1) * ((M / TP_BM + 1) / 2) * (N / tn); }
// Tile width (index into kLocal[which]) for operands read where they are: waves of the persistent grid times the clocks of a tile, which are those of the plain GEMM (gemm_sm100.cu: choose).
// *exchange: the exchanging form is the faster one.  That is so for gemm_rs with a long k and few tiles: summing all ranks' k in one accumulator has 1 / n of the tiles, each n times as long, and leaves the chip idle
// where the ranks' own products would fill it.  The exchange costs a fifth more than its tiles and 8 us.  Of 89 shapes the rule picks the slower form, by more than 2 %, for none (us, exchanging and
// reading: 8 ranks 1024 x 256 x 4096 40 / 94, 2048 x 256 x 4096 47 / 95, 2048 x 1280 x 1664 68 / 72, 4 ranks 1024 x 1024 x 4096 39 / 51, 3 ranks 384 x 512 x 4096 33 / 37; on the other side 8 ranks 3072 x 1024 x 4096
// 174 / 165, 1024 x 512 x 960 28.7 / 25.5, 4 ranks 512 x 2048 x 4096 57 / 50, 2 ranks 512 x 256 x 4096 33 / 26).
static int tp_local_width(int n, int M, int N, int K, int which, int pairs, bool* exchange) {
  const long long kb = (which ? K : (long long)n * K) / TP_BK;
  int best = 0; double best_cost = 0;
  auto waves = [&](long long tiles) { return (double)((tiles + pairs - 1) / pairs); };
  for (int v = 0; v < 3; v++) {
    const int tn = kLocal[which][v].tn;
    const double cost = waves(tp_local_tiles(n, M, N, which, tn)) * ((tn == 256 ? 136 : tn == 128 ? 84 : 70) * 4.0 * kb + 10.0 * tn);
    if (v == 0 || cost < best_cost) { best = v; best_cost = cost; }
  }
  *exchange = false;
  if (which == 0) {
    const long long mb = M / n / TP_BM, tiles = n * (((n - 1) * mb + 1) / 2 + (mb + 1) / 2) * (N / TP_BN);      // (pairs of row blocks for others and of own ones)
    const double other = waves(tiles) * (136 * 4.0 * (K / TP_BK) + 10.0 * TP_BN);
    // (the narrowest tiles of a long chain take 80 clocks: the ring of stages is shorter than memory is far)
    *exchange = best_cost * (kLocal[0][best].tn == 64 ? 80.0 / 70.0 : 1.0) > 1.2 * other + 15000;
  }
  return best;
}

static int tp_launch(piccl_comm** cs, int n, const void* const* A, const void* const* B, void* const* out, int M, int N, int K, int which, cudaStream_t stream) {
  int rc = tp_common_checks(cs, n, M, N, K, which); if (rc) return rc;
  piccl_comm* c0 = cs[0];
  const int nr = c0->nranks;
  struct Guard {
    int prev = -1, dev;
    explicit Guard(int d) : dev(d) { cudaGetDevice(&prev); if (prev != dev) cudaSetDevice(dev); }
    ~Guard() { if (prev >= 0 && prev != dev) cudaSetDevice(prev); }
  } guard(c0->device);
  TpArgs a; memset(&a, 0, sizeof a);
  a.n = nr; a.M = M; a.N = N; a.K = K;
  a.flag_off = c0->h_ctx.tp_flag_off + (which ? TP_FLAG_KERNEL : 0);   // the two kernels keep their flags apart
  // ... and their payload: each kernel owns one half of the workspace, and each call one half of that, chosen by the parity of
  // the kernel's own call count.  Neither these places nor the flags' depend on the shape: a rank that is one call ahead (the other kernel, or
  // the same kernel with another shape) never writes where a peer still reads the call before.
  const long long quarter = tp_quarter(c0->h_ctx.tp_bytes);
  const unsigned next_epoch = (which ? c0->tp_epoch_ag : c0->tp_epoch_rs) + 1;
  a.data_off = c0->h_ctx.tp_data_off + (which ? 2 * quarter : 0) + (long long)(next_epoch & 1) * quarter;
  a.n_part = ag_parts(M);
  const int smem_bytes = which ? PairSmem<TP_BN, AG_STAGES, AgPolicy::EXTRA_BYTES>::DYNAMIC : PairSmem<TP_BN, RS_STAGES, RsPolicy::EXTRA_BYTES, RsPolicy::NSTAGE>::DYNAMIC;
  const int threads = which ? AG_THREADS : PAIR_THREADS;
  auto fn = which ? ag_gemm_kernel : gemm_rs_kernel;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem_bytes; cfg.stream = stream;
  cudaLaunchAttribute at[1];
  if (!c0->tp_pairs[which]) {
    // pairs that can be resident at once (a pair needs two SMs of one GPC): the persistent grid is never larger, the ranks wait for one another
    if (cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess) return fail(PICCL_CUDA_ERROR, "cannot get %d bytes of shared memory", smem_bytes);
    at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(c0->sm_count / 2 * 2); cfg.attrs = at; cfg.numAttrs = 1;
    int active = 0;
    if (cudaOccupancyMaxActiveClusters(&active, fn, &cfg) != cudaSuccess || active < 1) { cudaGetLastError(); return fail(PICCL_CUDA_ERROR, "no room for a pair of CTAs with %d bytes of shared memory each", smem_bytes); }
    c0->tp_pairs[which] = std::min(active, c0->sm_count / 2);
  }
  a.nv = n; a.one_gpu = n == nr;
  bool ok = true;
  bool local = tp_local(cs, n, A, B, out, M, N, K, which), exchange = false;
  const LocalVariant& lv = kLocal[which][local ? tp_local_width(n, M, N, K, which, c0->tp_pairs[which], &exchange) : 0];
  if (local && exchange) {
    // (not while the stream is being captured: the exchange's epoch is a launch argument, a replay would reuse it)
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) { cudaGetLastError(); cap = cudaStreamCaptureStatusNone; }
    local = cap != cudaStreamCaptureStatusNone;
  }
  for (int i = 0; i < n && ok; i++) {
    piccl_comm* c = cs[i];
    TpRank& R = a.r[i];
    a.one_gpu &= c->device == c0->device;
    R.rank = c->rank; R.out = (bf16*)out[i]; R.a_shard = (const bf16*)A[i];
    for (int p = 0; p < nr; p++) R.heap[p] = c->h_ctx.heap[p];
    if (!c->d_tp_status) { if (cudaMalloc(&c->d_tp_status, sizeof(int)) != cudaSuccess) { ok = false; break; } cudaMemset(c->d_tp_status, 0, sizeof(int)); }
    R.status = c->d_tp_status;
    if (which == 0) {
      ok &= make_tmap_bf16_k64(&R.ta, A[i], (uint64_t)M, (uint64_t)K, (uint64_t)K, TP_BM);
      R.ta2 = R.ta;
      if (!local) a.epoch = ++c->tp_epoch_rs;
    } else {
      ok &= make_tmap_bf16_k64(&R.ta, A[i], (uint64_t)(M / nr), (uint64_t)K, (uint64_t)K, TP_BM);
      if (!local) { ok &= make_tmap_bf16_k64(&R.ta2, c->heap + a.data_off, (uint64_t)M, (uint64_t)K, (uint64_t)K, TP_BM); a.epoch = ++c->tp_epoch_ag; }
    }
    ok &= make_tmap_bf16_k64(&R.tb, B[i], (uint64_t)N, (uint64_t)K, (uint64_t)K, local ? lv.tn / 2 : TP_BN / 2);
    ok &= make_tmap_bf16_k64(&R.tc, out[i], (uint64_t)(which ? M : M / nr), (uint64_t)N, (uint64_t)N, 32);
  }
  if (!ok) return fail(PICCL_CUDA_ERROR, "tensor map or status set-up failed");
  if (local) {
    const int bit = 1 << (3 * which + (int)(&lv - kLocal[which]));
    if (!(c0->tp_local_ready & bit)) {
      if (cudaFuncSetAttribute((const void*)lv.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, lv.smem) != cudaSuccess) return fail(PICCL_CUDA_ERROR, "cannot get %d bytes of shared memory", lv.smem);
      c0->tp_local_ready |= bit;
    }
    const long long tiles = tp_local_tiles(n, M, N, which, lv.tn);
    cfg.gridDim = dim3(2 * (unsigned)std::min<long long>(tiles, c0->tp_pairs[which])); cfg.blockDim = dim3(PAIR_THREADS); cfg.dynamicSmemBytes = lv.smem;
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, lv.fn, a);
    if (e != cudaSuccess) return fail(PICCL_CUDA_ERROR, "fused kernel launch failed: %s", cudaGetErrorString(e));
    for (int i = 0; i < n; i++) cs[i]->stats.launches++;
    return PICCL_OK;
  }
  // ranks wait for one another inside the kernel: with several virtual ranks on one device all CTAs must be resident at once
  at[0].id = cudaLaunchAttributeCooperative; at[0].val.cooperative = 1;
  cfg.gridDim = dim3(2 * c0->tp_pairs[which]); cfg.attrs = at; cfg.numAttrs = n > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, a);
  if (e != cudaSuccess) return fail(PICCL_CUDA_ERROR, "fused kernel launch failed: %s", cudaGetErrorString(e));
  for (int i = 0; i < n; i++) cs[i]->stats.launches++;
  return PICCL_OK;
}

}  // namespace piccl

using namespace piccl;

extern "C" {

long long piccl_tp_workspace_bytes(int which, int nranks, int M, int N, int K) {
  // four quarters (two kernels x two calls in flight), each large enough for one call of this shape
  return 4 * ((tp_need_per_call(which, nranks, M, N, K) + 1023) / 1024 * 1024);
}
int piccl_tp_flag_range(int which, int nranks, int M, int N, int parity, long long* begin, long long* end) {
  if (which < 0 || which > 1 || nranks < 1 || nranks > TP_MAX_RANKS || M <= 0 || M % (TP_BM * nranks) || N <= 0 || N % TP_BN || parity < 0 || parity > 1) return fail(PICCL_INVALID_ARGUMENT, "no such call");
  const long long per_src = tp_flags_per_src(which, nranks, M, N), base = which ? TP_FLAG_KERNEL : 0;
  if (nranks * per_src * 4 > TP_FLAG_CALL) return fail(PICCL_UNSUPPORTED, "too many tiles for the flag area");
  *begin = base + tp_flag_at(parity, 0, per_src, 0); *end = base + tp_flag_at(parity, nranks - 1, per_src, per_src - 1) + 4;
  return PICCL_OK;
}
// Columns of a tile where a launch carries all ranks on one GPU with `pairs` pairs of CTAs; 0: the ranks exchange.
int piccl_test_tp_width(int which, int nranks, int M, int N, int K, int pairs) {
  bool exchange = false;
  const int v = tp_local_width(nranks, M, N, K, which, pairs, &exchange);
  return exchange ? 0 : kLocal[which][v].tn;
}
int piccl_gemm_rs(piccl_comm_t* c, const void* A, const void* B, void* out, int M, int N, int K_local, void* stream) {
  if (!c) return fail(PICCL_INVALID_ARGUMENT, "null communicator");
  const void* as[1] = {A}; const void* bs[1] = {B}; void* os[1] = {out}; piccl_comm* cs[1] = {c};
  return tp_launch(cs, 1, as, bs, os, M, N, K_local, 0, (cudaStream_t)stream);
}
int piccl_ag_gemm(piccl_comm_t* c, const void* A_shard, const void* B, void* out, int M, int N_local, int K, void* stream) {
  if (!c) return fail(PICCL_INVALID_ARGUMENT, "null communicator");
  const void* as[1] = {A_shard}; const void* bs[1] = {B}; void* os[1] = {out}; piccl_comm* cs[1] = {c};
  return tp_launch(cs, 1, as, bs, os, M, N_local, K, 1, (cudaStream_t)stream);
}
int piccl_gemm_rs_group(piccl_comm_t** comms, int n, const void* const* A, const void* const* B, void* const* out, int M, int N, int K_local, void* stream) {
  return tp_launch(comms, n, A, B, out, M, N, K_local, 0, (cudaStream_t)stream);
}
int piccl_ag_gemm_group(piccl_comm_t** comms, int n, const void* const* A_shard, const void* const* B, void* const* out, int M, int N_local, int K, void* stream) {
  return tp_launch(comms, n, A_shard, B, out, M, N_local, K, 1, (cudaStream_t)stream);
}
int piccl_tp_status(piccl_comm_t* c) {
  if (!c || !c->d_tp_status) return 0;
  int v = 0; cudaMemcpy(&v, c->d_tp_status, sizeof v, cudaMemcpyDeviceToHost);
  return v;
}

}  // extern "C"

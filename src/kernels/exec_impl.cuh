// The fused collective executor: ONE kernel runs a whole collective.  Each CTA
// owns a fixed slice of every action; for each window of FIFO segments it walks
// the action program, and every (action, segment) is a step, a single pass
//     wait (bounded) -> load local + incoming slots -> reduce in registers ->
//     store local + peers' slots -> publish counters
// so reduction (reference: src/kernels/reduce_kernel.cu, one launch per step)
// and block placement (reference: src/kernels/permutation_kernel.cu) never
// exist as separate passes, and no ncclSend/ncclRecv is issued.
//
// Roles inside a CTA: one warp waits (credits and data of the next steps, up to
// kStepDepth ahead), all warps but two move data, one warp publishes (its fence
// waits for the acknowledgement of everything the CTA stored, a microsecond and
// more).  They meet through named barriers per step, so the chain
//     peer's stores -> its release -> my poll -> my loads
// of one step overlaps the data movement of others.  With one group of threads doing all of it in
// turn a 64 KiB step took 10 us, 3 of them for the data.
//
// Peer traffic is plain 16-byte stores into the peer's mapped heap (NVLink /
// NVSwitch P2P); ordering is a fence and a relaxed store on the producer and
// an acquiring load on the consumer, and the same way back for the slots that are free.  Every wait has a time limit; on expiry the CTA records
// where it gave up, raises the abort flag that all other waits poll, and the
// kernel returns.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "exec.cuh"
#include "../include/piccl_slice.h"

namespace piccl {

// ---------------------------------------------------------------- memory primitives
// Counters and fences, for ranks on several GPUs or all on one.  At system scope every fence also waits on the way to the host and the peers: with all
// ranks on one GPU all-reduce 8 x 4 MiB on the ring took 79 us, at GPU scope 56; all-gather 8 x 2 MiB 94 / 72, 4 x 1 MiB at odd addresses 35.6 / 28.5, all-reduce
// 8 x 64 MiB 370 / 360 (on a machine where that way was short 60 / 56, 76 / 72, 29.5 / 28.5 and 367 / 360).
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p, bool one_gpu) {
  unsigned long long v;
  if (one_gpu) asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  else asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v, bool one_gpu) {
  if (one_gpu) asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
  else asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void fence_ranks(bool one_gpu) {
  if (one_gpu) asm volatile("fence.acq_rel.gpu;" ::: "memory");
  else asm volatile("fence.acq_rel.sys;" ::: "memory");
}
__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// FIFO payload written by another GPU: read past L1.
__device__ __forceinline__ uint4 ld_slot(const void* p) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
// The same, and stores, with the priority that the line gets in L2: one that is done with goes first, so that the FIFO's slots, which another rank reads
// next, stay.
__device__ __forceinline__ unsigned long long l2_policy(bool first) {
  unsigned long long p;
  if (first) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  else asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint4 ld_hint(const void* p, unsigned long long policy) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.L2::cache_hint.v4.u32 {%0,%1,%2,%3}, [%4], %5;" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "l"(policy) : "memory");
  return v;
}
__device__ __forceinline__ void st_hint(void* p, const uint4& v, unsigned long long policy) {
  asm volatile("st.global.L2::cache_hint.v4.u32 [%0], {%1,%2,%3,%4}, %5;" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "l"(policy) : "memory");
}
__device__ __forceinline__ void st_vec(void* p, const uint4& v) { *reinterpret_cast<uint4*>(p) = v; }

// ---------------------------------------------------------------- element-wise maths
constexpr int OP_COPY = 4;            // collectives that only move data: no action has two operands
template <int OP, typename A> __device__ __forceinline__ A red(A x, A y) {
  if (OP == 0) return x + y;
  if (OP == 1) return x * y;
  if (OP == 2) return x > y ? x : y;
  return x < y ? x : y;
}

template <typename T> struct AccOf { typedef T type; };
template <> struct AccOf<__half> { typedef float type; };
template <> struct AccOf<__nv_bfloat16> { typedef float type; };

template <typename T> struct Cvt {
  typedef typename AccOf<T>::type A;
  static __device__ __forceinline__ A up(T v) { return (A)v; }
  static __device__ __forceinline__ T down(A v) { return (T)v; }
};
template <> struct Cvt<__half> {
  static __device__ __forceinline__ float up(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half down(float v) { return __float2half_rn(v); }
};
template <> struct Cvt<__nv_bfloat16> {
  static __device__ __forceinline__ float up(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 down(float v) { return __float2bfloat16_rn(v); }
};

template <typename T> struct Pack {
  static constexpr int N = 16 / sizeof(T);
  typedef typename AccOf<T>::type A;
  union U { uint4 v; T t[N]; };
  static __device__ __forceinline__ void up(const uint4& v, A (&a)[N]) {
    U u; u.v = v;
#pragma unroll
    for (int i = 0; i < N; i++) a[i] = Cvt<T>::up(u.t[i]);
  }
  static __device__ __forceinline__ uint4 down(const A (&a)[N]) {
    U u;
#pragma unroll
    for (int i = 0; i < N; i++) u.t[i] = Cvt<T>::down(a[i]);
    return u.v;
  }
};

template <typename A> __device__ __forceinline__ A scale_val(A v, float s) { return v; }
template <> __device__ __forceinline__ float scale_val<float>(float v, float s) { return v * s; }
template <> __device__ __forceinline__ double scale_val<double>(double v, float s) { return v * (double)s; }

// Operands to scale (avg): bit s, operand s is an original contribution; bit 8 + s, of another rank, which would have put it into a slot: it is rounded to the
// element type as it would be there, so that a call's result does not depend on how its operands came (coll/flow.cc says where it need not be rounded).  FLOW: only a data flow has such operands; in the executor, where the lone operand to scale is the
// rank's own, the test for them cost the loops of 16-bit types a tenth, also those that scale nothing (reduce of 8 x 16 MiB of bf16 in two rings 120 us, with it 133; reduce-scatter of 8 x 8 MiB averaged on the ring 211 and 218).
constexpr int kRoundedShift = 8;
template <typename T, bool FLOW, typename A> __device__ __forceinline__ A scale_operand(A v, int scaled, int s, float scale) {
  if (scaled >> s & 1) {
    v = scale_val<A>(v, scale);
    if (FLOW && (scaled >> (s + kRoundedShift) & 1)) v = Cvt<T>::up(Cvt<T>::down(v));
  }
  return v;
}

// ---------------------------------------------------------------- bounded wait
struct WaitCtx { RankCtx* ctx; unsigned long long timeout_ns; int cta, action, segment; bool one_gpu; };

// Returns false if the wait was given up (time limit or abort raised elsewhere).  `seen` (optional): the value last read.
static __device__ __noinline__ bool wait_counter(const unsigned long long* flag, unsigned long long want, const WaitCtx& w, int code, int peer, unsigned long long* seen = nullptr) {
  unsigned long long t0 = 0, have = 0;
  for (unsigned spins = 1;; spins++) {
    have = ld_acquire(flag, w.one_gpu);
    if (have >= want) { if (seen) *seen = have; return true; }
    if ((spins & 31u) == 0) {
      if (*(volatile int*)w.ctx->abort_flag) return false;
      unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > w.timeout_ns) break;
    }
  }
  // first CTA to give up records where; everybody else just leaves
  if (atomicCAS(w.ctx->abort_flag, 0, 1) == 0) {
    piccl_status_t* s = w.ctx->status;
    s->code = code; s->rank = w.ctx->rank; s->cta = w.cta; s->action = w.action; s->peer = peer; s->segment = w.segment;
    s->want = want; s->have = have;
    __threadfence_system();
    s->aborted = 1;
    __threadfence_system();
  }
  return false;
}

// ---------------------------------------------------------------- data movement
// (nt: the block's threads, from thread 0, that move data)
// value = reduce(src[0..nsrc)) -> dst[0..ndst), everything 16-byte aligned; `scaled`: see scale_operand.
// The operands' packs stay as they were loaded until they are combined, so a thread has NSRC * U loads of 16 bytes in flight and no array of
// accumulators; offsets are 32-bit (a segment is at most a slot).  Whatever U is, pack p is thread p % nt's, so a step may read what an earlier one
// wrote.  The last round is as wide as the others instead of being finished a pack at a time, which took up to U - 1 further round trips: what lies
// beyond the end loads the last pack again (loads under a condition made the compiler spill).  The slots' packs may
// have been written by another GPU and the local operand is read once: all loads go past L1.
template <typename T, int OP, bool FLOW, int NSRC, bool SCALE>
__device__ __forceinline__ uint4 combine(const uint4* v, int stride, int nsrc, int scaled, float scale) {      // v[s * stride]: operand s
  if constexpr (OP == OP_COPY) return v[0];
  else {
    typedef typename AccOf<T>::type A;
    constexpr int N = Pack<T>::N;
    if (NSRC == 1 && !SCALE) return v[0];
    A acc[N];
    Pack<T>::up(v[0], acc);
    if (SCALE) {
#pragma unroll
      for (int e = 0; e < N; e++) acc[e] = scale_operand<T, FLOW>(acc[e], scaled, 0, scale);
    }
#pragma unroll
    for (int s = 1; s < NSRC; s++) {
      if (s < nsrc) {
        A x[N]; Pack<T>::up(v[s * stride], x);
        if (SCALE) {
#pragma unroll
          for (int e = 0; e < N; e++) x[e] = scale_operand<T, FLOW>(x[e], scaled, s, scale);
        }
#pragma unroll
        for (int e = 0; e < N; e++) acc[e] = red<OP, A>(acc[e], x[e]);
      }
    }
    return Pack<T>::down(acc);
  }
}
// (Only the aligned loops take these: at odd addresses, with more than two operands, or with destinations read from the table (NDST 0), lines keep the normal priority.)
struct L2Hints { bool src_done, dst_done; int local_src, local_dst; };
// FLOW: all operands and results are the caller's (exec_flow.cuh).
template <typename T, int OP, bool FLOW, int NSRC, int NDST, int U, bool EXACT, bool SCALE = false>      // EXACT: nsrc == NSRC, else the first operand stands in for what is missing; NDST 0: any number, read from the table each time
__device__ __forceinline__ void stream(int nt, const char* const* src, int nsrc_rt, char* const* dst, int ndst, int n, int scaled, float scale, const L2Hints& h) {
  constexpr bool HINT_SRC = NSRC <= 2;                   // (more sources leave no registers for their policies)
  const int nsrc = EXACT ? NSRC : nsrc_rt, tid = threadIdx.x;
  const char* sp[NSRC]; char* dp[NDST ? NDST : 1];
#pragma unroll
  for (int s = 0; s < NSRC; s++) sp[s] = src[EXACT || s < nsrc ? s : 0];
#pragma unroll
  for (int d = 0; d < NDST; d++) dp[d] = dst[d];
  unsigned long long ps[HINT_SRC ? NSRC : 1], pd[NDST ? NDST : 1];
  const unsigned long long normal = l2_policy(false);
#pragma unroll
  for (int s = 0; s < NSRC; s++) if (HINT_SRC) ps[s] = h.src_done && (FLOW || s == h.local_src) ? l2_policy(true) : normal;
#pragma unroll
  for (int d = 0; d < NDST; d++) pd[d] = h.dst_done && (FLOW || d == h.local_dst) ? l2_policy(true) : normal;
  const unsigned long long every = FLOW && h.dst_done ? l2_policy(true) : normal;
  auto get = [&](int s, int off) { if constexpr (HINT_SRC) return ld_hint(sp[s] + off, ps[s]); else return ld_slot(sp[s] + off); };
  auto put = [&](int off, const uint4& o) {
#pragma unroll
    for (int d = 0; d < NDST; d++) st_hint(dp[d] + off, o, pd[d]);
    if (NDST == 0) {
      for (int d = 0; d < ndst; d++) if constexpr (FLOW) st_hint(dst[d] + off, o, every); else st_vec(dst[d] + off, o);
    }
  };
  int p = tid;
  for (; p + (U - 1) * nt < n; p += U * nt) {
    uint4 v[NSRC][U];
#pragma unroll
    for (int s = 0; s < NSRC; s++)
#pragma unroll
      for (int u = 0; u < U; u++) v[s][u] = get(s, (p + u * nt) * 16);
#pragma unroll
    for (int u = 0; u < U; u++) put((p + u * nt) * 16, combine<T, OP, FLOW, NSRC, SCALE>(&v[0][u], U, nsrc, scaled, scale));
  }
  if (U > 1 && p < n) {
    uint4 v[NSRC][U];
#pragma unroll
    for (int s = 0; s < NSRC; s++)
#pragma unroll
      for (int u = 0; u < U - 1; u++) v[s][u] = get(s, min(p + u * nt, n - 1) * 16);
#pragma unroll
    for (int u = 0; u < U - 1; u++) if (p + u * nt < n) put((p + u * nt) * 16, combine<T, OP, FLOW, NSRC, SCALE>(&v[0][u], U, nsrc, scaled, scale));
  }
}
template <typename T, int OP, bool FLOW>
__device__ __forceinline__ void move_aligned(int nt, const char* const* src, int nsrc, char* const* dst, int ndst, int n, int scaled, float scale, const L2Hints& h) {
  if (OP == OP_COPY || (nsrc == 1 && !scaled)) {
    if (ndst == 1) stream<T, OP, FLOW, 1, 1, 8, true>(nt, src, 1, dst, 1, n, 0, scale, h);
    else if (ndst == 2) stream<T, OP, FLOW, 1, 2, 8, true>(nt, src, 1, dst, 2, n, 0, scale, h);
    else stream<T, OP, FLOW, 1, 0, 4, true>(nt, src, 1, dst, ndst, n, 0, scale, h);
  } else if constexpr (OP != OP_COPY) {
    // Scaled operands (avg, which is a sum) have loops of their own too: in the general one a lone operand was loaded twice and the destinations read
    // from the table for each pack (25 MiB of bf16 averaged among four ranks: 155 us, now 136).
    if (scaled) {
      if constexpr (OP == 0) {
        if (nsrc == 1) {
          if (ndst == 1) stream<T, OP, FLOW, 1, 1, 8, true, true>(nt, src, 1, dst, 1, n, 1, scale, h);
          else stream<T, OP, FLOW, 1, 0, 4, true, true>(nt, src, 1, dst, ndst, n, 1, scale, h);
        }
        else if (nsrc == 2 && ndst == 1) stream<T, OP, FLOW, 2, 1, 4, true, true>(nt, src, 2, dst, 1, n, scaled, scale, h);
        else if (nsrc == 2 && ndst == 2) stream<T, OP, FLOW, 2, 2, 4, true, true>(nt, src, 2, dst, 2, n, scaled, scale, h);
        else if (nsrc <= 4) stream<T, OP, FLOW, 4, 0, 2, false, true>(nt, src, nsrc, dst, ndst, n, scaled, scale, h);
        else stream<T, OP, FLOW, kMaxActionPeers + 1, 0, 1, false, true>(nt, src, nsrc, dst, ndst, n, scaled, scale, h);
      }
    }
    else if (nsrc == 2 && ndst == 1) stream<T, OP, FLOW, 2, 1, 4, true>(nt, src, 2, dst, 1, n, 0, scale, h);
    else if (nsrc == 2 && ndst == 2) stream<T, OP, FLOW, 2, 2, 4, true>(nt, src, 2, dst, 2, n, 0, scale, h);
    else if (nsrc == 4) stream<T, OP, FLOW, 4, 0, 2, true>(nt, src, 4, dst, ndst, n, 0, scale, h);
    else if (nsrc == kMaxActionPeers + 1) stream<T, OP, FLOW, kMaxActionPeers + 1, 0, 1, true>(nt, src, nsrc, dst, ndst, n, 0, scale, h);
    else if (nsrc < 4) stream<T, OP, FLOW, 4, 0, 2, false>(nt, src, nsrc, dst, ndst, n, 0, scale, h);
    else stream<T, OP, FLOW, kMaxActionPeers + 1, 0, 1, false>(nt, src, nsrc, dst, ndst, n, 0, scale, h);
  }
}

// ---- user buffers that are not 16-byte aligned (a block of an all-gather or reduce-scatter whose length is odd, a view into a buffer)
// bytes [s, s + 16) of the 32 bytes lo, hi
__device__ __forceinline__ uint4 shift_pair(const uint4& lo, const uint4& hi, int s) {
  uint32_t e[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  if (s & 8) {
#pragma unroll
    for (int i = 0; i < 6; i++) e[i] = e[i + 2];
  }
  if (s & 4) {
#pragma unroll
    for (int i = 0; i < 5; i++) e[i] = e[i + 1];
  }
  const int b = (s & 3) * 8;
  return make_uint4(__funnelshift_r(e[0], e[1], b), __funnelshift_r(e[1], e[2], b), __funnelshift_r(e[2], e[3], b), __funnelshift_r(e[3], e[4], b));
}
// bytes [from, to) of v to p + [from, to), p 16-byte aligned
static __device__ __noinline__ void store_part(char* p, const uint4 v, int from, int to) {
  union { uint4 v; unsigned char b[16]; } u; u.v = v;
  for (int i = from; i < to; i++) reinterpret_cast<unsigned char*>(p)[i] = u.b[i];
}
// The same movement where sources or destinations are at any byte address: an unaligned source is read as the
// two aligned words around each pack, an unaligned destination is written as aligned
// words too, put together from a lane's pack and the one before it.  Only the two ends of the run of packs that a warp
// writes (2 to 8 blocks of 512 bytes) go out in bytes.  (1 MiB blocks at odd
// addresses, all-gather of four ranks: 30 us; an element at a time 171.)
// An aligned word that is read may reach up to 15 bytes beyond the operand's ends; it never leaves the 16-byte granule of a byte that
// belongs to the operand, and allocations are whole granules.
// The words of a run of packs that one warp moves: w[u] is lane's word of block u, and, for an operand that is off by m bytes, `last` the word after the run.  A pack's second
// word is the next lane's first one (of its block, or of the run), so it comes by shuffle: loaded again past L1, an operand
// costs the L2 twice its bytes (us: reduce-scatter of 8 x 2 MB of bf16 at odd addresses 119, now 104, 4 x 0.85 MB averaged 27.2 and 24.7; all-gather of 4 x 1 MiB 18.4 either way).
__device__ __forceinline__ int address_mod(const void* p) { return (int)(reinterpret_cast<uintptr_t>(p) & 15); }      // 0 for a slot
template <int RUN> struct RunWords { uint4 w[RUN], last; };
template <int RUN>
__device__ __forceinline__ void load_run(RunWords<RUN>& r, const char* src, int m, long long run, int lane, long long npack) {
  const char* const base = src - m;
  const long long top = m ? npack : npack - 1;         // beyond the end: the last word again (a load under a condition makes the compiler spill)
#pragma unroll
  for (int u = 0; u < RUN; u++) r.w[u] = ld_slot(base + min(run + u * 32 + lane, top) * 16);
  r.last = m ? ld_slot(base + min(run + RUN * 32, top) * 16) : r.w[0];
}
template <int RUN>
__device__ __forceinline__ uint4 run_pack(const RunWords<RUN>& r, int u, int m, int lane) {
  if (m == 0) return r.w[u];
  const uint4 mine = r.w[u], over = u + 1 < RUN ? r.w[u + 1 < RUN ? u + 1 : u] : r.last;
  // lane 0 offers the first word of the next block, which lane 31 needs; the others their own
  const uint4 offer = lane == 0 ? over : mine;
  const int from = (lane + 1) & 31;
  uint4 hi;
  hi.x = __shfl_sync(0xffffffffu, offer.x, from); hi.y = __shfl_sync(0xffffffffu, offer.y, from);
  hi.z = __shfl_sync(0xffffffffu, offer.z, from); hi.w = __shfl_sync(0xffffffffu, offer.w, from);
  return shift_pair(mine, hi, m);
}
// Packs o[] of a run to every destination.
template <int RUN>
__device__ __forceinline__ void store_run(const uint4 (&o)[RUN], int ndst, char* const* dst, long long run, int lane, long long npack) {
  for (int d = 0; d < ndst; d++) {
    const int dm = address_mod(dst[d]);
    if (dm == 0) {
#pragma unroll
      for (int u = 0; u < RUN; u++) { const long long p = run + u * 32 + lane; if (p < npack) st_vec(dst[d] + p * 16, o[u]); }
      continue;
    }
#pragma unroll
    for (int u = 0; u < RUN; u++) {
      const long long p = run + u * 32 + lane;
      // the pack before: lane 31 offers the block's before, which lane 0 needs
      const uint4 offer = lane == 31 && u > 0 ? o[u > 0 ? u - 1 : 0] : o[u];
      const int from = (lane + 31) & 31;
      uint4 prev;
      prev.x = __shfl_sync(0xffffffffu, offer.x, from); prev.y = __shfl_sync(0xffffffffu, offer.y, from);
      prev.z = __shfl_sync(0xffffffffu, offer.z, from); prev.w = __shfl_sync(0xffffffffu, offer.w, from);
      if (p < npack) {
        char* const w = dst[d] + p * 16 - dm;        // aligned word: the last dm bytes of the pack before, then this pack's first 16 - dm
        const uint4 v = shift_pair(prev, o[u], 16 - dm);
        if (u == 0 && lane == 0) store_part(w, v, dm, 16);
        else st_vec(w, v);
        if (p == npack - 1 || (u == RUN - 1 && lane == 31)) store_part(w + 16, shift_pair(o[u], o[u], 16 - dm), 0, dm);
      }
    }
  }
}
template <typename T, int OP, int RUN>
__device__ __noinline__ void copy_shift(int nt, const char* src, int ndst, char* const* dst, long long npack) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = nt >> 5;
  char* one[1] = {dst[0]};
  if (ndst == 1 && address_mod(dst[0])) {                               // (a shift for the source and one for the destination: all-gather of 4 x 1 MiB 20.5 us)  One destination: its whole words, for which one shift will do, and the bytes at both ends
    const int head = 16 - address_mod(dst[0]);
    if (warp == nwarp - 1 && lane < 16) {
      const long long at = lane < head ? lane : npack * 16 - 16 + lane;      // (the last bytes are the words' remainder)
      one[0][at] = *reinterpret_cast<const volatile char*>(src + at);
    }
    src += head; one[0] += head; npack -= 1; dst = one;
  }
  const int m = address_mod(src);
  for (long long run = (long long)warp * (32 * RUN); run < npack; run += (long long)nwarp * (32 * RUN)) {
    RunWords<RUN> r;
    load_run(r, src, m, run, lane, npack);
    uint4 o[RUN];
#pragma unroll
    for (int u = 0; u < RUN; u++) o[u] = run_pack(r, u, m, lane);
    store_run<RUN>(o, ndst, dst, run, lane, npack);
  }
}
template <typename T, int OP, bool FLOW, int RUN>
__device__ __noinline__ void reduce_shift(int nt, int nsrc, const char* const* src, int ndst, char* const* dst, long long npack, int scaled, float scale) {
  typedef typename AccOf<T>::type A;
  constexpr int N = Pack<T>::N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = nt >> 5;
  for (long long run = (long long)warp * (32 * RUN); run < npack; run += (long long)nwarp * (32 * RUN)) {
    A acc[RUN][N];
    auto operand = [&](const RunWords<RUN>& r, int u, int s, int m, A (&x)[N]) {
      Pack<T>::up(run_pack(r, u, m, lane), x);
      if (scaled >> s & 1) {
#pragma unroll
        for (int e = 0; e < N; e++) x[e] = scale_operand<T, FLOW>(x[e], scaled, s, scale);
      }
    };
    {                                                // two operands' loads in flight, beside no accumulators yet
      const int second = min(1, nsrc - 1), m = address_mod(src[0]), m2 = address_mod(src[second]);
      RunWords<RUN> r, r2;
      load_run(r, src[0], m, run, lane, npack);
      load_run(r2, src[second], m2, run, lane, npack);
#pragma unroll
      for (int u = 0; u < RUN; u++) {
        operand(r, u, 0, m, acc[u]);
        if (nsrc > 1) {
          A x[N]; operand(r2, u, 1, m2, x);
#pragma unroll
          for (int e = 0; e < N; e++) acc[u][e] = red<OP, A>(acc[u][e], x[e]);
        }
      }
    }
#pragma unroll 1
    for (int s = 2; s < nsrc; s++) {
      const int m = address_mod(src[s]);
      RunWords<RUN> r;
      load_run(r, src[s], m, run, lane, npack);
#pragma unroll
      for (int u = 0; u < RUN; u++) {
        A x[N]; operand(r, u, s, m, x);
#pragma unroll
        for (int e = 0; e < N; e++) acc[u][e] = red<OP, A>(acc[u][e], x[e]);
      }
    }
    uint4 o[RUN];
#pragma unroll
    for (int u = 0; u < RUN; u++) o[u] = Pack<T>::down(acc[u]);
    store_run<RUN>(o, ndst, dst, run, lane, npack);
  }
}
// A warp takes runs of 2, 4 or 8 blocks (sums: 2 or 4): as few rounds as can be, and then over as many warps.
template <typename T, int OP, bool FLOW>
__device__ __forceinline__ void reduce_copy_shift(int nt, int nsrc, const char* const* src, int ndst, char* const* dst, long long npack, int scaled, float scale) {
  const long long blocks = (npack + nt - 1) / nt;      // per warp
  if (OP == OP_COPY || (nsrc == 1 && !scaled)) {
    if (blocks > 4) copy_shift<T, OP, 8>(nt, src[0], ndst, dst, npack);
    else if (blocks > 2) copy_shift<T, OP, 4>(nt, src[0], ndst, dst, npack);
    else copy_shift<T, OP, 2>(nt, src[0], ndst, dst, npack);
  } else if constexpr (OP != OP_COPY) {
    if (blocks > 2) reduce_shift<T, OP, FLOW, 4>(nt, nsrc, src, ndst, dst, npack, scaled, scale);
    else reduce_shift<T, OP, FLOW, 2>(nt, nsrc, src, ndst, dst, npack, scaled, scale);
  }
}

// Element-wise path: the last, partial pack of an action, an operand after the other.  (A data flow's has all operands on their way first, exec_flow.cuh.  In this kernel that form, which needs a register
// for each operand, makes the loops above slower although it hardly ever runs: reduce of 8 x 16 MiB in two rings 111 us, with it 123, in rings of four 101 and 110; 8 x 52 MiB of fp64 averaged by DIRECT 267 and 292.
// With bytes it is the other way round: maximum of 8 x 4 MiB on the ring 73.7, with it 69.9.)
template <typename T, int OP>
__device__ __noinline__ void reduce_copy_elem(int nt, int nsrc, const char* const* src, int local_src, int ndst, char* const* dst,
                                                 long long first, long long nelem, bool do_scale, float scale) {
  typedef typename AccOf<T>::type A;
  for (long long i = first + threadIdx.x; i < nelem; i += nt) {
    auto load = [&](int s) { const T* const p = reinterpret_cast<const T*>(src[s]) + i; return local_src == s ? *p : *reinterpret_cast<const volatile T*>(p); };
    A acc = A();
    if constexpr (sizeof(T) == 1) {
      T raw[kMaxActionPeers + 1];
#pragma unroll
      for (int s = 0; s < kMaxActionPeers + 1; s++) if (s < nsrc) raw[s] = load(s);
#pragma unroll
      for (int s = 0; s < kMaxActionPeers + 1; s++) if (s < nsrc) { const A x = Cvt<T>::up(raw[s]); acc = s == 0 ? x : red<OP, A>(acc, x); }
    } else {
      for (int s = 0; s < nsrc; s++) {
        A x = Cvt<T>::up(load(s));
        if (do_scale && local_src == s) x = scale_val<A>(x, scale);
        acc = s == 0 ? x : red<OP, A>(acc, x);
      }
    }
    const T o = Cvt<T>::down(acc);
    for (int d = 0; d < ndst; d++) reinterpret_cast<T*>(dst[d])[i] = o;
  }
}

// ---------------------------------------------------------------- the kernel
constexpr int kSliceCache = 192;      // actions kept in shared memory, with the CTA's slice of each

constexpr int kStepDepth = 4;         // steps the waiter may be ahead of the publisher
struct StepDesc {
  const char* src[kMaxActionPeers + 1];      // operands in rank order: receive peers below me, my own buffer, receive peers above me
  char* dst[kMaxActionPeers + 1];            // local destination first, then the send peers
  long long len;                             // elements
  int action, nsrc, ndst, local_src, local_dst, flags;
};
enum : int { STEP_SCALE = 1, STEP_ALIGNED = 2, STEP_LOCAL_DEP = 4, STEP_FAIL = 8, STEP_END = 16, STEP_SRC_DONE = 32, STEP_DST_DONE = 64 };
__device__ __forceinline__ void bar_sync_n(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive_n(int id, int n) { __threadfence_block(); asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// SHIFT = true: for calls with operands that are not 16-byte aligned (a kernel of its own: the mere presence of that path cost the aligned one
// 15 % in registers).
template <typename T, int OP, bool SHIFT>
__global__ void __launch_bounds__(kMaxBlock + kCtlThreads, 1) exec_kernel(const KernelArgs ka) {
  const int vr = blockIdx.x / ka.n_cta, cta = blockIdx.x % ka.n_cta;
  const LaunchRank& L = ka.r[vr];
  RankCtx* __restrict__ ctx = L.ctx;
  const int tid = threadIdx.x, lane = tid & 31, ndata = (int)blockDim.x - kCtlThreads;
  constexpr int esz = (int)sizeof(T);

  __shared__ StepDesc s_step[kStepDepth];
  __shared__ char* s_heap[kMaxRanks];
  __shared__ long long s_lo[kSliceCache], s_hi[kSliceCache];
  __shared__ Action s_act[kSliceCache];
  __shared__ int s_maxseg;
  __shared__ volatile int s_published;             // steps whose descriptor may be used again

  // everything read from the context more than once is fetched once, in parallel
  const int rank = ctx->rank, nranks = ctx->nranks, max_cta = ctx->max_cta;
  const long long tail_off = ctx->tail_off, head_off = ctx->head_off, fifo_off = ctx->fifo_off, scratch_off = ctx->scratch_off, chan_bytes = ctx->nslot * ctx->slot_bytes;
  if (tid < nranks) s_heap[tid] = ctx->heap[tid];
  if (tid == 0) { s_maxseg = 0; s_published = 0; }
  __syncthreads();
  const long long seg_bytes = ka.seg_bytes, seg_elems = (seg_bytes / 16) * (esz >= 16 ? 1 : 16 / esz);
  {
    int m = 0;
    for (int ai = tid; ai < L.n_actions; ai += blockDim.x) {
      const Action a = L.actions[ai];
      const Slice sl = slice_of(a.count, esz, cta, ka.n_cta, seg_bytes);
      if (ai < kSliceCache) { s_lo[ai] = sl.lo; s_hi[ai] = sl.hi; s_act[ai] = a; }
      m = max(m, sl.nseg);
    }
    if (m) atomicMax(&s_maxseg, m);
  }
  __syncthreads();
  const int maxseg = s_maxseg;
  char* const my_heap = s_heap[rank];
  // barriers: 1 .. kStepDepth a step's descriptor is ready (waiter arrives, data warps wait), then as many for its data being moved (data warps
  // arrive, publisher waits), then one among the data warps
  constexpr int kReady = 1, kDone = 1 + kStepDepth, kData = 1 + 2 * kStepDepth;

  if (tid < ndata) {                               // ---------------- data warps
    for (int k = 0;; k++) {
      const int d = k % kStepDepth;
      bar_sync_n(kReady + d, ndata + 32);
      const StepDesc& st = s_step[d];
      const int flags = st.flags;
      if (!(flags & (STEP_END | STEP_FAIL))) {
        // an operand that earlier steps wrote: its elements were written by the threads that read them now, or by their warp; the barrier makes it plain
        if (flags & STEP_LOCAL_DEP) bar_sync_n(kData, ndata);
        const char* const* const src = st.src; char* const* const dst = st.dst;
        const long long len = st.len;
        const int nsrc = st.nsrc, ndst = st.ndst, local_src = st.local_src;
        const bool do_scale = flags & STEP_SCALE;
        constexpr int N = Pack<T>::N;
        const long long nfull = (SHIFT || (flags & STEP_ALIGNED)) ? len / N : 0;
        if constexpr (SHIFT) { if (nfull && ndst) reduce_copy_shift<T, OP, false>(ndata, nsrc, src, ndst, dst, nfull, do_scale ? 1 << local_src : 0, ka.scale); }
        else if (nfull) move_aligned<T, OP, false>(ndata, src, nsrc, dst, ndst, (int)nfull, do_scale ? 1 << local_src : 0, ka.scale, L2Hints{(flags & STEP_SRC_DONE) != 0, (flags & STEP_DST_DONE) != 0, local_src, st.local_dst});
        if (nfull * N < len) reduce_copy_elem<T, OP>(ndata, nsrc, src, local_src, ndst, dst, nfull * N, len, do_scale, ka.scale);
      }
      bar_arrive_n(kDone + d, ndata + 32);
      if (flags & (STEP_END | STEP_FAIL)) return;
    }
  }

  // waiter and publisher: lane l has the connections with peers l and l + 32, and counts their entries on its own
  unsigned long long sent[2] = {0, 0}, rcvd[2] = {0, 0};
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int p = lane + 32 * q;
    if (p < nranks) { sent[q] = ctx->sent[p * max_cta + cta]; rcvd[q] = ctx->rcvd[p * max_cta + cta]; }
  }
  const unsigned nslot = (unsigned)ka.nslot;
  const long long mine = (long long)(rank * max_cta + cta) * kFlagStride;      // my counters in a peer's heap

  if (tid < ndata + 32) {                          // ---------------- waiter
    WaitCtx w; w.ctx = ctx; w.timeout_ns = ka.timeout_ns; w.cta = cta; w.one_gpu = ka.one_gpu;
    unsigned long long seen_head[2] = {0, 0};      // what a peer had consumed when last looked: no need to look again while that is credit enough
    int k = 0;
    bool failed = false;
    // the descriptor of step k - kStepDepth has served; the publisher waits for nobody but the data warps, which wait for nothing beyond this warp
    auto free_desc = [&]() {
      unsigned long long t0 = 0;
      for (unsigned spins = 1; s_published < k - kStepDepth + 1; spins++) {
        if ((spins & 1023u) == 0) {
          const unsigned long long now = globaltimer_ns();
          if (t0 == 0) t0 = now;
          else if (now - t0 > ka.timeout_ns) { *(volatile int*)ctx->abort_flag = 1; return; }
        }
      }
      __threadfence_block();
    };
    for (int seg0 = 0; seg0 < maxseg && !failed; seg0 += ka.window) {
      for (int ai = 0; ai < L.n_actions && !failed; ai++) {
        const Action& ac = ai < kSliceCache ? s_act[ai] : L.actions[ai];
        long long sl_lo, sl_hi;
        if (ai < kSliceCache) { sl_lo = s_lo[ai]; sl_hi = s_hi[ai]; }
        else { const Slice sl = slice_of(ac.count, esz, cta, ka.n_cta, seg_bytes); sl_lo = sl.lo; sl_hi = sl.hi; }
        const bool has_src = ac.src_buf != BUF_NONE, has_dst = ac.dst_buf != BUF_NONE;
        for (int seg = seg0; seg < seg0 + ka.window; seg++) {
          const long long lo = sl_lo + (long long)seg * seg_elems;
          if (lo >= sl_hi) break;
          free_desc();
          StepDesc& st = s_step[k % kStepDepth];
          bool ok = true;
          w.action = ai; w.segment = seg;
#pragma unroll
          for (int q = 0; q < 2; q++) {
            const int p = lane + 32 * q;
            const long long theirs = (long long)(p * max_cta + cta) * kFlagStride;      // peer p's counters in my heap
            for (int j = 0; j < ac.n_send; j++) if (ac.send_peer[j] == p) {
              st.dst[j + has_dst] = s_heap[p] + fifo_off + (long long)(rank * max_cta + cta) * chan_bytes + (long long)(sent[q] % nslot) * seg_bytes;
              if (++sent[q] > seen_head[q] + nslot && ok)
                ok = wait_counter(reinterpret_cast<const unsigned long long*>(my_heap + head_off + theirs), sent[q] - nslot, w, 1, p, &seen_head[q]);
            }
            for (int j = 0; j < ac.n_recv; j++) if (ac.recv_peer[j] == p) {
              st.src[j + (has_src && j >= ac.self_pos)] = my_heap + fifo_off + (long long)(p * max_cta + cta) * chan_bytes + (long long)(rcvd[q] % nslot) * seg_bytes;
              ++rcvd[q];
              if (ok) ok = wait_counter(reinterpret_cast<const unsigned long long*>(my_heap + tail_off + theirs), rcvd[q], w, 2, p);
            }
          }
          ok = __all_sync(0xffffffffu, ok);
          if (lane == 0) {
            const char* lsrc = nullptr; char* ldst = nullptr;
            if (has_src) { lsrc = (ac.src_buf == BUF_IN ? (const char*)L.in : ac.src_buf == BUF_OUT ? (const char*)L.out : my_heap + scratch_off) + (ac.src_off + lo) * esz; st.src[ac.self_pos] = lsrc; }
            if (has_dst) { ldst = (ac.dst_buf == BUF_OUT ? (char*)L.out : my_heap + scratch_off) + (ac.dst_off + lo) * esz; st.dst[0] = ldst; }
            st.len = (lo + seg_elems < sl_hi ? lo + seg_elems : sl_hi) - lo;
            st.action = ai; st.nsrc = ac.n_recv + has_src; st.ndst = ac.n_send + has_dst; st.local_src = has_src ? ac.self_pos : -1; st.local_dst = has_dst ? 0 : -1;
            st.flags = (ka.avg && (ac.flags & ACT_SCALE_SRC) && has_src ? STEP_SCALE : 0) | (((reinterpret_cast<uintptr_t>(lsrc) | reinterpret_cast<uintptr_t>(ldst)) & 15) == 0 ? STEP_ALIGNED : 0) |
                       (has_src && ac.src_buf != BUF_IN ? STEP_LOCAL_DEP : 0) | ((ka.leave_first & 1) && (ac.flags & ACT_SRC_DONE) ? STEP_SRC_DONE : 0) | ((ka.leave_first & 2) && (ac.flags & ACT_DST_DONE) ? STEP_DST_DONE : 0) | (ok ? 0 : STEP_FAIL);
          }
          __syncwarp();
          bar_arrive_n(kReady + k % kStepDepth, ndata + 32);
          k++;
          if (!ok) { failed = true; break; }
        }
        if (failed) break;
      }
    }
    if (!failed) {
      free_desc();
      if (lane == 0) s_step[k % kStepDepth].flags = STEP_END;
      __syncwarp();
      bar_arrive_n(kReady + k % kStepDepth, ndata + 32);
    }
    return;
  }

  for (int k = 0;; k++) {                          // ---------------- publisher: the data to the consumers, the freed slots to the producers
    const int d = k % kStepDepth;
    bar_sync_n(kDone + d, ndata + 32);
    const int flags = s_step[d].flags, ai = s_step[d].action;
    if (flags & (STEP_END | STEP_FAIL)) break;
    const Action& ac = ai < kSliceCache ? s_act[ai] : L.actions[ai];
    // One fence for both: what the data warps stored comes before the consumers' counters, what they read before the producers'.  It waits for the
    // acknowledgement of everything the CTA stored, so a credit costs up to a microsecond at the end of a call: 1 MiB blocks of an all-gather, with system scope, 31.6 us, 29.9
    // with plain stores for the heads, which nothing orders behind the reads.  A release per counter took 38.0, a warp of its own for the heads 32.5.  (With GPU scope the call takes 28.7; the others were not timed again.)
    fence_ranks(ka.one_gpu);
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int p = lane + 32 * q;
      for (int j = 0; j < ac.n_send; j++) if (ac.send_peer[j] == p) st_relaxed(reinterpret_cast<unsigned long long*>(s_heap[p] + tail_off + mine), ++sent[q], ka.one_gpu);
      for (int j = 0; j < ac.n_recv; j++) if (ac.recv_peer[j] == p) st_relaxed(reinterpret_cast<unsigned long long*>(s_heap[p] + head_off + mine), ++rcvd[q], ka.one_gpu);
    }
    __syncwarp();
    if (lane == 0) { __threadfence_block(); s_published = k + 1; }
  }
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int p = lane + 32 * q;
    if (p < nranks) { ctx->sent[p * max_cta + cta] = sent[q]; ctx->rcvd[p * max_cta + cta] = rcvd[q]; }
  }
}

}  // namespace piccl

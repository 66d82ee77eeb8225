// Low-latency variant of the fused executor for small messages of ANY collective
// and algorithm: the same action programs, but FIFO entries are 16-byte lines of
// {4 B data, 4 B sequence, 4 B data, 4 B sequence} in a separate small FIFO.  A line
// is complete when both sequence words equal the entry's number, so the producer
// needs neither a fence nor a tail counter and the consumer polls the data itself.
// Slot reuse is guarded by a head counter the consumer advances with a plain
// store once its reads are done (the producer only looks at it when the ring of
// kLLFifoSlots entries is about to wrap).  Entry numbers never repeat for a slot,
// and the region is zero at start, so stale lines can never look complete.
#pragma once
#include "exec_impl.cuh"
#include "exec_flow.cuh"

namespace piccl {

template <typename T> struct LLUnit {
  static constexpr int E = 8 / sizeof(T);
  union U { uint2 v; T t[E]; };
};

template <typename T, int OP>
__global__ void __launch_bounds__(kLLBlock) exec_ll_kernel(const KernelArgs ka) {
  typedef typename AccOf<T>::type A;
  constexpr int E = LLUnit<T>::E;
  constexpr int esz = (int)sizeof(T);
  const int vr = blockIdx.x / ka.n_cta, cta = blockIdx.x % ka.n_cta;
  const LaunchRank& L = ka.r[vr];
  RankCtx* __restrict__ ctx = L.ctx;
  const int tid = threadIdx.x;

  __shared__ unsigned s_send[2][kMaxRanks], s_recv[2][kMaxRanks];      // entry numbers of an action, by the action's parity
  __shared__ int s_credit[2];                                          // an action has to look for credit before it sends
  __shared__ long long s_lo[kSliceCache], s_hi[kSliceCache];
  __shared__ char* s_heap[kMaxRanks];
  __shared__ Action s_act[kSliceCache];
  __shared__ int s_maxseg;

  const int rank = ctx->rank, nranks = ctx->nranks;
  const long long llf_off = ctx->llf_off, llf_head_off = ctx->llf_head_off, scratch_off = ctx->scratch_off;
  unsigned long long my_sent = 0, my_rcvd = 0, seen_head = 0;      // seen_head: what peer `tid` had consumed when last looked
  if (tid < nranks) { s_heap[tid] = ctx->heap[tid]; my_sent = ctx->sent_ll[tid * kLLFifoCta + cta]; my_rcvd = ctx->rcvd_ll[tid * kLLFifoCta + cta]; }
  if (tid == 0) { s_maxseg = 0; s_credit[0] = s_credit[1] = 0; }
  __syncthreads();
  constexpr long long kPayload = kLLFifoSlotBytes / 2;
  const long long seg_elems = (kPayload / 16) * (16 / esz);
  if (tid < nranks) seen_head = ld_acquire(reinterpret_cast<const unsigned long long*>(s_heap[rank] + llf_head_off + (long long)(tid * kLLFifoCta + cta) * kFlagStride), ka.one_gpu);
  {
    // From the last thread down: the first ones wait for the line above, behind which an acquiring thread's loads queue (us: reduce-scatter of 4 KiB between two ranks 7.8, now 6.2, broadcast
    // of 2 KB among three on the ring 8.2 and 6.2, reduce of 32 KiB among four 7.9 and 6.2).
    int m = 0;
    for (int ai = (int)blockDim.x - 1 - tid; ai < L.n_actions; ai += blockDim.x) {
      const Action a = L.actions[ai];
      const Slice sl = slice_of(a.count, esz, cta, ka.n_cta, kPayload);
      if (ai < kSliceCache) { s_act[ai] = a; s_lo[ai] = sl.lo; s_hi[ai] = sl.hi; }
      m = max(m, sl.nseg);
    }
    if (m) atomicMax(&s_maxseg, m);
  }
  __syncthreads();
  const int maxseg = s_maxseg;
  char* const my_heap = s_heap[rank];
  WaitCtx w; w.ctx = ctx; w.timeout_ns = ka.timeout_ns; w.cta = cta; w.one_gpu = ka.one_gpu;
  unsigned long long rcvd_done = 0;
  bool failed = false, freed = false;                  // freed: entries from peer `tid` are read, and the peer does not know yet
  unsigned long long t0 = 0;
  int step = 0;
  // The slots of what was read (its data went through registers) are the producer's again: a plain store.
  auto free_slots = [&]() {
    if (freed) *reinterpret_cast<volatile unsigned long long*>(s_heap[tid] + llf_head_off + (long long)(rank * kLLFifoCta + cta) * kFlagStride) = rcvd_done;
    freed = false;
  };

  // One barrier to an action: behind it all threads are done with the action before, whose slots are given back then, beside this action's polling.  (With a second one after the
  // data, slices worked out anew and the heads read for every entry, all through the slots: all-reduce of 4 KiB on the ring, eight ranks, 38.9 us, now 28.5, of 16 KiB among four 19.4
  // and 14.4; all-gather of 16 KiB by PRM, eight ranks, 30.3 and 22.6; reduce-scatter of 8 KiB, four ranks, 12.4 and 10.8.)  What is left is a line's way through the L2 and the poll that sees it.
  bool over = false;                                   // given up, by all threads
  for (int seg = 0; seg < maxseg && !over; seg++) {
    for (int ai = 0; ai < L.n_actions; ai++) {
      const Action& ac = ai < kSliceCache ? s_act[ai] : L.actions[ai];
      long long sl_lo, sl_hi;
      if (ai < kSliceCache) { sl_lo = s_lo[ai]; sl_hi = s_hi[ai]; }
      else { const Slice sl = slice_of(ac.count, esz, cta, ka.n_cta, kPayload); sl_lo = sl.lo; sl_hi = sl.hi; }
      const long long lo = sl_lo + (long long)seg * seg_elems;
      if (lo >= sl_hi) continue;
      const long long hi = (lo + seg_elems < sl_hi) ? lo + seg_elems : sl_hi;
      const long long len = hi - lo;
      const int par = step++ & 1;
      const unsigned* const s_send_seq = s_send[par];
      const unsigned* const s_recv_seq = s_recv[par];

      bool sends = false;
      if (tid < nranks) {
        for (int j = 0; j < ac.n_send; j++) if (ac.send_peer[j] == tid) {
          s_send[par][tid] = (unsigned)++my_sent;
          sends = true;
          if (my_sent > seen_head + (unsigned long long)kLLFifoSlots) s_credit[par] = 1;
        }
        for (int j = 0; j < ac.n_recv; j++) if (ac.recv_peer[j] == tid) s_recv[par][tid] = (unsigned)++my_rcvd;
      }
      if (__syncthreads_or(failed)) { failed = over = true; break; }
      if (tid < nranks) {
        free_slots();
        for (int j = 0; j < ac.n_recv; j++) if (ac.recv_peer[j] == tid) { rcvd_done = my_rcvd; freed = true; }
      }
      if (s_credit[par]) {                             // (after the slots above are free: two ranks may wait for each other's)
        if (sends && my_sent > seen_head + (unsigned long long)kLLFifoSlots) {
          w.action = ai; w.segment = seg;
          failed = !wait_counter(reinterpret_cast<const unsigned long long*>(my_heap + llf_head_off + (long long)(tid * kLLFifoCta + cta) * kFlagStride), my_sent - kLLFifoSlots, w, 1, tid, &seen_head);
        }
        if (__syncthreads_or(failed)) { failed = over = true; break; }
        if (tid == 0) s_credit[par] = 0;               // (set again two actions on, behind the next action's barrier)
      }

      const bool has_src = ac.src_buf != BUF_NONE;
      const T* lsrc = nullptr; T* ldst = nullptr;
      if (has_src) lsrc = reinterpret_cast<const T*>(ac.src_buf == BUF_IN ? (const char*)L.in : ac.src_buf == BUF_OUT ? (const char*)L.out : my_heap + scratch_off) + ac.src_off + lo;
      if (ac.dst_buf != BUF_NONE) ldst = reinterpret_cast<T*>(ac.dst_buf == BUF_OUT ? (char*)L.out : my_heap + scratch_off) + ac.dst_off + lo;
      const int do_scale = ka.avg && (ac.flags & ACT_SCALE_SRC) && has_src ? 1 : 0;
      const long long nunits = (len + E - 1) / E;
      // a unit of a buffer, in one load where it is whole and stands at a multiple of its size
      auto load_unit = [&](const T* from, long long u, bool whole, int scaled, A (&v)[E]) {
        typename LLUnit<T>::U un;
        if (whole && u * E + E <= len) un.v = *reinterpret_cast<const uint2*>(from + u * E);
        else {
          un.v = make_uint2(0, 0);
#pragma unroll
          for (int e = 0; e < E; e++) if (u * E + e < len) un.t[e] = from[u * E + e];
        }
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = scale_operand<T, false>(Cvt<T>::up(un.t[e]), scaled, 0, ka.scale);
      };
      const bool src_whole = (reinterpret_cast<uintptr_t>(lsrc) & 7) == 0, dst_whole = (reinterpret_cast<uintptr_t>(ldst) & 7) == 0;

      for (long long u = tid; u < nunits && !failed; u += blockDim.x) {
        A acc[E], mine[E];
        bool have = false;
        if (has_src) load_unit(lsrc, u, src_whole, do_scale, mine);      // on its way while the lines come
        for (int j = 0; j <= ac.n_recv; j++) {
          if (j == ac.self_pos && has_src) {
#pragma unroll
            for (int e = 0; e < E; e++) acc[e] = have ? red<OP, A>(acc[e], mine[e]) : mine[e];
            have = true;
          }
          if (j == ac.n_recv) break;
          const int p = ac.recv_peer[j];
          const unsigned seq = s_recv_seq[p];
          const char* src = my_heap + llf_off + ((long long)(p * kLLFifoCta + cta) * kLLFifoSlots + (seq - 1) % kLLFifoSlots) * kLLFifoSlotBytes + u * 16;
          uint4 line;
          for (unsigned spins = 1;; spins++) {
            line = ld_slot(src);
            if (line.y == seq && line.w == seq) break;
            if ((spins & 63u) == 0) {
              if (*(volatile int*)ctx->abort_flag) { failed = true; break; }
              unsigned long long now = globaltimer_ns();
              if (!t0) t0 = now;
              else if (now - t0 > ka.timeout_ns) {
                if (atomicCAS(ctx->abort_flag, 0, 1) == 0) {
                  piccl_status_t* st = ctx->status;
                  st->code = 2; st->rank = rank; st->cta = cta; st->action = ai; st->peer = p; st->segment = seg; st->want = seq; st->have = line.y;
                  __threadfence_system(); st->aborted = 1; __threadfence_system();
                }
                failed = true; break;
              }
            }
          }
          if (failed) break;
          typename LLUnit<T>::U un; un.v = make_uint2(line.x, line.z);
#pragma unroll
          for (int e = 0; e < E; e++) { A x = Cvt<T>::up(un.t[e]); acc[e] = have ? red<OP, A>(acc[e], x) : x; }
          have = true;
        }
        if (failed) break;
        typename LLUnit<T>::U out;
#pragma unroll
        for (int e = 0; e < E; e++) out.t[e] = Cvt<T>::down(acc[e]);
        for (int j = 0; j < ac.n_send; j++) {
          const int p = ac.send_peer[j];
          const unsigned seq = s_send_seq[p];
          char* dst = s_heap[p] + llf_off + ((long long)(rank * kLLFifoCta + cta) * kLLFifoSlots + (seq - 1) % kLLFifoSlots) * kLLFifoSlotBytes + u * 16;
          asm volatile("st.volatile.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(dst), "r"(out.v.x), "r"(seq), "r"(out.v.y), "r"(seq) : "memory");
        }
        if (ldst && dst_whole && u * E + E <= len) *reinterpret_cast<uint2*>(ldst + u * E) = out.v;
        else if (ldst) {
#pragma unroll
          for (int e = 0; e < E; e++) { const long long idx = u * E + e; if (idx < len) ldst[idx] = out.t[e]; }
        }
      }
    }
    // (a thread that failed goes on to the next barrier, which tells the others)
  }
  if (!__syncthreads_or(failed) && tid < nranks) free_slots();
  if (tid < nranks) { ctx->sent_ll[tid * kLLFifoCta + cta] = my_sent; ctx->rcvd_ll[tid * kLLFifoCta + cta] = my_rcvd; }
}

}  // namespace piccl

#define PICCL_INSTANTIATE_EXEC(T, DT)                                                              \
  namespace piccl {                                                                                \
  ExecKernelFn exec_table_##DT[4] = {exec_kernel<T, 0, false>, exec_kernel<T, 1, false>, exec_kernel<T, 2, false>, exec_kernel<T, 3, false>}; \
  ExecKernelFn exec_shift_table_##DT[4] = {exec_kernel<T, 0, true>, exec_kernel<T, 1, true>, exec_kernel<T, 2, true>, exec_kernel<T, 3, true>}; \
  FlowKernelFn exec_flow_table_##DT[8] = {exec_flow_kernel<T, 0, false>, exec_flow_kernel<T, 1, false>, exec_flow_kernel<T, 2, false>, exec_flow_kernel<T, 3, false>,              \
                                          exec_flow_kernel<T, 0, true>, exec_flow_kernel<T, 1, true>, exec_flow_kernel<T, 2, true>, exec_flow_kernel<T, 3, true>};               \
  ExecKernelFn exec_ll_table_##DT[4] = {exec_ll_kernel<T, 0>, exec_ll_kernel<T, 1>, exec_ll_kernel<T, 2>, exec_ll_kernel<T, 3>}; \
  }

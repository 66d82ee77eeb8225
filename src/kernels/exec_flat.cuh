// Calls in which no action waits for another: every operand stands in a buffer that nobody writes during the call (share.cc), as in each all-gather and
// broadcast, and in the reductions that are one exchange.  Such a call needs neither counters nor all its CTAs at the same time, so it is an ordinary grid of small
// blocks, one slice of one action of one rank each, as many to an SM as there are registers for, and is launched while the kernel before it ends.
// Blocks of the same slice of all actions are neighbours: an operand that several ranks read comes from memory once.
// Bound by memory for large messages, by the launch for small ones.  Figures at flat_slices (comm.cu).
#pragma once
#include "exec_impl.cuh"

namespace piccl {

template <typename T, int OP, bool SHIFT>
__global__ void __launch_bounds__(kFlatBlock, 3) exec_flat_kernel(const KernelArgs ka) {
  constexpr int esz = (int)sizeof(T), N = Pack<T>::N;
  __shared__ const char* s_src[kMaxActionPeers + 1];
  __shared__ char* s_dst[1];
  int total = 0;
  for (int r = 0; r < ka.n_vrank; r++) total += ka.r[r].n_actions;
  if (total == 0) return;
  int ai = blockIdx.x % total, rank = 0;
  const int slice = blockIdx.x / total;
  while (ai >= ka.r[rank].n_actions) ai -= ka.r[rank++].n_actions;
  const LaunchRank& L = ka.r[rank];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const Action ac = L.actions[ai];
  const SharedOps* const x = L.shared + ai;
  const Slice sl = slice_of(ac.count, esz, slice, ka.n_cta, ka.seg_bytes);
  if (sl.lo >= sl.hi) return;
  const bool has_src = ac.src_buf != BUF_NONE;
  if (threadIdx.x <= ac.n_recv) {
    const int j = threadIdx.x;                         // receive operand j, or the rank's own
    if (j < ac.n_recv) s_src[j + (has_src && j >= ac.self_pos)] = (x->buf[j] == BUF_IN ? (const char*)ka.r[x->from[j]].in : (const char*)ka.r[x->from[j]].out) + (x->off[j] + sl.lo) * esz;
    else {
      if (has_src) s_src[ac.self_pos] = (ac.src_buf == BUF_IN ? (const char*)L.in : (const char*)L.out) + (ac.src_off + sl.lo) * esz;
      s_dst[0] = (char*)L.out + (ac.dst_off + sl.lo) * esz;
    }
  }
  __syncthreads();
  const int nsrc = ac.n_recv + has_src;
  int scaled = 0;
  if (ka.avg) {
    for (int j = 0; j < ac.n_recv; j++) if (x->scaled >> j & 1) scaled |= (x->from[j] == rank ? 1 : 1 | 1 << kRoundedShift) << (j + (has_src && j >= ac.self_pos));
    if (has_src && (ac.flags & ACT_SCALE_SRC)) scaled |= 1 << ac.self_pos;
  }
  const long long len = sl.hi - sl.lo, nfull = len / N;
  const int local_src = has_src ? ac.self_pos : -1;
  if constexpr (SHIFT) { if (nfull) reduce_copy_shift<T, OP>(kFlatBlock, nsrc, s_src, 1, s_dst, 0, nfull, scaled, ka.scale); }
  else if (nfull) move_aligned<T, OP>(kFlatBlock, s_src, nsrc, s_dst, 1, (int)nfull, scaled, ka.scale, L2Hints{(ka.leave_first & 1) && (ac.flags & ACT_SRC_DONE), (ka.leave_first & 2) && (ac.flags & ACT_DST_DONE), local_src, 0});
  if (nfull * N < len) reduce_copy_elem<T, OP>(kFlatBlock, nsrc, s_src, local_src, 1, s_dst, nfull * N, len, scaled, ka.scale);
}

}  // namespace piccl

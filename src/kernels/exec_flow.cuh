// Launches that carry all ranks on one GPU, from what the call computes (coll/flow.cc): each operation reads elements of the ranks' send buffers, folds them as the ranks' programs would, and
// stores the result in every receive buffer that takes it.  Nothing waits, so this needs neither counters nor all blocks at the same time: an ordinary grid of small blocks, one slice of one
// operation each, as many to an SM as there are registers for, launched while the kernel before it ends.  Blocks of the same slice of all operations are neighbours: what several operations
// read comes from memory once.  Large messages are bound by memory (each operand read and each result written once), small ones by the launch.  Figures in coll/flow.cc.
#pragma once
#include <type_traits>
#include "exec_impl.cuh"

namespace piccl {

// The accumulators of nested results (FlowOp).  Which one a leaf goes to is the same for all threads; they are named, not indexed, so that they stay in registers.
// LEVELS: four operands need two at most, (a + b) + (c + d).
template <typename T, int OP, int LEVELS> struct FlowAcc {
  typedef typename AccOf<T>::type A;
  static constexpr int N = Pack<T>::N;
  A s0[N], s1[N], s2[LEVELS > 2 ? N : 1], s3[LEVELS > 2 ? N : 1];
  static __device__ __forceinline__ void round(A (&s)[N]) {
    if constexpr (sizeof(T) != sizeof(A)) {
#pragma unroll
      for (int e = 0; e < N; e++) s[e] = Cvt<T>::up(Cvt<T>::down(s[e]));
    }
  }
  static __device__ __forceinline__ void fold(A (&s)[N], const A (&x)[N], bool first) {
    if (first) {
#pragma unroll
      for (int e = 0; e < N; e++) s[e] = x[e];
    } else {
#pragma unroll
      for (int e = 0; e < N; e++) s[e] = red<OP, A>(s[e], x[e]);
    }
  }
  static __device__ __forceinline__ void fold_before(A (&s)[N], const A (&x)[N]) {
#pragma unroll
    for (int e = 0; e < N; e++) s[e] = red<OP, A>(x[e], s[e]);
  }
  __device__ __forceinline__ void leaf(const uint4& v, int i, int place, bool before, int scaled, float scale) {
    A x[N];
    Pack<T>::up(v, x);
    if (scaled >> i & 1) {
#pragma unroll
      for (int e = 0; e < N; e++) x[e] = scale_operand<T, true>(x[e], scaled, i, scale);
    }
    int level = place & 3;
    const bool first = place & 4;
    if (OP >= 2 && before) {                               // (sums and products are the same either way round)
      if (level == 0) fold_before(s0, x);
      else if (LEVELS == 2 || level == 1) fold_before(s1, x);
      else if constexpr (LEVELS > 2) { if (level == 2) fold_before(s2, x); else fold_before(s3, x); }
    }
    else if (level == 0) fold(s0, x, first);
    else if (LEVELS == 2 || level == 1) fold(s1, x, first);
    else if constexpr (LEVELS > 2) { if (level == 2) fold(s2, x, first); else fold(s3, x, first); }
    int merges = place >> 5;
    for (int k = place >> 3 & 3; k > 0; k--, merges >>= 1) {
      if (level == 0) round(s0);
      else if (LEVELS == 2 || level == 1) { round(s1); if (merges & 1) fold(s0, s1, false); }
      else if constexpr (LEVELS > 2) {
        if (level == 2) { round(s2); if (merges & 1) fold(s1, s2, false); }
        else { round(s3); if (merges & 1) fold(s2, s3, false); }
      }
      level -= merges & 1;
    }
  }
};

// The shapes that most calls have, without a branch per leaf: the general form works as long as it waits (us, general and this: reduce-scatter 8 x 8 MiB on the ring 128 / 98, reduce 8 x 16 MiB
// 38 / 28, all-reduce 4 x 25 MiB averaged by recursive doubling 43 / 38, maximum of 8 x 8 MB in fours and pairs 53 / 31).
template <typename T, int OP> struct FlowEval {
  typedef typename AccOf<T>::type A;
  static constexpr int N = Pack<T>::N;
  typedef FlowAcc<T, OP, 2> Acc;
  static __device__ __forceinline__ void get(const uint4& v, int i, int scaled, float scale, A (&x)[N]) {
    Pack<T>::up(v, x);
    if (scaled >> i & 1) {
#pragma unroll
      for (int e = 0; e < N; e++) x[e] = scale_operand<T, true>(x[e], scaled, i, scale);
    }
  }
  // one accumulator: a ring's hops
  template <int LEAVES, class V> static __device__ __forceinline__ void chain(const V& v, const FlowOp& op, int scaled, float scale, A (&s)[N]) {
    get(v(0), 0, scaled, scale, s);
#pragma unroll
    for (int i = 1; i < LEAVES; i++) {
      if (i < op.n_leaf) {
        A x[N];
        get(v(i), i, scaled, scale, x);
        if (OP >= 2 && (op.before >> i & 1)) Acc::fold_before(s, x); else Acc::fold(s, x, false);
        if (op.place[i] >> 3 & 3) Acc::round(s);
      }
    }
  }
  template <int FIRST, int R0, int R1, int R2, class V> static __device__ __forceinline__ void tree(const V& v, int scaled, float scale, A (&s)[N]) {
    if constexpr (R2 > 1) {
      tree<FIRST, R0, R1, 1>(v, scaled, scale, s); Acc::round(s);
      A x[N];
      tree<FIRST + R0 * R1, R0, R1, 1>(v, scaled, scale, x); Acc::round(x);
      Acc::fold(s, x, false);
    } else if constexpr (R1 > 1) {
      tree<FIRST, R0, 1, 1>(v, scaled, scale, s); Acc::round(s);
#pragma unroll
      for (int b = 1; b < R1; b++) {
        A x[N];
        if (b == 1) tree<FIRST + R0, R0, 1, 1>(v, scaled, scale, x);
        else if (b == 2) tree<(R1 > 2 ? FIRST + 2 * R0 : 0), R0, 1, 1>(v, scaled, scale, x);
        else tree<(R1 > 3 ? FIRST + 3 * R0 : 0), R0, 1, 1>(v, scaled, scale, x);
        Acc::round(x);
        Acc::fold(s, x, false);
      }
    } else {
      get(v(FIRST), FIRST, scaled, scale, s);
#pragma unroll
      for (int a = 1; a < R0; a++) { A x[N]; get(v(FIRST + a), FIRST + a, scaled, scale, x); Acc::fold(s, x, false); }
    }
  }
};

// Packs of an operation with nested results; LEAVES: at least as many as it has.
template <typename T, int OP, int LEAVES, int U>
__device__ __forceinline__ void flow_tree(const FlowOp& op, const char* const* src, char* const* dst, int n, int scaled, float scale, bool dst_done) {
  const unsigned long long policy = l2_policy(dst_done);
  const char* sp[LEAVES];
#pragma unroll
  for (int i = 0; i < LEAVES; i++) sp[i] = src[i < op.n_leaf ? i : 0];
  for (int p = threadIdx.x; p < n; p += U * kFlowBlock) {
    uint4 v[LEAVES][U];
#pragma unroll
    for (int i = 0; i < LEAVES; i++)
#pragma unroll
      for (int u = 0; u < U; u++) v[i][u] = ld_slot(sp[i] + (size_t)min(p + u * kFlowBlock, n - 1) * 16);
#pragma unroll
    for (int u = 0; u < U; u++) {
      typedef FlowEval<T, OP> E;
      typename E::A s[E::N];
      auto leaf = [&](int i) -> const uint4& { return v[i][u]; };
      if (op.shape == FLOW_CHAIN) E::template chain<LEAVES>(leaf, op, scaled, scale, s);
      else if (op.shape == (2 | 2 << 4)) E::template tree<0, 2, 2, LEAVES / 4>(leaf, scaled, scale, s);
      else if (LEAVES == 8 && op.shape == (4 | 2 << 4)) { if constexpr (LEAVES == 8) E::template tree<0, 4, 2, 1>(leaf, scaled, scale, s); }
      else if (LEAVES == 8 && op.shape == (2 | 4 << 4)) { if constexpr (LEAVES == 8) E::template tree<0, 2, 4, 1>(leaf, scaled, scale, s); }
      else {
        // a loop over an array in local memory: written out per leaf, the code is so long that a small call spends 5 us fetching it
        FlowAcc<T, OP, LEAVES <= 4 ? 2 : kFlowLevels> acc;
        uint4 w[LEAVES];
#pragma unroll
        for (int i = 0; i < LEAVES; i++) w[i] = v[i][u];
#pragma unroll 1
        for (int i = 0; i < op.n_leaf; i++) acc.leaf(w[i], i, op.place[i], op.before >> i & 1, scaled, scale);
#pragma unroll
        for (int e = 0; e < E::N; e++) s[e] = acc.s0[e];
      }
      const uint4 o = Pack<T>::down(s);
      if (p + u * kFlowBlock < n) for (int d = 0; d < op.n_dst; d++) st_hint(dst[d] + (size_t)(p + u * kFlowBlock) * 16, o, policy);
    }
  }
}
// The same at any address, a warp's block of 32 packs at a time.
template <typename T, int OP>
__device__ __noinline__ void flow_tree_shift(const FlowOp& op, const char* const* src, char* const* dst, long long npack, int scaled, float scale) {
  const int lane = threadIdx.x & 31;
  for (long long run = threadIdx.x & ~31; run < npack; run += kFlowBlock) {
    FlowAcc<T, OP, kFlowLevels> acc;      // (the general form: what comes at odd addresses is bound by its shifts; a loop over an array, as above, takes half as long again)
#pragma unroll 1
    for (int i0 = 0; i0 < op.n_leaf; i0 += 4) {            // four leaves' loads in flight
      RunWords<1> r[4];
      int m[4];
#pragma unroll
      for (int i = 0; i < 4; i++) { const char* const s = src[min(i0 + i, op.n_leaf - 1)]; m[i] = address_mod(s); load_run(r[i], s, m[i], run, lane, npack); }
#pragma unroll
      for (int i = 0; i < 4; i++) if (i0 + i < op.n_leaf) acc.leaf(run_pack(r[i], 0, m[i], lane), i0 + i, op.place[i0 + i], op.before >> (i0 + i) & 1, scaled, scale);
    }
    const uint4 o[1] = {Pack<T>::down(acc.s0)};
    store_run<1>(o, op.n_dst, dst, run, lane, npack);
  }
}

// The last, partial pack of an operation without nested results.  All operands are on their way before the first is used: one after the other, eight cost six microseconds at the end of a call.
template <typename T, int OP>
__device__ __noinline__ void flow_elem(const FlowOp& op, const char* const* src, char* const* dst, long long first, long long nelem, int scaled, float scale) {
  typedef typename AccOf<T>::type A;
  for (long long i = first + threadIdx.x; i < nelem; i += kFlowBlock) {
    T raw[kFlowLeaves];
#pragma unroll
    for (int s = 0; s < kFlowLeaves; s++) if (s < op.n_leaf) raw[s] = *reinterpret_cast<const volatile T*>(reinterpret_cast<const T*>(src[s]) + i);
    A acc = A();
#pragma unroll
    for (int s = 0; s < kFlowLeaves; s++)
      if (s < op.n_leaf) {
        const A x = scale_operand<T, true>(Cvt<T>::up(raw[s]), scaled, s, scale);
        acc = s == 0 ? x : red<OP, A>(acc, x);
      }
    const T o = Cvt<T>::down(acc);
    for (int d = 0; d < op.n_dst; d++) reinterpret_cast<T*>(dst[d])[i] = o;
  }
}

template <typename T, int OP, bool SHIFT>
__global__ void __launch_bounds__(kFlowBlock, 3) exec_flow_kernel(const FlowArgs fa) {
  constexpr int esz = (int)sizeof(T), N = Pack<T>::N;
  __shared__ FlowOp op;
  __shared__ const char* s_src[kFlowLeaves];
  __shared__ char* s_dst[kFlowLeaves];
  const int tid = threadIdx.x, slice = blockIdx.x / fa.n_ops;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  static_assert(sizeof(FlowOp) % 8 == 0 && sizeof(FlowOp) / 8 <= kFlowBlock, "copied by the block");
  if (tid < (int)(sizeof(FlowOp) / 8)) reinterpret_cast<unsigned long long*>(&op)[tid] = reinterpret_cast<const unsigned long long*>(fa.ops + blockIdx.x % fa.n_ops)[tid];
  __syncthreads();
  const Slice sl = slice_of(op.count, esz, slice, fa.n_slices, fa.slice_bytes);
  if (sl.lo >= sl.hi) return;
  if (tid < op.n_leaf) s_src[tid] = (op.leaf_buf[tid] == BUF_IN ? (const char*)fa.in[op.leaf_rank[tid]] : (const char*)fa.out[op.leaf_rank[tid]]) + (op.leaf_off[tid] + sl.lo) * esz;
  if (tid < op.n_dst) s_dst[tid] = (char*)fa.out[op.dst_rank[tid]] + (op.dst_off[tid] + sl.lo) * esz;
  __syncthreads();
  const int scaled = fa.avg ? op.scaled | op.rounded << kRoundedShift : 0;
  const long long len = sl.hi - sl.lo, nfull = len / N;
  const bool dst_done = fa.leave_first & 2;
  constexpr bool NESTED = OP != OP_COPY && !std::is_integral<T>::value;      // (integers are folded flat)
  if (NESTED && op.nested) {
    if constexpr (NESTED) {
      if constexpr (SHIFT) flow_tree_shift<T, OP>(op, s_src, s_dst, nfull, scaled, fa.scale);
      else if (op.n_leaf <= 4) flow_tree<T, OP, 4, 2>(op, s_src, s_dst, (int)nfull, scaled, fa.scale, dst_done);
      else flow_tree<T, OP, 8, 1>(op, s_src, s_dst, (int)nfull, scaled, fa.scale, dst_done);
      if (tid < len - nfull * N) {                         // the last, partial pack, an element a thread
        typedef typename AccOf<T>::type A;
        A s[kFlowLevels];
        T raw[kFlowLeaves];
#pragma unroll
        for (int i = 0; i < kFlowLeaves; i++) if (i < op.n_leaf) raw[i] = *reinterpret_cast<const volatile T*>(reinterpret_cast<const T*>(s_src[i]) + nfull * N + tid);
#pragma unroll 1
        for (int i = 0; i < op.n_leaf; i++) {
          const A x = scale_operand<T, true>(Cvt<T>::up(raw[i]), scaled, i, fa.scale);
          int level = op.place[i] & 3, merges = op.place[i] >> 5;
          s[level] = op.place[i] & 4 ? x : op.before >> i & 1 ? red<OP, A>(x, s[level]) : red<OP, A>(s[level], x);
          for (int k = op.place[i] >> 3 & 3; k > 0; k--, merges >>= 1) {
            s[level] = Cvt<T>::up(Cvt<T>::down(s[level]));
            if (merges & 1) { level--; s[level] = red<OP, A>(s[level], s[level + 1]); }
          }
        }
        for (int d = 0; d < op.n_dst; d++) reinterpret_cast<T*>(s_dst[d])[nfull * N + tid] = Cvt<T>::down(s[0]);
      }
    }
    return;
  }
  if constexpr (SHIFT) { if (nfull) reduce_copy_shift<T, OP, true>(kFlowBlock, op.n_leaf, s_src, op.n_dst, s_dst, nfull, scaled, fa.scale); }
  else if (nfull) move_aligned<T, OP, true>(kFlowBlock, s_src, op.n_leaf, s_dst, op.n_dst, (int)nfull, scaled, fa.scale, L2Hints{(fa.leave_first & 1) && op.once, dst_done, 0, 0});
  if (nfull * N < len) flow_elem<T, OP>(op, s_src, s_dst, nfull * N, len, scaled, fa.scale);
}

}  // namespace piccl

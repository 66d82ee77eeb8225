// What a collective computes, without the way it takes: for launches that carry all ranks on one GPU, where every rank's buffers are equally near.
//
// A program says which operands are combined where, in which order, and through which slots the values travel.  Between GPUs that way is the point; on one GPU it is
// several passes over memory for each hop.  `data_flow` follows the entries of all ranks' programs back and keeps what they compute: each element of a
// receive buffer as an expression over the send buffers, with the operands of each action in its order and each partial result rounded to the element type where it would
// have been put into a slot, so that the results are bit for bit those of the programs,
// or of the low-latency kernel that a small call would take.  (But for bf16 averages among 2, 4 or 8 ranks of elements whose share is
// below 2^-126, its normal range: such shares are not rounded on their way.)  A sum that one rank makes and others receive, or that several ranks make alike, is
// computed once and stored in all their buffers.  Nothing in such a call waits (kernels/exec_flow.cuh).
//
// us through the slots and this, one B200: all-reduce 4 x 25 MiB averaged by recursive doubling 131 / 38, 8 x 64 MiB on the ring 353 / 188, 8 x 280 KB 45 / 4.8, 8 x 4 KB 37 / 4.7; all-gather 4 x 1 MiB at
// odd addresses 28.7 / 10.3, 8 x 8 MiB 195 / 98; reduce-scatter 2 x 32 MiB 55.5 / 34, 8 x 8 MiB on the ring 195 / 94; broadcast 8 x 16 MiB 103 / 27; reduce 8 x 16 MiB on the ring 92 / 28, in two rings 120 / 56.
#include <algorithm>
#include <array>
#include <map>
#include "coll_internal.h"

namespace piccl {

namespace {

struct Ref { int rank = -1, act = -1; bool operator<(const Ref& o) const { return rank != o.rank ? rank < o.rank : act < o.act; } };

struct Flow {
  const std::vector<Program>& progs;
  std::vector<std::vector<std::vector<Ref>>> producer;      // [rank][action][receive operand]
  FlowOp op;                                                // the expression being built
  bool ok = true;
  FlowKind kind;
  Flow(const std::vector<Program>& p, FlowKind k) : progs(p), producer(p.size()), kind(k) {}

  // the k-th entry pushed on a connection is the k-th one popped; false: the programs do not fit together
  bool match() {
    const int n = (int)progs.size();
    std::vector<std::vector<int>> pushed((size_t)n * n);
    std::vector<size_t> popped((size_t)n * n, 0);
    for (int s = 0; s < n; s++) {
      producer[s].resize(progs[s].actions.size());
      for (size_t i = 0; i < progs[s].actions.size(); i++)
        for (int j = 0; j < progs[s].actions[i].n_send; j++) pushed[(size_t)s * n + progs[s].actions[i].send_peer[j]].push_back((int)i);
    }
    for (int d = 0; d < n; d++)
      for (size_t i = 0; i < progs[d].actions.size(); i++) {
        const Action& a = progs[d].actions[i];
        for (int j = 0; j < a.n_recv; j++) {
          const size_t c = (size_t)a.recv_peer[j] * n + d;
          if (popped[c] >= pushed[c].size()) return false;
          const int act = pushed[c][popped[c]++];
          if (progs[a.recv_peer[j]].actions[act].count != a.count) return false;
          producer[d][i].push_back({(int)a.recv_peer[j], act});
        }
      }
    for (size_t c = 0; c < pushed.size(); c++) if (popped[c] != pushed[c].size()) return false;
    return true;
  }
  // the last action of rank s in [begin, end) that stores any of the range (-1: none), and whether it stores exactly that
  int writer(int s, int begin, int end, uint8_t buf, int64_t off, int64_t n, bool* exact) const {
    for (int i = end; i-- > begin;) {
      const Action& a = progs[s].actions[i];
      if (a.dst_buf != buf || a.dst_off >= off + n || off >= a.dst_off + a.count) continue;
      *exact = a.dst_off == off && a.count == n;
      return i;
    }
    return -1;
  }
  // where the value of an action that only hands on (one operand) comes from: the action that makes it, or one whose operand is a buffer's elements
  Ref maker(Ref at) {
    for (;;) {
      const Action& a = progs[at.rank].actions[at.act];
      if (a.n_recv == 1 && a.src_buf == BUF_NONE) { at = producer[at.rank][at.act][0]; continue; }
      if (a.n_recv == 0 && a.src_buf != BUF_IN) {
        bool exact = false;
        const int w = writer(at.rank, 0, at.act, a.src_buf, a.src_off, a.count, &exact);
        if (w >= 0 && exact) { at.act = w; continue; }
        if (w >= 0 || a.src_buf != BUF_OUT) ok = false;
      }
      return at;
    }
  }
  void leaf(int rank, uint8_t buf, int64_t off, bool scaled, bool rounded, int level, bool first) {
    if (op.n_leaf == kFlowLeaves) { ok = false; return; }
    const int i = op.n_leaf++;
    op.leaf_rank[i] = (uint8_t)rank; op.leaf_buf[i] = buf; op.leaf_off[i] = off;
    op.place[i] = (uint8_t)(level | (first ? 4 : 0));
    if (scaled) op.scaled |= (uint8_t)(1u << i);
    // One half, quarter or eighth of an element is itself an element unless it is below the normal range.  Where it is taken for one all ranks' averages are one expression; otherwise each rank's own share is the
    // one that is not rounded in its own result (fp16, us: 4 x 25 MiB by recursive doubling 37 and 45.6, through the slots 131; 8 x 8 MB in eights 24 and 68, 202).
    if (scaled && (kind == FLOW_ALL_SHARES || (rounded && (kind == FLOW_SMALL_SHARES || (progs.size() & (progs.size() - 1)) != 0)))) op.rounded |= (uint8_t)(1u << i);
  }
  void event(bool merge) {                                  // after the last leaf
    uint8_t& p = op.place[op.n_leaf - 1];
    const int k = p >> 3 & 3;
    if (k == 3) { ok = false; return; }
    p = (uint8_t)((p & ~0x18) | (k + 1) << 3 | (merge ? 0x20 << k : 0));
    op.nested = 1;
  }
  // The operands of the action that makes `at`, folded into accumulator `level`.
  void fold(Ref at, int level) {
    if (!ok) return;
    if (level >= kFlowLevels) { ok = false; return; }
    const Action& a = progs[at.rank].actions[at.act];
    struct Operand { Ref from; bool own; };                 // own: the rank's elements of the send buffer
    std::vector<Operand> operands;
    for (int j = 0; j <= a.n_recv && ok; j++) {
      if (j == a.self_pos && a.src_buf == BUF_IN) operands.push_back({at, true});
      else if (j == a.self_pos && a.src_buf != BUF_NONE) {
        bool exact = false;
        const int w = writer(at.rank, 0, at.act, a.src_buf, a.src_off, a.count, &exact);
        if (w < 0 || !exact) { ok = false; return; }
        operands.push_back({maker({at.rank, w}), false});
      }
      if (j < a.n_recv) operands.push_back({maker(producer[at.rank][at.act][j]), false});
    }
    if (!ok) return;
    auto simple = [&](const Operand& o) { return o.own || progs[o.from.rank].actions[o.from.act].n_recv == 0; };
    bool first = true;
    auto emit = [&](const Operand& o, bool before) {
      if (!ok) return;
      const Action& b = progs[o.from.rank].actions[o.from.act];
      if (o.own) leaf(at.rank, BUF_IN, a.src_off, (a.flags & ACT_SCALE_SRC) != 0, false, level, first);
      else if (simple(o)) leaf(o.from.rank, b.src_buf, b.src_off, (b.flags & ACT_SCALE_SRC) && b.src_buf == BUF_IN, true, level, first);
      else if (first) { fold(o.from, level); if (ok) event(false); }
      else { fold(o.from, level + 1); if (ok) event(true); }
      if (ok && before) op.before |= (uint8_t)(1u << (op.n_leaf - 1));
      first = false;
    };
    // a result behind a leaf: the result first, the leaf as its left operand (a ring's hops would need an accumulator each)
    const bool turned = operands.size() >= 2 && simple(operands[0]) && !simple(operands[1]);
    if (turned) { emit(operands[1], false); emit(operands[0], true); }
    for (size_t q = turned ? 2 : 0; q < operands.size(); q++) emit(operands[q], false);
  }
};

}  // namespace

// Integers: one fold of all operands, whatever the nesting was, in the ranks' order so that all ranks' expressions are alike.  Evaluated as nested expressions, 8-bit elements, sixteen to a pack, were
// slower than through the slots (us through the slots, nested, and this: maximum of 8 x 16 MiB of bytes in two rings 197, 1018, 35; product of 8 x 5 KB in fours 8.8, 23.6, 4.7; reduce-scatter of 8 x 2 MB on the ring at odd
// addresses 532, 812, 78).
static void flatten(FlowOp& op) {
  std::array<int, kFlowLeaves> order;
  for (int i = 0; i < op.n_leaf; i++) order[i] = i;
  std::sort(order.begin(), order.begin() + op.n_leaf, [&](int a, int b) { return std::make_pair(op.leaf_rank[a], op.leaf_off[a]) < std::make_pair(op.leaf_rank[b], op.leaf_off[b]); });
  const FlowOp was = op;
  for (int i = 0; i < op.n_leaf; i++) {
    op.leaf_rank[i] = was.leaf_rank[order[i]]; op.leaf_buf[i] = was.leaf_buf[order[i]]; op.leaf_off[i] = was.leaf_off[order[i]];
    op.place[i] = i == 0 ? 4 : 0;
  }
  op.nested = op.scaled = op.rounded = op.before = 0;
}

bool data_flow(const std::vector<Program>& progs, std::vector<FlowOp>& ops, FlowKind kind) {
  const int n = (int)progs.size();
  ops.clear();
  Flow f(progs, kind);
  if (n < 2 || n > kFlowLeaves || !f.match()) return false;
  std::map<Ref, int> made;                                  // the operation of what an action makes
  auto alike = [](const FlowOp& a, const FlowOp& b) {
    if (a.count != b.count || a.n_leaf != b.n_leaf || a.nested != b.nested || a.scaled != b.scaled || a.rounded != b.rounded || a.before != b.before) return false;
    for (int i = 0; i < a.n_leaf; i++) if (a.leaf_rank[i] != b.leaf_rank[i] || a.leaf_buf[i] != b.leaf_buf[i] || a.leaf_off[i] != b.leaf_off[i] || a.place[i] != b.place[i]) return false;
    return true;
  };
  for (int r = 0; r < n; r++)
    for (size_t i = 0; i < progs[r].actions.size(); i++) {
      const Action& a = progs[r].actions[i];
      if (a.dst_buf != BUF_OUT) continue;
      bool exact = false;
      if (f.writer(r, (int)i + 1, (int)progs[r].actions.size(), a.dst_buf, a.dst_off, a.count, &exact) >= 0) { if (!exact) return false; continue; }      // stored for a later step only
      const Ref m = f.maker({r, (int)i});
      if (!f.ok) return false;
      const Action& b = progs[m.rank].actions[m.act];
      f.op = FlowOp();
      f.op.count = a.count;
      int at = -1;
      if (b.n_recv == 0) {
        // A copy has one destination: the operand comes from the cache again for the next (all-gather 8 x 8 MiB 97.5 us, 107 with eight destinations; 4 x 1 MiB at odd addresses, where a
        // copy to one place is shifted once, 10.4 and 15.2).  The maker's own copy of a scaled operand is the value that others receive.
        f.leaf(m.rank, b.src_buf, b.src_off, (b.flags & ACT_SCALE_SRC) && b.src_buf == BUF_IN, false, 0, true);
      } else {
        const auto it = made.find(m);
        if (it != made.end()) at = it->second;
        else {
          f.fold(m, 0);
          if (kind == FLOW_INTEGERS && f.ok) flatten(f.op);
          for (size_t q = 0; q < ops.size() && f.ok && at < 0; q++) if (ops[q].n_leaf > 1 && alike(ops[q], f.op)) at = (int)q;
        }
      }
      if (!f.ok) return false;
      if (at < 0) { at = (int)ops.size(); ops.push_back(f.op); }
      else if (ops[at].n_dst == kFlowLeaves) {               // the same once more, for further destinations
        FlowOp again = ops[at];
        again.n_dst = 0;
        at = (int)ops.size(); ops.push_back(again);
      }
      if (b.n_recv != 0) made[m] = at;
      FlowOp& op = ops[at];
      op.dst_rank[op.n_dst] = (uint8_t)r; op.dst_off[op.n_dst++] = a.dst_off;
    }
  // Shapes that the kernel has straight code for: one accumulator (rings), and even trees of 4 and 8 operands in pairs and fours (recursive algorithms).
  auto even_tree = [](const FlowOp& op, int r0, int r1, int r2) {
    if (op.n_leaf != r0 * r1 * r2 || op.before) return false;
    for (int i = 0; i < op.n_leaf; i++) {
      const int a = i % r0, b = i / r0 % r1, c = i / (r0 * r1);
      // groups behind the first of their kind have an accumulator of their own, one up for each kind
      const int level = (b > 0) + (c > 0);
      int place = level | (a == 0 ? 4 : 0), done = 0;
      if (a == r0 - 1) { place |= b > 0 ? 0x20 << done : 0; done++; }
      if (a == r0 - 1 && b == r1 - 1 && r2 > 1) { place |= c > 0 ? 0x20 << done : 0; done++; }
      if (op.place[i] != (place | done << 3)) return false;
    }
    return true;
  };
  for (FlowOp& op : ops) {
    if (!op.nested) continue;
    bool chain = true;
    for (int i = 0; i < op.n_leaf; i++) chain &= (op.place[i] & 3) == 0;
    if (chain) op.shape = FLOW_CHAIN;
    else if (even_tree(op, 2, 2, 1) || even_tree(op, 2, 2, 2)) op.shape = 2 | 2 << 4;
    else if (even_tree(op, 4, 2, 1)) op.shape = 4 | 2 << 4;
    else if (even_tree(op, 2, 4, 1)) op.shape = 2 | 4 << 4;
  }
  // Elements of a buffer that no other operation reads may leave the cache with their use.
  for (size_t i = 0; i < ops.size(); i++) {
    bool again = false;
    for (size_t q = 0; q < ops.size() && !again; q++)
      for (int l = 0; l < ops[i].n_leaf && q != i && !again; l++)
        for (int k = 0; k < ops[q].n_leaf; k++)
          again |= ops[q].leaf_rank[k] == ops[i].leaf_rank[l] && ops[q].leaf_buf[k] == ops[i].leaf_buf[l] && ops[q].leaf_off[k] < ops[i].leaf_off[l] + ops[i].count && ops[i].leaf_off[l] < ops[q].leaf_off[k] + ops[q].count;
    ops[i].once = !again;
  }
  return !ops.empty();
}

const char* check_flow(const std::vector<FlowOp>& ops, const CollArgs& a) {
  const int64_t st = a.block_stride ? a.block_stride : a.count;
  const int64_t in_elems = a.coll == COLL_REDUCE_SCATTER ? (a.nranks - 1) * st + a.count : a.count, out_elems = a.coll == COLL_ALLGATHER ? (a.nranks - 1) * st + a.count : a.count;
  for (const FlowOp& op : ops) {
    if (op.count <= 0 || op.n_leaf < 1 || op.n_leaf > kFlowLeaves || op.n_dst < 1 || op.n_dst > kFlowLeaves) return "bad number of operands, destinations or elements";
    int level = 0;
    bool begun[kFlowLevels] = {false};
    for (int i = 0; i < op.n_leaf; i++) {
      if (op.leaf_rank[i] >= a.nranks || (a.coll == COLL_BROADCAST && op.leaf_rank[i] != a.root)) return "operand of a rank that has none";
      if (op.leaf_buf[i] != BUF_IN && !(op.leaf_buf[i] == BUF_OUT && a.in_place)) return "operand that is not in a send buffer";
      if (op.leaf_off[i] < 0 || op.leaf_off[i] + op.count > (op.leaf_buf[i] == BUF_IN ? in_elems : out_elems)) return "operand outside its buffer";
      level = op.place[i] & 3;
      if (((op.place[i] & 4) != 0) == begun[level]) return "an accumulator that is begun twice, or not at all";
      begun[level] = true;
      if (!op.nested && (level || (op.place[i] >> 3) || ((op.place[i] & 4) != 0) != (i == 0))) return "a nested expression that says it is flat";
      for (int k = 0; k < (op.place[i] >> 3 & 3); k++)
        if (op.place[i] >> (5 + k) & 1) {
          if (level == 0 || !begun[level - 1]) return "fold into an accumulator that holds nothing";
          begun[level--] = false;
        }
    }
    if (level != 0) return "accumulators left";
    for (int i = 1; i < kFlowLevels; i++) if (begun[i]) return "accumulators left";
    for (int i = 0; i < op.n_dst; i++) {
      if (op.dst_rank[i] >= a.nranks || (a.coll == COLL_REDUCE && op.dst_rank[i] != a.root)) return "destination of a rank that has none";
      if (op.dst_off[i] < 0 || op.dst_off[i] + op.count > out_elems) return "destination outside its buffer";
    }
  }
  return nullptr;
}

}  // namespace piccl

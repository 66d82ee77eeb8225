// Data flows (src/coll/flow.cc) looked at from inside; prints what is wrong, or OK.  flow_main CHECK
#include <cstdio>
#include <cstring>
#include "piccl_sched.h"

using namespace piccl;

static int bad(const char* what, const CollArgs& a) {
  printf("%s: collective %d algorithm %d radix %d ranks %d count %lld\n", what, (int)a.coll, (int)a.algo, a.k, a.nranks, (long long)a.count);
  return 1;
}
template <class F> static int each_call(F f) {
  for (int coll = 0; coll < COLL_COUNT; coll++)
    for (int algo : {ALGO_RING, ALGO_K_RING, ALGO_RD, ALGO_RM, ALGO_PRD, ALGO_PRM, ALGO_DIRECT})
      for (int n = 2; n <= 8; n++)
        for (int k : {-1, 2, 4, 8})
          for (long long count : {1LL, 257LL, 4096LL}) {
            CollArgs a; a.coll = (Coll)coll; a.algo = (Algo)algo; a.k = k; a.nranks = n; a.root = n / 2; a.count = count;
            std::vector<Program> progs;
            for (int r = 0; r < n; r++) progs.push_back(compile(a, r));
            if (int rc = f(a, progs)) return rc;
          }
  return 0;
}

// Integers: one fold of different operands, an operand of each rank to a sum, and no expression twice but for its destinations.
static int integers() {
  return each_call([](const CollArgs& a, const std::vector<Program>& progs) {
    std::vector<FlowOp> ops;
    if (!data_flow(progs, ops, FLOW_INTEGERS)) return bad("no data flow", a);
    const bool sums = a.coll == COLL_ALLREDUCE || a.coll == COLL_REDUCE || a.coll == COLL_REDUCE_SCATTER;
    for (size_t q = 0; q < ops.size(); q++) {
      const FlowOp& op = ops[q];
      if (op.nested || op.before || (sums && (op.scaled || op.rounded))) return bad("not flat", a);
      if (!sums) continue;
      if (op.n_leaf != a.nranks) return bad("operands missing", a);
      for (int i = 0; i < op.n_leaf; i++) if (op.leaf_rank[i] != i || op.place[i] != (i == 0 ? 4 : 0)) return bad("operands not in the ranks' order", a);
      for (size_t p = 0; p < q; p++) if (ops[p].leaf_off[0] == op.leaf_off[0] && ops[p].n_dst < kFlowLeaves) return bad("an expression twice", a);
    }
    return 0;
  });
}

// A sum that eight ranks store at two places each has more destinations than one operation holds: a second one with the same expression.
static int destinations() {
  const int n = 8, count = 16;
  std::vector<Program> progs(n);
  for (int r = 0; r < n; r++) {
    progs[r].rank = r; progs[r].nranks = n;
    Action get, twice;
    get.count = twice.count = count; get.dst_buf = BUF_OUT;
    if (r == 0) {
      get.src_buf = BUF_IN; get.n_recv = get.n_send = n - 1;
      for (int p = 1; p < n; p++) get.recv_peer[p - 1] = get.send_peer[p - 1] = (uint8_t)p;
    } else {
      Action put;
      put.count = count; put.src_buf = BUF_IN; put.n_send = 1; put.send_peer[0] = 0;
      progs[r].actions.push_back(put);
      get.n_recv = 1; get.recv_peer[0] = 0;
    }
    twice.src_buf = twice.dst_buf = BUF_OUT; twice.dst_off = count;
    progs[r].actions.push_back(get);
    progs[r].actions.push_back(twice);
  }
  std::vector<FlowOp> ops;
  if (!data_flow(progs, ops)) { printf("no data flow\n"); return 1; }
  int stored[8][2] = {{0}};
  for (const FlowOp& op : ops) {
    if (op.n_leaf != n || op.count != count || op.n_dst < 1 || op.n_dst > kFlowLeaves) { printf("an operation of %d operands and %d destinations\n", op.n_leaf, op.n_dst); return 1; }
    for (int i = 0; i < n; i++) if (op.leaf_rank[i] != i || op.leaf_buf[i] != BUF_IN || op.leaf_off[i] != 0) { printf("wrong operands\n"); return 1; }
    for (int i = 0; i < op.n_dst; i++) stored[op.dst_rank[i]][op.dst_off[i] / count]++;
  }
  for (auto& r : stored) for (int s : r) if (s != 1) { printf("stored %d times\n", s); return 1; }
  return 0;
}

// Every call's operations pass the check, whole and of every kind; with one of their fields set wrong they do not.
static int checked() {
  return each_call([](const CollArgs& given, const std::vector<Program>& given_progs) {
    CollArgs a = given;
    std::vector<Program> progs = given_progs;
    for (bool in_place : {false, true}) {
      if (in_place) {
        if (a.coll != COLL_ALLGATHER && a.coll != COLL_BROADCAST) break;
        a.in_place = true;
        for (int r = 0; r < a.nranks; r++) progs[r] = compile(a, r);
      }
      for (FlowKind kind : {FLOW_FLOATS, FLOW_INTEGERS, FLOW_SMALL_SHARES, FLOW_ALL_SHARES}) {
        std::vector<FlowOp> ops;
        if (!data_flow(progs, ops, kind)) return bad("no data flow", a);
        if (const char* why = check_flow(ops, a)) { printf("%s\n", why); return bad("refused", a); }
        const int64_t in = a.coll == COLL_REDUCE_SCATTER ? a.nranks * a.count : a.count, out = a.coll == COLL_ALLGATHER ? a.nranks * a.count : a.count;
        int missed = 0;
        auto wrong = [&](auto set) {
          for (size_t q = 0; q < ops.size(); q += 7) {
            const FlowOp was = ops[q];
            set(ops[q]);
            missed += check_flow(ops, a) == nullptr;
            ops[q] = was;
          }
        };
        wrong([&](FlowOp& op) { op.count = 0; });
        wrong([&](FlowOp& op) { op.n_leaf = 0; });
        wrong([&](FlowOp& op) { op.n_leaf = kFlowLeaves + 1; });
        wrong([&](FlowOp& op) { op.n_dst = 0; });
        wrong([&](FlowOp& op) { op.n_dst = kFlowLeaves + 1; });
        wrong([&](FlowOp& op) { op.leaf_rank[0] = (uint8_t)a.nranks; });
        wrong([&](FlowOp& op) { op.leaf_buf[op.n_leaf - 1] = BUF_SCRATCH; });
        wrong([&](FlowOp& op) { op.leaf_off[op.n_leaf - 1] = (op.leaf_buf[op.n_leaf - 1] == BUF_IN ? in : out) - op.count + 1; });
        wrong([&](FlowOp& op) { op.leaf_off[0] = -1; });
        wrong([&](FlowOp& op) { op.place[0] &= (uint8_t)~4; });
        wrong([&](FlowOp& op) { op.place[op.n_leaf - 1] = (uint8_t)((op.place[op.n_leaf - 1] & ~3) | 4 | 1); });
        wrong([&](FlowOp& op) { op.dst_rank[op.n_dst - 1] = (uint8_t)a.nranks; });
        wrong([&](FlowOp& op) { op.dst_off[op.n_dst - 1] = out - op.count + 1; });
        wrong([&](FlowOp& op) { op.dst_off[0] = -1; });
        if (missed) return bad("a wrong operation passed", a);
      }
    }
    return 0;
  });
}

int main(int argc, char** argv) {
  const char* what = argc > 1 ? argv[1] : "";
  const int rc = !strcmp(what, "integers") ? integers() : !strcmp(what, "destinations") ? destinations() : !strcmp(what, "checked") ? checked() : 2;
  if (rc == 0) printf("OK\n");
  return rc;
}

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

int main(int argc, char** argv) {
  const char* what = argc > 1 ? argv[1] : "";
  const int rc = !strcmp(what, "integers") ? integers() : 2;
  if (rc == 0) printf("OK\n");
  return rc;
}

// Programs of ranks that can read each other's buffers: all ranks in one launch on one GPU.
//
// There every buffer is as near to one rank as to another, so an entry that only hands elements on, unchanged, needs no slot: its reader takes them from where
// they stand.  `share_operands` traces the value of each entry back to its origin:
//   - a caller's send buffer, which nobody writes during the call: no wait, and no hop that only forwards it;
//   - elements that a rank stored for good, its share of an all-reduce, say: readable once that rank's progress counter has passed the action that stored them.
// Sums that are on their way still travel through the slots, hop by hop, and are combined by the same ranks in the same order.  Waits are a subset of the
// transitive waits of the programs that came in, so what did not deadlock before does not now.
// us through the slots and with this, one B200: all-reduce 4 x 25 MiB averaged by recursive doubling 131 and 89, 8 x 64 MiB on the ring 353 and 294, 8 x 32 MiB doubling 472 and 271;
// all-gather 4 x 16 MiB 130 and 81; reduce-scatter 2 x 32 MiB 55 and 41; broadcast 8 x 16 MiB 110 and 41; reduce 8 x 16 MiB in two rings 120 and 92.
// A sum that is stored only to be overwritten by the next step's (recursive all-reduces) is not stored any more: the rank reads it again from the slot that it
// has just filled.
#include <algorithm>
#include "coll_internal.h"

namespace piccl {

namespace {

struct Origin { bool ok = false; int rank = 0; uint8_t buf = BUF_NONE; int64_t off = 0; int after = -1; bool scaled = false; };
struct Ref { int rank = -1, act = -1; };

bool touches(uint8_t buf, int64_t off, int64_t n, uint8_t buf2, int64_t off2, int64_t n2) { return buf == buf2 && off < off2 + n2 && off2 < off + n; }

struct Tracer {
  const std::vector<Program>& progs;
  std::vector<std::vector<std::vector<Ref>>> producer;      // [rank][action][receive operand]
  std::vector<std::vector<Origin>> memo;
  std::vector<std::vector<uint8_t>> known;
  explicit Tracer(const std::vector<Program>& p) : progs(p), producer(p.size()), memo(p.size()), known(p.size()) {}

  // the k-th entry pushed on a connection is the k-th one popped; false: the programs do not fit together
  bool match() {
    const int n = (int)progs.size();
    std::vector<std::vector<int>> pushed((size_t)n * n);
    std::vector<size_t> popped((size_t)n * n, 0);
    for (int s = 0; s < n; s++) {
      memo[s].resize(progs[s].actions.size()); known[s].assign(progs[s].actions.size(), 0); producer[s].resize(progs[s].actions.size());
      for (size_t i = 0; i < progs[s].actions.size(); i++)
        for (int j = 0; j < progs[s].actions[i].n_send; j++) pushed[(size_t)s * n + progs[s].actions[i].send_peer[j]].push_back((int)i);
    }
    for (int d = 0; d < n; d++)
      for (size_t i = 0; i < progs[d].actions.size(); i++) {
        const Action& a = progs[d].actions[i];
        for (int j = 0; j < a.n_recv; j++) {
          const int s = a.recv_peer[j];
          const size_t c = (size_t)s * n + d;
          if (popped[c] >= pushed[c].size()) return false;
          const int act = pushed[c][popped[c]++];
          if (progs[s].actions[act].count != a.count) return false;
          producer[d][i].push_back({s, act});
        }
      }
    for (size_t c = 0; c < pushed.size(); c++) if (popped[c] != pushed[c].size()) return false;
    return true;
  }

  // the last action of rank s before `end` that writes any of the range; -1: none
  int writer(int s, int begin, int end, uint8_t buf, int64_t off, int64_t n) const {
    for (int i = end; i-- > begin;) { const Action& a = progs[s].actions[i]; if (touches(a.dst_buf, a.dst_off, a.count, buf, off, n)) return i; }
    return -1;
  }
  Origin stored(int s, int i, uint8_t buf, int64_t off, int64_t n) const {      // by action i (-1: before the call), and never overwritten
    Origin o;
    if (writer(s, i + 1, (int)progs[s].actions.size(), buf, off, n) >= 0) return o;
    o.ok = true; o.rank = s; o.buf = buf; o.off = off; o.after = i;
    return o;
  }
  Origin origin(int s, int i) {
    if (known[s][i]) return memo[s][i];
    known[s][i] = 1;                                  // (programs have no cycles: a value comes from earlier ones)
    const Action& a = progs[s].actions[i];
    Origin o;
    if (a.n_recv == 0 && a.src_buf == BUF_IN) {
      o.ok = true; o.rank = s; o.buf = BUF_IN; o.off = a.src_off; o.scaled = (a.flags & ACT_SCALE_SRC) != 0;
    } else if (a.n_recv == 0) {                       // elements of its own that the rank stored earlier
      const int w = writer(s, 0, i, a.src_buf, a.src_off, a.count);
      if (w < 0) { if (a.src_buf == BUF_OUT) o = stored(s, -1, a.src_buf, a.src_off, a.count); }
      else if (progs[s].actions[w].dst_off == a.src_off && progs[s].actions[w].count == a.count) {
        o = origin(s, w);
        if (!(o.ok && o.buf == BUF_IN)) o = stored(s, w, a.src_buf, a.src_off, a.count);
      }
    } else if (a.n_recv == 1 && a.src_buf == BUF_NONE) {
      o = origin(producer[s][i][0].rank, producer[s][i][0].act);
      if (!o.ok && a.dst_buf != BUF_NONE) o = stored(s, i, a.dst_buf, a.dst_off, a.count);
    } else if (a.dst_buf != BUF_NONE) {
      o = stored(s, i, a.dst_buf, a.dst_off, a.count);
    }
    return memo[s][i] = o;
  }
};

}  // namespace

bool share_operands(std::vector<Program>& progs, std::vector<std::vector<SharedOps>>& shared) {
  const int n = (int)progs.size();
  Tracer t(progs);
  if (n < 2 || n > kMaxActionPeers + 1 || !t.match()) return false;
  std::vector<std::vector<Origin>> of(n);
  for (int r = 0; r < n; r++) for (size_t i = 0; i < progs[r].actions.size(); i++) of[r].push_back(t.origin(r, (int)i));

  // operands that are read where they stand, and entries that nobody takes from a slot any more
  bool any = false;
  std::vector<Program> next = progs;
  std::vector<std::vector<int>> place(n);
  shared.assign(n, {});
  for (int r = 0; r < n; r++) {
    std::vector<Action> kept;
    for (size_t i = 0; i < progs[r].actions.size(); i++) {
      Action a = progs[r].actions[i];
      SharedOps x;
      for (int j = 0; j < a.n_recv; j++) {
        const Ref p = t.producer[r][i][j];
        const Origin& o = of[p.rank][p.act];
        if (!o.ok) continue;
        a.recv_peer[j] = kSharedPeer;
        x.buf[j] = o.buf; x.from[j] = (uint8_t)o.rank; x.off[j] = o.off; x.after[j] = o.after;
        if (o.scaled) x.scaled |= (uint8_t)(1u << j);
        any = true;
      }
      if (of[r][i].ok) a.n_send = 0;
      place[r].push_back((int)kept.size());
      if (a.dst_buf == BUF_NONE && a.n_send == 0) continue;
      kept.push_back(a); shared[r].push_back(x);
    }
    next[r].actions = std::move(kept);
  }
  for (int r = 0; r < n; r++)
    for (size_t i = 0; i < next[r].actions.size(); i++)
      for (int j = 0; j < next[r].actions[i].n_recv; j++)
        if (next[r].actions[i].recv_peer[j] == kSharedPeer && shared[r][i].after[j] >= 0) shared[r][i].after[j] = place[shared[r][i].from[j]][shared[r][i].after[j]];

  // sums on their way that the rank would store, read once and overwrite
  for (int r = 0; r < n; r++) {
    std::vector<Action>& as = next[r].actions;
    size_t busy = 0;                                  // one at a time
    for (size_t i = 0; i < as.size(); i++) {
      Action& a = as[i];
      if (i < busy || a.dst_buf == BUF_NONE || a.n_send == 0) continue;
      size_t k = i + 1;
      for (; k < as.size(); k++)
        if (touches(as[k].dst_buf, as[k].dst_off, as[k].count, a.dst_buf, a.dst_off, a.count) || touches(as[k].src_buf, as[k].src_off, as[k].count, a.dst_buf, a.dst_off, a.count)) break;
      if (k == as.size()) continue;
      Action& b = as[k];
      if (b.src_buf != a.dst_buf || b.src_off != a.dst_off || b.dst_buf != a.dst_buf || b.dst_off != a.dst_off || b.count != a.count) continue;
      bool again = false;                             // the slot is this rank's until it sends to that peer again
      for (size_t q = i + 1; q <= k; q++) for (int j = 0; j < as[q].n_send; j++) again |= as[q].send_peer[j] == a.send_peer[0];
      if (again) continue;
      a.dst_buf = BUF_NONE; a.keep = 1; b.src_buf = BUF_KEPT;
      busy = k;
      any = true;
    }
  }
  if (!any) return false;

  // which elements come up again, other ranks' reads included
  for (int r = 0; r < n; r++) {
    std::vector<Action>& as = next[r].actions;
    auto elsewhere = [&](uint8_t buf, int64_t off, int64_t cnt) {
      for (int o = 0; o < n; o++)
        for (size_t i = 0; i < next[o].actions.size(); i++)
          for (int j = 0; j < next[o].actions[i].n_recv; j++)
            if (next[o].actions[i].recv_peer[j] == kSharedPeer && shared[o][i].from[j] == r && touches(shared[o][i].buf[j], shared[o][i].off[j], next[o].actions[i].count, buf, off, cnt)) return true;
      return false;
    };
    for (size_t i = 0; i < as.size(); i++) {
      Action& a = as[i];
      if ((a.flags & ACT_SRC_DONE) && elsewhere(a.src_buf, a.src_off, a.count)) a.flags &= (uint8_t)~ACT_SRC_DONE;
      if ((a.flags & ACT_DST_DONE) && elsewhere(a.dst_buf, a.dst_off, a.count)) a.flags &= (uint8_t)~ACT_DST_DONE;
    }
  }
  progs = std::move(next);
  return true;
}

bool nothing_waits(const std::vector<Program>& progs, const std::vector<std::vector<SharedOps>>& shared) {
  for (size_t r = 0; r < progs.size(); r++)
    for (size_t i = 0; i < progs[r].actions.size(); i++) {
      const Action& a = progs[r].actions[i];
      if (a.dst_buf != BUF_OUT || a.n_send || (a.src_buf != BUF_NONE && a.src_buf != BUF_IN)) return false;
      for (int j = 0; j < a.n_recv; j++) if (a.recv_peer[j] != kSharedPeer || shared[r][i].after[j] >= 0 || shared[r][i].buf[j] == BUF_SCRATCH) return false;
    }
  return true;
}

// The same for the low-latency variant, whose entries carry their own flags and which has no progress counters: what stands in a buffer before the call is read there, and
// every other value goes from the action that makes it straight to all that use it, instead of being handed on.
bool share_lines(std::vector<Program>& progs, std::vector<std::vector<SharedOps>>& shared) {
  const int n = (int)progs.size();
  Tracer t(progs);
  if (n < 2 || n > kMaxActionPeers + 1 || !t.match()) return false;
  // the action that makes the value which action i of rank r sends
  auto maker = [&](int r, int i) {
    Ref at{r, i};
    for (;;) {
      const Action& a = progs[at.rank].actions[at.act];
      if (a.n_recv == 1 && a.src_buf == BUF_NONE) at = t.producer[at.rank][at.act][0];
      else if (a.n_recv == 0 && a.src_buf != BUF_IN) {
        const int w = t.writer(at.rank, 0, at.act, a.src_buf, a.src_off, a.count);
        if (w < 0 || progs[at.rank].actions[w].dst_off != a.src_off || progs[at.rank].actions[w].count != a.count) return at;
        at.act = w;
      } else return at;
    }
  };
  std::vector<Program> next = progs;
  shared.assign(n, {});
  for (int r = 0; r < n; r++) { shared[r].resize(progs[r].actions.size()); for (Action& a : next[r].actions) a.n_send = 0; }
  bool any = false;
  std::vector<std::vector<std::vector<Ref>>> from(n);         // the entries that are left, by who takes them
  for (int r = 0; r < n; r++) {
    from[r].resize(progs[r].actions.size());
    for (size_t i = 0; i < progs[r].actions.size(); i++)
      for (int j = 0; j < progs[r].actions[i].n_recv; j++) {
        const Ref p = t.producer[r][i][j];
        const Origin o = t.origin(p.rank, p.act);
        if (o.ok && o.after < 0) {
          next[r].actions[i].recv_peer[j] = kSharedPeer;
          SharedOps& x = shared[r][i];
          x.buf[j] = o.buf; x.from[j] = (uint8_t)o.rank; x.off[j] = o.off; x.after[j] = -1;
          if (o.scaled) x.scaled |= (uint8_t)(1u << j);
          any = true;
          continue;
        }
        const Ref m = maker(p.rank, p.act);
        Action& a = next[m.rank].actions[m.act];
        if (m.rank == r || a.n_send == kMaxActionPeers) return false;
        for (int q = 0; q < a.n_send; q++) if (a.send_peer[q] == r) return false;
        a.send_peer[a.n_send++] = (uint8_t)r;
        next[r].actions[i].recv_peer[j] = (uint8_t)m.rank;
        from[r][i].push_back(m);
        any |= m.rank != p.rank || m.act != p.act;
      }
  }
  if (!any) return false;
  // entries of a connection are taken in the order in which they are sent, still
  for (int s = 0; s < n; s++)
    for (int d = 0; d < n; d++) {
      int last = -1;
      for (size_t i = 0; i < from[d].size(); i++) for (const Ref& m : from[d][i]) if (m.rank == s) { if (m.act <= last) return false; last = m.act; }
    }
  for (int r = 0; r < n; r++) {
    std::vector<Action> kept;
    std::vector<SharedOps> ops;
    for (size_t i = 0; i < next[r].actions.size(); i++) {
      if (next[r].actions[i].dst_buf == BUF_NONE && next[r].actions[i].n_send == 0) continue;
      kept.push_back(next[r].actions[i]); ops.push_back(shared[r][i]);
    }
    next[r].actions = std::move(kept); shared[r] = std::move(ops);
  }
  progs = std::move(next);
  return true;
}

}  // namespace piccl

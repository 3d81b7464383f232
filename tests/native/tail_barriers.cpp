// Test harness (CPU): the named barriers of the dense tail's factorisation
// (tail_barriers.hpp) in every order in which the warps can come to them.
// A barrier's phase ends with the arrival of as many warps as take part,
// whichever they are, and releases those that wait. Loaded by
// tests/test_tail_barriers_cpu.py.
#include <algorithm>
#include <array>
#include <cstdint>
#include <set>
#include <vector>

#include "tail_barriers.hpp"

namespace {

struct Op {
  enum Kind { kArrive, kWait, kWrite, kRead } kind;
  int id;  // barrier; written or read: the column
};
struct Recorder {
  std::vector<Op> ops;
  void arrive(int id) { ops.push_back({Op::kArrive, id}); }
  void wait(int id) { ops.push_back({Op::kWait, id}); }
};

constexpr int kBars = 16;
struct State {
  std::array<uint8_t, 16> at{};       // next operation of each warp
  std::array<uint8_t, 16> blocked{};  // 1 + the barrier it waits at
  std::array<uint8_t, kBars> came{};  // arrivals in the barrier's phase
  bool operator<(const State& o) const {
    if (at != o.at) return at < o.at;
    if (blocked != o.blocked) return blocked < o.blocked;
    return came < o.came;
  }
};

}  // namespace

extern "C" {

// 0: every order ends, and every column is read only when it is complete;
// 1: an order in which no warp can go on; 2: a column used too early;
// 3: a barrier left with arrivals. one_barrier: all columns published at one
// barrier. states: orders looked at.
int tail_barriers_check(int n, int warps, int one_barrier, int64_t* states) {
  Recorder lead, follow;
  // the lead's next(c) takes column c + 1 with columns 0 .. c - 1 subtracted;
  // the others' subtract(c) needs column c scaled
  rpgo::tail_lead(
      n, lead, [&](int c) { lead.ops.push_back({Op::kWrite, c}); }, [&](int c) { lead.ops.push_back({Op::kRead, c - 1}); });
  rpgo::tail_follow(n, follow, [&](int c) {
    follow.ops.push_back({Op::kRead, c});
    follow.ops.push_back({Op::kWrite, c});
  });
  if (one_barrier)
    for (auto* r : {&lead, &follow})
      for (Op& o : r->ops)
        if (o.kind < Op::kWrite && o.id == rpgo::tail_published(1)) o.id = rpgo::tail_published(0);
  // columns that the operations before position k have written
  auto writes = [](const std::vector<Op>& ops) {
    std::vector<int> w(ops.size() + 1, 0);
    for (size_t k = 0; k < ops.size(); ++k) w[k + 1] = w[k] + (ops[k].kind == Op::kWrite);
    return w;
  };
  const std::vector<int> lead_w = writes(lead.ops), follow_w = writes(follow.ops);
  auto ops = [&](int w) -> const std::vector<Op>& { return w == 0 ? lead.ops : follow.ops; };
  std::set<State> seen;
  std::vector<State> todo{State{}};
  seen.insert(State{});
  int bad = 0;
  while (!todo.empty() && !bad) {
    const State s = todo.back();
    todo.pop_back();
    bool moved = false, done = true;
    for (int w = 0; w < warps && !bad; ++w) {
      if (s.at[w] == ops(w).size()) continue;
      done = false;
      if (s.blocked[w]) continue;
      moved = true;
      State t = s;
      const Op o = ops(w)[s.at[w]];
      if (o.kind == Op::kRead) {
        if (w == 0) {
          for (int v = 1; v < warps; ++v) bad = follow_w[s.at[v]] < o.id + 1 ? 2 : bad;
        } else if (lead_w[s.at[0]] < o.id + 1) {
          bad = 2;
        }
      }
      if (o.kind == Op::kRead || o.kind == Op::kWrite) {
        ++t.at[w];
      } else {
        if (o.kind == Op::kArrive) ++t.at[w];
        else t.blocked[w] = (uint8_t)(1 + o.id);
        if (++t.came[o.id] == warps) {
          t.came[o.id] = 0;
          for (int v = 0; v < warps; ++v)
            if (t.blocked[v] == 1 + o.id) {
              t.blocked[v] = 0;
              ++t.at[v];
            }
        }
      }
      // the other warps are alike: one order of them
      std::vector<std::array<uint8_t, 2>> rest;
      for (int v = 1; v < warps; ++v) rest.push_back({t.at[v], t.blocked[v]});
      std::sort(rest.begin(), rest.end());
      for (int v = 1; v < warps; ++v) t.at[v] = rest[v - 1][0], t.blocked[v] = rest[v - 1][1];
      if (seen.insert(t).second) todo.push_back(t);
    }
    if (!bad && !moved && !done) bad = 1;
    if (!bad && done)
      for (int b = 0; b < kBars; ++b)
        if (s.came[b]) bad = 3;
  }
  *states = (int64_t)seen.size();
  return bad;
}
}

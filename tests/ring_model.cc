// Model of the decode step kernel's ring: a producer that asks for boxes a pass at a time, warps that consume them at
// random speeds, barriers that are waited on by phase parity.  Checks that no wait ever passes in a phase other than its own
// and that every position finds its own box.  With UNORDERED lanes ask as soon as their own stage is free.
// ring_model <stages> <runs> <seed>: 0 if all runs are right, 1 and the first fault otherwise.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "ring_order.h"

namespace {

constexpr int kWarps = 11;

struct Barrier {
  int completed = 0;  // phases
  bool passes(int parity) const { return ((completed + 1) & 1) == parity; }  // the phase before the present one has it
};

struct Op {
  bool attention;
  int n;  // boxes, or tiles (two to an item)
};

struct Model {
  int S;
  std::vector<Op> ops;
  std::mt19937 rng;
  std::vector<Barrier> full, empty;
  std::vector<int> content;            // position whose box the stage holds
  std::vector<int> in_flight;          // positions asked for and not landed
  const char* fault = nullptr;
  int fault_at = 0;

  // producer
  int p_op = 0, p_base = 0, p_pos = 0;
  std::vector<char> pending;
  // warps
  struct Warp {
    int op = 0, at = -1;   // place within its own sequence of the op
    int step = 0;          // see consume()
    int busy = 0;
    double speed = 1.0;
  } warps[kWarps];
  int ring_base[64];
  int finished = 0;        // warps that are through the present op

  Model(int stages, std::vector<Op> o, unsigned seed)
      : S(stages), ops(std::move(o)), rng(seed), full(stages), empty(stages), content(stages, -1), pending(stages) {
    int base = 0;
    for (size_t i = 0; i < ops.size(); ++i) ring_base[i] = base, base += ops[i].n;
    for (Warp& w : warps) w.at = 0;
    const int slow = rng() % 4;
    for (int i = 0; i < slow; ++i) warps[rng() % kWarps].speed = 1.0 / (2 << rng() % 9);
    begin_pass();
  }
  void fail(const char* what, int pos) {
    if (fault == nullptr) fault = what, fault_at = pos;
  }
  void begin_pass() {
    while (p_op < static_cast<int>(ops.size()) && p_base >= ops[p_op].n) p_pos += ops[p_op].n, p_base = 0, ++p_op;
    for (int l = 0; l < S; ++l) pending[l] = p_op < static_cast<int>(ops.size()) && p_base + l < ops[p_op].n;
  }
  void produce() {
    if (p_op >= static_cast<int>(ops.size())) return;
    const Op& op = ops[p_op];
    const int ahead = op.attention ? 0 : S;
    unsigned ready = 0, waiting = 0;
    for (int l = 0; l < S; ++l) {
      if (!pending[l]) continue;
      const int at = p_pos + p_base + l, s = at % S, use = at / S;
      const bool free = empty[s].passes((use & 1) ^ 1);
      if (free && empty[s].completed != use) fail("a box asked for in a phase not its own", at);
      (free ? ready : waiting) |= 1u << l;
    }
    const int aw = mld::ring_attn_warps(S, kWarps);
    const int distance = op.attention ? mld::ring_attn_distance(S, aw) : mld::ring_distance(S, kWarps);
    bool left = false;
    for (int l = 0; l < S; ++l) {
      bool go = (ready >> l & 1u) != 0 && (p_base + l >= ahead || (ready & ((1u << l) - 1u)) == 0);
#ifndef UNORDERED
      go = go && (waiting & mld::ring_lanes_before(l, distance)) == 0;
#endif
      if (go) {
        pending[l] = 0;
        in_flight.push_back(p_pos + p_base + l);
      }
      left = left || pending[l];
    }
    (void)distance;
    if (!left) p_base += S, begin_pass();
  }
  void land() {
    if (in_flight.empty()) return;
    const size_t i = rng() % in_flight.size();
    const int pos = in_flight[i];
    in_flight.erase(in_flight.begin() + i);
    if (full[pos % S].completed != pos / S) fail("a box landed in a phase not its own", pos);
    content[pos % S] = pos;
    ++full[pos % S].completed;
  }
  bool wait_empty(int pos) {
    const Barrier& b = empty[pos % S];
    const int use = pos / S;
    if (!b.passes((use & 1) ^ 1)) return false;
    if (b.completed != use) fail("a release waited for in a phase not its own", pos);
    return true;
  }
  bool wait_full(int pos) {
    const Barrier& b = full[pos % S];
    if (!b.passes((pos / S) & 1)) return false;
    if (b.completed != pos / S + 1 || content[pos % S] != pos) fail("a box consumed that is not the position's", pos);
    return true;
  }
  void consume(int wi) {
    Warp& w = warps[wi];
    if (w.op >= static_cast<int>(ops.size())) return;
    if (w.busy > 0) {
      --w.busy;
      return;
    }
    const Op& op = ops[w.op];
    const int aw = mld::ring_attn_warps(S, kWarps);
    const int unit = op.attention ? 2 : 1, across = op.attention ? aw : kWarps;
    const int rel = unit * (w.at * across + wi);
    if (wi >= across || rel >= op.n) {  // through with the op: the warps meet
      if (w.step != 100) w.step = 100, ++finished;
      if (finished == kWarps) {
        finished = 0;
        for (Warp& o : warps) ++o.op, o.at = 0, o.step = 0;
      }
      return;
    }
    const int pos = ring_base[w.op] + rel;
    // steps 2 u: the stage's last use released (beyond the op's first ring's length); 2 u + 1: its box there; then work
    if (w.step < 2 * unit) {
      const int u = w.step >> 1;
      const bool through = (w.step & 1) == 0 ? rel + u < S || wait_empty(pos + u) : wait_full(pos + u);
      if (through && ++w.step == 2 * unit) w.busy = rng() % 4;
      return;
    }
    // release (an item's two stages one after the other)
    ++empty[(pos + w.step - 2 * unit) % S].completed;
    if (++w.step == 3 * unit) w.step = 0, ++w.at;
  }
  bool run() {
    std::uniform_real_distribution<double> chance(0.0, 1.0);
    const double land_rate = chance(rng) < 0.5 ? 1.0 : 0.3;
    for (long tick = 0; fault == nullptr; ++tick) {
      bool all = true;
      for (const Warp& w : warps) all = all && w.op >= static_cast<int>(ops.size());
      if (all) return true;
      if (tick > 2000000) fail("nothing moves", 0);
      produce();
      for (int i = 0; i < 4; ++i)
        if (chance(rng) < land_rate) land();
      for (int i = 0; i < kWarps; ++i)
        if (chance(rng) < warps[i].speed) consume(i);
    }
    return false;
  }
};

}  // namespace

int main(int argc, char** argv) {
  if (argc != 4) return 2;
  const int stages = atoi(argv[1]), runs = atoi(argv[2]);
  std::mt19937 rng(atoi(argv[3]));
  for (int r = 0; r < runs; ++r) {
    std::vector<Op> ops;
    for (int o = 0; o < 5; ++o) {
      const bool attention = rng() % 3 == 0;
      const int n = rng() % (6 * stages);
      ops.push_back({attention, attention ? n / 2 * 2 : n});
    }
    Model m(stages, ops, rng());
    if (!m.run()) {
      printf("run %d of %d stages: %s (position %d)\n", r, stages, m.fault, m.fault_at);
      return 1;
    }
  }
  return 0;
}

// The pass planner (everett_gb300/csrc/ev_tile.cuh, plan_passes) on the host.
//
// "same": its passes against the rule written out over a list that is copied
// from pass to pass, on random circuits of every op kind, in circuit order
// and reordered.
// "time": ns per gate of plans of 10 000 and of 400 000 gates.
// "tiles SMS": the default tile bits of every register, complex128 and complex64.
#include <chrono>
#include <cstdio>
#include <cstring>
#include <random>

#include "ev_tile.cuh"

using namespace ev;

namespace {

struct Builder {
  std::vector<ev_op> ops;
  std::vector<uint64_t> pool;
  ev_circuit circuit(int n) const {
    ev_circuit c{};
    c.num_qubits = uint64_t(n);
    c.ops = ops.data();
    c.nops = ops.size();
    c.ctrl_pool = pool.data();
    return c;
  }
  void one(int q, double re, double im) {
    ev_op o{};
    o.kind = EV_OP_APPLY1;
    o.q0 = uint32_t(q);
    o.m[0] = re, o.m[1] = im, o.m[6] = re, o.m[7] = -im;
    ops.push_back(o);
  }
  void controlled(int t, std::vector<int> ctrls) {
    ev_op o{};
    o.kind = EV_OP_CONTROLLED;
    o.q0 = uint32_t(t);
    o.nctrl = uint32_t(ctrls.size());
    o.ctrl_off = uint32_t(pool.size());
    for (int q : ctrls) pool.push_back(uint64_t(q));
    o.m[0] = 0.6, o.m[2] = -0.8, o.m[4] = 0.8, o.m[6] = 0.6;
    ops.push_back(o);
  }
  // 0 CNOT, 1 CZ, 2 SWAP, 3 diagonal
  void two(int kind, int a, int b) {
    ev_op o{};
    o.kind = EV_OP_APPLY2;
    o.q0 = uint32_t(a);
    o.q1 = uint32_t(b);
    const int to[4][4] = {{0, 1, 3, 2}, {0, 1, 2, 3}, {0, 2, 1, 3}, {0, 1, 2, 3}};
    for (int r = 0; r < 4; ++r) o.m[2 * (4 * r + to[kind][r])] = 1.0;
    if (kind == 1) o.m[30] = -1.0;
    if (kind == 3) o.m[0] = 0.6, o.m[1] = 0.8;
    ops.push_back(o);
  }
};

bool rule_moves(const ev_op& o) {
  if (o.kind != EV_OP_APPLY2) return false;
  Builder b;
  for (int kind = 0; kind < 3; ++kind) b.two(kind, 0, 1);
  for (const ev_op& m : b.ops)
    if (std::memcmp(m.m, o.m, sizeof(o.m)) == 0) return true;
  return false;
}

std::vector<Pass> rule(const ev_circuit* c, int n, int k, int L, uint64_t max_ops, bool reorder) {
  std::vector<Pass> out;
  std::vector<uint64_t> pending, rest;
  std::vector<char> moves;
  for (uint64_t j = 0; j < c->nops; ++j) {
    pending.push_back(j);
    moves.push_back(rule_moves(c->ops[j]));
  }
  while (!pending.empty()) {
    Pass p;
    uint64_t set = (uint64_t(1) << L) - 1, blocked = 0;
    bool behind = false;
    rest.clear();
    for (uint64_t j : pending) {
      const ev_op& o = c->ops[j];
      uint64_t data = uint64_t(1) << o.q0;
      if (o.kind == EV_OP_APPLY2) data |= uint64_t(1) << o.q1;
      uint64_t all = data;
      for (uint32_t i = 0; o.kind == EV_OP_CONTROLLED && i < o.nctrl; ++i)
        all |= uint64_t(1) << c->ctrl_pool[o.ctrl_off + i];
      const bool may_jump = reorder || moves[j] || !behind;
      if ((reorder || rest.size() < kPlanWindow) && p.ops.size() < max_ops && !(all & blocked) &&
          may_jump && __builtin_popcountll(set | data) <= k) {
        set |= data;
        p.ops.push_back(j);
      } else {
        blocked |= all;
        behind = behind || !moves[j];
        rest.push_back(j);
      }
    }
    for (int q = 0; q < n && __builtin_popcountll(set) < k; ++q) set |= uint64_t(1) << q;
    p.tset = set;
    out.push_back(p);
    pending.swap(rest);
  }
  return out;
}

// idle: a qubit that no op touches
Builder random_circuit(std::mt19937_64& rng, int n, int count, int idle) {
  Builder b;
  auto qubit = [&](uint64_t avoid) {
    for (;;) {
      const int q = int(rng() % uint64_t(n));
      if (q != idle && !((avoid >> q) & 1)) return q;
    }
  };
  for (int i = 0; i < count; ++i) {
    const int kind = int(rng() % 8), a = qubit(0), d = qubit(uint64_t(1) << a);
    if (kind < 3) b.one(a, 0.6, 0.8);
    else if (kind == 3) b.controlled(a, {d, qubit((uint64_t(1) << a) | (uint64_t(1) << d))});
    else b.two(kind - 4, a, d);
  }
  return b;
}

// rotations on every qubit, then a brick of CNOTs
Builder layers(int n, size_t gates, int idle) {
  Builder b;
  for (int d = 0; b.ops.size() < gates; ++d) {
    for (int q = 0; q < n; ++q)
      for (int r = 0; r < 3 && q != idle; ++r) b.one(q, 0.6, 0.8);
    for (int q = d & 1; q + 1 < n; q += 2)
      if (q != idle && q + 1 != idle) b.two(0, q, q + 1);
  }
  return b;
}

int same() {
  std::mt19937_64 rng(7);
  int bad = 0, cases = 0;
  auto check = [&](const Builder& b, int n, int k, int L, uint64_t max_ops, bool reorder) {
    const ev_circuit c = b.circuit(n);
    const std::vector<Pass> got = plan_passes(&c, 0, c.nops, n, k, L, max_ops, reorder);
    const std::vector<Pass> want = rule(&c, n, k, L, max_ops, reorder);
    bool ok = got.size() == want.size();
    for (size_t i = 0; ok && i < got.size(); ++i)
      ok = got[i].ops == want[i].ops && got[i].tset == want[i].tset;
    ++cases;
    bad += !ok;
  };
  for (int n : {4, 5, 9, 14, 26})
    for (int k : {4, 8, 12}) {
      if (k > n) continue;
      for (bool reorder : {false, true})
        for (uint64_t max_ops : {uint64_t(48), ~uint64_t(0)})
          for (int idle : {-1, n - 1}) {
            check(random_circuit(rng, n, 600, idle), n, k, 2, max_ops, reorder);
            check(layers(n, 800, idle), n, k, 2, max_ops, reorder);
          }
    }
  // beyond the window: a long run of ops that cannot join stands before one
  // that could
  for (bool reorder : {false, true}) {
    Builder b;
    for (size_t i = 0; i < kPlanWindow + 300; ++i) b.two(i & 1 ? 0 : 2, 8, 9 + (i & 3));
    for (int q = 0; q < 6; ++q) b.two(0, q, q + 1);
    check(b, 13, 4, 2, 48, reorder);
    Builder w = layers(13, 2 * kPlanWindow, -1);  // one pass whatever its length
    check(w, 13, 13, 2, ~uint64_t(0), reorder);
  }
  std::printf("%d plans, %d differ\n", cases, bad);
  return bad != 0;
}

double ns_per_gate(int n, int k, size_t gates, int idle, bool reorder) {
  const Builder b = layers(n, gates, idle);
  const ev_circuit c = b.circuit(n);
  double best = 1e300;
  for (int i = 0; i < (gates < 100000 ? 5 : 2); ++i) {
    const auto t = std::chrono::steady_clock::now();
    const std::vector<Pass> p = plan_passes(&c, 0, c.nops, n, k, 2, 48, reorder);
    const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count();
    if (s < best && !p.empty()) best = s;
  }
  return best * 1e9 / double(b.ops.size());
}

int times() {
  for (int n : {10, 17, 26})
    for (int idle : {-1, n - 2})
      for (bool reorder : {false, true}) {
        const int k = n <= 17 ? 8 : 12;
        std::printf("%d %d %d %.1f %.1f\n", n, idle, int(reorder),
                    ns_per_gate(n, k, 10000, idle, reorder), ns_per_gate(n, k, 400000, idle, reorder));
      }
  return 0;
}

}  // namespace

int main(int argc, char** argv) {
  if (argc > 2 && std::strcmp(argv[1], "tiles") == 0) {
    for (int n = 1; n <= 34; ++n)
      std::printf("%d %d %d\n", n, default_tile_bits(EV_C128, n, std::atoi(argv[2])),
                  default_tile_bits(EV_C64, n, std::atoi(argv[2])));
    return 0;
  }
  return argc > 1 && std::strcmp(argv[1], "time") == 0 ? times() : same();
}

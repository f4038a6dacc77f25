// The fused planner's arithmetic (everett_gb300/csrc/ev_fuse.h): a block's
// unitary after random gate records, entry by entry, against the rounding it
// states written out with std::fma.  Prints the entries that differ.
#include <cstdio>
#include <cstring>
#include <random>

#include "ev_fuse.h"

using ev::apply_to_unitary;
using cd = std::complex<double>;

namespace {

double re_of(cd m, cd x) { return std::fma(m.real(), x.real(), -(m.imag() * x.imag())); }
double im_of(cd m, cd x) { return std::fma(m.imag(), x.real(), m.real() * x.imag()); }
double im_first(cd m, cd x) { return std::fma(m.real(), x.imag(), m.imag() * x.real()); }

cd entry(const ev_op& o, int i) { return cd(o.m[2 * i], o.m[2 * i + 1]); }

// qubit q is local bit q
void plain(const ev_circuit* c, const ev_op& o, int d, std::vector<cd>* U) {
  std::vector<cd> out = *U;
  uint64_t ctrl = 0;
  for (uint32_t j = 0; o.kind == EV_OP_CONTROLLED && j < o.nctrl; ++j)
    ctrl |= uint64_t(1) << c->ctrl_pool[o.ctrl_off + j];
  for (int row = 0; row < d; ++row)
    for (int col = 0; col < d; ++col) {
      double re = 0.0, im = 0.0;
      if (o.kind == EV_OP_APPLY2) {
        const int r = 2 * ((row >> o.q0) & 1) + ((row >> o.q1) & 1);
        for (int k = 0; k < 4; ++k) {
          const int from = (row & ~(1 << o.q0) & ~(1 << o.q1)) | ((k >> 1) << o.q0) | ((k & 1) << o.q1);
          const cd m = entry(o, 4 * r + k), x = (*U)[size_t(from) * d + col];
          re += re_of(m, x);
          im += r == 0 ? im_first(m, x) : im_of(m, x);
        }
      } else {
        if ((uint64_t(row) & ctrl) != ctrl) continue;
        const int r = (row >> o.q0) & 1, r0 = row & ~(1 << o.q0);
        const cd x = (*U)[size_t(r0) * d + col], y = (*U)[size_t(r0 | (1 << o.q0)) * d + col];
        re = re_of(entry(o, 2 * r), x) + re_of(entry(o, 2 * r + 1), y);
        im = im_of(entry(o, 2 * r), x) + im_of(entry(o, 2 * r + 1), y);
      }
      out[size_t(row) * d + col] = cd(re, im);
    }
  *U = out;
}

}  // namespace

int main() {
  std::mt19937_64 rng(3);
  std::normal_distribution<double> normal;
  long entries = 0, differ = 0;
  for (int k = 2; k <= 6; ++k)
    for (int block = 0; block < 20; ++block) {
      const int d = 1 << k;
      std::vector<int> F;
      for (int q = 0; q < k; ++q) F.push_back(q);
      std::vector<uint64_t> pool;
      std::vector<cd> got(size_t(d) * d), want;
      for (cd& v : got) v = cd(normal(rng), normal(rng));
      want = got;
      for (int g = 0; g < 40; ++g) {
        ev_op o{};
        const int a = int(rng() % uint64_t(k)), b = (a + 1 + int(rng() % uint64_t(k - 1))) % k;
        const int kind = int(rng() % 6);
        o.q0 = uint64_t(a);
        o.q1 = uint64_t(b);
        if (kind < 2) {
          o.kind = EV_OP_APPLY1;
          for (int i = 0; i < 8; ++i) o.m[i] = 0.5 * normal(rng);
        } else if (kind == 2) {
          o.kind = EV_OP_CONTROLLED;
          o.nctrl = 1;
          o.ctrl_off = pool.size();
          pool.push_back(uint64_t(b));
          for (int i = 0; i < 8; ++i) o.m[i] = 0.5 * normal(rng);
        } else {
          o.kind = EV_OP_APPLY2;
          const int to[3][4] = {{0, 1, 3, 2}, {0, 1, 2, 3}, {0, 2, 1, 3}};
          if (kind == 3)  // dense, some entries zero
            for (int i = 0; i < 32; ++i) o.m[i] = rng() % 4 ? 0.4 * normal(rng) : 0.0;
          else if (kind == 4)
            for (int r = 0; r < 4; ++r) o.m[10 * r] = std::cos(0.3 + r), o.m[10 * r + 1] = std::sin(0.3 + r);
          else {
            const int p = int(rng() % 3);
            for (int r = 0; r < 4; ++r) o.m[2 * (4 * r + to[p][r])] = 1.0;
            if (p == 1) o.m[30] = -1.0;
          }
        }
        ev_circuit c{};
        c.ctrl_pool = pool.data();
        apply_to_unitary(&c, o, F, &got);
        plain(&c, o, d, &want);
      }
      for (size_t i = 0; i < got.size(); ++i) {
        ++entries;
        differ += !(got[i] == want[i]);
      }
    }
  std::printf("%ld entries, %ld differ\n", entries, differ);
  return differ != 0;
}

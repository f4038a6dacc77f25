// ev_fuse.h -- the fused planner's arithmetic on the host: gate records
// multiplied into a block's unitary, row by row.
//
// On rows of interleaved doubles: std::complex multiplies through a library
// call that checks for NaN, which made fusing the blocks of a 16-qubit run
// take longer than running them.  Every fused multiply-add is written out,
// so that the rounding is the same on every host and with every compiler
// (plain expressions are contracted one way or another, or not at all).  The
// forms, the first row of a 4x4 apart, are those that GCC gave the
// std::complex expressions on aarch64: a fused run's amplitudes are theirs to
// the last bit.
#pragma once

#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

#include "ev_internal.h"

namespace ev {

// Re and Im of (mr + i mi) (xr + i xi).  Both are x's real part times the one
// part of m plus its imaginary part times (-mi, mr): two lanes of one form.
inline double product_re(double mr, double mi, double xr, double xi) {
  return std::fma(mr, xr, -mi * xi);
}
inline double product_im(double mr, double mi, double xr, double xi) {
  return std::fma(mi, xr, mr * xi);
}

// (x, y) <- (m0 x + m1 y, m2 x + m3 y) over two rows of n complex values
inline void mix_rows(const double* m, double* __restrict__ x, double* __restrict__ y, int n) {
  const double a = m[0], ai = m[1], b = m[2], bi = m[3], c = m[4], ci = m[5], d = m[6], di = m[7];
  for (int i = 0; i < 2 * n; i += 2) {
    const double xr = x[i], xi = x[i + 1], yr = y[i], yi = y[i + 1];
    x[i] = product_re(a, ai, xr, xi) + product_re(b, bi, yr, yi);
    x[i + 1] = product_im(a, ai, xr, xi) + product_im(b, bi, yr, yi);
    y[i] = product_re(c, ci, xr, xi) + product_re(d, di, yr, yi);
    y[i + 1] = product_im(c, ci, xr, xi) + product_im(d, di, yr, yi);
  }
}

// Left-multiplies U (d x d, local bit i <-> F[i]) by one gate record: the
// gate combines whole rows of U.
inline void apply_to_unitary(const ev_circuit* c, const ev_op& op, const std::vector<int>& F,
                             std::vector<std::complex<double>>* U) {
  const int d = int(1u << F.size());
  auto loc = [&](uint64_t q) { return int(std::find(F.begin(), F.end(), int(q)) - F.begin()); };
  auto row = [&](int r) { return reinterpret_cast<double*>(U->data() + size_t(r) * d); };
  if (op.kind == EV_OP_APPLY2) {
    const int ba = 1 << loc(op.q0), bb = 1 << loc(op.q1);
    const Kind2 kind = classify2(op.m);
    double out[4][2 * 64];
    for (int base = 0; base < d; ++base) {
      if (base & (ba | bb)) continue;
      double* in[4] = {row(base), row(base | bb), row(base | ba), row(base | ba | bb)};
      if (kind == K2_CNOT || kind == K2_SWAP) {
        std::swap_ranges(in[2], in[2] + 2 * d, kind == K2_CNOT ? in[3] : in[1]);
        continue;
      }
      if (kind == K2_CZ) {
        for (int i = 0; i < 2 * d; ++i) in[3][i] = -in[3][i];
        continue;
      }
      for (int r = 0; r < 4; ++r) {
        std::fill(out[r], out[r] + 2 * d, 0.0);
        for (int k = 0; k < 4; ++k) {
          const double re = op.m[2 * (4 * r + k)], im = op.m[2 * (4 * r + k) + 1];
          if (re == 0.0 && im == 0.0) continue;
          const double* v = in[k];
          for (int i = 0; i < 2 * d; i += 2) {
            out[r][i] += product_re(re, im, v[i], v[i + 1]);
            out[r][i + 1] += r == 0 ? std::fma(re, v[i + 1], im * v[i]) : product_im(re, im, v[i], v[i + 1]);
          }
        }
      }
      for (int r = 0; r < 4; ++r) std::copy(out[r], out[r] + 2 * d, in[r]);
    }
    return;
  }
  const int tb = 1 << loc(op.q0);
  int cmask = 0;
  if (op.kind == EV_OP_CONTROLLED)
    for (uint32_t j = 0; j < op.nctrl; ++j) cmask |= 1 << loc(c->ctrl_pool[op.ctrl_off + j]);
  for (int i0 = 0; i0 < d; ++i0)
    if (!(i0 & tb) && (i0 & cmask) == cmask) mix_rows(op.m, row(i0), row(i0 | tb), d);
}

}  // namespace ev

// ev_stage.cuh -- runs of complex64 gate records applied to amplitudes held
// in registers, 16 a thread (tiles of 2^12 amplitudes and more in the tile
// pass, of 2^11 and more in the batched runner).
//
// A stage names four positions of the tile; each thread gathers the
// amplitudes that agree outside them, applies every record of the stage to
// them in circuit order and scatters them.  A record needs its moved positions (1-qubit target, CNOT target,
// both of a SWAP or a dense 4x4) among them; a position it only reads (a control, the bits a
// diagonal entry depends on) may also be a bit of the thread's index, where
// it selects threads or the entry.  So a whole ladder of controlled phases
// or a Trotter step's Rzz run rides along with the rotations around it.
//
// One shared-memory sweep and barrier per record is issue-bound: about 20
// instructions per amplitude and record, most of them index arithmetic and
// loop control (complex64 QFT pass, 25 qubits: 540 us for ~34 records against
// 80 us of HBM time).  Here a record costs its arithmetic plus ~45
// instructions of dispatch per 16 amplitudes (25-qubit QFT, device time 5.4
// -> 3.2 ms); 32 amplitudes a thread spill and leave half the warps (3.6 ms).
// A record waits ~10 branches for its case, though, so small tiles, where
// latency counts, keep the sweeps (14 qubits, depth 20: 0.22 ms against
// 0.27).  Every amplitude sees the operations of record-by-record application
// in the same order.
//
// Tiles are stored swizzled (the low four index bits xor the next four), so
// that gathers over low positions spread over the banks.
#pragma once

#include "ev_tile.cuh"

namespace ev {

constexpr int kStageBits = 4;
constexpr uint8_t K1_RX = 6;  // real diagonal, imaginary off-diagonal

// Where local amplitude l of a tile is stored (linear over xor, and its own
// inverse).
__device__ __forceinline__ uint32_t stage_slot(uint32_t l) { return l ^ ((l >> 4) & 15u); }

// Keeps the compiler from merging the cases of a switch whose bodies differ
// only in which registers they touch: merged, every operand becomes a chain
// of selects.
template <int TAG>
__device__ __forceinline__ void own_case() {
  asm volatile("// case %0" ::"n"(TAG));
}

// The updates below form every product that reads an amplitude before the
// sums that replace it, so a result can take its operand's register.  With
// the products interleaved (as the compiler orders the plain expressions)
// old and new values overlap, and the loop over records copied every
// amplitude back to its register: about 90 moves per record and thread,
// 43 % of all instructions.
__device__ __forceinline__ void formed(float& a, float& b) { asm volatile("" : "+f"(a), "+f"(b)); }
__device__ __forceinline__ void formed(float& a, float& b, float& c, float& d) {
  asm volatile("" : "+f"(a), "+f"(b), "+f"(c), "+f"(d));
}

// A plain exchange is renaming to the compiler, and the renamed registers of
// one case force copies of all 16 amplitudes onto every other case.
__device__ __forceinline__ void exchange(float2& x, float2& y) {
  float2 p = y, q = x;
  formed(p.x, p.y, q.x, q.y);
  x = p;
  y = q;
}

// x <- d x, as cmul
__device__ __forceinline__ void mul_to(float2 d, float2& x) {
  float t = __fmul_rn(d.y, x.y), u = __fmul_rn(d.y, x.x);
  formed(t, u);
  x.x = __fmaf_rn(d.x, x.x, -t);
  x.y = __fmaf_rn(d.x, x.y, u);
}
// x <- m0 x + m1 y, y <- m2 x + m3 y for real entries
__device__ __forceinline__ void real_to(float m0, float m1, float m2, float m3, float& x, float& y) {
  float p = __fmul_rn(m0, x), q = __fmul_rn(m1, y), r = __fmul_rn(m2, x), s = __fmul_rn(m3, y);
  formed(p, q, r, s);
  x = __fadd_rn(p, q);
  y = __fadd_rn(r, s);
}

// f on the register pairs that differ in bit POS (the rmask bits set in both).
template <int POS, int R, typename F>
__device__ __forceinline__ void reg_pairs(float2 (&a)[R], F f) {
  if constexpr ((1 << POS) < R) {
    own_case<POS>();
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (!((r >> POS) & 1)) f(a[r], a[r | (1 << POS)]);
    own_case<POS>();
  }
}
template <int POS, int R, typename F>
__device__ __forceinline__ void reg_pairs_masked(float2 (&a)[R], uint32_t rmask, F f) {
  if constexpr ((1 << POS) < R) {
    own_case<POS>();
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (!((r >> POS) & 1) && (uint32_t(r) & rmask) == rmask) f(a[r], a[r | (1 << POS)]);
    own_case<POS>();
  }
}
// f on the registers whose index has the bits of M.
template <int M, int R, typename F>
__device__ __forceinline__ void reg_subset(float2 (&a)[R], F f) {
  if constexpr (M < R) {
    own_case<M>();
#pragma unroll
    for (int r = 0; r < R; ++r)
      if ((r & M) == M) f(a[r]);
    own_case<M>();
  }
}
template <int POS, int R, typename F>
__device__ __forceinline__ void reg_half(float2 (&a)[R], F f) {
  reg_subset<1 << POS>(a, f);
}
template <int X, int Y, int R, typename F>
__device__ __forceinline__ void reg_quarter(float2 (&a)[R], F f) {
  reg_subset<(1 << X) | (1 << Y)>(a, f);
}
template <int R, typename F>
__device__ __forceinline__ void reg_masked(float2 (&a)[R], uint32_t mask, F f) {
#pragma unroll
  for (int r = 0; r < R; ++r)
    if ((uint32_t(r) & mask) == mask) f(a[r]);
}
// Registers with bit POS clear times d0, set times d1.
template <int POS, int R>
__device__ __forceinline__ void reg_diag(float2 (&a)[R], float2 d0, float2 d1) {
  if constexpr ((1 << POS) < R) {
    own_case<POS>();
#pragma unroll
    for (int r = 0; r < R; ++r) mul_to(((r >> POS) & 1) ? d1 : d0, a[r]);
    own_case<POS>();
  }
}
// Register r times entry 2 * bit Y + bit X of the diagonal of the 4x4 mm.
template <int X, int Y, int R>
__device__ __forceinline__ void reg_diag2(float2 (&a)[R], const double* mm) {
  if constexpr ((1 << Y) < R) {
    own_case<8 * Y + X>();
    const float2 e[4] = {ldm<float2>(mm, 0), ldm<float2>(mm, 5), ldm<float2>(mm, 10),
                         ldm<float2>(mm, 15)};
#pragma unroll
    for (int r = 0; r < R; ++r) mul_to(e[2 * ((r >> Y) & 1) + ((r >> X) & 1)], a[r]);
    own_case<8 * Y + X>();
  }
}
// The same with p0 at register bit POS and p1's bit, b1, among the threads.
template <int POS, int R>
__device__ __forceinline__ void reg_diag2_half(float2 (&a)[R], const double* mm, uint32_t b1) {
  reg_diag<POS>(a, ldm<float2>(mm, int(5u * b1)), ldm<float2>(mm, int(10u + 5u * b1)));
}
// Exchanges the registers that differ in bit T and have the control bit C.
template <int C, int T, int R, typename F>
__device__ __forceinline__ void reg_cnot(float2 (&a)[R], F f) {
  if constexpr ((1 << C) < R && (1 << T) < R) {
    own_case<8 * T + C>();
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (((r >> C) & 1) && !((r >> T) & 1)) f(a[r], a[r | (1 << T)]);
    own_case<8 * T + C>();
  }
}
template <int X, int Y, int R, typename F>
__device__ __forceinline__ void reg_swap(float2 (&a)[R], F f) {
  if constexpr ((1 << Y) < R) {
    own_case<8 * Y + X>();
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (((r >> X) & 1) && !((r >> Y) & 1)) f(a[r], a[r ^ (1 << X) ^ (1 << Y)]);
    own_case<8 * Y + X>();
  }
}

// What a staged record does to the registers, one jump-table case each: the
// base codes below plus a register bit, a register mask or a pair of bits.
// Position-by-position tests inside a switch on the kind took 13 branches a
// record.
enum StageCode : uint8_t {
  SC_NONE = 0,
  SC_CNOT = 1,            // + target bit: exchange (control, if any, among the threads)
  SC_DIAG = 5,            // + bit: times m0 / m3
  SC_RX = 9,              // + bit, as are the next three
  SC_REAL = 13,
  SC_DENSE = 17,
  SC_ANTI = 21,
  SC_DIAG_MASKED = 25,    // + bit: with register controls, as are the next four
  SC_RX_MASKED = 29,
  SC_REAL_MASKED = 33,
  SC_DENSE_MASKED = 37,
  SC_ANTI_MASKED = 41,
  SC_PHASE = 45,          // all registers times m3
  SC_PHASE_HALF = 46,     // + bit: those with the bit
  SC_PHASE_QUARTER = 50,  // + pair: those with both bits
  SC_PHASE_MASKED = 56,   // those with the control bits and the target bit
  SC_NEG = 57,            // all negated; + bit, + pair as above
  SC_NEG_HALF = 58,
  SC_NEG_QUARTER = 62,
  SC_TDIAG = 68,          // times m0 or m3 by the thread's bit
  SC_TDIAG_MASKED = 69,
  SC_CNOT_REG = 70,       // + 4 * target bit + control bit
  SC_SWAP = 86,           // + pair
  SC_DENSE2 = 92,
  SC_DIAG2 = 93,          // + pair: entry by both register bits, p0 the higher
  SC_DIAG2_HALF = 99,     // + bit of p0, p1 among the threads
  SC_DIAG2_THREAD = 103   // both among the threads
};
// Index 0..5 of an unordered pair of register bits x < y.
__host__ __device__ __forceinline__ int bit_pair(int x, int y) { return x + (y * (y - 1)) / 2; }

// One record on the R amplitudes whose local indices are l0 plus the stage's
// positions.  Fields as mark_stages leaves them.
template <int R, typename Op>
__device__ __forceinline__ void stage_record(float2 (&a)[R], uint32_t l0, const Op& op,
                                             const double* mats) {
  const uint32_t lmask = op.lmask;
  if ((l0 & lmask) != lmask) return;
  const double* mm = rec_m(op, mats);
  const uint32_t rmask = uint32_t(op.ins >> 8) & 15u;
  const float2 m0 = ldm<float2>(mm, 0), m1 = ldm<float2>(mm, 1);
  const float2 m2 = ldm<float2>(mm, 2), m3 = ldm<float2>(mm, 3);
  auto rx = [=](float2& x, float2& y) {
    float p = __fmul_rn(m1.y, y.y), q = __fmul_rn(m1.y, y.x);
    float r = __fmul_rn(m2.y, x.y), s = __fmul_rn(m2.y, x.x);
    formed(p, q, r, s);
    x.x = __fmaf_rn(m0.x, x.x, -p);
    x.y = __fmaf_rn(m0.x, x.y, q);
    y.x = __fmaf_rn(m3.x, y.x, -r);
    y.y = __fmaf_rn(m3.x, y.y, s);
  };
  auto real = [=](float2& x, float2& y) {
    real_to(m0.x, m1.x, m2.x, m3.x, x.x, y.x);
    real_to(m0.x, m1.x, m2.x, m3.x, x.y, y.y);
  };
  auto dense = [=](float2& x, float2& y) {
    float2 p = cmul(m0, x), q = cmul(m1, y), r = cmul(m2, x), s = cmul(m3, y);
    formed(p.x, p.y, q.x, q.y);
    formed(r.x, r.y, s.x, s.y);
    x = cadd(p, q);
    y = cadd(r, s);
  };
  auto anti = [=](float2& x, float2& y) {
    float2 p = cmul(m1, y), q = cmul(m2, x);
    formed(p.x, p.y, q.x, q.y);
    x = p;
    y = q;
  };
  auto both = [=](float2& x, float2& y) {
    mul_to(m0, x);
    mul_to(m3, y);
  };
  auto swap1 = [](float2& x, float2& y) { exchange(x, y); };
  auto times3 = [=](float2& x) { mul_to(m3, x); };
  auto negate = [](float2& x) { x = cneg(x); };
// the cases of an operation at each register bit, and at each pair of them
#define EV_BITS(code, fn, ...)                 \
  case code + 0: fn<0>(a, __VA_ARGS__); break; \
  case code + 1: fn<1>(a, __VA_ARGS__); break; \
  case code + 2: fn<2>(a, __VA_ARGS__); break; \
  case code + 3: fn<3>(a, __VA_ARGS__); break;
#define EV_PAIRS(code, fn, ...)                   \
  case code + 0: fn<0, 1>(a, __VA_ARGS__); break; \
  case code + 1: fn<0, 2>(a, __VA_ARGS__); break; \
  case code + 2: fn<1, 2>(a, __VA_ARGS__); break; \
  case code + 3: fn<0, 3>(a, __VA_ARGS__); break; \
  case code + 4: fn<1, 3>(a, __VA_ARGS__); break; \
  case code + 5: fn<2, 3>(a, __VA_ARGS__); break;
#define EV_CNOTS(t, c0, c1, c2)                                    \
  case SC_CNOT_REG + 4 * t + c0: reg_cnot<c0, t>(a, swap1); break; \
  case SC_CNOT_REG + 4 * t + c1: reg_cnot<c1, t>(a, swap1); break; \
  case SC_CNOT_REG + 4 * t + c2: reg_cnot<c2, t>(a, swap1); break;
  const int code = op.nins;
  switch (code) {
    EV_BITS(SC_CNOT, reg_pairs, swap1)
    EV_BITS(SC_DIAG, reg_diag, m0, m3)
    EV_BITS(SC_RX, reg_pairs, rx)
    EV_BITS(SC_REAL, reg_pairs, real)
    EV_BITS(SC_DENSE, reg_pairs, dense)
    EV_BITS(SC_ANTI, reg_pairs, anti)
    EV_BITS(SC_DIAG_MASKED, reg_pairs_masked, rmask, both)
    EV_BITS(SC_RX_MASKED, reg_pairs_masked, rmask, rx)
    EV_BITS(SC_REAL_MASKED, reg_pairs_masked, rmask, real)
    EV_BITS(SC_DENSE_MASKED, reg_pairs_masked, rmask, dense)
    EV_BITS(SC_ANTI_MASKED, reg_pairs_masked, rmask, anti)
    case SC_PHASE: reg_subset<0>(a, times3); break;
    EV_BITS(SC_PHASE_HALF, reg_half, times3)
    EV_PAIRS(SC_PHASE_QUARTER, reg_quarter, times3)
    case SC_PHASE_MASKED: {
      const uint32_t b = uint32_t(op.ins) & 15u;
      reg_masked(a, rmask | (b < 15u ? 1u << b : 0u), times3);
      break;
    }
    case SC_NEG: reg_subset<0>(a, negate); break;
    EV_BITS(SC_NEG_HALF, reg_half, negate)
    EV_PAIRS(SC_NEG_QUARTER, reg_quarter, negate)
    case SC_TDIAG:
    case SC_TDIAG_MASKED: {
      const float2 d = ((l0 >> op.p0) & 1u) ? m3 : m0;
      reg_masked(a, code == SC_TDIAG ? 0u : rmask, [=](float2& x) { mul_to(d, x); });
      break;
    }
    EV_CNOTS(0, 1, 2, 3)
    EV_CNOTS(1, 0, 2, 3)
    EV_CNOTS(2, 0, 1, 3)
    EV_CNOTS(3, 0, 1, 2)
    EV_PAIRS(SC_SWAP, reg_swap, swap1)
    case SC_DENSE2: {  // register bits 1 (p0) and 0 (p1), rows summed left to right
#pragma unroll
      for (int q = 0; q < R; q += 4) {
        float2 acc[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          acc[r] = cmul(ldm<float2>(mm, 4 * r), a[q]);
#pragma unroll
          for (int c = 1; c < 4; ++c) acc[r] = cadd(acc[r], cmul(ldm<float2>(mm, 4 * r + c), a[q + c]));
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          formed(acc[r].x, acc[r].y);
          a[q + r] = acc[r];
        }
      }
      break;
    }
    EV_PAIRS(SC_DIAG2, reg_diag2, mm)
    EV_BITS(SC_DIAG2_HALF, reg_diag2_half, mm, (l0 >> op.p1) & 1u)
    case SC_DIAG2_THREAD: {
      const uint32_t b0 = (l0 >> op.p0) & 1u, b1 = (l0 >> op.p1) & 1u;
      const float2 d = ldm<float2>(mm, int(5u * (2u * b0 + b1)));
      reg_subset<0>(a, [=](float2& x) { mul_to(d, x); });
      break;
    }
    default: break;  // SC_NONE
  }
#undef EV_BITS
#undef EV_PAIRS
#undef EV_CNOTS
}

// A stage of `run` records; `base` is the
// tile's base index (controls outside the tile).
template <typename Op>
__device__ __forceinline__ void tile_stage(float2* t, int k, const Op* ops, int run,
                                           const double* mats, uint64_t base) {
  constexpr int NB = kStageBits, R = 1 << NB;
  const uint32_t sorted = uint32_t(ops[0].ins >> 16) & 0xFFFFu;
  const uint32_t order = uint32_t(ops[0].ins >> 32) & 0xFFFFu;
  const int np = k < NB ? k : NB;
  uint32_t slot[NB];
#pragma unroll
  for (int i = 0; i < NB; ++i)
    slot[i] = i < np ? stage_slot(1u << ((order >> (4 * i)) & 15u)) : 0u;
  const uint32_t groups = 1u << (k - np);
  for (uint32_t g = threadIdx.x; g < groups; g += blockDim.x) {
    uint32_t l0 = g;
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (i < np) l0 = ins0(l0, int((sorted >> (4 * i)) & 15u));
    const uint32_t at = stage_slot(l0);
    float2 a[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      uint32_t off = 0;
#pragma unroll
      for (int i = 0; i < NB; ++i) off ^= (r >> i) & 1 ? slot[i] : 0u;
      a[r] = (r >> np) == 0 ? t[at ^ off] : make_float2(0.f, 0.f);
    }
#pragma unroll 1
    for (int j = 0; j < run; ++j) {
      const Op& op = ops[j];
      if ((base & op.emask) == op.emask) stage_record(a, l0, op, mats);  // uniform
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      uint32_t off = 0;
#pragma unroll
      for (int i = 0; i < NB; ++i) off ^= (r >> i) & 1 ? slot[i] : 0u;
      if ((r >> np) == 0) t[at ^ off] = a[r];
    }
  }
}

// ---- host -----------------------------------------------------------------------

// Positions a record moves: they have to be among the stage's.
inline uint32_t moved_positions(const TileOp& o) {
  switch (o.kind) {
    case T_1Q:
      return o.k1 == K1_DIAG || o.k1 == K1_PHASE || o.k1 == K1_IDENT ? 0u : 1u << o.p0;
    case T_CNOT: return 1u << o.p1;
    case T_SWAP:
    case T_DENSE2: return (1u << o.p0) | (1u << o.p1);
    default: return 0u;
  }
}
inline uint32_t read_positions(const TileOp& o) {
  return o.kind == T_1Q ? o.lmask | (1u << o.p0) : (1u << o.p0) | (1u << o.p1);
}

// The code for the registers with the bits of a mask: code (all), then one
// per bit, one per pair, and `masked` for larger masks.
inline uint8_t subset_code(uint32_t mask, uint8_t code, uint8_t masked) {
  const int n = popc(mask);
  if (n == 0) return code;
  const int lo = __builtin_ctz(mask), hi = 31 - __builtin_clz(mask);
  if (n == 1) return uint8_t(code + 1 + lo);
  return n == 2 ? uint8_t(code + 5 + bit_pair(lo, hi)) : masked;
}

// The code of a record whose p0, p1 and local controls sit at register bits
// b0, b1 (15: a thread bit) and rmask.
inline uint8_t stage_code(const TileOp& o, int b0, int b1, uint32_t rmask) {
  const uint32_t r0 = b0 < 15 ? 1u << b0 : 0u, r1 = b1 < 15 ? 1u << b1 : 0u;
  const int pair = b0 < 15 && b1 < 15 ? bit_pair(std::min(b0, b1), std::max(b0, b1)) : 0;
  switch (o.kind) {
    case T_1Q:
      switch (o.k1) {
        case K1_RX: return uint8_t((rmask ? SC_RX_MASKED : SC_RX) + b0);
        case K1_REAL: return uint8_t((rmask ? SC_REAL_MASKED : SC_REAL) + b0);
        case K1_DENSE: return uint8_t((rmask ? SC_DENSE_MASKED : SC_DENSE) + b0);
        case K1_ANTI: return uint8_t((rmask ? SC_ANTI_MASKED : SC_ANTI) + b0);
        case K1_PHASE: return subset_code(rmask | r0, SC_PHASE, SC_PHASE_MASKED);
        case K1_DIAG:
          if (b0 >= 15) return rmask ? SC_TDIAG_MASKED : SC_TDIAG;
          return uint8_t((rmask ? SC_DIAG_MASKED : SC_DIAG) + b0);
        default: return SC_NONE;
      }
    case T_CNOT: return uint8_t(b0 < 15 ? SC_CNOT_REG + 4 * b1 + b0 : SC_CNOT + b1);
    case T_CZ: return subset_code(r0 | r1, SC_NEG, SC_NONE);
    case T_SWAP: return uint8_t(SC_SWAP + pair);
    case T_DIAG2:
      if (b0 < 15 && b1 < 15) return uint8_t(SC_DIAG2 + pair);
      return uint8_t(b0 < 15 ? SC_DIAG2_HALF + b0 : SC_DIAG2_THREAD);
    default: return SC_DENSE2;
  }
}

// Cuts a complex64 pass's records (matrices already packed to f32) into
// stages of at most maxrun records: run on the first record
// of each (0 on the others), the stage code in nins, the thread-bit conditions
// in lmask, and in ins: bits 0-3 and 4-7 the register bit of p0 and p1 (15: a
// thread bit), 8-11 the register bits of the local controls, and on the first
// record 16-31 the stage's positions ascending, 32-47 in register-bit order.
inline void mark_stages(TileOp* ops, size_t nops, int k, size_t maxrun) {
  const int np = std::min(k, kStageBits);
  for (size_t j = 0; j < nops;) {
    uint32_t set = 0;
    int pos[kStageBits], cnt = 0;
    size_t e = j;
    int uses[16] = {};
    for (; e < nops && e - j < std::min<size_t>(maxrun, 255); ++e) {
      const TileOp& o = ops[e];
      const uint32_t need = moved_positions(o);
      // a dense 4x4 has its operands at register bits 1 and 0
      if (o.kind == T_DENSE2 && !(cnt == 0 || (cnt >= 2 && pos[0] == o.p1 && pos[1] == o.p0))) break;
      if (popc(set | need) > np) break;
      if (o.kind == T_DENSE2 && cnt == 0) {
        pos[cnt++] = o.p1;
        pos[cnt++] = o.p0;
      } else {
        for (int p = 0; p < k; ++p)
          if ((need & ~set) >> p & 1u) pos[cnt++] = p;
      }
      set |= need;
      for (int p = 0; p < k; ++p) uses[p] += int(read_positions(o) >> p & 1u);
    }
    // the rest: the positions the records read most (a register bit selects
    // registers, a thread bit idles lanes), high ones first
    while (cnt < np) {
      int best = -1;
      for (int p = k - 1; p >= 0; --p)
        if (!(set >> p & 1u) && (best < 0 || uses[p] > uses[best])) best = p;
      pos[cnt++] = best;
      set |= 1u << best;
    }
    uint64_t sorted = 0, order = 0;
    int s = 0;
    for (int p = 0; p < k; ++p)
      if (set >> p & 1u) sorted |= uint64_t(p) << (4 * s++);
    for (int i = 0; i < np; ++i) order |= uint64_t(pos[i]) << (4 * i);
    for (size_t i = j; i < e; ++i) {
      TileOp& o = ops[i];
      auto bit_of = [&](int p) {
        for (int b = 0; b < np; ++b)
          if (pos[b] == p) return b;
        return 15;
      };
      int b0 = bit_of(o.p0), b1 = o.kind == T_1Q ? 15 : bit_of(o.p1);
      // a diagonal takes its operands in either order: p0 at the higher
      // register bit, or the one that has a register bit
      if (o.kind == T_DIAG2 && (b0 == 15 || (b1 != 15 && b1 > b0)) && b1 != 15) {
        std::swap(b0, b1);
        std::swap(o.p0, o.p1);
        float f[32];  // entries 5 and 10 trade places
        std::memcpy(f, o.m, sizeof(f));
        std::swap(f[10], f[20]);
        std::swap(f[11], f[21]);
        std::memcpy(o.m, f, sizeof(f));
      }
      uint32_t rmask = 0;
      if (o.kind == T_1Q) {
        for (int b = 0; b < np; ++b)
          if (o.lmask >> pos[b] & 1u) rmask |= 1u << b;
        o.lmask &= ~set;
        if (o.k1 == K1_PHASE && b0 >= 15) o.lmask |= 1u << o.p0;
        if (o.k1 == K1_DENSE) {
          float f[8];
          std::memcpy(f, o.m, sizeof(f));
          if (f[1] == 0.f && f[7] == 0.f && f[2] == 0.f && f[4] == 0.f) o.k1 = K1_RX;
        }
      } else {
        o.lmask = 0;
        if ((o.kind == T_CNOT || o.kind == T_CZ) && b0 >= 15) o.lmask |= 1u << o.p0;
        if (o.kind == T_CZ && b1 >= 15) o.lmask |= 1u << o.p1;
      }
      o.nins = stage_code(o, b0, b1, rmask);
      o.ins = uint64_t(b0) | uint64_t(b1) << 4 | uint64_t(rmask) << 8;
      if (i == j) o.ins |= sorted << 16 | order << 32;
      o.run = uint8_t(i == j ? e - j : 0);
    }
    j = e;
  }
}

}  // namespace ev

// pfa_tile64.cuh -- tiles of the FP64 step kernels (2D, and 3D plane by plane).
// Included by .cu files only.
#pragma once

#include "pfa_device.cuh"

namespace pfa {
namespace {

using namespace dev;

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// A tile of TX x TY cells.  A warp owns a block of 8 x 4 of them: an FP64
// operation costs a warp the same whatever its active lanes, and a precipitate
// touches fewer compact blocks than rows of 32.  The warps past the tile's own
// stage its halo, so that a cell's solve and its update are never behind
// another cell's in the same warp; the corners only where the stencil reads
// them (an 8 x 8 tile's halo without them is one warp).
template <int TX_, int TY_, bool CORNERS>
struct Tile {
  static constexpr int TX = TX_, TY = TY_;
  static constexpr int EX = TX + 2, EY = TY + 2;  // staged cells
  // elements per staged row: 8 modulo 16, so that the two rows of 8 that a
  // half warp reads fall into different banks
  static constexpr int kPitch = (EX + 7) / 16 * 16 + 8;
  static constexpr int kOwn = TX * TY, kHalo = 2 * (TX + TY) + 4 * CORNERS;
  static constexpr int kThreads = kOwn + (kHalo + 31) / 32 * 32;
  static_assert(TX % 8 == 0 && TY % 4 == 0 && kPitch >= EX, "whole warp blocks");
  template <class T>
  using Plane = T[EY][kPitch];

  // this thread's cell (ex, ey) of the staged tile: its own output cell in the
  // first kOwn threads, a halo cell in the rest (false: none, a duplicate of
  // the last one)
  static __device__ __forceinline__ bool cell(int& ex, int& ey) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w < kOwn / 32) {
      ex = w % (TX / 8) * 8 + (lane & 7) + 1;
      ey = w / (TX / 8) * 4 + (lane >> 3) + 1;
      return true;
    }
    const int i = int(threadIdx.x) - kOwn, h = i < kHalo ? i : kHalo - 1;
    if (h < 2 * TX) {
      ey = h < TX ? 0 : TY + 1;
      ex = 1 + (h < TX ? h : h - TX);
    } else if (h < 2 * (TX + TY)) {
      const int k = h - 2 * TX;
      ey = 1 + (k < TY ? k : k - TY);
      ex = k < TY ? 0 : TX + 1;
    } else {
      const int k = h - 2 * (TX + TY);
      ey = k < 2 ? 0 : TY + 1;
      ex = k & 1 ? TX + 1 : 0;
    }
    return i < kHalo;
  }
};

// One staged cell: its values and x^gamma.  phase: the tile must look at the
// phases at all (an all-zero phase field stays zero: its Laplacian, p' and
// well vanish; compositions that are not finite make 0 x NaN, see kBigHi).
// g1, g2: x^gamma, the bits of its FP64 values or (FIXED, not wide) 2^58 times
// it.
struct Cell64 {
  double X, Y, pd, pl;
  long long g1, g2;
  double v1, v2;  // !HOT: x^gamma in FP64
  size_t i;       // element of the fields
  bool solved, phase, big;
  bool wide;  // FIXED: outside the range of the fixed-point sums
};

// a phase that solve_fixed takes: in [0, 1], or too small for p to count
__device__ __forceinline__ bool fraction(double v) {
  const unsigned hi = unsigned(__double2hiint(v));
  return mag_hi(v) < kSolveHi || hi < 0x3ff00000u || (hi == 0x3ff00000u && __double2loint(v) == 0);
}

// x^gamma of a cell next to a precipitate; take: in the range of solve_fixed;
// kinds: the forms of it that the warp needs; range: of the fixed-point sums.
// (A call: its registers would weigh on the cells that need none.)
struct Gamma64 {
  long long g1, g2;
  bool wide;
};
static __device__ __noinline__ Gamma64 gamma_cell(double X, double Y, double pd, double pl, bool take, int kinds,
                                                  Range60 range) {
  Gamma64 g;
  int64_t h1, h2;
  const uint64_t x = fix64(X) >> 1, y = fix64(Y) >> 1;
  const uint64_t fd = mag_hi(pd) < kSolveHi ? 0 : fix63(pd), fl = mag_hi(pl) < kSolveHi ? 0 : fix63(pl);
  if (take && (kinds == 3   ? solve_fixed<3>(x, y, fd, fl, h1, h2)
               : kinds == 1 ? solve_fixed<1>(x, y, fd, fl, h1, h2)
                            : solve_fixed<2>(x, y, fd, fl, h1, h2))) {
    g.wide = min(h1, h2) < range.low || max(h1, h2) >= range.most;
    g.g1 = g.wide ? __double_as_longlong(value60(h1)) : (h1 + 2) >> 2;
    g.g2 = g.wide ? __double_as_longlong(value60(h2)) : (h2 + 2) >> 2;
  } else {
    double g1, g2;
    gamma64(X, Y, pd, pl, g1, g2);
    g.wide = true;
    g.g1 = __double_as_longlong(g1);
    g.g2 = __double_as_longlong(g2);
  }
  return g;
}

// whole warp.  FIXED: x^gamma for the fixed-point sums; HOT: the solve in fixed
// point (else in FP64, inline: no call, so that a kernel with many waves of
// tiles without precipitate keeps its occupancy)
template <bool FIXED, bool HOT>
__device__ __forceinline__ Cell64 cell64(double X, double Y, double pd, double pl, Range60 range) {
  Cell64 c;
  c.X = X;
  c.Y = Y;
  c.pd = pd;
  c.pl = pl;
  const bool unit = in_unit(X) && in_unit(Y);
  c.big = !unit && max(mag_hi(X), mag_hi(Y)) >= kBigHi;
  const int m = max(mag_hi(pd), mag_hi(pl));
  c.phase = (m | __double2loint(pd) | __double2loint(pl)) != 0 || c.big;
  c.solved = m >= kSolveHi || c.big;
  c.wide = !FIXED || !unit;
  if constexpr (HOT) {
    c.g1 = c.wide ? __double_as_longlong(X) : fix58(X);
    c.g2 = c.wide ? __double_as_longlong(Y) : fix58(Y);
    if (__any_sync(0xffffffffu, c.solved)) {
      // next to a precipitate of one kind the other's fraction is below 10
      // 2^-70 and zero in fixed point
      const bool take = c.solved && unit && fraction(pd) && fraction(pl);
      const int kinds = int(__any_sync(0xffffffffu, take && mag_hi(pd) >= kSolveHi)) +
                        2 * int(__any_sync(0xffffffffu, take && mag_hi(pl) >= kSolveHi));
      if (c.solved) {
        const Gamma64 g = gamma_cell(X, Y, pd, pl, take, kinds, FIXED ? range : kRangeNone);
        c.g1 = g.g1;
        c.g2 = g.g2;
        c.wide = g.wide;
      }
    }
  } else {
    double g1 = X, g2 = Y;
    solve64(c.solved, c.big, X, Y, pd, pl, g1, g2);
    c.v1 = g1;
    c.v2 = g2;
    // (the bounds of the ranges used here have no low word)
    const int low = __double2hiint(double(-range.low) * 0x1p-60), most = __double2hiint(double(range.most) * 0x1p-60);
    auto out = [&](double g) { return mag_hi(g) >= (__double2hiint(g) < 0 ? low : most); };
    bool fixed = !c.wide;
    if (c.solved) {
      fixed = fixed && !out(g1) && !out(g2);
      c.g1 = fixed ? fix58_signed(g1) : __double_as_longlong(g1);
      c.g2 = fixed ? fix58_signed(g2) : __double_as_longlong(g2);
    } else {
      c.g1 = fixed ? fix58(X) : __double_as_longlong(X);
      c.g2 = fixed ? fix58(Y) : __double_as_longlong(Y);
    }
    c.wide = !fixed;
  }
  return c;
}

// x^gamma in FP64 from g1, g2 of its cell
__device__ __forceinline__ double2 gamma_values(const Cell64& c, long long g1, long long g2) {
  if (c.wide) return make_double2(__longlong_as_double(g1), __longlong_as_double(g2));
  return c.solved ? make_double2(value58(g1), value58(g2)) : make_double2(c.X, c.Y);
}

// the bits that are zero with a double (its sign aside)
__device__ __forceinline__ int value_bits(double v) { return mag_hi(v) | __double2loint(v); }

// Allen-Cahn of one phase of a cell.  none: the phase is zero at the cell and
// its neighbours, and stays so; lap() forms its Laplacian, gamma() its
// x^gamma.
template <int I, class Lap, class Gam>
__device__ __forceinline__ double phase64(const Coef64& K, const Cell64& c, bool none, Lap lap, Gam gamma) {
  if (none && !c.big) return 0.0;
  const double ph = I == 0 ? c.pd : c.pl, pj = I == 0 ? c.pl : c.pd;
  if (mag_hi(ph) < kLinearHi && mag_hi(pj) < kLoneHi && !c.big && K.linear)
    return allen_cahn_linear64<I>(K, ph, lap());
  constexpr double x1 = kXe[0][0], x2 = kXe[0][1];
  const double2 g = gamma();
  return allen_cahn64<I>(K, ph, pj, ph * pj, lap(), g.x - x1, g.y - x2);
}

}  // namespace
}  // namespace pfa

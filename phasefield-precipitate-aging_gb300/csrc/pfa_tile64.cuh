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
// well vanish; compositions that are not finite make 0 x NaN, see kBigHi)
struct Cell64 {
  double X, Y, pd, pl, g1, g2;
  size_t i;  // element of the fields
  bool solved, phase, big;
  bool unit;  // both compositions in [2^-11, 1)
};

// whole warp
__device__ __forceinline__ Cell64 cell64(double X, double Y, double pd, double pl) {
  Cell64 c;
  c.X = X;
  c.Y = Y;
  c.pd = pd;
  c.pl = pl;
  c.g1 = X;
  c.g2 = Y;
  c.unit = in_unit(X) && in_unit(Y);
  c.big = !c.unit && max(mag_hi(X), mag_hi(Y)) >= kBigHi;
  const int m = max(mag_hi(pd), mag_hi(pl));
  c.phase = (m | __double2loint(pd) | __double2loint(pl)) != 0 || c.big;
  c.solved = m >= kSolveHi || c.big;
  solve64(c.solved, c.big, X, Y, pd, pl, c.g1, c.g2);
  return c;
}

// outside the fixed-point forms' range, with |x^gamma| bounded by the high
// word `hi` (the neighbour sum has to stay below 2^5)
__device__ __forceinline__ bool wide64(const Cell64& c, int hi) {
  return !c.unit || (c.solved && max(mag_hi(c.g1), mag_hi(c.g2)) >= hi);
}

// x^gamma in fixed point (not wide)
__device__ __forceinline__ void fix_cell(const Cell64& c, long long& f1, long long& f2) {
  if (c.solved) {
    f1 = fix58_signed(c.g1);
    f2 = fix58_signed(c.g2);
  } else {
    f1 = fix58(c.X);
    f2 = fix58(c.Y);
  }
}

// the bits that are zero with a double (its sign aside)
__device__ __forceinline__ int value_bits(double v) { return mag_hi(v) | __double2loint(v); }

// Allen-Cahn of one phase of a cell.  none: the phase is zero at the cell and
// its neighbours, and stays so; lap() forms its Laplacian.
template <int I, class Lap>
__device__ __forceinline__ double phase64(const Coef64& K, const Cell64& c, bool none, Lap lap) {
  if (none && !c.big) return 0.0;
  const double ph = I == 0 ? c.pd : c.pl, pj = I == 0 ? c.pl : c.pd;
  if (mag_hi(ph) < kLinearHi && mag_hi(pj) < kLoneHi && !c.big)
    return allen_cahn_linear64<I>(K, ph, lap());
  constexpr double x1 = kXe[0][0], x2 = kXe[0][1];
  return allen_cahn64<I>(K, ph, pj, ph * pj, lap(), c.g1 - x1, c.g2 - x2);
}

}  // namespace
}  // namespace pfa

// pfa_rows.cuh -- the cells of a grid dealt to the warps of a launch.
// Included by .cu files only.
#pragma once

namespace pfa {
namespace {

// A warp takes pieces of 32 cells of a row, every W-th one (W: the launch's
// warps, numbered so that consecutive ones are in different blocks), which
// spreads the cells next to a precipitate, those that cost most; divisions per
// thread, none per cell.  Rows are (y, z).
struct RowWalk {
  unsigned chunks, Ny, Nz;
  unsigned c, y, z;     // the current piece
  unsigned dc, dy, dz;  // the step to the warp's next one
  __device__ RowWalk(int Nx, int Ny_, int Nz_, unsigned warp, unsigned warps) : Ny(Ny_), Nz(Nz_) {
    chunks = (Nx + 31) / 32;
    auto split = [&](unsigned u, unsigned& c, unsigned& y, unsigned& z) {
      const unsigned row = u / chunks;
      c = u - row * chunks;
      z = row / Ny;
      y = row - z * Ny;
    };
    split(warp, c, y, z);
    split(warps, dc, dy, dz);
  }
  __device__ bool more() const { return z < Nz; }
  __device__ void next() {
    c += dc;
    y += dy;
    z += dz;
    if (c >= chunks) {
      c -= chunks;
      y++;
    }
    if (y >= Ny) {
      y -= Ny;
      z++;
    }
  }
};

}  // namespace
}  // namespace pfa

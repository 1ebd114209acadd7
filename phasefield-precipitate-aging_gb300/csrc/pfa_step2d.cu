// pfa_step2d.cu -- 2D step kernels of libpfa_gb300 (sm_103a).
//
// One fused kernel per explicit Euler step replaces the reference's 29
// launches (src/main.cpp:289-305): zero-flux boundary fill, fictitious
// gamma compositions (src/discretization.cu:50-74), 5- or 9-point mask
// convolution (:550-603), Cahn-Hilliard (:843-886) and Allen-Cahn (:888-980).
// Each CTA stages one tile plus its one-cell halo in shared memory with
// x^gamma per staged cell, then forms the Laplacians and both updates of its
// interior cells.  Domain edges are handled by clamped (mirrored) indexing,
// which is what the reference's halo fill produces.
//
// The FP64 pipe bounds it (19 cycles per warp instruction and SM), so the
// arithmetic is in the reduced forms of pfa_device.cuh: no FP64 operations in
// a cell where both phases are exactly zero around it, 7 per phase in the
// phases' far tails, about 65 next to a precipitate (the reference's
// expressions: about 300 everywhere).  us a step with 4 particles: 4096^2 7780
// -> 248, 2048^2 1950 -> 65, 256^2 38.4 -> 6.1.
//
// Layout: the reference's, (Ny + 2) rows of pitch elements with a one-cell
// ghost ring, interior cell (x, y) at (y + 1) * pitch + x + 1.  The FP32
// precision form has its own kernel and layout (pfa_step2d_f32.cu).
#include <algorithm>
#include <cstdint>

#include "pfa_device.cuh"
#include "pfa_kernels.h"
#include "pfa_tile64.cuh"

namespace pfa {

using namespace dev;

namespace {

// The ghost cells that mirror interior cell (gx, gy) of the domain's edge
// (corners take the diagonal value).
__device__ __noinline__ void store_ghosts(double* f, int pitch, int gx, int gy, int Nx, int Ny, double v) {
  const size_t row = size_t(gy + 1) * pitch;
  const bool l = gx == 0, r = gx == Nx - 1, b = gy == 0, t = gy == Ny - 1;
  if (l) f[row] = v;
  if (r) f[row + Nx + 1] = v;
  if (b) {
    f[gx + 1] = v;
    if (l) f[0] = v;
    if (r) f[Nx + 1] = v;
  }
  if (t) {
    const size_t top = size_t(Ny + 1) * pitch;
    f[top + gx + 1] = v;
    if (l) f[top] = v;
    if (r) f[top + Nx + 1] = v;
  }
}

// the four new values of interior cell (gx, gy), element i of the fields
__device__ __forceinline__ void store_cell(const Step2DArgs& a, size_t i, int gx, int gy, double cr,
                                           double nb, double pd, double pl) {
  static_cast<double*>(a.out[0])[i] = cr;
  static_cast<double*>(a.out[1])[i] = nb;
  static_cast<double*>(a.out[2])[i] = pd;
  static_cast<double*>(a.out[3])[i] = pl;
  if (a.write_halo && (gx == 0 || gx == a.Nx - 1 || gy == 0 || gy == a.Ny - 1)) {
    const double v[4] = {cr, nb, pd, pl};
#pragma unroll
    for (int k = 0; k < 4; k++)
      store_ghosts(static_cast<double*>(a.out[k]), a.pitch, gx, gy, a.Nx, a.Ny, v[k]);
  }
}

// ---------------------------------------------------------------------------
// Plain FP64 fused step over tiles of pfa_tile64.cuh.  MASK: the kind of
// Coef64::mask.
// Laplacian (iso masks: over the weight, which Coef64 folds into its factors)
template <int MASK, int P>
__device__ __forceinline__ double lap64(const Step2DArgs& a, const double (*s)[P], int ex, int ey) {
  if constexpr (MASK == kMaskIso) {
    return fma(a.c.iso_c, s[ey][ex],
               (s[ey - 1][ex] + s[ey + 1][ex]) + (s[ey][ex - 1] + s[ey][ex + 1]));
  } else if constexpr (MASK == kMaskFive) {
    double v = a.m.mask[0] * s[ey - 1][ex];
    v = fma(a.m.mask[1], s[ey][ex - 1], v);
    v = fma(a.m.mask[2], s[ey][ex], v);
    v = fma(a.m.mask[3], s[ey][ex + 1], v);
    return fma(a.m.mask[4], s[ey + 1][ex], v);
  } else if constexpr (MASK == kMaskIso9) {
    const double f = (s[ey - 1][ex] + s[ey + 1][ex]) + (s[ey][ex - 1] + s[ey][ex + 1]);
    const double k = (s[ey - 1][ex - 1] + s[ey + 1][ex + 1]) + (s[ey - 1][ex + 1] + s[ey + 1][ex - 1]);
    return fma(a.c.iso_c, s[ey][ex], fma(4.0, f, k));
  } else {
    double v = a.mask9[0] * s[ey - 1][ex - 1];
    v = fma(a.mask9[1], s[ey - 1][ex], v);
    v = fma(a.mask9[2], s[ey - 1][ex + 1], v);
    v = fma(a.mask9[3], s[ey][ex - 1], v);
    v = fma(a.mask9[4], s[ey][ex], v);
    v = fma(a.mask9[5], s[ey][ex + 1], v);
    v = fma(a.mask9[6], s[ey + 1][ex - 1], v);
    v = fma(a.mask9[7], s[ey + 1][ex], v);
    return fma(a.mask9[8], s[ey + 1][ex + 1], v);
  }
}

// the same over a staged fixed-point array (iso masks; exact)
template <int MASK, int P>
__device__ __forceinline__ long long sum58(const long long (*s)[P], int ex, int ey) {
  const long long f = (s[ey - 1][ex] + s[ey + 1][ex]) + (s[ey][ex - 1] + s[ey][ex + 1]);
  if constexpr (MASK == kMaskIso) return f - 4 * s[ey][ex];
  const long long k = (s[ey - 1][ex - 1] + s[ey + 1][ex + 1]) + (s[ey - 1][ex + 1] + s[ey + 1][ex - 1]);
  return 4 * f + k - 20 * s[ey][ex];
}

// whether a staged phase is zero at a cell and all its neighbours
template <int MASK, int P>
__device__ __forceinline__ bool none64(const double (*s)[P], int ex, int ey) {
  auto b = [&](int y, int x) { return value_bits(s[y][x]); };
  int m = b(ey, ex) | b(ey - 1, ex) | b(ey + 1, ex) | b(ey, ex - 1) | b(ey, ex + 1);
  if constexpr (MASK == kMaskIso9 || MASK == kMaskNine)
    m |= b(ey - 1, ex - 1) | b(ey - 1, ex + 1) | b(ey + 1, ex - 1) | b(ey + 1, ex + 1);
  return m == 0;
}

template <bool FIXED, bool HOT>
__device__ __forceinline__ Cell64 stage64(const Step2DArgs& a, int gx, int gy, Range60 range) {
  const size_t i = size_t(clampi(gy, 0, a.Ny - 1) + 1) * a.pitch + clampi(gx, 0, a.Nx - 1) + 1;
  Cell64 c = cell64<FIXED, HOT>(__ldg(static_cast<const double*>(a.in[0]) + i),
                           __ldg(static_cast<const double*>(a.in[1]) + i),
                           __ldg(static_cast<const double*>(a.in[2]) + i),
                           __ldg(static_cast<const double*>(a.in[3]) + i), range);
  c.i = i;
  return c;
}

// Allen-Cahn of both phases, src/discretization.cu:888-980
template <int MASK, int P, class Gam>
__device__ __forceinline__ void update_phases(const Step2DArgs& a, const Cell64& c, const double (*s_pd)[P],
                                              const double (*s_pl)[P], int ex, int ey, Gam gamma,
                                              double& od, double& ol) {
  od = phase64<0>(a.c, c, none64<MASK>(s_pd, ex, ey), [&] { return lap64<MASK>(a, s_pd, ex, ey); }, gamma);
  ol = phase64<1>(a.c, c, none64<MASK>(s_pl, ex, ey), [&] { return lap64<MASK>(a, s_pl, ex, ey); }, gamma);
}

// tile rows past what a grid's second dimension holds go on in the third
// (tiles past the domain store nothing)
__device__ __forceinline__ int tile_row() { return int(blockIdx.z * gridDim.y + blockIdx.y); }

template <int MASK, int TX, int TY>
using Tile2 = Tile<TX, TY, MASK == kMaskIso9 || MASK == kMaskNine>;
// resident blocks asked for: 1152 threads per SM (56 registers), 1408 (46)
constexpr int blocks2(int threads, bool hot) { return (hot ? 1152 : 1408) / threads; }

// MASK: Coef64::mask.  HOT: see cell64.  Bound by the FP64 pipe next to
// precipitates, by integer issue and memory latency elsewhere.
template <int MASK, int TX, int TY, bool HOT>
__global__ void __launch_bounds__(Tile2<MASK, TX, TY>::kThreads, blocks2(Tile2<MASK, TX, TY>::kThreads, HOT))
    k_step2d_f64(const __grid_constant__ Step2DArgs a) {
  using T = Tile2<MASK, TX, TY>;
  constexpr bool kFixed = MASK == kMaskIso || MASK == kMaskIso9;
  constexpr Range60 kRange = MASK == kMaskIso9 ? kRangeCorners : kRangeFaces;
  // x^gamma as doubles, or (kFixed) in fixed point
  __shared__ typename T::template Plane<long long> s_g1, s_g2;
  __shared__ typename T::template Plane<double> s_pd, s_pl;
  auto as_double = [](long long (*s)[T::kPitch]) { return reinterpret_cast<double (*)[T::kPitch]>(s); };
  int ex, ey;
  const bool staged = T::cell(ex, ey);
  const int gx = int(blockIdx.x) * TX + ex - 1, gy = tile_row() * TY + ey - 1;
  const Cell64 c = stage64<kFixed, HOT>(a, gx, gy, kRange);
  if (staged) {
    s_g1[ey][ex] = c.g1;
    s_g2[ey][ex] = c.g2;
    s_pd[ey][ex] = c.pd;
    s_pl[ey][ex] = c.pl;
  }
  const bool phases = __syncthreads_or(c.phase);
  const bool fixed = kFixed && !__syncthreads_or(c.wide);
  if (kFixed && !fixed) {  // the whole tile in FP64
    if (staged && !c.wide) {
      const double2 g = gamma_values(c, s_g1[ey][ex], s_g2[ey][ex]);
      as_double(s_g1)[ey][ex] = g.x;
      as_double(s_g2)[ey][ex] = g.y;
    }
    __syncthreads();
  }
  if (threadIdx.x >= T::kOwn || gx >= a.Nx || gy >= a.Ny) return;
  // Cahn-Hilliard, composition_kernel src/discretization.cu:843-865
  const Coef64& K = a.c;
  double ocr, onb;
  if (fixed) {
    const long long S1 = sum58<MASK>(s_g1, ex, ey), S2 = sum58<MASK>(s_g2, ex, ey);
    ocr = advance58(c.X, K.Dfix[0][0], S1, K.Dfix[0][1], S2);
    onb = advance58(c.Y, K.Dfix[1][0], S1, K.Dfix[1][1], S2);
  } else {
    const double l1 = lap64<MASK>(a, as_double(s_g1), ex, ey);
    const double l2 = lap64<MASK>(a, as_double(s_g2), ex, ey);
    ocr = c.X + fma(K.D[0][0], l1, K.D[0][1] * l2);
    onb = c.Y + fma(K.D[1][0], l1, K.D[1][1] * l2);
  }
  double od = 0.0, ol = 0.0;
  if (phases) {
    auto gamma = [&] {
      if constexpr (!HOT) return make_double2(c.v1, c.v2);
      if (fixed) return gamma_values(c, s_g1[ey][ex], s_g2[ey][ex]);
      return make_double2(as_double(s_g1)[ey][ex], as_double(s_g2)[ey][ex]);
    };
    update_phases<MASK>(a, c, s_pd, s_pl, ex, ey, gamma, od, ol);
  }
  store_cell(a, c.i, gx, gy, ocr, onb, od, ol);
}

// ---------------------------------------------------------------------------
// Plain FP64 step with the variable-mobility Cahn-Hilliard (5-point mask):
// the reference's disabled mobility kernels, chemical_convolution_Cr/Nb
// (src/discretization.cu:175-358, 618-778) and the commented update of
// composition_kernel (:848-856), in the reduced form: with paraboloid
// energies the phases' fictitious compositions share their diffusion
// potentials, the 16 coefficient-weighted gradients sum to D(X, Y) grad
// x^gamma (to the 1e-14 the potentials' rounding leaves), and the flux through
// a face is (D_n + D_c)(u_n - u_c).  Each staged cell forms D once (three
// exponentials), each face's flux is formed once: a thread forms its east and
// lower faces, the halo warps the west faces of the first column and the
// upper faces of the first row.
//
// ISO (equal spacings): all of it in fixed point where every cell of the tile
// is in range: u in units of 2^-58, D of 2^-67 (pfa_fixed64.cuh), the fluxes of
// 2^-65, whose sum is rounded once into the composition (a sum that leaves 64
// bits is formed in FP64); else, and with other spacings, in FP64.  Bound by integer issue; with the matrix and
// the fluxes in FP64, bound by that pipe, 512^2 took 38.9 us a step for 20.9,
// 2048^2 521 for 236.
struct Matrix64 {
  double d[4];
};
static __device__ __noinline__ Matrix64 matrix64(const Coef64& K, double X, double Y, bool unit) {
  Matrix64 m;
  dmatrix64_scaled(K, X, Y, unit, m.d[0], m.d[1], m.d[2], m.d[3]);
  return m;
}

// X and its faces' fluxes (units of 2^-65) where their sum leaves 64 bits
static __device__ __noinline__ double advance_faces(double X, long long n, long long s, long long e, long long w) {
  return X + ((double(n) - double(s)) + (double(e) - double(w))) * 0x1p-65;
}

template <bool ISO, int TX, int TY>
__global__ void __launch_bounds__(Tile<TX, TY, false>::kThreads, TX == 16 ? 3 : 8)
    k_step2d_f64_varmob(const __grid_constant__ Step2DArgs a) {
  using T = Tile<TX, TY, false>;
  // fixed point, or the bits of FP64 values
  __shared__ typename T::template Plane<long long> s_g1, s_g2, s_d[4];
  __shared__ typename T::template Plane<double> s_pd, s_pl;
  __shared__ long long s_fx[2][TY][TX + 1], s_fy[2][TY + 1][TX];
  const Coef64& K = a.c;
  int ex, ey;
  const bool staged = T::cell(ex, ey);
  const int gx = int(blockIdx.x) * TX + ex - 1, gy = tile_row() * TY + ey - 1;
  const Cell64 c = stage64<ISO, true>(a, gx, gy, kRangeFlux);
  const bool unit = in_unit(c.X) && in_unit(c.Y);
  bool wide = true;
  long long d[4];
  if constexpr (ISO) {
    const uint64_t x = fix64(c.X), y = fix64(c.Y);
    wide = c.wide || !K.vm_fixed || uint64_t(x + y) <= x || !diffusivities(K, x, y, d);
  }
  auto stage_matrix = [&] {
    const Matrix64 m = matrix64(K, c.X, c.Y, unit);
#pragma unroll
    for (int k = 0; k < 4; k++) s_d[k][ey][ex] = __double_as_longlong(m.d[k]);
  };
  if (staged) {
    s_g1[ey][ex] = c.g1;
    s_g2[ey][ex] = c.g2;
    s_pd[ey][ex] = c.pd;
    s_pl[ey][ex] = c.pl;
    if (wide) {
      stage_matrix();
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) s_d[k][ey][ex] = d[k];
    }
  }
  const bool phases = __syncthreads_or(c.phase);
  const bool fixed = ISO && !__syncthreads_or(wide);
  if (ISO && !fixed) {  // the whole tile in FP64
    if (staged && !c.wide) {
      const double2 g = gamma_values(c, c.g1, c.g2);
      s_g1[ey][ex] = __double_as_longlong(g.x);
      s_g2[ey][ex] = __double_as_longlong(g.y);
    }
    if (staged && !wide) stage_matrix();
    __syncthreads();
  }
  // flux into (ex, ey) from (nx, ny): component k is (D_n + D_c)_k . (u_n - u_c)
  auto flux = [&](int x, int y, int nx, int ny, long long& f1, long long& f2) {
    if (fixed) {
      const long long u1 = (s_g1[ny][nx] - s_g1[y][x]) << 4, u2 = (s_g2[ny][nx] - s_g2[y][x]) << 4;
      f1 = __mul64hi(s_d[0][ny][nx] + s_d[0][y][x], u1) + __mul64hi(s_d[1][ny][nx] + s_d[1][y][x], u2);
      f2 = __mul64hi(s_d[2][ny][nx] + s_d[2][y][x], u1) + __mul64hi(s_d[3][ny][nx] + s_d[3][y][x], u2);
    } else {
      auto v = [](const long long (*s)[T::kPitch], int y, int x) { return __longlong_as_double(s[y][x]); };
      const double u1 = v(s_g1, ny, nx) - v(s_g1, y, x), u2 = v(s_g2, ny, nx) - v(s_g2, y, x);
      const double m0 = v(s_d[0], ny, nx) + v(s_d[0], y, x), m1 = v(s_d[1], ny, nx) + v(s_d[1], y, x);
      const double m2 = v(s_d[2], ny, nx) + v(s_d[2], y, x), m3 = v(s_d[3], ny, nx) + v(s_d[3], y, x);
      f1 = __double_as_longlong(fma(m0, u1, m1 * u2));
      f2 = __double_as_longlong(fma(m2, u1, m3 * u2));
    }
  };
  const bool own = threadIdx.x < T::kOwn;
  if (own) {
    flux(ex, ey, ex + 1, ey, s_fx[0][ey - 1][ex], s_fx[1][ey - 1][ex]);
    flux(ex, ey, ex, ey + 1, s_fy[0][ey][ex - 1], s_fy[1][ey][ex - 1]);
  } else if (staged && ex == 0 && ey >= 1 && ey <= TY) {
    flux(0, ey, 1, ey, s_fx[0][ey - 1][0], s_fx[1][ey - 1][0]);
  } else if (staged && ey == 0 && ex >= 1 && ex <= TX) {
    flux(ex, 0, ex, 1, s_fy[0][0][ex - 1], s_fy[1][0][ex - 1]);
  }
  __syncthreads();
  if (!own || gx >= a.Nx || gy >= a.Ny) return;
  const int tx = ex - 1, ty = ey - 1;
  auto sum = [&](int k, double X) {  // the faces' fluxes added to a composition
    const long long n = s_fy[k][ty + 1][tx], s = s_fy[k][ty][tx], e = s_fx[k][ty][tx + 1], w = s_fx[k][ty][tx];
    if (fixed) {
      int64_t t;
      return face_sum(n, s, e, w, t) ? advance_by(X, (t >> 1) + (t & 1)) : advance_faces(X, n, s, e, w);
    }
    return X + fma(K.vm_qy, __longlong_as_double(n) - __longlong_as_double(s),
                   __longlong_as_double(e) - __longlong_as_double(w));
  };
  const double ocr = sum(0, c.X), onb = sum(1, c.Y);
  double od = 0.0, ol = 0.0;
  if (phases) {
    auto gamma = [&] {
      if (fixed) return gamma_values(c, c.g1, c.g2);
      return make_double2(__longlong_as_double(s_g1[ey][ex]), __longlong_as_double(s_g2[ey][ex]));
    };
    update_phases<ISO ? kMaskIso : kMaskFive>(a, c, s_pd, s_pl, ex, ey, gamma, od, ol);
  }
  store_cell(a, c.i, gx, gy, ocr, onb, od, ol);
}

constexpr long long kHotTiles = 12288, kWideTiles = 8192;

template <int TX, int TY>
long long tiles(const Step2DArgs& a) {
  return (long long)((a.Nx + TX - 1) / TX) * ((a.Ny + TY - 1) / TY);
}

template <int TX, int TY, bool VM, bool HOT>
cudaError_t launch_tiles(const Step2DArgs& a, cudaStream_t s) {
  const int ny = (a.Ny + TY - 1) / TY;
  const dim3 grid((a.Nx + TX - 1) / TX, std::min(ny, 65535), (ny + 65534) / 65535);
  if constexpr (VM) {
    constexpr int n = Tile<TX, TY, false>::kThreads;
    if (a.c.mask == kMaskIso)
      k_step2d_f64_varmob<true, TX, TY><<<grid, n, 0, s>>>(a);
    else
      k_step2d_f64_varmob<false, TX, TY><<<grid, n, 0, s>>>(a);
  } else {
    constexpr int n5 = Tile2<kMaskIso, TX, TY>::kThreads, n9 = Tile2<kMaskIso9, TX, TY>::kThreads;
    if (a.c.mask == kMaskIso9) {
      k_step2d_f64<kMaskIso9, TX, TY, HOT><<<grid, n9, 0, s>>>(a);
    } else if (a.c.mask == kMaskNine) {
      k_step2d_f64<kMaskNine, TX, TY, HOT><<<grid, n9, 0, s>>>(a);
    } else if constexpr (TX == 8) {  // (16 x 8: 9 points only)
      if (a.c.mask == kMaskIso)
        k_step2d_f64<kMaskIso, TX, TY, HOT><<<grid, n5, 0, s>>>(a);
      else
        k_step2d_f64<kMaskFive, TX, TY, HOT><<<grid, n5, 0, s>>>(a);
    }
  }
  return cudaGetLastError();
}

}  // namespace

// ---------------------------------------------------------------------------
cudaError_t launch_step2d_f64(const Step2DArgs& a, cudaStream_t s) {
  if (a.varmob && a.nine) return cudaErrorInvalidValue;  // refused by the host before
  // A tile next to a precipitate takes its SM's FP64 pipe for microseconds, and
  // a step is as long as its most loaded SM: small tiles spread such work, and
  // 8 x 8 has the least halo for its size (with corners 36 cells, two warps: the
  // 9-point form takes 16 x 8 from 8192 tiles of 8 x 8).  The solve in fixed
  // point (HOT) shortens tiles next to precipitates, but its call costs
  // registers (56 for 40, fewer tiles in flight), which many waves of tiles
  // without precipitate feel.  us a step with 6 particles, HOT / FP64, 5
  // points, 8 x 8: 64 x 48 5.1 / 5.8, 256^2 6.6 / 7.4, 512^2 9.0 / 9.8, 1000 x
  // 733 14.2 / 14.3, 1024^2 17.4 / 16.6, 2048^2 73.6 / 64.8 (HOT 8 x 4: 5.3, 7.1,
  // 10.9, 19.0, 24.6, 92; 16 x 8: 5.9, 7.5, 9.9, 15.1, 18.0, 78); 9 points 8 x 8
  // 64 x 48 5.6 / 6.2, 512^2 11.0 / 13.4, 1000 x 733 17.6 / 18.9, 1024^2 21.8 /
  // 21.6, 2048^2 91 / 84; 16 x 8 6.5 / 7.3, 12.0 / 14.5, 17.0 / 18.8, 19.5 / 19.5,
  // 81 / 74.
  if (!a.varmob) {
    const bool hot = tiles<8, 8>(a) <= kHotTiles, corners = a.c.mask == kMaskIso9 || a.c.mask == kMaskNine;
    if (corners && tiles<8, 8>(a) > kWideTiles)
      return hot ? launch_tiles<16, 8, false, true>(a, s) : launch_tiles<16, 8, false, false>(a, s);
    return hot ? launch_tiles<8, 8, false, true>(a, s) : launch_tiles<8, 8, false, false>(a, s);
  }
  // every staged cell has its mobilities, so large grids take the tile with
  // the smallest share of halo: 8 x 8 / 16 x 16 64 x 48 6.5 / 9.9, 192^2 7.7 /
  // 9.6, 320^2 11.2 / 12.5, 384^2 13.8 / 13.1, 512^2 21.5 / 20.8, 2048^2 279 /
  // 237 (16 x 8: 271; 16 x 16 at two and four CTAs per SM: 272 and 243)
  return tiles<16, 16>(a) < 576 ? launch_tiles<8, 8, true, true>(a, s) : launch_tiles<16, 16, true, true>(a, s);
}

}  // namespace pfa

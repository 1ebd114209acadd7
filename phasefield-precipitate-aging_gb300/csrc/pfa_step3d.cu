// pfa_step3d.cu -- 3D step with the 7-point Laplacian (sm_103a).
//
// The reference supports 2D only (src/main.cpp:418-421); this extends its
// equations unchanged to a 7-point stencil with six-face zero-flux ghost
// fill.  Two kernels stream along z:
//   k_stream3d_f64: plain FP64 in the reduced forms of pfa_device.cuh,
//        ghost-ring layout ((Nz+2) planes of (Ny+2) rows of Nx+2 doubles, one
//        array per field); tiles of 8 x 8 columns, described below.
//   k_stream3d_f32: the precision form (FP32 arithmetic, every field
//        Kahan-compensated, the equilibrium-referenced gamma solve) on
//        interior-only records (pfa_step2d_f32.cu): A = float4 {x_Cr, x_Nb,
//        phi_del, phi_lav}, B = the four compensations as packed 16-bit
//        counts (uint2); tiles of 32 x 13 output cells, records staged by
//        TMA, described below.
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <type_traits>

#include "pfa_device.cuh"
#include "pfa_kernels.h"
#include "pfa_tile64.cuh"
#include "pfa_tma.cuh"

namespace pfa {

using namespace dev;

namespace {

template <class R>
struct Nb3 {
  R gcr, gnb, pd, pl;  // gcr, gnb: the deviations u = x^gamma - xe_gamma
};

template <class R>
struct Raw3 {
  R x, y, pd, pl;
  uint2 cq;  // packed Kahan compensations
};

// FP64 store of the interior cell (x, y, z) and of every ghost cell whose
// nearest interior cell it is (the six-face fill; edges and corners take the
// nearest interior cell).
__device__ __noinline__ void store64(double* f, const Step3DArgs& a, int x, int y, int z, double v) {
  int xs[3] = {x, 0, 0}, ys[3] = {y, 0, 0}, zs[3] = {z, 0, 0};
  int nx = 1, ny = 1, nz = 1;
  if (x == 0) xs[nx++] = -1;
  if (x == a.Nx - 1) xs[nx++] = a.Nx;
  if (y == 0) ys[ny++] = -1;
  if (y == a.Ny - 1) ys[ny++] = a.Ny;
  if (z == 0) zs[nz++] = -1;
  if (z == a.Nz - 1) zs[nz++] = a.Nz;
  for (int k = 0; k < nz; k++)
    for (int j = 0; j < ny; j++)
      for (int i = 0; i < nx; i++)
        f[((long long)(zs[k] + 1) * (a.Ny + 2) + (ys[j] + 1)) * a.pitch + (xs[i] + 1)] = v;
}

// ---- plain FP64 ----
// Tiles of 8 x 8 columns (pfa_tile64.cuh) streaming along z: a thread keeps
// its cell's last three planes (x^gamma, phases) and the records of the next
// two, publishes x^gamma (fixed point, pfa_device.cuh) and the phases of
// plane z in shared memory and passes one barrier per plane.  ISO: equal
// spacings, which the fixed-point sum needs; other spacings, and planes with
// a composition outside its range, take the FP64 sums.  Bound by the FP64
// pipe next to precipitates, elsewhere by the latency of a plane's chain:
// compact tiles put the fewest warps on a precipitate's surface, and three
// warps per CTA wait least for one another.  us a step at the best split, 32
// x 8 tiles in rows of 32 / 16 x 16 / 16 x 8 / 8 x 8 (eight CTAs per SM asked
// for; six: 139, 506): 128^3 184 / 168 / 158 / 132, 256^3 543 / 569 / 557 / 470.
using Tile3 = Tile<8, 8, false>;
struct Plane64 {
  Tile3::Plane<long long> g1, g2;
  Tile3::Plane<double> pd, pl;
};

template <bool ISO, bool HOT>
__global__ void __launch_bounds__(Tile3::kThreads, HOT ? 7 : 8)
    k_stream3d_f64(const __grid_constant__ Step3DArgs a) {
  __shared__ Plane64 sh[2];
  __shared__ int s_wide[3];
  int ex, ey;
  const bool staged = Tile3::cell(ex, ey);
  const int xt = (a.Nx + Tile3::TX - 1) / Tile3::TX, by = int(blockIdx.x) / xt, bx = int(blockIdx.x) - by * xt;
  const int x = bx * Tile3::TX + ex - 1, y = by * Tile3::TY + ey - 1;
  const int cx = clampi(x, 0, a.Nx - 1), cy = clampi(y, 0, a.Ny - 1);
  const bool own = threadIdx.x < Tile3::kOwn && x < a.Nx && y < a.Ny;
  const int z0 = blockIdx.y * a.zrows, z1 = min(z0 + a.zrows, a.Nz);
  const size_t plane = size_t(a.Ny + 2) * a.pitch, col = size_t(cy + 1) * a.pitch + cx + 1;
  const Coef64& K = a.c;
  const bool edge = cx == 0 || cx == a.Nx - 1 || cy == 0 || cy == a.Ny - 1;
  if (threadIdx.x < 3) s_wide[threadIdx.x] = 0;

  struct Record {
    double X, Y, pd, pl;
  };
  auto load = [&](int z) {
    const size_t i = size_t(clampi(z, 0, a.Nz - 1) + 1) * plane + col;
    return Record{__ldg(static_cast<const double*>(a.in[0]) + i), __ldg(static_cast<const double*>(a.in[1]) + i),
                  __ldg(static_cast<const double*>(a.in[2]) + i), __ldg(static_cast<const double*>(a.in[3]) + i)};
  };
  auto stage = [&](const Record& r) { return cell64<ISO, HOT>(r.X, r.Y, r.pd, r.pl, kRangeFaces); };
  Cell64 P, C, N;  // planes z - 1, z, z + 1 of the thread's column
  Record next;     // the record of the plane after them
  if constexpr (HOT) {
    next = load(z0 - 1);
    P = stage(next);
    next = load(z0);
    C = stage(next);
    next = load(z0 + 1);
  } else {
    // the first three planes are requested together: one wait, not three (us a
    // step 192^3 251 -> 241, 256^3 465 -> 455; with the solve's call the records
    // do not fit the registers: 128^3 123 -> 128)
    const Record r0 = load(z0 - 1), r1 = load(z0);
    next = load(z0 + 1);
    P = stage(r0);
    C = stage(r1);
  }
  __syncthreads();  // s_wide is set
  int w = 0;  // slot of s_wide
  for (int z = z0; z < z1; z++) {
    N = stage(next);
    if (z + 1 < z1) next = load(z + 2);
    Plane64& S = sh[z & 1];
    auto dg1 = reinterpret_cast<double (*)[Tile3::kPitch]>(S.g1), dg2 = reinterpret_cast<double (*)[Tile3::kPitch]>(S.g2);
    if (staged) {
      S.g1[ey][ex] = C.g1;
      S.g2[ey][ex] = C.g2;
      if (ISO && (P.wide || C.wide || N.wide)) s_wide[w] = 1;
      S.pd[ey][ex] = C.pd;
      S.pl[ey][ex] = C.pl;
    }
    // buffer z & 1 was last read before the previous barrier; slot w + 2 of
    // s_wide was last read before this one
    const bool phases = __syncthreads_or(staged && (P.phase || C.phase || N.phase));
    const bool fixed = ISO && s_wide[w] == 0;
    const int w2 = w == 0 ? 2 : w - 1;  // (w + 2) % 3
    if (threadIdx.x == 0) s_wide[w2] = 0;
    w = w == 2 ? 0 : w + 1;
    if (ISO && !fixed) {  // the whole plane in FP64
      if (staged && !C.wide) {
        const double2 g = gamma_values(C, C.g1, C.g2);
        dg1[ey][ex] = g.x;
        dg2[ey][ex] = g.y;
      }
      __syncthreads();
    }
    if (own) {
      double ocr, onb, od = 0.0, ol = 0.0;
      const double mx = a.m.idx2[0], my = a.m.idx2[1], mz = a.m.idx2[2];
      auto lap = [&](double zm, double zp, const double (*s)[Tile3::kPitch], double c) {
        const double sx = s[ey][ex - 1] + s[ey][ex + 1], sy = s[ey - 1][ex] + s[ey + 1][ex];
        if constexpr (ISO)
          return fma(K.iso_c, c, ((zm + zp) + sy) + sx);
        else
          return fma(mz, zm + zp, fma(my, sy, fma(mx, sx, -2. * (mx + my + mz) * c)));
      };
      if (fixed) {
        auto sum = [&](long long zm, long long zp, const long long (*s)[Tile3::kPitch], long long c) {
          return (zm + zp) + (s[ey - 1][ex] + s[ey + 1][ex]) + (s[ey][ex - 1] + s[ey][ex + 1]) - 6 * c;
        };
        const long long S1 = sum(P.g1, N.g1, S.g1, C.g1), S2 = sum(P.g2, N.g2, S.g2, C.g2);
        ocr = advance58(C.X, K.Dfix[0][0], S1, K.Dfix[0][1], S2);
        onb = advance58(C.Y, K.Dfix[1][0], S1, K.Dfix[1][1], S2);
      } else {
        // (fixed: within 2^-58 of the plane's own values, 1e-20 in the sum)
        auto value = [](const Cell64& c, long long g) { return ISO && !c.wide ? value58(g) : __longlong_as_double(g); };
        const double l1 = lap(value(P, P.g1), value(N, N.g1), dg1, dg1[ey][ex]);
        const double l2 = lap(value(P, P.g2), value(N, N.g2), dg2, dg2[ey][ex]);
        ocr = C.X + fma(K.D[0][0], l1, K.D[0][1] * l2);
        onb = C.Y + fma(K.D[1][0], l1, K.D[1][1] * l2);
      }
      if (phases) {
        auto none = [&](double zm, double zp, const double (*s)[Tile3::kPitch]) {
          auto b = [&](int y, int x) { return value_bits(s[y][x]); };
          return (value_bits(zm) | value_bits(zp) | b(ey, ex) | b(ey - 1, ex) | b(ey + 1, ex) |
                  b(ey, ex - 1) | b(ey, ex + 1)) == 0;
        };
        auto gamma = [&] { return gamma_values(C, C.g1, C.g2); };
        od = phase64<0>(K, C, none(P.pd, N.pd, S.pd), [&] { return lap(P.pd, N.pd, S.pd, C.pd); }, gamma);
        ol = phase64<1>(K, C, none(P.pl, N.pl, S.pl), [&] { return lap(P.pl, N.pl, S.pl, C.pl); }, gamma);
      }
      const double v[4] = {ocr, onb, od, ol};
      const size_t i = size_t(z + 1) * plane + col;
#pragma unroll
      for (int k = 0; k < 4; k++) static_cast<double*>(a.out[k])[i] = v[k];
      if (edge || z == 0 || z == a.Nz - 1) {
#pragma unroll
        for (int k = 0; k < 4; k++) store64(static_cast<double*>(a.out[k]), a, cx, cy, z, v[k]);
      }
    }
    P = C;
    C = N;
  }
}

// ---- FP32 form, two planes per barrier ----
// A CTA covers 32 x-columns by 13 y-rows of output and streams along z.
// Warps 0..12 own one row each, every lane an output column; warps 13..15
// solve the 94 halo cells around the tile (the rows above and below, 34
// cells each, and the columns left and right, 13 cells each).  Every thread
// publishes its solved cell into a 15 x 34 plane in shared memory, and the
// row warps read all four in-plane neighbours from there (no shuffles); z
// neighbours come from a register window.  With 32 output columns per CTA a
// power-of-two grid side splits into whole tiles.
// Planes reach shared memory through a four-plane ring filled by TMA: one
// thread issues, per plane, a tiled copy of the CTA's 15 x 36 box of A
// records and one of B records, from two columns left of the tile (so that
// the box of 8-byte B records starts on a 16-byte boundary), both
// completing on the plane slot's mbarrier; every thread reads its own
// (clamped) record from the slot, at the same index in both boxes.  Records
// outside the grid arrive as zeros and are never read (threads past an edge
// read the clamped record).  Each
// iteration solves planes z+1 and z+2, publishes them and passes one barrier
// for both updates; a plane's record is read from the ring once, for its
// solve, and kept in registers until its update.
constexpr int kRing3 = 4;                      // planes in the ring (a power of two)
constexpr int kW3 = 16;                        // warps per CTA
constexpr int kRows3 = 13;                     // output rows (warps 0..12)
constexpr int kCols3 = 32;                     // output columns
constexpr int kPR = kRows3 + 2;                // rows of a staged or published plane
constexpr int kPC = kCols3 + 2;                // columns of a published plane
constexpr int kBox3 = kCols3 + 4;              // records per staged row, from x0 - 2
constexpr int kHalo3 = 2 * kPC + 2 * kRows3;   // halo cells (94 <= 3 warps)
static_assert(kHalo3 <= 32 * (kW3 - kRows3), "the halo warps cover the halo");
constexpr uint32_t kBoxBytesA = kPR * kBox3 * sizeof(float4);  // 8640
constexpr uint32_t kBoxBytesB = kPR * kBox3 * sizeof(uint2);   // 4320
constexpr uint32_t kSlotA = (kBoxBytesA + 127) / 128 * 128, kSlotB = (kBoxBytesB + 127) / 128 * 128;
constexpr uint32_t kTxPlane = kBoxBytesA + kBoxBytesB;  // bytes one plane's two copies deliver
struct Smem3 {
  float4 ra[kRing3][kSlotA / sizeof(float4)];
  uint2 rc[kRing3][kSlotB / sizeof(uint2)];
  // two published planes per iteration, two iterations; the cell past the
  // plane takes the writes of the two idle halo lanes
  Nb3<float> sh[4][kPR * kPC + 1];
  unsigned long long bar[kRing3];
};
static_assert(offsetof(Smem3, rc) % 128 == 0, "ring slots must stay 128-byte aligned");
constexpr size_t kSmem3 = sizeof(Smem3) + 128;  // + slack to align the base to 128 B

// gamma solve of one cell (warp-uniform bulk / equilibrium-referenced forms)
__device__ __forceinline__ Nb3<float> solve32(const Step3DArgs& a, const Raw3<float>& r) {
  const float2 h = cq_halves(r.cq.x);
  const float cx = h.x * kCqXi, cy = h.y * kCqXi;
  Nb3<float> n;
  n.pd = r.pd;
  n.pl = r.pl;
  if (__all_sync(0xffffffffu, fmaxf(fabsf(r.pd), fabsf(r.pl)) < kBulkPhi))
    gamma_bulk32(a.k, r.x, r.y, cx, cy, n.gcr, n.gnb);
  else
    gamma_u32(a.k, r.x, r.y, cx, cy, r.pd, r.pl, n.gcr, n.gnb);
  return n;
}

// update of one output cell (record i) from its seven neighbours' solves
__device__ __forceinline__ void update32(const Step3DArgs& a, long long i, const Nb3<float>& up,
                                         const Nb3<float>& c, const Nb3<float>& dn,
                                         const Nb3<float>& s, const Nb3<float>& n,
                                         const Nb3<float>& wv, const Nb3<float>& e,
                                         const Raw3<float>& rc) {
  const float i2x = a.idx2f[0], i2y = a.idx2f[1], i2z = a.idx2f[2];
  auto lap = [&](float z0, float y0, float x0, float vc, float x1, float y1, float z1) {
    const float sx = (x0 - vc) + (x1 - vc);
    const float sy = (y0 - vc) + (y1 - vc);
    const float sz = (z0 - vc) + (z1 - vc);
    return fmaf(sx, i2x, fmaf(sy, i2y, sz * i2z));
  };
  const float lapCr = lap(up.gcr, s.gcr, wv.gcr, c.gcr, e.gcr, n.gcr, dn.gcr);
  const float lapNb = lap(up.gnb, s.gnb, wv.gnb, c.gnb, e.gnb, n.gnb, dn.gnb);
  const float lapD = lap(up.pd, s.pd, wv.pd, c.pd, e.pd, n.pd, dn.pd);
  const float lapL = lap(up.pl, s.pl, wv.pl, c.pl, e.pl, n.pl, dn.pl);
  const float4 cc = cq_unpack(rc.cq);
  const float X = rc.x, Y = rc.y, pd = rc.pd, pl = rc.pl;
  const float ycr = fmaf(a.dtD[0][0], lapCr, a.dtD[0][1] * lapNb) - cc.x, tcr = X + ycr;
  const float ynb = fmaf(a.dtD[1][0], lapCr, a.dtD[1][1] * lapNb) - cc.y, tnb = Y + ynb;
  const FastCoef& K = a.k;
  const float u1 = c.gcr, u2 = c.gnb;
  const float dFd = fmaf(-a.kap[0], lapD, dF_local32(pd, pl, quad2(K.dP[0], u1, u2), a.om2[0], a.alpha2));
  const float dFl = fmaf(-a.kap[1], lapL, dF_local32(pl, pd, quad2(K.dP[1], u1, u2), a.om2[1], a.alpha2));
  const float yd = fmaf(-a.dtL[0], dFd, -cc.z), td = pd + yd;
  const float yl = fmaf(-a.dtL[1], dFl, -cc.w), tl = pl + yl;
  static_cast<float4*>(a.out[0])[i] = make_float4(tcr, tnb, td, tl);
  static_cast<uint2*>(a.out[1])[i] =
      cq_pack((tcr - X) - ycr, (tnb - Y) - ynb, (td - pd) - yd, (tl - pl) - yl);
}

// SKIP: the instantiation with the test hook (Step3DArgs::skip_plane)
template <bool SKIP>
__global__ void __launch_bounds__(32 * kW3, 2)
    k_stream3d_f32(Step3DArgs a, const __grid_constant__ Tma3 t) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = tma::smem_addr(smem_raw);
  Smem3& sm = *reinterpret_cast<Smem3*>(smem_raw + ((128u - (raw & 127u)) & 127u));
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int xa = blockIdx.x * kCols3 - 1;    // first column of the published plane
  const int yb = blockIdx.y * kRows3 - 1;    // first row of the staged boxes / published plane
  // this thread's cell in the published plane (pr, pc): a row warp's own
  // cell, or a halo cell (h = 94, 95 solve a duplicate and publish it past
  // the plane)
  const bool row = w < kRows3;
  int pr = w + 1, pc = lane + 1;
  bool pub = true;
  if (!row) {
    const int h = (w - kRows3) * 32 + lane;
    if (h < kPC) {
      pr = 0;
      pc = h;
    } else if (h < 2 * kPC) {
      pr = kPR - 1;
      pc = h - kPC;
    } else if (h < 2 * kPC + kRows3) {
      pr = 1 + h - 2 * kPC;
      pc = 0;
    } else {
      pr = 1 + min(h - 2 * kPC - kRows3, kRows3 - 1);
      pc = kPC - 1;
      pub = h < kHalo3;
    }
  }
  const int x = xa + pc, y = yb + pr;
  const int cx = min(max(x, 0), a.Nx - 1), cy = min(max(y, 0), a.Ny - 1);
  const bool out = row && x < a.Nx && y < a.Ny;
  // records in a plane and this thread's record in it: both below 2^31 (a
  // plane of records fits a 32-bit index; the plane offset is 64-bit)
  const int col = cy * a.pitch + cx, plane = a.Ny * a.pitch;
  const int ib = (cy - yb) * kBox3 + (cx - xa + 1);  // this thread's record in the staged boxes
  const int op = pub ? pr * kPC + pc : kPR * kPC;   // its cell in a published plane
  const int z0 = blockIdx.z * a.zrows;
  const int z1 = min(z0 + a.zrows, a.Nz);
  const uint32_t bar0 = tma::smem_addr(&sm.bar[0]);
  const uint32_t dA = tma::smem_addr(&sm.ra[0][0]), dB = tma::smem_addr(&sm.rc[0][0]);
  if (tid == 0) {
    tma::prefetch_map(&t.a);
    tma::prefetch_map(&t.b);
    for (int k = 0; k < kRing3; k++) tma::bar_init(bar0 + 8 * k, 1);
    tma::bar_init_fence();
  }
  __syncthreads();
  // plane p lives in ring slot (p - z0 + 1) & 3 and completes that slot's
  // phase (p - z0 + 1) >> 2; planes past z1 are never issued.  The slot
  // arguments below are compile-time constants.
  int last[kRing3] = {-2, -2, -2, -2};  // thread 0: last plane issued into each slot
  // A thread whose wait gave up stops waiting (later waits give up after
  // their first polls; it computes from whatever the ring holds and the
  // handle reports the failure); thread 0, once its own wait gave up, issues
  // nothing more, so the copies in flight are exactly those its final drain
  // waits for.  SKIP: the test hook that withholds one plane's copies in
  // the first CTA.
  bool gave_up = false;
  const bool skip =
      SKIP && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && a.skip_plane >= 0;
  auto issue = [&](int p, int sl) {
    if (tid == 0 && p <= z1 && !gave_up && !(skip && p == a.skip_plane)) {
      const int zc = min(max(p, 0), a.Nz - 1);
      tma::proxy_fence();  // the slot's earlier reads (ordered by the barrier) come first
      tma::bar_arrive_tx(bar0 + 8 * sl, kTxPlane);
      tma::load3(dA + sl * kSlotA, &t.a, 4 * (xa - 1), yb, zc, bar0 + 8 * sl);
      tma::load3(dB + sl * kSlotB, &t.b, 2 * (xa - 1), yb, zc, bar0 + 8 * sl);
      last[sl] = p;
    }
  };
  auto wait = [&](int p, int sl) {
    if (!tma::bar_wait(bar0 + 8 * sl, uint32_t((p - z0 + 1) >> 2) & 1u,
                       gave_up ? 0ull : tma::kWaitNs))
      gave_up = true;
  };
  auto fetch = [&](int sl) {
    const float4 v = sm.ra[sl][ib];
    return Raw3<float>{v.x, v.y, v.z, v.w, sm.rc[sl][ib]};
  };
  auto update = [&](int z, const Nb3<float>& up, const Nb3<float>& c, const Nb3<float>& dn,
                    const Raw3<float>& rc, const Nb3<float>* P) {
    if (out)
      update32(a, (long long)z * plane + col, up, c, dn, P[op - kPC], P[op + kPC], P[op - 1],
               P[op + 1], rc);
  };
  for (int k = -1; k <= 2; k++) issue(z0 + k, k + 1);
  wait(z0 - 1, 0);
  wait(z0, 1);
  Raw3<float> rB = fetch(1), rC, rD;  // raw records kept for the updates
  Nb3<float> nA = solve32(a, fetch(0)), nB = solve32(a, rB), nC, nD;
  __syncthreads();  // slots 0 and 1 are read before the first pair refills them
  // two planes z, z+1; issued up to plane z+2 on entry.  Q = (z - z0) & 3
  // (0 or 2) fixes the ring slots and the exchange slots.
  auto pair = [&](auto q, int z) {
    constexpr int Q = decltype(q)::value;
    constexpr int s1 = (2 + Q) & 3, s2 = (3 + Q) & 3, s3 = Q & 3, s4 = (1 + Q) & 3;
    // the slots of planes z-1 and z: read before the previous barrier
    issue(z + 3, s3);
    issue(z + 4, s4);
    wait(z + 1, s1);
    rC = fetch(s1);
    wait(z + 2, s2);
    rD = fetch(s2);
    nC = solve32(a, rC);
    nD = solve32(a, rD);
    Nb3<float>* b0 = sm.sh[Q];
    Nb3<float>* b1 = sm.sh[Q + 1];
    b0[op] = nB;
    b1[op] = nC;
    // these exchange slots were last read two pairs ago, before the previous
    // pair's barrier
    __syncthreads();
    update(z, nA, nB, nC, rB, b0);
    update(z + 1, nB, nC, nD, rC, b1);
    nA = nC;
    nB = nD;
    rB = rD;
  };
  int z = z0;
  for (; z + 3 < z1; z += 4) {
    pair(std::integral_constant<int, 0>{}, z);
    pair(std::integral_constant<int, 2>{}, z + 2);
  }
  int q = 0;  // (z - z0) & 3
  if (z + 1 < z1) {
    pair(std::integral_constant<int, 0>{}, z);
    z += 2;
    q = 2;
  }
  if (z < z1) {  // one plane left; plane z+1 (<= z1) was issued by the last pair
    const int s1 = (2 + q) & 3;
    wait(z + 1, s1);
    nC = solve32(a, fetch(s1));
    Nb3<float>* b0 = sm.sh[q];
    b0[op] = nB;
    __syncthreads();
    update(z, nA, nB, nC, rB, b0);
  }
  if (gave_up && a.status) atomicExch(a.status, 3);
  // thread 0 waits for every plane it issued, so its copies have all landed
  // unless one of its waits gave up: then it waits again (bounded) before
  // the block exits
  if (tid == 0 && gave_up)
    for (int k = 0; k < kRing3; k++)
      if (last[k] >= z0 - 1) tma::bar_wait(bar0 + 8 * k, uint32_t((last[k] - z0 + 1) >> 2) & 1u);
}

// FP64 ghost-ring fields <-> FP32 records (3D): a thread per cell of the side
// that is written (records; ghost-ring fields, whose ghost cells read their
// nearest interior record), the launch grid covering (x, y) with its blocks
// and z with gridDim.z (looping when there are more planes), so no index needs
// a division and every store is coalesced (256^3: import 196 us, export 190; a
// thread per record that also stored the ghost cells it mirrors took 2.38 ms).
__global__ void k_import3d(Conv3DArgs a) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= a.Nx || y >= a.Ny) return;
  for (int z = blockIdx.z; z < a.Nz; z += gridDim.z) {
    const long long i64 = ((long long)(z + 1) * (a.Ny + 2) + (y + 1)) * (a.Nx + 2) + (x + 1);
    const long long r = ((long long)z * a.Ny + y) * a.pitch32 + x;
    float hi[4], c[4];
#pragma unroll
    for (int k = 0; k < 4; k++) split_f64(a.f64[k][i64], hi[k], c[k]);  // value = hi - c
    reinterpret_cast<float4*>(a.A)[r] = make_float4(hi[0], hi[1], hi[2], hi[3]);
    static_cast<uint2*>(a.B)[r] = cq_pack(c[0], c[1], c[2], c[3]);
  }
}

__global__ void k_export3d(Conv3DArgs a) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= a.Nx + 2 || y >= a.Ny + 2) return;
  const int cx = clampi(x - 1, 0, a.Nx - 1), cy = clampi(y - 1, 0, a.Ny - 1);
  for (int z = blockIdx.z; z < a.Nz + 2; z += gridDim.z) {
    const long long r = ((long long)clampi(z - 1, 0, a.Nz - 1) * a.Ny + cy) * a.pitch32 + cx;
    const long long i64 = ((long long)z * (a.Ny + 2) + y) * (a.Nx + 2) + x;
    const float4 v = reinterpret_cast<const float4*>(a.A)[r];
    double val[4];
    merge_record(v, static_cast<const uint2*>(a.B)[r], val);
#pragma unroll
    for (int k = 0; k < 4; k++) a.f64[k][i64] = val[k];
  }
}

// z planes per segment, tiles of tx x ty output cells per plane.  Large grids:
// whole waves of resident CTAs, two extra planes of gamma solves per segment.
// Small ones are bound by a segment's serial planes (0.85 us each), so the
// segments are as short as fill the SMs once, then the resident slots once and
// twice (us a step at that length, and in whole waves of at least 16 planes:
// 32^3 3.5 and 16, 48^3 5.2 and 16, 64^3 6.9 and 16, 80^3 12.3 and 16, 47 x 191 x
// 85 16.1 and 17.4, 110^3 21.0 and 23.7, 128^3 26.2 and 26.7, 178 x 47 x 202 23.4
// and 25.8; from 150^3 on, 42 and 38, whole waves are the better way).
int segment_planes(int Nx, int Ny, int Nz, int resident, int tx, int ty) {
  const long long cols = (long long)((Nx + tx - 1) / tx) * ((Ny + ty - 1) / ty);
  const long long n = cols * Nz, r = resident;  // planes of tiles, CTAs
  auto parts = [&](long long ctas) { return int(std::min<long long>((n + ctas - 1) / ctas, Nz)); };
  if (2 * n <= 5 * r) return parts(std::max(1ll, r / 2));
  if (n <= 10 * r) return parts(r);
  if (n <= 20 * r) return parts(2 * r);
  int best = Nz;
  double best_score = 0.0;
  for (int waves = 1; waves <= 256; waves++) {
    const long long segs = waves * r / cols;
    if (segs < 1) continue;
    const int planes = int((Nz + segs - 1) / segs);
    if (planes < 16 && segs > 1) break;
    const long long used = cols * ((Nz + planes - 1) / planes);
    const long long slots = ((used + r - 1) / r) * r;
    const double score = double(used) / double(slots) / (1.0 + 2.0 / planes);
    if (score > best_score) {
      best_score = score;
      best = planes;
    }
  }
  return best;
}

// FP64: a column next to a precipitate costs several times one in the matrix,
// so short segments that spread the precipitates over the SMs beat whole
// waves of equal ones.  us per step at 1 / 2 / 3 / 6 / 12 planes: 32^3 15 / 18
// / 22 / 38 / 70, 64^3 44 / 40 / 39 / 44 / 73, 96^3 79 / 71 / 71 / 80 / 94, 200
// x 100 x 60 94 / 84 / 81 / 86 / 108, 128^3 146 / 130 / 123 / 124 / 133, 192^3
// 362 / 285 / 263 / 250 / 252, 256^3 768 / 588 / 528 / 475 / 458.
int segment_planes_f64(long long columns, int Nz) {
  const long long n = columns * Nz;  // planes of tiles
  const int planes = n <= 1024 ? 1 : n <= 16384 ? 2 : (n <= 65536 ? 3 : (n <= 180000 ? 6 : 16));
  return std::min(std::max(planes, (Nz + 65534) / 65535), Nz);
}

// up to here the solve in fixed point (cell64's HOT) pays for its registers
// (pfa_step2d.cu), us a step fixed / FP64: 32^3 15.1 / 21.7, 64^3 39.6 / 56, 96^3
// 71 / 86, 128^3 123 / 132, 192^3 265 / 241, 256^3 503 / 455
constexpr long long kHotPlanes = 65536;

int g_resident3 = 0;  // resident CTAs of the FP32 kernel

}  // namespace

cudaError_t prepare_step3d() {
  cudaError_t e = cudaFuncSetAttribute(k_stream3d_f32<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(kSmem3));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_stream3d_f32<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(kSmem3));
  int dev = 0, sms = 0, per = 0;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_stream3d_f32<false>, 32 * kW3, kSmem3);
  g_resident3 = sms * (per > 0 ? per : 1);
  return e;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (the
// library links the static runtime, not the driver library)
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                 const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

cudaError_t encode_step3d_maps(Tma3* t, const void* A, const void* B, int Nx, int Ny, int Nz,
                               int pitch) {
  static EncodeTiled encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    const cudaError_t e =
        cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q);
    if (e != cudaSuccess) return e;
    if (q != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
    encode = reinterpret_cast<EncodeTiled>(fn);
  }
  const cuuint32_t box_a[3] = {4 * kBox3, kPR, 1}, box_b[3] = {2 * kBox3, kPR, 1}, one[3] = {1, 1, 1};
  const cuuint64_t dim_a[3] = {4ull * Nx, cuuint64_t(Ny), cuuint64_t(Nz)};
  const cuuint64_t dim_b[3] = {2ull * Nx, cuuint64_t(Ny), cuuint64_t(Nz)};
  const cuuint64_t str_a[2] = {16ull * pitch, 16ull * pitch * Ny};
  const cuuint64_t str_b[2] = {8ull * pitch, 8ull * pitch * Ny};
  CUresult r = encode(&t->a, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(A), dim_a, str_a,
                      box_a, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_SUCCESS)
    r = encode(&t->b, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<void*>(B), dim_b, str_b, box_b,
               one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t launch_step3d(Step3DArgs a, bool f64, const Tma3* t, cudaStream_t s) {
  if (f64) {
    const long long cols = (long long)((a.Nx + Tile3::TX - 1) / Tile3::TX) * ((a.Ny + Tile3::TY - 1) / Tile3::TY);
    a.zrows = segment_planes_f64(cols, a.Nz);
    const dim3 grid((unsigned)cols, (a.Nz + a.zrows - 1) / a.zrows);
    const bool hot = cols * a.Nz <= kHotPlanes;
    auto launch = [&](auto kernel) { kernel<<<grid, Tile3::kThreads, 0, s>>>(a); };
    if (a.c.mask == kMaskIso)
      launch(hot ? k_stream3d_f64<true, true> : k_stream3d_f64<true, false>);
    else
      launch(hot ? k_stream3d_f64<false, true> : k_stream3d_f64<false, false>);
  } else {
    if (!t) return cudaErrorInvalidValue;
    const int resident = g_resident3 > 0 ? g_resident3 : 152;
    a.zrows = segment_planes(a.Nx, a.Ny, a.Nz, resident, kCols3, kRows3);
    const dim3 grid((a.Nx + kCols3 - 1) / kCols3, (a.Ny + kRows3 - 1) / kRows3, (a.Nz + a.zrows - 1) / a.zrows);
    if (a.skip_plane >= 0)
      k_stream3d_f32<true><<<grid, 32 * kW3, kSmem3, s>>>(a, *t);
    else
      k_stream3d_f32<false><<<grid, 32 * kW3, kSmem3, s>>>(a, *t);
  }
  return cudaGetLastError();
}

dim3 conv3d_grid(int nx, int ny, int nz) {
  return dim3((nx + 31) / 32, (ny + 7) / 8, std::min(nz, 65535));
}

cudaError_t launch_import3d(const Conv3DArgs& a, cudaStream_t s) {
  k_import3d<<<conv3d_grid(a.Nx, a.Ny, a.Nz), dim3(32, 8), 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_export3d(const Conv3DArgs& a, cudaStream_t s) {
  k_export3d<<<conv3d_grid(a.Nx + 2, a.Ny + 2, a.Nz + 2), dim3(32, 8), 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace pfa

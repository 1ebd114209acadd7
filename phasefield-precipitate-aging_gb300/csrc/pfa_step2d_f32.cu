// pfa_step2d_f32.cu -- the FP32 precision form of the 2D step (sm_103a).
//
// Same step as the FP64 kernel (src/main.cpp:289-305 fused), arithmetic in
// FP32 with every field Kahan-compensated (value = hi - c).  The gamma
// solve is the equilibrium-referenced form (pfa_device.cuh, gamma_u32),
// which keeps FP32 accurate inside precipitates where the plain num / den
// form loses it to cancellation; cells whose phases are below 1e-5 skip the
// solve (x^gamma = X there), and rows whose phases are all zero the
// Allen-Cahn update.  Grids larger than the L2 take two steps per pass, small
// ones several steps per launch.  At 48 bytes per cell and pass the HBM budget
// leaves ~250 instructions per cell, so the kernels are organised for
// instruction economy:
//  * each warp owns a strip of 30 output columns (lanes 1..30; lanes 0 and
//    31 carry the neighbour columns) and streams down a segment of rows; the
//    three rows a 5- or 9-point Laplacian needs live in registers, rotated by
//    a 3x-unrolled loop, so each cell's gamma solve runs once and nothing
//    goes through shared memory;
//  * left / right neighbours come from __shfl_up / __shfl_down (with the
//    9-point mask each row carries its x-difference sums, formed once);
//  * the state is stored as two records per cell -- A = {x_Cr, x_Nb, phi_del,
//    phi_lav} (16 bytes) and B = the four compensations, packed into 16-bit
//    counts (8 bytes, PACK) or as FP32 (16 bytes) -- so a row costs one
//    128-bit and one 64-bit (128-bit) load and store and a single address per
//    lane; records of the row after next are loaded one iteration ahead (the
//    batched kernel stages rows through a per-warp cp.async ring instead).
//
// Record layout: Ny rows of `pitch` records (pitch a multiple of 32), interior
// cell (x, y) at record y * pitch + x, no ghost ring; zero-flux edges come
// from clamped indexing (the mirror the reference's halo fill produces).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "pfa_device.cuh"
#include "pfa_kernels.h"

namespace pfa {

using namespace dev;

namespace {

constexpr int kWarps = 4;  // warps (strips) per CTA
constexpr int kCols = 30;  // output columns per warp; lanes 0 and 31 are halo

// The values a neighbour needs: the gamma compositions as deviations
// u = x^gamma - xe_gamma (the variable of the grand-potential difference;
// their Laplacian is that of x^gamma) and the phases.
struct Nb {
  float u1, u2, pd, pl;
};

// With the 9-point mask a row also carries its x-difference sums
// h = (v_w - v) + (v_e - v), formed once per row (two shuffles per field),
// so the diagonal neighbours of the rows above and below cost no shuffles.
struct Nb9 {
  float u1, u2, pd, pl;
  float h1, h2, hd, hl;
};

// With the variable mobility a row also carries each cell's diffusivity
// matrix D(X, Y), scaled by dt / (2 dx^2) (dev::dmat32), for the face sums of
// the divergence.
struct NbV {
  float u1, u2, pd, pl;
  float d00, d01, d10, d11;
};

template <bool NINE, bool VM = false>
using NbT = typename std::conditional<NINE, Nb9,
                                      typename std::conditional<VM, NbV, Nb>::type>::type;

// Compensation record: packed 16-bit counts or four FP32 values.
template <bool PACK>
using CompT = typename std::conditional<PACK, uint2, float4>::type;

template <bool PACK>
struct Raw {
  float4 a;       // x_Cr, x_Nb, phi_del, phi_lav
  CompT<PACK> c;  // Kahan compensations
};

// Per-warp staging ring in shared memory (the batched kernel): rows are
// copied with cp.async kDepth-2 rows ahead of the row being solved, so a warp
// keeps several rows of loads in flight without holding them in registers.
constexpr int kDepth = 4;  // a power of two
template <bool PACK>
struct Ring {
  float4 a[kDepth][32];
  CompT<PACK> c[kDepth][32];
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// the composition compensations only (what the gamma solve needs)
template <bool PACK>
__device__ __forceinline__ float2 comps_x(const CompT<PACK>& c) {
  if constexpr (PACK) {
    const float2 h = cq_halves(c.x);
    return make_float2(h.x * kCqXi, h.y * kCqXi);
  } else {
    return make_float2(c.x, c.y);
  }
}

// the phases' compensations, and the bits that are zero with them (signs of
// FP32 zeros aside)
template <bool PACK>
__device__ __forceinline__ float2 comps_p(const CompT<PACK>& c) {
  if constexpr (PACK) {
    const float2 h = cq_halves(c.y);
    return make_float2(h.x * kCqPi, h.y * kCqPi);
  } else {
    return make_float2(c.z, c.w);
  }
}
__device__ __forceinline__ unsigned comp_bits(const uint2& c) { return c.y; }
__device__ __forceinline__ unsigned comp_bits(const float4& c) {
  return __float_as_uint(c.z) | __float_as_uint(c.w);
}

template <bool PACK, bool NINE, bool VM = false>
struct Stream {
  const Step2DArgs& a;
  const float4* A;        // this lane's column, row 0
  const CompT<PACK>* B;
  float4* Ao;
  CompT<PACK>* Bo;
  int Ny, P;
  bool out;  // this lane writes its column

  __device__ __forceinline__ int row(int y) const { return min(max(y, 0), Ny - 1) * P; }

  __device__ __forceinline__ Raw<PACK> load(int off) const {
    return Raw<PACK>{__ldg(A + off), __ldg(B + off)};
  }

  __device__ __forceinline__ void store(int y, const Raw<PACK>& r) const {
    if (out) {
      const int i = y * P;
      Ao[i] = r.a;
      Bo[i] = r.c;
    }
  }

  // The record of a row one step on, from its window (up, c, dn); rc = its
  // raw record.  still: the phases and their compensations are zero in all
  // three rows (Row::still): they stay zero.
  __device__ __forceinline__ Raw<PACK> step(const NbT<NINE, VM>& up, const NbT<NINE, VM>& c,
                                            const NbT<NINE, VM>& dn, const Raw<PACK>& rc,
                                            bool still) const {
    float lapCr, lapNb, lapD = 0.0f, lapL = 0.0f;
    if constexpr (VM) {
      // variable mobility: lapCr, lapNb hold dt times the divergence of
      // D grad u over the four faces, ((D_n + D_c)(u_n - u_c) summed), the
      // matrices already scaled by dt / (2 dx^2), y faces weighted by qy.
      // Each lane forms the flux through its east face; its west face's is
      // the east flux of the lane to its left (so both cells of a face use
      // the same number, and the x fluxes conserve each component exactly).
      auto dn1 = [](float v) { return __shfl_down_sync(0xffffffffu, v, 1); };
      auto up1 = [](float v) { return __shfl_up_sync(0xffffffffu, v, 1); };
      NbV e;
      e.u1 = dn1(c.u1);
      e.u2 = dn1(c.u2);
      e.d00 = dn1(c.d00);
      e.d01 = dn1(c.d01);
      e.d10 = dn1(c.d10);
      e.d11 = dn1(c.d11);
      // flux of component row (n0 + c0, n1 + c1) into the centre from neighbour n
      auto in = [&](const NbV& n, float n0, float n1, float c0, float c1) {
        return fmaf(n0 + c0, n.u1 - c.u1, (n1 + c1) * (n.u2 - c.u2));
      };
      const float fCr = in(e, e.d00, e.d01, c.d00, c.d01), fNb = in(e, e.d10, e.d11, c.d10, c.d11);
      const float qy = a.vm_qy;
      lapCr = (fCr - up1(fCr)) +
              qy * (in(up, up.d00, up.d01, c.d00, c.d01) + in(dn, dn.d00, dn.d01, c.d00, c.d01));
      lapNb = (fNb - up1(fNb)) +
              qy * (in(up, up.d10, up.d11, c.d10, c.d11) + in(dn, dn.d10, dn.d11, c.d10, c.d11));
      if (!still) {
        Nb w;
        w.pd = up1(c.pd);
        w.pl = up1(c.pl);
        e.pd = dn1(c.pd);
        e.pl = dn1(c.pl);
        const float idx2 = a.idx2f[0], idy2 = a.idx2f[1];
        auto lap = [&](float vw, float ve, float vn, float vs, float vc) {
          return fmaf((vw - vc) + (ve - vc), idx2, ((vn - vc) + (vs - vc)) * idy2);
        };
        lapD = lap(w.pd, e.pd, up.pd, dn.pd, c.pd);
        lapL = lap(w.pl, e.pl, up.pl, dn.pl, c.pl);
      }
    } else if constexpr (NINE) {
      // sum over the eight neighbours of w (v - v_c): with sy = (v_up - v_c)
      // + (v_dn - v_c) the corners add up to h_up + h_dn + 2 sy; then the
      // sum of the nine weights times the centre value (zero for dx = dy up
      // to rounding; k = that sum times xe_gamma for the deviations u)
      const float ex = a.lap9[0], ey = a.lap9[1], cw = a.lap9[2], sw = a.lap9[3];
      auto lap = [&](float hu, float hc, float hd, float vu, float vc, float vd, float k) {
        const float sy = (vu - vc) + (vd - vc);
        float t = fmaf(sw, vc, k);
        t = fmaf(cw, fmaf(2.0f, sy, hu + hd), t);
        t = fmaf(ey, sy, t);
        return fmaf(ex, hc, t);
      };
      lapCr = lap(up.h1, c.h1, dn.h1, up.u1, c.u1, dn.u1, a.lap9xe[0]);
      lapNb = lap(up.h2, c.h2, dn.h2, up.u2, c.u2, dn.u2, a.lap9xe[1]);
      if (!still) {
        lapD = lap(up.hd, c.hd, dn.hd, up.pd, c.pd, dn.pd, 0.0f);
        lapL = lap(up.hl, c.hl, dn.hl, up.pl, c.pl, dn.pl, 0.0f);
      }
    } else {
      Nb w, e;
      w.u1 = __shfl_up_sync(0xffffffffu, c.u1, 1);
      w.u2 = __shfl_up_sync(0xffffffffu, c.u2, 1);
      e.u1 = __shfl_down_sync(0xffffffffu, c.u1, 1);
      e.u2 = __shfl_down_sync(0xffffffffu, c.u2, 1);
      const float idx2 = a.idx2f[0], idy2 = a.idx2f[1];
      auto lap = [&](float vw, float ve, float vn, float vs, float vc) {
        const float sx = (vw - vc) + (ve - vc);
        const float sy = (vn - vc) + (vs - vc);
        return fmaf(sx, idx2, sy * idy2);
      };
      lapCr = lap(w.u1, e.u1, up.u1, dn.u1, c.u1);
      lapNb = lap(w.u2, e.u2, up.u2, dn.u2, c.u2);
      if (!still) {
        w.pd = __shfl_up_sync(0xffffffffu, c.pd, 1);
        w.pl = __shfl_up_sync(0xffffffffu, c.pl, 1);
        e.pd = __shfl_down_sync(0xffffffffu, c.pd, 1);
        e.pl = __shfl_down_sync(0xffffffffu, c.pl, 1);
        lapD = lap(w.pd, e.pd, up.pd, dn.pd, c.pd);
        lapL = lap(w.pl, e.pl, up.pl, dn.pl, c.pl);
      }
    }
    const float2 cx = comps_x<PACK>(rc.c);
    // Cahn-Hilliard
    const float X = rc.a.x, Y = rc.a.y;
    float ycr, ynb;
    if constexpr (VM) {
      ycr = lapCr - cx.x;
      ynb = lapNb - cx.y;
    } else {
      ycr = fmaf(a.dtD[0][0], lapCr, a.dtD[0][1] * lapNb) - cx.x;
      ynb = fmaf(a.dtD[1][0], lapCr, a.dtD[1][1] * lapNb) - cx.y;
    }
    const float tcr = X + ycr, tnb = Y + ynb;
    const float ox = (tcr - X) - ycr, oy = (tnb - Y) - ynb;
    Raw<PACK> r;
    if (still) {
      r.a = make_float4(tcr, tnb, 0.0f, 0.0f);
      if constexpr (PACK)
        r.c = make_uint2(cq_pair(ox * kCqX, oy * kCqX), 0u);
      else
        r.c = make_float4(ox, oy, 0.0f, 0.0f);
      return r;
    }
    // Allen-Cahn
    const FastCoef& K = a.k;
    const float2 cp = comps_p<PACK>(rc.c);
    const float phd = c.pd, phl = c.pl;
    const float dFd = fmaf(-a.kap[0], lapD, dF_local32(phd, phl, quad2(K.dP[0], c.u1, c.u2), a.om2[0], a.alpha2));
    const float dFl = fmaf(-a.kap[1], lapL, dF_local32(phl, phd, quad2(K.dP[1], c.u1, c.u2), a.om2[1], a.alpha2));
    const float yd = fmaf(-a.dtL[0], dFd, -cp.x), td = phd + yd;
    const float yl = fmaf(-a.dtL[1], dFl, -cp.y), tl = phl + yl;
    r.a = make_float4(tcr, tnb, td, tl);
    const float od = (td - phd) - yd, ol = (tl - phl) - yl;
    if constexpr (PACK)
      r.c = cq_pack(ox, oy, od, ol);
    else
      r.c = make_float4(ox, oy, od, ol);
    return r;
  }

  // What a step needs of a row's raw record: the gamma solve, and whether
  // the whole warp's phases and their compensations are zero (compositions
  // that are not finite make 0 x NaN in the Allen-Cahn terms and are not
  // still).  Whole warp.
  __device__ __forceinline__ NbT<NINE, VM> solve(const Raw<PACK>& r, bool& still) const {
    const FastCoef& K = a.k;
    const float2 cxy = comps_x<PACK>(r.c);
    NbT<NINE, VM> n;
    n.pd = r.a.z;
    n.pl = r.a.w;
    const unsigned cb = PACK ? comp_bits(r.c) : comp_bits(r.c) & 0x7fffffffu;
    const unsigned z = __float_as_uint(fmaf(r.a.x, 0.0f, fmaf(r.a.y, 0.0f, fabsf(r.a.z)))) |
                       __float_as_uint(fabsf(r.a.w)) | cb;
    still = __all_sync(0xffffffffu, z == 0u);
    // a cell of pure gamma needs no solve; each cell takes its own form,
    // whatever its neighbours in the warp do, so that results do not depend
    // on how a grid is cut into strips
    if (fmaxf(fabsf(r.a.z), fabsf(r.a.w)) >= kBulkPhi)
      gamma_u32(K, r.a.x, r.a.y, cxy.x, cxy.y, r.a.z, r.a.w, n.u1, n.u2);
    else
      gamma_bulk32(K, r.a.x, r.a.y, cxy.x, cxy.y, n.u1, n.u2);
    if constexpr (VM) dmat32(a.vm_pre, r.a.x, r.a.y, n.d00, n.d01, n.d10, n.d11);
    if constexpr (NINE) {
      auto hx = [](float v) {
        return (__shfl_up_sync(0xffffffffu, v, 1) - v) + (__shfl_down_sync(0xffffffffu, v, 1) - v);
      };
      n.h1 = hx(n.u1);
      n.h2 = hx(n.u2);
      if (still) {
        n.hd = n.hl = 0.0f;
      } else {
        n.hd = hx(n.pd);
        n.hl = hx(n.pl);
      }
    }
    return n;
  }
};

// Rows y0 .. y1-1 of the warp's strip, kShortRows at most: all its rows are
// requested at once, so that the warp waits for memory once instead of row by
// row.  (The variable-mobility form has the registers for a fourth row.)
template <bool VM>
constexpr int kShortRows = VM ? 4 : 3;
template <bool PACK, bool NINE, bool VM>
__device__ __forceinline__ void short_segment(const Stream<PACK, NINE, VM>& S, int y0, int y1) {
  bool z0, z1, z2;
  const Raw<PACK> ra = S.load(S.row(y0 - 1)), rb = S.load(S.row(y0)), rc = S.load(S.row(y0 + 1)),
                  rd = S.load(S.row(y0 + 2)), re = S.load(S.row(y0 + 3));
  Raw<PACK> rf;
  if constexpr (VM) rf = S.load(S.row(y0 + 4));
  NbT<NINE, VM> na = S.solve(ra, z0), nb = S.solve(rb, z1), nc = S.solve(rc, z2);
  S.store(y0, S.step(na, nb, nc, rb, z0 && z1 && z2));
  if (y0 + 1 >= y1) return;
  na = S.solve(rd, z0);
  S.store(y0 + 1, S.step(nb, nc, na, rc, z0 && z1 && z2));
  if (y0 + 2 >= y1) return;
  nb = S.solve(re, z1);
  S.store(y0 + 2, S.step(nc, na, nb, rd, z0 && z1 && z2));
  if constexpr (VM) {
    if (y0 + 3 >= y1) return;
    nc = S.solve(rf, z2);
    S.store(y0 + 3, S.step(na, nb, nc, re, z0 && z1 && z2));
  }
}

// One warp updates the strip of output columns x0 .. x0+29 over rows
// y0 .. y1-1 of one grid (the unit of work of both the single-grid and the
// batched kernels).  Whole warp; x0 < Nx.  Rows reach the registers either
// directly (one row ahead, !STAGED) or through the warp's staging ring
// (STAGED): the batched kernel's units are short, and the ring's deeper
// prefetch hides the start-up latency each unit pays.
template <bool PACK, bool STAGED, bool NINE = false, bool VM = false>
__device__ __forceinline__ void stream_strip(const Step2DArgs& a, const float4* Ain,
                                             const CompT<PACK>* Bin, float4* Aout,
                                             CompT<PACK>* Bout, int Nx, int Ny, int P, int x0,
                                             int y0, int y1, Ring<PACK>* ring) {
  const int lane = threadIdx.x & 31;
  const int gx = x0 - 1 + lane;  // lanes 0 and 31 hold the neighbour columns
  const int cx = min(max(gx, 0), Nx - 1);
  static_assert(!(STAGED && NINE), "the staged (batched) form has the 5-point mask only");
  static_assert(!(STAGED && VM), "the staged (batched) form has the constant mobility only");
  static_assert(!(NINE && VM), "the variable-mobility form has the 5-point mask only");
  const Stream<PACK, NINE, VM> S{a, Ain + cx, Bin + cx, Aout + cx, Bout + cx,
                             Ny, P, lane >= 1 && lane <= kCols && gx < Nx};
  bool z0, z1, z2;  // rows y-1, y, y+1 are still
  if constexpr (!STAGED) {
    if (y1 - y0 <= kShortRows<VM>) {
      short_segment(S, y0, y1);
      return;
    }
    // window rows y-1, y, y+1 and raw records of rows y, y+1, y+2
    Raw<PACK> r0 = S.load(S.row(y0)), r1 = S.load(S.row(y0 + 1)), r2;
    NbT<NINE, VM> n0 = S.solve(S.load(S.row(y0 - 1)), z0), n1 = S.solve(r0, z1), n2;
    // three rows per iteration with rotated roles: no register moves
    int y = y0;
    for (; y + 2 < y1; y += 3) {
      r2 = S.load(S.row(y + 2));
      n2 = S.solve(r1, z2);
      S.store(y, S.step(n0, n1, n2, r0, z0 && z1 && z2));
      r0 = S.load(S.row(y + 3));
      n0 = S.solve(r2, z0);
      S.store(y + 1, S.step(n1, n2, n0, r1, z0 && z1 && z2));
      r1 = S.load(S.row(y + 4));
      n1 = S.solve(r0, z1);
      S.store(y + 2, S.step(n2, n0, n1, r2, z0 && z1 && z2));
    }
    for (; y < y1; y++) {
      r2 = S.load(S.row(y + 2));
      n2 = S.solve(r1, z2);
      S.store(y, S.step(n0, n1, n2, r0, z0 && z1 && z2));
      n0 = n1;
      n1 = n2;
      z0 = z1;
      z1 = z2;
      r0 = r1;
      r1 = r2;
    }
  } else {
    if (y1 - y0 <= kShortRows<VM>) {
      short_segment(S, y0, y1);
      return;
    }
    // ring slot k holds rows y0-1+k, y0-1+k+kDepth, ...; each lane copies and
    // reads back only its own column's records, so the wait needs no warp sync
    const uint32_t sa = uint32_t(__cvta_generic_to_shared(&ring->a[0][lane]));
    const uint32_t sc = uint32_t(__cvta_generic_to_shared(&ring->c[0][lane]));
    constexpr uint32_t kSlotA = 32 * sizeof(float4), kSlotC = 32 * sizeof(CompT<PACK>);
    auto issue = [&](int y, int slot) {
      if (y <= y1) {  // rows past y1 are never read
        const int off = S.row(y);
        cp_async16(sa + slot * kSlotA, S.A + off);
        if constexpr (PACK)
          cp_async8(sc + slot * kSlotC, S.B + off);
        else
          cp_async16(sc + slot * kSlotC, S.B + off);
      }
      cp_commit();  // one group per row (empty past y1): the wait counts stay uniform
    };
    auto fetch = [&](int slot) { return Raw<PACK>{ring->a[slot][lane], ring->c[slot][lane]}; };
#pragma unroll
    for (int k = 0; k < kDepth; k++) issue(y0 - 1 + k, k);
    cp_wait<kDepth - 2>();  // rows y0-1 and y0 have landed
    Nb n0 = S.solve(fetch(0), z0), n1 = S.solve(fetch(1), z1), n2;
    int s = 0;  // slot of row y-1
    // row y: refill the slot of row y-1 (read for row y-1's update) with row
    // y-1+kDepth, wait for row y+1 (kDepth-2 newer groups stay in flight),
    // solve it, update row y.  Rows up to y1 were all waited for by the last
    // row, so no copy into the ring is pending when the strip ends.
    auto body = [&](int y, const Nb& up, const Nb& c, Nb& dn, bool& zdn) {
      issue(y - 1 + kDepth, s);
      s = (s + 1) & (kDepth - 1);
      cp_wait<kDepth - 2>();
      dn = S.solve(fetch((s + 1) & (kDepth - 1)), zdn);
      S.store(y, S.step(up, c, dn, fetch(s), z0 && z1 && z2));
    };
    int y = y0;
    for (; y + 2 < y1; y += 3) {
      body(y, n0, n1, n2, z2);
      body(y + 1, n1, n2, n0, z0);
      body(y + 2, n2, n0, n1, z1);
    }
    for (; y < y1; y++) {
      body(y, n0, n1, n2, z2);
      n0 = n1;
      n1 = n2;
      z0 = z1;
      z1 = z2;
    }
  }
}

// The packed form fits 9 CTAs per SM (56 registers, no spills): the extra
// warps cover load latency (4096^2: 0.1303 ms vs 0.1369 ms at 8); the FP32
// compensation form is faster at 8.  NINE: the 9-point mask (a window of
// eight values per row).
template <bool PACK, bool NINE, bool VM = false>
__global__ void __launch_bounds__(32 * kWarps, VM ? 6 : (PACK && !NINE ? 9 : 8))
    k_stream_f32(Step2DArgs a) {
  const int strip = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const int x0 = strip * kCols;  // first output column of the strip
  if (x0 >= a.Nx) return;        // whole warp leaves together
  const int y0 = blockIdx.y * a.rows;
  stream_strip<PACK, false, NINE, VM>(a, static_cast<const float4*>(a.in[0]),
                            static_cast<const CompT<PACK>*>(a.in[1]),
                            static_cast<float4*>(a.out[0]), static_cast<CompT<PACK>*>(a.out[1]),
                            a.Nx, a.Ny, a.pitch, x0, y0, min(y0 + a.rows, a.Ny), nullptr);
}

// the record of the lane that holds this lane's column
template <bool PACK>
__device__ __forceinline__ Raw<PACK> mirrored(const Raw<PACK>& r, int lane) {
  auto m = [&](float v) { return __shfl_sync(0xffffffffu, v, lane); };
  Raw<PACK> t;
  t.a = make_float4(m(r.a.x), m(r.a.y), m(r.a.z), m(r.a.w));
  if constexpr (PACK)
    t.c = make_uint2(__shfl_sync(0xffffffffu, r.c.x, lane), __shfl_sync(0xffffffffu, r.c.y, lane));
  else
    t.c = make_float4(m(r.c.x), m(r.c.y), m(r.c.z), m(r.c.w));
  return t;
}

// ---- two steps in one pass ----
// The strip of output columns x0 .. x0+27 over rows y0 .. y1-1, two steps on:
// row y+1 is advanced once (from rows y, y+1, y+2 as loaded), solved again,
// and row y advanced the second time from its once-advanced neighbours, all
// in registers, so a record crosses HBM once for two steps.  The values and
// their order of operations are those of two single steps (the packed
// compensations are rounded in between as the store would), so the result is
// the same bits.  Lanes 0, 1 and 30, 31 are halo: the first step is right on
// lanes 1 .. 30, the second on 2 .. 29.  A once-advanced record beyond the
// domain mirrors the one at its edge.
//
// Bound: latency and issue (124 instructions a cell and step, 74 % of the
// issue slots; HBM would allow 60 us a step at 4096^2).  Rows come through a
// per-warp cp.async ring, which holds the row whose first step is due besides
// the rows ahead and so leaves 80 registers without spills, 6 CTAs per SM
// (rows in registers, one ahead: 89.8 us; 7 or 8 CTAs with spills: 118 and
// 101).  4096^2: 129 us a step in single steps -> 71.7; FP32 compensations 176
// -> 85, 9 points 131 -> 91; 2048^2 35.3 -> 22.8.
constexpr int kCols2 = 28;
constexpr int kDepth2 = 8;  // rows in the ring (a power of two)
template <bool PACK>
struct Ring2 {
  float4 a[kDepth2][32];
  CompT<PACK> c[kDepth2][32];
};

template <bool PACK, bool NINE>
__device__ __forceinline__ void stream_strip2(const Step2DArgs& a, const float4* Ain,
                                              const CompT<PACK>* Bin, float4* Aout,
                                              CompT<PACK>* Bout, int Nx, int Ny, int P, int x0,
                                              int y0, int y1, Ring2<PACK>* ring) {
  const int lane = threadIdx.x & 31;
  const int gx = x0 - 2 + lane;
  const int cx = min(max(gx, 0), Nx - 1);
  const Stream<PACK, NINE> S{a, Ain + cx, Bin + cx, Aout + cx, Bout + cx, Ny, P,
                                 lane >= 2 && lane < 2 + kCols2 && gx < Nx};
  const bool edge = x0 == 0 || x0 + kCols2 >= Nx;  // whole warp
  const int mirror = cx - (x0 - 2);                // the lane holding column cx
  using N = NbT<NINE>;
  using R = Raw<PACK>;
  // ring slot k holds rows y0-2+k, y0-2+k+kDepth2, ...; each lane copies and
  // reads back only its own column's records, so the waits need no warp sync
  const uint32_t sa = uint32_t(__cvta_generic_to_shared(&ring->a[0][lane]));
  const uint32_t sc = uint32_t(__cvta_generic_to_shared(&ring->c[0][lane]));
  constexpr uint32_t kSlotA = 32 * sizeof(float4), kSlotC = 32 * sizeof(CompT<PACK>);
  auto issue = [&](int y, int slot) {
    if (y <= y1 + 1) {  // rows past y1 + 1 are never read
      const int off = S.row(y);
      cp_async16(sa + slot * kSlotA, S.A + off);
      if constexpr (PACK)
        cp_async8(sc + slot * kSlotC, S.B + off);
      else
        cp_async16(sc + slot * kSlotC, S.B + off);
    }
    cp_commit();  // one group per row (empty past y1 + 1): the wait counts stay uniform
  };
  auto fetch = [&](int slot) { return R{ring->a[slot][lane], ring->c[slot][lane]}; };
  // first step of a row
  auto first = [&](const N& up, const N& c, const N& dn, const R& rc, bool still) {
    const R r = S.step(up, c, dn, rc, still);
    return edge ? mirrored(r, mirror) : r;
  };
#pragma unroll
  for (int k = 0; k < kDepth2; k++) issue(y0 - 2 + k, k);
  cp_wait<kDepth2 - 4>();  // rows y0-2 .. y0+1 have landed
  // s: solves of the loaded rows y, y+1, y+2; u: solves of the once-advanced
  // rows y-1, y, y+1; t: once-advanced records of rows y, y+1
  N s0, s1, s2, u0, u1, u2;
  R t1, t2, t0;
  bool zs0, zs1, zs2, zu0, zu1, zu2;
  {
    bool za, zb;
    const N sa_ = S.solve(fetch(0), za), sb_ = S.solve(fetch(1), zb);
    s0 = S.solve(fetch(2), zs0);
    s1 = S.solve(fetch(3), zs1);
    t1 = first(sb_, s0, s1, fetch(2), zb && zs0 && zs1);
    t0 = y0 == 0 ? t1 : first(sa_, sb_, s0, fetch(1), za && zb && zs0);
    u0 = S.solve(t0, zu0);
    u1 = S.solve(t1, zu1);
  }
  issue(y0 - 2 + kDepth2, 0);
  issue(y0 - 1 + kDepth2, 1);
  int s = 2;  // slot of row y
  // one output row: row y's slot is refilled with row y+kDepth2, row y+2 waited
  // for (kDepth2-2 newer groups stay in flight); window (sa, sb, sc), window
  // (ua, ub, uc), records tb in, tc out
  auto body = [&](int y, const N& sa, const N& sb, N& sc, bool za, bool zb, bool& zc, const N& ua,
                  const N& ub, N& uc, bool wa, bool wb, bool& wc, const R& tb, R& tc) {
    issue(y + kDepth2, s);
    s = (s + 1) & (kDepth2 - 1);
    cp_wait<kDepth2 - 2>();
    sc = S.solve(fetch((s + 1) & (kDepth2 - 1)), zc);
    tc = first(sa, sb, sc, fetch(s), za && zb && zc);
    if (y + 1 >= Ny) tc = tb;
    uc = S.solve(tc, wc);
    S.store(y, S.step(ua, ub, uc, tb, wa && wb && wc));
  };
  int y = y0;
  for (; y + 2 < y1; y += 3) {
    body(y, s0, s1, s2, zs0, zs1, zs2, u0, u1, u2, zu0, zu1, zu2, t1, t2);
    body(y + 1, s1, s2, s0, zs1, zs2, zs0, u1, u2, u0, zu1, zu2, zu0, t2, t0);
    body(y + 2, s2, s0, s1, zs2, zs0, zs1, u2, u0, u1, zu2, zu0, zu1, t0, t1);
  }
  for (; y < y1; y++) {
    body(y, s0, s1, s2, zs0, zs1, zs2, u0, u1, u2, zu0, zu1, zu2, t1, t2);
    s0 = s1;
    s1 = s2;
    zs0 = zs1;
    zs1 = zs2;
    u0 = u1;
    u1 = u2;
    zu0 = zu1;
    zu1 = zu2;
    t1 = t2;
  }
  cp_wait<0>();  // only empty groups are left
}

template <bool PACK, bool NINE>
__global__ void __launch_bounds__(32 * kWarps, PACK && !NINE ? 6 : 4) k_stream2_f32(Step2DArgs a) {
  __shared__ Ring2<PACK> ring[kWarps];
  const int strip = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const int x0 = strip * kCols2;
  if (x0 >= a.Nx) return;
  const int y0 = blockIdx.y * a.rows;
  stream_strip2<PACK, NINE>(a, static_cast<const float4*>(a.in[0]),
                                static_cast<const CompT<PACK>*>(a.in[1]),
                                static_cast<float4*>(a.out[0]), static_cast<CompT<PACK>*>(a.out[1]),
                                a.Nx, a.Ny, a.pitch, x0, y0, min(y0 + a.rows, a.Ny),
                                &ring[threadIdx.x >> 5]);
}

// ---- several steps in one launch of tiles ----
// A CTA holds a region of 32 x kTileRows cells, a row per warp and a cell's
// record per thread, and takes it a.steps steps S on: in each a warp solves
// its row, publishes it for the rows above and below, and advances it; the
// rows and columns that are right shrink by one a side and step, and the
// region's middle (32 - 2 S) x (kTileRows - 2 S) cells are stored.  Records
// beyond the domain mirror its edge: a warp's lanes by a copy after each
// step, rows by reading the edge's own row.  The values and their order of
// operations are those of single steps (the packed compensations are rounded
// after each step as the store would), so the result is the same bits.
//
// What it saves is launches, 2.4 us each, of which a small grid's step itself
// takes a quarter; it is bound by the latency of a step's chain (0.65 us where
// an SM holds one CTA) and by issue.  Regions of 32 rows take 1.1 us a step:
// 64 x 48 1.5 us a step against 1.0, 128^2 1.5 / 1.15, 256^2 1.74 / 1.76.
constexpr int kTileRows = 16;
template <bool NINE, bool VM>
constexpr size_t tile_bytes() {  // at most 33 KB
  return 2 * kTileRows * (32 * sizeof(NbT<NINE, VM>) + sizeof(int));
}

template <bool PACK, bool NINE, bool VM>
__global__ void __launch_bounds__(32 * kTileRows, 2) k_tile_f32(Step2DArgs a) {
  using N = NbT<NINE, VM>;
  extern __shared__ float4 s_tile[];
  N* nb = reinterpret_cast<N*>(s_tile);                       // [2][kTileRows][32]
  int* still = reinterpret_cast<int*>(nb + 2 * kTileRows * 32);  // [2][kTileRows]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, S = a.steps;
  const int x0 = blockIdx.x * (32 - 2 * S), y0 = blockIdx.y * (kTileRows - 2 * S);
  const int gx = x0 - S + lane, gy = y0 - S + w;
  const int cx = min(max(gx, 0), a.Nx - 1);
  using C = CompT<PACK>;
  const Stream<PACK, NINE, VM> T{a, static_cast<const float4*>(a.in[0]) + cx, static_cast<const C*>(a.in[1]) + cx,
                                 static_cast<float4*>(a.out[0]) + cx, static_cast<C*>(a.out[1]) + cx,
                                 a.Ny, a.pitch, lane >= S && lane < 32 - S && gx < a.Nx};
  Raw<PACK> r = T.load(T.row(gy));
  const bool inside = gy >= 0 && gy < a.Ny;  // whole warp, as all below
  const bool edge = x0 - S < 0 || x0 + 32 - S > a.Nx;
  const int mirror = cx - (x0 - S);  // the lane holding column cx
  const int up = gy <= 0 ? w : w - 1, dn = gy >= a.Ny - 1 ? w : w + 1;
  for (int k = 0; k < S; k++) {
    N* rows = nb + (k & 1) * kTileRows * 32;
    int* z = still + (k & 1) * kTileRows;
    const bool solves = inside && w >= k && w < kTileRows - k;
    N n;
    bool own = true;
    if (solves) {
      n = T.solve(r, own);
      rows[w * 32 + lane] = n;
      if (lane == 0) z[w] = own;
    }
    // this buffer was last read before the barrier of step k - 1
    __syncthreads();
    if (solves && w > k && w < kTileRows - 1 - k) {
      r = T.step(rows[up * 32 + lane], n, rows[dn * 32 + lane], r, own && z[up] && z[dn]);
      if (edge) r = mirrored(r, mirror);
    }
  }
  if (inside && w >= S && w < kTileRows - S) T.store(gy, r);
}

// ---- many grids in one launch ----
// The units (grid, strip, row segment) of the batch's unit table, their count
// in counter[2] (TWO: counter[3]).  A persistent launch has one CTA per
// resident slot, whose warps claim units through an atomic counter
// (counter[parity]), so a captured launch stays valid while the table's
// contents change; the launch also zeroes the other parity's counter for the
// next launch, which stream order runs after this one.  The other shape has
// one warp per unit and leaves the balancing to the block scheduler; single
// steps then take the warp's own unit, with no claim to wait for, which small
// batches of short segments feel (us a step, best of the persistent shapes
// with segments of 6 and 12 rows -> segments of 3 rows, a warp each: 4 grids of
// 64-512 9.1 -> 6.6, 24 of 64-512 19.4 -> 13.8).  TWO: two steps in one pass
// (strips of 28 columns), else one (strips of 30).
template <bool TWO>
__global__ void __launch_bounds__(32 * kWarps, TWO ? 6 : 8) k_batch_f32(Step2DArgs a, BatchArgs b) {
  const int p = b.parity;
  if (blockIdx.x == 0 && threadIdx.x == 0) b.counter[p ^ 1] = 0;
  const int units = b.counter[TWO ? 3 : 2];
  using R = typename std::conditional<TWO, Ring2<true>, Ring<true>>::type;
  __shared__ R ring[kWarps];
  const bool claims = TWO || b.persistent;
  for (int u = blockIdx.x * kWarps + (threadIdx.x >> 5);; u = units) {
    if (claims) {
      if ((threadIdx.x & 31) == 0) u = atomicAdd(b.counter + p, 1);
      u = __shfl_sync(0xffffffffu, u, 0);
    }
    if (u >= units) return;
    const BatchUnit w = b.unit[u];
    const BatchGrid& g = b.grid[w.grid];
    R* r = &ring[threadIdx.x >> 5];
    if constexpr (TWO)
      stream_strip2<true, false>(a, g.A[p], g.B[p], g.A[p ^ 1], g.B[p ^ 1], g.Nx, g.Ny, g.pitch,
                                 w.x0, w.y0, w.y1, r);
    else
      stream_strip<true, true>(a, g.A[p], g.B[p], g.A[p ^ 1], g.B[p ^ 1], g.Nx, g.Ny, g.pitch,
                               w.x0, w.y0, w.y1, r);
  }
}

// ---- layout conversion between the reference's FP64 fields and the form ----
__global__ void k_import_records(ConvArgs a) {
  const int gx = blockIdx.x * blockDim.x + threadIdx.x;
  const int gy = a.y0 + int(blockIdx.y * blockDim.y + threadIdx.y);
  if (gx >= a.Nx || gy >= (a.y1 > 0 ? a.y1 : a.Ny)) return;
  const size_t i64 = size_t(gy + 1) * a.pitch64 + gx + 1;
  const size_t r = size_t(gy) * a.pitch32 + gx;
  float hi[4], c[4];
#pragma unroll
  for (int k = 0; k < 4; k++) split_f64(a.f64[k][i64], hi[k], c[k]);  // value = hi - c
  reinterpret_cast<float4*>(a.A)[r] = make_float4(hi[0], hi[1], hi[2], hi[3]);
  if (a.pack)
    static_cast<uint2*>(a.B)[r] = cq_pack(c[0], c[1], c[2], c[3]);
  else
    static_cast<float4*>(a.B)[r] = make_float4(c[0], c[1], c[2], c[3]);
}

__global__ void k_export_records(ConvArgs a) {
  const int gx = blockIdx.x * blockDim.x + threadIdx.x;
  const int gy = a.y0 + int(blockIdx.y * blockDim.y + threadIdx.y);
  if (gx >= a.Nx || gy >= (a.y1 > 0 ? a.y1 : a.Ny)) return;
  const size_t r = size_t(gy) * a.pitch32 + gx;
  const float4 v = reinterpret_cast<const float4*>(a.A)[r];
  double val[4];
  if (a.pack) {
    merge_record(v, static_cast<const uint2*>(a.B)[r], val);
  } else {
    const float4 c = static_cast<const float4*>(a.B)[r];
    val[0] = double(v.x) - double(c.x);
    val[1] = double(v.y) - double(c.y);
    val[2] = double(v.z) - double(c.z);
    val[3] = double(v.w) - double(c.w);
  }
  const size_t row = size_t(gy + 1) * a.pitch64;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    double* f = a.f64[k];
    f[row + gx + 1] = val[k];
    // ghost ring = mirror of the interior; corners take the diagonal cell
    const bool l = gx == 0, rr = gx == a.Nx - 1, b = gy == 0, t = gy == a.Ny - 1;
    if (l) f[row] = val[k];
    if (rr) f[row + a.Nx + 1] = val[k];
    if (b) {
      f[gx + 1] = val[k];
      if (l) f[0] = val[k];
      if (rr) f[a.Nx + 1] = val[k];
    }
    if (t) {
      const size_t top = size_t(a.Ny + 1) * a.pitch64;
      f[top + gx + 1] = val[k];
      if (l) f[top] = val[k];
      if (rr) f[top + a.Nx + 1] = val[k];
    }
  }
}

// at most 65535 segments (the launch grid's second dimension), none past Ny
int grid_rows(int rows, int Ny) { return std::min(std::max(rows, (Ny + 65534) / 65535), Ny); }

// Rows per warp segment of a single step.  Each segment solves two extra
// rows, but the more segments there are the better they balance, and a
// segment of up to three rows waits for memory once (a longer one row by row,
// about 0.4 us each where few warps share an SM).  us a step at 1 / 2 / 3 / 6
// / 12 rows: 256^2 2.7 / 3.1 / 3.4 / 5.2 / 8.0, 384^2 3.3 / 3.3 / 3.7 / 5.2 /
// 8.1, 700 x 433 4.5 / 4.1 / 4.4 / 5.7 / 8.4, 900 x 600 6.1 / 5.1 / 4.9 / 6.2
// / 8.9, 1024^2 10.0 / 7.5 / 7.0 / 7.9 / 10.1, 2048^2 45.8 / 33.5 / 30.2 /
// 33.0 / 36.3; the same order in the 9-point form.  The variable-mobility
// step, whose extra rows cost three exponentials a cell, takes 4 from four CTA
// rows per resident CTA on (us a step at 3 / 4 / 6 / 9 rows: 512^2 5.0 / 5.3 /
// 6.3 / 7.4, 900 x 600 7.0 / 6.7 / 7.7 / 8.6, 1024^2 10.5 / 10.3 / 11.1 / 11.5,
// 1531 x 1021 15.3 / 14.4 / 15.0 / 15.1, 4096^2 163 / 143 / 149 / 146).
int segment_rows(int Nx, int Ny, int resident, bool varmob) {
  const int nbx = ((Nx + kCols - 1) / kCols + kWarps - 1) / kWarps;
  const double load = double(nbx) * Ny / resident;  // CTA rows per resident CTA
  const int rows = load <= 1.0 ? 1 : load <= 2.5 ? 2 : !varmob || load <= 4.0 ? 3 : 4;
  return grid_rows(rows, Ny);
}

// resident CTAs: FP32 / packed variants, the batch kernel, the 9-point FP32 / packed
// variants, the variable-mobility FP32 / packed variants
int g_sms = 0;
int g_resident[12] = {};  // + 7: the two-step kernels (constant mobility), 11: the batch's

template <typename K>
cudaError_t query_resident(K kernel, int slot) {
  int dev = 0, sms = 0, per = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 32 * kWarps, 0);
  g_sms = sms;
  g_resident[slot] = sms * (per > 0 ? per : 1);
  return e;
}

template <bool PACK, bool NINE, bool VM = false>
cudaError_t launch_stream(Step2DArgs a, cudaStream_t s) {
  const int slot = VM ? 5 + PACK : (NINE ? 3 + PACK : PACK);
  const int resident = g_resident[slot] > 0 ? g_resident[slot] : 152 * 8;
  a.rows = segment_rows(a.Nx, a.Ny, resident, VM);
  const int strips = (a.Nx + kCols - 1) / kCols;
  dim3 grid((strips + kWarps - 1) / kWarps, (a.Ny + a.rows - 1) / a.rows);
  k_stream_f32<PACK, NINE, VM><<<grid, 32 * kWarps, 0, s>>>(a);
  return cudaGetLastError();
}

// Rows per segment of a two-step pass: each segment solves six extra rows and
// waits for its first four, fewer rows balance the CTAs better; the product
// of (1 + c / rows) and (1 + d rows / load) is least at sqrt(c load / d),
// with c / d = 6 from the sweeps (us a step at 6 / 9 / 15 / 24 / 36 / 96 rows:
// 2048^2 26.2 / 24.1 / 22.8 / 24.1 / 27.1 / 35.8, 4096^2 94.2 / 86.1 / 79.5 /
// 76.4 / 76.1 / 77.7); a multiple of the unrolled loop's three.
int segment_rows2(int Nx, int Ny, int resident) {
  const int nbx = ((Nx + kCols2 - 1) / kCols2 + kWarps - 1) / kWarps;
  const double load = double(nbx) * Ny / resident;  // CTA rows per resident CTA
  const int rows = 3 * std::max(2, int(std::sqrt(6.0 * load) / 3.0 + 0.5));
  return grid_rows(rows, Ny);
}

template <bool PACK, bool NINE, bool VM>
cudaError_t launch_tile(Step2DArgs a, int steps, cudaStream_t s) {
  a.steps = steps;
  const int nx = 32 - 2 * steps, ny = kTileRows - 2 * steps;
  const dim3 grid((a.Nx + nx - 1) / nx, (a.Ny + ny - 1) / ny);
  k_tile_f32<PACK, NINE, VM><<<grid, 32 * kTileRows, tile_bytes<NINE, VM>(), s>>>(a);
  return cudaGetLastError();
}

template <bool PACK, bool NINE>
cudaError_t launch_stream2(Step2DArgs a, cudaStream_t s) {
  const int slot = 7 + 2 * NINE + PACK;
  const int resident = g_resident[slot] > 0 ? g_resident[slot] : 152 * 4;
  a.rows = segment_rows2(a.Nx, a.Ny, resident);
  const int strips = (a.Nx + kCols2 - 1) / kCols2;
  dim3 grid((strips + kWarps - 1) / kWarps, (a.Ny + a.rows - 1) / a.rows);
  k_stream2_f32<PACK, NINE><<<grid, 32 * kWarps, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace

// Two steps in one pass save HBM traffic, which binds once the two record
// sets exceed the L2 (129 MB): at 1531 x 1021 (75 MB) single steps take 10.2
// us and double ones 12.0, at 1536^2 (113 MB) 17.0 and 14.7.  Smaller grids
// are bound by launches and latency, which a pass of twice the work does not
// shorten (256^2 2.96 and 3.09 us).  The variable-mobility step is bound by
// issue (4096^2 137.9 us, 133.8 in double passes): single steps.
bool two_steps_bytes(double bytes) { return bytes > 96e6; }

bool two_steps_f32(const Step2DArgs& a) {
  return !a.varmob && two_steps_bytes(double(a.pitch) * a.Ny * (a.full_comp ? 64 : 48));
}

// Steps per launch of tiles, 0: single steps are faster.  From the sweeps a
// launch takes 2.4 us and, with m CTAs on the most loaded SM, a step 0.25 +
// 0.4 m; past six CTAs per SM of three-step tiles single steps are (us a
// step in tiles / singly: 64 x 48 1.0 / 2.4, 128^2 1.15 / 2.4, 256^2 1.76 /
// 2.7, 384^2 2.7 / 3.3, 512^2 3.9 / 3.9, 700 x 433 4.1 / 4.1; 9 points 384^2
// 3.1 / 3.7, 512^2 4.6 / 4.3; variable mobility 64 x 48 1.25 / 2.5, 256^2 2.2 /
// 3.4, 384^2 3.6 / 4.3, 512^2 5.5 / 5.2).
int tile_steps(int Nx, int Ny) {
  const long long sms = g_sms > 0 ? g_sms : 152;
  auto tiles = [&](int s) {
    const int nx = 32 - 2 * s, ny = kTileRows - 2 * s;
    return ((Nx + nx - 1) / nx) * (long long)((Ny + ny - 1) / ny);
  };
  if (tiles(3) > 6 * sms) return 0;
  int best = 0;
  double least = 1e30;
  for (int s = 2; 2 * s < kTileRows; s++) {
    const double us = 2.4 / s + 0.25 + 0.4 * double((tiles(s) + sms - 1) / sms);
    if (us < least) {
      least = us;
      best = s;
    }
  }
  return best;
}

int pass_steps_f32(const Step2DArgs& a, int most) {
  if (most < 2) return 1;
  if (two_steps_f32(a)) return 2;
  const int s = tile_steps(a.Nx, a.Ny);
  if (s == 0) return 1;
  const int passes = (most + s - 1) / s;  // as even as they go
  return (most + passes - 1) / passes;
}

cudaError_t launch_step2d_f32(const Step2DArgs& a, int steps, cudaStream_t s) {
  if (a.varmob && a.nine) return cudaErrorInvalidValue;  // refused by the host before
  if (steps >= 2 && !two_steps_f32(a)) {
    if (a.varmob) return a.full_comp ? launch_tile<false, false, true>(a, steps, s) : launch_tile<true, false, true>(a, steps, s);
    if (a.nine) return a.full_comp ? launch_tile<false, true, false>(a, steps, s) : launch_tile<true, true, false>(a, steps, s);
    return a.full_comp ? launch_tile<false, false, false>(a, steps, s) : launch_tile<true, false, false>(a, steps, s);
  }
  if (a.varmob)
    return a.full_comp ? launch_stream<false, false, true>(a, s) : launch_stream<true, false, true>(a, s);
  if (steps == 2) {
    if (a.nine) return a.full_comp ? launch_stream2<false, true>(a, s) : launch_stream2<true, true>(a, s);
    return a.full_comp ? launch_stream2<false, false>(a, s) : launch_stream2<true, false>(a, s);
  }
  if (a.nine) return a.full_comp ? launch_stream<false, true>(a, s) : launch_stream<true, true>(a, s);
  return a.full_comp ? launch_stream<false, false>(a, s) : launch_stream<true, false>(a, s);
}

// occupancy of the FP32 kernels on the current device (outside any capture)
cudaError_t prepare_step2d_f32() {
  cudaError_t e = query_resident(k_stream_f32<false, false>, 0);
  if (e == cudaSuccess) e = query_resident(k_stream_f32<true, false>, 1);
  if (e == cudaSuccess) e = query_resident(k_batch_f32<false>, 2);
  if (e == cudaSuccess) e = query_resident(k_stream_f32<false, true>, 3);
  if (e == cudaSuccess) e = query_resident(k_stream_f32<true, true>, 4);
  if (e == cudaSuccess) e = query_resident(k_stream_f32<false, false, true>, 5);
  if (e == cudaSuccess) e = query_resident(k_stream_f32<true, false, true>, 6);
  if (e == cudaSuccess) e = query_resident(k_stream2_f32<false, false>, 7);
  if (e == cudaSuccess) e = query_resident(k_stream2_f32<true, false>, 8);
  if (e == cudaSuccess) e = query_resident(k_stream2_f32<false, true>, 9);
  if (e == cudaSuccess) e = query_resident(k_stream2_f32<true, true>, 10);
  if (e == cudaSuccess) e = query_resident(k_batch_f32<true>, 11);
  return e;
}

cudaError_t launch_batch_f32(const Step2DArgs& a, const BatchArgs& b, bool two, int ctas,
                             cudaStream_t s) {
  const int grid = b.persistent ? ctas : (b.units + kWarps - 1) / kWarps;
  if (grid <= 0) return cudaSuccess;
  if (two)
    k_batch_f32<true><<<grid, 32 * kWarps, 0, s>>>(a, b);
  else
    k_batch_f32<false><<<grid, 32 * kWarps, 0, s>>>(a, b);
  return cudaGetLastError();
}

int batch_resident_ctas(bool two) {
  const int n = g_resident[two ? 11 : 2];
  return n > 0 ? n : 152 * (two ? 6 : 8);
}
int batch_warps_per_cta() { return kWarps; }
int batch_strip_cols(bool two) { return two ? kCols2 : kCols; }

cudaError_t launch_import_f32(const ConvArgs& a, cudaStream_t s) {
  const int rows = (a.y1 > 0 ? a.y1 : a.Ny) - a.y0;
  if (rows <= 0) return cudaSuccess;
  dim3 block(32, 8);
  dim3 grid((a.Nx + 31) / 32, (rows + 7) / 8);
  k_import_records<<<grid, block, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_export_f32(const ConvArgs& a, cudaStream_t s) {
  const int rows = (a.y1 > 0 ? a.y1 : a.Ny) - a.y0;
  if (rows <= 0) return cudaSuccess;
  dim3 block(32, 8);
  dim3 grid((a.Nx + 31) / 32, (rows + 7) / 8);
  k_export_records<<<grid, block, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace pfa

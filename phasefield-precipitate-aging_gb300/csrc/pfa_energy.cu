// pfa_energy.cu -- on-device free energy of a grid (FP64).
//
// summarize_energy (src/alloy625.cpp:865-919) with gibbs (:752-786) and
// maskedgradient (:788-807), which the reference evaluates on the host at
// every output step: per interior node
//   chem = dV (pGam g_gam(x^gam) + pDel g_del(x^del) + pLav g_lav(x^lav)
//              + sum_i omega_i phi_i^2 (1 - phi_i)^2 + 2 Omega phi_del^2 phi_lav^2)
//   grad = dV sum_i kappa_i |grad phi_i|^2  (central differences over the
//          ghost ring at the edges)
// and the total of chem + grad.  The reference's atomic accumulation has no
// fixed order; here each of kSumBlocks blocks sums a fixed set of nodes in a
// fixed order and one block adds the partials, so the total is reproducible.
#include "pfa_device.cuh"
#include "pfa_reduce.h"
#include "pfa_rows.cuh"

namespace pfa {

using namespace dev;

namespace {

// A phase below 2^-600 adds nothing: its square is below the least double.
constexpr int kNoneHi = (1023 - 600) << 20;
// Below 2^-60 (kLinearHi) a phase's p (2^-176) adds nothing to gamma's energy,
// and its coupling to the other phase, 2 Omega / omega 2^-120 of the other's
// well, nothing to that.

// omega phi^2 (1 - phi)^2
__device__ __forceinline__ double well64(double omega, double ph, double sq) {
  const double u = 1.0 - ph;
  return omega * sq * (u * u);
}

// Chemical energy density of a phase PH (1 delta, 2 laves) below 1e-7 beside
// gamma: p g_PH at the composition PH has in pure gamma (p shifts it by less
// than half an ulp), where p counts, and the well
template <int PH>
__device__ __forceinline__ double trace64(double X, double Y, double omega, double ph) {
  double g = well64(omega, ph, ph * ph);
  if (mag_hi(ph) >= kLinearHi) {
    constexpr FictRow r = kFict[PH][0], q = kFict[PH][1];
    const double x = r.scale * fma(r.l[1], X, fma(r.m[1], Y, r.q[3]));
    const double y = q.scale * fma(q.l[1], X, fma(q.m[1], Y, q.q[3]));
    g = fma(p64(ph), g64<PH>(x, y), g);
  }
  return g;
}

// The FP64 pipe bounds the pass (19 cycles per warp instruction and SM), so a
// cell takes the cheapest form of the same value: 9 operations where both
// phases vanish around it (x^gamma is the composition itself), about 20 more
// per phase in its tails (below 1e-7), about 150 next to a precipitate.
// 1024^2: 423 us with the general form and 64-bit divisions everywhere, 61
// with these; 256^2 33 -> 20.
__global__ void __launch_bounds__(kSumThreads, 2) k_energy_partial(EnergyArgs a) {
  const int lane = threadIdx.x & 31;
  const size_t nx = size_t(a.Nx) + 2, plane = nx * (size_t(a.Ny) + 2);
  const double dV = a.dxyz[0] * a.dxyz[1] * (a.is3d ? a.dxyz[2] : 1.0);
  const double w[3] = {1.0 / (2.0 * a.dxyz[0]), 1.0 / (2.0 * a.dxyz[1]),
                       1.0 / (2.0 * a.dxyz[2])};
  double acc = 0.0;
  RowWalk it(a.Nx, a.Ny, a.is3d ? a.Nz : 1, (threadIdx.x >> 5) * kSumBlocks + blockIdx.x,
             kSumBlocks * (kSumThreads / 32));
  for (; it.more(); it.next()) {
    const int x = int(it.c) * 32 + lane;
    if (x >= a.Nx) continue;
    const size_t i = size_t(a.is3d ? it.z + 1 : 0) * plane + (size_t(it.y) + 1) * nx + (x + 1);
    const double X = a.f[0][i], Y = a.f[1][i];
    const double phi[2] = {a.f[2][i], a.f[3][i]};
    double g;
    if (below64(X, Y, phi[0], phi[1], kSolveHi)) {
      g = g64<0>(X, Y);
      if (mag_hi(phi[0]) >= kNoneHi) g += trace64<1>(X, Y, a.omega[0], phi[0]);
      if (mag_hi(phi[1]) >= kNoneHi) g += trace64<2>(X, Y, a.omega[1], phi[1]);
      if (min(mag_hi(phi[0]), mag_hi(phi[1])) >= kLinearHi)
        g += 2.0 * a.Omega * (phi[0] * phi[0]) * (phi[1] * phi[1]);
    } else {
      const double pD = p64(phi[0]), pL = p64(phi[1]);
      const double pG = 1.0 - pD - pL;
      Poly64 m;
      poly64(pD, pG, pL, m);
      g = pG * g64<0>(fict64<0, 0>(X, Y, m), fict64<0, 1>(X, Y, m));
      g += pD * g64<1>(fict64<1, 0>(X, Y, m), fict64<1, 1>(X, Y, m));
      g += pL * g64<2>(fict64<2, 0>(X, Y, m), fict64<2, 1>(X, Y, m));
      const double sq[2] = {phi[0] * phi[0], phi[1] * phi[1]};
#pragma unroll
      for (int k = 0; k < 2; k++) g += well64(a.omega[k], phi[k], sq[k]);
      g += 2.0 * a.Omega * sq[0] * sq[1];
    }
    double ge = 0.0;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const double* p = a.f[2 + k] + i;
      const double e = p[1], we = p[-1], n = p[nx], s = p[-(long long)nx];
      double u = 0.0, d = 0.0;
      if (a.is3d) {
        u = p[plane];
        d = p[-(long long)plane];
      }
      const int most = max(max(max(mag_hi(e), mag_hi(we)), max(mag_hi(n), mag_hi(s))), max(mag_hi(u), mag_hi(d)));
      if (most < kNoneHi) continue;
      const double gx = w[0] * (e - we), gy = w[1] * (n - s);
      double q = gx * gx + gy * gy;
      if (a.is3d) {
        const double gz = w[2] * (u - d);
        q += gz * gz;
      }
      ge += a.kappa[k] * q;
    }
    if (a.chem) a.chem[i] = g * dV;
    if (a.grad) a.grad[i] = ge * dV;
    acc += g + ge;
  }
  __shared__ double sh[kSumThreads];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int s = kSumThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) a.partial[blockIdx.x] = sh[0] * dV;
}

__global__ void __launch_bounds__(32) k_energy_total(const double* partial, int n, double* out) {
  double s = 0.0;
  for (int k = threadIdx.x; k < n; k += 32) s += partial[k];
  for (int w = 16; w > 0; w >>= 1) s += __shfl_down_sync(0xffffffffu, s, w);
  if (threadIdx.x == 0) *out = s;
}

}  // namespace

cudaError_t launch_energy(const EnergyArgs& a, cudaStream_t s) {
  k_energy_partial<<<kSumBlocks, kSumThreads, 0, s>>>(a);
  k_energy_total<<<1, 32, 0, s>>>(a.partial, kSumBlocks, a.out);
  return cudaGetLastError();
}

}  // namespace pfa

// pfa_reduce.cu -- on-device FP64 field summary of libpfa_gb300.
//
// summarize_fields (src/alloy625.cpp:811-863) averages x_Cr, x_Nb and the
// gamma / delta / laves phase fractions over the grid nodes on the host with
// an OpenMP critical section.  Here the sums run on the device, exactly in
// integers or in FP64 with Kahan compensation per thread, in a fixed two-level
// order (kSumBlocks partial sums, then one block), so repeated calls give
// identical bits.
#include "pfa_device.cuh"
#include "pfa_reduce.h"
#include "pfa_rows.cuh"

namespace pfa {

using namespace dev;

namespace {

// Kahan sum
struct Sum64 {
  double s, c;
  __device__ void add(double v) {
    const double y = v - c;
    const double t = s + y;
    c = (t - s) - y;
    s = t;
  }
};

// 2^64 times a sum of values in [2^-11, 1), exact
struct SumFix {
  unsigned long long lo;
  unsigned hi;
  __device__ void add(uint64_t v) {
    lo += v;
    hi += lo < v;
  }
};

// p of a phase below 2^-360 is below the least double
constexpr int kNoneHi = (1023 - 360) << 20;

// The FP64 pipe bounds the pass (19 cycles per warp instruction and SM; a
// compensated sum is four): compositions in the usual range are summed exactly
// in integers, phases only where they are not zero, and an FP32 record's
// fields take no FP64 conversion.  1024^2: 112 us with five compensated sums
// in every cell and 64-bit divisions, 21 with these.
template <bool F32>
__global__ void __launch_bounds__(kSumThreads, 2) k_sum_partial(SumArgs a) {
  const int lane = threadIdx.x & 31;
  Sum64 acc[5] = {};
  SumFix fx[2] = {};
  unsigned gamma = 0;  // cells of pure gamma
  RowWalk it(a.Nx, a.Ny, a.Nz, (threadIdx.x >> 5) * kSumBlocks + blockIdx.x,
             kSumBlocks * (kSumThreads / 32));
  for (; it.more(); it.next()) {
    const int x = int(it.c) * 32 + lane;
    if (x >= a.Nx) continue;
    const size_t cell = a.compact ? (size_t(it.z) * a.Ny + it.y) * a.pitch + x
                                  : (size_t(a.is3d ? it.z + 1 : 0) * (a.Ny + 2) + (it.y + 1)) * a.pitch + (x + 1);
    double v[4];
    if constexpr (F32) {
      const float4 r = static_cast<const float4*>(a.f[0])[cell];
      if (a.pack) {
        merge_record(r, static_cast<const uint2*>(a.comp)[cell], v);
      } else {
        const float4 c = static_cast<const float4*>(a.comp)[cell];
        v[0] = double(r.x) - double(c.x);
        v[1] = double(r.y) - double(c.y);
        v[2] = double(r.z) - double(c.z);
        v[3] = double(r.w) - double(c.w);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) v[k] = static_cast<const double*>(a.f[k])[cell];
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
      if (in_unit(v[k]))
        fx[k].add(fix64(v[k]));
      else
        acc[k].add(v[k]);
    }
    if (max(mag_hi(v[2]), mag_hi(v[3])) < kNoneHi) {
      gamma++;
    } else {
      const double pd = p64(v[2]), pl = p64(v[3]);
      acc[2].add((1.0 - pd) - pl);
      acc[3].add(pd);
      acc[4].add(pl);
    }
  }
  // the integer sums of the block, then their values in thread k of warp 0
  __shared__ uint64_t s_lo[2][kSumThreads / 32];
  __shared__ unsigned s_hi[2][kSumThreads / 32], s_gamma[kSumThreads / 32];
  __shared__ double sh[5][kSumThreads];
#pragma unroll
  for (int k = 0; k < 2; k++)
    for (int w = 16; w > 0; w >>= 1) {
      const unsigned hi = __shfl_down_sync(0xffffffffu, fx[k].hi, w);
      fx[k].add(__shfl_down_sync(0xffffffffu, fx[k].lo, w));
      fx[k].hi += hi;
    }
  gamma = __reduce_add_sync(0xffffffffu, gamma);
  if (lane == 0) {
    const int w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      s_lo[k][w] = fx[k].lo;
      s_hi[k][w] = fx[k].hi;
    }
    s_gamma[w] = gamma;
  }
  bool any = false;  // the FP64 sums of the block, where there are any
#pragma unroll
  for (int k = 0; k < 5; k++) any = any || acc[k].s != 0.0;
  any = __syncthreads_or(any);
  if (any) {
#pragma unroll
    for (int k = 0; k < 5; k++) sh[k][threadIdx.x] = acc[k].s - acc[k].c;
    __syncthreads();
    for (int w = kSumThreads / 2; w > 0; w >>= 1) {
      if (threadIdx.x < w)
        for (int k = 0; k < 5; k++) sh[k][threadIdx.x] += sh[k][threadIdx.x + w];
      __syncthreads();
    }
  }
  if (threadIdx.x < 5) {
    const int k = threadIdx.x;
    Sum64 t = {any ? sh[k][0] : 0.0, 0.0};
    if (k < 2) {
      SumFix f = {0, 0};
      for (int w = 0; w < kSumThreads / 32; w++) {
        f.add(s_lo[k][w]);
        f.hi += s_hi[k][w];
      }
      t.add(double(f.hi));
      t.add(double(unsigned(f.lo >> 32)) * 0x1p-32);
      t.add(double(unsigned(f.lo)) * 0x1p-64);
    } else if (k == 2) {
      unsigned n = 0;  // (a block's cells: below 2^32)
      for (int w = 0; w < kSumThreads / 32; w++) n += s_gamma[w];
      t.add(double(n));
    }
    a.partial[blockIdx.x * 5 + k] = t.s - t.c;
  }
}

// One warp per sum: each lane adds its share of the partials (compensated),
// then the lanes add up pairwise.  A single thread's chain over all of them
// took 32 us (an FP64 operation's latency is 64 cycles).
__global__ void __launch_bounds__(32 * 5) k_sum_final(const double* partial, int nblocks, double inv_n,
                                                      double* out) {
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double s = 0.0, c = 0.0;
  for (int b = lane; b < nblocks; b += 32) {
    const double y = partial[b * 5 + k] - c;
    const double t = s + y;
    c = (t - s) - y;
    s = t;
  }
  s -= c;
  for (int w = 16; w > 0; w >>= 1) s += __shfl_down_sync(0xffffffffu, s, w);
  if (lane == 0) out[k] = s * inv_n;
}

}  // namespace

cudaError_t launch_summarize(const SumArgs& a, cudaStream_t s) {
  if (a.is_f32)
    k_sum_partial<true><<<kSumBlocks, kSumThreads, 0, s>>>(a);
  else
    k_sum_partial<false><<<kSumBlocks, kSumThreads, 0, s>>>(a);
  const double n = double(a.Nx) * double(a.Ny) * double(a.Nz);
  k_sum_final<<<1, 32 * 5, 0, s>>>(a.partial, kSumBlocks, 1.0 / n, a.out);
  return cudaGetLastError();
}

}  // namespace pfa

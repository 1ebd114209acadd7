// pfa_fixed64.cuh -- parts of the FP64 steps in 64-bit fixed point.
//
// An FP64 operation takes an SM 19 cycles per warp, the high half of a 64 x 64
// bit product about three.  So for compositions in [2^-11, 1) and phase fields
// in [0, 1] these parts of a cell are formed in fixed point (every other cell
// takes the FP64 expressions):
//   solve_fixed: x^gamma of a cell with precipitate, 30 to 56 FP64 operations.
//     Error over the simplex (against 113 bits, units of 2^-53): at most 26,
//     0.08 on average; the FP64 forms 9800 and 18 (the cancellation inside
//     delta).  us a step: 256^2 with 8 particles 7.5 -> 6.6, 3D 64^3 56 -> 40.
//   mobilities: the weighted mobilities of the variable-mobility step, 59
//     operations with their three exponentials.  Error at most 1.6 (FP64: up
//     to 30 and, near x_Ni = 0, 4e4); 512^2 73.9 -> 38.9 us a step.
//   diffusivities: the matrix of that step, 26 operations.  Error in the usual
//     range of compositions, units of 2^-60: at most 1.6, 0.07 on average (FP64:
//     22 and 1.1); with the fluxes 512^2 38.9 -> 20.9 us a step.
// Compiles as host code too.
#pragma once

#include <cstdint>

#include "pfa_internal.h"
#include "pfa_model.h"

namespace pfa {
namespace dev {

#ifdef __CUDACC__
#define PFA_FIX_FN static __device__ __forceinline__
#else
#define PFA_FIX_FN static inline
#endif

PFA_FIX_FN uint64_t mul_hi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return uint64_t((unsigned __int128)a * b >> 64);
#endif
}

PFA_FIX_FN uint32_t mul_hi32(uint32_t a, uint32_t b) { return uint32_t(uint64_t(a) * b >> 32); }

// signed times unsigned 2^64
PFA_FIX_FN int64_t mul_hi_su(int64_t t, uint64_t u) { return int64_t(mul_hi(uint64_t(t), u) - (t < 0 ? u : 0)); }

PFA_FIX_FN int lead_zeros(uint64_t v) {  // v > 0
#ifdef __CUDA_ARCH__
  return __clzll((long long)v);
#else
  return __builtin_clzll(v);
#endif
}

// 2^z by table and polynomial (P. T. P. Tang, "Table-driven implementation of
// the exponential function in IEEE floating-point arithmetic", ACM TOMS 15,
// 1989): z = k + j / 128 + g / 128, 2^(j/128) from a table of 128 entries, and
// 2^(g/128) - 1 = sum_n (ln 2 / 128)^n g^n / n! to the sixth term (the seventh
// is below 2^-65).
// round(2^63 2^(j/128))
#ifdef __CUDACC__
static __device__
#else
static
#endif
const uint64_t kExp2[128] = {
    0x8000000000000000ull, 0x80b1ed4fd999ab6cull, 0x8164d1f3bc030773ull, 0x8218af4373fc25ecull,
    0x82cd8698ac2ba1d7ull, 0x8383594eefb6ee37ull, 0x843a28c3acde4046ull, 0x84f1f656379c1a29ull,
    0x85aac367cc487b15ull, 0x8664915b923fba04ull, 0x871f61969e8d1010ull, 0x87db357ff698d792ull,
    0x88980e8092da8527ull, 0x8955ee03618e5fddull, 0x8a14d575496efd9aull, 0x8ad4c6452c728924ull,
    0x8b95c1e3ea8bd6e7ull, 0x8c57c9c4646f4ddeull, 0x8d1adf5b7e5ba9e6ull, 0x8ddf042022e69cd6ull,
    0x8ea4398b45cd53c0ull, 0x8f6a8117e6c8e5c4ull, 0x9031dc431466b1dcull, 0x90fa4c8beee4b12bull,
    0x91c3d373ab11c336ull, 0x928e727d9531f9acull, 0x935a2b2f13e6e92cull, 0x9426ff0fab1c04b6ull,
    0x94f4efa8fef70961ull, 0x95c3fe86d6cc7fefull, 0x96942d3720185a00ull, 0x97657d49f17ab08eull,
    0x9837f0518db8a96full, 0x990b87e266c189aaull, 0x99e0459320b7fa65ull, 0x9ab62afc94ff864aull,
    0x9b8d39b9d54e5539ull, 0x9c6573682ec32c2dull, 0x9d3ed9a72cffb751ull, 0x9e196e189d472420ull,
    0x9ef5326091a111aeull, 0x9fd228256400dd06ull, 0xa0b0510fb9714fc2ull, 0xa18faeca8544b6e4ull,
    0xa27043030c496819ull, 0xa3520f68e802bb93ull, 0xa43515ae09e6809eull, 0xa5195786be9ef339ull,
    0xa5fed6a9b15138eaull, 0xa6e594cfeee86b1eull, 0xa7cd93b4e965356aull, 0xa8b6d5167b320e09ull,
    0xa9a15ab4ea7c0ef8ull, 0xaa8d2652ec907629ull, 0xab7a39b5a93ed337ull, 0xac6896a4be3fe929ull,
    0xad583eea42a14ac6ull, 0xae493452ca35b80eull, 0xaf3b78ad690a4375ull, 0xb02f0dcbb6e04584ull,
    0xb123f581d2ac2590ull, 0xb21a31a66618fe3bull, 0xb311c412a9112489ull, 0xb40aaea2654b9841ull,
    0xb504f333f9de6484ull, 0xb60093a85ed5f76cull, 0xb6fd91e328d17791ull, 0xb7fbefca8ca41e7cull,
    0xb8fbaf4762fb9ee9ull, 0xb9fcd2452c0b9debull, 0xbaff5ab2133e45fbull, 0xbc034a7ef2e9fb0dull,
    0xbd08a39f580c36bfull, 0xbe0f6809860993e2ull, 0xbf1799b67a731083ull, 0xc0213aa1f0d08db0ull,
    0xc12c4cca66709456ull, 0xc238d2311e3d6673ull, 0xc346ccda24976407ull, 0xc4563ecc5334cb33ull,
    0xc5672a115506daddull, 0xc67990b5aa245f79ull, 0xc78d74c8abb9b15dull, 0xc8a2d85c8ffe2c45ull,
    0xc9b9bd866e2f27a3ull, 0xcad2265e4290774eull, 0xcbec14fef2727c5dull, 0xcd078b86503dcdd2ull,
    0xce248c151f8480e4ull, 0xcf4318cf191918c1ull, 0xd06333daef2b2595ull, 0xd184df6251699ac6ull,
    0xd2a81d91f12ae45aull, 0xd3ccf099859ac379ull, 0xd4f35aabcfedfa1full, 0xd61b5dfe9f9bce07ull,
    0xd744fccad69d6af4ull, 0xd870394c6db32c84ull, 0xd99d15c278afd7b6ull, 0xdacb946f2ac9cc72ull,
    0xdbfbb797daf23755ull, 0xdd2d818508324c20ull, 0xde60f4825e0e9124ull, 0xdf9612deb8f04420ull,
    0xe0ccdeec2a94e111ull, 0xe2055afffe83d369ull, 0xe33f8972be8a5a51ull, 0xe47b6ca0373da88dull,
    0xe5b906e77c8348a8ull, 0xe6f85aaaee1fce22ull, 0xe8396a503c4bdc68ull, 0xe97c38406c4f8c57ull,
    0xeac0c6e7dd24392full, 0xec0718b64c1cbddcull, 0xed4f301ed9942b84ull, 0xee990f980da3025bull,
    0xefe4b99bdcdaf5cbull, 0xf13230a7ad094509ull, 0xf281773c59ffb13aull, 0xf3d28fde3a641a5bull,
    0xf5257d152486cc2cull, 0xf67a416c733f846eull, 0xf7d0df730ad13bb9ull, 0xf92959bb5dd4ba74ull,
    0xfa83b2db722a033aull, 0xfbdfed6ce5f09c49ull, 0xfd3e0c0cf486c175ull, 0xfe9e115c7b8f884cull,
};

// 2^63 2^(f 2^-64), rounded down; f: the fraction of z
PFA_FIX_FN uint64_t exp2_mantissa(uint64_t f) {
#ifdef __CUDA_ARCH__
  const uint64_t t = __ldg(reinterpret_cast<const unsigned long long*>(kExp2) + (f >> 57));
#else
  const uint64_t t = kExp2[f >> 57];
#endif
  const uint64_t h = f << 7;  // g 2^64
  const uint32_t hh = uint32_t(h >> 32);
  // Horner, in units of 2^-70; the high orders need few bits
  const uint32_t s = 0x2bb0ffdu + mul_hi32(0xa185u, hh);
  const uint64_t s4 = 0x9d955b7ddull + mul_hi32(s, hh);           // 36 bits
  const uint64_t s3 = 0x1c6b08d704a1ull + (uint64_t(uint32_t(s4 >> 4)) * hh >> 28);
  const uint64_t s2 = 0x3d7f7bff058b1dull + mul_hi(s3, h);
  const uint64_t s1 = 0x58b90bfbe8e7bcd6ull + mul_hi(s2, h);
  return t + (mul_hi(t, mul_hi(s1, h)) >> 6);
}

// the FP64 value of m 2^(e - 63), m >= 2^62 and the result normal
PFA_FIX_FN uint64_t pack64(uint64_t m, int e) {
  const int up = m >> 63 ? 0 : 1;
  m <<= up;
  return (uint64_t(1022 + e - up) << 52) + (m >> 11) + ((m >> 10) & 1);
}

// Weighted mobilities (e_Nb, e_Cr, e_Ni x_Ni of dmatrix64, times the
// prefactors vm_pre): m 2^(e - 63), 2^63 <= m.  x, y: the compositions times
// 2^64, 2^53 or more, x + y < 2^64.
struct Mobility {
  uint64_t m;
  int e;
};
PFA_FIX_FN void mobilities(const Coef64& K, uint64_t x, uint64_t y, Mobility v[3]) {
  const uint64_t n = 0 - (x + y);  // x_Ni
  auto normal = [](uint64_t m, int e) {  // m 2^(e - 62), 2^62 <= m
    const int up = m >> 63 ? 0 : 1;
    return Mobility{m << up, e + 1 - up};
  };
  auto weighted = [&](int64_t z, int q, int k) {  // vm_pre 2^(z 2^-q)
    return normal(mul_hi(exp2_mantissa(uint64_t(z) << (64 - q)), K.vm_m[k]), int(z >> q) + K.vm_e[k]);
  };
  // exponents times log2(e): 2^-57, 2^-59, 2^-54
  const int64_t zn = mul_hi_su(0x29a8bb8820a29949ll - int64_t(mul_hi(0x64f0372c225e9378ull, n)), y);
  const int64_t zc = mul_hi_su(0x26b6712afedfd131ll - int64_t(mul_hi(0x529296d39d336238ull, n)), x);
  const int64_t zi = (mul_hi_su(0x2e3564d412fda0f2ll - int64_t(mul_hi(0x625bca3fd59b5547ull, n)), x) >> 5) -
                     int64_t(mul_hi(0x004bdd4343eff6b2ull + mul_hi(0x9fa5039d40b0facaull, n), y));
  v[0] = weighted(zn, 57, 0);
  v[1] = weighted(zc, 59, 1);
  const Mobility i = weighted(zi, 54, 2);
  const int lead = lead_zeros(n);
  v[2] = normal(mul_hi(i.m, n << lead), i.e - lead - 1);
}

// FP64 bits of a mobility
PFA_FIX_FN uint64_t mobility_bits(const Mobility& v) { return pack64(v.m, v.e); }

// ---- diffusivities ----
PFA_FIX_FN constexpr uint64_t coef64(double c) { return uint64_t((c < 0 ? -c : c) * 0x1p64); }

// D_CrCr, D_CrNb, D_NbCr, D_NbNb of dmatrix64_scaled times 2^67 (false: one of
// them is 2^-5 or more).  The curvature weights are scaled by 2^-21 (to below
// 1), the mobilities by the power of two that brings the largest to [1/16,
// 1/8), so that no sum exceeds 1/2.
PFA_FIX_FN bool diffusivities(const Coef64& K, uint64_t x, uint64_t y, long long d[4]) {
  Mobility v[3];
  mobilities(K, x, y, v);
  const int top = v[0].e > v[1].e ? (v[0].e > v[2].e ? v[0].e : v[2].e) : (v[1].e > v[2].e ? v[1].e : v[2].e);
  uint64_t e[3];  // 2^64 2^-(top + 4) times the mobilities
  for (int k = 0; k < 3; k++) {
    const int down = 3 + top - v[k].e;
    e[k] = down < 64 ? v[k].m >> down : 0;
  }
  constexpr double q = 0x1p-21;
  auto column = [&](uint64_t hx, uint64_t hy, uint64_t hn, uint64_t hc, long long& dc, long long& dn) {
    const int64_t s = -int64_t((mul_hi(hx, x) + mul_hi(hy, y)) >> 1);  // 2^63, as all below
    const int64_t A = mul_hi_su(s + int64_t(hn >> 1), e[0]), B = mul_hi_su(s + int64_t(hc >> 1), e[1]);
    const int64_t W = mul_hi_su(B, x) + mul_hi_su(A, y) + mul_hi_su(s, e[2]);
    dc = mul_hi_su((B - W) << 1, x);
    dn = mul_hi_su((A - W) << 1, y);
  };
  column(coef64(kHCrCr * q), coef64(kHCrNb * q), coef64(kHCrNbAddA * q), coef64(kHCrCrAdd * q), d[0], d[2]);
  column(coef64(kHCrNb * q), coef64(kHNbNb * q), coef64(kHNbNbAdd * q), coef64(kHCrNbAddB * q), d[1], d[3]);
  const int up = top + 4 + 21 + 3;  // from 2^64 2^-(top + 25) to 2^67
  if (up < -60 || up > 60) return false;
  const uint64_t bound = up > 0 ? 1ull << 62 >> up : 1ull << 62;
  bool ok = true;
  for (int k = 0; k < 4; k++) {
    ok = ok && uint64_t(d[k]) + bound < 2 * bound;
    d[k] = up > 0 ? (long long)(uint64_t(d[k]) << up) : d[k] >> -up;
  }
  return ok;
}

// t = n - s + e - w, the fluxes through a cell's faces (units of 2^-65: each
// below 1/4); false where a sum leaves 64 bits.  Diffusivities up to 2^-5 let
// four faces reach 1/2 (found: 0.264 at 3.6 times the usual time step).  The
// test costs the step 0.6 % (512^2); fluxes in units of 2^-63 would need none,
// at two bits less.
PFA_FIX_FN bool face_sum(int64_t n, int64_t s, int64_t e, int64_t w, int64_t& t) {
  const uint64_t a = uint64_t(n) - uint64_t(s), b = uint64_t(e) - uint64_t(w), c = a + b;
  const uint64_t un = uint64_t(n), ue = uint64_t(e);
  t = int64_t(c);
  return int64_t(((un ^ uint64_t(s)) & (un ^ a)) | ((ue ^ uint64_t(w)) & (ue ^ b)) | ((a ^ c) & (b ^ c))) >= 0;
}

// ---- x^gamma ----
// All numbers are unsigned multiples of 2^-63 (1 is 2^63); signs are those of
// the coefficients (kFict, kDen), known at compile time.
constexpr uint64_t kOne63 = 1ull << 63;

PFA_FIX_FN uint64_t mul63(uint64_t a, uint64_t b) { return mul_hi(a, b) << 1; }
PFA_FIX_FN uint64_t by(uint64_t coef, uint64_t v) { return mul_hi(coef, v); }

// p(phi) = phi^3 (10 - 15 phi + 6 phi^2), the bracket in units of 2^-60
PFA_FIX_FN uint64_t p63(uint64_t f) {
  const uint64_t f2 = mul63(f, f), f3 = mul63(f2, f);
  const uint64_t q = (10ull << 60) + 6 * (f2 >> 3) - 15 * (f >> 3);
  return (mul_hi(f3, q) << 4) | (f3 * q >> 60);
}

// 2^126 / d, d >= 2^63: an FP32 reciprocal and two Newton steps
PFA_FIX_FN uint64_t reciprocal(uint64_t d) {
  union {
    uint32_t i;
    float f;
  } v;
  v.i = 0x3f800000u | (uint32_t(d >> 40) & 0x7fffffu);
  uint64_t y = uint64_t(uint32_t((1.0f / v.f) * 0x1p31f)) << 32;
  for (int k = 0; k < 2; k++) {
    const int64_t e = (1ll << 62) - int64_t(mul_hi(d, y));  // |e| < 2^41
    y += uint64_t(mul_hi_su(e << 20, y) >> 18);
  }
  return y;
}

// x^gamma in units of 2^-60 from the nested forms of gamma64 (pfa_device.cuh);
// KIND: 1 delta only, 2 laves only, 3 both (the same bits as 1 and 2 where the
// other fraction is zero).  x, y, fd, fl: compositions and phases times 2^63.
// false: fractions that add up to more than 1 or |x^gamma| of 2 and more.
template <int KIND>
PFA_FIX_FN bool solve_fixed(uint64_t x, uint64_t y, uint64_t fd, uint64_t fl, int64_t& h1, int64_t& h2) {
  constexpr bool D = KIND & 1, L = KIND & 2;
  const uint64_t pD = D ? p63(fd) : 0, pL = L ? p63(fl) : 0;
  if (pD > kOne63 || pL > kOne63 - pD) return false;  // (their sum wraps where both are 1)
  const uint64_t pG = kOne63 - pD - pL;
  constexpr FictRow a = kFict[0][0], b = kFict[0][1];
  static_assert(a.l[0] > 0 && a.l[2] > 0 && a.m[0] < 0 && a.m[2] < 0 && a.q[0] > 0 && a.q[1] > 0 &&
                    a.q[2] > 0 && a.q[4] < 0 && a.q[5] < 0,
                "the signs of x^gamma_Cr's terms");
  static_assert(b.l[0] > 0 && b.l[2] > 0 && b.m[0] < 0 && b.m[2] < 0 && b.q[0] > 0 && b.q[1] > 0 &&
                    b.q[2] > 0 && b.q[4] > 0 && b.q[5] > 0,
                "the signs of x^gamma_Nb's terms");
  uint64_t den = mul63(pG, pG);
  uint64_t l1 = pG, m1 = 0, l2 = 0, m2 = pG;
  int64_t n1 = 0, n2 = 0;
  if constexpr (D) {
    uint64_t d = by(coef64(kDen[0]), pD) + by(coef64(kDen[1]), pG);
    uint64_t q1 = by(coef64(a.q[0]), pD) + by(coef64(a.q[1]), pG);
    uint64_t q2 = by(coef64(b.q[0]), pD) + by(coef64(b.q[1]), pG);
    if constexpr (L) {
      d += by(coef64(kDen[2]), pL);
      q1 += by(coef64(a.q[2]), pL);
      q2 += by(coef64(b.q[2]), pL);
    }
    den += mul63(pD, d);
    n1 += int64_t(mul63(pD, q1));
    n2 -= int64_t(mul63(pD, q2));
    l1 += by(coef64(a.l[0]), pD);
    m1 += by(coef64(a.m[0]), pD);
    l2 += by(coef64(b.l[0]), pD);
    m2 += by(coef64(b.m[0]), pD);
  }
  if constexpr (L) {
    den += mul63(pL, by(coef64(kDen[4]), pG) + by(coef64(kDen[5]), pL));
    n1 -= int64_t(mul63(pL, by(coef64(a.q[4]), pG) + by(coef64(a.q[5]), pL)));
    n2 -= int64_t(mul63(pL, by(coef64(b.q[4]), pG) + by(coef64(b.q[5]), pL)));
    l1 += by(coef64(a.l[2]), pL);
    m1 += by(coef64(a.m[2]), pL);
    l2 += by(coef64(b.l[2]), pL);
    m2 += by(coef64(b.m[2]), pL);
  }
  n1 += int64_t(mul63(x, l1)) - int64_t(mul63(y, m1));
  n2 += int64_t(mul63(y, m2)) - int64_t(mul63(x, l2));
  const uint64_t most = uint64_t(n1 < 0 ? -n1 : n1) | uint64_t(n2 < 0 ? -n2 : n2);
  const int lead = lead_zeros(den);  // den is at least kDen[0]: below 11
  if (most >> 1 >= kOne63 >> lead) return false;
  const uint64_t r = reciprocal(den << lead);
  auto over = [&](int64_t n) {  // n / den 2^60
    const int64_t t = lead >= 2 ? int64_t(uint64_t(n) << (lead - 2)) : n >> (2 - lead);
    return mul_hi_su(t, r);
  };
  h1 = over(n1);
  h2 = over(n2);
  return true;
}

// The x^gamma, in units of 2^-60, whose weighted neighbour sums stay in range:
// low <= h < most.  A cell without a solve has x^gamma in [0, 1).
struct Range60 {
  int64_t low, most;
};
// The sums of 5 points (2D) and 7 (3D), weights 1 and -4 or -6, in units of
// 2^-58: a 64-bit sum holds +-32, these reach 4 x 2 + 4 x 2 = 16 and 24.
constexpr Range60 kRangeFaces = {-(1ll << 61), 1ll << 61};
// 9 points, weights 4, 1 and -20: 20 (1 + 9/16) = 31.25.
constexpr Range60 kRangeCorners = {-(9ll << 56), 1ll << 60};
// A face's difference for the fluxes of the variable mobility, in units of
// 2^-62: +-2 (the 2: h is rounded to units of 2^-58).
constexpr Range60 kRangeFlux = {-(1ll << 60), (1ll << 60) - 2};
constexpr Range60 kRangeNone = {0, 0};  // FP64 values are wanted

// FP64 bits of v 2^-q
PFA_FIX_FN uint64_t pack_signed(int64_t v, int q) {
  if (v == 0) return 0;
  const uint64_t m = v < 0 ? 0 - uint64_t(v) : uint64_t(v);
  const int lead = lead_zeros(m);
  return pack64(m << lead, 63 - lead - q) | (v < 0 ? 1ull << 63 : 0);
}

}  // namespace dev
}  // namespace pfa

// pfa_exp64.cuh -- the mobility exponentials in 64-bit integers.
//
// An FP64 operation takes an SM 19 cycles per warp, a 64 x 64 bit product
// about three, and the variable-mobility step's three exponentials per cell
// were half of its FP64 operations (48 of 83 per staged cell, with their
// arguments 59).  For compositions in [2^-11, 1) that add up to less than 1,
// everything up to the weighted mobilities e_Nb, e_Cr, e_Ni x_Ni is formed in
// fixed point and only the three results are rounded to FP64.
//
// 2^z by table and polynomial (P. T. P. Tang, "Table-driven implementation of
// the exponential function in IEEE floating-point arithmetic", ACM TOMS 15,
// 1989): z = k + j / 128 + g / 128, 2^(j/128) from a table of 128 entries, and
// 2^(g/128) - 1 = sum_n (ln 2 / 128)^n g^n / n! to the sixth term (the seventh
// is below 2^-65).
#pragma once

#include <cstdint>

#include "pfa_internal.h"

namespace pfa {
namespace dev {

#ifdef __CUDACC__
#define PFA_EXP_FN static __host__ __device__ __forceinline__
#else
#define PFA_EXP_FN static inline
#endif

PFA_EXP_FN uint64_t mul_hi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return uint64_t((unsigned __int128)a * b >> 64);
#endif
}

PFA_EXP_FN uint32_t mul_hi32(uint32_t a, uint32_t b) { return uint32_t(uint64_t(a) * b >> 32); }

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
PFA_EXP_FN uint64_t exp2_mantissa(uint64_t f) {
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
PFA_EXP_FN uint64_t pack64(uint64_t m, int e) {
  const int up = m >> 63 ? 0 : 1;
  m <<= up;
  return (uint64_t(1022 + e - up) << 52) + (m >> 11) + ((m >> 10) & 1);
}

// Weighted mobilities (e_Nb, e_Cr, e_Ni x_Ni of dmatrix64, times the
// prefactors pm 2^(pe - 63)) as FP64 bits.  x, y: the compositions times 2^64,
// 2^53 or more, x + y < 2^64.
PFA_EXP_FN void mobilities(const Coef64& K, uint64_t x, uint64_t y, uint64_t e[3]) {
  const uint64_t n = 0 - (x + y);  // x_Ni
  // signed * unsigned 2^64
  auto times = [](int64_t t, uint64_t u) { return int64_t(mul_hi(uint64_t(t), u) - (t < 0 ? u : 0)); };
  auto weighted = [&](int64_t z, int q, int k, uint64_t w) {  // pre 2^(z 2^-q) w
    const uint64_t m = mul_hi(exp2_mantissa(uint64_t(z) << (64 - q)), K.vm_m[k]);  // >= 2^62
    int lead = 0;
    if (w) {
#ifdef __CUDA_ARCH__
      lead = __clzll(w);
#else
      lead = __builtin_clzll(w);
#endif
    }
    const int ex = int(z >> q) + K.vm_e[k] + 1;
    if (!w) return pack64(m, ex);
    const uint64_t p = mul_hi(m << (m >> 63 ? 0 : 1), w << lead);
    return pack64(p, ex - (m >> 63 ? 0 : 1) - lead);
  };
  // exponents times log2(e): 2^-57, 2^-59, 2^-54
  const int64_t zn = times(0x29a8bb8820a29949ll - int64_t(mul_hi(0x64f0372c225e9378ull, n)), y);
  const int64_t zc = times(0x26b6712afedfd131ll - int64_t(mul_hi(0x529296d39d336238ull, n)), x);
  const int64_t zi = (times(0x2e3564d412fda0f2ll - int64_t(mul_hi(0x625bca3fd59b5547ull, n)), x) >> 5) -
                     int64_t(mul_hi(0x004bdd4343eff6b2ull + mul_hi(0x9fa5039d40b0facaull, n), y));
  e[0] = weighted(zn, 57, 0, 0);
  e[1] = weighted(zc, 59, 1, 0);
  e[2] = weighted(zi, 54, 2, n);
}

}  // namespace dev
}  // namespace pfa

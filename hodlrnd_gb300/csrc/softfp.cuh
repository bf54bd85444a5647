// Correctly rounded FP64 square roots and quotients on the integer pipe.
//
// GB300's FP64 pipe takes 20 cycles of an SM for one warp instruction, and a
// division or a square root takes 7.5 of them, while an integer instruction takes
// about 0.45: a square root and the division by it are 110 integer instructions
// (50 cycles) instead of 15 FP64 operations (300).  Results are IEEE
// round-to-nearest-even, bit for bit: the exact integer floor of the root or
// quotient with one extra bit (estimated by a third-order Newton step in 64-bit
// fixed point from a single-precision seed, then corrected by the exact
// remainder), rounded once.  Operands or results that are subnormal, infinite or
// NaN take the FP64 instructions.  Host code (the test against the host's FP64)
// uses the same integers.  (Products were tried too: 35 integer instructions in
// place of a 20-cycle multiplication did not pay, in any share of a residual's
// products: 425 -> 434 to 565 ms for a 3D N = 100003 build.)
#pragma once

#include <stdint.h>
#include <string.h>

#include <cmath>

#ifdef __CUDACC__
#define HODLR_HD __host__ __device__ __forceinline__
#define HODLR_HD_SLOW inline __host__ __device__ __noinline__  // rare: kept out of the callers' code
#else
#define HODLR_HD inline
#define HODLR_HD_SLOW inline
#endif

namespace hodlr {

HODLR_HD_SLOW double plain_sqrt(double x) {
#ifdef __CUDA_ARCH__
  return __dsqrt_rn(x);
#else
  return std::sqrt(x);
#endif
}
HODLR_HD_SLOW double plain_div(double c, double x) {
#ifdef __CUDA_ARCH__
  return __ddiv_rn(c, x);
#else
  return c / x;
#endif
}

HODLR_HD uint64_t soft_bits(double v) {
#ifdef __CUDA_ARCH__
  return static_cast<uint64_t>(__double_as_longlong(v));
#else
  uint64_t b;
  memcpy(&b, &v, 8);
  return b;
#endif
}
HODLR_HD double soft_double(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(static_cast<long long>(b));
#else
  double v;
  memcpy(&v, &b, 8);
  return v;
#endif
}
HODLR_HD uint64_t mulhi64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return uint64_t((static_cast<unsigned __int128>(a) * b) >> 64);
#endif
}
HODLR_HD uint32_t mulhi32(uint32_t a, uint32_t b) { return uint32_t((uint64_t(a) * b) >> 32); }

// Single-precision seeds 1 / sqrt(f), f in [1, 4), and 1 / f, f in [1, 2), as
// r 2^32 in (2^31, 2^32); anything within 2^-21 relative will do (CUDA's own are
// within 2^-22).
#ifndef HODLR_SOFT_SEED_NOISE
#define HODLR_SOFT_SEED_NOISE(r) (r)
#endif
HODLR_HD uint32_t soft_seed(float r) {
  uint32_t b;
#ifdef __CUDA_ARCH__
  b = __float_as_uint(r);
#else
  r = HODLR_SOFT_SEED_NOISE(r);
  memcpy(&b, &r, 4);
#endif
  return r >= 1.0f ? 0xffffffffu : r < 0.5f ? 0x80000000u : ((b & 0x7fffffu) | 0x800000u) << 8;
}
HODLR_HD float soft_float(uint32_t b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}

// A number taken apart: significand (53 bits), exponent
// field, sign; m = 0 for a zero; e = kSoftOdd for a subnormal, infinity or NaN.
struct SoftD {
  uint64_t m;
  int e;
  uint32_t sign;
};
constexpr int kSoftOdd = 1 << 20;
HODLR_HD SoftD soft_unpack(double v) {
  const uint64_t b = soft_bits(v);
  const uint32_t hi = uint32_t(b >> 32);
  SoftD s;
  s.e = int((hi >> 20) & 0x7ffu);
  s.sign = hi & 0x80000000u;
  s.m = (b & 0xfffffffffffffull) | 0x10000000000000ull;
  if (s.e == 0) {
    const bool zero = (b << 1) == 0;
    s.m = zero ? 0 : s.m;
    s.e = zero ? 0 : kSoftOdd;
  }
  if (s.e == 0x7ff) s.e = kSoftOdd;
  return s;
}

// floor of mc / s at 54 bits (53 for the quotient, one to round), from an
// approximate quotient `q` of that scale at most 3 off; both significands of
// 53 bits.  k = 53 when mc >= s, else 54.
HODLR_HD uint64_t soft_quotient(uint64_t mc, uint64_t s, uint64_t q, int k) {
  const int64_t r = int64_t((mc << k) - q * s);  // the remainder, modulo 2^64: a few s at most
  const int64_t d = int64_t(s);
  q += (r >= d ? 1 : 0) + (r >= 2 * d ? 1 : 0) + (r >= 3 * d ? 1 : 0);
  q -= (r < 0 ? 1 : 0) + (r < -d ? 1 : 0) + (r < -2 * d ? 1 : 0);
  return q;
}

// y (1 + c h + term2): the Newton step shared by root and quotient.  y0 =
// y 2^31 or 2^32, h in units of 2^-62.
HODLR_HD int64_t soft_y_h(uint32_t y0, int64_t h) {  // (y0 h) >> 32
  return int64_t(y0) * int32_t(h >> 32) + int64_t(mulhi32(y0, uint32_t(h)));
}

struct SoftRoot {
  uint64_t s;   // the rounded root's significand (53 bits)
  uint64_t y;   // 1 / sqrt(x), scaled: (2 / root) 2^62 with the root in [1, 2]
  int e;        // its exponent
};
// Root of a positive normal number.
HODLR_HD SoftRoot soft_root(uint64_t b) {
  const int ex = int(b >> 52) - 1023, odd = ex & 1;
  const uint64_t m = (b & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint64_t M = m << odd;   // [2^52, 2^54)
  const uint64_t X = M << 10;    // x / 4^(e + 1) in units of 2^-64: [1/4, 1)
#ifdef __CUDA_ARCH__
  const float r0 = rsqrtf(soft_float((uint32_t(127 + odd) << 23) | (uint32_t(b >> 29) & 0x7fffffu)));
#else
  const float r0 = 1.0f / std::sqrt(soft_float((uint32_t(127 + odd) << 23) | (uint32_t(b >> 29) & 0x7fffffu)));
#endif
  const uint32_t y0 = soft_seed(r0);  // 1 / sqrt(X) in units of 2^-31
  const int64_t h = int64_t(0x4000000000000000ull - mulhi64(X, uint64_t(y0) * y0));  // 1 - X y^2
  const int64_t hq = h >> 20;
  const uint64_t h2 = uint64_t(hq * hq) >> 22;  // h^2 in units of 2^-62
  // y (1 + h / 2 + 3 h^2 / 8); the next term, 5 h^3 / 16, is below 2^-61 (h below 2^-20)
  const uint64_t y = (uint64_t(y0) << 31) + uint64_t(soft_y_h(y0, h)) + ((uint64_t(y0) * (3u * uint32_t(h2))) >> 34);
  uint64_t S = mulhi64(X, y) >> 8;  // floor(sqrt(M 2^54)), at most one off
  const int64_t r = int64_t((M << 54) - S * S);
  S += r > int64_t(2 * S) ? 1 : 0;
  S -= r < 0 ? 1 : 0;
  SoftRoot R;
  R.s = (S + 1) >> 1;  // an odd S is never exact: no ties
  R.y = y;
  R.e = (ex - odd) >> 1;
  return R;
}
HODLR_HD bool soft_normal(uint64_t b) {  // positive and normal
  return (b >> 52) - 1u < 0x7feu;
}
HODLR_HD double soft_sqrt(double x) {
  const uint64_t b = soft_bits(x);
  if (!soft_normal(b)) return plain_sqrt(x);
  const SoftRoot R = soft_root(b);
  return soft_double((uint64_t(uint32_t(R.e + 1022)) << 52) + R.s);
}

// Rounded c / sqrt(x), the root rounded first (two roundings, as two operations).
HODLR_HD double soft_div_sqrt(const SoftD& c, double cv, double x) {
  const uint64_t b = soft_bits(x);
  if (soft_normal(b) && c.m != 0) {
    const SoftRoot R = soft_root(b);
    const int up = int(R.s >> 53);  // the root rounded up to 2
    const uint64_t s = R.s >> up;
    const int lt = c.m < s ? 1 : 0;
    const int e = c.e - (R.e + up) - lt;  // exponent field
    if (unsigned(e - 1) < 0x7fdu) {
      // c y 2^61 = quotient 2^62 (y of the root before it was rounded: 2^-53 off; halved when up)
      const uint64_t qx = mulhi64(c.m << 11, R.y);
      const uint64_t q = soft_quotient(c.m, s, (qx << up) >> (9 - lt), 53 + lt);
      return soft_double((uint64_t(uint32_t(e - 1)) << 52) + ((q + 1) >> 1) | (uint64_t(c.sign) << 32));
    }
  }
  return plain_div(cv, plain_sqrt(x));
}

// Rounded c / x.
HODLR_HD double soft_div(const SoftD& c, double cv, double x) {
  const SoftD d = soft_unpack(x);
  if (c.m != 0 && d.m != 0 && c.e != kSoftOdd && d.e != kSoftOdd) {
    const int lt = c.m < d.m ? 1 : 0;
    const int e = c.e - d.e + 1023 - lt;
    if (unsigned(e - 1) < 0x7fdu) {
      const float f = soft_float((127u << 23) | uint32_t((d.m >> 29) & 0x7fffffu));
#ifdef __CUDA_ARCH__
      const uint32_t y0 = soft_seed(__fdividef(1.0f, f));
#else
      const uint32_t y0 = soft_seed(1.0f / f);
#endif
      const int64_t h = int64_t(0x4000000000000000ull - mulhi64(d.m << 11, uint64_t(y0) << 31));  // 1 - s y
      const int64_t hq = h >> 20;
      const uint64_t h2 = uint64_t(hq * hq) >> 22;
      // y (1 + h + h^2), in units of 2^-62
      const uint64_t y = (uint64_t(y0) << 30) + uint64_t(soft_y_h(y0, h)) + ((uint64_t(y0) * h2) >> 32);
      const uint64_t q = soft_quotient(c.m, d.m, mulhi64(c.m << 11, y) >> (8 - lt), 53 + lt);
      return soft_double((uint64_t(uint32_t(e - 1)) << 52) + ((q + 1) >> 1) |
                         (uint64_t((c.sign ^ d.sign) & 0x80000000u) << 32));
    }
  }
  return plain_div(cv, x);
}

}  // namespace hodlr

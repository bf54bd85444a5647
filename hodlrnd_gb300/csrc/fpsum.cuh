// Sums of a few numbers with FP64's accuracy on the FP32 pipe (GB300's FP64 pipe
// takes 20 cycles of an SM for one warp instruction, its FP32 pipe a quarter of
// one).  Host code (the test against exact sums) runs the same operations.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define HODLR_HD __host__ __device__ __forceinline__
#else
#define HODLR_HD inline
#endif

namespace hodlr {

// One rounding each; no contraction.
HODLR_HD float add_rn(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(a, b);
#else
  return a + b;
#endif
}
HODLR_HD float sub_rn(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fsub_rn(a, b);
#else
  return a - b;
#endif
}
// a + b = s + e exactly (Knuth)
HODLR_HD void two_sum(float a, float b, float& s, float& e) {
  s = add_rn(a, b);
  const float bb = sub_rn(s, a);
  e = add_rn(sub_rn(a, sub_rn(s, bb)), sub_rn(b, bb));
}

// FP32 values (at most 32) summed as an FP32 pair, and whether the FP64 sum of
// the same rounds to the same FP32 value r.  With B the sum of the magnitudes:
// - rounds: the high part loses nothing and the low part, at most 32 errors of
//   2^-24 B, at most 32 roundings of 2^-24 of that, 2^-38 B in all; the FP64 sum is
//   within 2^-47 B of the exact one.  When every number within 2^-38 B of the pair
//   rounds to one FP32 value, that is the value of both.
// - exact: when no value but zeros is below 2^-18 B, all sums are multiples of
//   2^-42 B that 53 bits hold, and the low part's, at most 2^-18 B, 24 bits: both
//   sums are exact, ties included (which are common among values of like size).
// Zeros alone (their sign), infinities, NaNs and sums near FP32's limit pass neither.
struct PairSum {
  float s, c, b;
  HODLR_HD explicit PairSum(float v) : s(v), c(0.f), b(fabsf(v)) {}
  HODLR_HD void add(float v) {
    float e;
    two_sum(s, v, s, e);
    c = add_rn(c, e);
    b = add_rn(b, fabsf(v));
  }
  HODLR_HD bool rounds(float& r) const {
    float d;
    two_sum(s, c, r, d);
    const float eb = b * (1.0f / 137438953472.0f);  // 2^-37: b itself and the ends' own roundings
    return r != 0.f && add_rn(r, add_rn(d, eb)) == r && add_rn(r, sub_rn(d, eb)) == r;
  }
  template <typename At>
  HODLR_HD bool exact(int count, const At& at) const {
    float m = 2e38f;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int q = 0; q < count; q++) {
      const float v = fabsf(at(q));
      m = v > 0.f && v < m ? v : m;
    }
    return b < 1.5e38f && m < 1.5e38f && m >= b * (1.0f / 131072.0f);  // 2^-17: b's own roundings
  }
};

// The FP64 sum of the count FP32 values at(0), at(1), ... in that order, rounded to FP32.
template <typename At>
HODLR_HD float sum_in_fp64(int count, const At& at) {
  double acc = double(at(0));
  for (int q = 1; q < count; q++) acc += double(at(q));
  return float(acc);
}

// The same from the pair where that is the value (all but one sum in thousands).
template <typename At>
HODLR_HD float sum_as_fp64(int count, const At& at) {
  if (count <= 1) return at(0);
  if (count <= 32) {
    PairSum p(at(0));
    for (int q = 1; q < count; q++) p.add(at(q));
    float r;
    if (p.rounds(r) || p.exact(count, at)) return r;
  }
  return sum_in_fp64(count, at);
}

// The same for count <= U values in registers (zeros beyond count); false: the
// sum has to be formed in FP64.
template <int U>
HODLR_HD bool sum_few_as_fp64(int count, const float (&v)[U], float& r) {
  PairSum p(v[0]);
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int q = 1; q < U; q++) p.add(v[q]);
  const bool ok = p.rounds(r);
  if (count > 1) return ok || p.exact(U, [&](int q) { return v[q]; });
  r = v[0];
  return true;
}

// An unevaluated sum of three FP32 numbers: adding a pair to it loses 2^-24 of the
// third, about 2^-70 of the magnitudes added (FP64: 2^-53), for 20 operations of
// the FP32 pipe.
struct TripleSum {
  float s = 0.f, c = 0.f, t = 0.f;
  HODLR_HD void add(float x, float y, float z = 0.f) {
    float e1, e2, e3;
    two_sum(s, x, s, e1);
    two_sum(c, y, c, e2);
    two_sum(c, e1, c, e3);
    t = add_rn(add_rn(t, z), add_rn(e2, e3));
  }
  // rounded to FP64 (two roundings)
  HODLR_HD double value() const {
#ifdef __CUDA_ARCH__
    return __dadd_rn(double(s), __dadd_rn(double(c), double(t)));
#else
    return double(s) + (double(c) + double(t));
#endif
  }
  HODLR_HD bool finite() const { return fabsf(s) <= 3.4e38f && fabsf(c) <= 3.4e38f; }
};

}  // namespace hodlr

// Device-side helpers shared by the HODLRnD GB300 kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "softfp.cuh"

namespace hodlr {

// Process-wide count of this engine's kernel launches (hodlr_kernel_launches).
inline std::atomic<uint64_t> g_kernel_launches{0};
inline void count_launches(uint64_t k) { g_kernel_launches.fetch_add(k, std::memory_order_relaxed); }

// Kernel kinds (include/hodlrnd.h).
enum : int { kInvR = 1, kInvR2 = 2, kLogR = 3, kExpNegR = 4 };

struct KernelDev {
  int kind;
  double scale, diag;
};

// Points in tree order, structure of arrays: coordinate k of point i is
// x[k * ld + i].
struct PointsDev {
  const double* x;
  int64_t ld;
};

// The kernel of a squared distance, with one rounding per operation; square
// roots and divisions on the integer pipe (softfp.cuh: 3D assembly of near
// tiles 1.95 -> 0.71 ms at N = 100003).
inline __device__ __noinline__ double kernel_log_exp(int kind, double scale, double d2) {
  const double r = soft_sqrt(d2);
  return __dmul_rn(scale, kind == kLogR ? log(r) : exp(-r));
}
__device__ __forceinline__ double kernel_of(const KernelDev& K, double d2) {
  switch (K.kind) {
    case kInvR: return soft_div_sqrt(soft_unpack(K.scale), K.scale, d2);
    case kInvR2: return soft_div(soft_unpack(K.scale), K.scale, d2);
    default: return kernel_log_exp(K.kind, K.scale, d2);
  }
}

// One matrix entry A(i, j) for tree positions i, j (kernel_function::getRow /
// getCol / getMatrix + the user getMatrixEntry, include/kernel_function.hpp:20-53).
// d2 is accumulated in dimension order with one rounding per operation (the
// explicit _rn intrinsics keep the compiler from contracting into FMAs); sqrt
// and division are IEEE round-to-nearest on both sides, so the 1/r and 1/r^2
// entries are bit-identical to the scalar host code.  The log r and e^-r
// kinds call CUDA's log and exp, which need not round as the host's libm
// does: those entries agree to a few units in the last place.
template <int D>
__device__ __forceinline__ double kernel_entry(const PointsDev& P, const KernelDev& K, int64_t i, int64_t j,
                                               const double* xi) {
  if (i == j) return K.diag;
  double d2;
#pragma unroll
  for (int k = 0; k < D; k++) {
    const double t = __dsub_rn(xi[k], P.x[k * P.ld + j]);
    const double tt = __dmul_rn(t, t);
    d2 = k == 0 ? tt : __dadd_rn(d2, tt);  // 0 + tt is tt
  }
  return kernel_of(K, d2);
}

// The same entry from two staged coordinate vectors (stride ld between
// coordinates); same_point: the tree positions are equal (the diagonal).
template <int D>
__device__ __forceinline__ double kernel_entry_xy(const KernelDev& K, bool same_point, const double* xi,
                                                  const double* xj, int ld) {
  if (same_point) return K.diag;
  double d2;
#pragma unroll
  for (int k = 0; k < D; k++) {
    const double t = __dsub_rn(xi[k], xj[k * ld]);
    const double tt = __dmul_rn(t, t);
    d2 = k == 0 ? tt : __dadd_rn(d2, tt);  // 0 + tt is tt
  }
  return kernel_of(K, d2);
}

template <int D>
__device__ __forceinline__ void load_point(const PointsDev& P, int64_t i, double* xi) {
#pragma unroll
  for (int k = 0; k < D; k++) xi[k] = P.x[k * P.ld + i];
}

// a = hi + lo + e, |e| <= 2^-46 |a|: hi is a's sign, exponent and leading 24
// significand bits, lo the next 23 bits (truncated), both exact floats, built
// with integer operations only (GB300's FP64 pipe is far slower than its
// FP32 and integer pipes).  |a| < 2^-70 gives (0, 0), an absolute error below
// 8.5e-22; |a| >= 2^127 falls back to a rounding conversion.
__device__ __forceinline__ float2 split_d(double a) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(a));
  const unsigned hi32 = unsigned(b >> 32), lo32 = unsigned(b);
  const int e = int((hi32 >> 20) & 0x7ffu);
  if (e < 1023 - 70) return make_float2(0.f, 0.f);
  if (e > 1023 + 126) return make_float2(__double2float_rn(a), 0.f);
  const unsigned sign = hi32 & 0x80000000u;
  const unsigned m23 = ((hi32 & 0xfffffu) << 3) | (lo32 >> 29);
  const float hi = __uint_as_float(sign | (unsigned(e - 1023 + 127) << 23) | m23);
  // the next 23 bits r as a float (2^23 + r - 2^23, exact), times 2^(e - 1069)
  const float r = __fsub_rn(__uint_as_float(0x4B000000u | ((lo32 & 0x1fffffffu) >> 6)), 8388608.f);
  const float lo = __fmul_rn(r, __uint_as_float(unsigned(e - 1069 + 127) << 23));
  return make_float2(hi, __uint_as_float(__float_as_uint(lo) | sign));
}

// s + c += (a.x + a.y)(b.x + b.y)
__device__ __forceinline__ void dot2_add(float& s, float& c, float2 a, float2 b) {
  const float p = __fmul_rn(a.x, b.x);
  const float pe = __fmaf_rn(a.x, b.x, -p);
  const float t = __fmaf_rn(a.x, b.y, __fmaf_rn(a.y, b.x, pe));
  const float s2 = __fadd_rn(s, p);
  const float bb = __fsub_rn(s2, s);
  const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(s2, bb)), __fsub_rn(p, bb));
  s = s2;
  c = __fadd_rn(c, __fadd_rn(err, t));
}

// (s, c) + (s2, c2) as an unevaluated FP32 pair (TwoSum on the high parts).
__device__ __forceinline__ void pair_add(float& s, float& c, float s2, float c2) {
  const float t = __fadd_rn(s, s2);
  const float bb = __fsub_rn(t, s);
  const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bb)), __fsub_rn(s2, bb));
  s = t;
  c = __fadd_rn(__fadd_rn(c, c2), err);
}

// A pivot candidate's value as an integer that orders like its magnitude: the
// bits of |v|, with the sign below them (FP64 comparisons take GB300's slow FP64
// pipe, integer ones do not).  The largest (key >> 1) with the lowest index is the
// pivot; a NaN is no candidate (it compares false), nor is "none" = (0, INT_MAX),
// which loses the tie with a zero.
__device__ __forceinline__ unsigned long long pivot_key(double v) {
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v));
  return (b << 1) | (b >> 63);
}
__device__ __forceinline__ bool pivot_nan(unsigned long long key) { return (key >> 1) > 0x7ff0000000000000ull; }
__device__ __forceinline__ double pivot_value(unsigned long long key) {
  return __longlong_as_double(static_cast<long long>((key >> 1) | (key << 63)));
}
__device__ __forceinline__ bool pivot_better(unsigned long long k2, int i2, unsigned long long k, int i) {
  const unsigned long long a2 = k2 >> 1, a = k >> 1;
  return a2 > a || (a2 == a && i2 < i);
}

// ---------------------------------------------------------------- teams
// A "team" is the group of threads that compresses one block: a warp, or a
// whole CTA.  All members call every team function (uniform control flow).

struct WarpTeam {
  static constexpr int kSize = 32;
  __device__ __forceinline__ int tid() const { return threadIdx.x & 31; }
  __device__ __forceinline__ void sync() const { __syncwarp(); }
  __device__ __forceinline__ double sum(double v) const {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
  // The sums of a and b (one butterfly: lanes 0-15 end with a's, 16-31 with b's).
  __device__ __forceinline__ void sum2(double& a, double& b) const {
    const bool up = (threadIdx.x & 16) != 0;
    double v = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    a = __shfl_sync(0xffffffffu, v, 0);
    b = __shfl_sync(0xffffffffu, v, 16);
  }
  // Largest |v|, lowest index on ties (kernel_function::maxAbsVector keeps the
  // first maximum, include/kernel_function.hpp:55-68).
  __device__ __forceinline__ void argmax(unsigned long long& k, int& i) const {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long k2 = __shfl_xor_sync(0xffffffffu, k, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, i, o);
      if (pivot_better(k2, i2, k, i)) {
        k = k2;
        i = i2;
      }
    }
  }
  __device__ __forceinline__ int bcast(int v) const { return __shfl_sync(0xffffffffu, v, 0); }
  __device__ __forceinline__ double bcast(double v) const { return __shfl_sync(0xffffffffu, v, 0); }
};

// T lanes of one warp (T = 8 or 16): lanes 0..T-1, T..2T-1, ... each form a
// team of their own.  Teams of one warp may follow different control flow
// (their blocks differ); every shuffle names only the team's lanes.
template <int T>
struct SubTeam {
  static constexpr int kSize = T;
  unsigned mask;
  __device__ __forceinline__ SubTeam() : mask(((1u << T) - 1u) << ((threadIdx.x & 31) & ~(T - 1))) {}
  __device__ __forceinline__ int tid() const { return threadIdx.x & (T - 1); }
  __device__ __forceinline__ void sync() const { __syncwarp(mask); }
  __device__ __forceinline__ double sum(double v) const {
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, T);
    return v;
  }
  __device__ __forceinline__ void sum2(double& a, double& b) const {
    a = sum(a);
    b = sum(b);
  }
  __device__ __forceinline__ void argmax(unsigned long long& k, int& i) const {
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) {
      const unsigned long long k2 = __shfl_xor_sync(mask, k, o, T);
      const int i2 = __shfl_xor_sync(mask, i, o, T);
      if (pivot_better(k2, i2, k, i)) {
        k = k2;
        i = i2;
      }
    }
  }
  __device__ __forceinline__ int bcast(int v) const { return __shfl_sync(mask, v, 0, T); }
  __device__ __forceinline__ double bcast(double v) const { return __shfl_sync(mask, v, 0, T); }
};

template <int NT>
struct CtaTeam {
  static constexpr int kSize = NT;
  static constexpr int kWarps = NT / 32;
  double* red;    // shared, kWarps + 1
  double* red2;   // shared, kWarps + 1
  int* redi;      // shared, kWarps + 1
  double* terms;  // shared, kNormChunk: the norm estimate's terms of one pass (ACA)
  // terms[k] = v (the same in every lane of a warp)
  __device__ __forceinline__ void put_term(int k, double v) const {
    if ((threadIdx.x & 31) == 0) terms[k] = v;
  }
  __device__ __forceinline__ double term(int k) const { return terms[k]; }
  __device__ __forceinline__ int tid() const { return threadIdx.x; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
  __device__ __forceinline__ double sum(double v) const {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
      v = lane < kWarps ? red[lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[kWarps] = v;
    }
    __syncthreads();
    v = red[kWarps];
    __syncthreads();
    return v;
  }
  __device__ __forceinline__ void sum2(double& a, double& b) const {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    WarpTeam().sum2(a, b);
    if (lane == 0) {
      red[w] = a;
      red2[w] = b;
    }
    __syncthreads();
    if (w == 0) {
      a = lane < kWarps ? red[lane] : 0.0;
      b = lane < kWarps ? red2[lane] : 0.0;
      WarpTeam().sum2(a, b);
      if (lane == 0) {
        red[kWarps] = a;
        red2[kWarps] = b;
      }
    }
    __syncthreads();
    a = red[kWarps];
    b = red2[kWarps];
    __syncthreads();
  }
  __device__ __forceinline__ void argmax(unsigned long long& k, int& i) const {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    WarpTeam().argmax(k, i);
    __shared__ unsigned long long sk[kWarps + 1];
    if (lane == 0) {
      sk[w] = k;
      redi[w] = i;
    }
    __syncthreads();
    if (w == 0) {
      k = lane < kWarps ? sk[lane] : 0ull;
      i = lane < kWarps ? redi[lane] : 0x7fffffff;
      WarpTeam().argmax(k, i);
      if (lane == 0) {
        sk[kWarps] = k;
        redi[kWarps] = i;
      }
    }
    __syncthreads();
    k = sk[kWarps];
    i = redi[kWarps];
    __syncthreads();
  }
  __device__ __forceinline__ int bcast(int v) const {
    if (threadIdx.x == 0) redi[kWarps] = v;
    __syncthreads();
    v = redi[kWarps];
    __syncthreads();
    return v;
  }
  __device__ __forceinline__ double bcast(double v) const {
    if (threadIdx.x == 0) red[kWarps] = v;
    __syncthreads();
    v = red[kWarps];
    __syncthreads();
    return v;
  }
};

__host__ __device__ inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

}  // namespace hodlr

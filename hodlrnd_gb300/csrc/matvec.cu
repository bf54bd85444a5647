// HODLR matvec kernels (see matvec.h).
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "bulk.cuh"
#include "device.cuh"
#include "fpsum.cuh"
#include "matvec.h"

namespace hodlr {

__device__ unsigned int g_stream_timeouts = 0;

cudaError_t read_stream_timeouts(unsigned int* host, cudaStream_t st) {
  return cudaMemcpyFromSymbolAsync(host, g_stream_timeouts, sizeof(unsigned int), 0, cudaMemcpyDeviceToHost, st);
}

namespace {

constexpr int kWarpsPerCta = 8;

// BF16 storage element (bits only; arithmetic converts to FP32)
struct bf16 {
  unsigned short b;
};
__device__ __forceinline__ float bf2f(unsigned short b) { return __uint_as_float(uint32_t(b) << 16); }

template <typename T>
struct Vec16;
template <>
struct Vec16<bf16> {
  using type = uint4;  // 8 BF16 values
};
template <>
struct Vec16<float> {
  using type = float4;
};

// Two FP32 operations in one instruction (packed pairs), each rounded to nearest
// as the scalar one: the FP32 pipe takes as many operations a clock either way
// (128 per SM measured), but in half the issue slots, which the compensated and
// register-tiled products otherwise fill before the pipe (a compensated product
// of a loop of its own: 0.285 warp entries per clock and SM scalar, 0.347 packed;
// whole products: 3D N = 262144 FP32 factors 2.82 -> 2.63 ms, 4D N = 65536 BF16
// 1.27 -> 1.20).
__device__ __forceinline__ uint64_t pack_f2(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void unpack_f2(uint64_t v, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul_f2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add_f2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t sub_f2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Accumulators.  Acc<float> and Acc<double> are plain sums.  Acc<DF> is a
// compensated FP32 accumulator: the running value is hi + lo, each product
// of an FP32 matrix entry with an FP64 input split as xh + xl is formed
// exactly with an FMA (p + e == v * xh), and each addition keeps its
// rounding error (TwoSum), following Ogita, Rump and Oishi, "Accurate sum
// and dot product", SIAM J. Sci. Comput. 26 (2005), algorithm Dot2.  The
// result is about as accurate as FP64 accumulation while using only the
// FP32 pipe (GB300's FP64 rate is far below what a streaming matvec needs).
struct DF {
  float hi, lo;
};

template <typename T>
struct Acc;

template <>
struct Acc<float> {
  using A = float;
  using X = float;
  static __device__ __forceinline__ X in(float v) { return v; }
  static __device__ __forceinline__ X in(double v) { return float(v); }
  static __device__ __forceinline__ A zero() { return 0.f; }
  static __device__ __forceinline__ void fma(A& a, float v, X x) { a += v * x; }
  static __device__ __forceinline__ A add(A a, A b) { return a + b; }
  static __device__ __forceinline__ A scale(A a, float s) { return a * s; }
  static __device__ __forceinline__ X xscale(X x, float s) { return x * s; }
  static __device__ __forceinline__ A shfl_xor(A a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
  static __device__ __forceinline__ A shfl_down(A a, int o) { return __shfl_down_sync(0xffffffffu, a, o); }
  static __device__ __forceinline__ X shfl(X x, int src) { return __shfl_sync(0xffffffffu, x, src); }
  static __device__ __forceinline__ double value(A a) { return double(a); }
};

template <>
struct Acc<double> {
  using A = double;
  using X = double;
  static __device__ __forceinline__ X in(float v) { return double(v); }
  static __device__ __forceinline__ X in(double v) { return v; }
  static __device__ __forceinline__ A zero() { return 0.0; }
  static __device__ __forceinline__ void fma(A& a, float v, X x) { a += double(v) * x; }
  static __device__ __forceinline__ void fma(A& a, double v, X x) { a += v * x; }
  static __device__ __forceinline__ A add(A a, A b) { return a + b; }
  static __device__ __forceinline__ A scale(A a, float s) { return a * double(s); }
  static __device__ __forceinline__ X xscale(X x, float s) { return x * double(s); }
  static __device__ __forceinline__ A shfl_xor(A a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
  static __device__ __forceinline__ A shfl_down(A a, int o) { return __shfl_down_sync(0xffffffffu, a, o); }
  static __device__ __forceinline__ X shfl(X x, int src) { return __shfl_sync(0xffffffffu, x, src); }
  static __device__ __forceinline__ double value(A a) { return a; }
};

template <>
struct Acc<DF> {
  using A = DF;
  using X = DF;
  static __device__ __forceinline__ X in(double v) {
    const float h = __double2float_rn(v);
    return DF{h, __double2float_rn(v - double(h))};
  }
  static __device__ __forceinline__ X in(float v) { return DF{v, 0.f}; }
  static __device__ __forceinline__ X in(float2 v) { return DF{v.x, v.y}; }
  static __device__ __forceinline__ A zero() { return DF{0.f, 0.f}; }
  // hi + lo renormalised (FastTwoSum) as an input pair
  static __device__ __forceinline__ float2 to_pair(A a) {
    const float s = __fadd_rn(a.hi, a.lo);
    return make_float2(s, __fsub_rn(a.lo, __fsub_rn(s, a.hi)));
  }
  // a += v * (x.hi + x.lo)
  static __device__ __forceinline__ void fma(A& a, float v, X x) {
    const float p = __fmul_rn(v, x.hi);
    float e = __fmaf_rn(v, x.hi, -p);
    e = __fmaf_rn(v, x.lo, e);
    const float s = __fadd_rn(a.hi, p);
    const float bb = __fsub_rn(s, a.hi);
    const float t = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(p, bb));
    a.hi = s;
    a.lo = __fadd_rn(a.lo, __fadd_rn(t, e));
  }
  static __device__ __forceinline__ void fma(A& a, bf16 v, X x) { fma(a, bf2f(v.b), x); }
  // a += va * xa, b += vb * xb: the operations of fma() on packed pairs
  static __device__ __forceinline__ void fma2(A& a, A& b, float va, float vb, X xa, X xb) {
    const uint64_t v = pack_f2(va, vb), ah = pack_f2(a.hi, b.hi);
    const uint64_t p = mul_f2(v, pack_f2(xa.hi, xb.hi));
    uint64_t e = fma_f2(v, pack_f2(-xa.hi, -xb.hi), p);  // the negative of p's error
    e = fma_f2(v, pack_f2(-xa.lo, -xb.lo), e);
    const uint64_t s = add_f2(ah, p), bb = sub_f2(s, ah);
    const uint64_t t = add_f2(sub_f2(ah, sub_f2(s, bb)), sub_f2(p, bb));
    const uint64_t l = add_f2(pack_f2(a.lo, b.lo), sub_f2(t, e));
    unpack_f2(s, a.hi, b.hi);
    unpack_f2(l, a.lo, b.lo);
  }
  // (hi + lo) * s with the rounding error of hi * s kept (TwoProduct by FMA)
  static __device__ __forceinline__ A scale(A a, float s) {
    const float p = __fmul_rn(a.hi, s);
    return DF{p, __fmaf_rn(a.lo, s, __fmaf_rn(a.hi, s, -p))};
  }
  static __device__ __forceinline__ X xscale(X x, float s) { return scale(x, s); }
  static __device__ __forceinline__ A add(A a, A b) {
    const float s = __fadd_rn(a.hi, b.hi);
    const float bb = __fsub_rn(s, a.hi);
    const float t = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));
    return DF{s, __fadd_rn(__fadd_rn(a.lo, b.lo), t)};
  }
  static __device__ __forceinline__ A shfl_xor(A a, int o) {
    return DF{__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)};
  }
  static __device__ __forceinline__ A shfl_down(A a, int o) {
    return DF{__shfl_down_sync(0xffffffffu, a.hi, o), __shfl_down_sync(0xffffffffu, a.lo, o)};
  }
  static __device__ __forceinline__ X shfl(X x, int src) {
    return DF{__shfl_sync(0xffffffffu, x.hi, src), __shfl_sync(0xffffffffu, x.lo, src)};
  }
  static __device__ __forceinline__ double value(A a) { return double(a.hi) + double(a.lo); }
};

// Element types of a launch: the input vector buffer [x | z] (TI) and the
// outputs and partial sums (TY).  Compensated accumulation reads its inputs
// pre-split into (hi, lo) FP32 pairs, so its hot loops use no FP64 operation.
template <typename TACC>
struct IO;
template <>
struct IO<float> {
  using TI = float;
  using TY = float;
  static __device__ __forceinline__ TI from_double(double v) { return float(v); }
};
template <>
struct IO<double> {
  using TI = double;
  using TY = double;
  static __device__ __forceinline__ TI from_double(double v) { return v; }
};
template <>
struct IO<DF> {
  using TI = float2;
  using TY = double;
  static __device__ __forceinline__ TI from_double(double v) {
    const float h = __double2float_rn(v);
    return make_float2(h, __double2float_rn(v - double(h)));
  }
};

// Relaxed accumulation (Accum::kRelaxed): the inputs and outputs of DF
// (split FP64 inputs, FP64 outputs) with plain FP32 sums of the products of
// the FP32 factors with the inputs' high parts.  Cheaper, and accurate to
// about 1e-6 relative: what an inexact Krylov method may use once its
// residual has dropped far enough.
struct FH {};

template <>
struct Acc<FH> {
  using A = float;
  using X = float;
  static __device__ __forceinline__ X in(float2 v) { return v.x; }
  static __device__ __forceinline__ X in(float v) { return v; }
  static __device__ __forceinline__ A zero() { return 0.f; }
  static __device__ __forceinline__ void fma(A& a, float v, X x) { a = __fmaf_rn(v, x, a); }
  static __device__ __forceinline__ void fma(A& a, bf16 v, X x) { a = __fmaf_rn(bf2f(v.b), x, a); }
  static __device__ __forceinline__ A add(A a, A b) { return a + b; }
  static __device__ __forceinline__ A scale(A a, float s) { return a * s; }
  static __device__ __forceinline__ X xscale(X x, float s) { return x * s; }
  static __device__ __forceinline__ A shfl_xor(A a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
  static __device__ __forceinline__ A shfl_down(A a, int o) { return __shfl_down_sync(0xffffffffu, a, o); }
  static __device__ __forceinline__ X shfl(X x, int src) { return __shfl_sync(0xffffffffu, x, src); }
  static __device__ __forceinline__ double value(A a) { return double(a); }
};

template <>
struct IO<FH> {
  using TI = float2;
  using TY = double;
  static __device__ __forceinline__ TI from_double(double v) { return IO<DF>::from_double(v); }
};

// a += va * xa, b += vb * xb; compensated sums as packed pairs
template <typename TACC, typename V>
__device__ __forceinline__ void fma_pair(typename Acc<TACC>::A& a, typename Acc<TACC>::A& b, V va, V vb,
                                         typename Acc<TACC>::X xa, typename Acc<TACC>::X xb) {
  if constexpr (std::is_same_v<TACC, DF>) {
    Acc<DF>::fma2(a, b, va, vb, xa, xb);
  } else {
    Acc<TACC>::fma(a, va, xa);
    Acc<TACC>::fma(b, vb, xb);
  }
}

// acc[q] += a[q] * x for the components of a 16-byte vector
template <typename TACC, typename X>
__device__ __forceinline__ void axpy16(const float4& a, X x, typename Acc<TACC>::A* acc) {
  fma_pair<TACC>(acc[0], acc[1], a.x, a.y, x, x);
  fma_pair<TACC>(acc[2], acc[3], a.z, a.w, x, x);
}
template <typename TACC, typename X>
__device__ __forceinline__ void axpy16(const uint4& a, X x, typename Acc<TACC>::A* acc) {
  fma_pair<TACC>(acc[0], acc[1], __uint_as_float(a.x << 16), __uint_as_float(a.x & 0xffff0000u), x, x);
  fma_pair<TACC>(acc[2], acc[3], __uint_as_float(a.y << 16), __uint_as_float(a.y & 0xffff0000u), x, x);
  fma_pair<TACC>(acc[4], acc[5], __uint_as_float(a.z << 16), __uint_as_float(a.z & 0xffff0000u), x, x);
  fma_pair<TACC>(acc[6], acc[7], __uint_as_float(a.w << 16), __uint_as_float(a.w & 0xffff0000u), x, x);
}

template <typename T>
__device__ __forceinline__ T vzero();
template <>
__device__ __forceinline__ uint4 vzero<uint4>() {
  return make_uint4(0u, 0u, 0u, 0u);
}
template <>
__device__ __forceinline__ float4 vzero<float4>() {
  return make_float4(0.f, 0.f, 0.f, 0.f);
}
// Input value of column j of a segment: x_j, times the column scale of a BF16
// dense tile (cs non-null).
template <typename TACC, typename TX>
__device__ __forceinline__ typename Acc<TACC>::X seg_in(TX x, const float* cs, int j) {
  return cs ? Acc<TACC>::xscale(Acc<TACC>::in(x), __ldg(cs + j)) : Acc<TACC>::in(x);
}

// An input value back in the staged (hi, lo) form, after scaling.
template <typename TACC>
__device__ __forceinline__ float2 x_pair(typename Acc<TACC>::X x);
template <>
__device__ __forceinline__ float2 x_pair<DF>(DF x) {
  return make_float2(x.hi, x.lo);
}
template <>
__device__ __forceinline__ float2 x_pair<FH>(float x) {
  return make_float2(x, 0.f);
}

template <typename TACC>
__device__ __forceinline__ typename IO<TACC>::TI to_input(typename Acc<TACC>::A a) {
  return typename IO<TACC>::TI(Acc<TACC>::value(a));
}
template <>
__device__ __forceinline__ float2 to_input<DF>(DF a) {
  return Acc<DF>::to_pair(a);
}
template <>
__device__ __forceinline__ float2 to_input<FH>(float a) {
  return make_float2(a, 0.f);
}

// Phase 1: z_b = V_b^T x_s with V_b stored row major (n x vpad(r)).  The
// CPL = 16 / sizeof(TA) columns of a 16-byte load belong to one lane; P lanes
// cover a row's nk columns and the warp's G = 32 / P lane groups take
// consecutive rows, so each 16-byte read of the warp covers G whole rows.
// Each lane keeps CPL running sums, over rows g, g + G, g + 2G, ... of the
// item in that order; the groups are added by shuffles once at the end.  A
// block with more rows than one item takes writes partial sums (the last item
// adds them in order).
//
// An item that covers whole rows (k0 == 0, nk == vpad(r)) reads one
// contiguous run of V, and its inputs x[j0 .. j1) are contiguous too: both
// are staged through a per-warp ring of kZStages shared-memory stages by bulk
// copies, R rows per stage (R a multiple of G, so every lane's row order is
// the one above).  Other items (blocks of more than 128 FP32 or 64 FP64
// columns) load V directly.
// Ring shapes (stages x bytes) of the staged kernels; HODLR_TUNE_* override
// them at compile time for tuning runs.  Two stages per warp measured best on
// GB300: the shared memory per warp, not the stage count, limits the warps
// per SM, and more warps hide more latency than deeper rings.  A stage of V^T x
// holds its rows of V and after them their inputs, so that rows of any width fill
// it; 3.4 KB allow 8 CTAs per SM of the kernels that need 64 registers.  (With
// 4 KB of V and room for the inputs of the narrowest rows apart from it, 4 CTAs
// fitted.)  N = 262144 in 3D (FP32): 989 -> 919 us; 4D N = 65536 (BF16), where most
// items are two stages: 415 -> 312.
#ifndef HODLR_TUNE_Z_STAGES
#define HODLR_TUNE_Z_STAGES 2
#endif
#ifndef HODLR_TUNE_Z_BYTES
#define HODLR_TUNE_Z_BYTES 3488
#endif
#ifndef HODLR_TUNE_P_STAGES
#define HODLR_TUNE_P_STAGES 2
#endif
#ifndef HODLR_TUNE_P_BYTES
#define HODLR_TUNE_P_BYTES 4096
#endif
#ifndef HODLR_TUNE_S_STAGES
#define HODLR_TUNE_S_STAGES 2
#endif
#ifndef HODLR_TUNE_S_BYTES
#define HODLR_TUNE_S_BYTES 2048
#endif
#ifndef HODLR_TUNE_S_MINB
#define HODLR_TUNE_S_MINB 6  // leaf-panel CTAs per SM the register allocation must allow (no spills at 6)
#endif
constexpr int kZWarps = 4;                      // warps per CTA of zgemv_kernel
constexpr int kZStages = HODLR_TUNE_Z_STAGES;   // ring stages per warp
// V and input bytes per stage: R rows of V and of 8 input bytes, plus 2 x 15
// bytes of alignment slack, rounded to 16
constexpr int kZStageBytes = HODLR_TUNE_Z_BYTES;
constexpr int kZWarpSmem = 64 + kZStages * kZStageBytes;
static_assert(kZStageBytes % 16 == 0 && kZStageBytes >= 32 + 512 + 32 * 8, "bulk copy destinations must stay 16-byte aligned");

// Sum of `count` partial sums, `stride` apart, in an order that depends on
// count alone: one after another up to 8 of them; more (small operators, whose
// work is cut into many short items) go to 8 running sums, so that 8 loads are
// in flight instead of one load latency per part.  Read past L1: other SMs
// wrote the parts.
template <typename T>
__device__ __forceinline__ T sum_parts(const T* p, int count, int64_t stride) {
  T acc = T(0);
  if (count <= 8) {
    for (int q = 0; q < count; q++) acc += __ldcg(p + q * stride);
    return acc;
  }
  T a[8];
#pragma unroll
  for (int k = 0; k < 8; k++) a[k] = __ldcg(p + k * stride);
  int q = 8;
  for (; q + 8 <= count; q += 8) {
    T v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = __ldcg(p + (q + k) * stride);
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] += v[k];
  }
#pragma unroll
  for (int k = 0; k < 7; k++)
    if (q + k < count) a[k] += __ldcg(p + (q + k) * stride);
  return ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
}

// The end of an item: acc[q] (column p * CPL + q of the item) is summed over
// the G = 32 / P lanes sharing p by a transposed butterfly -- while a lane
// holds several columns, each exchange hands half of them to the partner
// lane and keeps the other half -- so lane l ends with the total of column
// p * CPL + coff(l) + k in acc[k], k < w; lanes that differ only in the bits
// of the plain exchanges that follow hold the same totals, and the one with
// those bits clear writes them.
template <typename TA, typename TACC>
__device__ __forceinline__ void z_finish(typename Acc<TACC>::A* acc, int P, int lane, const ZItem& it,
                                         const ZBlock& Z, typename IO<TACC>::TI* z,
                                         typename IO<TACC>::TY* zpart) {
  using AC = Acc<TACC>;
  constexpr int CPL = 16 / int(sizeof(TA));
  int coff = 0, w = CPL, o = 16;
#pragma unroll
  for (int lv = 0; (CPL >> lv) > 1; lv++, o >>= 1) {
    if (o < P) break;
    const int half = CPL >> (lv + 1);
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < CPL / 2; k++) {
      if (k < half) {
        const typename AC::A send = up ? acc[k] : acc[k + half];
        const typename AC::A keep = up ? acc[k + half] : acc[k];
        acc[k] = AC::add(keep, AC::shfl_xor(send, o));
      }
    }
    if (up) coff += half;
    w = half;
  }
  bool writer = true;
  for (; o >= P; o >>= 1) {  // w == 1 here
    acc[0] = AC::add(acc[0], AC::shfl_xor(acc[0], o));
    if (lane & o) writer = false;
  }
  const int p = lane % P;
  if (!writer || p * CPL >= it.nk) return;
#pragma unroll
  for (int k = 0; k < CPL; k++) {
    if (k < w) {
      const int c = p * CPL + coff + k;  // column within the item
      typename AC::A v = acc[k];
      // BF16: z columns carry the product of U's and V's column scales
      if (sizeof(TA) == 2 && Z.zscale && it.k0 + c < Z.r) v = AC::scale(v, __ldg(Z.zscale + it.k0 + c));
      if (it.part < 0) {
        if (it.k0 + c < Z.r) z[it.k0 + c] = to_input<TACC>(v);
      } else {
        zpart[it.part + c] = typename IO<TACC>::TY(AC::value(v));
      }
    }
  }
}

template <typename TA, typename TACC>
__global__ void __launch_bounds__(kZWarps * 32) zgemv_kernel(const ZBlock* __restrict__ zb,
                                                           const ZItem* __restrict__ items, int nitems,
                                                           typename IO<TACC>::TY* __restrict__ zpart,
                                                           typename IO<TACC>::TI* in) {
  using TX = typename IO<TACC>::TI;
  constexpr int CPL = 16 / int(sizeof(TA));
  using VT = typename Vec16<TA>::type;
  using AC = Acc<TACC>;
  extern __shared__ __align__(16) unsigned char zsm[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * kZWarps + wid;
  if (w >= nitems) return;
  const ZItem it = items[w];
  const ZBlock Z = zb[it.zb];
  const int64_t rp = vpad(Z.r, int(sizeof(TA)));
  const TX* x = in + Z.x_off;
  TX* z = in + Z.z_off;
  const int lanes = (it.nk + CPL - 1) / CPL;
  const int P = lanes <= 1 ? 1 : 1 << (32 - __clz(lanes - 1));  // next power of two >= lanes
  const int G = 32 / P, g = lane / P, p = lane % P;
  const bool cact = p < lanes;
  typename AC::A acc[CPL];
#pragma unroll
  for (int q = 0; q < CPL; q++) acc[q] = AC::zero();
  if (it.nst > 0) {
    // rows of rowb = rp * sizeof(TA) bytes (16 .. 512, a multiple of 16); V
    // is 16-byte aligned (factor chunks are, and every block's V starts on a
    // 16-byte boundary), so every stage's source and size are too.  The input
    // run is copied from its 16-byte boundary below to the one above; the
    // input buffers carry 16 bytes of padding at their end for that.  R and
    // nst come from z_item_stages: R a multiple of G whose rows fit a stage.
    unsigned char* base = zsm + wid * kZWarpSmem;
    uint64_t* bar = reinterpret_cast<uint64_t*>(base);
    unsigned char* vbuf = base + 64;
    const int rowb = int(rp) * int(sizeof(TA));
    const int R = it.R, nst = it.nst;
    const int nrows = it.j1 - it.j0;
    const TA* V = static_cast<const TA*>(Z.V) + int64_t(it.j0) * rp;
    const TX* xr = x + it.j0;
    if (lane == 0) {
#pragma unroll
      for (int s = 0; s < kZStages; s++) mbar_init(bar + s, 1);
      fence_mbar_init();
    }
    __syncwarp();
    auto issue = [&](int q) {  // lane 0
      const int s = q % kZStages;
      const int r0 = q * R, nr = min(R, nrows - r0);
      const uint32_t vb = uint32_t(nr) * uint32_t(rowb);
      const unsigned char* xs = reinterpret_cast<const unsigned char*>(xr + r0);
      const unsigned char* xa = static_cast<const unsigned char*>(align_down16(xs));
      const uint32_t xb = uint32_t((xs + size_t(nr) * sizeof(TX) - xa + 15) & ~size_t(15));
      fence_proxy_async();
      mbar_expect_tx(bar + s, vb + xb);
      bulk_g2s(vbuf + s * kZStageBytes, V + int64_t(r0) * rp, vb, bar + s);
      bulk_g2s(vbuf + s * kZStageBytes + R * rowb, xa, xb, bar + s);
    };
    if (lane == 0)
      for (int q = 0; q < min(kZStages, nst); q++) issue(q);
    for (int q = 0; q < nst; q++) {
      const int s = q % kZStages;
      const bool ok = __all_sync(0xffffffffu, mbar_wait(bar + s, uint32_t(q / kZStages) & 1u));
      if (!ok) {
        // give up: count it, let the copies still in flight land, return
        if (lane == 0) atomicAdd(&g_stream_timeouts, 1u);
        for (int t = q; t < min(q + kZStages, nst); t++) mbar_wait(bar + t % kZStages, uint32_t(t / kZStages) & 1u);
        return;
      }
      const int r0 = q * R, nr = min(R, nrows - r0);
      const int xo = int((reinterpret_cast<uintptr_t>(xr + r0) & 15u) / sizeof(TX));
      const TX* xsm = reinterpret_cast<const TX*>(vbuf + s * kZStageBytes + R * rowb) + xo;
      const unsigned char* vs = vbuf + s * kZStageBytes + p * 16;
      for (int i = g; i < nr; i += G) {
        const VT v = cact ? *reinterpret_cast<const VT*>(vs + i * rowb) : vzero<VT>();
        axpy16<TACC>(v, AC::in(xsm[i]), acc);
      }
      __syncwarp();
      if (lane == 0 && q + kZStages < nst) issue(q + kZStages);
    }
  } else {
    const TA* Vc = static_cast<const TA*>(Z.V) + it.k0 + p * CPL;
    int j = it.j0 + g;
    for (; j + 3 * G < it.j1; j += 4 * G) {
      VT v[4];
      typename AC::X xs[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        v[u] = cact ? __ldg(reinterpret_cast<const VT*>(Vc + int64_t(j + u * G) * rp)) : vzero<VT>();
        xs[u] = AC::in(x[j + u * G]);
      }
#pragma unroll
      for (int u = 0; u < 4; u++) axpy16<TACC>(v[u], xs[u], acc);
    }
    for (; j < it.j1; j += G) {
      const VT v = cact ? __ldg(reinterpret_cast<const VT*>(Vc + int64_t(j) * rp)) : vzero<VT>();
      axpy16<TACC>(v, AC::in(x[j]), acc);
    }
  }
  z_finish<TA, TACC>(acc, P, lane, it, Z, z, zpart);
}

// z of split blocks: each fix's columns summed over its parts.
template <typename TACC>
__global__ void __launch_bounds__(kZPart) zfix_kernel(const ZFix* __restrict__ fix,
                                                      const typename IO<TACC>::TY* __restrict__ zpart,
                                                      typename IO<TACC>::TI* __restrict__ in) {
  const ZFix F = fix[blockIdx.x];
  const int c = threadIdx.x;
  if (c < F.nk) in[F.zpos + c] = IO<TACC>::from_double(double(sum_parts(zpart + F.part + c, F.count, kZPart)));
}

// Phase 2, panels of at most 32 rows (leaves): lanes form 32 / mpad slices of
// mpad lanes (mpad = next power of two >= m), one lane per row; slice sl
// takes segments sl, sl + slices, ... of the item, each cut into pieces of at
// most cmax columns (a multiple of 16 bytes' worth of elements, so that every
// piece starts on a 16-byte boundary).  The warp runs in rounds: in round q
// every slice processes its q-th piece.  A piece (its m x c column-major
// block, rounded up to 16 bytes, and its input run, from the 16-byte boundary
// below to the one above) is staged in shared memory by bulk copies that the
// slice's first lane starts, kSStages rounds ahead; each round's mbarrier
// expects one arrival per slice.  Column j of a piece goes to accumulator
// j & 1; the slices are added by shuffles at the end.  For a BF16 dense tile
// the slice's lanes first multiply the staged inputs by the tile's column
// scales, in place (once per column rather than once per entry).
constexpr int kSWarps = 4;                     // warps per CTA of panel_small_kernel
constexpr int kSStages = HODLR_TUNE_S_STAGES;
constexpr int kSUBytes = HODLR_TUNE_S_BYTES;   // segment bytes per round (all slices)
// input bytes per round (all slices): twice as many for BF16, whose pieces
// hold more columns per byte of segment
template <typename TA>
__host__ __device__ constexpr int s_xbytes() { return sizeof(TA) == 2 ? 2 * kSUBytes : kSUBytes; }
template <typename TA>
__host__ __device__ constexpr int s_warp_smem() { return 64 + kSStages * (kSUBytes + s_xbytes<TA>()); }
// every slice's piece holds at least 16 bytes' worth of columns (cmax >= Q
// below) for any m <= 32 with these budgets
static_assert(kSUBytes >= 2048 && kSUBytes % 16 == 0, "leaf-panel stage too small");
static_assert(s_warp_smem<float>() % 16 == 0 && s_warp_smem<bf16>() % 16 == 0,
              "bulk copy destinations must stay 16-byte aligned");

template <typename TA, typename TACC>
__global__ void __launch_bounds__(kSWarps * 32, HODLR_TUNE_S_MINB)
    panel_small_kernel(const Panel* __restrict__ panels, const Seg* __restrict__ segs, const Item* __restrict__ items,
                       int nitems, const typename IO<TACC>::TI* __restrict__ in, typename IO<TACC>::TY* __restrict__ y,
                       typename IO<TACC>::TY* ypart) {
  using TX = typename IO<TACC>::TI;
  using TY = typename IO<TACC>::TY;
  using AC = Acc<TACC>;
  constexpr int esz = int(sizeof(TA));
  constexpr int Q = 16 / esz;  // piece columns are a multiple of Q
  constexpr int kSXBytes = s_xbytes<TA>(), kSWarpSmem = s_warp_smem<TA>();
  extern __shared__ __align__(16) unsigned char ssm[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * kSWarps + wid;
  if (w >= nitems) return;
  const Item it = items[w];
  const Panel P = panels[it.panel];
  const int m = P.m;
  const TX* inc = in;
  TY* yo = y + P.yoff;
  int mpad = 1;
  while (mpad < m) mpad <<= 1;
  const int slices = 32 / mpad;
  const int i = lane & (mpad - 1), sl = lane / mpad;
  // per slice and round: ub bytes of segment, xb bytes of inputs; a piece of
  // c columns needs c*m*esz + 15 and c*sizeof(TX) + 32 bytes at most
  const int ub = kSUBytes / slices, xb = kSXBytes / slices;
  const int cmax = min((ub - 15) / (m * esz), (xb - 32) / int(sizeof(TX))) / Q * Q;  // >= Q: ub, xb >= 64 mpad
  unsigned char* base = ssm + wid * kSWarpSmem;
  uint64_t* bar = reinterpret_cast<uint64_t*>(base);
  unsigned char* stage0 = base + 64;
  // rounds = the largest piece count over the slices
  int npieces = 0;
  for (int64_t q = it.seg_b + sl; q < it.seg_e; q += slices) npieces += (segs[q].K + cmax - 1) / cmax;
  int rounds = npieces;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rounds = max(rounds, __shfl_xor_sync(0xffffffffu, rounds, o));
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < kSStages; s++) mbar_init(bar + s, uint32_t(slices));
    fence_mbar_init();
  }
  __syncwarp();

  int64_t ps = it.seg_b + sl;  // producer cursor of this slice (used by its first lane)
  int pc = 0;
#define HODLR_SMALL_ISSUE(q_)                                                                                   \
  do {                                                                                                          \
    if (i != 0) break;                                                                                          \
    const int st_ = (q_) % kSStages;                                                                            \
    if (ps >= it.seg_e) {                                                                                       \
      mbar_arrive(bar + st_);                                                                                   \
      break;                                                                                                    \
    }                                                                                                           \
    const Seg S_ = segs[ps];                                                                                    \
    const int c_ = min(cmax, S_.K - pc);                                                                        \
    unsigned char* su_ = stage0 + st_ * (kSUBytes + kSXBytes) + sl * ub;                                        \
    unsigned char* sx_ = stage0 + st_ * (kSUBytes + kSXBytes) + kSUBytes + sl * xb;                             \
    /* pc is a multiple of Q, so the piece starts 16-byte aligned; the rounded                                 \
       size stays inside the block's storage (padded to 16 bytes) */                                            \
    const TA* A_ = static_cast<const TA*>(S_.A) + int64_t(pc) * m;                                              \
    const uint32_t bu_ = uint32_t((c_ * m * esz + 15) & ~15);                                                   \
    const unsigned char* xs_ = reinterpret_cast<const unsigned char*>(inc + S_.in_off + pc);                    \
    const unsigned char* xa_ = static_cast<const unsigned char*>(align_down16(xs_));                            \
    const uint32_t bx_ = uint32_t((xs_ + size_t(c_) * sizeof(TX) - xa_ + 15) & ~size_t(15));                    \
    fence_proxy_async();                                                                                        \
    mbar_expect_tx(bar + st_, bu_ + bx_);                                                                       \
    bulk_g2s(su_, A_, bu_, bar + st_);                                                                          \
    bulk_g2s(sx_, xa_, bx_, bar + st_);                                                                         \
    pc += c_;                                                                                                   \
    if (pc >= S_.K) {                                                                                           \
      ps += slices;                                                                                             \
      pc = 0;                                                                                                   \
    }                                                                                                           \
  } while (0)
  for (int q = 0; q < min(kSStages, rounds); q++) HODLR_SMALL_ISSUE(q);
  typename AC::A a0 = AC::zero(), a1 = AC::zero();
  int64_t cs = it.seg_b + sl;  // consumer cursor
  int cc = 0;
  for (int q = 0; q < rounds; q++) {
    const int st = q % kSStages;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(bar + st, uint32_t(q / kSStages) & 1u));
    if (!ok) {
      if (lane == 0) atomicAdd(&g_stream_timeouts, 1u);
      for (int t = q; t < min(q + kSStages, rounds); t++) mbar_wait(bar + t % kSStages, uint32_t(t / kSStages) & 1u);
      return;
    }
    if constexpr (sizeof(TA) == 2) {
      // BF16 dense tile: the slice's lanes multiply the staged inputs by the
      // column scales once, in place, before the products
      if (cs < it.seg_e) {
        const Seg S = segs[cs];
        if (S.cscale) {
          const int c = min(cmax, S.K - cc);
          const int xo = int((reinterpret_cast<uintptr_t>(inc + S.in_off + cc) & 15u) / sizeof(TX));
          TX* sx = reinterpret_cast<TX*>(stage0 + st * (kSUBytes + kSXBytes) + kSUBytes + sl * xb) + xo;
          for (int j = i; j < c; j += mpad) sx[j] = x_pair<TACC>(seg_in<TACC>(sx[j], S.cscale, cc + j));
        }
      }
      __syncwarp();
    }
    if (cs < it.seg_e) {
      const Seg S = segs[cs];
      const int c = min(cmax, S.K - cc);
      const TA* su = reinterpret_cast<const TA*>(stage0 + st * (kSUBytes + kSXBytes) + sl * ub);
      const int xo = int((reinterpret_cast<uintptr_t>(inc + S.in_off + cc) & 15u) / sizeof(TX));
      const TX* sx = reinterpret_cast<const TX*>(stage0 + st * (kSUBytes + kSXBytes) + kSUBytes + sl * xb) + xo;
      if (i < m) {
        int j = 0;
        for (; j + 1 < c; j += 2) {
          AC::fma(a0, su[j * m + i], AC::in(sx[j]));
          AC::fma(a1, su[(j + 1) * m + i], AC::in(sx[j + 1]));
        }
        if (j < c) AC::fma(a0, su[j * m + i], AC::in(sx[j]));
      }
      cc += c;
      if (cc >= S.K) {
        cs += slices;
        cc = 0;
      }
    }
    __syncwarp();  // round q's stage is refilled for round q + kSStages
    if (q + kSStages < rounds) HODLR_SMALL_ISSUE(q + kSStages);
  }
#undef HODLR_SMALL_ISSUE
  typename AC::A acc = AC::add(a0, a1);
  for (int o = mpad; o < 32; o <<= 1) acc = AC::add(acc, AC::shfl_xor(acc, o));
  // a panel whose columns are split over several items: partial rows at
  // ypart[part * tile_rows], added in part order by panel_fix_kernel
  if (sl == 0 && i < m) {
    if (it.part < 0)
      yo[i] = TY(AC::value(acc));
    else
      ypart[int64_t(it.part) * tile_rows(int(sizeof(TA))) + i] = TY(AC::value(acc));
  }
}

// Phase 2, panels of at most 32 rows, when the segments of every item lie
// in memory in segment order (the far field after its relayout in panel
// order, the near field as assembled).  All segments of a panel have its m
// rows, so an item's factors form one run of m-row columns (after each
// segment up to 15 bytes of padding, and for a BF16 dense tile its column
// scales).  The run is streamed through a per-warp ring of kLStages stages;
// a stage is the bytes of a run of whole columns -- at most l_bytes, at
// most l_cols columns -- fetched by ONE bulk copy (from the 16-byte boundary
// at or below its first column), and the input values of those columns,
// gathered into the stage by the lanes with 4- or 8-byte asynchronous copies
// (cp.async) that complete on the stage's mbarrier.  Relaxed products read
// only the high part of a split input, so only that part is staged.  Both
// are issued kLStages - 1 stages ahead of the products, so neither the
// factor bytes nor the scattered inputs (read from L2: x and z are small)
// are waited for in the loop.
//
// The warp plans each stage together: lane k reads the record of the k-th
// next segment (one coalesced load per 32 segments; the first 32 of each
// plan are loaded one stage ahead), a warp scan places each segment's
// columns in the stage, and every lane then fills the stage's column table
// (the element offset of each column in the stage buffer) and starts the
// gathers of columns lane, lane + 32, ... (for BF16 dense tiles also the
// gathers of their column scales).  After the wait the lanes multiply the
// staged inputs of BF16 dense tiles by their scales, once per column.  The
// products then read only shared memory, whose reads bound this kernel (a
// factor entry, an input of 8 bytes and a column offset are four clocks of an
// SM's shared memory against three of FP32 operations when a lane has one row):
// a lane has two rows, L = ceil(m / 2) lanes make up a slice, and slice sl of S =
// 32 / L (not a power of two: 17 rows fill 27 lanes, where one row per lane in
// slices of a power of two left 15 of 32 idle) takes the stage's columns sl,
// sl + S, ...  4D N = 65536 BF16: 412 -> 316 us, 3D N = 262144 FP32: 407 -> 342,
// its FP64 near field 138 -> 127.
#ifndef HODLR_TUNE_L_STAGES
#define HODLR_TUNE_L_STAGES 2
#endif
constexpr int kLWarps = 4;
constexpr int kLStages = HODLR_TUNE_L_STAGES;
// factor bytes and columns per stage at most, CTAs per SM to compile for: BF16
// columns are half as long, and with smaller stages a sixth CTA fits (4D N =
// 65536: 340 -> 315 us); FP32 and FP64 columns would fill them too early (3D N =
// 262144 FP32: 344 -> 360 us)
#ifndef HODLR_TUNE_L_BYTES  // 0: by type, as below
#define HODLR_TUNE_L_BYTES 0
#endif
#ifndef HODLR_TUNE_L_COLS
#define HODLR_TUNE_L_COLS 0
#endif
#ifndef HODLR_TUNE_L_MINB
#define HODLR_TUNE_L_MINB 0
#endif
template <typename TA>
inline constexpr int l_bytes = HODLR_TUNE_L_BYTES ? HODLR_TUNE_L_BYTES : sizeof(TA) == 2 ? 3072 : 4096;
template <typename TA>
inline constexpr int l_cols = HODLR_TUNE_L_COLS ? HODLR_TUNE_L_COLS : sizeof(TA) == 2 ? 96 : 128;
template <typename TA>
inline constexpr int l_minb = HODLR_TUNE_L_MINB ? HODLR_TUNE_L_MINB : sizeof(TA) == 2 ? 6 : 5;
constexpr int kLHead = 64;                        // barriers and stage descriptors
static_assert(kLStages >= 2 && kLStages <= 4, "leaf ring: 2 to 4 stages");
static_assert(32 + kLStages * 8 <= kLHead, "leaf ring header too small");
// The staged input of one column: the input element, or for relaxed products
// (which read only the high part of a split input) that high part alone.
template <typename TACC>
struct LeafX {
  using T = typename IO<TACC>::TI;
};
template <>
struct LeafX<FH> {
  using T = float;
};
// An input after scaling, in its staged form.
__device__ __forceinline__ void put_staged(float2& d, DF x) { d = make_float2(x.hi, x.lo); }
__device__ __forceinline__ void put_staged(float& d, float x) { d = x; }
// stage: factor bytes | inputs (kCols x TX) | column offsets (kCols x u16) | BF16 scales (kCols x f32)
template <typename TA, typename TX>
__host__ __device__ constexpr int l_stage_smem() {
  return l_bytes<TA> + l_cols<TA> * (int(sizeof(TX)) + 2 + (sizeof(TA) == 2 ? 4 : 0));
}
template <typename TA, typename TX>
__host__ __device__ constexpr int l_warp_smem() { return kLHead + kLStages * l_stage_smem<TA, TX>(); }

__device__ __forceinline__ void cp_async_gather(void* dst, const void* src, int bytes) {
  if (bytes == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
// the stage's mbarrier also waits for this thread's earlier cp.async copies
// (its pending count is raised now and lowered when they land)
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.shared.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Two elements next to each other in shared memory; EVEN: one load (the first one
// is aligned for it).
template <bool EVEN>
__device__ __forceinline__ void load_two(const float* p, float& a, float& b) {
  if constexpr (EVEN) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    a = v.x, b = v.y;
  } else {
    a = p[0], b = p[1];
  }
}
template <bool EVEN>
__device__ __forceinline__ void load_two(const double* p, double& a, double& b) {
  if constexpr (EVEN) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    a = v.x, b = v.y;
  } else {
    a = p[0], b = p[1];
  }
}
template <bool EVEN>
__device__ __forceinline__ void load_two(const bf16* p, float& a, float& b) {
  if constexpr (EVEN) {
    const uint32_t v = *reinterpret_cast<const uint32_t*>(p);
    a = __uint_as_float(v << 16), b = __uint_as_float(v & 0xffff0000u);
  } else {
    a = bf2f(p[0].b), b = bf2f(p[1].b);
  }
}

// The products of one staged stage for one lane (two rows of slice sl, su: the
// first of them in column 0): columns sl, sl + S, sl + 2 S, ... of the stage.
template <bool EVEN, typename TA, typename TX, typename TACC>
__device__ __forceinline__ void leaf_products(const TA* __restrict__ su, const TX* __restrict__ xs,
                                              const uint16_t* __restrict__ co, int C, int sl, int S,
                                              typename Acc<TACC>::A& a0, typename Acc<TACC>::A& a1) {
  using AC = Acc<TACC>;
  using V = std::conditional_t<sizeof(TA) == 8, double, float>;
  const TX* px = xs + sl;
  const uint16_t* pc = co + sl;
  int c = sl;
  for (; c + S < C; c += 2 * S, px += 2 * S, pc += 2 * S) {
    V v0, v1, w0, w1;
    load_two<EVEN>(su + pc[0], v0, v1);
    load_two<EVEN>(su + pc[S], w0, w1);
    const typename AC::X x = AC::in(px[0]), y = AC::in(px[S]);
    fma_pair<TACC>(a0, a1, v0, v1, x, x);
    fma_pair<TACC>(a0, a1, w0, w1, y, y);
  }
  if (c < C) {
    V v0, v1;
    load_two<EVEN>(su + pc[0], v0, v1);
    const typename AC::X x = AC::in(px[0]);
    fma_pair<TACC>(a0, a1, v0, v1, x, x);
  }
}

template <typename TA, typename TACC>
__global__ void __launch_bounds__(kLWarps * 32, l_minb<TA>)
    panel_leaf_kernel(const Panel* __restrict__ panels, const Seg* __restrict__ segs, const Item* __restrict__ items,
                      int nitems, const typename IO<TACC>::TI* __restrict__ in, typename IO<TACC>::TY* __restrict__ y,
                      typename IO<TACC>::TY* ypart) {
  using TI = typename IO<TACC>::TI;
  using TX = typename LeafX<TACC>::T;
  using TY = typename IO<TACC>::TY;
  using AC = Acc<TACC>;
  constexpr int esz = int(sizeof(TA));
  constexpr bool kScaled = esz == 2;
  constexpr int kStage = l_stage_smem<TA, TX>(), kWarpSmem = l_warp_smem<TA, TX>();
  constexpr int kLStageBytes = l_bytes<TA>, kLCols = l_cols<TA>;
  constexpr int kXOff = kLStageBytes, kOOff = kXOff + kLCols * int(sizeof(TX)), kSOff = kOOff + kLCols * 2;
  extern __shared__ __align__(16) unsigned char lsm[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * kLWarps + wid;
  if (w >= nitems) return;
  const Item it = items[w];
  const Panel P = panels[it.panel];
  const int m = P.m;
  const int colb = m * esz;  // bytes per column
  const TI* inc = in;
  TY* yo = y + P.yoff;
  // L lanes of two rows each per slice; the lanes beyond S L have no work
  const int L = (m + 1) >> 1, S = 32 / L;
  const int sl = lane / L, i = 2 * (lane - sl * L);
  unsigned char* base = lsm + wid * kWarpSmem;
  uint64_t* bar = reinterpret_cast<uint64_t*>(base);
  int2* meta = reinterpret_cast<int2*>(base + 32);  // per stage: column count, unused
  unsigned char* ring = base + kLHead;
  const int32_t qe = it.seg_e;
  const char* a0 = static_cast<const char*>(segs[it.seg_b].A);  // 16-byte aligned: every segment starts on 16 bytes
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < kLStages; s++) mbar_init(bar + s, 1u);
    fence_mbar_init();
  }
  __syncwarp();

  // next column to stage (the same in every lane): segment pq, column pj
  int32_t pq = it.seg_b, pj = 0;
  // lane k's record of segment rq + k, loaded a stage ahead of its use (the
  // first window of the next plan), so that its latency overlaps the products
  int32_t rq = -1, rK = 0, rso = 0;
  int64_t rino = 0;
  const float* rcs = nullptr;
  auto prefetch = [&]() {
    rq = pq;
    rK = 0;
    rso = 0;
    rino = 0;
    rcs = nullptr;
    if (pq + lane < qe) {
      const Seg S = segs[pq + lane];
      rK = S.K;
      rso = int32_t(static_cast<const char*>(S.A) - a0);
      rino = S.in_off;
      rcs = S.cscale;
    }
  };
  // Plans the stage from (pq, pj) into slot st and issues its copies; false
  // when every column is staged.  Warp-uniform.
  auto issue = [&](int st) -> bool {
    if (pq >= qe) return false;
    unsigned char* su = ring + st * kStage;
    TX* xs = reinterpret_cast<TX*>(su + kXOff);
    uint16_t* co = reinterpret_cast<uint16_t*>(su + kOOff);
    float* sc = reinterpret_cast<float*>(su + kSOff);
    int32_t sbase = 0, cols = 0, end = 0;
    bool first = true, more = true;
    while (more) {
      // lane k: segment pq + k, its first column to stage (pj for k = 0)
      const int32_t q = pq + lane;
      int32_t K = 0, so = 0;
      int64_t ino = 0;
      const float* cs = nullptr;
      if (pq == rq) {  // warp-uniform
        K = rK;
        so = rso;
        ino = rino;
        cs = rcs;
      } else if (q < qe) {
        const Seg S = segs[q];
        K = S.K;
        so = int32_t(static_cast<const char*>(S.A) - a0);
        ino = S.in_off;
        cs = S.cscale;
      }
      const int32_t j0 = lane == 0 ? pj : 0;
      const int32_t avail = max(K - j0, 0);
      if (first) sbase = (__shfl_sync(0xffffffffu, so + j0 * colb, 0)) & ~15;
      first = false;
      // columns of this segment whose end stays within the stage's bytes
      const int32_t room = sbase + kLStageBytes - so;
      int32_t fit = room >= colb * (j0 + 1) ? room / colb - j0 : 0;
      int32_t take = min(avail, fit);
      // segments after the first one that is not taken whole take nothing
      const unsigned part = __ballot_sync(0xffffffffu, take < avail || q >= qe);
      const int stop_at = part ? __ffs(part) - 1 : 32;  // first lane not taken whole
      if (lane > stop_at) take = 0;
      // the column cap: exclusive prefix sum of the takes
      int32_t pre = take;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t v = __shfl_up_sync(0xffffffffu, pre, o);
        if (lane >= o) pre += v;
      }
      pre -= take;
      take = max(0, min(take, kLCols - cols - pre));
      // column table and gathers for this window: the taken columns in order
      int32_t incl = pre + take;  // columns before the end of this lane's share
      const int32_t total = __shfl_sync(0xffffffffu, incl, 31);
      const int32_t wcols = min(total, kLCols - cols);
      for (int c0 = 0; c0 < wcols; c0 += 32) {  // every lane takes part in the shuffles
        const int c = c0 + lane;
        // the lane k whose share holds column c: the shares with columns are
        // those of lanes 0, 1, ... in column order, so k is the number of
        // shares starting before column c0, plus the shares starting in
        // c0 .. c, minus one (one warp vote and one OR-reduction of the
        // share starts, no search)
        const bool owns = take > 0;
        const int k0 = __popc(__ballot_sync(0xffffffffu, owns && pre < c0));
        const uint32_t starts =
            __reduce_or_sync(0xffffffffu, owns && pre >= c0 && pre < c0 + 32 ? 1u << (pre - c0) : 0u);
        const int k = k0 - 1 + __popc(starts & (0xffffffffu >> (31 - lane)));
        const int32_t pk = __shfl_sync(0xffffffffu, pre, k);
        const int32_t jk = __shfl_sync(0xffffffffu, j0, k) + (c - pk);
        const int32_t sok = __shfl_sync(0xffffffffu, so, k);
        const int64_t ink = __shfl_sync(0xffffffffu, ino, k);
        unsigned long long csk = 0;
        if constexpr (kScaled) csk = __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(cs), k);
        if (c < wcols) {
          co[cols + c] = uint16_t((sok + jk * colb - sbase) / esz);
          // relaxed products stage only the high part (the first member) of a split input
          cp_async_gather(xs + cols + c, reinterpret_cast<const TX*>(inc + ink + jk), int(sizeof(TX)));
          if constexpr (kScaled) {
            if (csk)
              cp_async_gather(sc + cols + c, reinterpret_cast<const float*>(csk) + jk, 4);
            else
              sc[cols + c] = 1.f;
          }
        }
      }
      // the last lane with columns ends the stage's bytes and moves the cursor
      const unsigned has = __ballot_sync(0xffffffffu, take > 0);
      if (has) {
        const int kl = 31 - __clz(has);
        const int32_t e = __shfl_sync(0xffffffffu, so + (j0 + take) * colb, kl);
        const int32_t tk = __shfl_sync(0xffffffffu, take, kl), ak = __shfl_sync(0xffffffffu, avail, kl);
        const int32_t jl = __shfl_sync(0xffffffffu, j0, kl);
        end = e;
        if (tk < ak) {
          pq += kl;
          pj = jl + tk;
        } else {
          pq += kl + 1;
          pj = 0;
        }
      }
      cols += wcols;
      // another window of 32 segments only when all 32 were taken whole
      more = has == 0xffffffffu && stop_at == 32 && cols < kLCols && pq < qe;
    }
    cp_async_arrive(bar + st);
    if (lane == 0) meta[st] = make_int2(cols, 0);
    __syncwarp();
    if (lane == 0) {
      // end rounded up to 16 bytes stays inside the last segment's storage
      // (every segment occupies a multiple of 16 bytes), and end - sbase <= kLStageBytes
      const uint32_t bytes = uint32_t(((end + 15) & ~15) - sbase);
      fence_proxy_async();
      mbar_expect_tx(bar + st, bytes);
      bulk_g2s(su, a0 + sbase, bytes, bar + st);
    }
    return true;
  };

  int nissued = 0;
  prefetch();
  for (int s = 0; s < kLStages; s++) {
    if (!issue(s)) break;
    nissued++;
    prefetch();
  }
  typename AC::A a0acc = AC::zero(), a1acc = AC::zero();
  for (int k = 0; k < nissued; k++) {
    const int st = k % kLStages;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(bar + st, uint32_t(k / kLStages) & 1u));
    if (!ok) {
      if (lane == 0) atomicAdd(&g_stream_timeouts, 1u);
      for (int t = k; t < nissued; t++) mbar_wait(bar + t % kLStages, uint32_t(t / kLStages) & 1u);
      cp_async_wait_all();
      return;
    }
    const int C = meta[st].x;
    const unsigned char* sb = ring + st * kStage;
    const TA* su = reinterpret_cast<const TA*>(sb);
    const TX* xs = reinterpret_cast<const TX*>(sb + kXOff);
    const uint16_t* co = reinterpret_cast<const uint16_t*>(sb + kOOff);
    const float* sc = reinterpret_cast<const float*>(sb + kSOff);
    if constexpr (kScaled) {
      // BF16: the staged inputs times their column scales, once per column
      // (lane c % 32 gathered column c and scales it), before the products
      TX* xw = const_cast<TX*>(xs);
      for (int c = lane; c < C; c += 32) put_staged(xw[c], AC::xscale(AC::in(xw[c]), sc[c]));
      __syncwarp();
    }
    // an even row count keeps every pair of rows aligned; of an odd one the last
    // lane's second row is whatever follows the column and is not stored
    if (sl < S) {
      if (m & 1)
        leaf_products<false, TA, TX, TACC>(su + i, xs, co, C, sl, S, a0acc, a1acc);
      else
        leaf_products<true, TA, TX, TACC>(su + i, xs, co, C, sl, S, a0acc, a1acc);
    }
    __syncwarp();  // stage k's slot is refilled for stage k + kLStages
    if (issue(st)) {
      nissued++;
      prefetch();
    }
  }
  // slices in pairs, in an order that depends on S alone
  for (int n = S; n > 1;) {
    const int half = (n + 1) >> 1;
    const typename AC::A o0 = AC::shfl_down(a0acc, half * L), o1 = AC::shfl_down(a1acc, half * L);
    if (sl + half < n) {
      a0acc = AC::add(a0acc, o0);
      a1acc = AC::add(a1acc, o1);
    }
    n = half;
  }
  if (sl == 0) {
    TY* dst = it.part < 0 ? yo + i : ypart + int64_t(it.part) * tile_rows(int(sizeof(TA))) + i;
    dst[0] = TY(AC::value(a0acc));
    if (i + 1 < m) dst[1] = TY(AC::value(a1acc));
  }
}

// Phase 2, panels of more than 32 rows: item chunk = row tile t of the
// panel (T = 512 / sizeof(TA) rows; a lane owns RPL = 16 / sizeof(TA) rows
// t*T + g*RPL ..).  A tile of rows <= 16 RPL rows needs fewer than 32 lanes
// per column: the warp then splits into slices of L lanes (L = the row
// groups rounded up to a power of two), slice sl taking the columns
// j = sl (mod 32 / L) of each segment, so that every lane has work (a
// 64-row BF16 tile keeps 8 lanes per column and 4 columns in flight).  Every
// segment's tile is h x K, column major with column stride h (h = the tile's
// row count rounded up to height_quantum rows), so a run of its columns is one contiguous byte
// range, and so is the run of their input values.  Both are staged through a
// per-warp ring of kPStages shared-memory stages by bulk copies, at most
// kPStageBytes of tile and kPCols columns per stage.  Within one stage a
// slice's k-th column goes to accumulator set k & 1; the slices' sums are
// added by shuffles at the end.  BF16 dense tiles: the warp multiplies the
// staged inputs by the column scales first, once, in place.
constexpr int kPWarps = 4;           // warps per CTA of panel_tile_kernel
constexpr int kPStages = HODLR_TUNE_P_STAGES;
constexpr int kPStageBytes = HODLR_TUNE_P_BYTES;
constexpr int kPCols = 64;           // columns per stage at most
constexpr int kPXBytes = kPCols * 8 + 32;
constexpr int kPWarpSmem = 64 + kPStages * (kPStageBytes + kPXBytes);
static_assert(kPWarpSmem % 16 == 0 && kPXBytes % 16 == 0, "bulk copy destinations must stay 16-byte aligned");

// CTAs per SM the register allocation must allow: a sixth (80 registers) helps
// the four rows of a lane's FP32 load (3D N = 262144: 1020 -> 1001 us), not the
// eight of a BF16 one, whose sums alone take 32 (4D N = 65536: 135 -> 143 us)
#ifndef HODLR_TUNE_P_MINB  // 0: by type
#define HODLR_TUNE_P_MINB 0
#endif
template <typename TA>
inline constexpr int p_minb = HODLR_TUNE_P_MINB ? HODLR_TUNE_P_MINB : sizeof(TA) == 2 ? 4 : 6;
template <typename TA, typename TACC>
__global__ void __launch_bounds__(kPWarps * 32, p_minb<TA>)
    panel_tile_kernel(const Panel* __restrict__ panels, const Seg* __restrict__ segs, const Item* __restrict__ items,
                      int nitems, typename IO<TACC>::TY* __restrict__ ypart,
                      const typename IO<TACC>::TI* __restrict__ in, typename IO<TACC>::TY* __restrict__ y) {
  using TX = typename IO<TACC>::TI;
  using TY = typename IO<TACC>::TY;
  constexpr int RPL = 16 / int(sizeof(TA));
  constexpr int T = 32 * RPL;
  using VT = typename Vec16<TA>::type;
  using AC = Acc<TACC>;
  extern __shared__ __align__(16) unsigned char psm[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * kPWarps + wid;
  if (w >= nitems) return;
  const Item it = items[w];
  const Panel P = panels[it.panel];
  const int m = P.m;
  const TX* inc = in;
  const int t = it.chunk;
  const int rows = min(T, m - t * T);
  const int64_t h = tile_height(m, t, int(sizeof(TA)));
  const int colb = int(h) * int(sizeof(TA));  // bytes per tile column: 16 .. 512, a multiple of 16
  const int cps = min(kPCols, kPStageBytes / colb);
  int lg = 1;  // lanes per slice
  while (lg * RPL < rows) lg <<= 1;
  const int slices = 32 / lg;
  const int g = lane & (lg - 1), sl = lane / lg;
  const bool act = g * RPL < rows;
  typename AC::A a0[RPL], a1[RPL];
#pragma unroll
  for (int q = 0; q < RPL; q++) a0[q] = a1[q] = AC::zero();

  unsigned char* base = psm + wid * kPWarpSmem;
  uint64_t* bar = reinterpret_cast<uint64_t*>(base);
  unsigned char* ubuf = base + 64;
  unsigned char* xbuf = ubuf + kPStages * kPStageBytes;
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < kPStages; s++) mbar_init(bar + s, 1);
    fence_mbar_init();
  }
  __syncwarp();
  // producer cursor (segment, first column); every lane keeps it, lane 0 issues
  int64_t ps = it.seg_b;
  int pc = 0, issued = 0;
#define HODLR_PANEL_ISSUE_NEXT()                                                                                  \
  do {                                                                                                            \
    while (ps < it.seg_e && pc >= segs[ps].K) {                                                                   \
      ps++;                                                                                                       \
      pc = 0;                                                                                                     \
    }                                                                                                             \
    if (ps >= it.seg_e) break;                                                                                    \
    const Seg S_ = segs[ps];                                                                                      \
    const int nc_ = min(cps, S_.K - pc);                                                                          \
    if (lane == 0) {                                                                                              \
      const int st_ = issued % kPStages;                                                                          \
      /* U tile t starts at element t*T*K: 16-byte aligned since T * sizeof(TA) = 512 */                          \
      const TA* src_ = static_cast<const TA*>(S_.A) + int64_t(t) * T * S_.K + int64_t(pc) * h;                    \
      const uint32_t ub_ = uint32_t(nc_) * uint32_t(colb);                                                        \
      const unsigned char* xs_ = reinterpret_cast<const unsigned char*>(inc + S_.in_off + pc);                    \
      const unsigned char* xa_ = static_cast<const unsigned char*>(align_down16(xs_));                            \
      const uint32_t xb_ = uint32_t((xs_ + size_t(nc_) * sizeof(TX) - xa_ + 15) & ~size_t(15));                   \
      fence_proxy_async();                                                                                        \
      mbar_expect_tx(bar + st_, ub_ + xb_);                                                                       \
      bulk_g2s(ubuf + st_ * kPStageBytes, src_, ub_, bar + st_);                                                  \
      bulk_g2s(xbuf + st_ * kPXBytes, xa_, xb_, bar + st_);                                                       \
    }                                                                                                             \
    pc += nc_;                                                                                                    \
    issued++;                                                                                                     \
  } while (0)
  for (int q = 0; q < kPStages; q++) HODLR_PANEL_ISSUE_NEXT();
  // consumer cursor
  int64_t cs = it.seg_b;
  int cc = 0;
  for (int q = 0; q < issued; q++) {
    while (cc >= segs[cs].K) {
      cs++;
      cc = 0;
    }
    const Seg S = segs[cs];
    const int nc = min(cps, S.K - cc);
    const int st = q % kPStages;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(bar + st, uint32_t(q / kPStages) & 1u));
    if (!ok) {
      if (lane == 0) atomicAdd(&g_stream_timeouts, 1u);
      for (int u = q; u < issued; u++) mbar_wait(bar + u % kPStages, uint32_t(u / kPStages) & 1u);
      return;
    }
    const int xo = int((reinterpret_cast<uintptr_t>(inc + S.in_off + cc) & 15u) / sizeof(TX));
    const TX* xsm = reinterpret_cast<const TX*>(xbuf + st * kPXBytes) + xo;
    const unsigned char* us = ubuf + st * kPStageBytes + g * 16;
    if constexpr (sizeof(TA) == 2) {
      // BF16 dense tile: the staged inputs times the column scales, once, in place
      if (S.cscale) {
        TX* xw = const_cast<TX*>(xsm);
        for (int j = lane; j < nc; j += 32) xw[j] = x_pair<TACC>(seg_in<TACC>(xw[j], S.cscale, cc + j));
        __syncwarp();
      }
    }
#define HODLR_XIN(j_) AC::in(xsm[j_])
    // this slice's columns of the stage: segment columns cc + j, j = sl (mod slices)
    int j = (sl - cc) & (slices - 1);
    for (; j + slices < nc; j += 2 * slices) {
      const VT v0 = act ? *reinterpret_cast<const VT*>(us + j * colb) : vzero<VT>();
      const VT v1 = act ? *reinterpret_cast<const VT*>(us + (j + slices) * colb) : vzero<VT>();
      axpy16<TACC>(v0, HODLR_XIN(j), a0);
      axpy16<TACC>(v1, HODLR_XIN(j + slices), a1);
    }
    if (j < nc) {
      const VT v0 = act ? *reinterpret_cast<const VT*>(us + j * colb) : vzero<VT>();
      axpy16<TACC>(v0, HODLR_XIN(j), a0);
    }
#undef HODLR_XIN
    cc += nc;
    __syncwarp();
    HODLR_PANEL_ISSUE_NEXT();  // the next run, if any, into the stage just consumed
  }
#undef HODLR_PANEL_ISSUE_NEXT
#pragma unroll
  for (int q = 0; q < RPL; q++) {
    a0[q] = AC::add(a0[q], a1[q]);
    for (int o = lg; o < 32; o <<= 1) a0[q] = AC::add(a0[q], AC::shfl_xor(a0[q], o));
  }
  if (act && sl == 0) {
    const int i = t * T + g * RPL;
    TY* dst = it.part < 0 ? y + P.yoff + i : ypart + int64_t(it.part) * T + g * RPL;
#pragma unroll
    for (int q = 0; q < RPL; q++)
      if (i + q < m) dst[q] = TY(AC::value(a0[q]));
  }
}

// Adds the partial row blocks of split panel chunks, in part order.
template <typename TX>
__global__ void __launch_bounds__(256) panel_fix_kernel(const Panel* __restrict__ panels,
                                                        const PanelFix* __restrict__ fix, int nfix, int rows,
                                                        const TX* __restrict__ ypart, TX* __restrict__ y) {
  const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int f = int(t / rows), q = int(t % rows);
  if (f >= nfix) return;
  const PanelFix F = fix[f];
  const Panel P = panels[F.panel];
  const int i = F.chunk * rows + q;
  if (i >= P.m) return;
  y[P.yoff + i] = sum_parts(ypart + int64_t(F.part) * rows + q, F.count, rows);
}

// ---- FP64 factors ------------------------------------------------------------
// z = V^T x and the panels are the same product: sums over columns j of
// A(i, j) x(j) for at most 64 rows i that lie together in memory (V is stored
// row major, so a column j of the product is a point's row of V).  GB300's
// FP64 pipe -- 2 multiply-adds per clock and SM, 4.9 TB/s of factors -- bounds
// it, so what matters is that no lane multiplies padding and that the pipe
// always has a warp ready.  8 lanes take a column, lane g rows g, g + 8, ...
// (R = ceil(rows / 8) of them: at most 7 idle lanes, where 16-byte loads with
// the next power of two of lanes idled up to half), and the warp's 4 slices of
// lanes take 4 consecutive columns; the slices are added by shuffles at the
// end.  Every kind of item goes into one launch (z items first, then the
// panels): in a small operator a launch lasts as long as its longest item, and
// one launch waits for one of them.
// One product with FP64 factors: 2D N = 2000 130 -> 77 us, 2D N = 10000 165 ->
// 94 us, 3D N = 30011 764 -> 606 us (0.37 G multiply-adds per ms, 60% of the
// pipe; the rest is leaf segments of 8 columns and less).
// Whether this warp, whose lanes have written their partial sums, is the last
// of `count` to finish on counter *cnt; the last one resets the counter.  (Used
// by the FP64 items only: in the staged kernels the wait for the partial sums'
// stores and the registers of the sums cost a large operator more than the two
// fix-up launches do -- 3D N = 262144 FP32 factors 2.82 -> 3.10 ms.)
__device__ __forceinline__ bool last_part(unsigned int* cnt, int count, int lane) {
  __threadfence();
  __syncwarp();
  int last = 0;
  if (lane == 0) {
    last = atomicAdd(cnt, 1u) == unsigned(count - 1);
    if (last) *cnt = 0u;
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return false;
  __threadfence();
  return true;
}

// The end of a split z item: the last one adds the parts into z.
__device__ __forceinline__ void z_fixup(const ZFix* __restrict__ fix, unsigned int* zcnt, int f, const double* zpart,
                                        double* in, int lane) {
  const ZFix F = fix[f];
  if (!last_part(zcnt + f, F.count, lane)) return;
  for (int c = lane; c < F.nk; c += 32) in[F.zpos + c] = sum_parts(zpart + F.part + c, F.count, kZPart);
}

// The end of a split panel item (rows rows from row0 of the panel, parts T rows apart).
__device__ __forceinline__ void panel_fixup(const PanelFix* __restrict__ fix, unsigned int* pcnt, int f,
                                            const double* ypart, double* y, int rows, int lane) {
  const PanelFix F = fix[f];
  if (!last_part(pcnt + f, F.count, lane)) return;
  for (int i = lane; i < rows; i += 32) y[i] = sum_parts(ypart + int64_t(F.part) * 64 + i, F.count, 64);
}

struct Items64 {
  const ZBlock* zb;
  const ZItem* zitems;
  int nz;
  const ZFix* zfix;
  unsigned int* zcnt;
  double* zpart;
  PanelItems L;
  double* ypart;
  double* in;
  double* y;
};

// acc[q] += sum_j A(g + 8 q, j) x(j), j = sl, sl + 4, ... < K; A points at row
// g of column 0; okl: row g + 8 (R - 1) exists.
template <int R>
__device__ __forceinline__ void cols64(const double* __restrict__ A, int64_t ld, const double* x, int K, bool okl,
                                       int sl, double (&acc)[R]) {
  constexpr int U = R <= 2 ? 4 : R <= 4 ? 2 : 1;  // columns in flight per slice
  for (int b = 0; b < K; b += 4 * U) {
    double v[U][R], xv[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (b + 4 * u < K) {  // warp-uniform
        const int j = b + 4 * u + sl;
        const bool in = j < K;
        xv[u] = in ? x[j] : 0.0;
        const double* Aj = A + int64_t(j) * ld;
#pragma unroll
        for (int q = 0; q < R; q++) v[u][q] = in && (q < R - 1 || okl) ? __ldg(Aj + 8 * q) : 0.0;
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (b + 4 * u < K) {
#pragma unroll
        for (int q = 0; q < R; q++) acc[q] += v[u][q] * xv[u];
      }
    }
  }
}

// acc[q] += sum_j A(g + 8 q, j) x(j) over this slice's own K columns (Km: the
// most of any slice).
template <int R>
__device__ __forceinline__ void segs64(const double* __restrict__ A, int64_t ld, const double* x, int K, int Km,
                                       bool okl, double (&acc)[R]) {
  constexpr int U = 4;
  for (int b = 0; b < Km; b += U) {
    double v[U][R], xv[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int j = b + u;
      const bool in = j < K;
      xv[u] = in ? x[j] : 0.0;
      const double* Aj = A + int64_t(j) * ld;
#pragma unroll
      for (int q = 0; q < R; q++) v[u][q] = in && (q < R - 1 || okl) ? __ldg(Aj + 8 * q) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (b + u < Km) {
#pragma unroll
        for (int q = 0; q < R; q++) acc[q] += v[u][q] * xv[u];
      }
  }
}

// One item: its segments' records one per lane (loaded 32 at a time), rows
// rows with column stride ld, the sums to dst[0 .. rows).  zA / zx / zK: the
// single segment of a z item (zA non-null).
template <int R>
__device__ __forceinline__ void item64(const Seg* __restrict__ segs, int32_t sb, int32_t se, int64_t tile_off,
                                       const double* zA, int64_t zx, int zK, int rows, int64_t ld, const double* in,
                                       double* dst, int lane) {
  const int g = lane & 7, sl = lane >> 3;
  const bool okl = g + 8 * (R - 1) < rows;
  double acc[R];
#pragma unroll
  for (int q = 0; q < R; q++) acc[q] = 0.0;
  if (zA) {
    cols64<R>(zA + g, ld, in + zx, zK, okl, sl, acc);
  } else {
    for (int32_t s0 = sb; s0 < se; s0 += 32) {
      const double* rA = nullptr;
      int64_t ro = 0;
      int rK = 0;
      if (s0 + lane < se) {
        const Seg S = segs[s0 + lane];
        rA = static_cast<const double*>(S.A) + tile_off * S.K;
        ro = S.in_off;
        rK = S.K;
      }
      const int n = min(32, se - s0);
      if constexpr (R <= 2) {
        // few rows, and columns of a leaf's few points: a segment for each
        // slice, so that four of them are in flight
        for (int k0 = 0; k0 < n; k0 += 4) {
          const int k = min(k0 + sl, n - 1);
          const double* A = reinterpret_cast<const double*>(
              __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(rA), k));
          const int64_t off = __shfl_sync(0xffffffffu, ro, k);
          int K = __shfl_sync(0xffffffffu, rK, k);
          if (k0 + sl >= n) K = 0;
          int Km = max(K, __shfl_xor_sync(0xffffffffu, K, 8));
          Km = max(Km, __shfl_xor_sync(0xffffffffu, Km, 16));
          segs64<R>(A + g, ld, in + off, K, Km, okl, acc);
        }
        continue;
      }
      for (int k = 0; k < n; k++) {
        const double* A = reinterpret_cast<const double*>(
            __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(rA), k));
        const int64_t off = __shfl_sync(0xffffffffu, ro, k);
        const int K = __shfl_sync(0xffffffffu, rK, k);
        cols64<R>(A + g, ld, in + off, K, okl, sl, acc);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < R; q++) {
    acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], 8);
    acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], 16);
  }
  if (sl == 0) {
#pragma unroll
    for (int q = 0; q < R; q++)
      if (q < R - 1 || okl) dst[g + 8 * q] = acc[q];
  }
}

__global__ void __launch_bounds__(kWarpsPerCta * 32, 4) items64_kernel(const Items64 a) {
  const int lane = threadIdx.x & 31;
  int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  int rows, part, fix;
  int32_t sb = 0, se = 0;
  int64_t tile_off = 0, ld, zx = 0;
  const double* zA = nullptr;
  int zK = 0;
  double *dst, *out;
  const bool isz = w < a.nz;
  if (isz) {
    const ZItem it = a.zitems[w];
    const ZBlock Z = a.zb[it.zb];
    rows = min(it.nk, Z.r - it.k0);  // without the padding columns of V's rows
    ld = vpad(Z.r, 8);
    zA = static_cast<const double*>(Z.V) + int64_t(it.j0) * ld + it.k0;
    zx = Z.x_off + it.j0;
    zK = it.j1 - it.j0;
    part = it.part;
    fix = it.fix;
    out = a.in + Z.z_off + it.k0;
    dst = part < 0 ? out : a.zpart + part;
  } else {
    w -= a.nz;
    if (w >= a.L.nbig + a.L.nsmall) return;
    const bool big = w < a.L.nbig;
    const Item it = big ? a.L.big[w] : a.L.small[w - a.L.nbig];
    const Panel P = a.L.panels[it.panel];
    constexpr int T = 64;  // tile_rows(8)
    const int t = big ? it.chunk : 0;
    rows = min(T, P.m - t * T);
    ld = P.m > 32 ? tile_height(P.m, t, 8) : P.m;
    tile_off = int64_t(t) * T;
    sb = it.seg_b;
    se = it.seg_e;
    part = it.part;
    fix = it.fix;
    out = a.y + P.yoff + t * T;
    dst = part < 0 ? out : a.ypart + int64_t(part) * T;
  }
#define HODLR_R64(r_)                                                              \
  case r_:                                                                         \
    item64<r_>(a.L.segs, sb, se, tile_off, zA, zx, zK, rows, ld, a.in, dst, lane); \
    break;
  switch ((rows + 7) / 8) {
    HODLR_R64(1)
    HODLR_R64(2)
    HODLR_R64(3)
    HODLR_R64(4)
    HODLR_R64(5)
    HODLR_R64(6)
    HODLR_R64(7)
    HODLR_R64(8)
    default:
      break;
  }
#undef HODLR_R64
  if (part < 0) return;
  if (isz)
    z_fixup(a.zfix, a.zcnt, fix, a.zpart, a.in, lane);
  else
    panel_fixup(a.L.fix, a.L.pcnt, fix, a.ypart, out, rows, lane);
}

// Leaf panels of many tiny segments (PanelItems::plain), which latency bounds:
// slices of mpad lanes (the next power of two of the rows), a segment for each
// slice and a row for each lane, in so few registers that an SM holds twice the
// warps of items64_kernel.
__global__ void __launch_bounds__(kWarpsPerCta * 32)
    panel_small64_kernel(const PanelItems L, const double* __restrict__ in, double* __restrict__ ypart,
                         double* __restrict__ y) {
  const int w = blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= L.nplain) return;
  const Item it = L.plain[w];
  const Panel P = L.panels[it.panel];
  const int m = P.m;
  int mpad = 1;
  while (mpad < m) mpad <<= 1;
  const int slices = 32 / mpad;
  const int i = lane & (mpad - 1), sl = lane / mpad;
  double a0 = 0.0, a1 = 0.0;
  if (i < m) {
    for (int64_t s = it.seg_b + sl; s < it.seg_e; s += slices) {
      const Seg S = L.segs[s];
      const double* A = static_cast<const double*>(S.A) + i;
      const double* x = in + S.in_off;
      int j = 0;
      for (; j + 3 < S.K; j += 4) {
        const double v0 = __ldg(A + int64_t(j) * m), v1 = __ldg(A + int64_t(j + 1) * m);
        const double v2 = __ldg(A + int64_t(j + 2) * m), v3 = __ldg(A + int64_t(j + 3) * m);
        const double x0 = x[j], x1 = x[j + 1], x2 = x[j + 2], x3 = x[j + 3];
        a0 += v0 * x0;
        a1 += v1 * x1;
        a0 += v2 * x2;
        a1 += v3 * x3;
      }
      for (; j < S.K; j++) a0 += __ldg(A + int64_t(j) * m) * x[j];
    }
  }
  double acc = a0 + a1;
  for (int o = mpad; o < 32; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  double* out = y + P.yoff;
  if (sl == 0 && i < m) (it.part < 0 ? out : ypart + int64_t(it.part) * 64)[i] = acc;
  if (it.part >= 0) panel_fixup(L.fix, L.pcnt, it.fix, ypart, out, m, lane);
}

template <typename TX, typename TO>
__global__ void combine_kernel(const TX* __restrict__ y, int64_t ld_y, int nslots, int64_t n,
                               const int64_t* __restrict__ perm, TO* __restrict__ out, int64_t ld_out) {
  const int c = blockIdx.y;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const TX* yc = y + int64_t(c) * nslots * ld_y + i;
    double acc = double(yc[0]);
    for (int s = 1; s < nslots; s++) acc += double(yc[int64_t(s) * ld_y]);
    out[(perm ? perm[i] : i) + c * ld_out] = TO(acc);
  }
}

template <typename TS, typename TD>
__global__ void gather_kernel(const TS* __restrict__ src, int64_t ld_src, const int64_t* __restrict__ perm, int64_t n,
                              TD* __restrict__ dst, int64_t ld_dst) {
  const int c = blockIdx.y;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    dst[i + c * ld_dst] = TD(src[(perm ? perm[i] : i) + c * ld_src]);
}

template <int D, typename TO>
__global__ void __launch_bounds__(256) assemble_kernel(PointsDev P, KernelDev K, const TileDesc* __restrict__ tiles,
                                                       int ntiles, TO* __restrict__ out) {
  const int w = blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= ntiles) return;
  const TileDesc T = tiles[w];
  TO* o = out + T.off;
  const int64_t total = int64_t(T.m) * T.n;
  for (int64_t e = lane; e < total; e += 32) {
    const int i = int(e % T.m), j = int(e / T.m);
    double xi[D];
    load_point<D>(P, T.t_begin + i, xi);
    o[elem_offset(i, j, T.m, T.n, int(sizeof(TO)))] = TO(kernel_entry<D>(P, K, T.t_begin + i, T.s_begin + j, xi));
  }
}

template <int D, typename TO>
__global__ void __launch_bounds__(256) compact_kernel(PointsDev P, KernelDev K, const double* __restrict__ ws,
                                                      const int32_t* __restrict__ lmap,
                                                      const CompactDesc* __restrict__ blocks, int nblocks) {
  const CompactDesc B = blocks[blockIdx.x];
  TO* u = static_cast<TO*>(B.u_dst);
  double* u64 = static_cast<double*>(B.u64_dst);  // the FP64 copy too, when asked for
  constexpr int esz = int(sizeof(TO));
  if (B.kscale != 0.0) K.scale = B.kscale;
  if (B.dense) {
    const int64_t total = int64_t(B.m) * B.n;
    for (int64_t e = threadIdx.x; e < total; e += blockDim.x) {
      const int i = int(e % B.m), j = int(e / B.m);
      double xi[D];
      load_point<D>(P, B.t_begin + i, xi);
      const double a = kernel_entry<D>(P, K, B.t_begin + i, B.s_begin + j, xi);
      u[elem_offset(i, j, B.m, B.n, esz)] = TO(a);
      if (u64) u64[elem_offset(i, j, B.m, B.n, 8)] = a;
    }
  } else {
    const double* U = ws + B.ws;
    const int64_t nu = int64_t(B.m) * B.rank;
    for (int64_t e = threadIdx.x; e < nu; e += blockDim.x) {
      const int i = int(e % B.m), k = int(e / B.m);
      const int64_t row = lmap[B.t_map + i] - B.t_begin;
      u[elem_offset(row, k, B.m, B.rank, esz)] = TO(U[e]);
      if (u64) u64[elem_offset(row, k, B.m, B.rank, 8)] = U[e];
    }
    // V follows U's full workspace (m x cap); stored row major, n x vpad(rank)
    const double* Vw = ws + B.ws + int64_t(B.m) * B.cap;
    TO* v = static_cast<TO*>(B.v_dst);
    double* v64 = static_cast<double*>(B.v64_dst);
    const int64_t rp = vpad(B.rank, esz), rp64 = vpad(B.rank, 8);
    const int64_t nv = int64_t(B.n) * B.rank;
    for (int64_t e = threadIdx.x; e < nv; e += blockDim.x) {
      const int j = int(e % B.n), k = int(e / B.n);
      const int64_t row = lmap[B.s_map + j] - B.s_begin;
      v[row * rp + k] = TO(Vw[e]);
      if (v64) v64[row * rp64 + k] = Vw[e];
    }
  }
}

// BF16 storage of the same blocks, every factor scaled per column.  A dense
// tile keeps, per column j, the FP32 scale c_j = max_i |A_ij| (in s_dst) and
// the BF16 entries A_ij / c_j (round to nearest even); a low-rank block keeps
// per column k the scales su_k = max_i |U_ik|, sv_k = max_j |V_jk| and
// U_ik / su_k, V_jk / sv_k in BF16, with su_k * sv_k (the scale of
// z_k = V_k^T x) in s_dst.  A zero column gets scale 1.  One warp per column.
__device__ __forceinline__ unsigned short to_bf16_bits(double v) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(float(v)));
}
__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <int D>
__global__ void __launch_bounds__(256) compact_bf16_kernel(PointsDev P, KernelDev K, const double* __restrict__ ws,
                                                           const int32_t* __restrict__ lmap,
                                                           const CompactDesc* __restrict__ blocks, int nblocks) {
  const CompactDesc B = blocks[blockIdx.x];
  unsigned short* u = static_cast<unsigned short*>(B.u_dst);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (B.kscale != 0.0) K.scale = B.kscale;
  if (B.dense) {
    for (int j = warp; j < B.n; j += nw) {
      double mx = 0.0;
      for (int i = lane; i < B.m; i += 32) {
        double xi[D];
        load_point<D>(P, B.t_begin + i, xi);
        mx = fmax(mx, fabs(kernel_entry<D>(P, K, B.t_begin + i, B.s_begin + j, xi)));
      }
      mx = warp_max(mx);
      const float sc = mx > 0.0 ? float(mx) : 1.0f;
      for (int i = lane; i < B.m; i += 32) {
        double xi[D];
        load_point<D>(P, B.t_begin + i, xi);
        u[elem_offset(i, j, B.m, B.n, 2)] = to_bf16_bits(kernel_entry<D>(P, K, B.t_begin + i, B.s_begin + j, xi) / sc);
      }
      if (lane == 0) B.s_dst[j] = sc;
    }
  } else {
    const double* Vw = ws + B.ws + int64_t(B.m) * B.cap;
    unsigned short* v = static_cast<unsigned short*>(B.v_dst);
    const int64_t rp = vpad(B.rank, 2);
    for (int k = warp; k < B.rank; k += nw) {
      const double* Uk = ws + B.ws + int64_t(k) * B.m;
      const double* Vk = Vw + int64_t(k) * B.n;
      double mu = 0.0, mv = 0.0;
      for (int i = lane; i < B.m; i += 32) mu = fmax(mu, fabs(Uk[i]));
      for (int j = lane; j < B.n; j += 32) mv = fmax(mv, fabs(Vk[j]));
      mu = warp_max(mu);
      mv = warp_max(mv);
      const float su = mu > 0.0 ? float(mu) : 1.0f, sv = mv > 0.0 ? float(mv) : 1.0f;
      for (int i = lane; i < B.m; i += 32)
        u[elem_offset(lmap[B.t_map + i] - B.t_begin, k, B.m, B.rank, 2)] = to_bf16_bits(Uk[i] / su);
      for (int j = lane; j < B.n; j += 32) v[(lmap[B.s_map + j] - B.s_begin) * rp + k] = to_bf16_bits(Vk[j] / sv);
      if (lane == 0) B.s_dst[k] = su * sv;
    }
  }
}

unsigned warps_grid(int64_t items) { return unsigned((items + kWarpsPerCta - 1) / kWarpsPerCta); }

unsigned vec_grid(int64_t n) {
  int64_t g = (n + 255) / 256;
  if (g > 152 * 8) g = 152 * 8;
  if (g < 1) g = 1;
  return unsigned(g);
}

}  // namespace

void z_item_stages(ZItem& it, int r, int esz) {
  const int rp = int(vpad(r, esz));
  it.R = it.nst = 0;
  if (it.k0 != 0 || it.nk != rp || it.j1 <= it.j0) return;
  const int lanes = (it.nk + 16 / esz - 1) / (16 / esz);
  int P = 1;
  while (P < lanes) P <<= 1;
  const int G = 32 / P, rowb = rp * esz;
  it.R = (kZStageBytes - 32) / (rowb + 8) / G * G;  // >= G: rowb <= 16 P
  it.nst = (it.j1 - it.j0 + it.R - 1) / it.R;
}

template <typename TA, typename TACC>
static void zgemv_t(const ZBlock* zb, const ZItem* items, int nitems, const ZFix* fix, int nfix, void* zpart, void* in,
                    cudaStream_t st) {
  using TI = typename IO<TACC>::TI;
  using TY = typename IO<TACC>::TY;
  const unsigned g = unsigned((nitems + kZWarps - 1) / kZWarps);
  cudaFuncSetAttribute(zgemv_kernel<TA, TACC>, cudaFuncAttributeMaxDynamicSharedMemorySize, kZWarps * kZWarpSmem);
  zgemv_kernel<TA, TACC><<<g, kZWarps * 32, kZWarps * kZWarpSmem, st>>>(zb, items, nitems, static_cast<TY*>(zpart),
                                                                         static_cast<TI*>(in));
  if (nfix > 0)
    zfix_kernel<TACC><<<unsigned(nfix), kZPart, 0, st>>>(fix, static_cast<const TY*>(zpart), static_cast<TI*>(in));
}

cudaError_t launch_items64(const ZBlock* zb, const ZItem* zitems, int nitems, const ZFix* fix, unsigned int* zcnt,
                           double* zpart, const PanelItems& L, double* ypart, double* in, double* y, cudaStream_t st,
                           bool contig) {
  Items64 a{zb, zitems, nitems, fix, zcnt, zpart, L, ypart, in, y};
  if (contig) a.L.nsmall = 0;
  const int64_t total = int64_t(nitems) + a.L.nsmall + L.nbig;
  if (total > 0) {
    count_launches(1);
    // as few warps a CTA as fill the SMs: items on one SM share its FP64 pipe
    int warps = 1;
    while (warps < kWarpsPerCta && total > 152 * warps) warps *= 2;
    items64_kernel<<<unsigned((total + warps - 1) / warps), unsigned(warps * 32), 0, st>>>(a);
  }
  if (L.nplain > 0) {
    count_launches(1);
    panel_small64_kernel<<<warps_grid(L.nplain), kWarpsPerCta * 32, 0, st>>>(L, in, ypart, y);
  }
  if (contig && L.nsmall > 0) {
    count_launches(1);
    constexpr int bytes = kLWarps * l_warp_smem<double, double>();
    cudaFuncSetAttribute(panel_leaf_kernel<double, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    panel_leaf_kernel<double, double><<<unsigned((L.nsmall + kLWarps - 1) / kLWarps), kLWarps * 32, bytes, st>>>(
        L.panels, L.segs, L.small, L.nsmall, in, y, ypart);
  }
  return cudaGetLastError();
}

cudaError_t launch_zgemv(Prec a, Prec x, const ZBlock* zb, const ZItem* items, int nitems, const ZFix* fix, int nfix,
                         unsigned int* zcnt, void* zpart, void* in, cudaStream_t st, Accum acc) {
  if (nitems <= 0) return cudaSuccess;
  if (a == Prec::kD && x == Prec::kD)
    return launch_items64(zb, items, nitems, fix, zcnt, static_cast<double*>(zpart), PanelItems{}, nullptr,
                          static_cast<double*>(in), nullptr, st, false);
  count_launches(nfix > 0 ? 2 : 1);
  if (a == Prec::kF && x == Prec::kD && acc == Accum::kCompensated)
    zgemv_t<float, DF>(zb, items, nitems, fix, nfix, zpart, in, st);
  else if (a == Prec::kF && x == Prec::kD && acc == Accum::kRelaxed)
    zgemv_t<float, FH>(zb, items, nitems, fix, nfix, zpart, in, st);
  else if (a == Prec::kB && x == Prec::kD && acc == Accum::kRelaxed)
    zgemv_t<bf16, FH>(zb, items, nitems, fix, nfix, zpart, in, st);
  else if (a == Prec::kB && x == Prec::kD)
    zgemv_t<bf16, DF>(zb, items, nitems, fix, nfix, zpart, in, st);
  else if (a == Prec::kF && x == Prec::kF)
    zgemv_t<float, float>(zb, items, nitems, fix, nfix, zpart, in, st);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

// FP32 and BF16 storage: the bulk-copy staged kernels
template <typename TA, typename TACC>
static void panels_t(const PanelItems& L, const void* in, void* ypart, void* y, cudaStream_t st, bool contig) {
  using TI = typename IO<TACC>::TI;
  using TY = typename IO<TACC>::TY;
  const TI* ti = static_cast<const TI*>(in);
  TY *ty = static_cast<TY*>(y), *tp = static_cast<TY*>(ypart);
  if (L.nbig > 0) {
    // above the default 48 KB of dynamic shared memory; set on every launch
    // (the attribute is per device and cheap to set)
    cudaFuncSetAttribute(panel_tile_kernel<TA, TACC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kPWarps * kPWarpSmem);
    panel_tile_kernel<TA, TACC><<<unsigned((L.nbig + kPWarps - 1) / kPWarps), kPWarps * 32, kPWarps * kPWarpSmem, st>>>(
        L.panels, L.segs, L.big, L.nbig, tp, ti, ty);
  }
  if (L.nsmall > 0 && contig) {
    using TX = typename LeafX<TACC>::T;
    constexpr int bytes = kLWarps * l_warp_smem<TA, TX>();
    cudaFuncSetAttribute(panel_leaf_kernel<TA, TACC>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    panel_leaf_kernel<TA, TACC><<<unsigned((L.nsmall + kLWarps - 1) / kLWarps), kLWarps * 32, bytes, st>>>(
        L.panels, L.segs, L.small, L.nsmall, ti, ty, tp);
  } else if (L.nsmall > 0) {
    constexpr int bytes = kSWarps * s_warp_smem<TA>();
    cudaFuncSetAttribute(panel_small_kernel<TA, TACC>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    panel_small_kernel<TA, TACC><<<unsigned((L.nsmall + kSWarps - 1) / kSWarps), kSWarps * 32, bytes, st>>>(
        L.panels, L.segs, L.small, L.nsmall, ti, ty, tp);
  }
  if (L.nfix > 0) {
    const int rows = int(tile_rows(int(sizeof(TA))));
    panel_fix_kernel<TY><<<unsigned((int64_t(L.nfix) * rows + 255) / 256), 256, 0, st>>>(L.panels, L.fix, L.nfix, rows,
                                                                                          tp, ty);
  }
}

bool small_items_contiguous(const std::vector<Panel>& panels, const std::vector<Seg>& segs,
                            const std::vector<Item>& small, int esz) {
  for (const Item& it : small) {
    const int64_t m = panels[size_t(it.panel)].m;
    if (m < 1 || m > 32) return false;
    const char* a0 = static_cast<const char*>(segs[size_t(it.seg_b)].A);
    if (reinterpret_cast<uintptr_t>(a0) % 16 != 0) return false;
    const char* next = a0;  // end of the previous segment's columns
    for (int32_t q = it.seg_b; q < it.seg_e; q++) {
      const char* a = static_cast<const char*>(segs[size_t(q)].A);
      // each segment starts on 16 bytes after the previous one's data; offsets
      // from the item's first segment stay far below 2^31
      if (a < next || reinterpret_cast<uintptr_t>(a) % 16 != 0 || a - a0 > (int64_t(1) << 30)) return false;
      next = a + m * int64_t(segs[size_t(q)].K) * esz;
    }
  }
  return true;
}

cudaError_t launch_panels(Prec a, Prec x, const PanelItems& L, void* ypart, const void* in, void* y, cudaStream_t st,
                          Accum acc, bool contig) {
  if (L.nsmall + L.nbig + L.nplain <= 0) return cudaSuccess;
  if (a == Prec::kD && x == Prec::kD)
    return launch_items64(nullptr, nullptr, 0, nullptr, nullptr, nullptr, L, static_cast<double*>(ypart),
                          static_cast<double*>(const_cast<void*>(in)), static_cast<double*>(y), st, contig);
  count_launches(uint64_t(L.nbig > 0) + uint64_t(L.nsmall > 0) + uint64_t(L.nfix > 0));
  if (a == Prec::kF && x == Prec::kD && acc == Accum::kCompensated)
    panels_t<float, DF>(L, in, ypart, y, st, contig);
  else if (a == Prec::kF && x == Prec::kD && acc == Accum::kRelaxed)
    panels_t<float, FH>(L, in, ypart, y, st, contig);
  else if (a == Prec::kB && x == Prec::kD && acc == Accum::kRelaxed)
    panels_t<bf16, FH>(L, in, ypart, y, st, contig);
  else if (a == Prec::kB && x == Prec::kD)
    panels_t<bf16, DF>(L, in, ypart, y, st, contig);
  else if (a == Prec::kF && x == Prec::kF)
    panels_t<float, float>(L, in, ypart, y, st, contig);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

template <typename T>
__global__ void __launch_bounds__(256) batch_gather_kernel(const BatchInst* __restrict__ inst, const T* __restrict__ x,
                                                           T* __restrict__ in) {
  const BatchInst I = inst[blockIdx.y];
  for (int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r < I.n; r += int64_t(gridDim.x) * blockDim.x)
    in[I.in_base + r] = x[I.x_base + I.perm[r]];
}

template <typename T>
__global__ void __launch_bounds__(256) batch_combine_kernel(const BatchInst* __restrict__ inst, const T* __restrict__ y,
                                                            T* __restrict__ out) {
  const BatchInst I = inst[blockIdx.y];
  for (int64_t r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r < I.n; r += int64_t(gridDim.x) * blockDim.x) {
    const T* yc = y + I.y_base + r;
    double acc = double(yc[0]);
    for (int s = 1; s < I.nslots; s++) acc += double(yc[int64_t(s) * I.n]);
    out[I.x_base + I.perm[r]] = T(acc);
  }
}

namespace {
dim3 batch_grid(int count, int64_t max_n) {
  int64_t g = (max_n + 255) / 256;
  if (g > 64) g = 64;
  if (g < 1) g = 1;
  return dim3(unsigned(g), unsigned(count));
}
}  // namespace

cudaError_t launch_batch_gather(Prec x, const BatchInst* inst, int count, int64_t max_n, const void* src, void* in,
                                cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  count_launches(1);
  if (x == Prec::kD)
    batch_gather_kernel<double><<<batch_grid(count, max_n), 256, 0, st>>>(inst, static_cast<const double*>(src),
                                                                           static_cast<double*>(in));
  else
    batch_gather_kernel<float><<<batch_grid(count, max_n), 256, 0, st>>>(inst, static_cast<const float*>(src),
                                                                          static_cast<float*>(in));
  return cudaGetLastError();
}

cudaError_t launch_batch_combine(Prec x, const BatchInst* inst, int count, int64_t max_n, const void* y, void* out,
                                 cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  count_launches(1);
  if (x == Prec::kD)
    batch_combine_kernel<double><<<batch_grid(count, max_n), 256, 0, st>>>(inst, static_cast<const double*>(y),
                                                                            static_cast<double*>(out));
  else
    batch_combine_kernel<float><<<batch_grid(count, max_n), 256, 0, st>>>(inst, static_cast<const float*>(y),
                                                                           static_cast<float*>(out));
  return cudaGetLastError();
}

__global__ void __launch_bounds__(128) copy16_kernel(const CopyDesc* __restrict__ d) {
  const CopyDesc D = d[blockIdx.x];
  const int4* s = static_cast<const int4*>(D.src);
  int4* t = static_cast<int4*>(D.dst);
  for (uint64_t i = threadIdx.x; i < D.bytes / 16; i += blockDim.x) t[i] = s[i];
}

// One CTA per descriptor: 16-byte units of every row.
__global__ void __launch_bounds__(128) copy_rows_kernel(const RowCopy* __restrict__ d) {
  const RowCopy D = d[blockIdx.x];
  const int units = D.row_bytes / 16;
  const int64_t total = int64_t(units) * D.rows;
  for (int64_t e = threadIdx.x; e < total; e += blockDim.x) {
    const int64_t row = e / units, u = e - row * units;
    *reinterpret_cast<int4*>(static_cast<char*>(D.dst) + row * D.dst_pitch + u * 16) =
        *reinterpret_cast<const int4*>(static_cast<const char*>(D.src) + row * D.src_pitch + u * 16);
  }
}

cudaError_t launch_copy_rows(const RowCopy* d, int n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  count_launches(1);
  copy_rows_kernel<<<unsigned(n), 128, 0, st>>>(d);
  return cudaGetLastError();
}

cudaError_t launch_copy16(const CopyDesc* d, int n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  count_launches(1);
  copy16_kernel<<<unsigned(n), 128, 0, st>>>(d);
  return cudaGetLastError();
}

__global__ void split_kernel(const double* __restrict__ x, float2* __restrict__ out, int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const double v = x[i];
    const float h = __double2float_rn(v);
    out[i] = make_float2(h, __double2float_rn(v - double(h)));
  }
}

cudaError_t launch_split(const double* x, void* out, int64_t n, cudaStream_t st) {
  count_launches(1);
  split_kernel<<<vec_grid(n), 256, 0, st>>>(x, static_cast<float2*>(out), n);
  return cudaGetLastError();
}

template <typename T, bool SPLIT>
__global__ void prep_kernel(const T* __restrict__ x, const int64_t* __restrict__ perm, int64_t n, T* __restrict__ in,
                            float2* __restrict__ in2, T* __restrict__ y, int nslots) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const T v = x[perm ? perm[i] : i];
    in[i] = v;
    if constexpr (SPLIT) {
      const float h = __double2float_rn(v);
      in2[i] = make_float2(h, __double2float_rn(v - double(h)));
    }
    for (int s = 1; s < nslots; s++) y[int64_t(s) * n + i] = T(0);
  }
}

cudaError_t launch_prep(Prec x, const void* src, const int64_t* perm, int64_t n, void* in, void* in2, void* y,
                        int nslots, cudaStream_t st) {
  count_launches(1);
  const unsigned g = vec_grid(n);
  if (x == Prec::kF)
    prep_kernel<float, false><<<g, 256, 0, st>>>(static_cast<const float*>(src), perm, n, static_cast<float*>(in),
                                                 nullptr, static_cast<float*>(y), nslots);
  else if (in2)
    prep_kernel<double, true><<<g, 256, 0, st>>>(static_cast<const double*>(src), perm, n, static_cast<double*>(in),
                                                 static_cast<float2*>(in2), static_cast<double*>(y), nslots);
  else
    prep_kernel<double, false><<<g, 256, 0, st>>>(static_cast<const double*>(src), perm, n, static_cast<double*>(in),
                                                  nullptr, static_cast<double*>(y), nslots);
  return cudaGetLastError();
}

cudaError_t launch_combine(Prec x, const void* y, int64_t ld_y, int nslots, int64_t n, int nrhs, const int64_t* perm,
                           void* out, Prec out_prec, int64_t ld_out, cudaStream_t st) {
  count_launches(1);
  dim3 g(vec_grid(n), unsigned(nrhs));
  if (x == Prec::kD && out_prec == Prec::kD)
    combine_kernel<double, double><<<g, 256, 0, st>>>(static_cast<const double*>(y), ld_y, nslots, n, perm,
                                                      static_cast<double*>(out), ld_out);
  else if (x == Prec::kF && out_prec == Prec::kF)
    combine_kernel<float, float><<<g, 256, 0, st>>>(static_cast<const float*>(y), ld_y, nslots, n, perm,
                                                    static_cast<float*>(out), ld_out);
  else if (x == Prec::kF && out_prec == Prec::kD)
    combine_kernel<float, double><<<g, 256, 0, st>>>(static_cast<const float*>(y), ld_y, nslots, n, perm,
                                                     static_cast<double*>(out), ld_out);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_gather(const void* src, Prec sp, int64_t ld_src, const int64_t* perm, int64_t n, int nrhs, void* dst,
                          Prec dp, int64_t ld_dst, cudaStream_t st) {
  count_launches(1);
  dim3 g(vec_grid(n), unsigned(nrhs));
  if (sp == Prec::kD && dp == Prec::kD)
    gather_kernel<double, double><<<g, 256, 0, st>>>(static_cast<const double*>(src), ld_src, perm, n,
                                                     static_cast<double*>(dst), ld_dst);
  else if (sp == Prec::kD && dp == Prec::kF)
    gather_kernel<double, float><<<g, 256, 0, st>>>(static_cast<const double*>(src), ld_src, perm, n,
                                                    static_cast<float*>(dst), ld_dst);
  else if (sp == Prec::kF && dp == Prec::kD)
    gather_kernel<float, double><<<g, 256, 0, st>>>(static_cast<const float*>(src), ld_src, perm, n,
                                                    static_cast<double*>(dst), ld_dst);
  else
    gather_kernel<float, float><<<g, 256, 0, st>>>(static_cast<const float*>(src), ld_src, perm, n,
                                                   static_cast<float*>(dst), ld_dst);
  return cudaGetLastError();
}

template <int D>
static void assemble_d(const PointsDev& P, const KernelDev& K, const TileDesc* tiles, int ntiles, void* out, Prec op,
                       cudaStream_t st) {
  if (op == Prec::kD)
    assemble_kernel<D, double><<<warps_grid(ntiles), 256, 0, st>>>(P, K, tiles, ntiles, static_cast<double*>(out));
  else
    assemble_kernel<D, float><<<warps_grid(ntiles), 256, 0, st>>>(P, K, tiles, ntiles, static_cast<float*>(out));
}

cudaError_t launch_assemble(int ndim, const PointsDev& P, const KernelDev& K, const TileDesc* tiles, int ntiles,
                            void* out, Prec op, cudaStream_t st) {
  if (ntiles <= 0) return cudaSuccess;
  count_launches(1);
  switch (ndim) {
    case 1: assemble_d<1>(P, K, tiles, ntiles, out, op, st); break;
    case 2: assemble_d<2>(P, K, tiles, ntiles, out, op, st); break;
    case 3: assemble_d<3>(P, K, tiles, ntiles, out, op, st); break;
    case 4: assemble_d<4>(P, K, tiles, ntiles, out, op, st); break;
    case 5: assemble_d<5>(P, K, tiles, ntiles, out, op, st); break;
    case 6: assemble_d<6>(P, K, tiles, ntiles, out, op, st); break;
    case 7: assemble_d<7>(P, K, tiles, ntiles, out, op, st); break;
    case 8: assemble_d<8>(P, K, tiles, ntiles, out, op, st); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

template <int D>
static void compact_d(const PointsDev& P, const KernelDev& K, const double* ws, const int32_t* lmap,
                      const CompactDesc* blocks, int nblocks, Prec op, cudaStream_t st) {
  if (op == Prec::kD)
    compact_kernel<D, double><<<unsigned(nblocks), 256, 0, st>>>(P, K, ws, lmap, blocks, nblocks);
  else if (op == Prec::kB)
    compact_bf16_kernel<D><<<unsigned(nblocks), 256, 0, st>>>(P, K, ws, lmap, blocks, nblocks);
  else
    compact_kernel<D, float><<<unsigned(nblocks), 256, 0, st>>>(P, K, ws, lmap, blocks, nblocks);
}

template <int D>
static cudaError_t compact_preload_d() {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, compact_kernel<D, double>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, compact_kernel<D, float>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, compact_bf16_kernel<D>);
  return e;
}

cudaError_t compact_preload(int ndim) {
  switch (ndim) {
    case 1: return compact_preload_d<1>();
    case 2: return compact_preload_d<2>();
    case 3: return compact_preload_d<3>();
    case 4: return compact_preload_d<4>();
    case 5: return compact_preload_d<5>();
    case 6: return compact_preload_d<6>();
    case 7: return compact_preload_d<7>();
    case 8: return compact_preload_d<8>();
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_compact(int ndim, const PointsDev& P, const KernelDev& K, const double* ws, const int32_t* lmap,
                           const CompactDesc* blocks, int nblocks, Prec op, cudaStream_t st) {
  if (nblocks <= 0) return cudaSuccess;
  count_launches(1);
  switch (ndim) {
    case 1: compact_d<1>(P, K, ws, lmap, blocks, nblocks, op, st); break;
    case 2: compact_d<2>(P, K, ws, lmap, blocks, nblocks, op, st); break;
    case 3: compact_d<3>(P, K, ws, lmap, blocks, nblocks, op, st); break;
    case 4: compact_d<4>(P, K, ws, lmap, blocks, nblocks, op, st); break;
    case 5: compact_d<5>(P, K, ws, lmap, blocks, nblocks, op, st); break;
    case 6: compact_d<6>(P, K, ws, lmap, blocks, nblocks, op, st); break;
    case 7: compact_d<7>(P, K, ws, lmap, blocks, nblocks, op, st); break;
    case 8: compact_d<8>(P, K, ws, lmap, blocks, nblocks, op, st); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}


// ============================================================================
// Several right-hand sides at once: FP32 factors, FP32 vectors, FP32 sums.
// A chunk of kMR right-hand sides is interleaved: entry e of a vector buffer
// holds its kMR values contiguously (byte offset e * 4 kMR), so one input row
// or z row is one 128-byte run that the bulk-copy engine stages next to the
// factor bytes, and every factor entry read from HBM feeds kMR FMAs; grid.y runs
// over chunks.
// ============================================================================
namespace {

constexpr int kMWarps = 4;
constexpr int kMStages = 2;
constexpr int kMStageBytes = 7424;             // factor and input bytes per stage
constexpr int kMRowBytes = kMR * 4;            // one interleaved entry
// a lane's column loads may run up to 496 bytes beyond the last row: 512 bytes at the end
constexpr int kMWarpSmem = 64 + kMStages * kMStageBytes + 512;
static_assert(kMWarpSmem % 16 == 0 && kMStageBytes % 16 == 0, "bulk copy destinations must stay 16-byte aligned");

// Products of the wide items (V rows of up to 128 columns, U tiles of up to 128
// rows): out(c, r) += A(k, c) x(k, r), every row k of A and of x staged in
// shared memory.  A value read from shared memory costs its register write-back
// (128 bytes per clock and SM: a 16-byte load of a warp 4 clocks, whether or
// not the lanes read the same address) against a quarter clock per FMA
// instruction, so with one right-hand side per lane and the factors broadcast
// the loads took four times as long as the FMAs.  A lane therefore keeps a tile
// of 4 NQ columns by 8 right-hand sides: lane 4 cg + rg has columns 32 q + 4 cg ..
// + 3 (q < NQ) and right-hand sides 4 rg .. + 3 and 16 + 4 rg .. + 3, and 2 + NQ
// loads of 16 bytes feed 32 NQ FMAs.  Columns beyond the item's are computed
// from whatever follows in the warp's shared memory and never stored.
// 24 3D operators (420,000 points), 32 right-hand sides: V^T x 4.44 -> 1.52 ms, node
// panels 2.19 -> 1.24 ms, leaf panels 3.65 -> 1.43 ms (whole product 11.1 -> 4.6 ms;
// the FMAs alone would take 1.4).
template <int NQ>
__device__ __forceinline__ void mr_wide(const unsigned char* as, int rowb, const float* xs, int nr, int lane,
                                        float (&acc)[4 * NQ][8]) {
  const int cg = lane >> 2, rg = lane & 3;
  const unsigned char* ap = as + cg * 16;
  const float4* x4 = reinterpret_cast<const float4*>(xs) + rg;
#pragma unroll 2
  for (int i = 0; i < nr; i++) {
    const float4 xa = x4[i * 8], xb = x4[i * 8 + 4];
    const float x[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      const float4 v4 = *reinterpret_cast<const float4*>(ap + i * rowb + q * 128);
      const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
      for (int e = 0; e < 4; e++)
#pragma unroll
        for (int r = 0; r < 8; r++) acc[4 * q + e][r] = __fmaf_rn(v[e], x[r], acc[4 * q + e][r]);
    }
  }
}

// The sums of columns c < n to dst + c * kMR.
template <int NQ>
__device__ __forceinline__ void mr_store(float* dst, int n, int lane, const float (&acc)[4 * NQ][8]) {
  const int cg = lane >> 2, rg = lane & 3;
#pragma unroll
  for (int q = 0; q < NQ; q++)
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int c = 32 * q + 4 * cg + e;
      const float* a = acc[4 * q + e];
      if (c < n) {
        *reinterpret_cast<float4*>(dst + int64_t(c) * kMR + 4 * rg) = make_float4(a[0], a[1], a[2], a[3]);
        *reinterpret_cast<float4*>(dst + int64_t(c) * kMR + 16 + 4 * rg) = make_float4(a[4], a[5], a[6], a[7]);
      }
    }
}

// z_b = V_b^T X_s: item = rows [j0, j1) of block zb, columns [k0, k0 + nk) (at
// most 128); runs of V rows and their input rows staged by bulk copies in a ring
// of kMStages: one copy for a run of whole rows (WHOLE), or one for each row of just
// the item's columns.
template <int NQ, bool WHOLE>
__device__ __forceinline__ void zgemv_mr_item(const ZItem& it, const ZBlock& Z, const float* V, int64_t rp,
                                              const float* xr, float* dst, unsigned char* base, int lane) {
  uint64_t* bar = reinterpret_cast<uint64_t*>(base);
  unsigned char* stage0 = base + 64;
  const int rowb = WHOLE ? int(rp) * 4 : it.nk * 4;  // a multiple of 16, as k0
  const int R = kMStageBytes / (rowb + kMRowBytes);  // rows per stage: their factors, then their inputs
  const int nrows = it.j1 - it.j0;
  const int total = (nrows + R - 1) / R;
  auto issue = [&](int q) {  // rows q R ..
    const int s = q % kMStages, r0 = q * R, nr = min(R, nrows - r0);
    unsigned char* st = stage0 + s * kMStageBytes;
    fence_proxy_async();
    if (lane == 0) {
      mbar_expect_tx(bar + s, uint32_t(nr) * uint32_t(rowb + kMRowBytes));
      if (WHOLE) bulk_g2s(st, V + int64_t(r0) * rp, uint32_t(nr * rowb), bar + s);
      bulk_g2s(st + R * rowb, xr + int64_t(r0) * kMR, uint32_t(nr * kMRowBytes), bar + s);
    }
    if (!WHOLE) {
      __syncwarp();
      for (int r = lane; r < nr; r += 32)
        bulk_g2s(st + r * rowb, V + int64_t(r0 + r) * rp + it.k0, uint32_t(rowb), bar + s);
    }
  };
  const bool copies = !WHOLE || lane == 0;
  if (copies)
    for (int q = 0; q < min(kMStages, total); q++) issue(q);
  float acc[4 * NQ][8];
#pragma unroll
  for (int c = 0; c < 4 * NQ; c++)
#pragma unroll
    for (int r = 0; r < 8; r++) acc[c][r] = 0.f;
  for (int q = 0; q < total; q++) {
    const int s = q % kMStages;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(bar + s, uint32_t(q / kMStages) & 1u));
    if (!ok) {
      if (lane == 0) atomicAdd(&g_stream_timeouts, 1u);
      for (int t = q; t < min(q + kMStages, total); t++) mbar_wait(bar + t % kMStages, uint32_t(t / kMStages) & 1u);
      return;
    }
    const unsigned char* st = stage0 + s * kMStageBytes;
    mr_wide<NQ>(st + (WHOLE ? it.k0 * 4 : 0), rowb, reinterpret_cast<const float*>(st + R * rowb),
                min(R, nrows - q * R), lane, acc);
    __syncwarp();
    if (copies && q + kMStages < total) issue(q + kMStages);
  }
  mr_store<NQ>(dst, it.part < 0 ? min(it.nk, Z.r - it.k0) : it.nk, lane, acc);
}

__global__ void __launch_bounds__(kMWarps * 32, 3)
    zgemv_mr_kernel(const ZBlock* __restrict__ zb, const ZItem* __restrict__ items, int nitems,
                    float* __restrict__ zpart, int64_t zpart_ld, float* in, int64_t ld_in) {
  extern __shared__ __align__(16) unsigned char msm[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * kMWarps + wid;
  if (w >= nitems) return;
  const ZItem it = items[w];
  const ZBlock Z = zb[it.zb];
  const int64_t rp = vpad(Z.r, 4);
  float* inc = in + int64_t(blockIdx.y) * ld_in * kMR;
  float* zp = zpart + int64_t(blockIdx.y) * zpart_ld * kMR;
  const float* V = static_cast<const float*>(Z.V) + int64_t(it.j0) * rp;
  const float* xr = inc + (Z.x_off + it.j0) * kMR;
  float* dst = it.part < 0 ? inc + (Z.z_off + it.k0) * kMR : zp + int64_t(it.part) * kMR;
  unsigned char* base = msm + wid * kMWarpSmem;
  if (lane == 0) {
    uint64_t* bar = reinterpret_cast<uint64_t*>(base);
#pragma unroll
    for (int s = 0; s < kMStages; s++) mbar_init(bar + s, 1);
    fence_mbar_init();
  }
  __syncwarp();
  // just the item's columns where a stage does not hold two whole rows (rank above
  // 928: 4D N = 40000, ranks up to 1227, 2.3 ms; whole rows read by plain loads
  // instead took 7.0); below, the short copies of an item of few columns cost more
  // than the rows' other columns (2D N = 6934, d' = 1, ranks about 130: 353 us
  // against 191)
  if (it.nk < rp && rp * 4 > kMStageBytes / 2) {
    zgemv_mr_item<4, false>(it, Z, V, rp, xr, dst, base, lane);
    return;
  }
  switch ((it.nk + 31) / 32) {
    case 1: zgemv_mr_item<1, true>(it, Z, V, rp, xr, dst, base, lane); break;
    case 2: zgemv_mr_item<2, true>(it, Z, V, rp, xr, dst, base, lane); break;
    case 3: zgemv_mr_item<3, true>(it, Z, V, rp, xr, dst, base, lane); break;
    default: zgemv_mr_item<4, true>(it, Z, V, rp, xr, dst, base, lane); break;
  }
}

// z row zpos (all kMR values) = sum of the item partials, in order.
__global__ void __launch_bounds__(256) zfix_mr_kernel(const ZFix* __restrict__ fix, int nfix,
                                                     const float* __restrict__ zpart, int64_t zpart_ld,
                                                     float* __restrict__ in, int64_t ld_in) {
  const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int64_t fc = t / kMR;
  const int f = int(fc / kZPart), k = int(fc % kZPart), c = int(t % kMR);
  if (f >= nfix) return;
  const ZFix F = fix[f];
  if (k >= F.nk) return;
  const float* zp = zpart + int64_t(blockIdx.y) * zpart_ld * kMR;
  float acc = 0.f;
  for (int q = 0; q < F.count; q++) acc += zp[(int64_t(F.part) + int64_t(q) * kZPart + k) * kMR + c];
  in[int64_t(blockIdx.y) * ld_in * kMR + (F.zpos + k) * kMR + c] = acc;
}

// Leaf panels (m <= 32): one warp per item.  The item's segments are cut into
// pieces that are packed, in order, into stages of at most kMSUBytes of factor
// bytes (each piece 16-byte aligned, a multiple of 4 columns unless it ends its
// segment) and kMSRows columns, each lane planning and copying a segment and noting
// where its columns start.  Lane tiles as in mr_wide, for
// columns of few rows at any alignment: RR = 1, 2 or 4 groups of lanes take RL =
// ceil(m / RR) <= 8 (made even) rows each, 4 lanes their 8 right-hand sides each, and the 8 / RR
// slices left every (8 / RR)-th column of the stage, added by shuffles at the end.
constexpr int kMSUBytes = 4096;
constexpr int kMSRows = 32;
constexpr int kMSXBytes = kMSRows * kMRowBytes;
constexpr int kMSStage = kMSUBytes + kMSXBytes + kMSRows * 4;  // factors, inputs, column offsets
constexpr int kMSWarpSmem = 64 + kMStages * kMSStage;
static_assert(kMSWarpSmem % 16 == 0 && kMSStage % 16 == 0, "bulk copy destinations must stay 16-byte aligned");

template <int RL>
__device__ __forceinline__ void small_mr_item(const Seg* __restrict__ segs, const Item& it, int m, int RR,
                                              const float* inc, float* dst, unsigned char* base, int lane) {
  uint64_t* bar = reinterpret_cast<uint64_t*>(base);
  unsigned char* stage0 = base + 64;
  const int rg = lane & 3, rr = (lane >> 2) & (RR - 1), SL = 8 / RR, sl = (lane >> 2) / RR;
  // packing cursor (the same in every lane): segment ps, column pc; lane k has the record of segment win + k
  int32_t ps = it.seg_b, pc = 0, win = it.seg_b - 32;
  const char* rA = nullptr;
  int64_t ro = 0;
  int rK = 0;
  // Packs and issues the next stage; its column count (0: nothing left).  Lane
  // k takes segment win + k (from column pc for the cursor's): whole segments
  // while they fit, or as many columns of the first one as do.  Each lane raises
  // the stage's transaction count (no arrival) and starts its piece's two copies;
  // the stage's one arrival comes after them all, so the phase cannot complete
  // before every copy is accounted for.
  auto issue = [&](int st) -> int {
    if (ps >= it.seg_e) return 0;
    unsigned char* su = stage0 + st * kMSStage;
    int* co = reinterpret_cast<int*>(su + kMSUBytes + kMSXBytes);
    if (ps >= win + 24 || ps < win) {  // at least 8 segments in the window (it ends at the item's end)
      win = ps;
      rK = 0;
      if (win + lane < it.seg_e) {
        const Seg S = segs[win + lane];
        rA = static_cast<const char*>(S.A);
        ro = S.in_off;
        rK = S.K;
      }
    }
    const int k0 = ps - win, c0 = lane == k0 ? pc : 0;
    int take = lane >= k0 ? rK - c0 : 0;
    int cols = take, bytes = (take * m * 4 + 15) & ~15;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int vc = __shfl_up_sync(0xffffffffu, cols, o), vb = __shfl_up_sync(0xffffffffu, bytes, o);
      if (lane >= o) {
        cols += vc;
        bytes += vb;
      }
    }
    // the lanes from k0 whose segments fit whole: a run, as both sums grow
    const bool fits = lane >= k0 && take > 0 && cols <= kMSRows && bytes <= kMSUBytes;
    const unsigned whole = __ballot_sync(0xffffffffu, fits);
    int n;
    if (whole == 0u) {
      // the cursor's segment is longer than a stage: a multiple of 4 columns, which keeps 16-byte alignment
      n = min(kMSRows, kMSUBytes / (m * 4)) / 4 * 4;
      take = lane == k0 ? n : 0;
      cols = n;
      bytes = n * m * 4;
      pc += n;
    } else {
      const int last = 31 - __clz(whole);
      n = __shfl_sync(0xffffffffu, cols, last);
      if (!fits) take = 0;
      ps = win + last + 1;
      pc = 0;
    }
    if (take > 0) {
      const int pb = (take * m * 4 + 15) & ~15, row0 = cols - take, off = bytes - pb;
      fence_proxy_async();
      mbar_expect_tx_only(bar + st, uint32_t(pb + take * kMRowBytes));
      bulk_g2s(su + off, rA + int64_t(c0) * m * 4, uint32_t(pb), bar + st);
      bulk_g2s(su + kMSUBytes + row0 * kMRowBytes, inc + (ro + c0) * kMR, uint32_t(take * kMRowBytes), bar + st);
      for (int j = 0; j < take; j++) co[row0 + j] = off + j * m * 4;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(bar + st);
    return n;
  };
  static_assert(kMStages == 2, "two column counts");
  uint64_t acc2[RL][4];  // pairs of right-hand sides: half the instructions (1.52 -> 1.43 ms for the two launches)
#pragma unroll
  for (int i = 0; i < RL; i++)
#pragma unroll
    for (int r = 0; r < 4; r++) acc2[i][r] = 0;
  // the last group's rows beyond m read whatever follows in the warp's share and are never stored
  const int row0 = rr * RL;
  bool gave_up = false;
  // q = -2, -1 fill the ring; from then on stage q is consumed and refilled (one
  // copy of the code: several row counts run on an SM at a time, and unrolled
  // over the stages they did not fit its instruction cache)
  int cur = 0, next = 0;
#pragma unroll 1
  for (int q = -kMStages; q < 0 || cur > 0; q++) {
    const int st = q & 1;
    if (q >= 0) {
      if (!__all_sync(0xffffffffu, mbar_wait(bar + st, uint32_t(q >> 1) & 1u))) {
        if (lane == 0) atomicAdd(&g_stream_timeouts, 1u);
        if (next > 0) mbar_wait(bar + (st ^ 1), uint32_t((q + 1) >> 1) & 1u);
        gave_up = true;
        break;
      }
      const unsigned char* su = stage0 + st * kMSStage;
      const float4* x4 = reinterpret_cast<const float4*>(su + kMSUBytes) + rg;
      const int* co = reinterpret_cast<const int*>(su + kMSUBytes + kMSXBytes);
#pragma unroll 1
      for (int c = sl; c < cur; c += SL) {
        const float* a = reinterpret_cast<const float*>(su + co[c]) + row0;
        const float4 xa = x4[c * 8], xb = x4[c * 8 + 4];
        const uint64_t x[4] = {pack_f2(xa.x, xa.y), pack_f2(xa.z, xa.w), pack_f2(xb.x, xb.y), pack_f2(xb.z, xb.w)};
#pragma unroll
        for (int i = 0; i < RL; i++) {
          const uint64_t v = pack_f2(a[i], a[i]);
#pragma unroll
          for (int r = 0; r < 4; r++) acc2[i][r] = fma_f2(v, x[r], acc2[i][r]);
        }
      }
      __syncwarp();
    }
    cur = next;
    next = issue(st);  // into the stage just consumed
  }
  float acc[RL][8];
#pragma unroll
  for (int i = 0; i < RL; i++)
#pragma unroll
    for (int r = 0; r < 4; r++) unpack_f2(acc2[i][r], acc[i][2 * r], acc[i][2 * r + 1]);
  for (int o = 4 * RR; o < 32; o <<= 1)
#pragma unroll
    for (int i = 0; i < RL; i++)
#pragma unroll
      for (int r = 0; r < 8; r++) acc[i][r] += __shfl_xor_sync(0xffffffffu, acc[i][r], o);
  if (sl == 0 && !gave_up) {
#pragma unroll
    for (int i = 0; i < RL; i++)
      if (row0 + i < m) {
        float* d = dst + int64_t(row0 + i) * kMR + 4 * rg;
        *reinterpret_cast<float4*>(d) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        *reinterpret_cast<float4*>(d + 16) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
      }
  }
}

__global__ void __launch_bounds__(kMWarps * 32, 4)
    panel_small_mr_kernel(const Panel* __restrict__ panels, const Seg* __restrict__ segs,
                          const Item* __restrict__ items, int nitems, const float* __restrict__ in, int64_t ld_in,
                          float* __restrict__ y, int64_t ld_y, float* __restrict__ ypart, int64_t ypart_ld) {
  extern __shared__ __align__(16) unsigned char msm[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * kMWarps + wid;
  if (w >= nitems) return;
  const Item it = items[w];
  const Panel P = panels[it.panel];
  const int m = P.m;
  const float* inc = in + int64_t(blockIdx.y) * ld_in * kMR;
  // split panels: partial rows at the part's 128-row block of ypart (panel_fix_mr_kernel)
  float* dst = it.part < 0 ? y + int64_t(blockIdx.y) * ld_y * kMR + P.yoff * kMR
                           : ypart + int64_t(blockIdx.y) * ypart_ld * kMR + int64_t(it.part) * 128 * kMR;
  unsigned char* base = msm + wid * kMSWarpSmem;
  if (lane == 0) {
    uint64_t* bar = reinterpret_cast<uint64_t*>(base);
#pragma unroll
    for (int s = 0; s < kMStages; s++) mbar_init(bar + s, 1);
    fence_mbar_init();
  }
  __syncwarp();
  // rows per lane rounded up to 2, 4, 6 or 8
  const int RR = m <= 8 ? 1 : m <= 16 ? 2 : 4;
#define HODLR_SMALL_MR(rl_)                                            \
  case rl_:                                                            \
    small_mr_item<2 * rl_>(segs, it, m, RR, inc, dst, base, lane);         \
    break;
  switch (((m + RR - 1) / RR + 1) / 2) {
    HODLR_SMALL_MR(1)
    HODLR_SMALL_MR(2)
    HODLR_SMALL_MR(3)
    HODLR_SMALL_MR(4)
    default: break;
  }
#undef HODLR_SMALL_MR
}

// Panels of more than 32 rows: item = row tile t (up to 128 rows) times a
// run of segments; runs of tile columns and their input rows are staged
// (mr_wide: the tile's columns are the rows of A).
template <int NQ>
__device__ __forceinline__ void panel_tile_mr_item(const Seg* __restrict__ segs, const Item& it, int rows, int64_t h,
                                                   const float* inc, float* dst, unsigned char* base, int lane) {
  constexpr int T = 128;
  const int t = it.chunk;
  const int colb = int(h) * 4;
  const int cps = kMStageBytes / (colb + kMRowBytes);  // columns per stage, then their inputs
  float acc[4 * NQ][8];
#pragma unroll
  for (int c = 0; c < 4 * NQ; c++)
#pragma unroll
    for (int r = 0; r < 8; r++) acc[c][r] = 0.f;
  uint64_t* bar = reinterpret_cast<uint64_t*>(base);
  unsigned char* stage0 = base + 64;
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < kMStages; s++) mbar_init(bar + s, 1);
    fence_mbar_init();
  }
  __syncwarp();
  int64_t ps = it.seg_b;
  int pc = 0, issued = 0;
#define HODLR_MRT_ISSUE()                                                                          \
  do {                                                                                             \
    while (ps < it.seg_e && pc >= segs[ps].K) {                                                    \
      ps++;                                                                                        \
      pc = 0;                                                                                      \
    }                                                                                              \
    if (ps >= it.seg_e) break;                                                                     \
    const Seg S_ = segs[ps];                                                                       \
    const int nc_ = min(cps, S_.K - pc);                                                           \
    if (lane == 0) {                                                                               \
      const int st_ = issued % kMStages;                                                           \
      unsigned char* dst_ = stage0 + st_ * kMStageBytes;                                           \
      const float* src_ = static_cast<const float*>(S_.A) + int64_t(t) * T * S_.K + int64_t(pc) * h; \
      fence_proxy_async();                                                                         \
      mbar_expect_tx(bar + st_, uint32_t(nc_) * uint32_t(colb + kMRowBytes));                      \
      bulk_g2s(dst_, src_, uint32_t(nc_ * colb), bar + st_);                                       \
      bulk_g2s(dst_ + cps * colb, inc + (S_.in_off + pc) * kMR, uint32_t(nc_ * kMRowBytes), bar + st_); \
    }                                                                                              \
    pc += nc_;                                                                                     \
    issued++;                                                                                      \
  } while (0)
  for (int q = 0; q < kMStages; q++) HODLR_MRT_ISSUE();
  int64_t cs = it.seg_b;
  int cc = 0;
  for (int q = 0; q < issued; q++) {
    while (cc >= segs[cs].K) {
      cs++;
      cc = 0;
    }
    const int nc = min(cps, segs[cs].K - cc);
    const int st = q % kMStages;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(bar + st, uint32_t(q / kMStages) & 1u));
    if (!ok) {
      if (lane == 0) atomicAdd(&g_stream_timeouts, 1u);
      for (int u = q; u < issued; u++) mbar_wait(bar + u % kMStages, uint32_t(u / kMStages) & 1u);
      return;
    }
    const unsigned char* us = stage0 + st * kMStageBytes;
    const float* xs = reinterpret_cast<const float*>(us + cps * colb);
    mr_wide<NQ>(us, colb, xs, nc, lane, acc);
    cc += nc;
    __syncwarp();
    HODLR_MRT_ISSUE();
  }
#undef HODLR_MRT_ISSUE
  mr_store<NQ>(dst, rows, lane, acc);
}

__global__ void __launch_bounds__(kMWarps * 32, 3)
    panel_tile_mr_kernel(const Panel* __restrict__ panels, const Seg* __restrict__ segs,
                         const Item* __restrict__ items, int nitems, float* __restrict__ ypart, int64_t ypart_ld,
                         const float* __restrict__ in, int64_t ld_in, float* __restrict__ y, int64_t ld_y) {
  constexpr int T = 128;
  extern __shared__ __align__(16) unsigned char msm[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * kMWarps + wid;
  if (w >= nitems) return;
  const Item it = items[w];
  const Panel P = panels[it.panel];
  const float* inc = in + int64_t(blockIdx.y) * ld_in * kMR;
  const int rows = min(T, P.m - it.chunk * T);
  const int64_t h = tile_height(P.m, it.chunk, 4);
  float* dst = it.part < 0 ? y + int64_t(blockIdx.y) * ld_y * kMR + (P.yoff + int64_t(it.chunk) * T) * kMR
                           : ypart + int64_t(blockIdx.y) * ypart_ld * kMR + int64_t(it.part) * T * kMR;
  unsigned char* base = msm + wid * kMWarpSmem;
  switch (int(h + 31) / 32) {
    case 1: panel_tile_mr_item<1>(segs, it, rows, h, inc, dst, base, lane); break;
    case 2: panel_tile_mr_item<2>(segs, it, rows, h, inc, dst, base, lane); break;
    case 3: panel_tile_mr_item<3>(segs, it, rows, h, inc, dst, base, lane); break;
    default: panel_tile_mr_item<4>(segs, it, rows, h, inc, dst, base, lane); break;
  }
}

// One CTA per split panel chunk, a warp per row (a lane per right-hand side).
__global__ void __launch_bounds__(256) panel_fix_mr_kernel(const Panel* __restrict__ panels,
                                                           const PanelFix* __restrict__ fix,
                                                           const float* __restrict__ ypart, int64_t ypart_ld,
                                                           float* __restrict__ y, int64_t ld_y) {
  constexpr int rows = 128;
  const int lane = threadIdx.x & 31;
  const PanelFix F = fix[blockIdx.x];
  const Panel P = panels[F.panel];
  const float* yp = ypart + int64_t(blockIdx.y) * ypart_ld * kMR + int64_t(F.part) * rows * kMR + lane;
  float* yo = y + int64_t(blockIdx.y) * ld_y * kMR + (P.yoff + F.chunk * rows) * kMR + lane;
  const int n = min(rows, P.m - F.chunk * rows);
  for (int i = threadIdx.x >> 5; i < n; i += 8)
    yo[int64_t(i) * kMR] = sum_parts(yp + int64_t(i) * kMR, F.count, int64_t(rows) * kMR);
}

// in (chunk ch, interleaved) <- x (caller order, column major total_n x k): 32
// points of the caller's order at a time, read column by column, written as
// whole rows at their tree positions.
__global__ void __launch_bounds__(256) batch_gather_mr_kernel(const BatchInst* __restrict__ inst,
                                                              const float* __restrict__ x, int64_t total_n, int k,
                                                              float* __restrict__ in, int64_t ld_in, int ch) {
  __shared__ float tile[32][kMR + 1];
  const BatchInst I = inst[blockIdx.y];
  float* inc = in + int64_t(ch) * ld_in * kMR;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int64_t p0 = int64_t(blockIdx.x) * 32; p0 < I.n; p0 += int64_t(gridDim.x) * 32) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int c = wid * 4 + q, col = ch * kMR + c;
      tile[lane][c] = col < k && p0 + lane < I.n ? x[int64_t(col) * total_n + I.x_base + p0 + lane] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int64_t p = p0 + wid * 4 + q;
      if (p < I.n) inc[(I.in_base + I.iperm[p]) * kMR + lane] = tile[wid * 4 + q][lane];
    }
    __syncthreads();
  }
}

// A CTA takes 32 points of one instance in the caller's order: each warp reads
// whole 128-byte rows of the slots (at the points' tree positions), and the sums
// are written from shared memory as runs of 32 points of a column (written row
// by row in tree order, each value was a sector of its own: 313 us for 420,000
// points against 60).  A row is the FP64 sum of its slots, formed on the FP32 pipe
// where that gives the same value (fpsum.cuh; 20 us more than a plain FP32 pair).
// Q rows of up to U slots are read before their sums (others one by one).
template <int U, int Q>
__global__ void __launch_bounds__(256) batch_combine_mr_kernel(const BatchInst* __restrict__ inst,
                                                               const float* __restrict__ y, int64_t ld_y,
                                                               float* __restrict__ out, int64_t total_n, int k, int ch) {
  __shared__ float tile[32][kMR + 1];
  const BatchInst I = inst[blockIdx.y];
  const float* yc = y + int64_t(ch) * ld_y * kMR;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t stride = I.n * kMR;
  const bool live = ch * kMR + lane < k, few = I.nslots <= U;
  for (int64_t p0 = int64_t(blockIdx.x) * 32; p0 < I.n; p0 += int64_t(gridDim.x) * 32) {
#pragma unroll 1
    for (int q0 = 0; q0 < 4; q0 += Q) {  // four rows a warp
      const float* yr[Q];
      float v[Q][U];
#pragma unroll
      for (int q = 0; q < Q; q++) {
        const int64_t p = p0 + wid * 4 + q0 + q;
        yr[q] = p < I.n && live ? yc + (I.y_base + I.iperm[p]) * kMR + lane : nullptr;
#pragma unroll
        for (int s = 0; s < U; s++) v[q][s] = yr[q] && few && s < I.nslots ? yr[q][s * stride] : 0.f;
      }
#pragma unroll
      for (int q = 0; q < Q; q++) {
        float r = 0.f;
        const bool ok = few && sum_few_as_fp64(I.nslots, v[q], r);
        if (yr[q])
          tile[wid * 4 + q0 + q][lane] = ok ? r : sum_as_fp64(I.nslots, [&](int s) { return yr[q][s * stride]; });
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int c = wid * 4 + q, col = ch * kMR + c;
      if (col < k && p0 + lane < I.n) out[int64_t(col) * total_n + I.x_base + p0 + lane] = tile[lane][c];
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) invert_perm_kernel(const int64_t* __restrict__ perm, int64_t n,
                                                          int32_t* __restrict__ iperm) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    iperm[perm[i]] = int32_t(i);
}

}  // namespace

cudaError_t launch_zgemv_mr(const ZBlock* zb, const ZItem* items, int nitems, const ZFix* fix, int nfix, float* zpart,
                            int64_t zpart_ld, float* in, int64_t ld_in, int nchunks, cudaStream_t st) {
  if (nitems <= 0) return cudaSuccess;
  count_launches(nfix > 0 ? 2 : 1);
  cudaFuncSetAttribute(zgemv_mr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMWarps * kMWarpSmem);
  dim3 g(unsigned((nitems + kMWarps - 1) / kMWarps), unsigned(nchunks));
  zgemv_mr_kernel<<<g, kMWarps * 32, kMWarps * kMWarpSmem, st>>>(zb, items, nitems, zpart, zpart_ld, in, ld_in);
  if (nfix > 0) {
    dim3 gf(unsigned((int64_t(nfix) * kZPart * kMR + 255) / 256), unsigned(nchunks));
    zfix_mr_kernel<<<gf, 256, 0, st>>>(fix, nfix, zpart, zpart_ld, in, ld_in);
  }
  return cudaGetLastError();
}

cudaError_t launch_panels_mr(const Panel* panels, const Seg* segs, const Item* small, int nsmall, const Item* big,
                             int nbig, const PanelFix* fix, int nfix, float* ypart, int64_t ypart_ld, const float* in,
                             int64_t ld_in, float* y, int64_t ld_y, int nchunks, cudaStream_t st) {
  if (nsmall + nbig <= 0) return cudaSuccess;
  count_launches(uint64_t(nbig > 0) + uint64_t(nsmall > 0) + uint64_t(nfix > 0));
  if (nbig > 0) {
    cudaFuncSetAttribute(panel_tile_mr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMWarps * kMWarpSmem);
    dim3 g(unsigned((nbig + kMWarps - 1) / kMWarps), unsigned(nchunks));
    panel_tile_mr_kernel<<<g, kMWarps * 32, kMWarps * kMWarpSmem, st>>>(panels, segs, big, nbig, ypart, ypart_ld, in,
                                                                          ld_in, y, ld_y);
  }
  if (nsmall > 0) {
    cudaFuncSetAttribute(panel_small_mr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMWarps * kMSWarpSmem);
    dim3 g(unsigned((nsmall + kMWarps - 1) / kMWarps), unsigned(nchunks));
    panel_small_mr_kernel<<<g, kMWarps * 32, kMWarps * kMSWarpSmem, st>>>(panels, segs, small, nsmall, in, ld_in, y,
                                                                           ld_y, ypart, ypart_ld);
  }
  if (nfix > 0) {
    panel_fix_mr_kernel<<<dim3(unsigned(nfix), unsigned(nchunks)), 256, 0, st>>>(panels, fix, ypart, ypart_ld, y, ld_y);
  }
  return cudaGetLastError();
}

cudaError_t launch_batch_gather_mr(const BatchInst* inst, int count, int64_t max_n, const float* x, int64_t total_n,
                                   int k, float* in, int64_t ld_in, int nchunks, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  for (int ch = 0; ch < nchunks; ch++) {
    count_launches(1);
    batch_gather_mr_kernel<<<dim3(unsigned(std::min<int64_t>((max_n + 31) / 32, 2048)), unsigned(count)), 256, 0, st>>>(inst, x, total_n, k, in, ld_in, ch);
  }
  return cudaGetLastError();
}

cudaError_t launch_invert_perm(const int64_t* perm, int64_t n, int32_t* iperm, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  count_launches(1);
  invert_perm_kernel<<<vec_grid(n), 256, 0, st>>>(perm, n, iperm);
  return cudaGetLastError();
}

cudaError_t launch_batch_combine_mr(const BatchInst* inst, int count, int64_t max_n, int max_slots, const float* y,
                                    int64_t ld_y, float* out, int64_t total_n, int k, int nchunks, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  const dim3 g(unsigned(std::min<int64_t>((max_n + 31) / 32, 2048)), unsigned(count));
  for (int ch = 0; ch < nchunks; ch++) {
    count_launches(1);
    // (deep trees: 1D N = 8104, three operators, 206 us with <8, 4>, 200 with <16, 2>)
    if (max_slots <= 8)
      batch_combine_mr_kernel<8, 4><<<g, 256, 0, st>>>(inst, y, ld_y, out, total_n, k, ch);
    else
      batch_combine_mr_kernel<16, 2><<<g, 256, 0, st>>>(inst, y, ld_y, out, total_n, k, ch);
  }
  return cudaGetLastError();
}

}  // namespace hodlr

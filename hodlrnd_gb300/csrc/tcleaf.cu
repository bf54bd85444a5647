// Leaf-level products for up to 64 right-hand sides (tc.h): the near tiles, the
// dense far tiles and the low-rank blocks of panels of at most 32 rows.
//
// These blocks are tiny (4D N = 65536: 2 million of 16 x 16 points and rank 8)
// and there is one pass to make over each, so what bounds them is the traffic
// and latency around the products, not the products.  As two phases through
// the tcgen05 kernels (tcgen05.cu) every block's z = V^T x went out to memory
// and back (512 bytes per z row, 8 GB in all against 0.9 GB of factors) and
// every step of 32 columns of a 16-row tile paid for staging, barriers and a
// tensor-memory round trip.  Here a warp owns a panel (or a run of its
// segments): its accumulators, 64 right-hand sides by up to 32 rows, stay in
// registers, and a block is applied whole -- z^T = x^T V into an accumulator
// fragment, which, scaled and split into BF16 high and low parts, already is
// the operand fragment of y^T += z^T U^T -- by register-level MMAs
// (mma.m16n8k16, BF16 operands, FP32 sums; the high and low parts of 8 columns
// make up one K = 16), whose 8-point pieces fit ragged leaves.  The inputs lie
// in memory as operand fragments (2 KB per 8 points, "units").  The 8 warps of a
// CTA take 8 panels next to each other -- siblings, mostly, with nearly the same
// sources -- and walk the union of their sources together: a batch of sources is
// staged in shared memory once for all of them by bulk copies (two stages), and
// each warp applies its own segments of the batch, asking for the next one's
// factors before it multiplies.
// 4D N = 65536, 64 right-hand sides: 2.1 ms against 5.3 for these blocks through
// the tcgen05 kernels (the whole product 7.28 -> 3.5 ms).  Of it 0.5 ms waits for
// factor loads; the rest is instructions (43% of the issue slots) and the padding
// of ranks, points and rows to 8.  Measured and not kept: sources read through L1
// by each warp (3.2 ms), records fetched by each warp (2.8 ms), prefetching the
// next batch's factors into L2 (2.2 ms).
#include <cuda_runtime.h>

#include <algorithm>

#include "device.cuh"
#include "tc.h"
#include "umma.cuh"

namespace hodlr {
namespace {

// c (16 x 8) += (high + low) B: A's columns 0-7 are the high parts (a.x, a.y),
// 8-15 the low parts (a.z, a.w) of the same 8 columns, B's rows 0-7 and 8-15 both
// the 8 x 8 matrix b.  Lane = 4 g + t holds A rows g, g + 8, columns 2 t, 2 t + 1,
// B rows 2 t, 2 t + 1 of column g, and C rows g (c0, c1) and g + 8 (c2, c3), columns
// 2 t, 2 t + 1.
__device__ __forceinline__ void mma16(float (&c)[4], const uint4& a, uint32_t b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %8}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b));
}
// c += d rounded to nearest: the MMA's own sum is cut off towards zero, which over
// the hundreds of blocks of a panel adds up (4D N = 65536, against the compensated
// product: 5.9e-6 with sums in the MMA, 2.4-3.3e-6 so; 2.03 -> 2.18 ms)
__device__ __forceinline__ void add4(float (&c)[4], const float (&d)[4]) {
#pragma unroll
  for (int q = 0; q < 4; q += 2)  // two additions in one instruction
    asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\t"
        "add.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "+f"(c[q]), "+f"(c[q + 1])
        : "f"(d[q]), "f"(d[q + 1]));
}
// 8 x 8 BF16 matrix transposed across the warp (lane 4 g + t: row g, columns 2 t, 2 t + 1)
__device__ __forceinline__ uint32_t transpose8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {  // BF16, rounded to nearest even
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float low_f(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float high_f(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
__device__ __forceinline__ uint32_t ldu16(const uint16_t* p) { return __ldg(p); }
// A stage: the sources' units, the batch's segment records, its header.  Shared
// memory of a CTA: the stages' full and empty barriers, the stop flag, then the
// stages.
constexpr int kLeafStages = 2;
constexpr int kLeafStop = 64;  // byte offset of the stop flag
constexpr int kStageSegs = kTcLeafUnits * kTcUnitBytes;
constexpr int kStageHead = kStageSegs + kTcLeafSegs * int(sizeof(TcLeafSeg));
constexpr int kStageBytes = kStageHead + int(sizeof(TcLeafBatch));
constexpr int kLeafSmem = 128 + kLeafStages * kStageBytes;
static_assert(sizeof(TcLeafSeg) % 16 == 0 && sizeof(TcLeafBatch) % 16 == 0 && kStageBytes % 16 == 0,
              "bulk copies: sizes and destinations are multiples of 16 bytes");

// A segment is applied in steps: 8 columns c .. c + 7 of U and V for a low-rank
// block, unit c (8 points) for a tile.  The factor values of a step, as loaded
// and one step ahead of their use (nothing is computed from them before then,
// so that no warp waits for them early): entries of U or of the tile for rows
// 8 nt + g, columns 2 t and 2 t + 1; V's rows of units 0 .. 3; scales.
template <int NT, bool NEAR>
struct LeafRaw;
template <int NT>
struct LeafRaw<NT, false> {
  uint32_t a[NT][2], v[4];
  float sc0, sc1;
};
template <int NT>
struct LeafRaw<NT, true> {
  double a[NT][2];
};

__device__ __forceinline__ uint32_t load_v(const TcLeafSeg& S, int c, int u, int lane) {
  const int j = 8 * u + (lane >> 2), k = c + 2 * (lane & 3);
  // V's rows hold vpad(rank) columns, a multiple of 8: those beyond the rank are masked when used
  return j < S.n && k < S.K ? __ldg(reinterpret_cast<const uint32_t*>(S.V + int64_t(j) * S.vstride + k)) : 0u;
}

template <int NT, bool NEAR>
__device__ __forceinline__ void load_step(const TcLeafSeg& S, int c, int m, int lane, LeafRaw<NT, NEAR>& L) {
  const int g = lane >> 2, t = lane & 3;
  if constexpr (NEAR) {
    const int j = 8 * c + 2 * t;
    const double* A = static_cast<const double*>(S.A) + int64_t(j) * m + g;
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      const bool in = 8 * nt + g < m;
      L.a[nt][0] = in && j < S.n ? __ldg(A + 8 * nt) : 0.0;
      L.a[nt][1] = in && j + 1 < S.n ? __ldg(A + m + 8 * nt) : 0.0;
    }
  } else {
    // columns k, k + 1 of U, or points k, k + 1 of a dense tile
    const bool lr = S.V != nullptr;
    const int k = (lr ? c : 8 * c) + 2 * t, K = lr ? S.K : S.n;
    const uint16_t* A = static_cast<const uint16_t*>(S.A) + k * m + g;
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      const bool in = 8 * nt + g < m;
      L.a[nt][0] = in && k < K ? ldu16(A + 8 * nt) : 0u;
      L.a[nt][1] = in && k + 1 < K ? ldu16(A + m + 8 * nt) : 0u;
    }
    L.sc0 = k < K ? __ldg(S.scale + k) : 0.f;
    L.sc1 = k + 1 < K ? __ldg(S.scale + k + 1) : 0.f;
    if (lr) {
#pragma unroll
      for (int u = 0; u < 4; u++) L.v[u] = load_v(S, c, u, lane);
    }
  }
}

// y^T (16 mtn right-hand sides x 8 NT rows) += one step of a segment; X: its
// source's units
template <int MT, int NT, bool NEAR>
__device__ __forceinline__ void leaf_step(const TcLeafSeg& S, int c, const LeafRaw<NT, NEAR>& L, const uint4* X, int lane,
                                          float (&acc)[MT][NT][4]) {
  const int t = lane & 3;
  if constexpr (NEAR) {
    // FP64 entries in three BF16 terms: a = t0 + t1 + t2 + O(2^-24 a)
    uint32_t b[NT][3];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      float f0 = float(L.a[nt][0]), f1 = float(L.a[nt][1]);
      b[nt][0] = pack2(f0, f1);
      f0 -= low_f(b[nt][0]);
      f1 -= high_f(b[nt][0]);
      b[nt][1] = pack2(f0, f1);
      b[nt][2] = pack2(f0 - low_f(b[nt][1]), f1 - high_f(b[nt][1]));
    }
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
      {
        const uint4 x = X[(c * 4 + mt) * 32];
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
          float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int q = 2; q >= 0; q--) mma16(d, x, b[nt][q]);
          add4(acc[mt][nt], d);
        }
      }
  } else if (S.V) {
    const int units = (S.n + 7) >> 3, k = c + 2 * t;
    float z[MT][4];
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int q = 0; q < 4; q++) z[mt][q] = 0.f;
    const uint32_t mask = k + 1 < S.K ? 0xffffffffu : 0x0000ffffu;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (u < units) {
        const uint32_t v = transpose8(L.v[u] & mask);
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
        mma16(z[mt], X[(u * 4 + mt) * 32], v);
      }
    }
    for (int u = 4; u < units; u++) {
      const uint32_t v = transpose8(load_v(S, c, u, lane) & mask);
#pragma unroll
      for (int mt = 0; mt < MT; mt++)
        mma16(z[mt], X[(u * 4 + mt) * 32], v);
    }
    uint32_t ub[NT];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) ub[nt] = L.a[nt][0] | (L.a[nt][1] << 16);
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
      {
        // z times its scale, in BF16 high and low parts (2^-17)
        const float z0 = z[mt][0] * L.sc0, z1 = z[mt][1] * L.sc1, z2 = z[mt][2] * L.sc0, z3 = z[mt][3] * L.sc1;
        uint4 zz;
        zz.x = pack2(z0, z1);
        zz.y = pack2(z2, z3);
        zz.z = pack2(z0 - low_f(zz.x), z1 - high_f(zz.x));
        zz.w = pack2(z2 - low_f(zz.y), z3 - high_f(zz.y));
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
          float d[4] = {0.f, 0.f, 0.f, 0.f};
          mma16(d, zz, ub[nt]);
          add4(acc[mt][nt], d);
        }
      }
  } else {
    // dense tile: stored entry times its column's scale in two BF16 terms (2^-16)
    uint32_t b[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      const float f0 = bf16_value(uint16_t(L.a[nt][0])) * L.sc0, f1 = bf16_value(uint16_t(L.a[nt][1])) * L.sc1;
      b[nt][0] = pack2(f0, f1);
      b[nt][1] = pack2(f0 - low_f(b[nt][0]), f1 - high_f(b[nt][0]));
    }
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
      {
        const uint4 x = X[(c * 4 + mt) * 32];
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
          float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int q = 1; q >= 0; q--) mma16(d, x, b[nt][q]);
          add4(acc[mt][nt], d);
        }
      }
  }
}

// One warp's share of a group's run of batches.  Every wait is bounded.  A warp
// that gives one up counts it in *a.status and raises the CTA's stop flag; from
// then on no warp reads a stage it has not seen complete, nothing more is
// copied, and warp 0 waits (again with a bound) for the copies in flight before
// it leaves.
template <int MT, int NT, bool NEAR>
__device__ __forceinline__ void leaf_run(const TcLeafArgs& a, const TcLeafRun& R, int m, float* out,
                                         unsigned char* smem, int wid, int lane) {
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + kLeafStages;
  volatile int* stop = reinterpret_cast<volatile int*>(smem + kLeafStop);
  unsigned char* ring = smem + 128;
  auto give_up = [&]() {
    if (lane == 0) {
      atomicAdd(a.status, 1u);
      *stop = 1;
    }
  };
  float acc[MT][NT > 0 ? NT : 1][4];
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int nt = 0; nt < NT; nt++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[mt][nt][q] = 0.f;
  const int nb = R.batch_e - R.batch_b;
  const TcLeafSeg* segs = NEAR ? a.near_segs : a.far_segs;
  // warp 0 copies a batch: its lanes a source's units each (they lie together),
  // lane 0 the segment records and the header
  auto issue = [&](int b) {
    if (b == a.drop_copies) return;
    const TcLeafBatch* B = a.batches + R.batch_b + b;
    unsigned char* stage = ring + (b % kLeafStages) * kStageBytes;
    uint64_t* bar = full + b % kLeafStages;
    const int q = B->src_b + lane, ns = B->warp_off[kTcLeafGroup];
    TcLeafSrc S{0, 0};
    if (q < B->src_e) S = a.srcs[q];
    const uint32_t bytes = uint32_t((S.n + 7) >> 3) * kTcUnitBytes;
    uint32_t off = bytes;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, off, o);
      if (lane >= o) off += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, off, 31);
    if (lane == 0) {
      const uint32_t sb = uint32_t(ns) * uint32_t(sizeof(TcLeafSeg));
      fence_proxy_async();
      mbar_expect_tx(bar, total + sb + uint32_t(sizeof(TcLeafBatch)));
      bulk_g2s(stage + kStageSegs, segs + B->seg_b, sb, bar);
      bulk_g2s(stage + kStageHead, B, uint32_t(sizeof(TcLeafBatch)), bar);
    }
    __syncwarp();
    if (bytes) bulk_g2s(stage + off - bytes, a.xunits + int64_t(S.xunit) * 128, bytes, bar);
  };
  int issued = min(kLeafStages, nb);  // warp 0's count of batches asked for
  if (wid == 0)
    for (int b = 0; b < issued; b++) issue(b);
  int b = 0;
  for (; b < nb; b++) {
    const int st = b % kLeafStages;
    const uint32_t phase = uint32_t(b / kLeafStages) & 1u;
    const unsigned char* stage = ring + st * kStageBytes;
    if (!__all_sync(0xffffffffu, mbar_wait(full + st, phase, a.wait_ns))) {
      give_up();
      break;
    }
    if (__any_sync(0xffffffffu, *stop != 0)) break;
    if constexpr (NT > 0) {
      const TcLeafBatch* H = reinterpret_cast<const TcLeafBatch*>(stage + kStageHead);
      const TcLeafSeg* rec = reinterpret_cast<const TcLeafSeg*>(stage + kStageSegs);
      int k = H->warp_off[wid], c = 0;
      const int ke = H->warp_off[wid + 1];
      if (k < ke) {
        TcLeafSeg S = rec[k];
        LeafRaw<NT, NEAR> L;
        load_step<NT, NEAR>(S, 0, m, lane, L);
        for (;;) {
          // the next step: of this segment, or of the next one
          TcLeafSeg Sn = S;
          int cn = !NEAR && S.V ? c + 8 : c + 1;
          bool more = true;
          if (cn >= (!NEAR && S.V ? S.K : (S.n + 7) >> 3)) {
            cn = 0;
            more = ++k < ke;
            if (more) Sn = rec[k];
          }
          LeafRaw<NT, NEAR> Ln;
          if (more) load_step<NT, NEAR>(Sn, cn, m, lane, Ln);
          const uint4* X = reinterpret_cast<const uint4*>(stage + S.unit * kTcUnitBytes) + lane;
          leaf_step<MT, NT, NEAR>(S, c, L, X, lane, acc);
          if (!more) break;
          S = Sn;
          c = cn;
          L = Ln;
        }
      }
    }
    __syncwarp();
    if (lane == 0 && !(wid == 1 && b == a.drop_release)) mbar_arrive(empty + st);
    if (wid == 0 && b + kLeafStages < nb) {
      // refilled once every warp has left the stage
      if (!__all_sync(0xffffffffu, mbar_wait(empty + st, phase, a.wait_ns))) {
        give_up();
        b++;  // this batch's copies are done
        break;
      }
      issue(b + kLeafStages);
      issued++;
    }
  }
  if (b < nb) {
    if (wid == 0)
      for (; b < issued; b++) mbar_wait(full + b % kLeafStages, uint32_t(b / kLeafStages) & 1u, a.wait_ns);
    return;
  }
  if constexpr (NT > 0) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
      {
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
          const int i = 8 * nt + 2 * t, r = 16 * mt + g;
          if (i < m) {
            out[i * kTcRhs + r] = acc[mt][nt][0];
            out[i * kTcRhs + r + 8] = acc[mt][nt][2];
          }
          if (i + 1 < m) {
            out[(i + 1) * kTcRhs + r] = acc[mt][nt][1];
            out[(i + 1) * kTcRhs + r + 8] = acc[mt][nt][3];
          }
        }
      }
  }
}

template <int MT>
__global__ void __launch_bounds__(kTcLeafGroup * 32, 2) tc_leaf_kernel(const TcLeafArgs a) {
  extern __shared__ __align__(128) unsigned char lsm[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const TcLeafRun R = a.runs[blockIdx.x];
  uint64_t* full = reinterpret_cast<uint64_t*>(lsm);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < kLeafStages; s++) {
      mbar_init(full + s, 1u);
      mbar_init(full + kLeafStages + s, kTcLeafGroup);
    }
    *reinterpret_cast<volatile int*>(lsm + kLeafStop) = 0;
    fence_mbar_init();
  }
  __syncthreads();
  const int p = wid < R.count ? R.panel0 + wid : -1;
  int m = 0;
  float* out = nullptr;
  if (p >= 0) {
    const int pi = R.near ? a.near_list[p] : a.far_list[p];
    const Panel P = R.near ? a.near_panels[pi] : a.far_panels[pi];
    m = P.m;
    out = R.part < 0 ? a.y + P.yoff * kTcRhs
                     : (R.near ? a.part_near : a.part_far) +
                           (int64_t(R.part) + int64_t(wid) * R.part_stride) * kTcRows * kTcRhs;
  }
  // per warp; at most 32 rows (host); without a panel the warp keeps the ring going
#define HODLR_LEAF_RUN(nt_)                              \
  case nt_:                                              \
    if (R.near)                                          \
      leaf_run<MT, nt_, true>(a, R, m, out, lsm, wid, lane); \
    else                                                 \
      leaf_run<MT, nt_, false>(a, R, m, out, lsm, wid, lane); \
    break;
  switch ((m + 7) >> 3) {
    HODLR_LEAF_RUN(1)
    HODLR_LEAF_RUN(2)
    HODLR_LEAF_RUN(3)
    HODLR_LEAF_RUN(4)
    default: leaf_run<MT, 0, false>(a, R, m, out, lsm, wid, lane); break;
  }
#undef HODLR_LEAF_RUN
}

// The sources' inputs as operand fragments: thread (unit, m-tile, lane) packs
// points 2 t, 2 t + 1 of the unit for right-hand sides 16 mt + g and + 8, high
// parts then low parts; points beyond the source are zero.
__global__ void __launch_bounds__(256) tc_units_kernel(const uint32_t* __restrict__ in, const TcUnit* __restrict__ units,
                                                       int64_t total, uint4* __restrict__ out) {
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < total; e += int64_t(gridDim.x) * blockDim.x) {
    const int lane = int(e & 31), mt = int((e >> 5) & 3);
    const TcUnit U = units[e >> 7];
    const int g = lane >> 2, t = lane & 3, r = 16 * mt + g;
    const uint32_t* p = in + (U.x_off + 2 * t) * kTcRhs + r;
    const bool ok0 = 2 * t < U.n, ok1 = 2 * t + 1 < U.n;
    const uint32_t w0 = ok0 ? p[0] : 0u, w1 = ok1 ? p[kTcRhs] : 0u;
    const uint32_t v0 = ok0 ? p[8] : 0u, v1 = ok1 ? p[kTcRhs + 8] : 0u;
    out[e] = make_uint4(__byte_perm(w0, w1, 0x5410), __byte_perm(v0, v1, 0x5410), __byte_perm(w0, w1, 0x7632),
                        __byte_perm(v0, v1, 0x7632));
  }
}

}  // namespace

cudaError_t launch_tc_units(const uint32_t* in, const TcUnit* units, int64_t nunits, uint4* out, cudaStream_t st) {
  if (nunits <= 0) return cudaSuccess;
  count_launches(1);
  const int64_t total = nunits * 128;
  tc_units_kernel<<<unsigned(std::min<int64_t>((total + 255) / 256, 152 * 16)), 256, 0, st>>>(in, units, total, out);
  return cudaGetLastError();
}

template <int MT>
static cudaError_t launch_leaf(const TcLeafArgs& a, cudaStream_t st) {
  const cudaError_t e = cudaFuncSetAttribute(tc_leaf_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLeafSmem);
  if (e != cudaSuccess) return e;
  count_launches(1);
  tc_leaf_kernel<MT><<<unsigned(a.nruns), kTcLeafGroup * 32, kLeafSmem, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_tc_leaf(const TcLeafArgs& a, int nrhs, cudaStream_t st) {
  if (a.nruns <= 0) return cudaSuccess;
  if (nrhs < 1 || nrhs > kTcRhs) return cudaErrorInvalidValue;
  // groups of 16 right-hand sides, known at compile time
  return nrhs <= 16 ? launch_leaf<1>(a, st) : nrhs <= 32 ? launch_leaf<2>(a, st) : launch_leaf<4>(a, st);
}

}  // namespace hodlr

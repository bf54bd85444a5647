// Restarted GMRES on the device (see gmres.h).
#include "cluster.cuh"
#include "device.cuh"
#include "fpsum.cuh"
#include "gmres.h"

#include <algorithm>
#include <cmath>

namespace hodlr {

namespace {

#define HODLR_TRY(x)                      \
  do {                                    \
    cudaError_t e_ = (x);                 \
    if (e_ != cudaSuccess) return e_;     \
  } while (0)

constexpr int kThreads = 256;

__device__ __forceinline__ double to_d(double v) { return v; }
__device__ __forceinline__ double to_d(float v) { return double(v); }

// a - h * b with one rounding per operation in FP64, rounded to T.
__device__ __forceinline__ double axmy(double a, double h, double b) { return __dsub_rn(a, __dmul_rn(h, b)); }

// Block-wide sum; every thread gets the result.
__device__ double block_sum(double v) {
  __shared__ double sh[kThreads / 32 + 1];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (wid == 0) {
    v = lane < kThreads / 32 ? sh[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) sh[kThreads / 32] = v;
  }
  __syncthreads();
  v = sh[kThreads / 32];
  __syncthreads();
  return v;
}

// Sum of the kVecCtas partials in a fixed order (each CTA gets the same value).
__device__ double reduce_parts(const double* part) {
  double v = 0.0;
  for (int i = threadIdx.x; i < kVecCtas; i += kThreads) v += part[i];
  return block_sum(v);
}

template <typename T>
__global__ void __launch_bounds__(kThreads) dot_partial_kernel(const T* a, const T* b, int64_t n, double* part) {
  double acc = 0.0;
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n; i += int64_t(kVecCtas) * kThreads)
    acc += to_d(a[i]) * to_d(b[i]);
  acc = block_sum(acc);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// partials of |sum_{s = s0}^{s1 - 1} y[s * n + i]|^2 over i
template <typename T>
__global__ void __launch_bounds__(kThreads) slots_partial_kernel(const T* y, int64_t n, int s0, int s1, double* part) {
  double acc = 0.0;
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n; i += int64_t(kVecCtas) * kThreads) {
    double v = 0.0;
    for (int s = s0; s < s1; s++) v += to_d(y[int64_t(s) * n + i]);
    acc += v * v;
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// h = <w, v_k> from part_in; w -= h v_k; part_out = partials of <w, next>.
template <typename T>
__global__ void __launch_bounds__(kThreads)
    mgs_step_kernel(T* w, const T* vk, const T* next, int64_t n, const double* part_in, double* part_out, double* hout) {
  const double h = reduce_parts(part_in);
  if (blockIdx.x == 0 && threadIdx.x == 0) *hout = h;
  double acc = 0.0;
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n; i += int64_t(kVecCtas) * kThreads) {
    const T wi = T(axmy(to_d(w[i]), h, to_d(vk[i])));
    w[i] = wi;
    acc += to_d(wi) * to_d(next ? next[i] : wi);
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) part_out[blockIdx.x] = acc;
}

// Classical Gram-Schmidt, one pass (applied twice per Arnoldi step: CGS2).
// Its O(n * nv) products run on the FP32 pipe: GB300's FP64 pipe, not HBM,
// bounded the FP64 versions (84% FP64-pipe busy, 12% of DRAM bandwidth).
// Each FP64 value is split into two floats from its bits alone (split_d,
// device.cuh),
// products are formed as in Dot2 (Ogita, Rump and Oishi, SIAM J. Sci.
// Comput. 26 (2005)): the product of the high parts exactly by FMA, the cross
// terms rounded, every addition's error kept.  Dots and updates come out
// within about 1e-14 of the exact values (FP64 summation of the same terms
// is within n * 1.1e-16); only O(n) operations stay on the FP64 pipe.

__device__ __forceinline__ float2 split_t(double a) { return split_d(a); }
__device__ __forceinline__ float2 split_t(float a) { return make_float2(a, 0.f); }

// cgs_dots: part[j * kVecCtas + cta] = this CTA's share of <w, v_j> for
// j < nv and cta < kDotCtas.  Grid kDotCtas x ceil(nv / 8): CTA (cta, g)
// takes vectors 8g .. 8g + 7, so every group runs at once and each thread
// keeps eight loads in flight over about n / (kDotCtas * 256) elements; the
// CTA's sums are combined as FP32 pairs (the FP64 pipe would bound a
// reduction in FP64), and a partial's summation order depends only on cta.
constexpr int kDotGroup = 8;
constexpr int kDotCtas = 152;
template <typename T>
__global__ void __launch_bounds__(kThreads)
    cgs_dots_kernel(const T* __restrict__ w, const T* __restrict__ V, int64_t n, int nv, double* __restrict__ part) {
  constexpr int U = kDotGroup;
  __shared__ float shs[U][kThreads / 32], shc[U][kThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int j0 = blockIdx.y * U;
  const int jn = min(U, nv - j0);
  float as[U], ac[U];
#pragma unroll
  for (int u = 0; u < U; u++) as[u] = ac[u] = 0.f;
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n; i += int64_t(kDotCtas) * kThreads) {
    const float2 wi = split_t(w[i]);
#pragma unroll
    for (int u = 0; u < U; u++)
      if (u < jn) dot2_add(as[u], ac[u], split_t(V[int64_t(j0 + u) * n + i]), wi);
  }
#pragma unroll
  for (int u = 0; u < U; u++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      pair_add(as[u], ac[u], __shfl_xor_sync(0xffffffffu, as[u], o), __shfl_xor_sync(0xffffffffu, ac[u], o));
    if (lane == 0) {
      shs[u][wid] = as[u];
      shc[u][wid] = ac[u];
    }
  }
  __syncthreads();
  if (threadIdx.x < jn) {
    float vs = 0.f, vc = 0.f;
    for (int q = 0; q < kThreads / 32; q++) pair_add(vs, vc, shs[threadIdx.x][q], shc[threadIdx.x][q]);
    part[int64_t(j0 + threadIdx.x) * kVecCtas + blockIdx.x] = __dadd_rn(double(vs), double(vc));
  }
}

// Sum of the first kDotCtas partials in a fixed order (each CTA gets the same value).
__device__ double reduce_dot_parts(const double* part) {
  double v = 0.0;
  for (int i = threadIdx.x; i < kDotCtas; i += kThreads) v += part[i];
  return block_sum(v);
}

// One CTA per basis vector j: hc[j] = <w, v_j> from the partial sums (fixed
// order); the Hessenberg column gets hc (first pass) or hc added (second).
__global__ void __launch_bounds__(kThreads)
    cgs_reduce_kernel(const double* __restrict__ part, double* __restrict__ hc, double* __restrict__ hcol, int second) {
  const int j = blockIdx.x;
  const double v = reduce_dot_parts(part + int64_t(j) * kVecCtas);
  if (threadIdx.x == 0) {
    hc[j] = v;
    hcol[j] = second ? __dadd_rn(hcol[j], v) : v;
  }
}

// w -= sum_j hc[j] v_j: the sum of the products as above, then one FP64
// subtraction, rounded to T once; with part, also the partial sums of |w|^2
// for the normalisation (as FP32 pairs until one FP64 value per CTA).
// nv <= kMaxBasis (the restart length + 1).
constexpr int kMaxBasis = 1001;
template <typename T>
__global__ void __launch_bounds__(kThreads) cgs_update_kernel(T* __restrict__ w, const T* __restrict__ V, int64_t n,
                                                              int nv, const double* __restrict__ hc,
                                                              double* __restrict__ part) {
  __shared__ float2 hs[kMaxBasis];
  __shared__ float ps[kThreads / 32], pc[kThreads / 32];
  for (int j = threadIdx.x; j < nv; j += kThreads) hs[j] = split_d(hc[j]);
  __syncthreads();
  float ns = 0.f, nc = 0.f;
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n; i += int64_t(kVecCtas) * kThreads) {
    float s = 0.f, c = 0.f;
#pragma unroll 8
    for (int j = 0; j < nv; j++) dot2_add(s, c, split_t(V[int64_t(j) * n + i]), hs[j]);
    const T t = T(__dsub_rn(to_d(w[i]), __dadd_rn(double(s), double(c))));
    w[i] = t;
    const float2 ts = split_t(t);
    dot2_add(ns, nc, ts, ts);
  }
  if (part) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      pair_add(ns, nc, __shfl_xor_sync(0xffffffffu, ns, o), __shfl_xor_sync(0xffffffffu, nc, o));
    if (lane == 0) {
      ps[wid] = ns;
      pc[wid] = nc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      float vs = 0.f, vc = 0.f;
      for (int q = 0; q < kThreads / 32; q++) pair_add(vs, vc, ps[q], pc[q]);
      part[blockIdx.x] = __dadd_rn(double(vs), double(vc));
    }
  }
}

// h = sqrt(<w, w>) from part; v_next = (1 / h) * w (GMRES.hpp:241-242).
template <typename T>
__global__ void __launch_bounds__(kThreads)
    normalize_kernel(const T* w, T* vnext, int64_t n, const double* ih_ptr) {
  const double ih = *ih_ptr;
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n; i += int64_t(kVecCtas) * kThreads)
    vnext[i] = T(__dmul_rn(ih, to_d(w[i])));
}

// h = sqrt(<w, w>) from part into *hout and 1 / h into *ihout, once (one CTA):
// every CTA of normalize_kernel then multiplies by the same value without
// summing the partials and dividing itself.
__global__ void __launch_bounds__(kThreads) norm_recip_kernel(const double* part, double* hout, double* ihout) {
  const double h = sqrt(reduce_parts(part));
  if (threadIdx.x == 0) {
    *hout = h;
    *ihout = 1.0 / h;
  }
}

// v0 = r * (1 / beta) (GMRES.hpp:220); s = beta e_0.
template <typename T>
__global__ void __launch_bounds__(kThreads)
    start_cycle_kernel(const T* r, T* v0, int64_t n, const double* scal, double* s, int restart) {
  const double ib = 1.0 / scal[1];
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n; i += int64_t(kVecCtas) * kThreads)
    v0[i] = T(__dmul_rn(to_d(r[i]), ib));
  if (blockIdx.x == 0)
    for (int k = threadIdx.x; k <= restart; k += kThreads) s[k] = k == 0 ? scal[1] : 0.0;
}

__device__ __forceinline__ void apply_rot(double& dx, double& dy, double cs, double sn) {
  const double t = __dadd_rn(__dmul_rn(cs, dx), __dmul_rn(sn, dy));
  dy = __dadd_rn(__dmul_rn(-sn, dx), __dmul_rn(cs, dy));
  dx = t;
}

__device__ __forceinline__ void gen_rot(double dx, double dy, double& cs, double& sn) {
  if (dy == 0.0) {
    cs = 1.0;
    sn = 0.0;
  } else if (fabs(dy) > fabs(dx)) {
    const double t = dx / dy;
    sn = 1.0 / sqrt(__dadd_rn(1.0, __dmul_rn(t, t)));
    cs = __dmul_rn(t, sn);
  } else {
    const double t = dy / dx;
    cs = 1.0 / sqrt(__dadd_rn(1.0, __dmul_rn(t, t)));
    sn = __dmul_rn(t, cs);
  }
}

// Rotations for column i of H and the residual estimate (GMRES.hpp:244-250).
// The running entry stays in a register (H and rot do not alias), so the
// loads of the next entry and rotation are not held up by the stores.
__global__ void givens_kernel(double* __restrict__ H, int ldh, double* __restrict__ rot, int restart, int i,
                              double* __restrict__ scal) {
  double* cs = rot;
  double* sn = rot + (restart + 1);
  double* s = rot + 2 * (restart + 1);
  double* h = H + int64_t(i) * ldh;
  double hk = h[0];
  for (int k = 0; k < i; k++) {
    double hk1 = h[k + 1];
    apply_rot(hk, hk1, cs[k], sn[k]);
    h[k] = hk;
    hk = hk1;
  }
  double hi1 = h[i + 1];
  gen_rot(hk, hi1, cs[i], sn[i]);
  apply_rot(hk, hi1, cs[i], sn[i]);
  h[i] = hk;
  h[i + 1] = hi1;
  apply_rot(s[i], s[i + 1], cs[i], sn[i]);
  scal[0] = fabs(s[i + 1]) / scal[2];
}

// ---- one Arnoldi step in one launch ------------------------------------------
// Everything after the product A v_i -- the orthogonalisation, the norm,
// v_{i+1}, the rotations and the residual estimate -- in one kernel, for
// vectors short enough that the separate kernels are all start-up (MGS: i + 2
// launches of 4-8 us; CGS2: nine, 65 us at n = 20011).

// The rotations and the residual estimate (givens_kernel) by one thread, from
// shared memory: first the earlier rotations cs, sn applied to the Hessenberg
// column h[0 .. i] (hcol gets its entries 0 .. i - 1; the running entry i is
// returned), then, once the column's last entry hn is known, the new rotation.
__device__ __forceinline__ double step_rotate(const double* h, const double* cs, const double* sn, int i, double* hcol) {
  double hk = h[0];
  for (int k = 0; k < i; k++) {
    double hk1 = h[k + 1];
    apply_rot(hk, hk1, cs[k], sn[k]);
    hcol[k] = hk;
    hk = hk1;
  }
  return hk;
}
__device__ __forceinline__ void step_new_rotation(double hk, double hn, int i, double* hcol, double* rot, int restart,
                                                  double* scal, double* hres) {
  double* rcs = rot;
  double* rsn = rot + (restart + 1);
  double* rs = rot + 2 * (restart + 1);
  double hi1 = hn, c, s;
  gen_rot(hk, hi1, c, s);
  apply_rot(hk, hi1, c, s);
  rcs[i] = c;
  rsn[i] = s;
  hcol[i] = hk;
  hcol[i + 1] = hi1;
  double s0 = rs[i], s1 = rs[i + 1];
  apply_rot(s0, s1, c, s);
  rs[i] = s0;
  rs[i + 1] = s1;
  const double res = fabs(s1) / scal[2];
  scal[0] = res;
  *hres = res;
}

template <typename T>
struct StepArgs {
  T* w;
  T* V;
  int64_t n;
  int i;        // Arnoldi index: w against v_0 .. v_i, v_{i+1} written
  double* H;
  int ldh;
  double* rot;
  int restart;  // the allocated one (rot's layout)
  double* scal;
  double* hres;  // host-visible: [0] residual estimate, [1] nonzero after a wait gave up
  // CGS2
  float2* part;             // kStepMaxBasis x kStepGrid partial pairs, two sets, and the norm's
  unsigned long long* bar;  // grid barrier arrivals
  int cached;               // the basis slices fit in shared memory
  uint64_t wait_ns;         // longest wait at a barrier
  int phase;                // one phase per launch: which
  int redo;                 // a one-launch attempt of this step gave up
};

// MGS: a cluster of CTAs (16, or 8 where 16 do not fit), each with a slice of
// the vectors; w stays in registers and the next basis vector is loaded before
// the sum is waited for.  A sum over the cluster is one store per CTA into
// every other CTA's shared memory and a hardware cluster barrier.  FP64
// operations (16 cycles a warp on an SM) bound the rest, so a CTA has few
// threads with up to 8 elements each, and one warp finishes each sum.
// About 3 us per basis vector (n = 10000, 19 steps: 33 us a step against 100 for
// the separate kernels); with 640 one-element threads per CTA the FP64 sums of
// idle-handed warps made it 8 us.
constexpr int64_t kStepMaxN = 40960;
constexpr int kStepMaxBasis = 256;  // restart + 1 at most
constexpr int kStepCtas = 16;
constexpr int kStepEpt = 8;         // elements per thread at most
constexpr int kStepThreads = 640;   // 8 CTAs x 640 x 8 = kStepMaxN

__host__ __device__ inline int64_t step_slice(int64_t n, int ctas) { return (n + ctas - 1) / ctas; }

template <typename T>
__global__ void __launch_bounds__(kStepThreads, 1) mgs_cluster_kernel(const StepArgs<T> a) {
  __shared__ double slots[2][kStepCtas];  // the CTAs' sums, used in turn
  __shared__ double red[kStepThreads / 32], total;
  __shared__ double h[kStepMaxBasis], cs[kStepMaxBasis], sn[kStepMaxBasis];
  const uint32_t me = cluster_rank(), nc = cluster_size();
  const int64_t E = step_slice(a.n, int(nc)), e0 = int64_t(me) * E;
  const int cnt = int(max(int64_t(0), min(E, a.n - e0)));
  const int t = threadIdx.x, nt = blockDim.x, nv = a.i + 1;
  const int lane = t & 31, wid = t >> 5, nw = nt >> 5;
  T* V = a.V + e0;
  if (me == 0)
    for (int k = t; k < a.i; k += nt) {
      cs[k] = a.rot[k];
      sn[k] = a.rot[a.restart + 1 + k];
    }
  T wr[kStepEpt], vr[kStepEpt], vn[kStepEpt];
#pragma unroll
  for (int q = 0; q < kStepEpt; q++) {
    const int e = t + q * nt;
    wr[q] = e < cnt ? a.w[e0 + e] : T(0);
    vr[q] = e < cnt ? V[e] : T(0);
    vn[q] = T(0);
  }
  double acc = 0.0;
#pragma unroll
  for (int q = 0; q < kStepEpt; q++)
    if (q * nt < cnt) acc += to_d(wr[q]) * to_d(vr[q]);
  // no CTA stores into another's shared memory before that one has started
  cluster_barrier();
  int set = 0;
  // the sum of acc over the cluster, the same value in every thread
  auto cluster_sum = [&](double v) -> double {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (wid == 0) {
      v = lane < nw ? red[lane] : 0.0;
      for (int o = 16; o > 0; o >>= 1)
        if (o < nw) v += __shfl_xor_sync(0xffffffffu, v, o);
      v = __shfl_sync(0xffffffffu, v, 0);
      if (lane < int(nc)) cluster_store(cluster_addr(&slots[set][me], uint32_t(lane)), v);
    }
    cluster_barrier();
    if (wid == 0) {
      v = lane < int(nc) ? slots[set][lane] : 0.0;
#pragma unroll
      for (int o = kStepCtas / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) total = v;
    }
    set ^= 1;
    __syncthreads();
    return total;
  };
  for (int k = 0; k < nv; k++) {
    if (k + 1 < nv) {
      const T* vk = V + int64_t(k + 1) * a.n;
#pragma unroll
      for (int q = 0; q < kStepEpt; q++) {
        const int e = t + q * nt;
        if (e < cnt) vn[q] = vk[e];
      }
    }
    const double hk = cluster_sum(acc);
    if (t == 0) h[k] = hk;
    acc = 0.0;
#pragma unroll
    for (int q = 0; q < kStepEpt; q++) {
      if (q * nt < cnt) {
        wr[q] = T(axmy(to_d(wr[q]), hk, to_d(vr[q])));
        vr[q] = vn[q];
        acc += to_d(wr[q]) * to_d(k + 1 < nv ? vr[q] : wr[q]);
      }
    }
  }
  const double hn = sqrt(cluster_sum(acc));
  const double ih = 1.0 / hn;
  T* out = V + int64_t(nv) * a.n;
#pragma unroll
  for (int q = 0; q < kStepEpt; q++) {
    const int e = t + q * nt;
    if (e < cnt) out[e] = T(__dmul_rn(ih, to_d(wr[q])));
  }
  if (me == 0 && t == 0) {
    double* hcol = a.H + int64_t(a.i) * a.ldh;
    step_new_rotation(step_rotate(h, cs, sn, a.i, hcol), hn, a.i, hcol, a.rot, a.restart, a.scal, a.hres);
  }
}

// CGS2: every SM has a slice of the vectors (a cooperative launch, whose CTAs
// meet at three grid barriers): the projections of a pass are each CTA's
// partial pairs, summed by every CTA after the barrier.  The products are those
// of cgs_dots_kernel and cgs_update_kernel (dot2_add, pair_add, one FP64
// subtraction per element and pass); the basis slices are split once into
// shared memory where they fit and serve both passes from there.
// n = 20011, 50 basis vectors: 37 us a step against 75 for the nine kernels; a
// cluster of 16 CTAs took 105 (its 16 SMs are bound by the splits and products).
// When other work holds some SMs for longer than kBarrierNs, a barrier gives up,
// and the step is done again in four launches that need no CTA beside another
// one: the same operations in the same order, so the results are the same to the last bit.
constexpr int kStepGrid = 152;
constexpr int kCgsThreads = 512;
constexpr int kCgsWarps = kCgsThreads / 32;
constexpr int kCgsSliceBytes = 128 * 1024;  // basis slices in shared memory at most

// a slice: a multiple of 32 elements
__host__ __device__ inline int cgs_slice(int64_t n) { return int((step_slice(n, kStepGrid - 1) + 31) / 32 * 32); }
// CTAs: one per slice and one for the rotations, kStepGrid at most
__host__ inline int cgs_grid(int64_t n) { return int((n + cgs_slice(n) - 1) / cgs_slice(n)) + 1; }
__host__ inline size_t cgs_smem(int64_t n, int nv, bool cached) {
  return size_t(cgs_slice(n)) * (sizeof(double) + sizeof(float2)) + (cached ? size_t(nv) * cgs_slice(n) * sizeof(float2) : 0);
}

// Arrives at the grid barrier and waits for every CTA (at most wait_ns); false
// after a give-up.
__device__ __forceinline__ bool grid_barrier(unsigned long long* bar, uint64_t wait_ns) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned long long g = gridDim.x, mine = atomicAdd(bar, 1ull), goal = (mine / g + 1) * g;
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    int good = 1;
    for (;;) {
      unsigned long long v;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(bar) : "memory");
      if (v >= goal) break;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
      if (t1 - t0 > wait_ns) {
        good = 0;
        break;
      }
    }
    __threadfence();
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// The sum of the G CTAs' partial pairs at part, by 8 lanes (each gets it; a warp
// takes four sums at a time, which all its lanes ask for).  Summed as FP32
// triples: more accurate than FP64 sums, and off the FP64 pipe, which a sum per
// basis vector on every SM would hold up.  Sums beyond FP32's range are formed in
// FP64.
__device__ __forceinline__ double sum_step_parts(const float2* part, int G, int lane) {
  const int sub = lane & 7;
  constexpr int Q = kStepGrid / 8;
  float2 p[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) p[q] = sub + 8 * q < G ? __ldcg(part + sub + 8 * q) : make_float2(0.f, 0.f);
  TripleSum a;
#pragma unroll
  for (int q = 0; q < Q; q++) {
    if (8 * q >= G) break;
    a.add(p[q].x, p[q].y);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
    a.add(__shfl_xor_sync(0xffffffffu, a.s, o), __shfl_xor_sync(0xffffffffu, a.c, o),
          __shfl_xor_sync(0xffffffffu, a.t, o));
  if (!__any_sync(0xffffffffu, !a.finite())) return a.value();
  double v = 0.0;
  for (int c = sub; c < G; c += 8) {
    const float2 p = __ldcg(part + c);
    v += __dadd_rn(double(p.x), double(p.y));
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
static_assert(kStepGrid % 8 == 0, "shares of 8 lanes");

// GRID: the whole step (a cooperative launch); else phase a.phase of it, after
// which w and the partial sums are in memory:
//   0: the first pass's projections
//   1: their sums and update, the second pass's projections
//   2: their sums and update, the earlier rotations, |w|'s share
//   3: |w|, v_{i+1}, the new rotation
// scal[5]: the right-hand side's entry i before the step, scal[6]: the column's
// running entry after the earlier rotations.
template <typename T, bool GRID>
__global__ void __launch_bounds__(kCgsThreads, 1) cgs2_step_kernel(const StepArgs<T> a) {
  extern __shared__ __align__(16) unsigned char csm[];
  __shared__ double h[kStepMaxBasis], cs[kStepMaxBasis], sn[kStepMaxBasis];
  __shared__ float2 hs[kStepMaxBasis], pairs[kCgsThreads];
  __shared__ double nrm;
  const int E = cgs_slice(a.n), G = gridDim.x, cta = blockIdx.x;
  const int64_t e0 = int64_t(cta) * E;
  const int cnt = int(max(int64_t(0), min(int64_t(E), a.n - e0)));
  double* wd = reinterpret_cast<double*>(csm);
  float2* sw = reinterpret_cast<float2*>(wd + E);
  float2* sv = sw + E;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nv = a.i + 1;
  T* V = a.V + e0;
  // the last CTA has no slice: it applies the earlier rotations to the column
  // while the others form the second pass's update (one thread, a chain of FP64
  // operations, 8 us at 50 columns)
  const bool rotor = cta == G - 1;
  double hk = 0.0;
  auto run = [&](int phase) { return GRID || a.phase == phase; };
  if (rotor && t == 0) {
    double* rs = a.rot + 2 * (a.restart + 1);
    if (GRID) {
      a.scal[5] = rs[a.i];
    } else if (a.phase == 0 && a.redo) {  // the attempt's rotation may have been applied
      rs[a.i] = a.scal[5];
      rs[a.i + 1] = 0.0;
    }
  }
  if (rotor)
    for (int k = t; k < a.i; k += kCgsThreads) {
      cs[k] = a.rot[k];
      sn[k] = a.rot[a.restart + 1 + k];
    }
  for (int e = t; e < E; e += kCgsThreads) {
    const T v = e < cnt ? a.w[e0 + e] : T(0);
    wd[e] = to_d(v);
    sw[e] = split_t(v);
  }
  const bool cached = GRID && a.cached;
  if (cached && !rotor) {
    for (int q = wid; q < nv; q += kCgsWarps)
#pragma unroll 4
      for (int e = lane; e < E; e += 32) sv[q * E + e] = e < cnt ? split_t(V[int64_t(q) * a.n + e]) : make_float2(0.f, 0.f);
  }
  __syncthreads();
  // the update's warps: EG groups of 32 elements by JG shares of the vectors
  const int EG = E / 32, JG = max(1, kCgsWarps / EG);
  const int eg0 = wid % min(EG, kCgsWarps), jg = wid / min(EG, kCgsWarps);
  float ns = 0.f, nk = 0.f;
  for (int pass = 0; pass < 2; pass++) {
    float2* part = a.part + int64_t(pass) * kStepMaxBasis * kStepGrid;
    for (int j = run(pass) ? wid : nv; j < nv; j += kCgsWarps) {
      float as = 0.f, ac = 0.f;
      if (rotor) {
      } else if (cached) {
        const float2* vj = sv + j * E;
#pragma unroll 4
        for (int e = lane; e < E; e += 32) dot2_add(as, ac, vj[e], sw[e]);
      } else {
        const T* vj = V + int64_t(j) * a.n;
#pragma unroll 8
        for (int e = lane; e < cnt; e += 32) dot2_add(as, ac, split_t(vj[e]), sw[e]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        pair_add(as, ac, __shfl_xor_sync(0xffffffffu, as, o), __shfl_xor_sync(0xffffffffu, ac, o));
      if (lane == 0) __stcg(part + int64_t(j) * kStepGrid + cta, make_float2(as, ac));
    }
    if (GRID && !grid_barrier(a.bar, a.wait_ns)) {
      if (t == 0) a.hres[1] = 1.0;
      return;
    }
    if (!run(pass + 1)) continue;
    for (int j0 = wid * 4; j0 < nv; j0 += kCgsWarps * 4) {
      const int j = min(j0 + (lane >> 3), nv - 1);
      const double v = sum_step_parts(part + int64_t(j) * kStepGrid, G, lane);
      double first = 0.0;  // the first pass's, for the column
      if (pass && rotor) first = GRID ? h[j] : sum_step_parts(a.part + int64_t(j) * kStepGrid, G, lane);
      if ((lane & 7) == 0 && j == j0 + (lane >> 3)) {
        h[j] = pass ? __dadd_rn(first, v) : v;
        hs[j] = split_d(v);
      }
    }
    __syncthreads();
    if (rotor) {
      if (pass && t == 0) {
        hk = step_rotate(h, cs, sn, a.i, a.H + int64_t(a.i) * a.ldh);
        if (!GRID) a.scal[6] = hk;
      }
      continue;
    }
    for (int b = 0; b < EG; b += kCgsWarps) {
      const int eg = b + eg0, e = eg * 32 + lane;
      const bool act = eg < EG && jg < JG;
      float s = 0.f, c = 0.f;
      if (act && e < cnt) {
        if (cached) {
#pragma unroll 4
          for (int j = jg; j < nv; j += JG) dot2_add(s, c, sv[j * E + e], hs[j]);
        } else {
#pragma unroll 8
          for (int j = jg; j < nv; j += JG) dot2_add(s, c, split_t(V[int64_t(j) * a.n + e]), hs[j]);
        }
      }
      pairs[t] = make_float2(s, c);
      __syncthreads();
      if (act && jg == 0 && e < cnt) {
        for (int g = 1; g < JG; g++) {
          const float2 q = pairs[(g * min(EG, kCgsWarps) + eg0) * 32 + lane];
          pair_add(s, c, q.x, q.y);
        }
        const T v = T(__dsub_rn(wd[e], __dadd_rn(double(s), double(c))));
        const float2 vs = split_t(v);
        wd[e] = to_d(v);
        sw[e] = vs;
        if (!GRID) a.w[e0 + e] = v;
        if (pass) dot2_add(ns, nk, vs, vs);
      }
      __syncthreads();
    }
  }
  // |w|: the CTA's pair, then every CTA's
  float2* npart = a.part + int64_t(2) * kStepMaxBasis * kStepGrid;
  if (run(2)) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      pair_add(ns, nk, __shfl_xor_sync(0xffffffffu, ns, o), __shfl_xor_sync(0xffffffffu, nk, o));
    if (lane == 0) pairs[wid] = make_float2(ns, nk);
    __syncthreads();
    if (t == 0) {
      ns = nk = 0.f;
      for (int q = 0; q < kCgsWarps; q++) pair_add(ns, nk, pairs[q].x, pairs[q].y);
      __stcg(npart + cta, make_float2(ns, nk));  // the last CTA's is zero, as its projections are
    }
  }
  if (GRID && !grid_barrier(a.bar, a.wait_ns)) {
    if (t == 0) a.hres[1] = 1.0;
    return;
  }
  if (!run(3)) return;
  if (wid == 0) {
    const double v = sum_step_parts(npart, G, lane);
    if (lane == 0) nrm = v;
  }
  __syncthreads();
  const double hn = sqrt(nrm);
  const double ih = 1.0 / hn;
  T* out = V + int64_t(nv) * a.n;
  for (int e = t; e < cnt; e += kCgsThreads) out[e] = T(__dmul_rn(ih, wd[e]));
  if (rotor && t == 0)
    step_new_rotation(GRID ? hk : a.scal[6], hn, a.i, a.H + int64_t(a.i) * a.ldh, a.rot, a.restart, a.scal, a.hres);
}

// What the MGS cluster of c CTAs is launched with.
cudaLaunchConfig_t mgs_config(int64_t n, int c, cudaLaunchAttribute* at, cudaStream_t st) {
  const int64_t E = step_slice(n, c);
  cudaLaunchConfig_t cfg{};
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = unsigned(c);
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg.gridDim = dim3(unsigned(c));
  // about 5 elements per thread, 8 at most
  cfg.blockDim = dim3(unsigned(std::min<int64_t>(kStepThreads, std::max<int64_t>(128, (E / 5 + 31) / 32 * 32))));
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// CTAs of the MGS cluster for vectors of n elements on this device; 0: the
// separate kernels.
template <typename T>
int mgs_ctas(int64_t n) {
  if (n > kStepMaxN) return 0;
  for (int c : {kStepCtas, kStepCtas / 2}) {
    cudaLaunchAttribute at{};
    const cudaLaunchConfig_t cfg = mgs_config(n, c, &at, nullptr);
    int clusters = 0;
    if (cudaFuncSetAttribute(&mgs_cluster_kernel<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&clusters, &mgs_cluster_kernel<T>, &cfg) == cudaSuccess && clusters > 0)
      return c;
    cudaGetLastError();
  }
  return 0;
}

// Whether the CGS2 step kernel takes vectors of n elements on this device.
template <typename T>
bool cgs_step_fits(int64_t n) {
  if (n > kStepMaxN) return false;
  int dev = 0, sms = 0, coop = 0, per = 0;
  const bool ok =
      cudaGetDevice(&dev) == cudaSuccess &&
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
      cudaFuncSetAttribute(&cgs2_step_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           int(kCgsSliceBytes + cgs_smem(kStepMaxN, 0, false))) == cudaSuccess &&
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, &cgs2_step_kernel<T, true>, kCgsThreads,
                                                    kCgsSliceBytes + cgs_smem(n, 0, false)) == cudaSuccess &&
      int64_t(per) * sms >= cgs_grid(n);
  if (!ok) cudaGetLastError();
  return ok;
}

template <typename T>
cudaError_t launch_mgs_step(const StepArgs<T>& a, int ctas, cudaStream_t st) {
  cudaLaunchAttribute at{};
  const cudaLaunchConfig_t cfg = mgs_config(a.n, ctas, &at, st);
  count_launches(1);
  return cudaLaunchKernelEx(&cfg, &mgs_cluster_kernel<T>, a);
}

template <typename T>
cudaError_t launch_cgs_step(StepArgs<T> a, cudaStream_t st) {
  const size_t basis = size_t(a.i + 1) * size_t(cgs_slice(a.n)) * sizeof(float2);
  a.cached = basis <= size_t(kCgsSliceBytes);
  count_launches(1);
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(&cgs2_step_kernel<T, true>), dim3(unsigned(cgs_grid(a.n))),
                                     dim3(kCgsThreads), args, cgs_smem(a.n, a.i + 1, a.cached != 0), st);
}

// The same step in four launches.
template <typename T>
cudaError_t launch_cgs_phases(StepArgs<T> a, bool redo, cudaStream_t st) {
  a.redo = redo;
  for (a.phase = 0; a.phase < 4; a.phase++) {
    count_launches(1);
    cgs2_step_kernel<T, false>
        <<<unsigned(cgs_grid(a.n)), kCgsThreads, cgs_smem(a.n, a.i + 1, false), st>>>(a);
  }
  return cudaGetLastError();
}

// Update (GMRES.hpp:132-146): back substitution into y.
// One CTA: thread j keeps y_j and subtracts column i of H times y_i as soon as y_i
// is known, the operations of the serial loop in its order; the next column is
// loaded meanwhile.  k < kMaxBasis <= 1024.
// 100 columns: 44 us against 428 for one thread (19: 14 us against 43).
static_assert(kMaxBasis <= 1024, "a thread per column");
__global__ void __launch_bounds__(1024) backsolve_kernel(const double* __restrict__ H, int ldh, double* rot, int restart,
                                                         int k) {
  __shared__ double yi[2];
  const double* s = rot + 2 * (restart + 1);
  double* y = rot + 3 * (restart + 1);
  const int j = threadIdx.x;
  double v = j <= k ? s[j] : 0.0;
  double hc = j <= k ? H[j + int64_t(k) * ldh] : 0.0, hn = 0.0;
  for (int i = k; i >= 0; i--) {
    if (j < i) hn = H[j + int64_t(i - 1) * ldh];
    if (j == i) {
      v = v / hc;
      yi[i & 1] = v;
      y[i] = v;
    }
    __syncthreads();
    if (j < i) {
      v = __dsub_rn(v, __dmul_rn(hc, yi[i & 1]));
      hc = hn;
    }
  }
}

void launch_backsolve(const double* H, int ldh, double* rot, int restart, int k, cudaStream_t st) {
  count_launches(1);
  backsolve_kernel<<<1, unsigned((k + 32) / 32 * 32), 0, st>>>(H, ldh, rot, restart, k);
}

// x += sum_j V_j y_j, accumulated j by j as the reference does.
template <typename T>
__global__ void __launch_bounds__(kThreads)
    update_x_kernel(T* x, const T* V, int64_t ldv, const double* rot, int restart, int k, int64_t n) {
  const double* y = rot + 3 * (restart + 1);
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n; i += int64_t(kVecCtas) * kThreads) {
    double xi = to_d(x[i]);
    for (int j = 0; j <= k; j++) xi = __dadd_rn(xi, __dmul_rn(to_d(V[j * ldv + i]), y[j]));
    x[i] = T(xi);
  }
}

// c = a - b and partial sums of |c|^2.
template <typename T>
__global__ void __launch_bounds__(kThreads) sub_norm_kernel(const T* a, const T* b, T* c, int64_t n, double* part) {
  double acc = 0.0;
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n; i += int64_t(kVecCtas) * kThreads) {
    const double v = __dsub_rn(to_d(a[i]), to_d(b[i]));
    const T tv = T(v);
    if (c) c[i] = tv;
    acc += to_d(tv) * to_d(tv);
  }
  acc = block_sum(acc);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

__global__ void finish_norm_kernel(const double* part, double* dst) {
  const double v = reduce_parts(part);
  if (threadIdx.x == 0) *dst = sqrt(v);
}

template <typename T>
__global__ void fill_zero_kernel(T* x, int64_t n) {
  for (int64_t i = blockIdx.x * int64_t(kThreads) + threadIdx.x; i < n; i += int64_t(kVecCtas) * kThreads) x[i] = T(0);
}

}  // namespace

template <typename T>
cudaError_t gmres_alloc(GmresWork<T>& W, int64_t n, int restart, cudaStream_t st) {
  gmres_free(W);
  W.n = n;
  W.restart = restart;
  HODLR_TRY(cudaMalloc(&W.V, sizeof(T) * size_t(n) * size_t(restart + 1)));
  HODLR_TRY(cudaMalloc(&W.w, sizeof(T) * size_t(n)));
  HODLR_TRY(cudaMalloc(&W.r, sizeof(T) * size_t(n)));
  HODLR_TRY(cudaMalloc(&W.tmp, sizeof(T) * size_t(n)));
  HODLR_TRY(cudaMalloc(&W.H, sizeof(double) * size_t(restart + 1) * size_t(restart)));
  HODLR_TRY(cudaMemsetAsync(W.H, 0, sizeof(double) * size_t(restart + 1) * size_t(restart), st));
  HODLR_TRY(cudaMalloc(&W.rot, sizeof(double) * 4 * size_t(restart + 1)));
  HODLR_TRY(cudaMemsetAsync(W.rot, 0, sizeof(double) * 4 * size_t(restart + 1), st));
  HODLR_TRY(cudaMalloc(&W.part, sizeof(double) * 2 * kVecCtas));
  HODLR_TRY(cudaMalloc(&W.partk, sizeof(double) * kVecCtas * size_t(restart + 1)));
  HODLR_TRY(cudaMalloc(&W.hc, sizeof(double) * size_t(restart + 1)));
  HODLR_TRY(cudaMalloc(&W.scal, sizeof(double) * 8));
  HODLR_TRY(cudaMallocHost(&W.hscal, sizeof(double) * 8));
  W.mgs_ctas = mgs_ctas<T>(n);
  W.cgs_step = cgs_step_fits<T>(n);
  if (W.cgs_step) {
    HODLR_TRY(cudaMalloc(&W.step_part, sizeof(float2) * (2 * kStepMaxBasis + 1) * kStepGrid));
    HODLR_TRY(cudaMalloc(&W.step_bar, sizeof(unsigned long long)));
    HODLR_TRY(cudaMemsetAsync(W.step_bar, 0, sizeof(unsigned long long), st));
  }
  return cudaStreamSynchronize(st);  // a solve may follow on any stream
}

template <typename T>
void gmres_free(GmresWork<T>& W) {
  cudaFree(W.V);
  cudaFree(W.w);
  cudaFree(W.r);
  cudaFree(W.tmp);
  cudaFree(W.H);
  cudaFree(W.rot);
  cudaFree(W.part);
  cudaFree(W.partk);
  cudaFree(W.hc);
  cudaFree(W.scal);
  cudaFree(W.step_part);
  cudaFree(W.step_bar);
  if (W.hscal) cudaFreeHost(W.hscal);
  W = GmresWork<T>();
}

template <typename T>
cudaError_t vec_sub_norm2(const T* a, const T* b, T* c, int64_t n, double* part, double* dst, cudaStream_t st) {
  count_launches(1);
  sub_norm_kernel<T><<<kVecCtas, kThreads, 0, st>>>(a, b, c, n, part);
  count_launches(1);
  finish_norm_kernel<<<1, kThreads, 0, st>>>(part, dst);
  return cudaGetLastError();
}

template <typename T>
cudaError_t vec_norm2(const T* a, int64_t n, double* part, double* dst, cudaStream_t st) {
  count_launches(1);
  dot_partial_kernel<T><<<kVecCtas, kThreads, 0, st>>>(a, a, n, part);
  count_launches(1);
  finish_norm_kernel<<<1, kThreads, 0, st>>>(part, dst);
  return cudaGetLastError();
}

template <typename T>
cudaError_t slots_norm2(const T* y, int64_t n, int s0, int s1, double* part, double* dst, cudaStream_t st) {
  count_launches(1);
  slots_partial_kernel<T><<<kVecCtas, kThreads, 0, st>>>(y, n, s0, s1, part);
  count_launches(1);
  finish_norm_kernel<<<1, kThreads, 0, st>>>(part, dst);
  return cudaGetLastError();
}

template <typename T>
cudaError_t gmres_solve(GmresWork<T>& W, const TreeMatvec<T>& A, const T* b, T* x, bool x0_zero, int restart,
                        int64_t max_iter, double tol, cudaStream_t st, GmresResult* res, Ortho ortho,
                        const std::function<void(double)>& progress) {
  const int64_t n = W.n;
  if (restart > W.restart || restart < 1) return cudaErrorInvalidValue;
  const int m = restart, ldh = W.restart + 1;
  double* part0 = W.part;
  double* part1 = W.part + kVecCtas;
  auto host_scal = [&](int count) -> cudaError_t {
    HODLR_TRY(cudaMemcpyAsync(W.hscal, W.scal, sizeof(double) * size_t(count), cudaMemcpyDeviceToHost, st));
    return cudaStreamSynchronize(st);
  };
  // normb = |b|; r = b - A x; beta = |r| (GMRES.hpp:186-197)
  HODLR_TRY(vec_norm2<T>(b, n, part0, W.scal + 2, st));
  if (x0_zero) {
    count_launches(1);
    fill_zero_kernel<T><<<kVecCtas, kThreads, 0, st>>>(x, n);
    HODLR_TRY(vec_sub_norm2<T>(b, x, W.r, n, part0, W.scal + 1, st));
  } else {
    HODLR_TRY(A(x, W.tmp));
    HODLR_TRY(vec_sub_norm2<T>(b, W.tmp, W.r, n, part0, W.scal + 1, st));
  }
  HODLR_TRY(host_scal(3));
  if (W.hscal[2] == 0.0) {
    W.hscal[2] = 1.0;
    HODLR_TRY(cudaMemcpyAsync(W.scal + 2, W.hscal + 2, sizeof(double), cudaMemcpyHostToDevice, st));
  }
  double resid = W.hscal[1] / W.hscal[2];
  res->converged = false;
  if (resid <= tol) {
    res->iterations = 0;
    res->resid = resid;
    res->converged = true;
    return cudaSuccess;
  }
  int64_t j = 1;
  const bool mgs = ortho == Ortho::kMGS;
  // whether this solve's steps take one launch each (its own cycle counts, not
  // the longest one the workspace has been allocated for)
  const bool one_launch = m + 1 <= kStepMaxBasis && (mgs ? W.mgs_ctas > 0 : W.cgs_step);
  bool busy = false;  // the device has no room for every CTA of a step at once
  while (j <= max_iter) {
    count_launches(1);
    start_cycle_kernel<T><<<kVecCtas, kThreads, 0, st>>>(W.r, W.V, n, W.scal, W.rot + 2 * (W.restart + 1), W.restart);
    for (int i = 0; i < m && j <= max_iter; i++, j++) {
      T* vi = W.V + int64_t(i) * n;
      HODLR_TRY(A(vi, W.w));
      if (one_launch) {
        const StepArgs<T> sa{W.w,       W.V,    n,       i,           W.H,
                             ldh,       W.rot,  W.restart, W.scal,    W.hscal,
                             static_cast<float2*>(W.step_part), W.step_bar, 0, W.step_wait_ns, 0, 0};
        W.hscal[1] = 0.0;
        W.steps++;
        HODLR_TRY(mgs ? launch_mgs_step<T>(sa, W.mgs_ctas, st)
                      : busy ? launch_cgs_phases<T>(sa, false, st) : launch_cgs_step<T>(sa, st));
        HODLR_TRY(cudaStreamSynchronize(st));
        if (W.hscal[1] != 0.0) {  // a barrier gave up: v_0 .. v_i and w are as they were
          busy = true;            // for the rest of this solve
          W.step_give_ups++;
          HODLR_TRY(cudaMemsetAsync(W.step_bar, 0, sizeof(unsigned long long), st));
          HODLR_TRY(launch_cgs_phases<T>(sa, true, st));
          HODLR_TRY(cudaStreamSynchronize(st));
        }
      } else {
        double* plast;
        if (mgs) {
          count_launches(1);
          dot_partial_kernel<T><<<kVecCtas, kThreads, 0, st>>>(W.w, W.V, n, part0);
          for (int k = 0; k <= i; k++) {
            const T* next = k < i ? W.V + int64_t(k + 1) * n : nullptr;
            double* pin = (k & 1) ? part1 : part0;
            double* pout = (k & 1) ? part0 : part1;
            count_launches(1);
            mgs_step_kernel<T><<<kVecCtas, kThreads, 0, st>>>(W.w, W.V + int64_t(k) * n, next, n, pin, pout,
                                                               W.H + k + int64_t(i) * ldh);
          }
          plast = (i & 1) ? part0 : part1;
        } else {
          // CGS2: two classical passes against v_0 .. v_i, |w|^2 from the second
          for (int pass = 0; pass < 2; pass++) {
            count_launches(3);
            cgs_dots_kernel<T><<<dim3(kDotCtas, unsigned((i + 1 + kDotGroup - 1) / kDotGroup)), kThreads, 0, st>>>(
                W.w, W.V, n, i + 1, W.partk);
            cgs_reduce_kernel<<<i + 1, kThreads, 0, st>>>(W.partk, W.hc, W.H + int64_t(i) * ldh, pass);
            cgs_update_kernel<T><<<kVecCtas, kThreads, 0, st>>>(W.w, W.V, n, i + 1, W.hc, pass == 1 ? part0 : nullptr);
          }
          plast = part0;
        }
        count_launches(2);
        norm_recip_kernel<<<1, kThreads, 0, st>>>(plast, W.H + (i + 1) + int64_t(i) * ldh, W.scal + 4);
        normalize_kernel<T><<<kVecCtas, kThreads, 0, st>>>(W.w, W.V + int64_t(i + 1) * n, n, W.scal + 4);
        count_launches(1);
        givens_kernel<<<1, 1, 0, st>>>(W.H, ldh, W.rot, W.restart, i, W.scal);
        HODLR_TRY(cudaGetLastError());
        HODLR_TRY(host_scal(1));
      }
      resid = W.hscal[0];
      if (progress) progress(resid);
      if (resid < tol) {
        launch_backsolve(W.H, ldh, W.rot, W.restart, i, st);
        count_launches(1);
        update_x_kernel<T><<<kVecCtas, kThreads, 0, st>>>(x, W.V, n, W.rot, W.restart, i, n);
        HODLR_TRY(cudaGetLastError());
        res->iterations = j;
        res->resid = resid;
        res->converged = true;
        return cudaStreamSynchronize(st);
      }
    }
    launch_backsolve(W.H, ldh, W.rot, W.restart, m - 1, st);
    count_launches(1);
    update_x_kernel<T><<<kVecCtas, kThreads, 0, st>>>(x, W.V, n, W.rot, W.restart, m - 1, n);
    if (progress) progress(1.0);  // the restart's true residual
    HODLR_TRY(A(x, W.tmp));
    HODLR_TRY(vec_sub_norm2<T>(b, W.tmp, W.r, n, part0, W.scal + 1, st));
    HODLR_TRY(host_scal(2));
    resid = W.hscal[1] / W.hscal[2];
    if (resid < tol) {
      res->iterations = j;
      res->resid = resid;
      res->converged = true;
      return cudaSuccess;
    }
  }
  res->iterations = max_iter;
  res->resid = resid;
  return cudaSuccess;
}

template cudaError_t gmres_alloc<double>(GmresWork<double>&, int64_t, int, cudaStream_t);
template cudaError_t gmres_alloc<float>(GmresWork<float>&, int64_t, int, cudaStream_t);
template void gmres_free<double>(GmresWork<double>&);
template void gmres_free<float>(GmresWork<float>&);
template cudaError_t gmres_solve<double>(GmresWork<double>&, const TreeMatvec<double>&, const double*, double*, bool,
                                         int, int64_t, double, cudaStream_t, GmresResult*, Ortho,
                                         const std::function<void(double)>&);
template cudaError_t gmres_solve<float>(GmresWork<float>&, const TreeMatvec<float>&, const float*, float*, bool, int,
                                        int64_t, double, cudaStream_t, GmresResult*, Ortho,
                                        const std::function<void(double)>&);
template cudaError_t vec_sub_norm2<double>(const double*, const double*, double*, int64_t, double*, double*,
                                           cudaStream_t);
template cudaError_t vec_sub_norm2<float>(const float*, const float*, float*, int64_t, double*, double*, cudaStream_t);
template cudaError_t vec_norm2<double>(const double*, int64_t, double*, double*, cudaStream_t);
template cudaError_t slots_norm2<double>(const double*, int64_t, int, int, double*, double*, cudaStream_t);
template cudaError_t vec_norm2<float>(const float*, int64_t, double*, double*, cudaStream_t);

}  // namespace hodlr

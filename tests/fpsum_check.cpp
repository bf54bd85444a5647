// Compares fpsum.cuh's FP32-pair sums with the FP64 sums they stand for, bit for
// bit, over random and edge operands; prints the number of mismatches.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>

#include "../hodlrnd_gb300/csrc/fpsum.cuh"
using namespace hodlr;

#ifdef __aarch64__
using Quad = long double;  // 113 bits
#else
using Quad = __float128;
#endif

static uint64_t rng_state = 88172645463325252ull;
static uint64_t rnd() {
  rng_state ^= rng_state << 13;
  rng_state ^= rng_state >> 7;
  rng_state ^= rng_state << 17;
  return rng_state;
}
static float make(int kind) {
  const uint64_t b = rnd();
  uint32_t e, m = uint32_t(b & 0x7fffff);
  switch (b >> 60 & 3) {  // random, few and many bits
    case 0: m &= 0x7f0000; break;
    case 1: m |= 0x00ffff; break;
    default: break;
  }
  switch (kind) {  // near 1, wide, the ends of the range, specials
    case 0: e = 120 + rnd() % 10; break;
    case 1: e = 90 + rnd() % 70; break;
    case 2: e = rnd() % 30; break;
    case 3: e = 225 + rnd() % 30; break;
    default: {
      const uint32_t ends[] = {0, 0, 1, 127, 254, 254, 255};
      e = ends[rnd() % 7];
      if ((e == 0 || e == 255) && rnd() % 2) m = 0;
    }
  }
  const uint32_t u = uint32_t(rnd() & 1) << 31 | e << 23 | m;
  float f;
  memcpy(&f, &u, 4);
  return f;
}
static uint32_t bits(float f) {
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  long bad = 0;
  for (long i = 0; i < n; i++) {
    float v[40];
    const int count = 1 + int(rnd() % (i % 50 ? 9 : 40)), kind = int(i % 16 < 8 ? 0 : i % 5);
    for (int q = 0; q < count; q++) {
      v[q] = make(kind);
      if (q && rnd() % 4 == 0) v[q] = -v[rnd() % q];  // cancellation
      if (q && rnd() % 16 == 0) v[q] = v[q - 1] * (1.f / 16777216.f);  // ties: half a unit in the last place
    }
    volatile double acc = double(v[0]);
    for (int q = 1; q < count; q++) acc = acc + double(v[q]);
    const float want = float(acc);
    auto at = [&](int q) { return v[q]; };
    auto same = [&](float got) { return bits(got) == bits(want) || (got != got && want != want); };
    bad += !same(sum_as_fp64(count, at));
    if (count <= 8) {
      float u[8], r;
      for (int q = 0; q < 8; q++) u[q] = q < count ? v[q] : 0.f;
      bad += !same(sum_few_as_fp64(count, u, r) ? r : sum_in_fp64(count, at));
    }
  }
  // triples of 152 pairs against sums in 113 bits: no further off than FP64 sums
  double e3 = 0.0, e64 = 0.0;
  for (long i = 0; i < n / 152; i++) {
    TripleSum t;
    Quad want = 0, mag = 0;
    volatile double acc = 0.0;
    for (int q = 0; q < 152; q++) {
      const float x = make(0), y = x * float(int64_t(rnd() >> 40)) * 0x1p-49f;
      const float sign = rnd() & 1 ? 1.f : -1.f;
      t.add(sign * x, sign * y);
      want += Quad(sign * x) + Quad(sign * y);
      mag += Quad(x < 0 ? -x : x);
      acc = acc + (double(sign * x) + double(sign * y));
    }
    const double a = double((Quad(t.value()) - want) / mag), b = double((Quad(acc) - want) / mag);
    e3 = std::max(e3, std::fabs(a));
    e64 = std::max(e64, std::fabs(b));
  }
  printf("%ld %.3e %.3e\n", bad, e3, e64);
  return bad || e3 > e64 || e3 > 0x1p-53 ? 1 : 0;
}

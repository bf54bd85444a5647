// Compares softfp.cuh with the host's FP64 operations, bit for bit, over random
// and edge operands; prints the number of mismatches per operation.  The seeds of
// the Newton steps are perturbed by up to 2^-21, so the results do not depend on
// whose single-precision reciprocals they come from.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
static uint64_t rng_state = 88172645463325252ull;
static uint64_t rnd() {
  rng_state ^= rng_state << 13;
  rng_state ^= rng_state >> 7;
  rng_state ^= rng_state << 17;
  return rng_state;
}
static float noise(float r) { return r * (1.0f + float(int(rnd() % 2001) - 1000) * (4.7e-7f / 1000.0f)); }
#define HODLR_SOFT_SEED_NOISE(r) noise(r)
#include "../hodlrnd_gb300/csrc/softfp.cuh"
using namespace hodlr;

static double make(int kind) {
  uint64_t b = rnd();
  uint64_t m = b & 0xfffffffffffffull;
  switch (rnd() % 8) {  // significands: random, nearly all zeros or ones, few bits
    case 0: m = 0; break;
    case 1: m = 0xfffffffffffffull; break;
    case 2: m = 1ull << (rnd() % 52); break;
    case 3: m = 0xfffffffffffffull ^ (1ull << (rnd() % 52)); break;
    case 4: m &= 0xfffffffull << (rnd() % 25); break;
    default: break;
  }
  uint64_t e;
  switch (kind) {  // exponents: near 0, anywhere normal, the ends and the specials
    case 0: e = 1023 + int(rnd() % 60) - 40; break;
    case 1: e = 1 + rnd() % 2046; break;
    default: {
      const uint64_t ends[] = {0, 0, 1, 2, 3, 511, 512, 1022, 1023, 2044, 2045, 2046, 2047};
      e = ends[rnd() % 13];
      if ((e == 0 || e == 2047) && rnd() % 2) m = 0;
    }
  }
  return soft_double((rnd() << 63) | (e << 52) | m);
}
static bool same(double a, double b) { return soft_bits(a) == soft_bits(b) || (a != a && b != b); }

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  long bad[3] = {0, 0, 0};
  for (long i = 0; i < n; i++) {
    const int kind = i % 8 < 5 ? 0 : i % 8 < 7 ? 1 : 2;
    volatile double a = make(kind), b = make(kind);
    volatile double q = a / b, s = std::sqrt(b), ds = a / s;
    bad[0] += !same(soft_sqrt(b), s);
    bad[1] += !same(soft_div_sqrt(soft_unpack(a), a, b), ds);
    bad[2] += !same(soft_div(soft_unpack(a), a, b), q);
    // squares of integers and their neighbours, exact products and quotients
    volatile double r = double(int64_t(rnd() >> 38)), r2 = soft_double(soft_bits(r * r) + rnd() % 3 - 1);
    volatile double sr = std::sqrt(r2), pr = r * a, qr = pr / r;
    bad[0] += !same(soft_sqrt(r2), sr);
    bad[2] += !same(soft_div(soft_unpack(pr), pr, r), qr);
  }
  printf("%ld %ld %ld\n", bad[0], bad[1], bad[2]);
  return bad[0] + bad[1] + bad[2] ? 1 : 0;
}

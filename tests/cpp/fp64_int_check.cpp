// Host check of fp64_int.cuh against the processor's FP64, bit for bit, over
// mantissas of all kinds.  Prints one line "name mismatches tested" per check.
#include <cmath>
#include <cstdio>

#include "fp64_int.cuh"

using namespace j3g;

static uint64_t state = 1;
static uint64_t next() {  // splitmix64
  uint64_t x = state += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

// fractions at random, with few bits, with long runs of ones or zeros
static uint64_t fraction() {
  const uint64_t r = next(), k = next() % 6;
  const int n = (int)(next() % 52);
  if (k == 0) return r & kIntFrac & ~0ull << n;
  if (k == 1) return (r | ~(~0ull << n)) & kIntFrac;
  if (k == 2) return next() % 2 ? 1ull << n : (1ull << n) - 1;
  if (k == 3) return (0ull - (1ull << n)) & kIntFrac;
  return r & kIntFrac;
}

int main() {
  const long long kN = 20000000;
  long long bad = 0;
  for (long long i = 0; i < kN; ++i) {
    double x = fx_double((next() % 2046 + 1) << 52 | fraction());
    if (i % 4 == 0) {  // squares and their neighbours
      const double r = fx_double((1000 + next() % 40) << 52 | (fraction() >> next() % 30));
      x = fx_double(fx_bits(r * r) + next() % 3 - 1);
    }
    bad += fx_bits(int_sqrt(x)) != fx_bits(std::sqrt(x));
  }
  std::printf("sqrt %lld %lld\n", bad, kN);
  bad = 0;
  for (long long i = 0; i < kN; ++i) {
    uint64_t n = fraction() | kIntOne, d = fraction() | kIntOne;
    if (i % 8 == 0) n = d + next() % 5 - 2;
    if (i % 8 == 1) {  // products: quotients with few bits, and their neighbours
      const double p = fx_double(1023ull << 52 | fraction()) * fx_double(1023ull << 52 | d);
      n = (fx_bits(p) & kIntFrac) | kIntOne;
      n += next() % 3 - 1;
    }
    n = (n & kIntFrac) | kIntOne;
    int down;
    const uint64_t z = int_quotient(n, d, down);
    bad += (double)z * (down ? 0.5 : 1.0) != (double)n / (double)d * 0x1p52;
    bad += z < kIntOne || z > 2 * kIntOne;
  }
  std::printf("quotient %lld %lld\n", bad, kN);
  bad = 0;
  for (long long i = 0; i < kN; ++i) {
    int64_t v = (int64_t)(next() >> (11 + next() % 53));
    if (i & 1) v = -v;
    if (i % 64 == 0) v = (int64_t)(i % 128 ? 1ull << 53 : 0);
    const int scale = (int)(next() % 100);
    bad += fx_bits(int_to_double(v, scale)) != fx_bits(std::ldexp((double)v, -scale));
  }
  std::printf("convert %lld %lld\n", bad, kN);
  bad = 0;
  for (long long i = 0; i < kN; ++i) {
    // exponents anywhere, gaps of 2 and of 35 at most; specials; cancellation
    const int e = (int)(next() % 2046) + 1, gap = (int)(next() % (i & 1 ? 4 : 70)) - (i & 1 ? 2 : 35);
    const int f = e + gap < 0 ? 0 : e + gap > 2047 ? 2047 : e + gap;
    double a = fx_double((next() & 1) << 63 | (uint64_t)e << 52 | fraction());
    double b = fx_double((next() & 1) << 63 | (uint64_t)f << 52 | fraction());
    static const double special[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, -2e-308, 1.7e308};
    if (i % 16 == 0) b = special[next() % 8];
    if (i % 16 == 1) b = fx_double(fx_bits(a) ^ 1ull << 63 ^ next() % 3);
    if (i & 8) {
      const double t = a;
      a = b;
      b = t;
    }
    const double got = int_add(a, b), want = a + b;
    bad += fx_bits(got) != fx_bits(want) && !(std::isnan(got) && std::isnan(want));
  }
  std::printf("add %lld %lld\n", bad, kN);
  return 0;
}

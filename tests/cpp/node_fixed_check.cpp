// Accuracy of the fixed-point node terms (csrc/node_fixed.cuh) on the host
// against long double: prints one line per set of offsets with the evaluated
// and left-out counts and the largest error of each component in units of its
// bound (test_node_fixed.py states the bounds).
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <random>

#include "node_fixed.cuh"

using namespace j3g;
static FxTables tables;
typedef long double LD;

static LD ln_sum(LD d, LD r, LD a, LD b) {  // log(d + r) without cancellation
  return d < 0 ? logl((a * a + b * b) / (r - d)) : logl(d + r);
}
static LD half_ulp(LD v) {
  int e;
  frexpl(v, &e);
  return ldexpl(1.0L, e - 54);
}

template <int MASK> static void run(const char *name, int set, long n) {
  std::mt19937_64 g(1000 + set);
  std::uniform_real_distribution<double> u(-1, 1);
  double worst[7] = {0};
  long left = 0;
  for (long i = 0; i < n; ++i) {
    double dx, dy, dz;
    switch (set) {
      case 0: dx = 3200 * u(g); dy = 3200 * u(g); dz = -1000 * fabs(u(g)) - 1; break;  // a survey
      case 1:  // eighteen binades, any sign
        dx = std::copysign(exp2(9 * u(g)), u(g));
        dy = std::copysign(exp2(9 * u(g)), u(g));
        dz = std::copysign(exp2(9 * u(g)), u(g));
        break;
      case 2: dx = 4800 * u(g); dy = u(g); dz = -1; break;            // nearly in line
      case 3: dx = 100 * u(g); dy = 100 * u(g); dz = -2e4 * u(g) - 3e4; break;  // far above
      case 4:  // stations on the mesh's planes and above its columns
        dx = 50.0 * (int)(4 * u(g)); dy = 50.0 * (int)(4 * u(g)); dz = -25.0 * (1 + (int)(3 * fabs(u(g))));
        if (u(g) < 0) dz = -dz;
        break;
      default: dx = 1e9 * u(g); dy = 1e-3 * u(g); dz = 1e3 * u(g); break;  // wide apart
    }
    double o[7];
    const FxColumn c = fx_column<MASK>(fx_axis(dx), fx_axis(dy), tables);
    if (!fx_node<MASK>(c, fx_axis(dz), tables, o)) {
      ++left;
      continue;
    }
    if (MASK & 1) o[0] = std::fma(dx, o[5], std::fma(dy, o[6], dz * o[0]));
    const LD x = dx, y = dy, z = dz, r = sqrtl(x * x + y * y + z * z);
    LD t[7], b[7];
    t[4] = dx == 0 && dy == 0 && dz < 0 ? -52 * logl(2.0L) : ln_sum(z, r, x, y);
    t[5] = ln_sum(y, r, x, z);
    t[6] = ln_sum(x, r, y, z);
    t[1] = atan2l(y * z, x * r);
    t[2] = atan2l(x * z, y * r);
    t[3] = atan2l(x * y, z * r);
    const LD a = atan2l(z * r, x * y);
    t[0] = x * t[5] + y * t[6] + z * a;
    const LD off[3] = {z, y, x}, arg[3] = {expl(t[4]), expl(t[5]), expl(t[6])};
    for (int k = 0; k < 3; ++k) {
      const LD cut = off[k] < 0 ? r / arg[k] : 1.0L;
      b[4 + k] = half_ulp(t[4 + k]) + ldexpl(1.0L, -54) + cut * ldexpl(1.0L, -56);
    }
    for (int k = 1; k < 4; ++k)
      b[k] = half_ulp(t[k]) + fminl(ldexpl(1.0L, -56), fabsl(t[k]) * ldexpl(1.0L, -48));
    b[0] = fabsl(x) * b[5] + fabsl(y) * b[6] + fabsl(z) * (half_ulp(a) + ldexpl(1.0L, -56)) +
           1.5L * ldexpl(1.0L, -52) * (fabsl(x * t[5]) + fabsl(y * t[6]) + fabsl(z * a));
    for (int k = 0; k < 7; ++k)
      if (MASK >> k & 1) {
        const LD e = fabsl((LD)o[k] - t[k]);
        if (!(e <= (LD)worst[k] * b[k])) worst[k] = b[k] > 0 ? (double)(e / b[k]) : (e > 0 ? 1e9 : 0);
      }
  }
  printf("%s %d %ld %ld", name, set, n, left);
  for (int k = 0; k < 7; ++k) printf(" %.4g", worst[k]);
  printf("\n");
}

int main() {
  tables.set(0, 1);
  for (int set = 0; set < 6; ++set) {
    run<127>("joint", set, 100000);
    run<126>("tensor", set, 100000);
    run<1>("scalar", set, 100000);
    run<8 + 32 + 64>("gradient", set, 100000);
  }
  return 0;
}

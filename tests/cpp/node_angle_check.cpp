// Error of the fixed-point angles (csrc/node_fixed.cuh) and of the same angles in
// FP64 (atan2 of products of doubles), in units of the last place, against long
// double: one line per component and power of two of the angle with the count, the
// root mean squares and the largest errors of both.
#include <cmath>
#include <cstdio>
#include <random>

#include "node_fixed.cuh"

using namespace j3g;
typedef long double LD;
static FxTables tables;

struct Stat {
  long n;
  double fx2, fp2, fx, fp;
};

int main() {
  tables.set(0, 1);
  std::mt19937_64 g(3);
  std::uniform_real_distribution<double> u(0, 1);
  static Stat stat[3][40];
  auto offset = [&](double scale) {
    const double v = scale * std::exp2(-12 * u(g));
    return u(g) < 0.5 ? -v : v;
  };
  for (int i = 0; i < 1500000; ++i) {
    const double scale = std::exp2(14 * u(g));
    const double dx = offset(scale), dy = offset(scale), dz = offset(scale);
    double o[7];
    const FxColumn c = fx_column<127>(fx_axis(dx), fx_axis(dy), tables);
    if (!fx_node<127>(c, fx_axis(dz), tables, o)) return 1;
    const LD x = dx, y = dy, z = dz, r = sqrtl(x * x + y * y + z * z);
    const double d = std::sqrt(std::fma(dx, dx, std::fma(dy, dy, dz * dz)));
    const LD exact[3] = {atan2l(y * z, x * r), atan2l(x * z, y * r), atan2l(x * y, z * r)};
    const double fp[3] = {std::atan2(dy * dz, dx * d), std::atan2(dx * dz, dy * d),
                          std::atan2(dx * dy, dz * d)};
    for (int k = 0; k < 3; ++k) {
      int e;
      frexpl(exact[k], &e);
      if (e > 2 || e <= -38) continue;
      Stat &s = stat[k][2 - e];
      const double a = fabsl(o[1 + k] - exact[k]) * exp2l(53 - e);
      const double b = fabsl(fp[k] - exact[k]) * exp2l(53 - e);
      ++s.n;
      s.fx2 += a * a;
      s.fp2 += b * b;
      s.fx = std::fmax(s.fx, a);
      s.fp = std::fmax(s.fp, b);
    }
  }
  for (int k = 0; k < 3; ++k)
    for (int b = 0; b < 40; ++b) {
      const Stat &s = stat[k][b];
      if (s.n)
        printf("%d %d %ld %.4f %.4f %.3f %.3f\n", k, 2 - b, s.n, std::sqrt(s.fx2 / s.n),
               std::sqrt(s.fp2 / s.n), s.fx, s.fp);
    }
  return 0;
}

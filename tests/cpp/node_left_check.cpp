// Offsets that the fixed-point node terms (csrc/node_fixed.cuh) leave to FP64 and the
// nearest ones that they take: prints "left" or "taken" per line of the list below.
#include <cmath>
#include <cstdio>
#include <limits>

#include "node_fixed.cuh"

using namespace j3g;
static FxTables tables;

int main() {
  tables.set(0, 1);
  const double inf = std::numeric_limits<double>::infinity(), top = std::exp2(41);
  const double last = std::nextafter(top, 0.0), low = std::exp2(-40);
  const double below = std::nextafter(low, 0.0), sub = std::numeric_limits<double>::denorm_min();
  const double offsets[][3] = {
      // taken: ends of the range on each axis, zero offsets but dz with another
      {last, 3.0, -5.0}, {2.0, -last, 7.0}, {2.0, 3.0, last}, {low, 3.0, -5.0},
      {2.0, -low, 7.0}, {2.0, 3.0, -low}, {0.0, 3.0, -5.0}, {2.0, 0.0, 7.0},
      {0.0, 0.0, -5.0}, {0.0, 0.0, 5.0}, {2.0, 3.0, 0.0},
      // left: beyond the range, dz and another zero, all zero, not finite
      {top, 3.0, -5.0}, {2.0, -top, 7.0}, {2.0, 3.0, top}, {below, 3.0, -5.0},
      {2.0, -below, 7.0}, {2.0, 3.0, sub}, {0.0, 3.0, 0.0}, {2.0, 0.0, 0.0},
      {0.0, 0.0, 0.0}, {inf, 3.0, -5.0}, {2.0, -inf, 7.0}, {2.0, 3.0, inf},
      {NAN, 3.0, -5.0}, {2.0, NAN, 7.0}, {2.0, 3.0, NAN}};
  for (const auto &o : offsets) {
    double v[7];
    const FxColumn c = fx_column<127>(fx_axis(o[0]), fx_axis(o[1]), tables);
    puts(fx_node<127>(c, fx_axis(o[2]), tables, v) ? "taken" : "left");
  }
  return 0;
}

// node_column.cuh -- what the kernels over node columns share: block shape and
// the z offsets that a block keeps for its columns.
#pragma once
#include "node_fixed.cuh"
#include "prism_math.cuh"

namespace j3g {

// 128 threads at 96 registers: five blocks, 20 warps, to an SM (256 threads at
// 128 registers: 16 warps, 1 to 7 % slower)
constexpr int kNodeThreads = 128;
constexpr int kNodeResident = 5;

struct ZOffset {
  FxAxis a;
  double d;
};

__device__ __forceinline__ ZOffset z_offset(double mz, double Z) {
  ZOffset o;
  o.d = sub(mz, Z);
  o.a = fx_axis(o.d);
  return o;
}

}  // namespace j3g

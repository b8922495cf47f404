// Device check of fp64_int.cuh and of the functions that use it: square roots
// against the FP64 instruction, flog, fatan2 and fatan2_pair with SPLIT against
// themselves without, sums against the instruction.  Prints one line "name mismatches tested" per check.
#include <cstdio>
#include <cuda_runtime.h>

#include "fp64_math.cuh"

using namespace j3g;

__device__ unsigned long long mix64(unsigned long long x) {  // splitmix64 finaliser
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
__device__ double value(unsigned long long r, int e0, int range) {
  unsigned long long m = r & kIntFrac;
  if ((r >> 60) == 0) m &= ~0ull << (r >> 54 & 51);  // few bits: breakpoints, exact cases
  return __longlong_as_double((long long)((unsigned long long)(e0 + mix64(r) % range) << 52 | m));
}
__device__ bool same(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}

__global__ void k_check(int which, unsigned long long n, unsigned long long *bad) {
  unsigned long long nb = 0;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long r = mix64(i), s = mix64(r);
    if (which == 0) {
      const double x = i & 1 ? value(r, 1, 2046) : value(r, 1000, 60);
      nb += !same(int_sqrt(x), sqrt(x));
    } else if (which == 1) {
      const double x = i & 1 ? value(r, 1, 2046) : value(r, 1021, 4);
      nb += !same(flog<true>(x), flog<false>(x));
    } else if (which == 3) {
      double x = value(r, 950, 100), y = value(s, i & 1 ? 1000 : 940, i & 1 ? 3 : 130);
      if (r >> 63) x = -x;
      if (s >> 63) y = -y;
      if (i % 32 == 7) y = -x;
      if (i % 32 == 8) y = 0.0;
      if (i % 32 == 9) y *= 0x1p-1000;
      nb += !same(int_add(x, y), __dadd_rn(x, y)) + !same(int_add(y, int_neg(x)), __dsub_rn(y, x));
    } else {
      // ratios near 1, over the breakpoints, tiny; every quadrant; zeros
      double y = value(r, 1000, i % 3 == 0 ? 2 : 40), x = value(s, 1000, 2);
      if (i % 3 == 2) y *= 0x1p-900;
      if (i % 64 == 5) y = 0.0;
      if (s >> 62 & 1) y = -y;
      if (s >> 63) x = -x;
      double a, b;
      fatan2_pair<true>(y, x, a, b);
      nb += !same(fatan2<true>(y, x), fatan2<false>(y, x));
      nb += !same(a, fatan2<false>(y, x)) + !same(b, fatan2<false>(x, y));
    }
  }
  atomicAdd(bad, nb);
}

int main() {
  const char *names[] = {"sqrt", "log", "atan2", "add"};
  unsigned long long *bad;
  if (cudaMalloc(&bad, 4 * sizeof *bad) != cudaSuccess) return 1;
  cudaMemset(bad, 0, 4 * sizeof *bad);
  const unsigned long long n = 1ull << 27;
  for (int w = 0; w < 4; ++w) k_check<<<1216, 256>>>(w, n, bad + w);
  unsigned long long h[4];
  if (cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  for (int w = 0; w < 4; ++w) std::printf("%s %llu %llu\n", names[w], h[w], n);
  return 0;
}

// Device check of chained.cuh: a launch that the runtime refuses (more threads than
// a block holds) returns its error and leaves none behind for the next launch's
// check; kernels in a chain run in order.  Prints "ok", or the first failure.
#include <cstdio>

#include "chained.cuh"

using namespace j3g;

__global__ void k_step(int i, int *v) {
  chain_begin();
  chain_wait();
  if (threadIdx.x == 0 && *v == i) *v = i + 1;
}

int main() {
  int *v = nullptr, got = 0;
  if (cudaMalloc(&v, sizeof(int)) != cudaSuccess || cudaMemset(v, 0, sizeof(int)) != cudaSuccess)
    return puts("no memory"), 1;
  if (launch_chained(k_step, dim3(1), 4096, 0, 0, 0, v) == cudaSuccess)
    return puts("4096 threads were accepted"), 1;
  if (cudaGetLastError() != cudaSuccess) return puts("the error was left behind"), 1;
  for (int i = 0; i < 20; ++i)
    if (launch_chained(k_step, dim3(1), 32, 0, 0, i, v) != cudaSuccess)
      return puts("a launch failed"), 1;
  if (cudaMemcpy(&got, v, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess || got != 20)
    return puts("out of order"), 1;
  puts("ok");
  return 0;
}

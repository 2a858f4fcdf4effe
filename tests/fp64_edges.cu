// Counts operands of given lists for which the branch-free IEEE sequences of
// sed_common.cuh differ from CUDA's own division and square root (compiled by
// test_gpu_fp64_edges.py).
#include "../pubsed_b200/csrc/sed_common.cuh"
using namespace sed;

__global__ void count(const double* a, const double* b, int n, unsigned long long* bad)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double x = a[i], y = b[i];
    if (div_rn(x, y) != x / y || div_rn(-x, y) != -x / y) atomicAdd(bad + 0, 1ull);
    if (rcp_rn(y) != 1.0 / y || rcp_rn(-y) != -1.0 / y) atomicAdd(bad + 1, 1ull);
    if (sqrt_rn(x) != sqrt(x)) atomicAdd(bad + 2, 1ull);
    if (rcp_sqrt_rn(x) != 1.0 / sqrt(x)) atomicAdd(bad + 3, 1ull);
  }
}

extern "C" int fp64_edges(const double* a, const double* b, int n, unsigned long long* bad)
{
  double* d;
  unsigned long long* c;
  if (cudaMalloc(&d, 2 * (size_t)n * sizeof(double)) != cudaSuccess || cudaMalloc(&c, 4 * sizeof *c) != cudaSuccess) return 1;
  cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemset(c, 0, 4 * sizeof *c);
  count<<<592, 256>>>(d, d + n, n, c);
  const cudaError_t e = cudaMemcpy(bad, c, 4 * sizeof *c, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(c);
  return e != cudaSuccess;
}

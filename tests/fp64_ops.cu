// Counts operands where the branch-free IEEE sequences of sed_common.cuh differ
// from CUDA's own division and square root (compiled by test_gpu_fp64_forms.py).
#include "../pubsed_b200/csrc/sed_common.cuh"
using namespace sed;

__device__ double operand(uint32_t a, uint32_t b, int lo, int hi)
{
  const uint64_t m = (((uint64_t)a << 20) ^ ((uint64_t)b * 0x9E3779B97F4A7C15ull >> 12)) & 0xFFFFFFFFFFFFFull;
  const int e = lo + (int)(b % (uint32_t)(hi - lo + 1));
  return __longlong_as_double(((int64_t)(e + 1023) << 52) | (int64_t)m);
}

__global__ void count(unsigned long long* bad, uint64_t n, int lo, int hi, double t, double th, double tl)
{
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const PhiloxOut o = philox4x32_10((uint32_t)i, (uint32_t)(i >> 32), 3, 4, 5, 6);
    const double a = operand(o.w[0], o.w[1], lo, hi), b = operand(o.w[2], o.w[3], lo, hi);
    if (div_rn(a, b) != a / b || div_rn(-a, b) != -a / b || div_rn(0.0, b) != 0.0) atomicAdd(bad + 0, 1ull);
    if (rcp_rn(b) != 1.0 / b) atomicAdd(bad + 1, 1ull);
    if (sqrt_rn(a) != sqrt(a) || sqrt_rn(0.0) != 0.0) atomicAdd(bad + 2, 1ull);
    if (rcp_sqrt_rn(a) != 1.0 / sqrt(a)) atomicAdd(bad + 3, 1ull);
    if (div_c(a) != a / C_LIGHT) atomicAdd(bad + 4, 1ull);
    if (div_by(a, t, th, tl) != a / t) atomicAdd(bad + 5, 1ull);
    const double m = floor(ldexp(w01(o.w[0]) + 1, 52)) + 0.5;  // radicands next to the midpoints of roots
    if (sqrt_rn(m * m) != sqrt(m * m)) atomicAdd(bad + 6, 1ull);
  }
}

extern "C" int fp64_ops(unsigned long long* bad, unsigned long long n, int lo, int hi, double t)
{
  unsigned long long* d;
  if (cudaMalloc(&d, 7 * 8) != cudaSuccess) return 1;
  cudaMemset(d, 0, 7 * 8);
  const double th = 1.0 / t, tl = fma(-t, th, 1.0) * th;
  count<<<592, 256>>>(d, n, lo, hi, t, th, tl);
  const cudaError_t e = cudaMemcpy(bad, d, 7 * 8, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e != cudaSuccess;
}

// Counts frequencies for which loc_within_mixed gives another bin than
// loc_within, the reference's rule (compiled by test_gpu_bin_lookup.py).
#include "../pubsed_b200/csrc/sed_ctx.h"
using namespace sed;

__global__ void count(DevLoc g, double top, uint64_t n, unsigned long long* bad)
{
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const PhiloxOut o = philox4x32_10((uint32_t)i, (uint32_t)(i >> 32), 7, 8, 9, 10);
    double x = g.min + (top - g.min) * (1.002 * u01(o.w[0], o.w[1]) - 0.001);  // over both ends
    if (i % 4 == 0)  // next to a wall
      x = g.right[o.w[2] % (uint32_t)g.n] * (1.0 + ((int)(o.w[3] % 5u) - 2) * 0x1p-52);
    if (loc_within_mixed(g, x) != loc_within(g, x)) atomicAdd(bad, 1ull);
  }
}

extern "C" int bin_lookup(int type, int nn, double min, double del, const double* right, unsigned long long n,
                          unsigned long long* bad)
{
  const sed_locate_grid lg{nn, type, min, del, right};
  const HostLoc h = host_loc(lg);
  DevBuf<double> d;
  DevBuf<unsigned long long> b;
  if (d.resize((size_t)nn) != cudaSuccess || b.resize(1) != cudaSuccess) return 1;
  cudaMemcpy(d.p, right, nn * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemset(b.p, 0, sizeof *b.p);
  count<<<592, 256>>>(dev_loc(h, d), right[nn - 1], n, b.p);
  const cudaError_t e = cudaMemcpy(bad, b.p, sizeof *bad, cudaMemcpyDeviceToHost);
  d.release();
  b.release();
  return e != cudaSuccess;
}

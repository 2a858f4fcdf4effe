// Counts the device allocations DevBuf makes for a list of sizes, with
// stand-ins for cudaMalloc and cudaFree: runs without a GPU (compiled by
// test_device_buffers.py).
#include <cstdlib>
#include <cuda_runtime.h>

static long n_alloc = 0, n_free = 0;
static size_t held = 0, most = 0, limit = 0;

template <typename T>
static cudaError_t counted_malloc(T** p, size_t bytes)
{
  if (limit && held + bytes > limit) return cudaErrorMemoryAllocation;
  size_t* q = static_cast<size_t*>(std::malloc(sizeof(size_t)));
  *q = bytes;
  *p = reinterpret_cast<T*>(q);
  ++n_alloc;
  held += bytes;
  if (held > most) most = held;
  return cudaSuccess;
}
static cudaError_t counted_free(void* p)
{
  held -= *static_cast<size_t*>(p);
  std::free(p);
  ++n_free;
  return cudaSuccess;
}
#define cudaMalloc counted_malloc
#define cudaFree counted_free
#define cudaGetLastError() cudaSuccess
#include "../pubsed_b200/csrc/sed_ctx.h"

// out: allocations, bytes held after the last size, most bytes held, sizes refused
extern "C" int devbuf_run(const long long* sizes, int n, long long max_bytes, long long* out)
{
  n_alloc = n_free = 0;
  held = most = 0;
  limit = (size_t)max_bytes;
  sed::DevBuf<double> b;
  long long refused = 0;
  for (int i = 0; i < n; ++i) {
    if (b.resize((size_t)sizes[i]) != cudaSuccess) {
      ++refused;
      if (b.p || b.n || b.cap) return 1;
      continue;
    }
    if (b.n != (size_t)sizes[i] || (sizes[i] > 0) != (b.p != nullptr)) return 1;
    if (sizes[i] > 0 && (b.cap < b.n || held != b.cap * sizeof(double))) return 1;
  }
  out[0] = n_alloc;
  out[1] = (long long)held;
  out[2] = (long long)most;
  out[3] = refused;
  b.release();
  return held == 0 && n_alloc == n_free ? 0 : 1;
}

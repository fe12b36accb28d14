// Device conversions of the tensor-core kernels against CUDA's own (built and
// called by test_gpu_conversions.py).  Each check counts the values that differ.
#include <algorithm>

#include "k_tcx.cu"

using namespace bgpu::dev;

namespace conversions {

__device__ bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }

// every f32
__global__ void f32_to_f64_kernel(unsigned long long* bad) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32); i += step) {
    const float x = __uint_as_float((uint32_t)i);
    if (!same(bgpu::tc::f32_to_f64(x), (double)x)) atomicAdd(bad, 1ull);
  }
}

// a 2^k: the conversion, rounded once, then an exact scaling
__global__ void scaled_kernel(const long long* a, int n, unsigned long long* bad) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int k = -960; k <= 960; k += 60)
      if (!same(scaled(a[i], k), scalbn((double)a[i], k))) atomicAdd(bad, 1ull);
}

// integers of digits and of accumulators
__global__ void integers_kernel(unsigned long long* bad) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  for (int x = -255 + t; x <= 255; x += step)
    for (int y = -255; y <= 255; ++y) {
      const uint32_t w = bf16x2_of(x, y);
      if (__uint_as_float(w << 16) != (float)x || __uint_as_float(w & 0xffff0000u) != (float)y) atomicAdd(bad, 1ull);
    }
  for (int x = -(1 << 22) + 1 + t; x < (1 << 22); x += step)
    if (as_int<true>(__float_as_uint((float)x)) != x || as_int<false>(__float_as_uint((float)x)) != x)
      atomicAdd(bad, 1ull);
}

template <class F>
long long counted(F launch) {
  unsigned long long *d = nullptr, h = 0;
  if (cudaMalloc(&d, sizeof h) != cudaSuccess) return -1;
  cudaMemset(d, 0, sizeof h);
  launch(d);
  const cudaError_t e = cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? (long long)h : -1;
}

}  // namespace conversions

using namespace conversions;

extern "C" long long check_f32_to_f64() {
  return counted([](unsigned long long* bad) { f32_to_f64_kernel<<<2048, 256>>>(bad); });
}
extern "C" long long check_integers() {
  return counted([](unsigned long long* bad) { integers_kernel<<<256, 256>>>(bad); });
}
extern "C" long long check_scaled(const long long* a, int n) {
  long long* d = nullptr;
  if (cudaMalloc(&d, n * sizeof(long long)) != cudaSuccess) return -1;
  cudaMemcpy(d, a, n * sizeof(long long), cudaMemcpyHostToDevice);
  const long long bad = counted([=](unsigned long long* b) { scaled_kernel<<<256, 256>>>(d, n, b); });
  cudaFree(d);
  return bad;
}

// Device functions and kernels of the library called one at a time, for the
// tests that check them against values computed on the host.
#include <cuda_runtime.h>

#include "kernels_common.cuh"

namespace {
template <typename T, class F>
__global__ void k_map(const T* x, int n, T* y, F f) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = f(x[i]);
}
template <typename T, class F>
int map(const T* x, int n, T* y, F f) {  // host arrays
  T *dx = nullptr, *dy = nullptr;
  cudaError_t e = cudaMalloc(&dx, n * sizeof(T));
  if (e == cudaSuccess) e = cudaMalloc(&dy, n * sizeof(T));
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, n * sizeof(T), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_map<<<148, 256>>>(dx, n, dy, f);
    e = cudaMemcpy(y, dy, n * sizeof(T), cudaMemcpyDeviceToHost);
  }
  cudaFree(dx);
  cudaFree(dy);
  return (int)e;
}
struct Root {
  __device__ double operator()(double x) const { return kifmm::rinv_cut(x); }
};
struct Seed {
  __device__ double operator()(double x) const {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
  }
};
struct Library {
  __device__ double operator()(double x) const { return rsqrt(x); }
};
}  // namespace

// which: 0 rinv_cut, 1 the seed of rsqrt_t, 2 CUDA's rsqrt()
extern "C" int harness_root(int which, const double* x, int n, double* y) {
  return which == 0 ? map(x, n, y, Root()) : which == 1 ? map(x, n, y, Seed()) : map(x, n, y, Library());
}

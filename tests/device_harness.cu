// Device functions and kernels of the library called one at a time, for the
// tests that check them against values computed on the host.
#include <cuda_runtime.h>

#include <vector>

#include "kernels_common.cuh"
#include "launch.hpp"

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

// the leaf pass's items (host side) of `nwork` leaves with tcnt[w] targets and
// nmid[w] W-list surfaces each, the near list of leaf w being the leaves
// nptr[w] .. nptr[w + 1] of nidx, with scnt sources; rows of 8: leaf, first
// target, first near segment, segments, skip, take, surfaces, output row.
// Returns the number of items.
extern "C" int harness_leaf_items(int nwork, const int* tcnt, const int* scnt, const int64_t* nptr, const int* nidx,
                                  const int64_t* mptr, int nsurf, int least, int num_sms, int* rows, int cap,
                                  int* nsplit, int* nparts) {
  std::vector<int> work(nwork), tbeg(nwork);
  for (int w = 0, t = 0; w < nwork; t += tcnt[w++]) work[w] = w, tbeg[w] = t;
  std::vector<unsigned char> l2t(nwork, 0);
  std::vector<kifmm::LeafItem> items;
  std::vector<kifmm::LeafSplit> splits;
  kifmm::leaf_items(nwork, work.data(), tcnt, scnt, nptr, nidx, mptr, l2t.data(), tbeg.data(), nsurf, least, num_sms,
                    &items, &splits, nparts);
  *nsplit = (int)splits.size();
  for (int i = 0; i < (int)items.size() && i < cap; i++) {
    const kifmm::LeafItem& it = items[i];
    const int r[8] = {it.g, it.tb, (int)it.nb, it.nn, it.skip, it.take, it.nm, it.out};
    for (int k = 0; k < 8; k++) rows[8 * i + k] = r[k];
  }
  return (int)items.size();
}

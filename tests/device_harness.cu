// Device functions and kernels of the library called one at a time, for the
// tests that check them against values computed on the host.
#include <cuda_runtime.h>

#include <algorithm>
#include <initializer_list>
#include <vector>

#include "kernels_common.cuh"
#include "launch.hpp"
#include "operators.hpp"

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

namespace {
template <typename T>
struct Dev {  // a device copy of a host array
  T* p = nullptr;
  cudaError_t e = cudaSuccess;
  Dev(const T* h, size_t n) {
    if (!h) return;
    e = cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T));
    if (e == cudaSuccess) e = cudaMemcpy(p, h, n * sizeof(T), cudaMemcpyHostToDevice);
  }
  ~Dev() { cudaFree(p); }
};
}  // namespace

// C[cidx[j]] (=|+=) scale(A (M x K) B[bidx[j]]) for j < ncol, by the library's node
// contractions: FP64, or with T = float the tensor-core ones, whose operator is
// split on the host.  B has nb columns of ldb values, C nc of ldc (host
// arrays); col_lvl (ncol) may be null.  Returns a cudaError, or -1 where a device-side
// wait timed out.
template <typename T>
static int node_gemm(int M, int K, const double* A, int nb, int ldb, const T* B, const int* bidx, int nc, int ldc, T* C,
                     const int* cidx, int ncol, int accumulate, int sd, const int* deg, const int* col_lvl,
                     int lvl_base, int num_sms) {
  Dev<T> b(B, (size_t)nb * ldb), c(C, (size_t)nc * ldc);
  Dev<int> bi(bidx, ncol), ci(cidx, ncol), lv(col_lvl, ncol);
  const int zero = 0;
  Dev<int> status(&zero, 1);
  kifmm::GemmScale sc;
  sc.col_lvl = lv.p;
  sc.lvl_base = lvl_base;
  sc.sd = sd;
  for (int s = 0; s < sd; s++) sc.deg[s] = deg[s];
  for (int e : std::initializer_list<int>{b.e, c.e, bi.e, ci.e, lv.e, status.e})
    if (e != cudaSuccess) return e;
  if constexpr (sizeof(T) == 8) {
    Dev<double> a(A, (size_t)M * K);
    if (a.e != cudaSuccess) return (int)a.e;
    kifmm::launch_node_gemm64(M, K, a.p, b.p, ldb, bi.p, c.p, ldc, ci.p, ncol, accumulate != 0, sc, num_sms, 0);
    cudaDeviceSynchronize();
  } else {
    std::vector<float> img;
    kifmm::TcOperator op;
    kifmm::tc_operator_images(M, K, A, &img, &op);
    Dev<float> a(img.data(), img.size());
    if (a.e != cudaSuccess) return (int)a.e;
    op.img = a.p;
    kifmm::launch_node_gemm_tc(op, b.p, ldb, bi.p, c.p, ldc, ci.p, ncol, accumulate != 0, sc, num_sms, status.p, 0);
    cudaDeviceSynchronize();
  }
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(C, c.p, (size_t)nc * ldc * sizeof(T), cudaMemcpyDeviceToHost);
  int timed_out = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&timed_out, status.p, sizeof(int), cudaMemcpyDeviceToHost);
  return e != cudaSuccess ? (int)e : timed_out ? -1 : 0;
}

extern "C" int harness_gemm64(int M, int K, const double* A, int nb, int ldb, const double* B, const int* bidx, int nc,
                              int ldc, double* C, const int* cidx, int ncol, int accumulate, int sd, const int* deg,
                              const int* col_lvl, int lvl_base, int num_sms) {
  return node_gemm<double>(M, K, A, nb, ldb, B, bidx, nc, ldc, C, cidx, ncol, accumulate, sd, deg, col_lvl, lvl_base,
                           num_sms);
}
extern "C" int harness_gemm32(int M, int K, const double* A, int nb, int ldb, const float* B, const int* bidx, int nc,
                              int ldc, float* C, const int* cidx, int ncol, int accumulate, int sd, const int* deg,
                              const int* col_lvl, int lvl_base, int num_sms) {
  return node_gemm<float>(M, K, A, nb, ldb, B, bidx, nc, ldc, C, cidx, ncol, accumulate, sd, deg, col_lvl, lvl_base,
                          num_sms);
}

// the library's truncated pseudo-inverse of a (m x n, row-major) as factors V (n x
// rank) and W (rank x m); returns the rank, or -1
extern "C" int harness_pinv(int m, int n, const double* a, double rel_cut, double* V, double* W) {
  std::vector<double> v, w;
  int rank = 0;
  if (!kifmm::pinv_factors(m, n, a, rel_cut, 4, &v, &w, &rank)) return -1;
  std::copy(v.begin(), v.end(), V);
  std::copy(w.begin(), w.end(), W);
  return rank;
}

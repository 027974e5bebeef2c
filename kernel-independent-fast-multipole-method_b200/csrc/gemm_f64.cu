// FP64 node GEMM for the surface contractions (gemm.cu has the operators and
// the reference lines they replace), on mma.m8n8k4.f64: rows = nodes, columns =
// operator rows, so that a lane's two results are adjacent in the node's output.
//
// A CTA computes 64 nodes x 32 NT operator rows (NT = 5: the ranks and surfaces of
// np >= 6, 152 of 160 columns at np = 6; NT = 2 for operators of at most 64 rows
// and where it pads less), 8 warps of 32 x 8 NT.  K advances 16 at a time through
// three stages of 16-byte cp.async copies; a lane reads two K steps of a row at
// once (K is summed in the order 0 2 4 6, 1 3 5 7 of each 8), rows 64 bytes apart,
// so fragment loads are conflict-free and take 28 % of the load path.  A launch
// with few tiles (the shallow levels, K = 8 r) splits K over a cluster of up to
// 8 CTAs, which add their tiles through distributed shared memory in rank
// order: no workspace and no second launch.
//
// Bound: the FP64 pipe (the matrix instructions run at its rate, 37 TFLOP/s).
// At 4M points, np = 6, the SIMT form this replaces (64 x 64 tiles of scalar
// multiply-adds, 8 deep, unpipelined) ran at 29 % of the pipe.
#include <cooperative_groups.h>

#include <algorithm>

#include "launch.hpp"

namespace kifmm {
namespace {

namespace cg = cooperative_groups;

constexpr int G_THREADS = 256, G_NODES = 64, G_BK = 16, G_STAGES = 3;

__device__ __forceinline__ void mma64(double* c, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// 16 bytes, or zeros where !ok
__device__ __forceinline__ void copy16(unsigned dst, const double* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

__device__ __forceinline__ double row_scale64(const GemmScale& sc, int lvl, int r) {
  const int s = sc.sd == 1 ? 0 : r % sc.sd;
  return ldexp(1.0, -lvl * (s == 0 ? sc.deg[0] : s == 1 ? sc.deg[1] : s == 2 ? sc.deg[2] : sc.deg[3]));
}

template <int NT>
__global__ void __launch_bounds__(G_THREADS, 2)
    k_node_gemm64(int M, int K, int kper, int ks, const double* __restrict__ A, const double* B, int64_t ldb,
                  const int* __restrict__ bidx, double* C, int64_t ldc, const int* __restrict__ cidx, int ncol,
                  int accumulate, GemmScale sc) {
  constexpr int OPS = 32 * NT, ROWS = G_NODES + OPS, STAGE = ROWS * G_BK;  // doubles per stage
  extern __shared__ __align__(16) double sm[];                            // [stage][half][row][8]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane >> 2, lk = lane & 3;
  const int z = ks > 1 ? (int)(blockIdx.x % ks) : 0;
  const int n0 = (int)(blockIdx.x / ks) * G_NODES, m0 = blockIdx.y * OPS;
  const int kb = z * kper, ke = min(K, kb + kper);
  // copies: this thread's 16 bytes (column 2 q of 16) of rows (tid >> 3) + 32 i
  const int q = tid & 7, r0 = tid >> 3;
  const double* bsrc[G_NODES / 32];
#pragma unroll
  for (int i = 0; i < G_NODES / 32; i++) {
    const int j = n0 + r0 + 32 * i;
    bsrc[i] = j < ncol ? B + (int64_t)bidx[j] * ldb + 2 * q : nullptr;
  }
  const double* asrc = A + (size_t)(m0 + r0) * K + 2 * q;
  const unsigned dst0 = (unsigned)__cvta_generic_to_shared(sm) + (((q >> 2) * ROWS + r0) * 8 + (q & 3) * 2) * 8;
  auto fill = [&](int stage, int k0) {
    const unsigned d = dst0 + stage * (STAGE * 8);
    const bool in = k0 + 2 * q < ke;
#pragma unroll
    for (int i = 0; i < G_NODES / 32; i++) {
      const bool ok = in && bsrc[i];
      copy16(d + i * (32 * 64), ok ? bsrc[i] + k0 : A, ok);
    }
#pragma unroll
    for (int i = 0; i < NT; i++) {
      const bool ok = in && m0 + r0 + 32 * i < M;
      copy16(d + (G_NODES + 32 * i) * 64, ok ? asrc + (size_t)(32 * i) * K + k0 : A, ok);
    }
  };
  double acc[4][NT][2];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < NT; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int wn = (warp & 1) * 32, wm = (warp >> 1) * (8 * NT);  // the warp's first node and operator row
  const int steps = ke > kb ? (ke - kb + G_BK - 1) / G_BK : 0;
  wait_for_previous();
  dependents_may_start();
#pragma unroll
  for (int s = 0; s < G_STAGES - 1; s++) {
    if (s < steps) fill(s, kb + s * G_BK);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int s = 0, st = 0; s < steps; s++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(G_STAGES - 2) : "memory");
    __syncthreads();  // stage st has landed for all, and the stage of step s - 1 has been read by all
    const int nst = st == 0 ? G_STAGES - 1 : st - 1;
    if (s + G_STAGES - 1 < steps) fill(nst, kb + (s + G_STAGES - 1) * G_BK);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const double* base = sm + st * STAGE;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const double* hb = base + h * (ROWS * 8) + lk * 2;
      double2 a[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = *reinterpret_cast<const double2*>(hb + (wn + 8 * i + lr) * 8);
#pragma unroll
      for (int j = 0; j < NT; j++) {
        const double2 b = *reinterpret_cast<const double2*>(hb + (G_NODES + wm + 8 * j + lr) * 8);
#pragma unroll
        for (int i = 0; i < 4; i++) mma64(acc[i][j], a[i].x, b.x);
#pragma unroll
        for (int i = 0; i < 4; i++) mma64(acc[i][j], a[i].y, b.y);
      }
    }
    st = st + 1 == G_STAGES ? 0 : st + 1;
  }
  auto store = [&](int j, int r, double v0, double v1) {  // results r, r + 1 (both < M, M even) of column j
    double* p = C + (int64_t)cidx[j] * ldc + r;
    if (sc.col_lvl) {
      const int lvl = sc.col_lvl[j] + sc.lvl_base;
      v0 *= row_scale64(sc, lvl, r);
      v1 *= row_scale64(sc, lvl, r + 1);
    }
    double2 v = make_double2(v0, v1);
    if (accumulate) {
      const double2 o = *reinterpret_cast<const double2*>(p);
      v.x += o.x;
      v.y += o.y;
    }
    *reinterpret_cast<double2*>(p) = v;
  };
  if (ks == 1) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int j = n0 + wn + 8 * i + lr;
      if (j >= ncol) continue;
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const int r = m0 + wm + 8 * t + 2 * lk;
        if (r < M) store(j, r, acc[i][t][0], acc[i][t][1]);
      }
    }
    return;
  }
  // K split over the cluster: every CTA leaves its tile in shared memory and
  // adds one part of all tiles, in rank order
  cg::cluster_group cl = cg::this_cluster();
  __syncthreads();
  double2* tile = reinterpret_cast<double2*>(sm);  // [64][OPS / 2]
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int t = 0; t < NT; t++)
      tile[(wn + 8 * i + lr) * (OPS / 2) + (wm + 8 * t) / 2 + lk] = make_double2(acc[i][t][0], acc[i][t][1]);
  cl.sync();
  for (int e = z * G_THREADS + tid; e < G_NODES * OPS / 2; e += ks * G_THREADS) {
    const int j = n0 + e / (OPS / 2), r = m0 + 2 * (e % (OPS / 2));
    if (j >= ncol || r >= M) continue;
    double2 s = make_double2(0.0, 0.0);
    for (int p = 0; p < ks; p++) {
      const double2 v = *cl.map_shared_rank(tile + e, p);
      s.x += v.x;
      s.y += v.y;
    }
    store(j, r, s.x, s.y);
  }
  cl.sync();  // no CTA ends while another reads its tile
}

template <int NT>
void launch_nt(int M, int K, const double* A, const double* B, int64_t ldb, const int* bidx, double* C, int64_t ldc,
               const int* cidx, int ncol, bool accumulate, const GemmScale& sc, int num_sms, cudaStream_t st) {
  const int nt = (ncol + G_NODES - 1) / G_NODES, mt = (M + 32 * NT - 1) / (32 * NT);
  // split K where the tiles leave SMs idle: at least four stages each
  int ks = 1;
  while (ks < 8 && nt * mt * ks * 2 <= num_sms && K >= 2 * ks * 4 * G_BK) ks *= 2;
  const int kper = ((K + ks - 1) / ks + G_BK - 1) / G_BK * G_BK;
  // a grid of at most one CTA per SM asks for more than half an SM's shared memory:
  // placed early beside the kernel before it, its CTAs would pair up on the SMs
  // that are freed first
  const bool few = (int64_t)nt * mt * ks <= num_sms;
  constexpr size_t stages = (size_t)G_STAGES * (G_NODES + 32 * NT) * G_BK * sizeof(double);
  constexpr size_t most = std::max(stages, (size_t)120 << 10);
  const size_t smem = few ? most : stages;
  auto kern = k_node_gemm64<NT>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);  // the same at every launch (launch.hpp)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nt * ks, mt, 1);
  cfg.blockDim = dim3(G_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ks;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = few ? 2 : 1;  // dependent (launch.hpp)
  cudaLaunchKernelEx(&cfg, kern, M, K, kper, ks, A, B, ldb, bidx, C, ldc, cidx, ncol, accumulate ? 1 : 0, sc);
}

}  // namespace

int launch_node_gemm64(int M, int K, const double* A, const double* B, int64_t ldb, const int* bidx, double* C,
                       int64_t ldc, const int* cidx, int ncol, bool accumulate, const GemmScale& sc, int num_sms,
                       cudaStream_t st) {
  if (ncol <= 0 || M <= 0 || K <= 0) return 0;
  // columns of padding: 32 NT per tile
  const int wide = (M + 159) / 160 * 160, narrow = (M + 63) / 64 * 64;
  if (M <= 64 || narrow * 5 < wide * 4)
    launch_nt<2>(M, K, A, B, ldb, bidx, C, ldc, cidx, ncol, accumulate, sc, num_sms, st);
  else
    launch_nt<5>(M, K, A, B, ldb, bidx, C, ldc, cidx, ncol, accumulate, sc, num_sms, st);
  return 1;
}

}  // namespace kifmm

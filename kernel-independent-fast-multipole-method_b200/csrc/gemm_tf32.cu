// Node GEMM for the FP32 surface contractions of the mixed-precision engine with
// few columns, the levels of a tree (gemm_tc.cu, tcgen05, has the large ones;
// gemm.cu the operators and the reference lines they replace), on mma.m16n8k8
// with both operands split into a TF32 head and a TF32 tail:
//
//   D[node][out] = sum_k data[node][k] * op[out][k]
//   head*head + head*tail + tail*head   (tail*tail, 2^-22 relative, is dropped)
//
// A CTA computes 64 nodes x 32 NT operator rows (NT = 5, or 2 for operators of at
// most 64 rows), 8 warps of 32 x 8 NT.  K advances in chunks of 32 through two
// stages of 16-byte cp.async copies: the node columns as they are, split in
// registers, and the operator's head and tail as laid out once on the host
// (tc_operator_images, 8 x 4 blocks of 128 bytes: a fragment is one
// conflict-free load).  Few tiles (the shallow tree levels, K = 8 r) split K
// over a cluster of up to 8 CTAs that add their tiles in FP64 through
// distributed shared memory, in rank order.
//
// Precision: the tensor core adds an MMA's products to its accumulator with one
// alignment, whose rounding error grows with every MMA folded into it.  Each
// chunk's 12 MMAs therefore start from zero and the chunks are summed in
// FP32 registers (round to nearest), which keeps the contractions -- which
// cancel strongly in the Sigma^-1 U^T factors -- in the error class of FP32
// multiply-add accumulation.
//
// Where the line to tcgen05 lies: a launch of fewer 128-node tiles than SMs.  There
// the tcgen05 form is bound by its chunk round trip (node load, split, MMA,
// TMEM drain) and needed K slices in a workspace and a second launch to add
// them: 28 + 5 us for 450 columns at K = 1,216, here 12.  mma.sync's TF32 rate (277
// TFLOP/s measured, a third of it useful) bounds the large launches: all levels
// of 4M points, upward 1.94 ms here against 1.69 on tcgen05.
#include <cooperative_groups.h>

#include <algorithm>

#include "launch.hpp"

namespace kifmm {
namespace {

namespace cg = cooperative_groups;

constexpr int F_THREADS = 256, F_NODES = 64, F_KC = 32, F_STAGES = 2;
constexpr int F_PITCH = 36;                     // floats per staged node row: fragment loads touch all banks
constexpr int F_ROWS = 160;                     // operator rows per image tile
constexpr int F_IMG = 2 * F_ROWS * F_KC;        // floats of one (tile, chunk) image: head, tail
constexpr int F_NODE = F_NODES * F_PITCH;

__device__ __forceinline__ void mma_tf32(float* c, const unsigned* a, unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ unsigned tf32_round(float x) { return (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u; }

// 16 bytes, or zeros where !ok
__device__ __forceinline__ void copy16(unsigned dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

// 2^e as a float (e in the normal range), else ldexpf
__device__ __forceinline__ float pow2f(int e) {
  return (e >= -126 && e <= 127) ? __int_as_float((e + 127) << 23) : ldexpf(1.0f, e);
}

template <int NT>
__global__ void __launch_bounds__(F_THREADS, 2)
    k_node_gemm_tf32(TcOperator A, int cper, int ks, const float* B, int64_t ldb, const int* __restrict__ bidx, float* C,
                     int64_t ldc, const int* __restrict__ cidx, int ncol, int accumulate, GemmScale sc) {
  constexpr int OPS = 32 * NT, IMG = 2 * OPS * F_KC, STAGE = F_NODE + IMG;  // floats
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane >> 2, lk = lane & 3;
  const int z = ks > 1 ? (int)(blockIdx.x % ks) : 0;
  const int n0 = (int)(blockIdx.x / ks) * F_NODES, y = blockIdx.y, m0 = y * A.ntile;
  const int nkt = A.Kp / F_KC, cb = z * cper, ce = min(nkt, cb + cper);
  // node copies: 16 bytes (floats 4 q ..) of rows (tid >> 3) and (tid >> 3) + 32
  const int q = tid & 7, r0 = tid >> 3;
  const float* bsrc[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int j = n0 + r0 + 32 * i;
    bsrc[i] = j < ncol ? B + (int64_t)bidx[j] * ldb + 4 * q : nullptr;
  }
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(sm);
  const float* img = A.img + (size_t)y * nkt * F_IMG;
  auto fill = [&](int stage, int c) {
    const unsigned d = sbase + stage * (STAGE * 4);
    const bool in = c * F_KC + 4 * q < A.K;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const bool ok = in && bsrc[i];
      copy16(d + ((r0 + 32 * i) * F_PITCH + 4 * q) * 4, ok ? bsrc[i] + c * F_KC : A.img, ok);
    }
    const float* s = img + (size_t)c * F_IMG;
#pragma unroll
    for (int i = 0; i < IMG / 4 / F_THREADS; i++) {  // head, then tail (their first OPS rows)
      const int e = tid + F_THREADS * i, half = e / (OPS * F_KC / 4), o = e % (OPS * F_KC / 4);
      copy16(d + (F_NODE + 4 * e) * 4, s + half * (F_ROWS * F_KC) + 4 * o, true);
    }
  };
  float acc[2][NT][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[i][j][e] = 0.f;
  const int wn = (warp & 1) * 32, wm = (warp >> 1) * NT;  // the warp's first node and 8-row operator block
  const int steps = max(ce - cb, 0);
  wait_for_previous();
  dependents_may_start();
  if (steps > 0) fill(0, cb);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int s = 0; s < steps; s++) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // chunk s has landed for all, and the other stage has been read by all
    if (s + 1 < steps) fill((s + 1) & 1, cb + s + 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* nd = sm + (s & 1) * STAGE + (wn + lr) * F_PITCH + lk;
    const unsigned* op = reinterpret_cast<const unsigned*>(sm + (s & 1) * STAGE + F_NODE) + wm * 256 + lane;
    float t[2][NT][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) t[i][j][e] = 0.f;
#pragma unroll
    for (int k8 = 0; k8 < F_KC / 8; k8++) {
      unsigned ah[2][4], al[2][4];
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) {  // (row, k), (row + 8, k), (row, k + 4), (row + 8, k + 4)
          const float v = nd[(16 * i + 8 * (e & 1)) * F_PITCH + 8 * k8 + 4 * (e >> 1)];
          ah[i][e] = tf32_round(v);
          al[i][e] = tf32_round(v - __uint_as_float(ah[i][e]));
        }
#pragma unroll
      for (int j = 0; j < NT; j++) {
        const unsigned* o = op + j * 256 + k8 * 64;
        const unsigned h0 = o[0], h1 = o[32], l0 = o[OPS * F_KC], l1 = o[OPS * F_KC + 32];
        // (an accumulator's three products two apart, so that a warp's MMAs overlap)
        mma_tf32(t[0][j], ah[0], h0, h1);
        mma_tf32(t[1][j], ah[1], h0, h1);
        mma_tf32(t[0][j], ah[0], l0, l1);
        mma_tf32(t[1][j], ah[1], l0, l1);
        mma_tf32(t[0][j], al[0], h0, h1);
        mma_tf32(t[1][j], al[1], h0, h1);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[i][j][e] += t[i][j][e];
  }
  // results r, r + 1 (r even, both below M) of column j
  auto scale = [&](int j, int r, float& f0, float& f1) {
    f0 = f1 = 1.f;
    if (!sc.col_lvl) return;
    const int lvl = sc.col_lvl[j] + sc.lvl_base, s0 = sc.sd == 1 ? 0 : r % sc.sd, s1 = sc.sd == 1 ? 0 : (r + 1) % sc.sd;
    auto deg = [&](int s) { return s == 0 ? sc.deg[0] : s == 1 ? sc.deg[1] : s == 2 ? sc.deg[2] : sc.deg[3]; };
    f0 = pow2f(-lvl * deg(s0));
    f1 = pow2f(-lvl * deg(s1));
  };
  if (ks == 1) {
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int j = n0 + wn + 16 * i + 8 * h + lr;
        if (j >= ncol) continue;
        float* crow = C + (int64_t)cidx[j] * ldc;
#pragma unroll
        for (int n = 0; n < NT; n++) {
          const int o = 8 * (wm + n) + 2 * lk, r = m0 + o;
          if (o >= A.ntile || r >= A.M) continue;
          float f0, f1;
          scale(j, r, f0, f1);
          float2 v = make_float2(acc[i][n][2 * h] * f0, acc[i][n][2 * h + 1] * f1);
          float2* p = reinterpret_cast<float2*>(crow + r);
          if (accumulate) {
            const float2 c = *p;
            v.x += c.x;
            v.y += c.y;
          }
          *p = v;
        }
      }
    return;
  }
  // K split over the cluster: every CTA leaves its tile in shared memory and
  // adds one part of all tiles, in FP64 and rank order
  cg::cluster_group cl = cg::this_cluster();
  __syncthreads();
  float2* tile = reinterpret_cast<float2*>(sm);  // [64][OPS / 2]
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int n = 0; n < NT; n++)
        tile[(wn + 16 * i + 8 * h + lr) * (OPS / 2) + 4 * (wm + n) + lk] =
            make_float2(acc[i][n][2 * h], acc[i][n][2 * h + 1]);
  cl.sync();
  for (int e = z * F_THREADS + tid; e < F_NODES * OPS / 2; e += ks * F_THREADS) {
    const int j = n0 + e / (OPS / 2), o = 2 * (e % (OPS / 2)), r = m0 + o;
    if (j >= ncol || o >= A.ntile || r >= A.M) continue;
    double v0 = 0.0, v1 = 0.0;
    for (int p = 0; p < ks; p++) {
      const float2 v = *cl.map_shared_rank(tile + e, p);
      v0 += (double)v.x;
      v1 += (double)v.y;
    }
    float f0, f1;
    scale(j, r, f0, f1);
    v0 *= (double)f0;
    v1 *= (double)f1;
    float2* p = reinterpret_cast<float2*>(C + (int64_t)cidx[j] * ldc + r);
    if (accumulate) {
      const float2 c = *p;
      v0 += (double)c.x;
      v1 += (double)c.y;
    }
    *p = make_float2((float)v0, (float)v1);
  }
  cl.sync();  // no CTA ends while another reads its tile
}

template <int NT>
void launch_nt(const TcOperator& A, const float* B, int64_t ldb, const int* bidx, float* C, int64_t ldc,
               const int* cidx, int ncol, bool accumulate, const GemmScale& sc, int num_sms, cudaStream_t st) {
  const int nt = (ncol + F_NODES - 1) / F_NODES, nkt = A.Kp / F_KC;
  // split K where the tiles leave SMs idle (two CTAs fit one): two chunks each at least
  int ks = 1;
  while (ks < 8 && (int64_t)nt * A.ntiles * ks <= num_sms && nkt >= 4 * ks) ks *= 2;
  const int cper = (nkt + ks - 1) / ks;
  // a grid of at most one CTA per SM asks for more than half an SM's shared memory:
  // placed early beside the kernel before it, its CTAs would pair up on the SMs
  // that are freed first
  const bool few = (int64_t)nt * A.ntiles * ks <= num_sms;
  constexpr size_t stages = (size_t)F_STAGES * (F_NODE + 2 * 32 * NT * F_KC) * sizeof(float);
  constexpr size_t most = std::max(stages, (size_t)120 << 10);
  const size_t smem = few ? most : stages;
  auto kern = k_node_gemm_tf32<NT>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);  // the same at every launch (launch.hpp)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nt * ks, A.ntiles, 1);
  cfg.blockDim = dim3(F_THREADS, 1, 1);
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
  cudaLaunchKernelEx(&cfg, kern, A, cper, ks, B, ldb, bidx, C, ldc, cidx, ncol, accumulate ? 1 : 0, sc);
}

}  // namespace

int launch_node_gemm_tf32(const TcOperator& A, const float* B, int64_t ldb, const int* bidx, float* C, int64_t ldc,
                          const int* cidx, int ncol, bool accumulate, const GemmScale& sc, int num_sms,
                          cudaStream_t st) {
  if (ncol <= 0 || A.M <= 0 || A.K <= 0) return 0;
  if (A.ntile <= 64)
    launch_nt<2>(A, B, ldb, bidx, C, ldc, cidx, ncol, accumulate, sc, num_sms, st);
  else
    launch_nt<5>(A, B, ldb, bidx, C, ldc, cidx, ncol, accumulate, sc, num_sms, st);
  return 1;
}

}  // namespace kifmm

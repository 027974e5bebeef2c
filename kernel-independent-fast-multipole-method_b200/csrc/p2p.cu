// Point <-> point and point <-> surface evaluation passes.
//
//   k_s2m_warp   S2M  : leaf sources -> its upward check surface      (SE2UC_dgemv, fmm3d/fmm3d.cpp:62-71)
//   k_s2l        S2L  : X-list leaf sources -> downward check surface  (SE2DC_dgemv, fmm3d/fmm3d.cpp:73-82)
//   k_leaf_warp  near : U list + direct W/X (SE2TC_dgemv, fmm3d/fmm3d.cpp:35-60), M2T from W-list
//                       upward equivalent surfaces (UE2TC_dgemv, :114-141) and L2T from the leaf's own
//                       downward equivalent surface (DE2TC_dgemv, :84-112), fused into one pass that
//                       writes each target once.
//
// S2M and the leaf pass run warps on leaves (see below); S2L, rare, CTAs on a
// node's check points with shared-memory tiles.  Every target accumulates in registers.
// Positions are stored relative to the centre of their leaf and re-centred on
// the target node's centre while staging, so FP32 differences lose no more
// than the node size's precision.
#include "host_parallel.hpp"
#include "kernels_common.cuh"
#include "launch.hpp"

namespace kifmm {

namespace {

constexpr int P2P_THREADS = 128;
constexpr int TILE = 256;

template <typename T, int SDMAX>
struct Tile {
  T x[TILE], y[TILE], z[TILE];
  T nx[TILE], ny[TILE], nz[TILE];
  T f[TILE * SDMAX];
};

template <typename T, int TDMAX>
struct Red {
  T v[P2P_THREADS * TDMAX];
};

// Packed staged source: (x, y, z, first density component); a single-dof
// single-layer interaction then reads one 16-byte (FP32) word, and lap_pairs a
// pair of sources as two of them.
template <typename T>
struct alignas(16) P4 {
  T x, y, z, w;
};

template <typename T, int KT>
__device__ __forceinline__ void accumulate_tile(const Tile<T, 4>& t, int cnt, int j0, int jstep, T px, T py, T pz,
                                                T* acc, const KConst<T>& kc) {
  constexpr int SD = KTraits<KT>::SD;
#pragma unroll 4
  for (int j = j0; j < cnt; j += jstep) {
    T nrm[3];
    if constexpr (KTraits<KT>::DL) {
      nrm[0] = t.nx[j];
      nrm[1] = t.ny[j];
      nrm[2] = t.nz[j];
    }
    keval<KT, T>(px - t.x[j], py - t.y[j], pz - t.z[j], nrm, &t.f[j * SD], acc, kc);
  }
}

template <typename T, int TD>
__device__ __forceinline__ void reduce_and_store(Red<T, 4>& red, const T* acc, int G, int nsplit, bool valid,
                                                 T* out, bool add) {
  int slot = threadIdx.x % G, sg = threadIdx.x / G;
  if (sg < nsplit) {
#pragma unroll
    for (int d = 0; d < TD; d++) red.v[(sg * G + slot) * TD + d] = acc[d];
  }
  __syncthreads();
  if (sg == 0 && valid) {
#pragma unroll
    for (int d = 0; d < TD; d++) {
      T s = red.v[slot * TD + d];
      for (int q = 1; q < nsplit; q++) s += red.v[(q * G + slot) * TD + d];
      if (add)
        out[d] += s;
      else
        out[d] = s;
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// S2L: CTA (w, b) sums the X-list sources of work item w at downward check
// points 32 b .. 32 b + 31, each point's sources over its four warps.  The list's
// leaves are small and many (they are finer than the node), so 128 of them at a
// time get a prefix sum and the sources are staged 256 at a time across leaf
// borders.  One CTA per node and a barrier pair per leaf, the form before, was
// latency: 44 us for 70 nodes of a 262,144-point tree, now 12.
template <typename T, int KT>
__global__ void __launch_bounds__(P2P_THREADS) k_s2l(P2PArgs<T> a, const int* work, const int64_t* ptr,
                                                      const int* idx, int rhs) {
  constexpr int SD = KTraits<KT>::SD, TD = KTraits<KT>::TD;
  constexpr bool DL = KTraits<KT>::DL;
  constexpr int G = 32, NSPLIT = P2P_THREADS / G;
  __shared__ Tile<T, 4> tile;
  __shared__ Red<T, 4> red;
  __shared__ int lbeg[P2P_THREADS], pre[P2P_THREADS + 1], wsum[NSPLIT];
  __shared__ T lx[P2P_THREADS], ly[P2P_THREADS], lz[P2P_THREADS];
  wait_for_previous();
  dependents_may_start();
  const int w = blockIdx.x, g = work[w], tid = threadIdx.x, lane = tid & 31;
  const T rad = (T)a.radius[g];
  const double cx = a.center[3 * g], cy = a.center[3 * g + 1], cz = a.center[3 * g + 2];
  const int ti = blockIdx.y * G + lane, sg = tid >> 5;
  const bool valid = ti < a.nsurf;
  T px = 0, py = 0, pz = 0;
  if (valid) {
    px = a.dc_unit[3 * ti] * rad;
    py = a.dc_unit[3 * ti + 1] * rad;
    pz = a.dc_unit[3 * ti + 2] * rad;
  }
  const T* den = a.sden + (size_t)rhs * a.ns * SD;
  T acc[4] = {0, 0, 0, 0};
  for (int64_t e0 = ptr[w]; e0 < ptr[w + 1]; e0 += P2P_THREADS) {
    const int nleaf = (int)min((int64_t)P2P_THREADS, ptr[w + 1] - e0);
    int c = 0;
    if (tid < nleaf) {
      const int s = idx[e0 + tid];
      lbeg[tid] = a.sbeg[s];
      c = a.scnt[s];
      lx[tid] = (T)(a.center[3 * s] - cx);
      ly[tid] = (T)(a.center[3 * s + 1] - cy);
      lz[tid] = (T)(a.center[3 * s + 2] - cz);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, c, o);
      if (lane >= o) c += v;
    }
    if (lane == 31) wsum[sg] = c;
    __syncthreads();
    for (int q = 0; q < sg; q++) c += wsum[q];
    pre[tid + 1] = c;
    if (tid == 0) pre[0] = 0;
    __syncthreads();
    const int total = pre[P2P_THREADS];
    for (int k0 = 0; k0 < total; k0 += TILE) {
      const int cnt = min(TILE, total - k0);
      for (int j = tid; j < cnt; j += P2P_THREADS) {
        int lo = 0, hi = nleaf;  // pre[lo] <= k0 + j < pre[hi]
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (pre[mid] <= k0 + j)
            lo = mid;
          else
            hi = mid;
        }
        const int p = lbeg[lo] + (k0 + j - pre[lo]);
        tile.x[j] = a.sx[p] + lx[lo];
        tile.y[j] = a.sy[p] + ly[lo];
        tile.z[j] = a.sz[p] + lz[lo];
        if constexpr (DL) {
          tile.nx[j] = a.snx[p];
          tile.ny[j] = a.sny[p];
          tile.nz[j] = a.snz[p];
        }
#pragma unroll
        for (int s = 0; s < SD; s++) tile.f[j * SD + s] = den[(size_t)p * SD + s];
      }
      __syncthreads();
      if (valid) accumulate_tile<T, KT>(tile, cnt, sg, NSPLIT, px, py, pz, acc, a.ku);
      __syncthreads();
    }
  }
  reduce_and_store<T, TD>(red, acc, G, NSPLIT, valid, a.tdncval + ((size_t)g * a.nsurf + ti) * TD, true);
}

// ---------------------------------------------------------------------------
// Warp-per-leaf forms.  A warp owns one leaf, stages its sources 32 at a time
// in a private slice of shared memory and synchronises with __syncwarp only,
// so the other warps of the SM keep issuing while it waits on its loads.
constexpr int WP_WARPS = 8;  // warps per CTA

template <typename T>
struct WarpSrc {  // one staged batch of 32 sources
  P4<T> p[32];
  T f[32 * 3];
  T n[32 * 3];
};

template <typename T>
struct WarpSrc64 {  // one staged batch of 64 sources
  P4<T> p[64];
  T f[64 * 3];
  T n[64 * 3];
};

// Single-dof Laplace sums in FP32 run on packed f32x2 arithmetic, two
// sources per instruction: the staged batch is then pair-interleaved,
// pair q = sources 2q, 2q + 1 as {x0, x1, y0, y1} {z0, z1, w0, w1}, so one
// pair is two 16-byte shared loads already in packed-register order.
template <typename T>
__device__ __forceinline__ void stage_src(WarpSrc64<T>& w, int j, P4<T> v, bool paired) {
  if (!paired) {
    w.p[j] = v;
    return;
  }
  T* q = reinterpret_cast<T*>(w.p) + 8 * (j >> 1) + (j & 1);
  q[0] = v.x;
  q[2] = v.y;
  q[4] = v.z;
  q[6] = v.w;
}

__device__ __forceinline__ unsigned long long pk2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void upk2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// s[k] = sum over the pairs q = sg, sg + nsplit, ... < npairs of w / |t_k - s|
// (the 1e-16 cut-off as in keval), for two targets t_k = (px, py, pz)[k]
__device__ __forceinline__ void lap_pairs(const WarpSrc64<float>& w, const float* px, const float* py,
                                          const float* pz, int sg, int nsplit, int npairs, float* s) {
  static_assert(alignof(WarpSrc64<float>) % alignof(float4) == 0, "16-byte loads of the staged sources");
  const float4* wp = reinterpret_cast<const float4*>(w.p);
  unsigned long long PX[2], PY[2], PZ[2], S[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    PX[k] = pk2(px[k], px[k]);
    PY[k] = pk2(py[k], py[k]);
    PZ[k] = pk2(pz[k], pz[k]);
    S[k] = pk2(0.f, 0.f);
  }
  const int rounds = sg < npairs ? (npairs - sg + nsplit - 1) / nsplit : 0;
#pragma unroll 4
  for (int r = 0; r < rounds; r++) {
    const int q = sg + r * nsplit;
    const float4 A = wp[2 * q], B = wp[2 * q + 1];
    const unsigned long long SX = pk2(A.x, A.y), SY = pk2(A.z, A.w), SZ = pk2(B.x, B.y), SW = pk2(B.z, B.w);
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const unsigned long long X = sub2(PX[k], SX), Y = sub2(PY[k], SY), Z = sub2(PZ[k], SZ);
      unsigned long long R2 = mul2(X, X);
      R2 = fma2(Y, Y, R2);
      R2 = fma2(Z, Z, R2);
      float r2a, r2b;
      upk2(R2, r2a, r2b);
      const float ria = (r2a >= 1e-16f) ? rsqrt_t(r2a) : 0.f, rib = (r2b >= 1e-16f) ? rsqrt_t(r2b) : 0.f;
      S[k] = fma2(pk2(ria, rib), SW, S[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    float sa, sb;
    upk2(S[k], sa, sb);
    s[k] = sa + sb;
  }
}

// u_k += c * sum over the sources sg, sg + nsplit, ... (`rounds` of them) of w / |t_k - s|
template <typename T>
__device__ __forceinline__ void lap_points(const WarpSrc64<T>& w, const T* px, const T* py, const T* pz, int sg,
                                           int nsplit, int rounds, T c, T* u0, T* u1) {
  T s0 = T(0), s1 = T(0);
#pragma unroll 4
  for (int r = 0; r < rounds; r++) {
    const P4<T> s = w.p[sg + r * nsplit];
    const T x0 = px[0] - s.x, y0 = py[0] - s.y, z0 = pz[0] - s.z;
    const T x1 = px[1] - s.x, y1 = py[1] - s.y, z1 = pz[1] - s.z;
    s0 += rinv_cut(x0 * x0 + y0 * y0 + z0 * z0) * s.w;
    s1 += rinv_cut(x1 * x1 + y1 * y1 + z1 * z1) * s.w;
  }
  *u0 += c * s0;
  *u1 += c * s1;
}

// S2M: a warp carries R rounds of 32 upward check points of one leaf, of
// `parts` warps that share its check points; every staged source (a broadcast
// load) updates all of them.  All R rounds are computed, the last ones on
// check points past the end where there are any: a test per round keeps
// the rounds' chains from overlapping.
template <typename T, int KT, int R>
__global__ void __launch_bounds__(32 * WP_WARPS)
    k_s2m_warp(P2PArgs<T> a, const int* work, int nwork, int parts, int rhs) {
  constexpr int SD = KTraits<KT>::SD, TD = KTraits<KT>::TD;
  constexpr bool DL = KTraits<KT>::DL;
  __shared__ WarpSrc<T> ws[WP_WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WarpSrc<T>& w = ws[warp];
  wait_for_previous();
  dependents_may_start();
  const T* den = a.sden + (size_t)rhs * a.ns * SD;
  const int nt = a.nuc;
  for (int64_t wi = blockIdx.x * WP_WARPS + warp; wi < (int64_t)nwork * parts; wi += gridDim.x * WP_WARPS) {
    const int g = work[wi / parts], t0 = (int)(wi % parts) * (32 * R) + lane;
    const T rad = (T)a.radius[g];
    const int sb = a.sbeg[g], sc = a.scnt[g];
    T px[R], py[R], pz[R], acc[R][TD];
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int ti = t0 + 32 * r;
      px[r] = py[r] = pz[r] = T(0);
      if (ti < nt) {
        px[r] = a.uc_unit[3 * ti] * rad;
        py[r] = a.uc_unit[3 * ti + 1] * rad;
        pz[r] = a.uc_unit[3 * ti + 2] * rad;
      }
#pragma unroll
      for (int d = 0; d < TD; d++) acc[r][d] = T(0);
    }
    // FP32 Laplace: packed f32x2 sums over pairs of this lane's check points
    constexpr bool PACKED = KT == 111 && sizeof(T) == 4;
    unsigned long long PX[R / 2 > 0 ? R / 2 : 1], PY[R / 2 > 0 ? R / 2 : 1], PZ[R / 2 > 0 ? R / 2 : 1],
        SP[R / 2 > 0 ? R / 2 : 1];
    float s_last = 0.f;
    if constexpr (PACKED) {
#pragma unroll
      for (int rp = 0; rp < R / 2; rp++) {
        PX[rp] = pk2(px[2 * rp], px[2 * rp + 1]);
        PY[rp] = pk2(py[2 * rp], py[2 * rp + 1]);
        PZ[rp] = pk2(pz[2 * rp], pz[2 * rp + 1]);
        SP[rp] = pk2(0.f, 0.f);
      }
    }
    for (int c0 = 0; c0 < sc; c0 += 32) {
      const int cnt = min(32, sc - c0);
      __syncwarp();
      if (lane < cnt) {
        const int p = sb + c0 + lane;
        T f[SD], nrm[3] = {T(0), T(0), T(0)};
#pragma unroll
        for (int s = 0; s < SD; s++) f[s] = den[(size_t)p * SD + s];
        if constexpr (DL) {
          nrm[0] = a.snx[p];
          nrm[1] = a.sny[p];
          nrm[2] = a.snz[p];
        }
        w.p[lane] = P4<T>{a.sx[p], a.sy[p], a.sz[p], f[0]};
#pragma unroll
        for (int s = 1; s < SD; s++) w.f[lane * (SD - 1) + s - 1] = f[s];
        if constexpr (DL) {
          w.n[3 * lane] = nrm[0];
          w.n[3 * lane + 1] = nrm[1];
          w.n[3 * lane + 2] = nrm[2];
        }
      }
      __syncwarp();
      for (int j = 0; j < cnt; j++) {
        const P4<T> sp = w.p[j];
        T f[SD];
        f[0] = sp.w;
#pragma unroll
        for (int k = 1; k < SD; k++) f[k] = w.f[j * (SD - 1) + k - 1];
        T nrm[3];
        if constexpr (DL) {
          nrm[0] = w.n[3 * j];
          nrm[1] = w.n[3 * j + 1];
          nrm[2] = w.n[3 * j + 2];
        }
        if constexpr (PACKED) {
          // check points 2 rp, 2 rp + 1 as one f32x2 pair; an odd last round scalar
          const unsigned long long SX = pk2(sp.x, sp.x), SY = pk2(sp.y, sp.y), SZ = pk2(sp.z, sp.z),
                                   SW = pk2(sp.w, sp.w);
#pragma unroll
          for (int rp = 0; rp < R / 2; rp++) {
            const unsigned long long X = sub2(PX[rp], SX), Y = sub2(PY[rp], SY), Z = sub2(PZ[rp], SZ);
            unsigned long long R2 = mul2(X, X);
            R2 = fma2(Y, Y, R2);
            R2 = fma2(Z, Z, R2);
            float r2a, r2b;
            upk2(R2, r2a, r2b);
            const float ria = (r2a >= 1e-16f) ? rsqrt_t(r2a) : 0.f, rib = (r2b >= 1e-16f) ? rsqrt_t(r2b) : 0.f;
            SP[rp] = fma2(pk2(ria, rib), SW, SP[rp]);
          }
          if constexpr (R % 2 == 1) {
            const float x = px[R - 1] - sp.x, y = py[R - 1] - sp.y, z = pz[R - 1] - sp.z;
            s_last += rinv_cut(x * x + y * y + z * z) * sp.w;
          }
        } else {
#pragma unroll
          for (int r = 0; r < R; r++) keval<KT, T>(px[r] - sp.x, py[r] - sp.y, pz[r] - sp.z, nrm, f, acc[r], a.ku);
        }
      }
    }
    if constexpr (PACKED) {  // sum f / r, times 1/(4 pi) once
#pragma unroll
      for (int rp = 0; rp < R / 2; rp++) {
        float sa, sb;
        upk2(SP[rp], sa, sb);
        acc[2 * rp][0] = a.ku.c0 * sa;
        acc[2 * rp + 1][0] = a.ku.c0 * sb;
      }
      if constexpr (R % 2 == 1) acc[R - 1][0] = a.ku.c0 * s_last;
    }
    T* outbase = a.supcval + (size_t)g * nt * TD;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int ti = t0 + 32 * r;
      if (ti < nt)
#pragma unroll
        for (int d = 0; d < TD; d++) outbase[(size_t)ti * TD + d] = acc[r][d];
    }
  }
}

// Leaf pass, one warp per work item: a round of up to 32 targets of one leaf
// against a range of the leaf's sources (leaf_items below cuts long ranges).
// lane = (target slot, source split) with two targets a slot, G = the power of
// two >= half the round's targets (<= 16) slots and 32 / G splits, so a leaf of
// 33-64 targets splits its last round's sources over the lanes its few targets
// leave; splits are summed with warp shuffles.  Two targets, because a staged
// source costs a lane 32 (FP64) or, for a pair of them, 32 (FP32) bytes of
// register fills, at 128 bytes a clock per SM 8 clocks a warp, against 6.5 clocks
// of FP64 pipe or 4 of reciprocal roots for one target's Laplace terms.  Sources are staged 64 at a time: point
// sources from the leaf's near list (segments = source leaves, found by
// bisection of the warp's prefix sums), then the W-list upward equivalent
// surfaces and the leaf's own downward equivalent surface.  An item of a cut
// range writes partial[out][slot][d] (T, the accumulator's type), which
// k_leaf_reduce adds up in item order.  Limits on the registers trade spills for
// warps, whose number hides the staging loads.  FP32: 64 registers (32 warps an
// SM) for the scalar single layers, 80 (24 warps) for the others, which spill at
// 64; leaf pass of 262,144 Laplace points 0.261 ms with 64, 0.263 with 80 and 0.327
// with 108, of 100,003 Stokes points 0.134, 0.126 and 0.142, of as many Navier points
// 0.132, 0.125 and 0.136.  FP64: 128, and for Laplace 96 (16 and 20 warps).
template <typename T>
struct WarpSegs {
  int beg[32];
  int pre[33];
  T shx[32], shy[32], shz[32], rad[32];
  const T* unit[32];
  const T* den[32];
};

// target slots of a round with `left` targets to go, two targets each
__host__ __device__ inline int leaf_slots(int left) {
  int G = 1;
  while (2 * G < left && G < 16) G <<= 1;
  return G;
}

// CTAs per SM that the registers are limited for (comment above)
template <typename T, int KT>
constexpr int leaf_ctas() {
  if (sizeof(T) == 8) return KT == 111 ? 5 : 4;
  return KTraits<KT>::TD == 1 && !KTraits<KT>::DL ? 4 : 3;
}

template <typename T, int KT, int NWARP>
__global__ void __launch_bounds__(32 * NWARP, leaf_ctas<T, KT>())
    k_leaf_warp(P2PArgs<T> a, const LeafItem* __restrict__ items, const int* __restrict__ nidx,
                const int* __restrict__ midx, int nitem, T* partial, int rhs) {
  constexpr int SD = KTraits<KT>::SD, TD = KTraits<KT>::TD;
  constexpr bool DL = KTraits<KT>::DL;
  constexpr int MM = KTraits<KT>::MM;
  constexpr int SDM = KTraits<MM>::SD;
  __shared__ WarpSrc64<T> ws[NWARP];
  __shared__ WarpSegs<T> wg[NWARP];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WarpSrc64<T>& w = ws[warp];
  WarpSegs<T>& sgt = wg[warp];
  wait_for_previous();
  dependents_may_start();
  // packed FP32 Laplace sums (near field for KT 111, surfaces for MM 111)
  constexpr bool PAIR_NEAR = KT == 111 && sizeof(T) == 4, PAIR_SURF = MM == 111 && sizeof(T) == 4;
  const T* den = a.sden + (size_t)rhs * a.ns * SD;
  const int nsurf = a.nsurf;
  for (int wi = blockIdx.x * NWARP + warp; wi < nitem; wi += gridDim.x * NWARP) {
    const LeafItem it = items[wi];
    const int g = it.g;
    const double cx = a.center[3 * g], cy = a.center[3 * g + 1], cz = a.center[3 * g + 2];
    const T rad = (T)a.radius[g];
    const int tb0 = a.tbeg[g], nt = a.tcnt[g];
    const int64_t nb = it.nb, ne = it.nb + it.nn;
    const int64_t mb = it.mb, me = it.mb + it.nm;
    const int nsurf_segs = it.nm + it.l2t;
    int left = it.take;  // point sources of this item still to come
    {
      const int G = leaf_slots(nt - it.tb);
      const int nsplit = 32 / G, slot = lane % G, sg = lane / G;
      bool valid[2];  // targets it.tb + slot and it.tb + slot + G
      T px[2], py[2], pz[2], acc[2][TD];
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int ti = it.tb + slot + k * G;
        valid[k] = ti < nt;
        px[k] = valid[k] ? a.tx[tb0 + ti] : T(0);
        py[k] = valid[k] ? a.ty[tb0 + ti] : T(0);
        pz[k] = valid[k] ? a.tz[tb0 + ti] : T(0);
#pragma unroll
        for (int d = 0; d < TD; d++) acc[k][d] = T(0);
      }
      // point sources, up to 32 source leaves per batch
      for (int64_t c0 = nb; c0 < ne; c0 += 32) {
        const int nseg = (int)min((int64_t)32, ne - c0);
        __syncwarp();
        int cntl = 0;
        if (lane < nseg) {
          const int s = nidx[c0 + lane];
          const int skip = c0 == nb && lane == 0 ? it.skip : 0;  // the item begins inside its first leaf
          sgt.beg[lane] = a.sbeg[s] + skip;
          cntl = a.scnt[s] - skip;
          sgt.shx[lane] = (T)(a.center[3 * s] - cx);
          sgt.shy[lane] = (T)(a.center[3 * s + 1] - cy);
          sgt.shz[lane] = (T)(a.center[3 * s + 2] - cz);
        }
        // inclusive scan of the segment sizes
        int incl = cntl;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        sgt.pre[lane + 1] = incl;
        if (lane == 0) sgt.pre[0] = 0;
        const int total = min(left, __shfl_sync(0xffffffffu, incl, 31));
        left -= total;
        __syncwarp();
        for (int k0 = 0; k0 < total; k0 += 64) {
          const int cnt = min(64, total - k0);
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int jl = lane + 32 * h;
            if (jl >= cnt) {
              // an odd batch's last pair: a zero-weight partner
              if (PAIR_NEAR && jl == cnt && (cnt & 1)) stage_src(w, jl, P4<T>{T(0), T(0), T(0), T(0)}, true);
              break;
            }
            const int k = k0 + jl;
            int lo = 0, hi = nseg;  // pre[lo] <= k < pre[hi]
            while (hi - lo > 1) {
              const int mid = (lo + hi) >> 1;
              if (sgt.pre[mid] <= k)
                lo = mid;
              else
                hi = mid;
            }
            const int p = sgt.beg[lo] + (k - sgt.pre[lo]);
            T f[SD];
#pragma unroll
            for (int s = 0; s < SD; s++) f[s] = den[(size_t)p * SD + s];
            stage_src(w, jl, P4<T>{a.sx[p] + sgt.shx[lo], a.sy[p] + sgt.shy[lo], a.sz[p] + sgt.shz[lo], f[0]},
                      PAIR_NEAR);
#pragma unroll
            for (int s = 1; s < SD; s++) w.f[jl * (SD - 1) + s - 1] = f[s];
            if constexpr (DL) {
              w.n[3 * jl] = a.snx[p];
              w.n[3 * jl + 1] = a.sny[p];
              w.n[3 * jl + 2] = a.snz[p];
            }
          }
          __syncwarp();
          if (valid[0]) {
            const int rounds = sg < cnt ? (cnt - sg + nsplit - 1) / nsplit : 0;
            if constexpr (PAIR_NEAR) {  // sum f / r on source pairs, times 1/(4 pi) once
              float s1[2];
              lap_pairs(w, px, py, pz, sg, nsplit, (cnt + 1) >> 1, s1);
              acc[0][0] += a.ku.c0 * s1[0];
              acc[1][0] += a.ku.c0 * s1[1];
            } else if constexpr (KT == 111) {  // FP64: sum f / r, times 1/(4 pi) once
              lap_points<T>(w, px, py, pz, sg, nsplit, rounds, a.ku.c0, acc[0], acc[1]);
            } else {
#pragma unroll 2
              for (int r = 0; r < rounds; r++) {
                const int j = sg + r * nsplit;
                const P4<T> s = w.p[j];
                T f[SD];
                f[0] = s.w;
#pragma unroll
                for (int k = 1; k < SD; k++) f[k] = w.f[j * (SD - 1) + k - 1];
                T nrm[3];
                if constexpr (DL) {
                  nrm[0] = w.n[3 * j];
                  nrm[1] = w.n[3 * j + 1];
                  nrm[2] = w.n[3 * j + 2];
                }
#pragma unroll
                for (int k = 0; k < 2; k++) keval<KT, T>(px[k] - s.x, py[k] - s.y, pz[k] - s.z, nrm, f, acc[k], a.ku);
              }
            }
          }
          __syncwarp();
        }
      }
      // surface sources: W-list upward equivalent surfaces and the leaf's own
      // downward equivalent surface, equivalent kernel
      for (int c0 = 0; c0 < nsurf_segs; c0 += 32) {
        const int nseg = min(32, nsurf_segs - c0);
        __syncwarp();
        if (lane < nseg) {
          const int e = c0 + lane;
          if (e < (int)(me - mb)) {
            const int s = midx[mb + e];
            sgt.shx[lane] = (T)(a.center[3 * s] - cx);
            sgt.shy[lane] = (T)(a.center[3 * s + 1] - cy);
            sgt.shz[lane] = (T)(a.center[3 * s + 2] - cz);
            sgt.rad[lane] = (T)a.radius[s];
            sgt.unit[lane] = a.ue_unit;
            sgt.den[lane] = a.supeden + (size_t)s * nsurf * SDM;
          } else {
            sgt.shx[lane] = sgt.shy[lane] = sgt.shz[lane] = T(0);
            sgt.rad[lane] = rad;
            sgt.unit[lane] = a.de_unit;
            sgt.den[lane] = a.tdneden + (size_t)g * nsurf * SDM;
          }
        }
        __syncwarp();
        const int total = nseg * nsurf;
        for (int k0 = 0; k0 < total; k0 += 64) {
          const int cnt = min(64, total - k0);
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int jl = lane + 32 * h;
            if (jl >= cnt) {
              if (PAIR_SURF && jl == cnt && (cnt & 1)) stage_src(w, jl, P4<T>{T(0), T(0), T(0), T(0)}, true);
              break;
            }
            const int k = k0 + jl;
            const int e = k / nsurf, m = k - e * nsurf;
            const T* u = sgt.unit[e];
            const T* sd = sgt.den[e];
            const T r = sgt.rad[e];
            stage_src(w, jl,
                      P4<T>{u[3 * m] * r + sgt.shx[e], u[3 * m + 1] * r + sgt.shy[e], u[3 * m + 2] * r + sgt.shz[e],
                            sd[(size_t)m * SDM]},
                      PAIR_SURF);
#pragma unroll
            for (int s = 1; s < SDM; s++) w.f[jl * (SDM - 1) + s - 1] = sd[(size_t)m * SDM + s];
          }
          __syncwarp();
          if (valid[0]) {
            const int rounds = sg < cnt ? (cnt - sg + nsplit - 1) / nsplit : 0;
            if constexpr (PAIR_SURF) {
              float s1[2];
              lap_pairs(w, px, py, pz, sg, nsplit, (cnt + 1) >> 1, s1);
              acc[0][0] += a.km.c0 * s1[0];
              acc[1][0] += a.km.c0 * s1[1];
            } else if constexpr (MM == 111) {
              lap_points<T>(w, px, py, pz, sg, nsplit, rounds, a.km.c0, acc[0], acc[1]);
            } else {
#pragma unroll 2
              for (int r = 0; r < rounds; r++) {
                const int j = sg + r * nsplit;
                const P4<T> s = w.p[j];
                T f[SDM];
                f[0] = s.w;
#pragma unroll
                for (int k = 1; k < SDM; k++) f[k] = w.f[j * (SDM - 1) + k - 1];
                T nrm[3];
#pragma unroll
                for (int k = 0; k < 2; k++) keval<MM, T>(px[k] - s.x, py[k] - s.y, pz[k] - s.z, nrm, f, acc[k], a.km);
              }
            }
          }
          __syncwarp();
        }
      }
      // sum the splits (lanes slot, slot + G, ...)
#pragma unroll
      for (int k = 0; k < 2; k++) {
#pragma unroll
        for (int d = 0; d < TD; d++)
          for (int o = G; o < 32; o <<= 1) acc[k][d] += __shfl_xor_sync(0xffffffffu, acc[k][d], o);
        if (valid[k] && sg == 0) {
          T* o = it.out >= 0 ? partial + ((size_t)it.out * 32 + slot + k * G) * TD
                             : a.tval + ((size_t)rhs * a.nt + tb0 + it.tb + slot + k * G) * TD;
#pragma unroll
          for (int d = 0; d < TD; d++) o[d] = acc[k][d];
        }
      }
    }
  }
}

// tval of one round = the sum of its items' partial potentials, in item order
template <typename T, int TD>
__global__ void k_leaf_reduce(const LeafSplit* __restrict__ splits, int n, const T* partial, T* tval) {
  wait_for_previous();
  dependents_may_start();
  const int e = blockIdx.x * blockDim.x + threadIdx.x, w = e / (32 * TD), k = e % (32 * TD);
  if (w >= n) return;
  const LeafSplit sp = splits[w];
  if (k >= sp.cnt * TD) return;
  T s = T(0);
#pragma unroll 4
  for (int p = 0; p < sp.parts; p++) s += partial[((size_t)(sp.first + p) * 32) * TD + k];
  tval[(size_t)sp.tbeg * TD + k] = s;
}

// sden_sorted[r][i][s] = srcden[r][perm[i]][s]
template <typename T>
__global__ void k_scatter_den(const double* srcden, const int* perm, int ns, int sd, int nrhs, T* out) {
  wait_for_previous();
  dependents_may_start();
  size_t n = (size_t)ns * sd * nrhs;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    size_t r = e / ((size_t)ns * sd);
    size_t rem = e % ((size_t)ns * sd);
    int i = (int)(rem / sd), s = (int)(rem % sd);
    out[e] = (T)srcden[r * ns * sd + (size_t)perm[i] * sd + s];
  }
}

// trgval[r][perm[i]][t] = tval[r][i][t]
template <typename T>
__global__ void k_gather_val(const T* tval, const int* perm, int nt, int td, int nrhs, double* trgval) {
  wait_for_previous();
  dependents_may_start();
  size_t n = (size_t)nt * td * nrhs;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    size_t r = e / ((size_t)nt * td);
    size_t rem = e % ((size_t)nt * td);
    int i = (int)(rem / td), d = (int)(rem % td);
    trgval[r * nt * td + (size_t)perm[i] * td + d] = (double)tval[e];
  }
}

// trgval[r][perm[i]][t] = tval[r][i][t] + near[r][i][t]: the FP32 passes'
// potentials plus an FP64 near-field sum
__global__ void k_gather_val_sum(const float* tval, const double* near, const int* perm, int nt, int td, int nrhs,
                                 double* trgval) {
  wait_for_previous();
  dependents_may_start();
  size_t n = (size_t)nt * td * nrhs;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    size_t r = e / ((size_t)nt * td);
    size_t rem = e % ((size_t)nt * td);
    int i = (int)(rem / td), d = (int)(rem % td);
    trgval[r * nt * td + (size_t)perm[i] * td + d] = (double)tval[e] + near[e];
  }
}

template <typename T, int KT>
void launch_p2p_kt(const P2PArgs<T>& a, const P2PWork& w, int which, int rhs, cudaStream_t st) {
  switch (which) {
    case P2P_S2M:
      if (w.n) {
        // rounds per warp.  FP32: all of a leaf's (152, 296 and 488 check points at
        // np = 4, 6 and 8 are 5, 10 and 16 rounds).  FP64: 5 or 4 of them, which
        // reuse a staged source often enough (two would) at half the registers.
        // Two rounds where the leaves alone leave the SMs below 32 warps, so that
        // one warp's rounds do not set the time, and for other np.
        const int rounds = (a.nuc + 31) / 32;
        int R = 2;
        if (w.n >= B200_SMS * 32) {
          if (sizeof(T) == 8)
            R = rounds % 5 == 0 ? 5 : rounds % 4 == 0 ? 4 : 2;
          else if (rounds == 5 || rounds == 10 || rounds == 16)
            R = rounds;
        }
        const int parts = (rounds + R - 1) / R;
        const int grid = (int)std::min<int64_t>(((int64_t)w.n * parts + WP_WARPS - 1) / WP_WARPS, B200_SMS * 32);
        if (R == 2)
          launch_dependent(k_s2m_warp<T, KT, 2>, grid, 32 * WP_WARPS, 0, st, a, w.work, w.n, parts, rhs);
        else if (R == 5)
          launch_dependent(k_s2m_warp<T, KT, 5>, grid, 32 * WP_WARPS, 0, st, a, w.work, w.n, parts, rhs);
        else if constexpr (sizeof(T) == 8)
          launch_dependent(k_s2m_warp<T, KT, 4>, grid, 32 * WP_WARPS, 0, st, a, w.work, w.n, parts, rhs);
        else if (R == 10)
          launch_dependent(k_s2m_warp<T, KT, 10>, grid, 32 * WP_WARPS, 0, st, a, w.work, w.n, parts, rhs);
        else
          launch_dependent(k_s2m_warp<T, KT, 16>, grid, 32 * WP_WARPS, 0, st, a, w.work, w.n, parts, rhs);
      }
      break;
    case P2P_S2L:
      if (w.n)
        launch_dependent(k_s2l<T, KT>, dim3(w.n, (a.nsurf + 31) / 32), P2P_THREADS, 0, st, a, w.work, w.ptr, w.idx,
                         rhs);
      break;
    case P2P_LEAF:
      if (w.n) {
        constexpr int nw = sizeof(T) == 4 ? 8 : 4;  // static shared memory: 64 staged sources per warp
        const int grid = std::min((w.nitem + nw - 1) / nw, B200_SMS * 32);
        launch_dependent(k_leaf_warp<T, KT, nw>, grid, 32 * nw, 0, st, a, w.items, w.idx, w.idx2, w.nitem,
                         static_cast<T*>(w.partial), rhs);
        if (w.nsplit > 0) {
          constexpr int TD = KTraits<KT>::TD;
          launch_dependent(k_leaf_reduce<T, TD>, (w.nsplit * 32 * TD + 255) / 256, 256, 0, st, w.splits, w.nsplit,
                           static_cast<const T*>(w.partial), a.tval + (size_t)rhs * a.nt * TD);
        }
      }
      break;
  }
}

}  // namespace

namespace {
// evaluations per lane of `all` sources at a round's targets: 32 / slots lanes
// share a source's two targets, a round of one target computes its second in vain
double leaf_cost(int64_t all, int left) { return (double)all * leaf_slots(left) / 16; }

// the items of leaves w0 .. w1 - 1 of leaf_items, partial rows counted from 0
void cut_leaves(int w0, int w1, const int* work, const int* tcnt, const int* scnt, const int64_t* nptr, const int* nidx,
                const int64_t* mptr, const unsigned char* l2t, const int* tbeg, int nsurf, double limit,
                const int64_t* nsrc, std::vector<LeafItem>* items, std::vector<LeafSplit>* splits,
                int* nparts) {
  for (int w = w0; w < w1; w++) {
    const int g = work[w], nt = tcnt[g];
    const int nseg = (int)(mptr[w + 1] - mptr[w]) + l2t[w];
    const int64_t all = nsrc[w] + (int64_t)nseg * nsurf;
    for (int tb = 0; tb < nt; tb += 32) {
      const double cost = leaf_cost(all, nt - tb);
      const int parts = cost > 1.5 * limit ? (int)std::min(cost / limit + 0.5, 65536.0) : 1;
      int64_t seg = nptr[w];  // the near segment the next item begins in, `skip` sources into it
      int skip = 0, s0 = 0;   // and its first surface
      int64_t k0 = 0;
      const int first = *nparts;
      int made = 0;
      for (int p = 0; p < parts; p++) {
        const bool last = p + 1 == parts;
        const int64_t cut = last ? all : (int64_t)((double)all * (p + 1) / parts);
        const int64_t k1 = last ? nsrc[w] : std::max(k0, std::min(nsrc[w], (cut + 63) / 64 * 64));
        int s1 = last ? nseg : std::max(s0, (int)((std::max(cut, nsrc[w]) - nsrc[w]) / nsurf));
        if (k1 == k0 && s1 == s0 && !(last && made == 0)) continue;
        LeafItem it;
        it.g = g;
        it.tb = tb;
        it.nb = seg;
        it.skip = skip;
        it.take = (int)(k1 - k0);
        int64_t left = k1 - k0;
        int64_t e = seg;
        while (left > 0) {
          const int64_t c = scnt[nidx[e]] - skip;
          if (left < c) {
            skip += (int)left;
            left = 0;
            break;
          }
          left -= c;
          skip = 0;
          e++;
        }
        it.nn = (int)(e - seg) + (skip > 0 ? 1 : 0);
        if (it.take == 0) it.nn = 0;
        seg = e;
        it.mb = mptr[w] + s0;
        it.l2t = s1 == nseg && s1 > s0 ? l2t[w] : 0;
        it.nm = s1 - s0 - it.l2t;
        it.out = parts > 1 ? (*nparts)++ : -1;
        made++;
        k0 = k1;
        s0 = s1;
        items->push_back(it);
      }
      if (parts > 1) {
        if (made == 1) {  // nothing was cut after all
          items->back().out = -1;
          (*nparts)--;
        } else {
          splits->push_back(LeafSplit{tbeg[g] + tb, std::min(32, nt - tb), first, made});
        }
      }
    }
  }
}
}  // namespace

// Work items of the leaf pass.  One warp per leaf, the form before, left a
// leaf with long lists to one warp (150,001 sources on an ellipsoid, targets
// in the volume: the coarse leaves' W lists hold hundreds of surfaces, 17.9 ms
// in that warp's tail) and a small tree's leaves on a few SMs (2,000 points:
// 56 warps, 0.15 ms).  A range costs its evaluations per lane (leaf_cost; with a
// round of one target counted at half of that, 150,001 ellipsoid sources to 5,000
// volume targets took 0.167 ms instead of 0.122); it is cut above `limit` = 1/8 of
// a warp's share when every SM holds 32 warps, and not below `least` sources
// (two staged batches in FP64, four in FP32, whose pairs take a quarter of the
// time), where starting an item and adding its partial sum would cost more than
// the sources.
void leaf_items(int nwork, const int* work, const int* tcnt, const int* scnt, const int64_t* nptr, const int* nidx,
                const int64_t* mptr, const unsigned char* l2t, const int* tbeg, int nsurf, int least, int num_sms,
                std::vector<LeafItem>* items, std::vector<LeafSplit>* splits, int* nparts) {
  // the leaves in contiguous ranges, one host thread each
  const int nthr = host_parallel_threads(nwork / 2048);
  auto run = [&](auto&& body) {  // body(t, first leaf, past the last)
    host_parallel(nthr, [&](int t, int n) {
      body(t, (int)((int64_t)nwork * t / n), (int)((int64_t)nwork * (t + 1) / n));
    });
  };
  std::vector<int64_t> nsrc(nwork);
  std::vector<double> totals(nthr, 0.0);
  run([&](int t, int w0, int w1) {
    double total = 0;
    for (int w = w0; w < w1; w++) {
      int64_t s = 0;
      for (int64_t k = nptr[w]; k < nptr[w + 1]; k++) s += scnt[nidx[k]];
      nsrc[w] = s;
      const int nt = tcnt[work[w]];
      const int64_t all = s + (mptr[w + 1] - mptr[w] + l2t[w]) * nsurf;
      for (int tb = 0; tb < nt; tb += 32) total += leaf_cost(all, nt - tb);
    }
    totals[t] = total;
  });
  double total = 0;
  for (double v : totals) total += v;
  const double limit = std::max((double)least, total / ((double)num_sms * 32 * 8));
  std::vector<std::vector<LeafItem>> pitems(nthr);
  std::vector<std::vector<LeafSplit>> psplits(nthr);
  std::vector<int> pparts(nthr, 0);
  run([&](int t, int w0, int w1) {
    cut_leaves(w0, w1, work, tcnt, scnt, nptr, nidx, mptr, l2t, tbeg, nsurf, limit, nsrc.data(), &pitems[t], &psplits[t],
               &pparts[t]);
  });
  items->clear();
  splits->clear();
  *nparts = 0;
  for (int t = 0; t < nthr; t++) {
    for (LeafItem& it : pitems[t]) {
      if (it.out >= 0) it.out += *nparts;
      items->push_back(it);
    }
    for (LeafSplit& sp : psplits[t]) {
      sp.first += *nparts;
      splits->push_back(sp);
    }
    *nparts += pparts[t];
  }
}

template <typename T>
void launch_p2p(int kt, const P2PArgs<T>& a, const P2PWork& w, int which, int rhs, cudaStream_t st) {
  switch (kt) {
    case 111: launch_p2p_kt<T, 111>(a, w, which, rhs, st); break;
    case 121: launch_p2p_kt<T, 121>(a, w, which, rhs, st); break;
    case 311: launch_p2p_kt<T, 311>(a, w, which, rhs, st); break;
    case 312: launch_p2p_kt<T, 312>(a, w, which, rhs, st); break;
    case 321: launch_p2p_kt<T, 321>(a, w, which, rhs, st); break;
    case 322: launch_p2p_kt<T, 322>(a, w, which, rhs, st); break;
    case 511: launch_p2p_kt<T, 511>(a, w, which, rhs, st); break;
    case 521: launch_p2p_kt<T, 521>(a, w, which, rhs, st); break;
  }
}
template void launch_p2p<double>(int, const P2PArgs<double>&, const P2PWork&, int, int, cudaStream_t);
template void launch_p2p<float>(int, const P2PArgs<float>&, const P2PWork&, int, int, cudaStream_t);

template <typename T>
void launch_scatter_den(const double* srcden, const int* perm, int ns, int sd, int nrhs, T* out, cudaStream_t st) {
  size_t n = (size_t)ns * sd * nrhs;
  if (!n) return;
  int grid = (int)std::min<size_t>((n + 255) / 256, B200_SMS * 16);
  launch_dependent(k_scatter_den<T>, grid, 256, 0, st, srcden, perm, ns, sd, nrhs, out);
}
template void launch_scatter_den<double>(const double*, const int*, int, int, int, double*, cudaStream_t);
template void launch_scatter_den<float>(const double*, const int*, int, int, int, float*, cudaStream_t);

template <typename T>
void launch_gather_val(const T* tval, const int* perm, int nt, int td, int nrhs, double* trgval, cudaStream_t st) {
  size_t n = (size_t)nt * td * nrhs;
  if (!n) return;
  int grid = (int)std::min<size_t>((n + 255) / 256, B200_SMS * 16);
  launch_dependent(k_gather_val<T>, grid, 256, 0, st, tval, perm, nt, td, nrhs, trgval);
}
template void launch_gather_val<double>(const double*, const int*, int, int, int, double*, cudaStream_t);

void launch_gather_val_sum(const float* tval, const double* near, const int* perm, int nt, int td, int nrhs,
                           double* trgval, cudaStream_t st) {
  size_t n = (size_t)nt * td * nrhs;
  if (!n) return;
  int grid = (int)std::min<size_t>((n + 255) / 256, B200_SMS * 16);
  launch_dependent(k_gather_val_sum, grid, 256, 0, st, tval, near, perm, nt, td, nrhs, trgval);
}
template void launch_gather_val<float>(const float*, const int*, int, int, int, double*, cudaStream_t);

}  // namespace kifmm

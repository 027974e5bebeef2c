// FP64 direct sum over all sources (Dense3d::eval, fmm3d/dense3d.cpp:38-57),
// absolute coordinates (3 x n interleaved): the check of an evaluation, and
// kifmm_direct / kifmm_direct_noalloc.
//
// A check has few targets and many sources, so the sources are split: CTA
// (b, c) of 128 threads evaluates the G targets of block b on chunk c of the
// sources, 128 / G threads sharing a target inside the CTA, and writes one
// partial potential per target; k_direct_reduce adds the chunks in order.
// Bound: the FP64 pipe (13 FP64 instructions per Laplace pair, 64 lanes per
// SM and clock).  One thread per target over all sources, the form before,
// ran 262,144 sources at 1,000 targets on 8 CTAs: 25.9 ms; split, 0.25 ms.
#include <algorithm>

#include "launch.hpp"

namespace kifmm {
namespace {

constexpr int DIR_THREADS = 128, DIR_TILE = 128;

struct alignas(16) Src4 {
  double x, y, z, w;
};

// partial[c][t][d] = sum over the sources of chunk c of K(trg_t - src) den
template <int KT, int G>
__global__ void __launch_bounds__(DIR_THREADS) k_direct_partial(const double* __restrict__ spos,
                                                                const double* __restrict__ snor,
                                                                const double* __restrict__ sden, int ns, int chunk,
                                                                const double* __restrict__ tpos, int nt,
                                                                double* __restrict__ partial, KConst<double> kc) {
  constexpr int SD = KTraits<KT>::SD, TD = KTraits<KT>::TD, NSPLIT = DIR_THREADS / G;
  constexpr bool DL = KTraits<KT>::DL;
  __shared__ Src4 sp[DIR_TILE];
  __shared__ double sf[SD > 1 ? DIR_TILE * (SD - 1) : 1], sn[DL ? DIR_TILE * 3 : 1];
  __shared__ double red[NSPLIT > 1 ? DIR_THREADS * TD : 1];
  const int slot = threadIdx.x % G, sg = threadIdx.x / G;
  const int t = blockIdx.x * G + slot;
  const int64_t s0 = (int64_t)blockIdx.y * chunk;
  const int n = (int)max((int64_t)0, min((int64_t)chunk, (int64_t)ns - s0));
  double px = 0, py = 0, pz = 0;
  if (t < nt) {
    px = tpos[3 * (size_t)t];
    py = tpos[3 * (size_t)t + 1];
    pz = tpos[3 * (size_t)t + 2];
  }
  double acc[TD];
#pragma unroll
  for (int d = 0; d < TD; d++) acc[d] = 0;
  for (int c0 = 0; c0 < n; c0 += DIR_TILE) {
    const int cnt = min(DIR_TILE, n - c0);
    __syncthreads();
    if ((int)threadIdx.x < cnt) {
      const int j = threadIdx.x;
      const size_t p = (size_t)(s0 + c0 + j);
      sp[j] = Src4{spos[3 * p], spos[3 * p + 1], spos[3 * p + 2], sden[p * SD]};
#pragma unroll
      for (int s = 1; s < SD; s++) sf[j * (SD - 1) + s - 1] = sden[p * SD + s];
      if constexpr (DL) {
        sn[3 * j] = snor[3 * p];
        sn[3 * j + 1] = snor[3 * p + 1];
        sn[3 * j + 2] = snor[3 * p + 2];
      }
    }
    __syncthreads();
    if (t < nt) {
      const int rounds = sg < cnt ? (cnt - sg + NSPLIT - 1) / NSPLIT : 0;
#pragma unroll 4
      for (int r = 0; r < rounds; r++) {
        const int j = sg + r * NSPLIT;
        const Src4 s = sp[j];
        double f[SD], nrm[3];
        f[0] = s.w;
#pragma unroll
        for (int k = 1; k < SD; k++) f[k] = sf[j * (SD - 1) + k - 1];
        if constexpr (DL) {
          nrm[0] = sn[3 * j];
          nrm[1] = sn[3 * j + 1];
          nrm[2] = sn[3 * j + 2];
        }
        keval<KT, double>(px - s.x, py - s.y, pz - s.z, nrm, f, acc, kc);
      }
    }
  }
  if constexpr (NSPLIT > 1) {
#pragma unroll
    for (int d = 0; d < TD; d++) red[threadIdx.x * TD + d] = acc[d];
    __syncthreads();
    if (sg > 0 || t >= nt) return;
#pragma unroll
    for (int d = 0; d < TD; d++)
      for (int q = 1; q < NSPLIT; q++) acc[d] += red[(q * G + slot) * TD + d];
  }
  if (t < nt)
#pragma unroll
    for (int d = 0; d < TD; d++) partial[((size_t)blockIdx.y * nt + t) * TD + d] = acc[d];
}

// out[e] = sum over the chunks of partial[c][e]: 32 outputs per CTA, 8
// threads taking every eighth chunk of each
__global__ void __launch_bounds__(256) k_direct_reduce(const double* __restrict__ partial, int nchunk, size_t n,
                                                       double* __restrict__ out) {
  __shared__ double red[8][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (size_t e0 = (size_t)blockIdx.x * 32; e0 < n; e0 += (size_t)gridDim.x * 32) {
    const size_t e = e0 + tx;
    double s = 0.0;
    if (e < n)
#pragma unroll 4
      for (int c = ty; c < nchunk; c += 8) s += partial[(size_t)c * n + e];
    red[ty][tx] = s;
    __syncthreads();
    if (ty == 0 && e < n) {
      for (int q = 1; q < 8; q++) s += red[q][tx];
      out[e] = s;
    }
    __syncthreads();
  }
}

template <int KT, int G>
void launch_partial(const DirectPlan& p, const double* spos, const double* snor, const double* sden, int ns,
                    const double* tpos, int nt, double* partial, const KConst<double>& kc, cudaStream_t st) {
  k_direct_partial<KT, G><<<dim3(p.tblocks, p.nchunk), DIR_THREADS, 0, st>>>(spos, snor, sden, ns, p.chunk, tpos, nt,
                                                                             partial, kc);
}

template <int KT>
void launch_partial_g(const DirectPlan& p, const double* spos, const double* snor, const double* sden, int ns,
                      const double* tpos, int nt, double* partial, const KConst<double>& kc, cudaStream_t st) {
  switch (p.G) {
    case 8: launch_partial<KT, 8>(p, spos, snor, sden, ns, tpos, nt, partial, kc, st); break;
    case 32: launch_partial<KT, 32>(p, spos, snor, sden, ns, tpos, nt, partial, kc, st); break;
    default: launch_partial<KT, 128>(p, spos, snor, sden, ns, tpos, nt, partial, kc, st); break;
  }
}

}  // namespace

// Targets per CTA: 128 once two such blocks are full (a staged tile of 128
// sources then serves 128 targets), else 32, or 8 for the fewest, whose lanes
// would stay empty.  Chunks of sources: about 16 CTAs per SM, a chunk no
// smaller than one staged tile, all partial sums within `capacity` doubles.
DirectPlan direct_plan(int ns, int nt, int td, int num_sms, size_t capacity) {
  DirectPlan p;
  p.G = nt >= 256 ? 128 : nt > 8 ? 32 : 8;
  p.tblocks = (nt + p.G - 1) / p.G;
  const size_t per_chunk = (size_t)nt * td;
  size_t nc = std::max<size_t>(1, (size_t)16 * num_sms / std::max(1, p.tblocks));
  nc = std::min(nc, std::max<size_t>(1, ((size_t)ns + DIR_TILE - 1) / DIR_TILE));
  nc = std::min(nc, std::max<size_t>(1, capacity / std::max<size_t>(1, per_chunk)));
  nc = std::min<size_t>(nc, 65535);
  const size_t per = (((size_t)ns + nc - 1) / nc + DIR_TILE - 1) / DIR_TILE * DIR_TILE;
  p.chunk = (int)std::max<size_t>(1, std::min<size_t>(per, (size_t)ns));
  p.nchunk = (int)std::max<size_t>(1, ((size_t)ns + p.chunk - 1) / p.chunk);
  p.scratch = p.nchunk > 1 ? (size_t)p.nchunk * per_chunk : 0;
  return p;
}

void launch_direct(int kt, const DirectPlan& p, const double* spos, const double* snor, const double* sden, int ns,
                   const double* tpos, int nt, double* out, double* scratch, const double* kc3, int num_sms,
                   cudaStream_t st) {
  if (nt <= 0) return;
  const KConst<double> kc{kc3[0], kc3[1], kc3[2]};
  const bool staged = p.nchunk > 1 || p.staged;
  double* partial = staged ? scratch : out;
  int td = 1;
  switch (kt) {
    case 111: launch_partial_g<111>(p, spos, snor, sden, ns, tpos, nt, partial, kc, st); break;
    case 121: launch_partial_g<121>(p, spos, snor, sden, ns, tpos, nt, partial, kc, st); break;
    case 311: launch_partial_g<311>(p, spos, snor, sden, ns, tpos, nt, partial, kc, st); td = 3; break;
    case 312: launch_partial_g<312>(p, spos, snor, sden, ns, tpos, nt, partial, kc, st); break;
    case 321: launch_partial_g<321>(p, spos, snor, sden, ns, tpos, nt, partial, kc, st); td = 3; break;
    case 322: launch_partial_g<322>(p, spos, snor, sden, ns, tpos, nt, partial, kc, st); break;
    case 511: launch_partial_g<511>(p, spos, snor, sden, ns, tpos, nt, partial, kc, st); td = 3; break;
    case 521: launch_partial_g<521>(p, spos, snor, sden, ns, tpos, nt, partial, kc, st); td = 3; break;
    default: return;
  }
  if (staged) {
    const size_t n = (size_t)nt * td;
    const int grid = (int)std::min<size_t>((n + 31) / 32, (size_t)num_sms * 8);
    k_direct_reduce<<<std::max(1, grid), 256, 0, st>>>(partial, p.nchunk, n, out);
  }
}

}  // namespace kifmm

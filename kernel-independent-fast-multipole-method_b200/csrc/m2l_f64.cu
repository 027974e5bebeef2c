// FP64 Hadamard accumulation of the V list (cptwvv, fmm3d/matmgnt3d.cpp:343-360)
// on the FP64 matrix instructions, for equivalent kernels of 1 x 1 (Laplace),
// 4 x 3 (Stokes) and 3 x 3 (Navier) dofs and np = 4, 6, 8.
//
// Per frequency, target parent Q and colleague direction d the children-to-
// children block M[i][j] = K(2d + oct(j) - oct(i)) is, along x, a 2 x 2 Toeplitz
// matrix of 4 x 4 complex blocks: three block products instead of four,
//   y0 = A + B, y1 = A + C,  A = t0 (x0 + x1), B = (t1 - t0) x1, C = (t-1 - t0) x0
// (the two halves x0, x1 are the children with x bit 0 and 1), each of them
// 8 x 8 in real arithmetic: with 8 target parents as rows, two
// mma.m8n8k4.f64 and no padding.  Directions and source dofs accumulate in
// the same registers, and A, B, C are combined once per parent.
//
// Why matrix instructions, which run at the FP64 pipe's rate (37.0 TFLOP/s
// measured, multiply-adds 36.4): the operands.  An operator value that a
// thread multiplies into one parent costs a 16-byte register fill per 4
// multiply-adds, and the load path fills 128 bytes a clock per SM even when
// all lanes read one address: the same sums with the factorisation along all
// three axes (27 products instead of 64, 146 FP64 instructions) ran at 34 % of
// the pipe, 80 % of the load path, 23.0 ms where this form takes 13.9.  Here a fill serves 8
// parents and the pipe is the bound.
//
// A CTA keeps NF frequencies and one target dof, whose operator for all source
// dofs (39,936 bytes per frequency and dof pair) it lays out in shared memory
// in fragment order, while each warp walks groups of 16 parents (two row
// tiles) at one frequency.  Rows gather their colleague's spectra straight
// from global memory (spectra_f64_index); neighbouring parents share
// colleagues, which L1 serves.  The layout keeps frequency pairs innermost: with
// the 8 children of one frequency contiguous, one load a row, this kernel is no
// faster and the forward pass, whose nodes then write half sectors, takes 8.2 ms
// instead of 2.6 (4M points).
// A group takes every direction that one of its 16 parents has, 1.05x the work in
// a volume and 1.4-2x on a surface (had64_groups groups the parents by direction
// sets; letting each tile of 8 skip its own, 1.3-1.8x the work, is slower: one
// tile alone waits for its operator fragments and rows).
//
// Measured, against one launch of the direct parent-pair sweep (m2l.cu) per dof
// pair on the transforms of 2 np points that it then had: Laplace np = 6, 4,194,304
// points in a volume 22.5 -> 10.4 ms (13.9 on 2 np points; matrix pipe 75 % busy);
// Stokes np = 6, 262,144 points on an ellipsoid 28.4 -> 3.0 ms; Navier np = 8, 1,048,576
// points on a sphere 45.9 -> 14.5 ms; Laplace np = 4, 32,768 points on a sphere 0.64 ->
// 0.03 ms.
#include <algorithm>
#include <cmath>

#include "host_parallel.hpp"
#include "launch.hpp"

namespace kifmm {
namespace {

constexpr int H_WARPS = 16, H_THREADS = 32 * H_WARPS;
constexpr int H_ROWS = 26 * 27;            // table values per frequency and dof pair: direction, x combination, dy, dz
constexpr int H_FRAGS = 26 * 3 * 32;       // fragment entries (double2: both k steps) per frequency and dof pair
constexpr int H_TILES = 2, H_GROUP = 8 * H_TILES;

__device__ __forceinline__ void mma(double* c, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

struct TileX {
  double2 x0, x1;  // this lane's child (y, z) of its row's colleague, x bit 0 and 1
};

template <int SD, int NF>
__global__ void __launch_bounds__(H_THREADS, 1)
    k_m2l_had64(const double2* __restrict__ tables, const double2* __restrict__ spectra, size_t plane, int nfc, int ngroup,
                int per_slice, const int2* __restrict__ ghead, const int* __restrict__ gtab,
                const int* __restrict__ gdesc, const int* __restrict__ gout, double2* __restrict__ effval) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* Bs = reinterpret_cast<double2*>(smem_raw);  // [NF][SD][26][3][32]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane >> 2, c = lane & 3;
  const int f0 = blockIdx.y * NF, t = blockIdx.z;
  // fragment order: lane (k = source child, n = target child and part), k step
  // 0 = real parts of the sources, 1 = imaginary parts
  for (int e = threadIdx.x; e < NF * SD * H_FRAGS; e += H_THREADS) {
    const int ln = e & 31, n = ln >> 2, j = ln & 3, i = n >> 1;
    const int r = e >> 5, kx = r % 3, ds = r / 3;  // ds = (f, s, direction)
    const int dy = (j >> 1) - (i >> 1), dz = (j & 1) - (i & 1);
    const double2 v = __ldg(tables + ((size_t)t * nfc + f0) * (SD * H_ROWS) + ds * 27 + kx * 9 + (dy + 1) * 3 + dz + 1);
    Bs[e] = (n & 1) ? make_double2(v.y, v.x) : make_double2(v.x, -v.y);  // columns im: (Ti, Tr), re: (Tr, -Ti)
  }
  __syncthreads();
  const int fw = warp % NF, f = f0 + fw;
  const double2* Bw = Bs + (size_t)fw * (SD * H_FRAGS) + lane;
  const size_t gstride = (size_t)nfc * 8;  // complex slots of a sibling group
  const size_t lbase = (size_t)(f >> 1) * 16 + 2 * c + (f & 1);
  const int g1 = min(ngroup, (int)(blockIdx.x + 1) * per_slice);
  for (int g = blockIdx.x * per_slice + warp / NF; g < g1; g += H_WARPS / NF) {
    const int2 head = ghead[g];  // first step and number of steps (even), per source dof
    const int* tab = gtab + (size_t)head.x * H_GROUP + row;
    const int* desc = gdesc + head.x;
    double acc[H_TILES][3][2];
#pragma unroll
    for (int n = 0; n < H_TILES; n++)
#pragma unroll
      for (int k = 0; k < 3; k++) acc[n][k][0] = acc[n][k][1] = 0.0;
    // two register sets: the next step's rows are loaded while this step's are
    // multiplied, from a descriptor and colleague indices that were loaded one
    // step earlier still (past the last step they wrap to the first again)
    TileX xa[H_TILES], xb[H_TILES];
    int ea, eb;  // B fragment offset
    int i = 0, s = 0, idx[H_TILES], de;
    auto fetch = [&] {
      de = __ldg(desc + i) + s * (26 * 96);
#pragma unroll
      for (int n = 0; n < H_TILES; n++) idx[n] = __ldg(tab + i * H_GROUP + 8 * n);
    };
    auto load = [&](TileX* x, int& e) {
      e = de;
      const double2* X = spectra + (size_t)s * plane + lbase;
#pragma unroll
      for (int n = 0; n < H_TILES; n++) {
        const double2* p = X + (size_t)idx[n] * gstride;
        x[n].x0 = __ldg(p);
        x[n].x1 = __ldg(p + 8);
      }
      if (++i == head.y) {
        i = 0;
        if (++s == SD) s = 0;
      }
      fetch();
    };
    auto multiply = [&](const TileX* x, int e) {
      const double2* B = Bw + e;
      const double2 b0 = B[0], b1 = B[32], b2 = B[64];
#pragma unroll
      for (int n = 0; n < H_TILES; n++) {
        mma(acc[n][1], x[n].x1.x, b1.x);
        mma(acc[n][2], x[n].x0.x, b2.x);
        mma(acc[n][0], x[n].x0.x + x[n].x1.x, b0.x);
      }
#pragma unroll
      for (int n = 0; n < H_TILES; n++) {
        mma(acc[n][1], x[n].x1.y, b1.y);
        mma(acc[n][2], x[n].x0.y, b2.y);
        mma(acc[n][0], x[n].x0.y + x[n].x1.y, b0.y);
      }
    };
    fetch();
    load(xa, ea);
    for (int st = 0; st < head.y * SD; st += 2) {
      load(xb, eb);
      multiply(xa, ea);
      load(xa, ea);
      multiply(xb, eb);
    }
    // a lane holds the real and imaginary part of target child c of its row
#pragma unroll
    for (int n = 0; n < H_TILES; n++) {
      const int o = gout[g * H_GROUP + 8 * n + row];  // the target's sibling group
      if (o < 0) continue;
      double2* y = effval + (size_t)t * plane + (size_t)o * gstride + lbase;
      y[0] = make_double2(acc[n][0][0] + acc[n][1][0], acc[n][0][1] + acc[n][1][1]);
      y[8] = make_double2(acc[n][0][0] + acc[n][2][0], acc[n][0][1] + acc[n][2][1]);
    }
  }
}

// tables[t][f][s][direction][k = x combination, dy + 1, dz + 1] from khat
// [343][td][sd][nf]: K(2d + (0, dy, dz)) for A, and its differences from
// K(2d + (1, dy, dz)) for B and K(2d + (-1, dy, dz)) for C
__global__ void k_had64_tables(const double2* __restrict__ khat, int nf, int sd, int td, double2* __restrict__ out) {
  const size_t n = (size_t)td * sd * nf * H_ROWS;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
    const int f = (int)(e % nf);  // fastest, so that the reads of khat are contiguous
    size_t r = e / nf;
    const int row = (int)(r % H_ROWS);
    r /= H_ROWS;
    const int s = (int)(r % sd), t = (int)(r / sd);
    const int dir = row / 27, k = row % 27, dd = dir < 13 ? dir : dir + 1;
    const int kx = k / 9;
    const int ox = 2 * (dd / 9 - 1) + 3, oy = 2 * ((dd / 3) % 3 - 1) + (k / 3) % 3 - 1 + 3,
              oz = 2 * (dd % 3 - 1) + k % 3 - 1 + 3;
    auto at = [&](int x) { return khat[(((size_t)(x * 49 + oy * 7 + oz) * td + t) * sd + s) * nf + f]; };
    double2 v = at(ox);
    if (kx > 0) {
      const double2 u = at(kx == 1 ? ox + 1 : ox - 1);
      v = make_double2(u.x - v.x, u.y - v.y);
    }
    out[(((size_t)t * nf + f) * sd + s) * H_ROWS + row] = v;
  }
}

template <int SD, int NF>
void launch_sd(const double* tables, const double* spectra, size_t plane, int nfc, int td, int ngroup,
               const Had64Groups& g, double* effval, int num_sms, cudaStream_t st) {
  // slices of the groups: the count whose CTAs (one per SM) fill their last
  // wave best, a CTA's start (its operator fragments) counted as one group a warp
  constexpr int LANES = H_WARPS / NF;  // groups in flight per CTA
  int best = 1;
  double cost = 1e300;
  for (int ns = 1; ns <= std::max(1, std::min(64, (ngroup + LANES - 1) / LANES)); ns++) {
    const int per = (ngroup + ns - 1) / ns;
    const double waves = std::ceil((double)ns * (nfc / NF) * td / num_sms);
    const double c = waves * (1.0 + (per + LANES - 1) / LANES);
    if (c < cost) {
      cost = c;
      best = ns;
    }
  }
  const int per = (ngroup + best - 1) / best;
  const size_t smem = (size_t)NF * SD * H_FRAGS * sizeof(double2);
  auto kern = k_m2l_had64<SD, NF>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  // (not a dependent launch: its read-only loads of the spectra may not be moved
  // above a wait in the kernel, and as plain loads they cost 7 % of an eval)
  kern<<<dim3((ngroup + per - 1) / per, nfc / NF, td), H_THREADS, smem, st>>>(
      reinterpret_cast<const double2*>(tables), reinterpret_cast<const double2*>(spectra), plane, nfc, ngroup, per,
      reinterpret_cast<const int2*>(g.head), g.tab, g.desc, g.out, reinterpret_cast<double2*>(effval));
}

}  // namespace

size_t had64_table_doubles(int nf, int sd, int td) { return (size_t)td * sd * nf * H_ROWS * 2; }

void launch_had64_tables(const double* khat, int nf, int sd, int td, double* tables, int num_sms, cudaStream_t st) {
  k_had64_tables<<<num_sms * 16, 256, 0, st>>>(reinterpret_cast<const double2*>(khat), nf, sd, td,
                                               reinterpret_cast<double2*>(tables));
}

// Groups of 16 target parents, two row tiles of 8.  A group takes every
// direction that one of its parents has, so inside windows of 4096 parents
// (Morton order, whose colleagues stay near) groups are filled greedily: a
// parent and, fifteen times, the one that adds the fewest directions (of those,
// the one that shares the most).  On a sphere of 1,048,576 points a group then
// takes 1.45 directions per direction of a parent, in Morton order 2.03.
void had64_groups(int nq, int zero_node, const int* qchd, const int* coll, Had64HostGroups* o) {
  constexpr int WINDOW = 4096;
  std::vector<unsigned> dirs(nq, 0u);
  std::vector<int> order(nq);
  auto window = [&](int b) {
    std::vector<int> left;
    int n = b;
    for (int w = b; w < std::min(nq, b + WINDOW); w++) {
      left.push_back(w);
      for (int d = 0; d < 26; d++)
        if (coll[(size_t)w * 26 + d] != zero_node) dirs[w] |= 1u << d;
    }
    while (!left.empty()) {
      // a group begins with the next parent of the Morton order
      unsigned m = dirs[left[0]];
      order[n++] = left[0];
      left.erase(left.begin());
      for (int k = 1; k < H_GROUP && !left.empty(); k++) {
        int best = 0, cost = 1 << 30;
        for (int e = 0; e < (int)left.size() && cost > -__builtin_popcount(m); e++) {
          const unsigned v = dirs[left[e]];
          const int c = 32 * __builtin_popcount(v & ~m) - __builtin_popcount(v & m);
          if (c < cost) {
            cost = c;
            best = e;
          }
        }
        m |= dirs[left[best]];
        order[n++] = left[best];
        left.erase(left.begin() + best);
      }
    }
  };
  const int windows = (nq + WINDOW - 1) / WINDOW;
  host_parallel(host_parallel_threads(windows), [&](int t, int n) {
    for (int k = t; k < windows; k += n) window(k * WINDOW);
  });
  const int ng = (nq + H_GROUP - 1) / H_GROUP, zero = (zero_node + 7) >> 3;
  o->head.clear();
  o->tab.clear();
  o->desc.clear();
  o->out.assign((size_t)ng * H_GROUP, -1);
  for (int g = 0; g < ng; g++) {
    unsigned m = 0;
    for (int r = 0; r < H_GROUP && g * H_GROUP + r < nq; r++) {
      const int w = order[g * H_GROUP + r];
      m |= dirs[w];
      o->out[g * H_GROUP + r] = (qchd[w] + 7) >> 3;
    }
    o->head.push_back((int)o->desc.size());
    int n = 0;
    for (int d = 0; d < 26; d++) {
      if (!((m >> d) & 1)) continue;
      o->desc.push_back(d * 96);
      for (int r = 0; r < H_GROUP; r++) {
        const int e = g * H_GROUP + r;
        o->tab.push_back(e < nq ? (coll[(size_t)order[e] * 26 + d] + 7) >> 3 : zero);
      }
      n++;
    }
    while (n == 0 || (n & 1)) {  // an even number of steps: one more of zeros
      o->desc.push_back(0);
      o->tab.insert(o->tab.end(), H_GROUP, zero);
      n++;
    }
    o->head.push_back(n);
  }
}

void launch_m2l_hadamard64(int nf, int sd, int td, const double* tables, const double* spectra, size_t plane, int nq,
                           const Had64Groups& g, double* effval, int num_sms, cudaStream_t st) {
  if (nq <= 0) return;
  const int ng = (nq + H_GROUP - 1) / H_GROUP;
  if (sd == 1)
    launch_sd<1, 2>(tables, spectra, plane, nf, td, ng, g, effval, num_sms, st);
  else if (sd == 3)
    launch_sd<3, 1>(tables, spectra, plane, nf, td, ng, g, effval, num_sms, st);
  else if (sd == 4)
    launch_sd<4, 1>(tables, spectra, plane, nf, td, ng, g, effval, num_sms, st);
}

}  // namespace kifmm

// Host-callable launchers of the device passes (one stream argument each;
// no synchronisation inside).  Argument structs hold device pointers only.
#pragma once

#include <cuda_runtime.h>
#include <complex>

#include <vector>
#include <stdint.h>

#include "kernels_common.cuh"

namespace kifmm {

// Dependent launches.  An evaluation is a chain of 12 to 40 kernels on one
// stream; a kernel launched by launch_dependent may start (its CTAs resident, its
// constant tables loaded) once every CTA of the kernel before it has
// called dependents_may_start(), and must call wait_for_previous() before it
// touches anything an earlier kernel of the stream writes or reads: the call
// returns when the kernel before has completed and its writes are visible.
// Every kernel of the chain waits, so completion is transitive.  What another
// kernel of the chain writes or reads is accessed through pointers without
// __restrict__ (and without __ldg): the compiler may take such memory for
// untouched by the wait and move accesses above it.  Set-up data may be qualified.
// A grid between one CTA per SM and many waves is launched normally: started early, its CTAs pair up on
// the SMs that the kernel before frees first (FP64 contractions of Stokes np=6:
// upward 1.29 -> 1.61 ms before the rule).  Measured on whole calls: Laplace np=4
// FP64 2,000 points 126 -> 107 us, 32,768 points 308 -> 280 us, np=6 mixed 262,144
// points 1174 -> 1110 us.
//
// Limits of dynamic shared memory.  cudaFuncAttributeMaxDynamicSharedMemorySize
// belongs to the kernel, not to a launch, and handles may be evaluated by several
// threads: a kernel whose launches differ in size sets it to its largest size
// every time, so that no thread lowers it between another's setting and launch.
constexpr int B200_SMS = 148;
#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dependents_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
inline void launch_dependent(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  const long long ctas = (long long)grid.x * grid.y * grid.z;
  cfg.numAttrs = ctas <= B200_SMS || ctas >= B200_SMS * 16 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}
#endif

// Device view of the tree, points and per-node surface data of one engine.
template <typename T>
struct P2PArgs {
  int nnodes = 0, ns = 0, nt = 0, nsurf = 0, nuc = 0;
  const int *sbeg = nullptr, *scnt = nullptr, *tbeg = nullptr, *tcnt = nullptr;
  const double *center = nullptr, *radius = nullptr;
  // sorted points, coordinates relative to their leaf centre
  const T *sx = nullptr, *sy = nullptr, *sz = nullptr, *snx = nullptr, *sny = nullptr, *snz = nullptr;
  const T* sden = nullptr;  // [rhs][ns][sd]
  const T *tx = nullptr, *ty = nullptr, *tz = nullptr;
  T* tval = nullptr;  // [rhs][nt][td]
  // unit surface grids (3 per point): UE radius 1, UC radius 3, DE radius 3, DC radius 1
  const T *ue_unit = nullptr, *uc_unit = nullptr, *de_unit = nullptr, *dc_unit = nullptr;
  // per-node surface data [node][point][dof] (one density vector at a time)
  const T* supeden = nullptr;
  const T* tdneden = nullptr;
  T* supcval = nullptr;
  T* tdncval = nullptr;
  KConst<T> ku{}, km{};  // user and equivalent kernel constants
};

enum { P2P_S2M = 0, P2P_S2L = 1, P2P_LEAF = 2 };

// One warp's work in the leaf pass: targets [tb, tb + 32) of leaf g against
// point sources (near-list segments nb .. nb + nn, from `skip` sources into the
// first, `take` in all), W-list surfaces mb .. mb + nm and, if l2t, the leaf's own
// downward equivalent surface; the sum goes to the leaf's potentials (out < 0)
// or to the partial sums' row `out`.
struct LeafItem {
  int64_t nb = 0, mb = 0;
  int g = 0, tb = 0, nn = 0, skip = 0, take = 0, nm = 0, l2t = 0, out = -1;
};
// A round of targets whose sources several items share: targets [tbeg, tbeg +
// cnt) = the sum of the partial rows first .. first + parts.
struct LeafSplit {
  int tbeg, cnt, first, parts;
};
// host side: the items of the leaves `work` (source counts scnt, near lists
// nptr/nidx, W-list surface counts from mptr, l2t flags per leaf), the rounds
// that were cut and their number of partial rows
void leaf_items(int nwork, const int* work, const int* tcnt, const int* scnt, const int64_t* nptr, const int* nidx,
                const int64_t* mptr, const unsigned char* l2t, const int* tbeg, int nsurf, int least, int num_sms,
                std::vector<LeafItem>* items, std::vector<LeafSplit>* splits, int* nparts);

struct P2PWork {
  const int* work = nullptr;  // node ids, one CTA each (S2M: one warp)
  int n = 0;
  const int64_t* ptr = nullptr;  // S2L: CSR over work items, X leaves
  const int* idx = nullptr;      // S2L: X leaves; LEAF: point-source leaves
  const int* idx2 = nullptr;     // LEAF: M2T source nodes
  // LEAF: the items, the cut rounds and their partial sums [row][32][td]
  const LeafItem* items = nullptr;
  int nitem = 0;
  const LeafSplit* splits = nullptr;
  int nsplit = 0;
  void* partial = nullptr;
};

template <typename T>
void launch_p2p(int kt, const P2PArgs<T>& a, const P2PWork& w, int which, int rhs, cudaStream_t st);

// Direct sum (direct.cu): the split of the sources into chunks, whose partial
// potentials take `scratch` doubles (0: one chunk, written straight to out).
// staged: one chunk takes nt * td doubles of scratch too, so that out is written
// only once every input has been read and may be one of the inputs.
struct DirectPlan {
  int G = 128, tblocks = 0, nchunk = 1, chunk = 1;
  size_t scratch = 0;
  bool staged = false;
};
DirectPlan direct_plan(int ns, int nt, int td, int num_sms, size_t capacity);
// snor is read for double-layer kernels only
void launch_direct(int kt, const DirectPlan& p, const double* spos, const double* snor, const double* sden, int ns,
                   const double* tpos, int nt, double* out, double* scratch, const double* kc3, int num_sms,
                   cudaStream_t st);

template <typename T>
void launch_scatter_den(const double* srcden, const int* perm, int ns, int sd, int nrhs, T* out, cudaStream_t st);
template <typename T>
void launch_gather_val(const T* tval, const int* perm, int nt, int td, int nrhs, double* trgval, cudaStream_t st);
// the same gather of tval + near (an FP64 near-field sum beside FP32 passes)
void launch_gather_val_sum(const float* tval, const double* near, const int* perm, int nt, int td, int nrhs,
                           double* trgval, cudaStream_t st);

// Batched node GEMM: for j < ncol,
//   C[cidx[j]*ldc + r] (=|+=) rs(j, r) * sum_k A[r*K + k] * B[bidx[j]*ldb + k]
// A is M x K row-major.  rs(j, r) = 2^(-(col_lvl[j] + lvl_base) * deg[r % sd])
// when col_lvl is set (homogeneous level scaling, one launch covering nodes of
// every level), else 1.
struct GemmScale {
  int sd = 1;
  int deg[4] = {0, 0, 0, 0};
  const int* col_lvl = nullptr;
  int lvl_base = 0;
};

// FP32 (gemm.cu); ws (FP64, ws_len doubles) lets a launch with few columns split
// K over several CTAs; pass nullptr to disable.  Returns the number of launches.
int launch_node_gemm(int M, int K, const float* A, const float* B, int64_t ldb, const int* bidx, float* C, int64_t ldc,
                     const int* cidx, int ncol, bool accumulate, const GemmScale& sc, double* ws, size_t ws_len,
                     int num_sms, cudaStream_t st);
// FP64 on the matrix instructions (gemm_f64.cu), one launch.  M, K, ldb and ldc
// even (every surface has an even number of points, ranks are padded to
// multiples of 8), A, B and C 16-byte aligned.
int launch_node_gemm64(int M, int K, const double* A, const double* B, int64_t ldb, const int* bidx, double* C,
                       int64_t ldc, const int* cidx, int ncol, bool accumulate, const GemmScale& sc, int num_sms,
                       cudaStream_t st);

// The same product on the tensor cores for FP32 data, both operands split into
// a TF32 head and a TF32 tail and three MMAs per product (head*head + head*tail +
// tail*head) accumulating in FP32: about 2^-21 relative, the FP32 rounding
// class.  The operator is split on the host into shared-memory images, one per
// (N tile, 32-wide K chunk): head then tail, each 160 rows x 32 columns in the
// no-swizzle K-major core-matrix layout (zero padded), so that one bulk copy moves
// a chunk.  Requires M, K, ldb and ldc multiples of 4 and 16-byte aligned B and C.
// Launches with at least as many tiles of 128 nodes as SMs run on tcgen05
// (gemm_tc.cu, kind::tf32; a bounded wait that times out sets bit 1 of *status), the
// others on mma.sync with K split over clusters (gemm_tf32.cu).  One launch.
struct TcOperator {
  const float* img = nullptr;  // [ntiles][Kp/32][2][160 x 32]
  int M = 0, K = 0, Np = 0, Kp = 0;
  int ntile = 0, ntiles = 0;  // rows per N tile (multiple of 16, <= 160), number of N tiles
};
int launch_node_gemm_tc(const TcOperator& A, const float* B, int64_t ldb, const int* bidx, float* C, int64_t ldc,
                        const int* cidx, int ncol, bool accumulate, const GemmScale& sc, int num_sms, int* status,
                        cudaStream_t st);
int launch_node_gemm_tf32(const TcOperator& A, const float* B, int64_t ldb, const int* bidx, float* C, int64_t ldc,
                          const int* cidx, int ncol, bool accumulate, const GemmScale& sc, int num_sms,
                          cudaStream_t st);
// host side: the images of a row-major M x K operator (fills A's sizes; img
// is left to the caller to upload)
void tc_operator_images(int M, int K, const double* A, std::vector<float>* img, TcOperator* desc);

// FFT-based M2L (MatMgnt3d::plnden2effden / UE2DC_dgemv / effval2plnval,
// fmm3d/matmgnt3d.cpp:223-361).
struct M2LGeom {
  int np = 0, n = 0, nh = 0, nfreq = 0, nsurf = 0;
  int nfc = 0;                // stored (Hermitian-canonical) frequencies per spectrum
  const int* fc2f = nullptr;  // device: compact -> full frequency index
  const int* ff2c = nullptr;  // device: full -> compact c, or -c-1 for conj(compact c)
  const int* surf_ijk = nullptr;  // device, 3 per surface point
  int sd = 1, td = 1;
  int deg[4] = {0, 0, 0, 0};
  int rootlvl = 0;
  // 2: the sibling-group-major layout holding FP16 pairs (below)
  // 0: spectra[node][s][f]; 1: sibling-group major, one plane per dof,
  // spectra[s][(node + 7) / 8][f / 4][(node + 7) % 8][f % 4] -- every sibling
  // group's spectra one block, and in it the 8 children's values of 4
  // frequencies contiguous (first children are 1 mod 8); in FP64 those of 2
  // (spectra_f64_index)
  int sg = 0;
  // sg == 2: each complex value x is stored as the FP16 pairs
  // {hi(re), hi(im)}, {lo(re), lo(im)} of x * 2^(14 - e), where 2^e >= the
  // FP32 value *bound (k_spectra_bound) -- the operands of the 16-bit
  // tensor-core Hadamard, in the 8 bytes (spectra_sg_index) the FP32 value
  // would take
  const unsigned* bound = nullptr;
  // accumulated spectra in the sibling-group-major layout of
  // sg 1 or 2 instead of [node][td][nfc] (written so by the FP16
  // tensor-core and the FP64 Hadamard)
  int effval_sg = 0;
  // complex slots per dof plane of the sibling-group-major spectra (dof s at
  // s * plane + spectra_sg_index)
  size_t plane = 0;
};
// complex index of (node, compact frequency c) in the sibling-group-major
// layout of nfc frequencies (a multiple of 4)
__host__ __device__ inline size_t spectra_sg_index(int nfc, int node, int c) {
  return (((size_t)((node + 7) >> 3) * (nfc >> 2) + (c >> 2)) * 8 + ((node + 7) & 7)) * 4 + (c & 3);
}
// complex index in the FP64 form's layout: [sibling group][f / 2][8 children][f % 2]
__host__ __device__ inline size_t spectra_f64_index(int nfc, int node, int c) {
  return (((size_t)((node + 7) >> 3) * (nfc >> 1) + (c >> 1)) * 8 + ((node + 7) & 7)) * 2 + (c & 1);
}

// spectra[node][s][f] (complex, interleaved re/im) of 2^(l*deg) * supeden[node]
template <typename T>
void launch_m2l_forward(const M2LGeom& g, const T* supeden, const int* nodes, int nnodes_work, const int* depth,
                        T* spectra, cudaStream_t st);
// effval[w][t][f] = sum_{s in V(work[w])} Khat[offset] * spectra[s]
template <typename T>
void launch_m2l_hadamard(const M2LGeom& g, const T* khat, const T* spectra, const int* work, int nwork,
                         const int64_t* vptr, const int* vidx, const int* path, T* effval, cudaStream_t st);
// Parent-pair form: effval[child of Q] for the nq target parents Q (first
// child qchd[q], colleague first children coll[q][26], the all-zero block
// zero_node when absent, V-list children mask[q]).  ktiles: operator spectra
// as [td][sd][ceil(nf/32)][343][32] complex, zero-padded; one pass per
// (target dof, source dof).  A mbarrier wait that times out sets bit 0 of
// *status.  Requires m2l_sweep_supported(nf, sd, td) (np = 4, 6, 8; dofs
// 1->1, 4->3, 3->3).
bool m2l_sweep_supported(int nf, int sd, int td);
template <typename T>
void launch_m2l_hadamard_sweep(int nf, int sd, int td, const T* ktiles, const T* spectra, int nq, const int* qchd,
                               const int* coll, const unsigned char* mask, T* effval, int zero_node, int* status,
                               int num_sms, cudaStream_t st);
// The same product with the 2 x 2 x 2 block-Toeplitz factorisation of each
// colleague block (27 instead of 64 complex products per direction), FP32.
// ttiles: [td][sd][ceil(nf/16)][26 directions][14][16][2] complex: for direction d
// and frequency lane l, the 27 transformed values k (padded to 28) stored as
// pairs (k, k+1) at [d][k/2][l][k%2].
void launch_m2l_hadamard_tz(int nf, int sd, int td, const float* ttiles, const float* spectra, int nq, const int* qchd,
                            const int* coll, const unsigned char* mask, float* effval, int zero_node, int* status,
                            int num_sms, cudaStream_t st);
// The FP64 form (m2l_f64.cu): spectra and accumulated spectra in the
// layout of spectra_f64_index, one plane per dof.  Tables [td][nf][sd][26][27] complex, had64_table_doubles doubles, made on
// the device from the operator spectra khat [343][td][sd][nf].  Parents in groups
// of 16 rows, a step per direction that one of them has: head [group] {first
// step, number of steps}, tab [step][16] the colleague's sibling group (the
// all-zero group for an absent one or a padding row), desc [step] the
// direction's operator fragments, out [group][16] the target sibling group (-1:
// padding).
struct Had64Groups {
  const int *head = nullptr, *tab = nullptr, *desc = nullptr, *out = nullptr;
};
struct Had64HostGroups {
  std::vector<int> head, tab, desc, out;
};
void had64_groups(int nq, int zero_node, const int* qchd, const int* coll, Had64HostGroups* o);
size_t had64_table_doubles(int nf, int sd, int td);
void launch_had64_tables(const double* khat, int nf, int sd, int td, double* tables, int num_sms, cudaStream_t st);
void launch_m2l_hadamard64(int nf, int sd, int td, const double* tables, const double* spectra, size_t plane, int nq,
                           const Had64Groups& g, double* effval, int num_sms, cudaStream_t st);
// The same product for single-dof kernels in FP32 on the tensor cores
// (m2l_tc.cu): tiles of 128 target parents, per frequency a split-TF32 MMA
// with the gathered colleague spectra in TMEM; spectra in the
// sibling-group-major layout.  img: per (chunk of 4
// frequencies, direction) the head and tail images of the 16 x 16 real
// blocks (m2l_tc_images); tile_dirs[t]: the directions present among tile
// t's parents (bit d; never 0).  A wait that times out sets bit 2 of *status.
bool m2l_tc_supported(int nf, int sd, int td);
void m2l_tc_images(int nf, const std::complex<double>* m2l, std::vector<float>* img);
void launch_m2l_hadamard_tc(int nf, const float* img, const float* spectra, int nq, const int* qchd,
                            const int* coll, const unsigned char* mask, const unsigned* tile_dirs, float* effval,
                            int zero_node, int* status, int num_sms, cudaStream_t st);
// The same product on the tensor cores with FP16-pair operands (kind::f16,
// m2l_tc16.cu): spectra written by the forward pass in the sg == 2 layout
// (scaled by the data bound *bound), img per (chunk of 4 frequencies,
// direction) the hi and lo FP16 images of the 16 x 16 real blocks, scaled by
// 1 / inv_sb[chunk] (m2l_tc16_images).  groups: producer warp groups = TMEM A
// stages (2 or 3 groups: 4 or 6 stages).  wait_limit bounds every pipeline
// wait (polls); a time-out sets bit 3 of *status.
// Equivalent kernels with sd x td dofs (1 x 1, Stokes 4 x 3, Navier 3 x 3):
// the images are [chunk][direction][td][sd]; the source spectra and the
// accumulated spectra hold one sibling-group-major plane of `plane` complex
// slots per dof, and a work item is (chunk, target dof, tile) whose steps
// are (direction, source dof).
bool m2l_tc16_supported(int nf, int sd, int td);
void m2l_tc16_images(int nf, int sd, int td, const std::complex<double>* m2l, std::vector<unsigned short>* img,
                     std::vector<float>* inv_sb);
// *bound = max over nodes and source dofs s of 2^((depth + rootlvl) deg[s]) *
// sum_k |supeden[node][k][s]| (FP32 bits)
void launch_spectra_bound(const float* supeden, const int* nodes, int n, const int* depth, int rootlvl,
                          const int* deg, int sd, int nsurf, unsigned* bound, int num_sms, cudaStream_t st);
void launch_m2l_hadamard_tc16(int groups, int nf, int sd, int td, const unsigned short* img,
                              const unsigned* spectra, int nq, const int* qchd, const int* ctab,
                              const unsigned* tile_dirs, float* effval, size_t plane, const unsigned* bound,
                              const float* inv_sb, int wait_limit, int* status, int num_sms, cudaStream_t st);
// colleague tables of the FP16 form: per tile of 128 target parents and
// direction, the sibling group ((first child + 7) / 8) of each row's colleague
// (the all-zero group for an absent one or a padding row), [tile][26][128]
void m2l_tc16_tables(int nq, int zero_node, const int* coll, std::vector<int>* ctab);
// tdncval[node] += extract(inverse(effval[node]))
template <typename T>
void launch_m2l_inverse(const M2LGeom& g, const T* effval, const int* work, int nwork, T* tdncval,
                        cudaStream_t st);

}  // namespace kifmm

// kifmm_direct_noalloc: the FP64 direct sum (the engine's Dense3d path)
// for callers that must not allocate device memory.
//
// Who needs it: a process whose device memory is owned by someone else --
// a serving runtime or framework that reserved the GPU's memory up front
// through its own caching allocator, or a plug-in host that forbids device
// allocations after start-up -- cannot call cudaMalloc between its own
// steps: the call fails once the budget is taken, bypasses the owner's
// accounting, and synchronises the device in the middle of a stream of
// work.  Such a caller allocates its inputs and outputs itself and needs
// an entry point that allocates nothing else.
//
// How: the sources are split into chunks evaluated by different CTAs (so a
// small target set still fills the GPU, direct.cu); each chunk's partial potentials go
// to a fixed scratch array in device global memory, declared below at file
// scope, and a second kernel adds the chunks up into the caller's output, which
// may therefore be one of the inputs.
// The scratch holds KIFMM_NOALLOC_SCRATCH_DOUBLES doubles (8 MiB) on every
// GPU that loads this library, for the life of the process.  A call needs
// nchunk * nt * tdof of them; nt * tdof above the capacity is rejected with
// KIFMM_ERR_CAPACITY before any launch.  Every slot a call reads was written
// earlier in the same call, so nothing needs clearing between calls; the
// array keeps the last call's partial sums.  All calls share the one array:
// two calls whose kernels overlap on the GPU (different streams, or
// different host threads) race on it and must be serialised by the caller.
//
// The array's device address is looked up with cudaGetSymbolAddress on
// every call, with the caller's device current (host code cannot use the
// symbol itself: on the host it names a stand-in, not device memory); the
// lookup allocates nothing and stays right after a cudaDeviceReset, which
// reloads the module and may move the array.  The first call on a device
// loads the module there and should come before any stream capture.
#include "../../include/kifmm.h"
#include "launch.hpp"

namespace kifmm {
namespace {

static __device__ __align__(256) double g_noalloc_scratch[KIFMM_NOALLOC_SCRATCH_DOUBLES];

}  // namespace
}  // namespace kifmm

extern "C" kifmm_status kifmm_direct_noalloc(int kt, int ncoef, const double* coefs, int ns, const double* d_srcpos,
                                             const double* d_srcnor, const double* d_srcden, int nt,
                                             const double* d_trgpos, double* d_trgval, void* stream) {
  using namespace kifmm;
  int td = 0;
  switch (kt) {
    case 111: case 121: case 312: case 322: td = 1; break;
    case 311: case 321: case 511: case 521: td = 3; break;
    default: return KIFMM_ERR_KERNEL;
  }
  int need = (kt == 511 || kt == 521) ? 2 : (kt == 111 || kt == 121) ? 0 : 1;
  if (ncoef < need || (ncoef > 0 && !coefs)) return KIFMM_ERR_KERNEL;
  if (ns < 0 || nt < 0) return KIFMM_ERR_ARG;
  if (nt == 0) return KIFMM_OK;
  if (!d_trgpos || !d_trgval || (ns > 0 && (!d_srcpos || !d_srcnor || !d_srcden))) return KIFMM_ERR_ARG;
  const size_t per_chunk = (size_t)nt * td;
  if (per_chunk > (size_t)KIFMM_NOALLOC_SCRATCH_DOUBLES) return KIFMM_ERR_CAPACITY;
  // an error left by the caller's earlier work is reported as such (and
  // left pending), not taken for a failure of this call's launches
  if (cudaPeekAtLastError() != cudaSuccess) return KIFMM_ERR_CUDA;
  int dev = 0, num_sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return KIFMM_ERR_NO_DEVICE;
  }
  // the scratch array's address on the current device (every call)
  double* scratch = nullptr;
  {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
      cudaGetLastError();
      return KIFMM_ERR_CUDA;
    }
    scratch = (double*)p;
  }
  cudaStream_t st = (cudaStream_t)stream;
  double kcd[3], cf[2] = {1.0, 0.25};
  for (int i = 0; i < ncoef && i < 2; i++) cf[i] = coefs[i];
  kernel_constants(kt, cf, kcd);
  DirectPlan plan = direct_plan(ns, nt, td, num_sms, (size_t)KIFMM_NOALLOC_SCRATCH_DOUBLES);
  plan.staged = true;  // the caller's output may be one of its inputs
  launch_direct(kt, plan, d_srcpos, d_srcnor, d_srcden, ns, d_trgpos, nt, d_trgval, scratch, kcd, num_sms, st);
  if (cudaGetLastError() != cudaSuccess) return KIFMM_ERR_CUDA;
  return KIFMM_OK;
}

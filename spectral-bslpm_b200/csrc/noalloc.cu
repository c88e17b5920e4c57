// Biot-Savart direct sum for callers that cannot allocate device memory.
//
// Some callers cannot let a library allocate: a host model that fixes its
// whole device footprint when it starts, or one that owns all device memory
// through its own allocator, must not see cudaMalloc / cudaMallocAsync /
// cudaFree calls appear inside the time loop.  The direct-sum kernels add
// their partial sums within a cluster's shared memory, so neither direct-sum
// entry point needs device scratch for them; this one keeps its own limits (its
// target count, and fewer source groups in mixed precision for large ones),
// which its callers' results and error handling depend on.  Results that
// overlay an input pass through a fixed array of this module (16 MiB, on the
// GPU once this file's code is loaded there); such calls share it.
#include <cuda_runtime.h>

#include <string>

#include "../../include/sbslpm.h"
#include "bve_kernels.cuh"
#include "internal.hpp"

namespace sbslpm {
namespace {
constexpr long kPartialDoubles = 1L << 21;  // 3 x targets x groups never exceeds this: 699,050 targets at most
__device__ __align__(256) double g_apart[kPartialDoubles];
}
}  // namespace sbslpm

using namespace sbslpm;

extern "C" sbslpm_status sbslpm_direct_sum_bve_noalloc(long nt, const double* tx, const double* ty, const double* tz,
                                                       long ns, const double* sx, const double* sy, const double* sz,
                                                       const double* s, double eps, int precision, double* ux,
                                                       double* uy, double* uz, void* stream) {
  if (nt < 0 || ns < 0) return set_last_error("sbslpm_direct_sum_bve_noalloc: negative size"), SBSLPM_ERR_ARG;
  if (precision != SBSLPM_FP64 && precision != SBSLPM_MIXED)
    return set_last_error("sbslpm_direct_sum_bve_noalloc: unknown precision"), SBSLPM_ERR_ARG;
  if ((nt > 0 && (!tx || !ty || !tz || !ux || !uy || !uz)) || (ns > 0 && (!sx || !sy || !sz || !s)))
    return set_last_error("sbslpm_direct_sum_bve_noalloc: null array"), SBSLPM_ERR_ARG;
  // a host array handed to the kernels would fault the caller's context
  if (any_on_host({tx, ty, tz, sx, sy, sz, s, ux, uy, uz}))
    return set_last_error("sbslpm_direct_sum_bve_noalloc: an array is host memory (device pointers expected)"),
           SBSLPM_ERR_ARG;
  if (3 * nt > kPartialDoubles) {
    set_last_error("sbslpm_direct_sum_bve_noalloc: " + std::to_string(nt) + " targets exceed its limit (" +
                   std::to_string(kPartialDoubles / 3) + " targets at most); use sbslpm_direct_sum_bve");
    return SBSLPM_ERR_ARG;
  }
  if (nt == 0) return SBSLPM_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaSuccess;
  if (ns == 0) {
    double* outs[3] = {ux, uy, uz};
    for (double* o : outs)
      if ((e = cudaMemsetAsync(o, 0, sizeof(double) * nt, st)) != cudaSuccess) break;
  } else {
    long groups = direct_groups(nt, ns);
    const long fit = kPartialDoubles / (3 * nt);
    if (groups > fit) groups = fit;
    double *out[3] = {ux, uy, uz}, *to[3] = {ux, uy, uz};
    void* apart = nullptr;
    if (direct_in_place(nt, {tx, ty, tz}, ns, {sx, sy, sz, s}, {ux, uy, uz})) {
      e = cudaGetSymbolAddress(&apart, g_apart);
      for (int k = 0; k < 3 && e == cudaSuccess; k++) out[k] = static_cast<double*>(apart) + k * nt;
    }
    if (e == cudaSuccess) {
      launch_direct_bve(nt, tx, ty, tz, ns, sx, sy, sz, s, eps, precision, (int)groups, out[0], out[1], out[2], st);
      e = cudaGetLastError();
    }
    for (int k = 0; k < 3 && apart && e == cudaSuccess; k++)
      e = cudaMemcpyAsync(to[k], out[k], sizeof(double) * nt, cudaMemcpyDeviceToDevice, st);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    set_last_error(std::string("sbslpm_direct_sum_bve_noalloc: ") + cudaGetErrorString(e));
    return SBSLPM_ERR_CUDA;
  }
  return SBSLPM_OK;
}

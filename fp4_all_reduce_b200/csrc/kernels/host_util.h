// Small host-side helpers shared by the translation units of the library.
#pragma once
#include <cuda_runtime.h>
#include "../include/fp4ar.h"

namespace fp4ar {

constexpr int kMaxRanksOps = FP4AR_MAX_RANKS;

// Remembers the text of the last failed CUDA call for fp4ar_last_cuda_error().
void set_last_cuda_error(cudaError_t e, const char* where);
int cuda_fail();                 // records cudaGetLastError(), returns FP4AR_ERR_CUDA
int cuda_check_launch();         // FP4AR_OK, or FP4AR_ERR_CUDA if the launch was rejected
int device_sm_count();           // multiprocessors of the current device (cached per device)

// Launch of a kernel that begins with pdl_wait_prior_grids(): as a programmatic dependent of what precedes it in the
// stream, so that its CTAs are set up while that still runs, and without the runtime's <<<>>> path (3.2 us of host time
// per launch against 2.2).
template <class... P, class... A>
int launch_dependent(void (*kernel)(P...), int grid, int block, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  if (e == cudaSuccess) return FP4AR_OK;
  set_last_cuda_error(e, "launch");
  cudaGetLastError();
  return FP4AR_ERR_CUDA;
}

}  // namespace fp4ar

// Launches that may overlap the end of the kernel before them (programmatic dependent launch): a block is scheduled, sets up its barriers
// and fetches its first instructions and tensor maps while the kernel before still runs, which is most of what a kernel of a few
// microseconds takes besides its work.  Training steps (us, without / with): 144 launches of a small model 739 / 692, 346 launches of a
// 512-wide one 4463 / 4364, 428 over long documents 7680 / 7435, 986 of a speech model 52490 / 50570.
#pragma once
#include <cuda_runtime.h>

namespace b200 {

bool launch_overlap();

// `kernel` calls wait_for_previous() in every thread before it touches memory that other kernels use, and let_next_start().
template <typename... P, typename... A>
const char* launch_overlapped(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = launch_overlap() ? 1 : 0;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, P(args)...);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace b200

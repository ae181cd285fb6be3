// Launches that may overlap the end of the kernel before them (programmatic dependent launch): a block is scheduled, sets up its barriers
// and fetches its first instructions and tensor maps while the kernel before still runs, which is most of what a kernel of a few
// microseconds takes besides its work.  Training steps (us, without / with): 144 launches of a small model 739 / 692, 346 launches of a
// 512-wide one 4463 / 4364, 428 over long documents 7680 / 7435, 986 of a speech model 52490 / 50570.
// Only blocks that have an SM to themselves are launched so (more than half of its shared memory, or one block to every second SM at most).
// Several to an SM are placed while the kernel before holds some of the SMs, crowd onto the others, and run there when the rest is
// free again: a product, dropout and LayerNorm of 3000 x 512 13.2 us without overlap, 15.3 with it everywhere, 11.8 so; 20000 x 1024
// 80.5 / 90.9 / 77.2; LayerNorm gradient, dropout gradient and two products of 1000 x 512 21.8 / 21.6 / 18.0.
#pragma once
#include <cuda_runtime.h>

namespace b200 {

bool launch_overlap();
int num_sms();
constexpr int kOwnSm = 116 * 1024;      // shared memory that keeps a second such block off the SM
inline bool overlaps(long blocks, size_t smem) { return launch_overlap() && (smem >= kOwnSm || 2 * blocks <= num_sms()); }

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
  cfg.numAttrs = overlaps(static_cast<long>(grid.x) * grid.y * grid.z, smem) ? 1 : 0;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, P(args)...);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

}  // namespace b200

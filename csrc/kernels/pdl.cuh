// Programmatic dependent launch: a kernel launched with it may start while the kernel in front of it in the stream is still running,
// once all of that kernel's blocks have issued `pdl_launch` or ended.  Rules that every kernel launched this way keeps:
//   * `pdl_wait` comes before the first access to memory that an earlier kernel writes, and before the first store (a buffer may still
//     be read by the kernel in front).  It returns when the kernel in front has ended and its stores are visible.
//   * `pdl_launch` comes after `pdl_wait`: when a kernel starts, only the one in front of it can still be running.
// Without the launch attribute both instructions do nothing.
#pragma once
#include <cuda_runtime.h>
#include <string.h>

namespace rb {
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
}  // namespace rb

namespace rbhost {
// Launches `kern` with programmatic dependent launch, in clusters of `cluster` blocks along x.
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, A&&... args) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}
}  // namespace rbhost

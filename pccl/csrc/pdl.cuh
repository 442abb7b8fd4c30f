// Launches that may start before the kernel in front of them in the stream has ended (programmatic dependent
// launch).  The blocks of such a kernel take their places on the device, set up their barriers and tensor
// memory, and then wait in pdl_wait() until every kernel in front has finished and its writes are visible; what is saved is
// the launch latency and the set-up, 2-3 us per kernel in a chain of small ones.
//
// Rules every kernel launched this way keeps:
//   * no thread touches global memory before its pdl_wait(), not even to read (its inputs may be on their way, its
//     outputs may still be read), and no bounded wait on another role starts before it;
//   * nothing is read through the non-coherent path (__ldg, or a const __restrict__ pointer): that path takes memory to be
//     constant for the life of the kernel, which here begins while the kernel in front still writes;
//   * every block calls pdl_wait(), so a kernel never ends before the ones in front of it;
//   * pdl_trigger(), which lets the next kernel's blocks in, comes after the block owns all it needs (tensor memory among it):
//     a block that waits must never hold what a running one still has to acquire.
// Kernels that wait for other ranks, or for copies that run beside them, are launched the ordinary way.
#pragma once
#include <cuda_runtime.h>

namespace pccl {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// cluster: blocks per cluster along x, 0 where the kernel itself declares it (or has none).
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, unsigned cluster, bool early,
                       A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (cluster > 0) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (early) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  return e != cudaSuccess ? e : cudaGetLastError();
}
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
  return launch_pdl(kernel, grid, block, smem, stream, 0u, true, args...);
}

}  // namespace pccl

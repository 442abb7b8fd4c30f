// Reduce-scatter and two-phase all-reduce of float32 inputs.
#include "collectives.cuh"

namespace pccl {

cudaError_t launch_reduce_scatter_f32(const ReduceScatterArgs& a, bool ragged, int nlanes, cudaStream_t stream) {
  return launch_reduce_scatter_of<kF32>(a, ragged, nlanes, stream);
}

cudaError_t launch_all_reduce_rsag_f32(const AllReduceRsAgArgs& a, bool ragged, int nlanes, cudaStream_t stream) {
  return launch_all_reduce_rsag_of<kF32>(a, ragged, nlanes, stream);
}

}  // namespace pccl

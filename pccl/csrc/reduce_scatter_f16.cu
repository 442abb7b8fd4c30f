// Reduce-scatter and two-phase all-reduce of float16 inputs.
#include "collectives.cuh"

namespace pccl {

cudaError_t launch_reduce_scatter_f16(const ReduceScatterArgs& a, bool ragged, int nlanes, cudaStream_t stream) {
  return launch_reduce_scatter_of<kF16>(a, ragged, nlanes, stream);
}

cudaError_t launch_all_reduce_rsag_f16(const AllReduceRsAgArgs& a, bool ragged, int nlanes, cudaStream_t stream) {
  return launch_all_reduce_rsag_of<kF16>(a, ragged, nlanes, stream);
}

}  // namespace pccl

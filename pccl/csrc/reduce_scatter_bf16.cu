// Reduce-scatter and two-phase all-reduce of bfloat16 inputs.
#include "collectives.cuh"

namespace pccl {

cudaError_t launch_reduce_scatter_bf16(const ReduceScatterArgs& a, bool ragged, int nlanes, cudaStream_t stream) {
  return launch_reduce_scatter_of<kBF16>(a, ragged, nlanes, stream);
}

cudaError_t launch_all_reduce_rsag_bf16(const AllReduceRsAgArgs& a, bool ragged, int nlanes, cudaStream_t stream) {
  return launch_all_reduce_rsag_of<kBF16>(a, ragged, nlanes, stream);
}

}  // namespace pccl

// Reduce-scatter of bfloat16 inputs.
#include "collectives.cuh"

namespace pccl {

cudaError_t launch_reduce_scatter_bf16(const ReduceScatterArgs& a, RsForm form, int nlanes, cudaStream_t stream) {
  return launch_reduce_scatter_of<kBF16>(a, form, nlanes, stream);
}

}  // namespace pccl

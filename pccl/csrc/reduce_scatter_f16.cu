// Reduce-scatter of float16 inputs.
#include "collectives.cuh"

namespace pccl {

cudaError_t launch_reduce_scatter_f16(const ReduceScatterArgs& a, RsForm form, int nlanes, cudaStream_t stream) {
  return launch_reduce_scatter_of<kF16>(a, form, nlanes, stream);
}

}  // namespace pccl

// Reduce-scatter of float32 inputs.
#include "collectives.cuh"

namespace pccl {

cudaError_t launch_reduce_scatter_f32(const ReduceScatterArgs& a, RsForm form, int nlanes, cudaStream_t stream) {
  return launch_reduce_scatter_of<kF32>(a, form, nlanes, stream);
}

}  // namespace pccl

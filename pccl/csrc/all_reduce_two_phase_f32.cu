// The all-reduce that runs a reduce-scatter and an all-gather in one launch, for float32.
#include "collectives.cuh"

namespace pccl {

cudaError_t launch_all_reduce_rsag_f32(const AllReduceRsAgArgs& a, RsForm form, int nlanes, cudaStream_t stream) {
  return launch_all_reduce_rsag_of<kF32>(a, form, nlanes, stream);
}

}  // namespace pccl

// The all-reduce that runs a reduce-scatter and an all-gather in one launch, for float16.
#include "collectives.cuh"

namespace pccl {

cudaError_t launch_all_reduce_rsag_f16(const AllReduceRsAgArgs& a, RsForm form, int nlanes, cudaStream_t stream) {
  return launch_all_reduce_rsag_of<kF16>(a, form, nlanes, stream);
}

}  // namespace pccl

// The all-reduce that runs a reduce-scatter and an all-gather in one launch, for bfloat16.
#include "collectives.cuh"

namespace pccl {

cudaError_t launch_all_reduce_rsag_bf16(const AllReduceRsAgArgs& a, RsForm form, int nlanes, cudaStream_t stream) {
  return launch_all_reduce_rsag_of<kBF16>(a, form, nlanes, stream);
}

}  // namespace pccl

// Host-callable launchers of the collective kernels.
// They take fully-resolved argument blocks and enqueue exactly one kernel on `stream`.
#pragma once
#include <cuda_runtime.h>

#include "device_types.h"

namespace pccl {

cudaError_t launch_all_gather(const AllGatherArgs& a, int nlanes, cudaStream_t stream);
cudaError_t launch_reduce_scatter(const ReduceScatterArgs& a, int nlanes, cudaStream_t stream);
cudaError_t launch_all_reduce(const AllReduceArgs& a, int nlanes, cudaStream_t stream);
cudaError_t launch_all_reduce_rsag(const AllReduceRsAgArgs& a, int nlanes, cudaStream_t stream);
cudaError_t launch_broadcast(const BroadcastArgs& a, int nlanes, cudaStream_t stream);
cudaError_t launch_barrier(const BarrierArgs& a, cudaStream_t stream);

// What reduce-scatter and the two-phase all-reduce choose between: a form of the kernel, and the input's type.
enum RsForm : int {
  kRsAligned = 0,    // every operand starts on a 16-byte boundary; the middle steps sum in thread loops
  kRsStreamed = 1,   // the same with the middle steps summed from shared memory, which the copy engine fills (16-bit types)
  kRsRagged = 2,     // misaligned operands, loaded in aligned vectors and shifted into place
};
RsForm rs_form(const ReduceScatterArgs& a);      // the rule
cudaError_t launch_reduce_scatter_bf16(const ReduceScatterArgs& a, RsForm form, int nlanes, cudaStream_t stream);
cudaError_t launch_reduce_scatter_f16(const ReduceScatterArgs& a, RsForm form, int nlanes, cudaStream_t stream);
cudaError_t launch_reduce_scatter_f32(const ReduceScatterArgs& a, RsForm form, int nlanes, cudaStream_t stream);
cudaError_t launch_all_reduce_rsag_bf16(const AllReduceRsAgArgs& a, RsForm form, int nlanes, cudaStream_t stream);
cudaError_t launch_all_reduce_rsag_f16(const AllReduceRsAgArgs& a, RsForm form, int nlanes, cudaStream_t stream);
cudaError_t launch_all_reduce_rsag_f32(const AllReduceRsAgArgs& a, RsForm form, int nlanes, cudaStream_t stream);

// Largest lane count (grid.x) that is guaranteed to be co-resident on `device`.
int max_resident_lanes(int device);

}  // namespace pccl

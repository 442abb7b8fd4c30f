// Host-callable launchers of the collective kernels (collectives.cu).
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

// What launch_reduce_scatter and launch_all_reduce_rsag choose between: the input's type, and the kernel for misaligned
// operands (the rule is at rs_ragged) or the one for aligned ones.
cudaError_t launch_reduce_scatter_bf16(const ReduceScatterArgs& a, bool ragged, int nlanes, cudaStream_t stream);
cudaError_t launch_all_reduce_rsag_bf16(const AllReduceRsAgArgs& a, bool ragged, int nlanes, cudaStream_t stream);
cudaError_t launch_reduce_scatter_f16(const ReduceScatterArgs& a, bool ragged, int nlanes, cudaStream_t stream);
cudaError_t launch_all_reduce_rsag_f16(const AllReduceRsAgArgs& a, bool ragged, int nlanes, cudaStream_t stream);
cudaError_t launch_reduce_scatter_f32(const ReduceScatterArgs& a, bool ragged, int nlanes, cudaStream_t stream);
cudaError_t launch_all_reduce_rsag_f32(const AllReduceRsAgArgs& a, bool ragged, int nlanes, cudaStream_t stream);

// Largest lane count (grid.x) that is guaranteed to be co-resident on `device`.
int max_resident_lanes(int device);

}  // namespace pccl

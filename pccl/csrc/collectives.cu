// The all-gather, one-shot all-reduce, broadcast and barrier kernels, and the choice of a reduce-scatter kernel.
#include "collectives.cuh"

namespace pccl {

namespace {

__global__ void __launch_bounds__(kCollThreads, 1) all_gather_kernel(const __grid_constant__ AllGatherArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  BulkPipe pipe;
  bulk_pipe_init(pipe, smem, a.g.timeout_ns);
  all_gather_body(a, pipe, 16, kCollAllGather);
}

// ============================================================================ all-reduce
// Two-shot in one kernel: member r reduces slice r (loading it from every heap) and writes
// the result back into slice r of every heap; nobody else touches slice r, so the
// operation is in place.  The composition reduce-scatter + all-gather is what
// pccl/src/yacl.cpp:146-177 of the reference does with two temporaries and two host loops.
template <int DT>
__global__ void __launch_bounds__(kCollThreads, 1) all_reduce_kernel(const __grid_constant__ AllReduceArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const GroupDev& g = a.g;
  const int P = g.size;
  const LaneCtx c{(int)blockIdx.y, g.first_local + (int)blockIdx.y, (int)blockIdx.x, kCollAllReduce};
  const int me = c.me;
  constexpr uint64_t S = Elem<DT>::size;
  const uint64_t per = (((a.elems + P - 1) / P) + 7) / 8 * 8;  // slice length, multiple of 8 elements
  char* data = a.data[c.li];
  char* buf = g.heap[me] + a.buf_off;
  const unsigned others = others_mask(P, me);
  BulkPipe pipe;
  bulk_pipe_init(pipe, smem, g.timeout_ns);

  auto slice = [&](int s, uint64_t* lo, uint64_t* cnt) {
    uint64_t b = (uint64_t)s * per, e = b + per;
    if (b > a.elems) b = a.elems;
    if (e > a.elems) e = a.elems;
    uint64_t l, h;
    lane_range(e - b, 8, c.lane, gridDim.x, &l, &h);
    *lo = b + l;
    *cnt = h - l;
  };

  if (P == 1) {
    uint64_t lo, cnt;
    slice(0, &lo, &cnt);
    char* p = (data != nullptr ? data : buf) + lo * S;
    if (a.scale != 1.0f) cta_reduce<DT, DT, DT, false>(&p, 1, p, nullptr, 0, cnt, a.scale);
    return;
  }

  if (data != nullptr)
    for (int s = 0; s < P; ++s) {
      uint64_t lo, cnt;
      slice(s, &lo, &cnt);
      if (!lane_copy1<false>(pipe, buf + lo * S, data + lo * S, cnt * S)) return;
    }
  publish_mask(pipe, g, c, kSlotEntry, others);
  if (!cta_wait_mask(g, c, kSlotEntry, others)) return;

  uint64_t lo, cnt;
  slice(me, &lo, &cnt);
  if (a.algo == kMultimem) {
    constexpr int EPV = 16 / (int)S;
    char* mc = g.mc_heap + a.buf_off + lo * S;
    const uint64_t nvec = cnt / EPV;
    for (uint64_t i = threadIdx.x; i < nvec; i += blockDim.x) {
      uint4 v = multimem_ld_reduce_v4<DT>(mc + (i << 4));
      if (a.scale != 1.0f) {
        if constexpr (DT == kF32) {
          v.x = __float_as_uint(__uint_as_float(v.x) * a.scale); v.y = __float_as_uint(__uint_as_float(v.y) * a.scale);
          v.z = __float_as_uint(__uint_as_float(v.z) * a.scale); v.w = __float_as_uint(__uint_as_float(v.w) * a.scale);
        } else {
          float f[8];
          Elem<DT>::unpack(v, f);
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] *= a.scale;
          v = Elem<DT>::pack(f);
        }
      }
      multimem_st_v4(mc + (i << 4), v);
    }
  } else {
    const char* w[kMaxReduceSrc];
    char* outs[kMaxRanks];
    int nw = 0, no = 0;
    outs[no++] = buf + lo * S;
    for (int k = 1; k < P; ++k) {
      const int p = pmod(me + k, P);
      w[nw++] = g.heap[p] + a.buf_off + lo * S;
      outs[no++] = g.heap[p] + a.buf_off + lo * S;
    }
    cta_reduce<DT, DT, DT, true>(outs, no, buf + lo * S, w, nw, cnt, a.scale);
  }
  cta_signal_mask(g, c, kSlotStep0, others);
  if (!cta_wait_mask(g, c, kSlotStep0, others)) return;

  if (data != nullptr)
    for (int s = 0; s < P; ++s) {
      uint64_t l2, c2;
      slice(s, &l2, &c2);
      if (!lane_copy1<true>(pipe, data + l2 * S, buf + l2 * S, c2 * S)) return;
    }
  cta_bulk_flush(pipe);
}

// ============================================================================ broadcast
__global__ void __launch_bounds__(kCollThreads, 1) broadcast_kernel(const __grid_constant__ BroadcastArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const GroupDev& g = a.g;
  const int P = g.size;
  const LaneCtx c{(int)blockIdx.y, g.first_local + (int)blockIdx.y, (int)blockIdx.x, kCollBroadcast};
  const int me = c.me;
  if (P == 1) return;
  uint64_t lo, hi;
  lane_range(a.bytes, 16, c.lane, gridDim.x, &lo, &hi);
  const uint64_t len = hi - lo;
  if (len == 0) return;
  BulkPipe pipe;
  bulk_pipe_init(pipe, smem, g.timeout_ns);
  char* data = a.data[c.li];
  char* buf = g.heap[me] + a.buf_off;
  const unsigned others = others_mask(P, me);
  if (me == a.root) {
    const char* src = data != nullptr ? data : buf;
    if (!cta_wait_mask(g, c, kSlotEntry, others)) return;
    if (a.use_multimem) {
      char* mc = g.mc_heap + a.buf_off + lo;
      for (uint64_t i = threadIdx.x; i < (len >> 4); i += blockDim.x) multimem_st_v4(mc + (i << 4), ld_v4(src + lo + (i << 4)));
    } else {
      char* dsts[kMaxRanks];
      int nd = 0;
      for (int k = 1; k < P; ++k) dsts[nd++] = g.heap[pmod(me + k, P)] + a.buf_off + lo;
      if (!lane_copy<false>(pipe, dsts, nd, src + lo, len)) return;
    }
    publish_mask(pipe, g, c, kSlotStep0, others);
  } else {
    cta_signal(g, c, kSlotEntry, a.root);
    if (!cta_wait(g, c, kSlotStep0, a.root)) return;
    if (data != nullptr && !lane_copy1<true>(pipe, data + lo, buf + lo, len)) return;
    cta_bulk_flush(pipe);
  }
}

// ============================================================================ barrier
__global__ void __launch_bounds__(64, 1) barrier_kernel(const __grid_constant__ BarrierArgs a) {
  const GroupDev& g = a.g;
  const LaneCtx c{(int)blockIdx.y, g.first_local + (int)blockIdx.y, 0, kCollBarrier};
  if (g.size == 1) return;
  const unsigned others = others_mask(g.size, c.me);
  cta_signal_mask(g, c, kSlotEntry, others);
  cta_wait_mask(g, c, kSlotEntry, others);
}

}  // namespace

cudaError_t launch_all_gather(const AllGatherArgs& a, int nlanes, cudaStream_t stream) {
  return launch(all_gather_kernel, a, nlanes, kCollThreads, kBulkSmemBytes, stream);
}
// Whether some vector of a reduce-scatter would be misaligned: a block of the input, of the staging area or of the
// result that does not start on a 16-byte boundary (an odd number of elements per block, or an offset tensor).  Such calls take the
// kernel with the shifting loads.  It is a kernel of its own because the registers those loads need cost the aligned
// loops a quarter of their speed (8 ranks, 6.3 M elements: 477 against 616 us); the aligned kernel sums such operands
// element by element (8 ranks, 1000003 elements, direct: 1000 against 180 us).
static bool rs_ragged(const ReduceScatterArgs& a) {
  const uint64_t sw = (uint64_t)dtype_size(a.wire_dtype);
  uint64_t m = a.dst_stride | a.out_sub_stride * (a.nsub > 1) | a.sub_stride * (a.nsub > 1);
  if (a.algo == kPull || a.algo == kMultimem) m |= a.in_off;
  else if (a.g.size > 1) m |= a.stage_off | a.stage_elems * sw;
  for (int i = 0; i < a.g.nlocal; ++i) m |= (uint64_t)reinterpret_cast<uintptr_t>(a.in[i]) | (uint64_t)reinterpret_cast<uintptr_t>(a.out[i]);
  return (m & 15u) != 0;
}

// The middle steps of the ring and halving schedules add one or two staged blocks to one of their own.  With little data
// the sums come from L2 and the thread loops are faster; once the inputs of this device's ranks exceed what L2 holds
// (126 MB) the copy engine keeps more loads in flight, for 16-bit types only.  Halving over eight ranks, with two staged sources in
// its last step, gains from half of that on.  It is a kernel of its own because either path costs the other 4-7 % beside it in
// one kernel (registers).  Measured on one device, thread loops / copy engine (us): 4 ranks, ring, 16 lanes of
// 200 KB / 700 KB / 4 MB 80 / 95, 224 / 213, 1181 / 992; 8 ranks, halving, 8 lanes of 200 KB / 700 KB 147 / 146, 437 / 376; 8 ranks, halving,
// 18 lanes of 700 KB 525 / 436; fp32, 8 ranks, ring, 8 lanes of 700 KB 314 / 355.
RsForm rs_form(const ReduceScatterArgs& a) {
  if (rs_ragged(a)) return kRsRagged;
  if (a.in_dtype == kF32 || a.wire_dtype != a.in_dtype || (a.algo != kRing && a.algo != kRecursive)) return kRsAligned;
  const uint64_t bytes = (uint64_t)a.g.nlocal * a.g.size * a.nsub * a.sub_elems * dtype_size(a.in_dtype);
  const uint64_t line = a.algo == kRecursive && a.g.size >= 8 ? 80ull << 20 : 160ull << 20;
  return bytes > line ? kRsStreamed : kRsAligned;
}
cudaError_t launch_reduce_scatter(const ReduceScatterArgs& a, int nlanes, cudaStream_t stream) {
  if (a.stage_elems < a.sub_elems) return cudaErrorInvalidValue;
  const RsForm form = rs_form(a);
  if (a.in_dtype == kBF16) return launch_reduce_scatter_bf16(a, form, nlanes, stream);
  if (a.in_dtype == kF16) return launch_reduce_scatter_f16(a, form, nlanes, stream);
  if (a.in_dtype == kF32) return launch_reduce_scatter_f32(a, form, nlanes, stream);
  return cudaErrorInvalidValue;
}

cudaError_t launch_all_reduce(const AllReduceArgs& a, int nlanes, cudaStream_t stream) {
  if (a.dtype == kBF16) return launch(all_reduce_kernel<kBF16>, a, nlanes, kCollThreads, kBulkSmemBytes, stream);
  if (a.dtype == kF16) return launch(all_reduce_kernel<kF16>, a, nlanes, kCollThreads, kBulkSmemBytes, stream);
  if (a.dtype == kF32) return launch(all_reduce_kernel<kF32>, a, nlanes, kCollThreads, kBulkSmemBytes, stream);
  return cudaErrorInvalidValue;
}
cudaError_t launch_all_reduce_rsag(const AllReduceRsAgArgs& a, int nlanes, cudaStream_t stream) {
  if (a.rs.stage_elems < a.rs.sub_elems) return cudaErrorInvalidValue;
  const RsForm form = rs_form(a.rs);
  if (a.rs.in_dtype == kBF16) return launch_all_reduce_rsag_bf16(a, form, nlanes, stream);
  if (a.rs.in_dtype == kF16) return launch_all_reduce_rsag_f16(a, form, nlanes, stream);
  if (a.rs.in_dtype == kF32) return launch_all_reduce_rsag_f32(a, form, nlanes, stream);
  return cudaErrorInvalidValue;
}

cudaError_t launch_broadcast(const BroadcastArgs& a, int nlanes, cudaStream_t stream) {
  return launch(broadcast_kernel, a, nlanes, kCollThreads, kBulkSmemBytes, stream);
}

cudaError_t launch_barrier(const BarrierArgs& a, cudaStream_t stream) {
  return launch(barrier_kernel, a, 1, 64, 0, stream);
}

int max_resident_lanes(int device) {
  int sms = 0, per_sm = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  if (cudaFuncSetAttribute(reinterpret_cast<const void*>(all_gather_kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kBulkSmemBytes) != cudaSuccess)
    return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, all_gather_kernel, kCollThreads, kBulkSmemBytes) != cudaSuccess)
    return 0;
  int m = sms * (per_sm > 0 ? 1 : 0);  // the kernels are written for one CTA per SM
  return m > kMaxLanes ? kMaxLanes : m;
}

}  // namespace pccl

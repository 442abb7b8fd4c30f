// Device-side building blocks of the collective kernels: system-scope flags with bounded
// waits, CTA-wide copies to and from peer memory, fp32-accumulating reductions and the
// NVLS multimem wrappers.
//
// Memory-ordering contract used throughout:
//   producer:  data stores (weak)  ->  bar.sync  ->  st.release.sys flag (cumulative: it covers what the barrier ordered
//              before it; a separate system fence in front of it would be a second one of the same kind)
//   consumer:  ld.acquire.sys flag (one thread)  ->  bar.sync  ->  data loads
// Flags and peer data are never read through the non-coherent (.nc) path.
// Flags carry the call number (epoch) of the group, so they are never reset and a rank
// that runs ahead by one call cannot be mistaken for the current one.
//
// The reference gets ordering from a host-side cudaEventSynchronize before every
// MPI_Sendrecv (pccl/src/all_gather.cpp:57-63); here nothing leaves the device.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "device_types.h"

namespace pccl {

constexpr int kCollThreads = 512;

// ---------------------------------------------------------------- raw accessors
__device__ __forceinline__ void st_release_sys(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_relaxed_sys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// 16-byte load that bypasses L1: used for memory that another GPU may have written.
__device__ __forceinline__ uint4 ld_volatile_v4(const void* p) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_v4(const void* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ void st_v4(void* p, uint4 v) { *reinterpret_cast<uint4*>(p) = v; }

// ---------------------------------------------------------------- status / failure
__device__ __forceinline__ void report_failure(const GroupDev& g, int li, uint32_t code, uint32_t coll,
                                               int me, int peer, int lane, int kind, uint32_t seen) {
  Status* st = g.status[li];
  if (st != nullptr && atomicCAS(&st->code, (uint32_t)kStatusOk, code) == kStatusOk) {
    st->epoch = g.epoch;
    st->rank = me;
    st->peer = peer;
    st->lane = lane;
    st->slot_kind = kind;
    st->seen = seen;
    st->collective = coll;
    __threadfence_system();
  }
  if (g.poison[li] != nullptr) atomicExch(g.poison[li], 1u);
}

// One thread spins until flag >= epoch (wrap-safe), the time limit runs out, or the
// communicator is poisoned.  Never traps, never spins without a limit.  (Polling with relaxed
// loads and one acquire fence at the end was tried and was not faster.)
__device__ __forceinline__ bool spin_until(const uint32_t* flag, uint32_t epoch, const GroupDev& g, int li,
                                           uint32_t* seen_out) {
  uint32_t v = ld_acquire_sys(flag);
  if ((int32_t)(v - epoch) >= 0) return true;
  const uint64_t t0 = global_timer_ns();
  const uint32_t* poison = g.poison[li];
  uint32_t it = 0;
  for (;;) {
    v = ld_acquire_sys(flag);
    if ((int32_t)(v - epoch) >= 0) return true;
    if ((++it & 63u) == 0u) {
      if (poison != nullptr && *reinterpret_cast<const volatile uint32_t*>(poison) != 0u) break;
      if (global_timer_ns() - t0 > g.timeout_ns) break;
      __nanosleep(64);
    }
  }
  *seen_out = v;
  return false;
}

struct LaneCtx {
  int li;     // local rank slot (blockIdx.y)
  int me;     // my group index
  int lane;   // blockIdx.x
  uint32_t coll;
};

// Debug hooks of every synchronisation point; both are off (two predictable branches) unless the
// communicator switched them on.  Called by one thread.
//  * stress mode: sleep a pseudo-random, bounded time, so that lanes and ranks meet their waits
//    and signals in orders a quiet machine never produces; results must not change.
//  * trace: append (time, epoch, rank, lane, slot kind, wait|signal) to the trace buffer.
__device__ __forceinline__ void debug_jitter(const GroupDev& g, const LaneCtx& c, int kind) {
  if (g.jitter_ns == 0u) return;
  uint32_t h = g.epoch * 0x9E3779B1u ^ (uint32_t)c.lane * 0x85EBCA77u ^ (uint32_t)c.me * 0xC2B2AE3Du ^ (uint32_t)kind * 0x27D4EB2Fu ^
               (uint32_t)global_timer_ns();
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 12;
  uint32_t ns = h % g.jitter_ns;
  while (ns > 0u) {                       // at most jitter_ns in total
    const uint32_t step = ns < 500000u ? ns : 500000u;
    __nanosleep(step);
    ns -= step;
  }
}
__device__ __forceinline__ void debug_trace(const GroupDev& g, const LaneCtx& c, int kind, bool is_signal) {
  TraceBuf* tb = g.trace;
  if (tb == nullptr) return;
  const unsigned long long i = atomicAdd(&tb->count, 1ull);
  if (i < tb->capacity) {
    TraceEvent e;
    e.t_ns = global_timer_ns();
    e.epoch = g.epoch;
    e.lane = (uint16_t)c.lane;
    e.rank = (uint8_t)c.me;
    e.what = (uint8_t)((kind & 63) | (is_signal ? 64 : 0));
    e.collective = c.coll;
    e.pad = 0;
    tb->ev[i] = e;
  }
}

// All threads of the CTA call this; thread 0 waits.  Returns false (to all threads) when
// the wait gave up; the status word then says where.
__device__ __forceinline__ bool cta_wait(const GroupDev& g, const LaneCtx& c, int kind, int src) {
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    debug_jitter(g, c, kind);
    uint32_t seen = 0;
    const uint32_t* flag = g.sig[c.me] + slot_index(c.lane, kind, src);
    bool ok = spin_until(flag, g.epoch, g, c.li, &seen);
    if (ok) debug_trace(g, c, kind, false);
    if (!ok) {
      const bool poisoned = g.poison[c.li] != nullptr &&
                            *reinterpret_cast<const volatile uint32_t*>(g.poison[c.li]) != 0u;
      report_failure(g, c.li, poisoned ? kStatusPoisoned : kStatusTimeout, c.coll, c.me, src, c.lane, kind, seen);
    }
    s_ok = ok ? 1 : 0;
  }
  __syncthreads();
  const int ok = s_ok;
  __syncthreads();
  return ok != 0;
}

// Wait for the same slot kind from every member whose bit is set in `mask`.
__device__ __forceinline__ bool cta_wait_mask(const GroupDev& g, const LaneCtx& c, int kind, unsigned mask) {
  __shared__ int s_ok_all;
  if (threadIdx.x == 0) {
    s_ok_all = 1;
    debug_jitter(g, c, kind);
  }
  __syncthreads();
  if (threadIdx.x < (unsigned)g.size && ((mask >> threadIdx.x) & 1u)) {
    uint32_t seen = 0;
    const int src = threadIdx.x;
    const uint32_t* flag = g.sig[c.me] + slot_index(c.lane, kind, src);
    if (!spin_until(flag, g.epoch, g, c.li, &seen)) {
      const bool poisoned = g.poison[c.li] != nullptr &&
                            *reinterpret_cast<const volatile uint32_t*>(g.poison[c.li]) != 0u;
      report_failure(g, c.li, poisoned ? kStatusPoisoned : kStatusTimeout, c.coll, c.me, src, c.lane, kind, seen);
      atomicExch(&s_ok_all, 0);
    }
  }
  __syncthreads();
  const int ok = s_ok_all;
  if (ok != 0 && threadIdx.x == 0) debug_trace(g, c, kind, false);
  __syncthreads();
  return ok != 0;
}

// Publish slot(lane, kind, me) = epoch in the pad of every member in `mask`.
// The leading bar.sync orders every thread's earlier stores before the release.
__device__ __forceinline__ void cta_signal_mask(const GroupDev& g, const LaneCtx& c, int kind, unsigned mask) {
  if (threadIdx.x == 0) {
    debug_jitter(g, c, kind);          // the whole CTA waits at the barrier below: the flags go out late
    debug_trace(g, c, kind, true);
  }
  __syncthreads();
  if (threadIdx.x < (unsigned)g.size && ((mask >> threadIdx.x) & 1u)) {
    st_release_sys(g.sig[threadIdx.x] + slot_index(c.lane, kind, c.me), g.epoch);
  }
}
__device__ __forceinline__ void cta_signal(const GroupDev& g, const LaneCtx& c, int kind, int dst) {
  cta_signal_mask(g, c, kind, 1u << dst);
}

__device__ __forceinline__ unsigned others_mask(int P, int me) { return ((1u << P) - 1u) & ~(1u << me); }

// ---------------------------------------------------------------- lane partition
// Split `total` bytes/elements into gridDim.x contiguous pieces on `gran` boundaries.
__device__ __forceinline__ void lane_range(uint64_t total, uint64_t gran, int lane, int nlanes, uint64_t* lo,
                                           uint64_t* hi) {
  const uint64_t units = (total + gran - 1) / gran;
  const uint64_t per = (units + nlanes - 1) / nlanes;
  uint64_t a = per * lane, b = a + per;
  if (a > units) a = units;
  if (b > units) b = units;
  a *= gran;
  b *= gran;
  if (a > total) a = total;
  if (b > total) b = total;
  *lo = a;
  *hi = b;
}

// ---------------------------------------------------------------- misaligned ranges
// A range whose source and destination do not share their position within 16 bytes (blocks of an odd number
// of elements: every rank's block then starts somewhere else) is still moved in 16-byte accesses: aligned vectors
// are loaded, each lane takes the vector behind its own from its neighbour, and the pair is shifted into place.  Every
// byte is loaded once, which matters most where the source is a peer's memory.  A vector is only loaded if it holds
// at least one byte of the range, so no access leaves the range's own 16-byte granules (and with them its pages).

// Bytes [sh, sh + 16) of the 32 bytes a, b.
__device__ __forceinline__ uint4 shift16(const uint4& a, const uint4& b, uint32_t sh) {
  uint32_t w0 = a.x, w1 = a.y, w2 = a.z, w3 = a.w, w4 = b.x, w5 = b.y, w6 = b.z;
  if (sh & 8u) w0 = w2, w1 = w3, w2 = w4, w3 = w5, w4 = w6, w5 = b.w;
  if (sh & 4u) w0 = w1, w1 = w2, w2 = w3, w3 = w4, w4 = w5;
  const uint32_t bits = (sh & 3u) * 8u;
  return make_uint4(__funnelshift_r(w0, w1, bits), __funnelshift_r(w1, w2, bits), __funnelshift_r(w2, w3, bits),
                    __funnelshift_r(w3, w4, bits));
}
__device__ __forceinline__ uint4 shfl_down_v4(const uint4& v) {
  return make_uint4(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1), __shfl_down_sync(0xffffffffu, v.z, 1),
                    __shfl_down_sync(0xffffffffu, v.w, 1));
}

// The same range to several destinations that share their position within 16 bytes, but not the source's.
// Called by all threads of the block.  Measured against the byte loop in its place, 8 x 2 MB blocks of an odd
// length on one device (all-gather, direct): 352 -> 46 us.
template <bool REMOTE_SRC>
__device__ __noinline__ void cta_copy_shifted(char* const* dsts, int ndst, const char* src, uint64_t n) {
  const uint64_t tid = threadIdx.x, nt = blockDim.x;
  const uint32_t lane = threadIdx.x & 31u;
  uint64_t head = (16 - (reinterpret_cast<uintptr_t>(dsts[0]) & 15u)) & 15u;
  if (head > n) head = n;
  const uint64_t nvec = (n - head) >> 4;
  const uint32_t sh = (uint32_t)(reinterpret_cast<uintptr_t>(src + head) & 15u);      // never 0 here
  const char* sa = src + head - sh;
  constexpr int U = 4;
  for (uint64_t i0 = tid - lane; i0 < nvec; i0 += U * nt) {                           // whole warps: the lanes exchange vectors
    uint4 v[U], last[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const uint64_t i = i0 + k * nt + lane;
      v[k] = last[k] = make_uint4(0u, 0u, 0u, 0u);
      if (i <= nvec) v[k] = REMOTE_SRC ? ld_volatile_v4(sa + (i << 4)) : ld_v4(sa + (i << 4));
      if (lane == 31u && i < nvec) last[k] = REMOTE_SRC ? ld_volatile_v4(sa + ((i + 1) << 4)) : ld_v4(sa + ((i + 1) << 4));
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const uint64_t i = i0 + k * nt + lane;
      uint4 next = shfl_down_v4(v[k]);
      if (lane == 31u) next = last[k];
      const uint4 out = shift16(v[k], next, sh);
      if (i < nvec)
        for (int d = 0; d < ndst; ++d) st_v4(dsts[d] + head + (i << 4), out);
    }
  }
  const uint64_t done = head + (nvec << 4);
  const volatile char* s = src;                  // a peer may have written the ends as well
  for (uint64_t j = tid; j < head; j += nt) {
    const char b = s[j];
    for (int d = 0; d < ndst; ++d) dsts[d][j] = b;
  }
  for (uint64_t j = done + tid; j < n; j += nt) {
    const char b = s[j];
    for (int d = 0; d < ndst; ++d) dsts[d][j] = b;
  }
}

// ---------------------------------------------------------------- CTA-wide copy
// REMOTE_SRC: the source may have been written by another GPU during this kernel.
// RAGGED: with the code for ranges that do not share their position within 16 bytes; without it they are
// copied byte by byte (kernels that leave it out are only launched where no such range occurs).
template <bool REMOTE_SRC, bool RAGGED>
__device__ __forceinline__ void cta_copy(char* __restrict__ dst, const char* __restrict__ src, uint64_t n) {
  if (n == 0 || dst == src) return;
  const uint64_t tid = threadIdx.x, nt = blockDim.x;
  const uintptr_t ds = reinterpret_cast<uintptr_t>(dst), ss = reinterpret_cast<uintptr_t>(src);
  if (((ds ^ ss) & 15u) == 0) {
    uint64_t head = (16 - (ss & 15u)) & 15u;
    if (head > n) head = n;
    for (uint64_t i = tid; i < head; i += nt) dst[i] = src[i];
    const uint64_t nvec = (n - head) >> 4;
    const char* s = src + head;
    char* d = dst + head;
    constexpr int U = 8;
    uint64_t i = tid;
    for (; i + (U - 1) * nt < nvec; i += U * nt) {
      uint4 v[U];
#pragma unroll
      for (int k = 0; k < U; ++k)
        v[k] = REMOTE_SRC ? ld_volatile_v4(s + ((i + k * nt) << 4)) : ld_v4(s + ((i + k * nt) << 4));
#pragma unroll
      for (int k = 0; k < U; ++k) st_v4(d + ((i + k * nt) << 4), v[k]);
    }
    for (; i < nvec; i += nt) {
      uint4 v = REMOTE_SRC ? ld_volatile_v4(s + (i << 4)) : ld_v4(s + (i << 4));
      st_v4(d + (i << 4), v);
    }
    const uint64_t done = head + (nvec << 4);
    for (uint64_t j = done + tid; j < n; j += nt) dst[j] = src[j];
  } else if constexpr (RAGGED) {
    char* d[1] = {dst};
    cta_copy_shifted<REMOTE_SRC>(d, 1, src, n);
  } else {
    const volatile char* s = src;
    for (uint64_t i = tid; i < n; i += nt) dst[i] = s[i];
  }
}

// The same range to several destinations in one pass: every vector is loaded once and stored
// ndst times (a pass per destination pays the load latency ndst times, which is most of the
// time of a small all-gather to seven peers).  Falls back to a pass per destination when the
// destinations do not share their position within 16 bytes.
template <bool REMOTE_SRC, bool RAGGED>
__device__ __forceinline__ void cta_copy_multi(char* const* dsts, int ndst, const char* __restrict__ src, uint64_t n) {
  if (n == 0 || ndst == 0) return;
  const uintptr_t ss = reinterpret_cast<uintptr_t>(src);
  bool together = true;
  for (int d = 1; d < ndst; ++d)
    together = together && ((reinterpret_cast<uintptr_t>(dsts[d]) ^ reinterpret_cast<uintptr_t>(dsts[0])) & 15u) == 0;
  const bool congruent = ((reinterpret_cast<uintptr_t>(dsts[0]) ^ ss) & 15u) == 0;
  if (ndst == 1 || !together || (!RAGGED && !congruent)) {
    for (int d = 0; d < ndst; ++d) cta_copy<REMOTE_SRC, RAGGED>(dsts[d], src, n);
    return;
  }
  if constexpr (RAGGED) {
    if (!congruent) {
      cta_copy_shifted<REMOTE_SRC>(dsts, ndst, src, n);
      return;
    }
  }
  const uint64_t tid = threadIdx.x, nt = blockDim.x;
  uint64_t head = (16 - (ss & 15u)) & 15u;
  if (head > n) head = n;
  for (uint64_t i = tid; i < head; i += nt) {
    const char b = src[i];
    for (int d = 0; d < ndst; ++d) dsts[d][i] = b;
  }
  const uint64_t nvec = (n - head) >> 4;
  const char* s = src + head;
  constexpr int U = 4;
  uint64_t i = tid;
  for (; i + (U - 1) * nt < nvec; i += U * nt) {
    uint4 v[U];
#pragma unroll
    for (int k = 0; k < U; ++k)
      v[k] = REMOTE_SRC ? ld_volatile_v4(s + ((i + k * nt) << 4)) : ld_v4(s + ((i + k * nt) << 4));
    for (int d = 0; d < ndst; ++d) {
      char* o = dsts[d] + head;
#pragma unroll
      for (int k = 0; k < U; ++k) st_v4(o + ((i + k * nt) << 4), v[k]);
    }
  }
  for (; i < nvec; i += nt) {
    const uint4 v = REMOTE_SRC ? ld_volatile_v4(s + (i << 4)) : ld_v4(s + (i << 4));
    for (int d = 0; d < ndst; ++d) st_v4(dsts[d] + head + (i << 4), v);
  }
  const uint64_t done = head + (nvec << 4);
  for (uint64_t j = done + tid; j < n; j += nt) {
    const char b = src[j];
    for (int d = 0; d < ndst; ++d) dsts[d][j] = b;
  }
}

// ---------------------------------------------------------------- typed 8-element vectors
template <int DT>
struct Elem;
template <>
struct Elem<kBF16> {
  static constexpr int size = 2;
  __device__ static __forceinline__ float load1(const char* p) {
    return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(p));
  }
  __device__ static __forceinline__ void store1(char* p, float f) {
    *reinterpret_cast<__nv_bfloat16*>(p) = __float2bfloat16_rn(f);
  }
  __device__ static __forceinline__ void unpack(const uint4& v, float* f) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
  __device__ static __forceinline__ uint4 pack(const float* f) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
      w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
};
template <>
struct Elem<kF16> {
  static constexpr int size = 2;
  __device__ static __forceinline__ float load1(const char* p) {
    return __half2float(*reinterpret_cast<const __half*>(p));
  }
  __device__ static __forceinline__ void store1(char* p, float f) {
    *reinterpret_cast<__half*>(p) = __float2half_rn(f);
  }
  __device__ static __forceinline__ void unpack(const uint4& v, float* f) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      f[2 * i] = t.x;
      f[2 * i + 1] = t.y;
    }
  }
  __device__ static __forceinline__ uint4 pack(const float* f) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __half2 h = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
      w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
};
template <>
struct Elem<kF32> {
  static constexpr int size = 4;
  __device__ static __forceinline__ float load1(const char* p) { return *reinterpret_cast<const float*>(p); }
  __device__ static __forceinline__ void store1(char* p, float f) { *reinterpret_cast<float*>(p) = f; }
};

// Load 8 consecutive elements as fp32.  p must be 16-byte aligned.
template <int DT, bool REMOTE>
__device__ __forceinline__ void load8(const char* p, float* f) {
  if constexpr (DT == kF32) {
    uint4 a = REMOTE ? ld_volatile_v4(p) : ld_v4(p);
    uint4 b = REMOTE ? ld_volatile_v4(p + 16) : ld_v4(p + 16);
    f[0] = __uint_as_float(a.x); f[1] = __uint_as_float(a.y); f[2] = __uint_as_float(a.z); f[3] = __uint_as_float(a.w);
    f[4] = __uint_as_float(b.x); f[5] = __uint_as_float(b.y); f[6] = __uint_as_float(b.z); f[7] = __uint_as_float(b.w);
  } else {
    uint4 a = REMOTE ? ld_volatile_v4(p) : ld_v4(p);
    Elem<DT>::unpack(a, f);
  }
}
template <int DT>
__device__ __forceinline__ void store8(char* p, const float* f) {
  if constexpr (DT == kF32) {
    st_v4(p, make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3])));
    st_v4(p + 16, make_uint4(__float_as_uint(f[4]), __float_as_uint(f[5]), __float_as_uint(f[6]), __float_as_uint(f[7])));
  } else {
    st_v4(p, Elem<DT>::pack(f));
  }
}
template <int DT>
__device__ __forceinline__ float load_scalar(const char* p) {
  return Elem<DT>::load1(p);
}

// ---------------------------------------------------------------- CTA-wide reduction
// out[i] = cast<TOUT>( scale * ( a[i] + sum_k w[k][i] ) ),  i in [0, count)
// `a` has TA elements (may be nullptr), the nw extra sources have TW elements; all sums in
// fp32, one rounding at the store.  REMOTE_W: the w sources may have been written by peers.
constexpr int kMaxReduceSrc = kMaxRanks;

template <int TOUT>
__device__ __forceinline__ void store8_all(char* const* outs, int nout, uint64_t byte_off, const float* f) {
  for (int o = 0; o < nout; ++o) store8<TOUT>(outs[o] + byte_off, f);
}

// outs: nout destinations that all receive the same result (nout > 1: the broadcast half
// of an all-reduce).
// 8 elements of type DT as they sit in memory (one 16-byte vector, two for fp32), and their sum into acc.
template <int DT>
struct Raw8 {
  uint4 v[Elem<DT>::size == 4 ? 2 : 1];
};
template <int DT, bool REMOTE>
__device__ __forceinline__ void load8_raw(const char* p, Raw8<DT>& r) {
  r.v[0] = REMOTE ? ld_volatile_v4(p) : ld_v4(p);
  if constexpr (DT == kF32) r.v[1] = REMOTE ? ld_volatile_v4(p + 16) : ld_v4(p + 16);
}
template <int DT>
__device__ __forceinline__ void add8_raw(const Raw8<DT>& r, float* acc) {
  if constexpr (DT == kF32) {
    acc[0] += __uint_as_float(r.v[0].x); acc[1] += __uint_as_float(r.v[0].y);
    acc[2] += __uint_as_float(r.v[0].z); acc[3] += __uint_as_float(r.v[0].w);
    acc[4] += __uint_as_float(r.v[1].x); acc[5] += __uint_as_float(r.v[1].y);
    acc[6] += __uint_as_float(r.v[1].z); acc[7] += __uint_as_float(r.v[1].w);
  } else {
    float t[8];
    Elem<DT>::unpack(r.v[0], t);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] += t[e];
  }
}

// The vector part of cta_reduce: G groups of 8 elements per thread and iteration, every load of
// up to KW sources at a time issued before the first add.  With a loop over the sources that adds as it
// loads, the (volatile) loads of peer memory run one round trip after another: seven peers cost
// seven NVLink latencies per iteration.  Sums are formed in source order, as before.
template <int TA, int TW, int TOUT, bool REMOTE_W, int G, int KW>
__device__ __forceinline__ uint64_t cta_reduce_groups(char* const* outs, int nout, const char* a, const char* const* w,
                                                      int nw, uint64_t i, uint64_t ngroups, float scale) {
  constexpr uint64_t SA = 8 * Elem<TA>::size, SW = 8 * Elem<TW>::size, SO = 8 * Elem<TOUT>::size;
  const uint64_t nt = blockDim.x;
  for (; i + (G - 1) * nt < ngroups; i += G * nt) {
    float acc[G][8];
    Raw8<TW> raw[G][KW];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (a != nullptr) {
        load8<TA, false>(a + (i + g * nt) * SA, acc[g]);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[g][e] = 0.f;
      }
    }
    for (int k0 = 0; k0 < nw; k0 += KW) {            // one pass unless there are more than KW sources
#pragma unroll
      for (int k = 0; k < KW; ++k)
        if (k0 + k < nw) {
#pragma unroll
          for (int g = 0; g < G; ++g) load8_raw<TW, REMOTE_W>(w[k0 + k] + (i + g * nt) * SW, raw[g][k]);
        }
#pragma unroll
      for (int k = 0; k < KW; ++k)
        if (k0 + k < nw) {
#pragma unroll
          for (int g = 0; g < G; ++g) add8_raw<TW>(raw[g][k], acc[g]);
        }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[g][e] *= scale;
      store8_all<TOUT>(outs, nout, (i + g * nt) * SO, acc[g]);
    }
  }
  return i;
}

// The vector part of cta_reduce for sources that lie anywhere (element-aligned): groups of 8 elements whose
// place in the outputs is 16-byte aligned; see "misaligned ranges" for the loads.  A warp sums 31 groups at a time, its
// last lane only lends the vector behind them: that costs 3 % of the lanes and saves a vector of registers
// per source.  Sums in source order.
template <int DT, bool REMOTE>
__device__ __forceinline__ void load8_shifted(const char* w, uint64_t i, uint64_t ngroups, Raw8<DT>& r) {
  constexpr int V = Elem<DT>::size == 4 ? 2 : 1;
  const uint32_t sh = (uint32_t)(reinterpret_cast<uintptr_t>(w) & 15u);
  const char* p = w - sh + i * (V * 16);
  r.v[0] = make_uint4(0u, 0u, 0u, 0u);
  if constexpr (V == 2) r.v[1] = r.v[0];
  if (i < ngroups || (i == ngroups && sh != 0u)) r.v[0] = REMOTE ? ld_volatile_v4(p) : ld_v4(p);
  if constexpr (V == 2) {
    if (i < ngroups) r.v[1] = REMOTE ? ld_volatile_v4(p + 16) : ld_v4(p + 16);
  }
}
template <int DT>
__device__ __forceinline__ void add8_shifted(const Raw8<DT>& r, const char* w, float* acc) {
  const uint32_t sh = (uint32_t)(reinterpret_cast<uintptr_t>(w) & 15u);
  if (sh == 0u) {                                  // the same for the whole block
    add8_raw<DT>(r, acc);
    return;
  }
  const uint4 next = shfl_down_v4(r.v[0]);
  Raw8<DT> o;
  if constexpr (Elem<DT>::size == 4) {
    o.v[0] = shift16(r.v[0], r.v[1], sh);
    o.v[1] = shift16(r.v[1], next, sh);
  } else {
    o.v[0] = shift16(r.v[0], next, sh);
  }
  add8_raw<DT>(o, acc);
}
template <int TA, int TW, int TOUT, bool REMOTE_W>
__device__ __forceinline__ void cta_reduce_shifted(char* const* outs, int nout, const char* a, const char* const* w, int nw,
                                                   uint64_t ngroups, float scale) {
  constexpr uint64_t SO = 8 * Elem<TOUT>::size;
  constexpr int KW = Elem<TW>::size == 4 ? 2 : 4;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t per_pass = (uint64_t)(blockDim.x >> 5) * 31;
  for (uint64_t i0 = (uint64_t)(threadIdx.x >> 5) * 31; i0 < ngroups; i0 += per_pass) {
    const uint64_t i = i0 + lane;
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    Raw8<TA> ra;
    if (a != nullptr) load8_shifted<TA, false>(a, i, ngroups, ra);
    for (int k0 = 0; k0 < nw || k0 == 0; k0 += KW) {
      Raw8<TW> raw[KW];
#pragma unroll
      for (int k = 0; k < KW; ++k)
        if (k0 + k < nw) load8_shifted<TW, REMOTE_W>(w[k0 + k], i, ngroups, raw[k]);
      if (k0 == 0 && a != nullptr) add8_shifted<TA>(ra, a, acc);
#pragma unroll
      for (int k = 0; k < KW; ++k)
        if (k0 + k < nw) add8_shifted<TW>(raw[k], w[k0 + k], acc);
    }
    if (lane < 31u && i < ngroups) {
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] *= scale;
      store8_all<TOUT>(outs, nout, i * SO, acc);
    }
  }
}

// RAGGED: with the code for misaligned operands (without it they are summed element by element).
template <int TA, int TW, int TOUT, bool REMOTE_W, bool RAGGED = false>
__device__ __forceinline__ void cta_reduce(char* const* outs, int nout, const char* a,
                                           const char* const* w, int nw, uint64_t count, float scale) {
  if (count == 0) return;
  const uint64_t tid = threadIdx.x, nt = blockDim.x;
  bool aligned = (a == nullptr || (reinterpret_cast<uintptr_t>(a) & 15u) == 0);
  for (int o = 0; o < nout; ++o) aligned = aligned && (reinterpret_cast<uintptr_t>(outs[o]) & 15u) == 0;
  for (int k = 0; k < nw; ++k) aligned = aligned && (reinterpret_cast<uintptr_t>(w[k]) & 15u) == 0;
  uint64_t done = 0;
  if (aligned) {
    const uint64_t ngroups = count >> 3;
    uint64_t i = tid;
    // at most 32 registers of source vectors in flight per thread
    constexpr int kWide = Elem<TW>::size == 4 ? 2 : 1;      // 16-byte vectors per 8 elements
    if (nw <= 1) i = cta_reduce_groups<TA, TW, TOUT, REMOTE_W, 2, 1>(outs, nout, a, w, nw, i, ngroups, scale);
    i = cta_reduce_groups<TA, TW, TOUT, REMOTE_W, 1, 4 / kWide>(outs, nout, a, w, nw, i, ngroups, scale);
    done = ngroups << 3;
  }
  // Element by element: what is left behind the vectors; for misaligned operands also what lies in front of the
  // outputs' first 16-byte boundary.
  uint64_t head = 0;
  if (RAGGED && !aligned) {
    const uintptr_t o0 = reinterpret_cast<uintptr_t>(outs[0]);
    bool shiftable = (o0 % Elem<TOUT>::size) == 0 && (a == nullptr || (reinterpret_cast<uintptr_t>(a) % Elem<TA>::size) == 0);
    for (int o = 1; o < nout; ++o) shiftable = shiftable && ((reinterpret_cast<uintptr_t>(outs[o]) ^ o0) & 15u) == 0;
    for (int k = 0; k < nw; ++k) shiftable = shiftable && (reinterpret_cast<uintptr_t>(w[k]) % Elem<TW>::size) == 0;
    if (shiftable) {
      head = ((16 - (o0 & 15u)) & 15u) / Elem<TOUT>::size;
      if (head > count) head = count;
      const uint64_t ngroups = (count - head) >> 3;
      if (ngroups > 0) {
        char* o2[kMaxRanks];
        const char* w2[kMaxReduceSrc];
        for (int o = 0; o < nout; ++o) o2[o] = outs[o] + head * Elem<TOUT>::size;
        for (int k = 0; k < nw; ++k) w2[k] = w[k] + head * Elem<TW>::size;
        cta_reduce_shifted<TA, TW, TOUT, REMOTE_W>(o2, nout, a != nullptr ? a + head * Elem<TA>::size : nullptr, w2, nw, ngroups, scale);
      }
      done = head + (ngroups << 3);
    }
  }
  for (uint64_t j = tid; j < head + (count - done); j += nt) {
    const uint64_t i = j < head ? j : done + (j - head);
    float acc = a != nullptr ? load_scalar<TA>(a + i * Elem<TA>::size) : 0.f;
    for (int k = 0; k < nw; ++k) {
      const char* p = w[k] + i * Elem<TW>::size;
      if constexpr (Elem<TW>::size == 4) {
        acc += __uint_as_float(REMOTE_W ? ld_relaxed_sys(reinterpret_cast<const uint32_t*>(p))
                                        : *reinterpret_cast<const uint32_t*>(p));
      } else {
        unsigned short bits = *reinterpret_cast<const volatile unsigned short*>(p);
        if constexpr (TW == kBF16) acc += __uint_as_float(uint32_t(bits) << 16);
        else acc += __half2float(__ushort_as_half(bits));
      }
    }
    for (int o = 0; o < nout; ++o) Elem<TOUT>::store1(outs[o] + i * Elem<TOUT>::size, acc * scale);
  }
}

// ---------------------------------------------------------------- NVLS (multimem) wrappers
// One instruction addresses the same offset of every GPU bound to the multicast object:
// ld_reduce sums inside the switch (fp32 accumulation for 16-bit types), st writes all.
template <int DT>
__device__ __forceinline__ uint4 multimem_ld_reduce_v4(const char* mc_ptr) {
  uint4 v;
  if constexpr (DT == kBF16) {
    asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v4.bf16x2 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(mc_ptr) : "memory");
  } else if constexpr (DT == kF16) {
    asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v4.f16x2 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(mc_ptr) : "memory");
  } else {
    asm volatile("multimem.ld_reduce.relaxed.sys.global.add.v4.f32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(mc_ptr) : "memory");
  }
  return v;
}
__device__ __forceinline__ void multimem_st_v4(char* mc_ptr, uint4 v) {
  asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(mc_ptr), "r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w)
               : "memory");
}

}  // namespace pccl

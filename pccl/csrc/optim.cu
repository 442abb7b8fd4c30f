// Elementwise training kernels of the ZeRO-3 engine: fused AdamW on a parameter shard,
// squared-norm partial sums for gradient clipping, and softmax cross-entropy computed
// forward and backward in one pass over the logits.
//
// The reference contains none of this (it hooks DeepSpeed, pccl/patch_deepspeed.py:95-126,
// and DeepSpeed brings its own optimizer); they exist here because the engine that stands
// in for DeepSpeed has to do the optimizer step inside the timed region.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "act.cuh"
#include "optim.h"
#include "pdl.cuh"

namespace pccl {

namespace {

constexpr int kOptThreads = 256;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <bool MAX>
__device__ __forceinline__ float block_reduce(float v, float* smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = MAX ? warp_max(v) : warp_sum(v);
  __syncthreads();
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  float r = MAX ? -INFINITY : 0.f;
  for (int i = 0; i < nw; ++i) r = MAX ? fmaxf(r, smem[i]) : r + smem[i];
  return r;
}

// ---------------------------------------------------------------- squared norm
// Grid-stride partial sums over 16-byte vectors (four in flight per thread), one atomicAdd per
// block into *out (zeroed by the caller).
template <typename T>
__device__ __forceinline__ float sq8(const uint4& q);
template <>
__device__ __forceinline__ float sq8<__nv_bfloat16>(const uint4& q) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  float a = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float lo = __uint_as_float(w[i] << 16), hi = __uint_as_float(w[i] & 0xffff0000u);
    a += lo * lo + hi * hi;
  }
  return a;
}
template <>
__device__ __forceinline__ float sq8<float>(const uint4& q) {
  const float a = __uint_as_float(q.x), b = __uint_as_float(q.y), c = __uint_as_float(q.z), d = __uint_as_float(q.w);
  return a * a + b * b + c * c + d * d;
}

template <typename T>
__global__ void __launch_bounds__(kOptThreads) sq_norm_kernel(const T* x, uint64_t n, float* out) {
  __shared__ float red[32];
  pdl_wait();
  pdl_trigger();
  constexpr uint64_t EPV = 16 / sizeof(T);
  float acc = 0.f;
  uint64_t done = 0;
  if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0) {
    const uint64_t nvec = n / EPV;
    const uint4* v = reinterpret_cast<const uint4*>(x);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3 * stride < nvec; i += 4 * stride) {
      const uint4 a = v[i], b = v[i + stride], c = v[i + 2 * stride], d = v[i + 3 * stride];
      acc += sq8<T>(a) + sq8<T>(b) + sq8<T>(c) + sq8<T>(d);
    }
    for (; i < nvec; i += stride) acc += sq8<T>(v[i]);
    done = nvec * EPV;
  }
  for (uint64_t i = done + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const float f = (float)x[i];
    acc += f * f;
  }
  acc = block_reduce<false>(acc, red);
  if (threadIdx.x == 0) atomicAdd(out, acc);
}

// ---------------------------------------------------------------- AdamW
// One pass over the shard: reads grad, master, m, v; writes master, m, v and the bf16
// working copy that the next all-gather sends out.  total_sq_norm (device scalar, may be
// null) holds the squared global gradient norm; the clip factor is derived on the device,
// so no host synchronisation sits between the norm all-reduce and the update.
template <typename G>
__global__ void __launch_bounds__(kOptThreads)
    adamw_kernel(float* __restrict__ master, float* __restrict__ m, float* __restrict__ v, const G* grad,
                 __nv_bfloat16* __restrict__ param, uint64_t n, AdamWArgs a, const float* total_sq_norm) {
  pdl_wait();
  pdl_trigger();
  float clip = 1.0f;
  if (total_sq_norm != nullptr && a.max_grad_norm > 0.f) {
    const float norm = sqrtf(*total_sq_norm) * a.grad_scale;
    clip = fminf(1.0f, a.max_grad_norm / (norm + 1e-6f));
  }
  const float gs = a.grad_scale * clip;
  auto update = [&](float g, float& p, float& mi, float& vi) {
    g *= gs;
    mi = a.beta1 * mi + (1.f - a.beta1) * g;
    vi = a.beta2 * vi + (1.f - a.beta2) * g * g;
    const float mhat = mi * a.bias1, vhat = vi * a.bias2;
    p = p * (1.f - a.lr * a.weight_decay) - a.lr * mhat / (sqrtf(vhat) + a.eps);
  };
  // Four elements per thread and iteration through 16-byte accesses (8 bytes for the bf16 sides),
  // two such groups in flight: the pass is pure streaming (28 bytes per parameter) and wants many
  // wide requests outstanding.  Pointers that are not 16-byte aligned take the scalar loop.
  uint64_t done = 0;
  const uintptr_t align = reinterpret_cast<uintptr_t>(master) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v) |
                          reinterpret_cast<uintptr_t>(grad) | reinterpret_cast<uintptr_t>(param);
  if ((align & 15u) == 0) {
    const uint64_t nvec = n / 4;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    float4* pm = reinterpret_cast<float4*>(master);
    float4* mm = reinterpret_cast<float4*>(m);
    float4* vv = reinterpret_cast<float4*>(v);
    auto load_g = [&](uint64_t i, float* g) {
      if constexpr (sizeof(G) == 2) {
        const uint2 q = __ldcs(reinterpret_cast<const uint2*>(grad) + i);
        g[0] = __uint_as_float(q.x << 16); g[1] = __uint_as_float(q.x & 0xffff0000u);
        g[2] = __uint_as_float(q.y << 16); g[3] = __uint_as_float(q.y & 0xffff0000u);
      } else {
        const float4 q = __ldcs(reinterpret_cast<const float4*>(grad) + i);
        g[0] = q.x; g[1] = q.y; g[2] = q.z; g[3] = q.w;
      }
    };
    auto one = [&](uint64_t i, const float* g, float4 p4, float4 m4, float4 v4) {
      update(g[0], p4.x, m4.x, v4.x);
      update(g[1], p4.y, m4.y, v4.y);
      update(g[2], p4.z, m4.z, v4.z);
      update(g[3], p4.w, m4.w, v4.w);
      __stcs(pm + i, p4);
      __stcs(mm + i, m4);
      __stcs(vv + i, v4);
      const __nv_bfloat162 lo = __floats2bfloat162_rn(p4.x, p4.y), hi = __floats2bfloat162_rn(p4.z, p4.w);
      uint2 o;
      o.x = *reinterpret_cast<const uint32_t*>(&lo);
      o.y = *reinterpret_cast<const uint32_t*>(&hi);
      reinterpret_cast<uint2*>(param)[i] = o;          // the working copy is read again soon: default caching
    };
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + stride < nvec; i += 2 * stride) {
      float g0[4], g1[4];
      load_g(i, g0);
      load_g(i + stride, g1);
      const float4 p0 = __ldcs(pm + i), m0 = __ldcs(mm + i), v0 = __ldcs(vv + i);
      const float4 p1 = __ldcs(pm + i + stride), m1 = __ldcs(mm + i + stride), v1 = __ldcs(vv + i + stride);
      one(i, g0, p0, m0, v0);
      one(i + stride, g1, p1, m1, v1);
    }
    for (; i < nvec; i += stride) {
      float g0[4];
      load_g(i, g0);
      one(i, g0, __ldcs(pm + i), __ldcs(mm + i), __ldcs(vv + i));
    }
    done = nvec * 4;
  }
  for (uint64_t i = done + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    float p = master[i], mi = m[i], vi = v[i];
    update((float)grad[i], p, mi, vi);
    master[i] = p;
    m[i] = mi;
    v[i] = vi;
    param[i] = __float2bfloat16_rn(p);
  }
}

// ---------------------------------------------------------------- softmax cross-entropy, fwd + bwd
// One CTA per row.  The row of logits is read from HBM once into shared memory and overwritten in place
// with d(loss)/d(logits) = (softmax - onehot) * grad_scale.  loss_sum accumulates the per-row losses: every
// CTA adds up its own rows, so the large sum is rounded once per CTA and not once per row.
//
// Every CTA walks over several rows, and the loop that forms the gradient of one row takes in the next one: per
// 16-byte vector, the load of the next row is issued, the vector of this row is turned into its gradient and stored, and
// then the new vector replaces it and joins the next row's running maximum and its sum of exponentials (rescaled when
// the maximum rises).  So loads, stores and both exponentials per element overlap all the time, a row meets the
// block's barriers only for its maximum and sum, and shared memory is each thread's own store (no other thread reads it).
// Bound by HBM (one read, one write) with the exponential unit close behind; two CTAs per SM at 50304 columns.
// Rows are taken from the last to the first: the product that wrote the logits finished with the last
// ones, which L2 still holds.  Measured against one row per CTA in three sweeps (calls back to back, buffers in turn):
// 2048 rows of 50304 (412 MB moved) 150 -> 92 us (4.5 TB/s, 0.68 of the copy rate), 64 rows 17.6 -> 9.2 us, 2048 rows of
// 1024 14.2 -> 5.6 us.  More warps with fewer registers (768 or 1024 threads) and 2 vectors in flight: no faster.
// The sum's error: a rescaling multiplies a thread's sum by another approximate exponential (2 units in its last
// place), and a thread sees about log(vectors) of them; over a row that stays below the rounding of its logarithm.  Measured
// against 64 bits, mean loss of 2048 rows of 50304: 1e-7 to 4e-7 (three sweeps and an atomic per row: 5e-7 to 1.3e-6), and
// the gradient's error is the same to six digits.
//
// e^(x - m): the difference is exact or nearly so, the exponential flushes results below 2^-126 to zero.  Keeping them costs
// three more instructions per element (2048 x 50304 91.8 -> 96.8 us) and changes neither error above.
__device__ __forceinline__ float exp_diff(float x, float m) { return ex2_hw((x - m) * 1.4426950408889634f); }

template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) ce_fwd_bwd_kernel(__nv_bfloat16* __restrict__ logits, const int64_t* targets,
                                                            float* loss_sum, int64_t rows, int vocab, int64_t row_stride,
                                                            float grad_scale, int64_t ignore_index, int* bad_targets) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint4* row_s = reinterpret_cast<uint4*>(smem_raw);
  __nv_bfloat16* tail_s = reinterpret_cast<__nv_bfloat16*>(smem_raw);
  __shared__ float red_m[2][THREADS / 32], red_s[2][THREADS / 32];
  __shared__ float loss_s;                                  // the losses of this CTA's rows
  if (threadIdx.x == 0) loss_s = 0.f;
  const int nvec = vocab >> 3;  // 8 bf16 = 16 bytes (row_stride is a multiple of 8)
  constexpr int nt = THREADS, nw = THREADS / 32, U = 4;     // U vectors in flight per thread
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float m = -INFINITY, s = 0.f;
  // m rises to the maximum of what comes in; while nothing above -inf has been seen the sum stays empty
  auto raise = [&](float top) {
    const float old = m;
    m = fmaxf(m, top);
    if (m != -INFINITY && old != m) s *= exp_diff(old, m);
    return m == -INFINITY ? 0.f : m;
  };
  auto top_of = [](const uint4& q) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    float top = -INFINITY;
#pragma unroll
    for (int e = 0; e < 4; ++e) top = fmaxf(top, fmaxf(__uint_as_float(w[e] << 16), __uint_as_float(w[e] & 0xffff0000u)));
    return top;
  };
  auto sum_of = [](const uint4& q, float mm) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    float a = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) a += exp_diff(__uint_as_float(w[e] << 16), mm) + exp_diff(__uint_as_float(w[e] & 0xffff0000u), mm);
    return a;
  };
  auto take = [&](const uint4& q) {
    const float mm = raise(top_of(q));
    s += sum_of(q, mm);
  };
  auto take_all = [&](const uint4 (&q)[U]) {
    float top = top_of(q[0]);
#pragma unroll
    for (int k = 1; k < U; ++k) top = fmaxf(top, top_of(q[k]));
    const float mm = raise(top);
#pragma unroll
    for (int k = 0; k < U; ++k) s += sum_of(q[k], mm);
  };
  const int64_t stride = gridDim.x;
  int64_t r = rows - 1 - (int64_t)blockIdx.x;
  {
    const __nv_bfloat16* first = logits + r * row_stride;
    int i = threadIdx.x;
    for (; i + (U - 1) * nt < nvec; i += U * nt) {
      uint4 q[U];
#pragma unroll
      for (int k = 0; k < U; ++k) q[k] = reinterpret_cast<const uint4*>(first)[i + k * nt];
#pragma unroll
      for (int k = 0; k < U; ++k) row_s[i + k * nt] = q[k];
      take_all(q);
    }
    for (; i < nvec; i += nt) {
      const uint4 q = reinterpret_cast<const uint4*>(first)[i];
      row_s[i] = q;
      take(q);
    }
    for (int c = (nvec << 3) + threadIdx.x; c < vocab; c += nt) {
      tail_s[c] = first[c];
      const float x = __bfloat162float(tail_s[c]);
      const float mm = raise(x);
      s += exp_diff(x, mm);
    }
  }
  for (int buf = 0; r >= 0; r -= stride, buf ^= 1) {
    __nv_bfloat16* row = logits + r * row_stride;
    const bool more = r >= stride;
    const __nv_bfloat16* next = row - stride * row_stride;
    const int64_t tgt = targets[r];
    // A target outside [0, vocab) that is not the ignore index would index past the row: such a row
    // counts as ignored (no loss, zero gradient) and is reported through *bad_targets, so a corrupt
    // label never becomes an out-of-bounds access.
    const bool out_of_range = tgt != ignore_index && (tgt < 0 || tgt >= (int64_t)vocab);
    const bool ignored = tgt == ignore_index || out_of_range;
    const int hot = ignored ? -8 : (int)tgt;                 // the column that loses grad_scale
    // ---- the row's maximum and sum: every thread's sum rescaled to the common maximum
    const float mw = warp_max(m);
    if (lane == 0) red_m[buf][warp] = mw;
    __syncthreads();
    float mx = -INFINITY;
    for (int w = 0; w < nw; ++w) mx = fmaxf(mx, red_m[buf][w]);
    // a thread that saw nothing above -inf has an empty (or NaN) sum, which needs no factor
    s = warp_sum(m == -INFINITY ? s : s * exp_diff(m, mx));
    if (lane == 0) red_s[buf][warp] = s;
    // the whole row lies in shared memory between these two barriers: nobody has begun to replace it
    float lt = 0.f;
    if (threadIdx.x == 0 && !ignored) lt = __bfloat162float(tail_s[hot]);
    __syncthreads();
    float sum = 0.f;
    for (int w = 0; w < nw; ++w) sum += red_s[buf][w];
    if (threadIdx.x == 0) {
      if (!ignored) loss_s += mx + logf(sum) - lt;
      if (out_of_range && bad_targets != nullptr) atomicAdd(bad_targets, 1);
    }
    const float inv = ignored ? 0.f : grad_scale / sum;
    auto grad = [&](int k, const uint4& q) {
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
      float f[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        f[2 * e] = exp_diff(__uint_as_float(w[e] << 16), mx) * inv;
        f[2 * e + 1] = exp_diff(__uint_as_float(w[e] & 0xffff0000u), mx) * inv;
      }
      if ((hot >> 3) == k) {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if ((hot & 7) == e) f[e] -= grad_scale;
      }
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
        o[e] = *reinterpret_cast<const uint32_t*>(&h);
      }
      reinterpret_cast<uint4*>(row)[k] = make_uint4(o[0], o[1], o[2], o[3]);
    };
    m = -INFINITY;
    s = 0.f;
    int i = threadIdx.x;
    for (; i + (U - 1) * nt < nvec; i += U * nt) {
      uint4 q[U];
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (more) q[k] = reinterpret_cast<const uint4*>(next)[i + k * nt];
#pragma unroll
      for (int k = 0; k < U; ++k) grad(i + k * nt, row_s[i + k * nt]);
      if (more) {
#pragma unroll
        for (int k = 0; k < U; ++k) row_s[i + k * nt] = q[k];
        take_all(q);
      }
    }
    for (; i < nvec; i += nt) {
      uint4 q = make_uint4(0u, 0u, 0u, 0u);
      if (more) q = reinterpret_cast<const uint4*>(next)[i];
      grad(i, row_s[i]);
      if (more) {
        row_s[i] = q;
        take(q);
      }
    }
    for (int c = (nvec << 3) + threadIdx.x; c < vocab; c += nt) {
      const float x = __bfloat162float(tail_s[c]);
      row[c] = __float2bfloat16_rn(exp_diff(x, mx) * inv - (c == hot ? grad_scale : 0.f));
      if (more) {
        tail_s[c] = next[c];
        const float y = __bfloat162float(tail_s[c]);
        const float mm = raise(y);
        s += exp_diff(y, mm);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) atomicAdd(loss_sum, loss_s);
}

int grid_for(uint64_t n, int threads, int per_thread) {
  uint64_t blocks = (n + (uint64_t)threads * per_thread - 1) / ((uint64_t)threads * per_thread);
  if (blocks < 1) blocks = 1;
  if (blocks > 148 * 8) blocks = 148 * 8;
  return (int)blocks;
}

}  // namespace

cudaError_t launch_sq_norm(const void* x, int dtype_is_bf16, uint64_t n, float* out, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const int grid = grid_for(n, kOptThreads, 16);
  if (dtype_is_bf16) return launch_pdl(sq_norm_kernel<__nv_bfloat16>, grid, kOptThreads, 0, s, (const __nv_bfloat16*)x, n, out);
  return launch_pdl(sq_norm_kernel<float>, grid, kOptThreads, 0, s, (const float*)x, n, out);
}

cudaError_t launch_adamw(float* master, float* m, float* v, const void* grad, int grad_is_bf16, void* param_bf16,
                         uint64_t n, const AdamWArgs& a, const float* total_sq_norm, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const int grid = grid_for(n, kOptThreads, 8);
  if (grad_is_bf16)
    return launch_pdl(adamw_kernel<__nv_bfloat16>, grid, kOptThreads, 0, s, master, m, v, (const __nv_bfloat16*)grad,
                      (__nv_bfloat16*)param_bf16, n, a, total_sq_norm);
  return launch_pdl(adamw_kernel<float>, grid, kOptThreads, 0, s, master, m, v, (const float*)grad, (__nv_bfloat16*)param_bf16, n,
                    a, total_sq_norm);
}

cudaError_t launch_ce_fwd_bwd(void* logits_bf16, const int64_t* targets, float* loss_sum, int64_t rows, int vocab,
                              int64_t row_stride, float grad_scale, int64_t ignore_index, int* bad_targets,
                              cudaStream_t s) {
  if (rows == 0) return cudaSuccess;
  const size_t smem = (size_t)vocab * sizeof(__nv_bfloat16);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;   // the row must fit into shared memory
  // the shared-memory limit is a per-device attribute of the function
  static bool configured[64] = {false};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    e = cudaFuncSetAttribute(ce_fwd_bwd_kernel<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  // short rows take smaller CTAs, of which more fit on an SM (1 KiB of shared memory per CTA is the system's)
  const int threads = vocab >= 16384 ? 512 : vocab >= 4096 ? 256 : 128;
  const int64_t per_sm = std::max<int64_t>(1, std::min<int64_t>(1024 / threads, (int64_t)(228 * 1024 / (smem + 1280))));
  const unsigned grid = (unsigned)std::min<int64_t>(rows, 148 * per_sm);
  auto* l = (__nv_bfloat16*)logits_bf16;
  if (threads == 512) return launch_pdl(ce_fwd_bwd_kernel<512>, grid, 512, smem, s, l, targets, loss_sum, rows, vocab, row_stride, grad_scale, ignore_index, bad_targets);
  if (threads == 256) return launch_pdl(ce_fwd_bwd_kernel<256>, grid, 256, smem, s, l, targets, loss_sum, rows, vocab, row_stride, grad_scale, ignore_index, bad_targets);
  return launch_pdl(ce_fwd_bwd_kernel<128>, grid, 128, smem, s, l, targets, loss_sum, rows, vocab, row_stride, grad_scale, ignore_index, bad_targets);
}

}  // namespace pccl

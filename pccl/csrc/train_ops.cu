// Memory-bound training kernels of the GPT forward and backward pass, each one pass over the
// activations: column sums (bias gradients), GELU forward, GELU backward fused with the
// column sum of its result, layer norm fused with the residual add in front of it, and
// layer-norm backward with its weight/bias gradients and the residual gradient added in.
//
// The reference has no model code; these serve the in-repo ZeRO-3 engine, where the stock
// framework kernels for the same jobs cost about a sixth of the step.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "act.cuh"
#include "optim.h"
#include "pdl.cuh"

namespace pccl {

namespace {

// ---------------------------------------------------------------- column sum
// out[c] = sum_r X[r, c]; X is [T, N] bf16 row-major with N % 8 == 0.  A block covers 256
// columns (a warp reads 512 contiguous bytes of one row) in eight row lanes, one per warp, and one slice of the
// rows; the last block to finish a column tile adds the slices' fp32 partial sums and writes bf16.  That
// last sum is a chain of loads from one SM at the end of everything, so the slices are few (col_sum_row_splits) and
// each thread keeps four of them in flight (more would cost the main loop its fourth block per SM).  Measured against 512-column tiles and up to 296 slices: 4096 x 1024
// 18.8 -> 5.6 us; GELU form 4096 x 4096 26.4 -> 20.4 us, with its arithmetic in pairs of elements.
// GELU form: X is the gradient of the GELU's output and U its input; the kernel writes
// DU = X * gelu'(U) and sums the columns of DU (as rounded to bf16), the bias gradient of
// the linear layer in front of the GELU.
// Concatenating form: the columns are those of three [T, N/3] matrices side by side (the
// gradients of q, k and v); the kernel writes the [T, N] concatenation to DU while it sums.
constexpr int kColTile = 256, kRowLanes = 8;
enum ColMode { kColSum = 0, kColGelu = 1, kColCat3 = 2 };

template <int MODE>
__device__ __forceinline__ void col_item(const uint4& q, const uint4& uq, __nv_bfloat16* DU, int64_t off, F2 (&acc)[4]) {
  if (MODE == kColGelu) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w}, uw[4] = {uq.x, uq.y, uq.z, uq.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      // the clamp of gelu_tanh_grad, on the packed pair (as there, NaN goes to a bound)
      __nv_bfloat162 u = *reinterpret_cast<const __nv_bfloat162*>(&uw[e]);
      u = __hmin2(__hmax2(u, __float2bfloat162_rn(-20.f)), __float2bfloat162_rn(20.f));
      float a, b;
      split(unpack2(w[e]) * gelu_tanh_grad2(unpack2(*reinterpret_cast<const uint32_t*>(&u))), a, b);
      const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);     // one rounding; the sums are of the rounded values
      o[e] = *reinterpret_cast<const uint32_t*>(&h);
      acc[e] = acc[e] + unpack2(o[e]);
    }
    *reinterpret_cast<uint4*>(DU + off) = make_uint4(o[0], o[1], o[2], o[3]);
    return;
  }
  if (MODE == kColCat3) *reinterpret_cast<uint4*>(DU + off) = q;
  acc[0] = acc[0] + unpack2(q.x);
  acc[1] = acc[1] + unpack2(q.y);
  acc[2] = acc[2] + unpack2(q.z);
  acc[3] = acc[3] + unpack2(q.w);
}

template <int MODE>
__global__ void __launch_bounds__(256, 4) col_sum_kernel(const __nv_bfloat16* X, int64_t T, int N,
                                                      __nv_bfloat16* __restrict__ out, float* __restrict__ partial,
                                                      int* __restrict__ counters, const __nv_bfloat16* U,
                                                      __nv_bfloat16* __restrict__ DU, const __nv_bfloat16* X2) {
  __shared__ __align__(16) float red[kRowLanes][kColTile];
  __shared__ int s_last;
  pdl_wait();
  pdl_trigger();
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int col_base = blockIdx.x * kColTile;
  const int col = col_base + tx * 8;
  const int R = gridDim.y;
  const int64_t rows_per = (T + R - 1) / R;
  const int64_t r0 = (int64_t)blockIdx.y * rows_per;
  const int64_t r1 = r0 + rows_per < T ? r0 + rows_per : T;
  F2 acc[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) acc[e] = f2(0.f);
  if (col < N) {
    // where this thread's 8 columns come from: X itself, or one of the three sources
    const __nv_bfloat16* src = X + col;
    int64_t ld = N;
    if (MODE == kColCat3) {
      const int w = N / 3, which = col / w;
      src = (which == 0 ? X : which == 1 ? U : X2) + (col - which * w);
      ld = w;
    }
    int64_t r = r0 + ty;
    for (; r + 3 * kRowLanes < r1; r += 4 * kRowLanes) {
      uint4 q[4], uq[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        q[k] = *reinterpret_cast<const uint4*>(src + (r + k * kRowLanes) * ld);
        uq[k] = MODE == kColGelu ? *reinterpret_cast<const uint4*>(U + (r + k * kRowLanes) * N + col) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) col_item<MODE>(q[k], uq[k], DU, (r + k * kRowLanes) * N + col, acc);
    }
    for (; r < r1; r += kRowLanes) {
      const uint4 q = *reinterpret_cast<const uint4*>(src + r * ld);
      const uint4 uq = MODE == kColGelu ? *reinterpret_cast<const uint4*>(U + r * N + col) : make_uint4(0, 0, 0, 0);
      col_item<MODE>(q, uq, DU, r * N + col, acc);
    }
  }
  // the eight row lanes' sums, column by column (256 threads, 256 columns)
  auto combine = [&]() {
#pragma unroll
    for (int e = 0; e < 4; ++e) split(acc[e], red[ty][tx * 8 + 2 * e], red[ty][tx * 8 + 2 * e + 1]);
    __syncthreads();
    float a = red[0][threadIdx.x];
#pragma unroll
    for (int l = 1; l < kRowLanes; ++l) a += red[l][threadIdx.x];
    return a;
  };
  const int mine = col_base + threadIdx.x;
  const float part = combine();
  if (mine < N) __stcg(partial + (int64_t)blockIdx.y * N + mine, part);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(counters + blockIdx.x, 1) == R - 1;
  __syncthreads();
  if (s_last) {
    __threadfence();
    // the row lanes split the slices; every thread adds 8 columns of its share, four slices at a time
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = f2(0.f);
    if (col < N) {
      for (int y0 = ty; y0 < R; y0 += 4 * kRowLanes) {
        float4 v[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int y = y0 + k * kRowLanes;
          const float* src = partial + (int64_t)y * N + col;
          v[2 * k] = v[2 * k + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (y < R) {
            v[2 * k] = __ldcg(reinterpret_cast<const float4*>(src));
            v[2 * k + 1] = __ldcg(reinterpret_cast<const float4*>(src + 4));
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          acc[0] = acc[0] + f2(v[2 * k].x, v[2 * k].y);
          acc[1] = acc[1] + f2(v[2 * k].z, v[2 * k].w);
          acc[2] = acc[2] + f2(v[2 * k + 1].x, v[2 * k + 1].y);
          acc[3] = acc[3] + f2(v[2 * k + 1].z, v[2 * k + 1].w);
        }
      }
    }
    const float total = combine();
    if (mine < N) out[mine] = __float2bfloat16_rn(total);
    if (threadIdx.x == 0) counters[blockIdx.x] = 0;   // ready for the next call
  }
}

// ---------------------------------------------------------------- layer-norm backward
// One pass over dy and x:  dx = rstd * (g - mean(g) - xhat * mean(g * xhat)),  g = dy * gamma,
// and per-block partial sums of dgamma = sum_r dy * xhat, dbeta = sum_r dy.  With `resid` the gradient that
// flows around the layer norm (the residual connection) is added to dx in the same pass (in fp32, before the one
// rounding); with `pdx` the kernel also sums the columns of dx (the bias gradient of the linear layer whose output
// gradient dx is).  A block leaves one partial row per array, and a second small kernel adds the blocks' partials.
//
// D / 8 threads work on one row (one 16-byte vector each), so the three column accumulators take 24 registers and
// 16 warps of 128 registers fit on an SM for every width.  A block takes two rows at a time, and the loads of
// the next two are issued before the reductions of the current ones: with one buffer of four rows instead, the memory
// system waits while the block reduces.  One barrier per two rows (the row sums are double-buffered); the
// arithmetic goes two elements per instruction.  Bound by HBM at many rows, by the chain of row reductions at few.
// Measured with residual and column sums, whole calls (the kernel that adds the partials among them), against 128 threads per
// row (256 at 2048 columns) and four rows in one buffer (us): 8192 rows of 1024 24.1 -> 20.0, of 2048 38.6 -> 34.6, of 4096
// 82.5 -> 72.8 (3.7 TB/s); 1501 rows of 4096 26.6 -> 22.2.
// AHEAD false: RB rows at a time, nothing in flight while they are reduced.  At 2048 columns with a residual
// gradient two blocks share an SM and cover for one another, and three rows of loads at once are worth more than two rows ahead:
// calls with residual and column sums, ahead / three rows (us): 500 rows 9.1 / 10.0, 1501 13.2 / 13.2, 4096 21.9 / 21.4,
// 8192 37.4 / 35.0, 32768 116.5 / 103.6.  (One block per SM at 4096 columns, four at 1024: ahead is the better form.)
template <int D, int RB, bool AHEAD>
__global__ void __launch_bounds__(D / 8, 4096 / D)
    ln_bwd_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* x, const float* mean, const float* rstd,
                  const __nv_bfloat16* gamma, const __nv_bfloat16* resid,
                  __nv_bfloat16* __restrict__ dx, float* __restrict__ pgamma, float* __restrict__ pbeta, float* __restrict__ pdx,
                  int64_t T) {
  pdl_wait();
  pdl_trigger();
  constexpr int NW = D / 256;
  __shared__ float2 red[2][RB][NW];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  F2 g[4], dgam[4], dbet[4], dxs[4];
  {
    const uint4 q = *reinterpret_cast<const uint4*>(gamma + t * 8);
    g[0] = unpack2(q.x), g[1] = unpack2(q.y), g[2] = unpack2(q.z), g[3] = unpack2(q.w);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) dgam[e] = dbet[e] = dxs[e] = f2(0.f);
  struct Rows {
    uint4 dy[RB], x[RB], r[RB];
    float mu[RB], rs[RB];
  };
  auto load = [&](Rows& b, int64_t base) {                  // rows past the end hold zeros
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int64_t r = base + j;
      b.mu[j] = b.rs[j] = 0.f;
      b.dy[j] = b.x[j] = b.r[j] = make_uint4(0, 0, 0, 0);
      if (r < T) {
        const int64_t off = r * D + t * 8;
        b.dy[j] = *reinterpret_cast<const uint4*>(dy + off);
        b.x[j] = *reinterpret_cast<const uint4*>(x + off);
        if (resid != nullptr) b.r[j] = *reinterpret_cast<const uint4*>(resid + off);
        b.mu[j] = mean[r];
        b.rs[j] = rstd[r];
      }
    }
  };
  constexpr float inv_d = 1.0f / (float)D;
  const int64_t step = (int64_t)RB * gridDim.x;
  Rows cur, nxt;
  if (AHEAD) load(cur, (int64_t)blockIdx.x * RB);
  int buf = 0;
  for (int64_t base = (int64_t)blockIdx.x * RB; base < T; base += step, buf ^= 1) {
    if (AHEAD) load(nxt, base + step);
    else load(cur, base);
    // ---- row sums and the weight/bias gradient sums
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const uint32_t aw[4] = {cur.dy[j].x, cur.dy[j].y, cur.dy[j].z, cur.dy[j].w}, bw[4] = {cur.x[j].x, cur.x[j].y, cur.x[j].z, cur.x[j].w};
      const F2 rs = f2(cur.rs[j]), nmr = f2(-cur.mu[j] * cur.rs[j]);
      F2 t1 = f2(0.f), t2 = f2(0.f);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const F2 a = unpack2(aw[e]), xhat = fma2(unpack2(bw[e]), rs, nmr), gg = a * g[e];
        t1 = t1 + gg;
        t2 = fma2(gg, xhat, t2);
        dgam[e] = fma2(a, xhat, dgam[e]);
        dbet[e] = dbet[e] + a;
      }
      float s1, s2, hi;
      split(t1, s1, hi);
      s1 += hi;
      split(t2, s2, hi);
      s2 += hi;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
      }
      if (lane == 0) red[buf][j][warp] = make_float2(s1, s2);
    }
    __syncthreads();
    // ---- dx = rs * (dy * gamma - m1 - xhat * m2) = dy * (gamma * rs) - x * c2 + c0
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const int64_t r = base + j;
      if (r < T) {
        float m1 = 0.f, m2 = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
          m1 += red[buf][j][w].x;
          m2 += red[buf][j][w].y;
        }
        m1 *= inv_d;
        m2 *= inv_d;
        const float c2 = cur.rs[j] * cur.rs[j] * m2;
        const F2 c0 = f2(fmaf(cur.mu[j], c2, -m1 * cur.rs[j])), nc2 = f2(-c2), rs = f2(cur.rs[j]);
        const uint32_t aw[4] = {cur.dy[j].x, cur.dy[j].y, cur.dy[j].z, cur.dy[j].w}, bw[4] = {cur.x[j].x, cur.x[j].y, cur.x[j].z, cur.x[j].w};
        const uint32_t qw[4] = {cur.r[j].x, cur.r[j].y, cur.r[j].z, cur.r[j].w};
        uint32_t ow[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          F2 o = fma2(unpack2(aw[e]), g[e] * rs, fma2(unpack2(bw[e]), nc2, c0));
          if (resid != nullptr) o = o + unpack2(qw[e]);                        // one rounding, at the store
          dxs[e] = dxs[e] + o;
          float lo, hi;
          split(o, lo, hi);
          const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
          ow[e] = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(dx + r * D + t * 8) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
      }
    }
    if (AHEAD) cur = nxt;
  }
  auto put = [&](float* row, const F2 (&acc)[4]) {
    float v[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) split(acc[e], v[2 * e], v[2 * e + 1]);
    float4* o = reinterpret_cast<float4*>(row + (int64_t)blockIdx.x * D + t * 8);
    o[0] = make_float4(v[0], v[1], v[2], v[3]);
    o[1] = make_float4(v[4], v[5], v[6], v[7]);
  };
  put(pgamma, dgam);
  put(pbeta, dbet);
  if (pdx != nullptr) put(pdx, dxs);
}

// Adds the per-block partial sums of up to three arrays (blockIdx.y picks the array): a block
// owns 32 columns, its 32 warps split the partials and keep four rows in flight each (up to 592 rows: five
// rounds; with 8 warps the rounds were what this kernel took).
struct LnBwdFinalizeArgs {
  const float* part[3];
  __nv_bfloat16* out[3];
};

__global__ void __launch_bounds__(1024) ln_bwd_finalize_kernel(LnBwdFinalizeArgs f, int nparts, int d) {
  pdl_wait();
  pdl_trigger();
  __shared__ float sa[32][33];
  const float* part = f.part[blockIdx.y];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;                // d is a multiple of 32
  float a = 0.f;
  for (int p = w; p < nparts; p += 128) {
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = p + 32 * k < nparts ? __ldcg(part + (int64_t)(p + 32 * k) * d + c) : 0.f;
    a += (v[0] + v[1]) + (v[2] + v[3]);
  }
  sa[w][lane] = a;
  __syncthreads();
  // warp w adds column w's 32 sums
  a = sa[lane][w];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if (lane == 0) f.out[blockIdx.y][blockIdx.x * 32 + w] = __float2bfloat16_rn(a);
}

// ---------------------------------------------------------------- GELU forward
__device__ __forceinline__ uint4 gelu8(const uint4& q) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  uint32_t o[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float a, b;
    split(gelu_tanh2(unpack2(w[e])), a, b);
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    o[e] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}
__global__ void __launch_bounds__(256) gelu_fwd_kernel(const uint4* in, uint4* __restrict__ out, int64_t nvec) {
  pdl_wait();
  pdl_trigger();
  const int64_t stride = (int64_t)gridDim.x * 256;
  int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  for (; i + 3 * stride < nvec; i += 4 * stride) {
    uint4 q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) q[k] = in[i + k * stride];
#pragma unroll
    for (int k = 0; k < 4; ++k) out[i + k * stride] = gelu8(q[k]);
  }
  for (; i < nvec; i += stride) out[i] = gelu8(in[i]);
}

// ---------------------------------------------------------------- residual add + layer norm
// With `branch` the row is x + branch, rounded to bf16 and written back over `branch` (it becomes the new residual
// stream); the statistics and the normalised output are taken from the rounded values, which is what the
// backward pass reads.  Writes y = (v - mean) * rstd * gamma + beta, mean and rstd (biased variance, from the
// deviations).
//
// A warp works on one row (two warps for 4096 columns) and keeps it as it is stored, eight 16-byte vectors per
// lane: all its loads are in flight at once, the row sums need no block barrier, and the packed row takes 32 registers.
// Bound by HBM.  Measured with branch against 128 threads per row, fp32 in registers and four barriers (us): 8192 rows of
// 1024 17.1 -> 11.4, of 2048 29.3 -> 21.9, of 4096 51.8 -> 43.4 (6.2 TB/s, 0.94 of the copy rate); 1501 rows of 4096 14.5 -> 9.9.
constexpr int kLnFwdWarps = 4;      // per block: small ones, so that few rows still reach every SM
template <int D>
__global__ void __launch_bounds__(32 * kLnFwdWarps, 6) ln_fwd_kernel(const __nv_bfloat16* x, __nv_bfloat16* branch,
                                                        const __nv_bfloat16* gamma, const __nv_bfloat16* beta,
                                                        __nv_bfloat16* __restrict__ y,
                                                        float* __restrict__ mean, float* __restrict__ rstd, int64_t T, float eps) {
  pdl_wait();
  pdl_trigger();
  constexpr int WPR = D > 2048 ? 2 : 1;                // warps per row
  constexpr int NV = D / (256 * WPR);                  // vectors per lane
  __shared__ float part[2][kLnFwdWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t r = ((int64_t)blockIdx.x * kLnFwdWarps + warp) / WPR;
  const bool live = r < T;                             // a block's last rows may not exist (the block meets at barriers if WPR > 1)
  const int c0 = ((warp % WPR) * 32 + lane) * 8;       // first column of vector k: c0 + k * 256 * WPR
  constexpr float inv_d = 1.0f / (float)D;
  uint4 v[NV];
  float s = 0.f;
  if (live) {
    const int64_t off = r * D + c0;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = *reinterpret_cast<const uint4*>(x + off + k * 256 * WPR);
    if (branch != nullptr) {
      uint4 b[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) b[k] = *reinterpret_cast<const uint4*>(branch + off + k * 256 * WPR);
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        uint32_t vw[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
        const uint32_t bw[4] = {b[k].x, b[k].y, b[k].z, b[k].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float lo, hi;
          split(unpack2(vw[e]) + unpack2(bw[e]), lo, hi);
          const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
          vw[e] = *reinterpret_cast<const uint32_t*>(&h);
        }
        v[k] = make_uint4(vw[0], vw[1], vw[2], vw[3]);
        *reinterpret_cast<uint4*>(branch + off + k * 256 * WPR) = v[k];
      }
    }
    F2 a = f2(0.f);
#pragma unroll
    for (int k = 0; k < NV; ++k) a = a + ((unpack2(v[k].x) + unpack2(v[k].y)) + (unpack2(v[k].z) + unpack2(v[k].w)));
    float hi;
    split(a, s, hi);
    s += hi;
  }
  auto row_sum = [&](float a, int which) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (WPR > 1) {
      if (lane == 0) part[which][warp] = a;
      __syncthreads();
      a = part[which][warp & ~1] + part[which][warp | 1];
    }
    return a;
  };
  const float mu = row_sum(s, 0) * inv_d;
  F2 dev = f2(0.f);
  const F2 nmu = f2(-mu);
  if (live) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const uint32_t vw[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const F2 c = unpack2(vw[e]) + nmu;
        dev = fma2(c, c, dev);
      }
    }
  }
  float s2, hi2;
  split(dev, s2, hi2);
  const float rs = rsqrtf(row_sum(s2 + hi2, 1) * inv_d + eps);
  if (!live) return;
  const F2 rs2 = f2(rs);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int c = c0 + k * 256 * WPR;
    const uint4 gq = *reinterpret_cast<const uint4*>(gamma + c), bq = *reinterpret_cast<const uint4*>(beta + c);
    const uint32_t vw[4] = {v[k].x, v[k].y, v[k].z, v[k].w}, gw[4] = {gq.x, gq.y, gq.z, gq.w}, bw[4] = {bq.x, bq.y, bq.z, bq.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float lo, hi;
      split(fma2((unpack2(vw[e]) + nmu) * rs2, unpack2(gw[e]), unpack2(bw[e])), lo, hi);
      const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
      o[e] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(y + r * D + c) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  if (lane == 0 && warp % WPR == 0) {
    mean[r] = mu;
    rstd[r] = rs;
  }
}

}  // namespace

int col_sum_row_splits(int64_t T, int N) {
  const int tiles = (N + kColTile - 1) / kColTile;
  int R = 148 * 4 / tiles;                                     // four blocks per SM and no second wave
  // The last sum in two rounds of loads, unless the main loop is long enough to want every SM: 65536 rows of 1024, 64
  // slices / 148 (us): GELU form 102.8 / 72.5, plain 29.1 / 26.1; 8192 rows of 1024 plain 8.4 / 9.6, 16384 11.2 / 11.5.
  if (T <= 16384 && R > 8 * kRowLanes) R = 8 * kRowLanes;
  const int64_t max_r = (T + 2 * kRowLanes - 1) / (2 * kRowLanes);
  if (R > max_r) R = (int)max_r;
  if (R < 1) R = 1;
  return R;
}

cudaError_t launch_col_sum(const void* X, int64_t T, int N, void* out, float* partial, int* counters, int R,
                           cudaStream_t s) {
  if (T <= 0 || N <= 0) return cudaSuccess;
  if (N % 8 != 0) return cudaErrorInvalidValue;
  dim3 grid((N + kColTile - 1) / kColTile, R);
  return launch_pdl(col_sum_kernel<kColSum>, grid, 256, 0, s, (const __nv_bfloat16*)X, T, N, (__nv_bfloat16*)out, partial, counters, nullptr,
                                               nullptr, nullptr);
}

cudaError_t launch_gelu_bwd_col_sum(const void* dg, const void* u, void* du, int64_t T, int N, void* out, float* partial,
                                    int* counters, int R, cudaStream_t s) {
  if (T <= 0 || N <= 0) return cudaSuccess;
  if (N % 8 != 0) return cudaErrorInvalidValue;
  dim3 grid((N + kColTile - 1) / kColTile, R);
  return launch_pdl(col_sum_kernel<kColGelu>, grid, 256, 0, s, (const __nv_bfloat16*)dg, T, N, (__nv_bfloat16*)out, partial, counters,
                                                (const __nv_bfloat16*)u, (__nv_bfloat16*)du, nullptr);
}

cudaError_t launch_cat3_col_sum(const void* a, const void* b, const void* c, void* cat, int64_t T, int N, void* out,
                                float* partial, int* counters, int R, cudaStream_t s) {
  if (T <= 0 || N <= 0) return cudaSuccess;
  if (N % 24 != 0) return cudaErrorInvalidValue;          // three sources of a multiple of 8 columns each
  dim3 grid((N + kColTile - 1) / kColTile, R);
  return launch_pdl(col_sum_kernel<kColCat3>, grid, 256, 0, s, (const __nv_bfloat16*)a, T, N, (__nv_bfloat16*)out, partial, counters,
                                                (const __nv_bfloat16*)b, (__nv_bfloat16*)cat, (const __nv_bfloat16*)c);
}

cudaError_t launch_gelu_fwd(const void* in, void* out, int64_t n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (n % 8 != 0) return cudaErrorInvalidValue;
  const int64_t nvec = n / 8;
  int64_t blocks = (nvec + 256 * 4 - 1) / (256 * 4);
  if (blocks > 148 * 8) blocks = 148 * 8;
  return launch_pdl(gelu_fwd_kernel, (int)blocks, 256, 0, s, (const uint4*)in, (uint4*)out, nvec);
}

cudaError_t launch_ln_fwd(const void* x, void* branch, const void* gamma, const void* beta, void* y, float* mean, float* rstd,
                          int64_t T, int d, float eps, cudaStream_t s) {
  if (T <= 0) return cudaSuccess;
  const int64_t blocks = (T * (d > 2048 ? 2 : 1) + kLnFwdWarps - 1) / kLnFwdWarps;
  auto* X = (const __nv_bfloat16*)x;
  auto* B = (__nv_bfloat16*)branch;
  auto* G = (const __nv_bfloat16*)gamma;
  auto* Be = (const __nv_bfloat16*)beta;
  auto* Y = (__nv_bfloat16*)y;
  cudaError_t e = cudaSuccess;
  switch (d / 128) {
    case 8: e = launch_pdl(ln_fwd_kernel<1024>, (unsigned)blocks, 32 * kLnFwdWarps, 0, s, X, B, G, Be, Y, mean, rstd, T, eps); break;
    case 16: e = launch_pdl(ln_fwd_kernel<2048>, (unsigned)blocks, 32 * kLnFwdWarps, 0, s, X, B, G, Be, Y, mean, rstd, T, eps); break;
    case 32: e = launch_pdl(ln_fwd_kernel<4096>, (unsigned)blocks, 32 * kLnFwdWarps, 0, s, X, B, G, Be, Y, mean, rstd, T, eps); break;
    default: return cudaErrorInvalidValue;
  }
  return e;
}

// Blocks of the widest grid: 4096 / d per SM, each leaves one partial row of d floats per array.
int ln_bwd_blocks(int d) { return 148 * (4096 / d); }

cudaError_t launch_ln_bwd(const void* dy, const void* x, const float* mean, const float* rstd, const void* gamma, void* dx,
                          const void* resid, void* dgamma, void* dbeta, void* dx_col_sum, float* scratch, int64_t T, int d,
                          cudaStream_t s) {
  if (T <= 0) return cudaSuccess;
  int blocks = ln_bwd_blocks(d);
  if ((int64_t)blocks * 2 > T) blocks = (int)((T + 1) / 2);                 // two rows per block and iteration
  auto* DY = (const __nv_bfloat16*)dy;
  auto* X = (const __nv_bfloat16*)x;
  auto* G = (const __nv_bfloat16*)gamma;
  auto* RS = (const __nv_bfloat16*)resid;
  auto* DX = (__nv_bfloat16*)dx;
  float* pgamma = scratch;
  float* pbeta = scratch + (int64_t)ln_bwd_blocks(d) * d;
  float* pdx = dx_col_sum != nullptr ? scratch + 2 * (int64_t)ln_bwd_blocks(d) * d : nullptr;
  auto run = [&](auto* kernel) { return launch_pdl(kernel, blocks, d / 8, 0, s, DY, X, mean, rstd, G, RS, DX, pgamma, pbeta, pdx, T); };
  cudaError_t e = cudaSuccess;
  switch (d / 128) {
    case 8: e = run(ln_bwd_kernel<1024, 2, true>); break;
    case 16:
      // the comment at the kernel has both sides of this line
      e = resid != nullptr && T >= 4096 ? run(ln_bwd_kernel<2048, 3, false>) : run(ln_bwd_kernel<2048, 2, true>);
      break;
    case 32: e = run(ln_bwd_kernel<4096, 2, true>); break;
    default: return cudaErrorInvalidValue;
  }
  if (e != cudaSuccess) return e;
  LnBwdFinalizeArgs f;
  f.part[0] = pgamma, f.part[1] = pbeta, f.part[2] = pdx;
  f.out[0] = (__nv_bfloat16*)dgamma, f.out[1] = (__nv_bfloat16*)dbeta, f.out[2] = (__nv_bfloat16*)dx_col_sum;
  return launch_pdl(ln_bwd_finalize_kernel, dim3((d + 31) / 32, pdx != nullptr ? 3 : 2), 1024, 0, s, f, blocks, d);
}

}  // namespace pccl

// Memory-bound kernels of the training step, written for sm_100a: fused dropout+residual+LayerNorm
// (and RMSNorm), softmax cross-entropy (loss and logit gradient in one pass over the row), rotated
// embedding gather/scatter, short-sequence causal attention, column sums for bias gradients,
// multi-tensor Adam(W) with value clipping, and small elementwise helpers.
// All tensors are bf16 unless stated; statistics and reductions are fp32.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <algorithm>
#include <string>
#include <cooperative_groups.h>
#include "common.cuh"
#include "launch.h"
#include "kernels.h"

using namespace rtp;

namespace {
thread_local std::string k_err;
int kfail(const char* what, cudaError_t e) {
  k_err = std::string(what) + ": " + cudaGetErrorString(e);
  return -1;
}
#define LAUNCH_CHECK(name)                                 \
  do {                                                     \
    cudaError_t e__ = cudaGetLastError();                  \
    if (e__ != cudaSuccess) return kfail(name, e__);       \
  } while (0)

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
// block-wide sum over up to 1024 threads; `red` is a 32-float smem scratch
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = (threadIdx.x < nw) ? red[threadIdx.x] : 0.f;
  if (w == 0) t = warp_sum(t);
  if (threadIdx.x == 0) red[0] = t;
  __syncthreads();
  return red[0];
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = (threadIdx.x < nw) ? red[threadIdx.x] : -INFINITY;
  if (w == 0) t = warp_max(t);
  if (threadIdx.x == 0) red[0] = t;
  __syncthreads();
  return red[0];
}
__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  f[0] = bf16_lo(u.x); f[1] = bf16_hi(u.x); f[2] = bf16_lo(u.y); f[3] = bf16_hi(u.y);
  f[4] = bf16_lo(u.z); f[5] = bf16_hi(u.z); f[6] = bf16_lo(u.w); f[7] = bf16_hi(u.w);
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}
// dropout keep flags for 8 consecutive elements starting at e (e % 8 == 0)
__device__ __forceinline__ void keep8(uint64_t seed, uint64_t offset, uint64_t e, uint32_t thresh, bool* k) {
  uint4 r0 = philox4x32(seed, offset, e >> 2), r1 = philox4x32(seed, offset, (e >> 2) + 1);
  k[0] = r0.x >= thresh; k[1] = r0.y >= thresh; k[2] = r0.z >= thresh; k[3] = r0.w >= thresh;
  k[4] = r1.x >= thresh; k[5] = r1.y >= thresh; k[6] = r1.z >= thresh; k[7] = r1.w >= thresh;
}
uint32_t host_thresh(float p) {
  if (p <= 0.f) return 0;
  double t = (double)p * 4294967296.0;
  if (t > 4294967295.0) t = 4294967295.0;
  return (uint32_t)t;
}

// ------------------------------------------------------------------------------------------------
// h = x + dropout(sub);  y = norm(h) * gamma (+ beta).  rms = 0: LayerNorm, 1: RMSNorm.
// One block of T threads per row; the row lives in registers (NG groups of 8 columns per thread, D <= 8 T NG), so
// global memory is touched exactly once per tensor.  Saves h (bf16) and the row statistics for backward.
//
// A block keeps the next row's words in flight while it reduces the current one, and a reduction is one barrier (its
// scratch alternates).  D <= 1024 takes 128 threads a row: seven blocks fit on an SM, so that the 1024 rows of a small
// training step are one wave.  Wider rows take 256; 128 threads with two groups of columns each were slower at every size
// (RMSNorm of 256 x 2048 2.8 us, 256 threads 2.3; 8192 x 2048 19.3 and 17.1).  Microseconds before and after: 650 x 768
// with residual 4.0 -> 2.3, 8192 x 2048 21.5 -> 17, 4096 x 5120 (RMSNorm) 35 -> 17, 3000 x 4096 23 -> 12; 1024 x 2048 with
// residual and dropout stays at 6.2.
// ------------------------------------------------------------------------------------------------
// Sums N values of every thread over its group of T threads (the block is G groups): `red` holds 2 x G x T / 32 x N floats,
// `turn` alternates between its halves.
template <int T, int N, int G = 1>
__device__ __forceinline__ void block_sum_n(float (&v)[N], float* red, int turn) {
  constexpr int W = T / 32;
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) % W;
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = warp_sum(v[i]);
  if (W == 1) return;
  float* mine = red + (turn * G + threadIdx.x / T) * (W * N);
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < N; ++i) mine[w * N + i] = v[i];
  }
  __syncthreads();
  // the warps' sums in the order of a butterfly: halves first
#pragma unroll
  for (int i = 0; i < N; ++i) {
    float t[W];
#pragma unroll
    for (int k = 0; k < W; ++k) t[k] = mine[k * N + i];
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < o; ++k) t[k] += t[k + o];
    v[i] = t[0];
  }
}

template <int T, int NG>
__global__ void __launch_bounds__(T, T == 128 ? 7 : NG == 1 ? 4 : 2) norm_fwd_kernel(
    const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ sub, const __nv_bfloat16* __restrict__ gamma,
    const __nv_bfloat16* __restrict__ beta, __nv_bfloat16* __restrict__ h_out, __nv_bfloat16* __restrict__ y,
    float* __restrict__ mean_out, float* __restrict__ rstd_out, int M, int D, float eps, int rms, uint32_t thresh,
    float drop_scale, uint64_t seed, uint64_t offset, const unsigned long long* __restrict__ step_ptr) {
  pdl_prologue();
  __shared__ float red[2 * (T / 32)];
  if (step_ptr) offset += __ldg(step_ptr) * 65536ull;
  const int c0 = threadIdx.x * 8;
  uint4 nx[NG], ns[NG], g[NG], bt[NG];
  auto fetch = [&](int row) {
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      const int c = q * T * 8 + c0;
      if (c < D) {
        nx[q] = __ldcs(reinterpret_cast<const uint4*>(x + (size_t)row * D + c));
        if (sub) ns[q] = __ldcs(reinterpret_cast<const uint4*>(sub + (size_t)row * D + c));
      }
    }
  };
  if ((int)blockIdx.x < M) fetch(blockIdx.x);
#pragma unroll
  for (int q = 0; q < NG; ++q) {
    const int c = q * T * 8 + c0;
    g[q] = bt[q] = make_uint4(0u, 0u, 0u, 0u);
    if (c < D) {
      g[q] = *reinterpret_cast<const uint4*>(gamma + c);
      if (beta) bt[q] = *reinterpret_cast<const uint4*>(beta + c);
    }
  }
  int turn = 0;
  for (int row = blockIdx.x; row < M; row += gridDim.x) {
    const size_t base = (size_t)row * D;
    float v[NG][8];
    float s[1] = {0.f};
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      const int c = q * T * 8 + c0;
      if (c < D) {
        unpack8(nx[q], v[q]);
        if (sub) {
          float u[8];
          unpack8(ns[q], u);
          if (thresh) {
            bool k[8];
            keep8(seed, offset, base + c, thresh, k);
#pragma unroll
            for (int i = 0; i < 8; ++i) u[i] = k[i] ? u[i] * drop_scale : 0.f;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) v[q][i] += u[i];
        }
        const uint4 hp = pack8(v[q]);   // round to bf16 first: backward sees exactly the saved h
        unpack8(hp, v[q]);
        if (h_out) *reinterpret_cast<uint4*>(h_out + base + c) = hp;
#pragma unroll
        for (int i = 0; i < 8; ++i) s[0] += v[q][i];
      }
    }
    if (row + (int)gridDim.x < M) fetch(row + gridDim.x);
    float mean = 0.f;
    if (!rms) {
      block_sum_n<T, 1>(s, red, turn);
      mean = s[0] / D;
      turn ^= 1;
    }
    float qq[1] = {0.f};
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      if (q * T * 8 + c0 < D) {
#pragma unroll
        for (int i = 0; i < 8; ++i) { const float d = v[q][i] - mean; qq[0] += d * d; }
      }
    }
    block_sum_n<T, 1>(qq, red, turn);
    const float rstd = rsqrtf(qq[0] / D + eps);
    turn ^= 1;
    if (threadIdx.x == 0) {
      if (mean_out) mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      const int c = q * T * 8 + c0;
      if (c < D) {
        float o[8], gf[8], bf[8];
        unpack8(g[q], gf);
        unpack8(bt[q], bf);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = (v[q][i] - mean) * rstd * gf[i] + bf[i];
        *reinterpret_cast<uint4*>(y + base + c) = pack8(o);
      }
    }
  }
}

// Backward: dh = d(norm)/dh (+ dres); dx = dh; dsub = dropout_mask * dh.  Per-thread dgamma / dbeta partials stay in
// registers across the rows of the block and are added to the fp32 outputs with one atomic per column at the end, so there
// are few blocks, each with many rows.  With `part_pitch` every block leaves its sums in a row of its own instead
// (dgamma + block * part_pitch, dbeta's D columns behind), which norm_param_grads_kernel adds up: no buffer has to be zeroed before
// and converted after.  R rows are in flight at once and share a reduction (two sums a row, one barrier):
// one row at a time left the block waiting for a load and two barriers per row.  Narrow rows take T < 256 threads and a
// block works on 256 / T groups of R rows side by side, whose column sums it adds up before the atomics.
// 256 x 256 6.6 -> 2.9 us, 650 x 768 8.1 -> 4.6, 1024 x 512 8.5 -> 4.8, 1024 x 2048 with dropout 11.0 -> 9.7,
// 8192 x 2048 30.4 -> 28.7, 4096 x 5120 51 -> 34.
// AHEAD: the next rows are fetched while the current ones are worked on.  It takes the registers of two more rows, so fewer
// are in flight at once, and pays where a block has many rows: 16384 x 1536 with dropout, four rows 76.7 us, two and two
// ahead 71.4; without dropout 60.2 and 48.5.
template <int T, int NG, int R, bool AHEAD = false>
__global__ void __launch_bounds__(256, 2) norm_bwd_kernel(
    const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ gamma,
    const float* __restrict__ mean_in, const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx,
    __nv_bfloat16* __restrict__ dsub, float* __restrict__ dgamma, float* __restrict__ dbeta, int M, int D, int rms,
    uint32_t thresh, float drop_scale, uint64_t seed, uint64_t offset, const __nv_bfloat16* __restrict__ dres,
    const unsigned long long* __restrict__ step_ptr, int vec_atomics, int part_pitch) {
  pdl_prologue();
  constexpr int G = 256 / T;                   // row groups of the block
  __shared__ float red[2 * 8 * 2 * R];
  __shared__ float colsum[G > 1 ? 2 * 2048 : 1];
  const int tid = threadIdx.x % T, grp = threadIdx.x / T;
  if (step_ptr) offset += __ldg(step_ptr) * 65536ull;
  uint4 g[NG];
  float pg[NG][8], pb[NG][8];
#pragma unroll
  for (int q = 0; q < NG; ++q) {
    const int c = (q * T + tid) * 8;
    g[q] = make_uint4(0u, 0u, 0u, 0u);
    if (c < D) g[q] = *reinterpret_cast<const uint4*>(gamma + c);
#pragma unroll
    for (int i = 0; i < 8; ++i) { pg[q][i] = 0.f; pb[q][i] = 0.f; }
  }
  uint4 nd[R][NG], nh[R][NG];
  float nmean[R], nrstd[R];
  auto fetch = [&](int row0) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = row0 + r;
      nmean[r] = nrstd[r] = 0.f;
      if (row < M) {
        if (!rms) nmean[r] = mean_in[row];
        nrstd[r] = rstd_in[row];
      }
#pragma unroll
      for (int q = 0; q < NG; ++q) {
        const int c = (q * T + tid) * 8;
        nd[r][q] = nh[r][q] = make_uint4(0u, 0u, 0u, 0u);
        if (c < D && row < M) {
          nd[r][q] = __ldcs(reinterpret_cast<const uint4*>(dy + (size_t)row * D + c));
          nh[r][q] = __ldcs(reinterpret_cast<const uint4*>(h + (size_t)row * D + c));
        }
      }
    }
  };
  if (AHEAD) fetch(blockIdx.x * (G * R) + grp * R);
  int turn = 0;
  for (int block0 = blockIdx.x * (G * R); block0 < M; block0 += gridDim.x * (G * R)) {
    const int row0 = block0 + grp * R;
    if (!AHEAD) fetch(row0);
    uint4 cd[R][NG], ch[R][NG];
    float mean[R], rstd[R], s[2 * R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      mean[r] = nmean[r];
      rstd[r] = nrstd[r];
#pragma unroll
      for (int q = 0; q < NG; ++q) {
        cd[r][q] = nd[r][q];
        ch[r][q] = nh[r][q];
      }
    }
    if (AHEAD) fetch(row0 + gridDim.x * (G * R));
#pragma unroll
    for (int r = 0; r < R; ++r) {
      s[2 * r] = s[2 * r + 1] = 0.f;
      if (row0 + r < M) {
#pragma unroll
        for (int q = 0; q < NG; ++q) {
          if ((q * T + tid) * 8 < D) {
            float d[8], hv[8], gf[8];
            unpack8(cd[r][q], d);
            unpack8(ch[r][q], hv);
            unpack8(g[q], gf);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float xh = (hv[i] - mean[r]) * rstd[r];
              const float dg = d[i] * gf[i];
              s[2 * r] += dg;
              s[2 * r + 1] += dg * xh;
              pg[q][i] += d[i] * xh;
              pb[q][i] += d[i];
            }
          }
        }
      }
    }
    block_sum_n<T, 2 * R, G>(s, red, turn);
    turn ^= 1;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = row0 + r;
      if (row >= M) break;
      const size_t base = (size_t)row * D;
      const float s1 = rms ? 0.f : s[2 * r] / D, s2 = s[2 * r + 1] / D;
#pragma unroll
      for (int q = 0; q < NG; ++q) {
        const int c = (q * T + tid) * 8;
        if (c < D) {
          float o[8], d[8], hv[8], gf[8];
          unpack8(cd[r][q], d);
          unpack8(ch[r][q], hv);
          unpack8(g[q], gf);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = (d[i] * gf[i] - s1 - (hv[i] - mean[r]) * rstd[r] * s2) * rstd[r];
          if (dres) {   // gradient that reaches h along a second path (pre-norm residual stream)
            float e[8];
            unpack8(__ldcs(reinterpret_cast<const uint4*>(dres + base + c)), e);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] += e[i];
          }
          *reinterpret_cast<uint4*>(dx + base + c) = pack8(o);
          if (dsub) {
            if (thresh) {
              bool k[8];
              keep8(seed, offset, base + c, thresh, k);
#pragma unroll
              for (int i = 0; i < 8; ++i) o[i] = k[i] ? o[i] * drop_scale : 0.f;
            }
            *reinterpret_cast<uint4*>(dsub + base + c) = pack8(o);
          }
        }
      }
    }
  }
  if (G > 1) {       // NG = 1: columns 8 tid .. 8 tid + 7 of every group
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      colsum[grp * (T * 8) + i * T + tid] = pg[0][i];
      colsum[2048 + grp * (T * 8) + i * T + tid] = pb[0][i];
    }
    __syncthreads();
    if (grp) return;
#pragma unroll
    for (int k = 1; k < G; ++k)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        pg[0][i] += colsum[k * (T * 8) + i * T + tid];
        pb[0][i] += colsum[2048 + k * (T * 8) + i * T + tid];
      }
  }
#pragma unroll
  for (int q = 0; q < NG; ++q) {
    const int c = (q * T + tid) * 8;
    if (c < D) {
      if (part_pitch) {
        float4* o = reinterpret_cast<float4*>(dgamma + (size_t)blockIdx.x * part_pitch + c);
        o[0] = make_float4(pg[q][0], pg[q][1], pg[q][2], pg[q][3]);
        o[1] = make_float4(pg[q][4], pg[q][5], pg[q][6], pg[q][7]);
        if (dbeta) {
          o = reinterpret_cast<float4*>(dbeta + (size_t)blockIdx.x * part_pitch + c);
          o[0] = make_float4(pb[q][0], pb[q][1], pb[q][2], pb[q][3]);
          o[1] = make_float4(pb[q][4], pb[q][5], pb[q][6], pb[q][7]);
        }
        continue;
      }
      if (!vec_atomics) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          atomicAdd(dgamma + c + i, pg[q][i]);
          if (dbeta) atomicAdd(dbeta + c + i, pb[q][i]);
        }
        continue;
      }
      // 16-byte vector reductions: four columns per atomic
      atomicAdd(reinterpret_cast<float4*>(dgamma + c), make_float4(pg[q][0], pg[q][1], pg[q][2], pg[q][3]));
      atomicAdd(reinterpret_cast<float4*>(dgamma + c + 4), make_float4(pg[q][4], pg[q][5], pg[q][6], pg[q][7]));
      if (dbeta) {
        atomicAdd(reinterpret_cast<float4*>(dbeta + c), make_float4(pb[q][0], pb[q][1], pb[q][2], pb[q][3]));
        atomicAdd(reinterpret_cast<float4*>(dbeta + c + 4), make_float4(pb[q][4], pb[q][5], pb[q][6], pb[q][7]));
      }
    }
  }
}

// out[c] = bf16(sum over n rows of part[r * pitch + y * D + c]): the gradients of gamma (y = 0) and beta (y = 1).  64 columns a
// block, 16 rows side by side, always in the same order.  Up to a few MB that are still in L2: bound by its launch.
__global__ void __launch_bounds__(256) norm_param_grads_kernel(const float* __restrict__ part, int n, int pitch, int D,
                                                               __nv_bfloat16* __restrict__ dgamma, __nv_bfloat16* __restrict__ dbeta) {
  pdl_prologue();
  __shared__ float4 sums[16][16];
  const int x = threadIdx.x & 15, y = threadIdx.x >> 4, c = blockIdx.x * 64 + x * 4;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c < D) {
    const float* p = part + (size_t)blockIdx.y * D + c;
#pragma unroll 8
    for (int r = y; r < n; r += 16) {
      const float4 v = *reinterpret_cast<const float4*>(p + (size_t)r * pitch);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
  }
  sums[y][x] = s;
  __syncthreads();
  if (y || c >= D) return;
#pragma unroll
  for (int k = 1; k < 16; ++k) {
    const float4 v = sums[k][x];
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  __nv_bfloat16* out = (blockIdx.y ? dbeta : dgamma) + c;
  out[0] = __float2bfloat16(s.x); out[1] = __float2bfloat16(s.y); out[2] = __float2bfloat16(s.z); out[3] = __float2bfloat16(s.w);
}

// ------------------------------------------------------------------------------------------------
// Softmax cross-entropy over rows of bf16 logits [M, V] (row pitch ld). Writes the per-row loss (fp32)
// and overwrites the logits with grad_scale * (softmax - onehot), i.e. the gradient of
// grad_scale * sum_rows(loss). Rows whose target equals ignore_index give zero loss and gradient.
// ------------------------------------------------------------------------------------------------
__global__ void ce_kernel(__nv_bfloat16* logits, long long ld, const long long* __restrict__ target,
                          float* __restrict__ loss, int M, int V, float grad_scale, long long ignore_index,
                          int write_grad, __nv_bfloat16* grad, long long ldg) {
  __shared__ float red[32];
  for (int row = blockIdx.x; row < M; row += gridDim.x) {
    __nv_bfloat16* lp = logits + (size_t)row * ld;
    __nv_bfloat16* gp = grad ? grad + (size_t)row * ldg : lp;   // the gradient may go to a buffer of its own
    const long long t = target[row];
    float mx = -INFINITY;
    for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
      float v[8];
      unpack8(*reinterpret_cast<const uint4*>(lp + c), v);
#pragma unroll
      for (int i = 0; i < 8; ++i) mx = fmaxf(mx, v[i]);
    }
    mx = block_max(mx, red);
    float se = 0.f;
    for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
      float v[8];
      unpack8(*reinterpret_cast<const uint4*>(lp + c), v);
#pragma unroll
      for (int i = 0; i < 8; ++i) se += __expf(v[i] - mx);
    }
    se = block_sum(se, red);
    const float lse = mx + __logf(se);
    const bool ignored = (t == ignore_index) || t < 0 || t >= V;
    if (threadIdx.x == 0) loss[row] = ignored ? 0.f : lse - __bfloat162float(lp[t]);
    __syncthreads();
    if (write_grad) {
      const float inv = 1.f / se;
      for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
        float v[8];
        unpack8(*reinterpret_cast<const uint4*>(lp + c), v);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float p = __expf(v[i] - mx) * inv;
          if (c + i == t) p -= 1.f;
          v[i] = ignored ? 0.f : p * grad_scale;
        }
        *reinterpret_cast<uint4*>(gp + c) = pack8(v);
      }
    }
    __syncthreads();
  }
}

// The same with the row in registers, for up to 32768 logits: every logit is read once and every gradient written once.  A
// block takes one row, NG 16-byte words a thread, all in flight at once; two (512 threads) or three blocks share an SM, so
// that one loads or stores while the other computes.  The two exponentials a logit (16 a clock and SM) and the unpacking
// bound it, not memory: 4096 x 32000 166 -> 114 us, 1024 x 8192 10.4 -> 7.2 against the kernel above, which reads a row three
// times.  Tried and dropped: the row in shared memory, filled and drained by bulk copies; 1024 threads with half the words
// (one block per SM).
// Up to 16384 logits 256 threads, which add up in the order of the kernel above.
constexpr int kCeMaxV = 65536;
template <int kCeThreads, int NG>
__global__ void __launch_bounds__(kCeThreads, kCeThreads == 512 ? 2 : 3) ce_row_kernel(
    const __nv_bfloat16* logits, long long ld, const long long* __restrict__ target, float* __restrict__ loss, int V,
    float grad_scale, const float* __restrict__ scale_ptr, long long ignore_index, __nv_bfloat16* grad, long long ldg) {
  pdl_prologue();
  __shared__ float red[32];
  const int row = blockIdx.x, tid = threadIdx.x, n = V >> 3;
  const uint4* lp = reinterpret_cast<const uint4*>(logits + (size_t)row * ld);
  const long long t = target[row];
  const bool ignored = t == ignore_index || t < 0 || t >= V;
  uint4 u[NG];
  const uint32_t kNegInf2 = 0xff80ff80u;                 // two bf16 -inf: words beyond the row count for nothing
#pragma unroll
  for (int q = 0; q < NG; ++q) {
    const int i = q * kCeThreads + tid;
    u[q] = i < n ? __ldcs(lp + i) : make_uint4(kNegInf2, kNegInf2, kNegInf2, kNegInf2);
  }
  const float lt = (tid == 0 && !ignored) ? __bfloat162float(logits[(size_t)row * ld + t]) : 0.f;
  if (scale_ptr) grad_scale *= __ldg(scale_ptr);
  float mx = -INFINITY;
#pragma unroll
  for (int q = 0; q < NG; ++q) {
    float v[8];
    unpack8(u[q], v);
#pragma unroll
    for (int k = 0; k < 8; ++k) mx = fmaxf(mx, v[k]);
  }
  mx = block_max(mx, red);
  float se = 0.f;
#pragma unroll
  for (int q = 0; q < NG; ++q) {
    if (q * kCeThreads + tid < n) {
      float v[8];
      unpack8(u[q], v);
#pragma unroll
      for (int k = 0; k < 8; ++k) se += __expf(v[k] - mx);
    }
  }
  se = block_sum(se, red);
  if (tid == 0) loss[row] = ignored ? 0.f : mx + __logf(se) - lt;
  if (!grad) return;
  const float inv = 1.f / se;
  uint4* gp = reinterpret_cast<uint4*>(grad + (size_t)row * ldg);
#pragma unroll
  for (int q = 0; q < NG; ++q) {
    const int i = q * kCeThreads + tid;
    if (i < n) {
      float v[8];
      unpack8(u[q], v);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float p = __expf(v[k] - mx) * inv;
        if (i * 8 + k == (int)t) p -= 1.f;
        v[k] = ignored ? 0.f : p * grad_scale;
      }
      __stcs(gp + i, pack8(v));
    }
  }
}

// The same sums in the same order (so the same bits), with the row read again for each pass instead of held: the second and
// third reads come from L2, little lives in registers and four blocks of 512 threads (eight of 256) share an SM.  A held row
// leaves two blocks an SM that wait for memory and then compute, and above 32768 logits it spills.  us, held / read again:
// loss and gradient of 8192 x 50304 451 / 296, 1024 x 40960 49 / 40, 64 x 65536 21.6 / 9.3, 8192 x 20480 140 / 138, 300 x
// 20480 8.1 / 10.6; loss alone of 8192 x 50304 280 / 136, 1024 x 57344 52 / 26, 2048 x 9216 10.6 / 8.7.
template <int T, bool GRAD>
__global__ void __launch_bounds__(T, 2048 / T) ce_stream_kernel(
    const __nv_bfloat16* logits, long long ld, const long long* __restrict__ target, float* __restrict__ loss, int V,
    float grad_scale, const float* __restrict__ scale_ptr, long long ignore_index, __nv_bfloat16* grad, long long ldg) {
  pdl_prologue();
  __shared__ float red[32];
  const int row = blockIdx.x, tid = threadIdx.x, n = V >> 3;
  const uint4* lp = reinterpret_cast<const uint4*>(logits + (size_t)row * ld);
  const long long t = target[row];
  const bool ignored = t == ignore_index || t < 0 || t >= V;
  const float lt = (tid == 0 && !ignored) ? __bfloat162float(logits[(size_t)row * ld + t]) : 0.f;
  float mx = -INFINITY;
#pragma unroll 4
  for (int i = tid; i < n; i += T) {
    float v[8];
    unpack8(lp[i], v);
#pragma unroll
    for (int k = 0; k < 8; ++k) mx = fmaxf(mx, v[k]);
  }
  mx = block_max(mx, red);
  float se = 0.f;
#pragma unroll 4
  for (int i = tid; i < n; i += T) {
    float v[8];
    unpack8(lp[i], v);
#pragma unroll
    for (int k = 0; k < 8; ++k) se += __expf(v[k] - mx);
  }
  se = block_sum(se, red);
  if (tid == 0) loss[row] = ignored ? 0.f : mx + __logf(se) - lt;
  if (!GRAD) return;
  if (scale_ptr) grad_scale *= __ldg(scale_ptr);
  const float inv = 1.f / se;
  uint4* gp = reinterpret_cast<uint4*>(grad + (size_t)row * ldg);
#pragma unroll 4
  for (int i = tid; i < n; i += T) {
    float v[8];
    unpack8(lp[i], v);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float p = __expf(v[k] - mx) * inv;
      if (i * 8 + k == (int)t) p -= 1.f;
      v[k] = ignored ? 0.f : p * grad_scale;
    }
    __stcs(gp + i, pack8(v));
  }
}

// n = number of targets that count (at least one), for the mean: out[0] = n, out[1] = 1 / n.
__global__ void ce_count_kernel(const long long* __restrict__ target, int M, long long ignore_index, float* out) {
  pdl_prologue();
  __shared__ int total;
  int c = 0;
  for (int i = threadIdx.x; i < M; i += blockDim.x) c += target[i] != ignore_index;
  c = __reduce_add_sync(0xffffffffu, c);
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) atomicAdd(&total, c);
  __syncthreads();
  if (threadIdx.x == 0) {
    const float n = (float)max(total, 1);
    out[0] = n;
    out[1] = 1.f / n;
  }
}
// g *= *scale, except by one: the usual gradient of a loss costs no pass over the logits' gradient.
__global__ void scale_unless_one_kernel(__nv_bfloat16* g, const float* __restrict__ scale, long long n8) {
  const float s = __ldg(scale);
  if (s == 1.f) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    float v[8];
    unpack8(reinterpret_cast<const uint4*>(g)[i], v);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] *= s;
    reinterpret_cast<uint4*>(g)[i] = pack8(v);
  }
}

// ------------------------------------------------------------------------------------------------
// Embedding gather for one visiting table shard [V, Ds]: out[t, col_off + c] =
//   dropout(table[ids[t], c] * scale + pe[t / tokens_per_pos, col_off + c])
// ------------------------------------------------------------------------------------------------
__global__ void embed_fwd_kernel(const __nv_bfloat16* __restrict__ table, const long long* __restrict__ ids,
                                 const __nv_bfloat16* __restrict__ pe, long long ld_pe, int tokens_per_pos,
                                 __nv_bfloat16* __restrict__ out, long long ld_out, int col_off, int T, int Ds, int D,
                                 float scale, uint32_t thresh, float drop_scale, uint64_t seed, uint64_t offset,
                                 const unsigned long long* __restrict__ step_ptr) {
  pdl_prologue();
  if (step_ptr) offset += __ldg(step_ptr) * 65536ull;
  const int per_row = Ds / 8;
  const long long total = (long long)T * per_row;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / per_row), c = (int)(i % per_row) * 8;
    float v[8];
    unpack8(*reinterpret_cast<const uint4*>(table + (size_t)ids[t] * Ds + c), v);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] *= scale;
    if (pe) {
      float p[8];
      unpack8(*reinterpret_cast<const uint4*>(pe + (size_t)(t / tokens_per_pos) * ld_pe + col_off + c), p);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += p[k];
    }
    if (thresh) {
      bool kp[8];
      keep8(seed, offset, (uint64_t)t * D + col_off + c, thresh, kp);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = kp[k] ? v[k] * drop_scale : 0.f;
    }
    *reinterpret_cast<uint4*>(out + (size_t)t * ld_out + col_off + c) = pack8(v);
  }
}
// Scatter-add of the output gradient into a (zeroed or incoming) table-shard gradient [V, Ds].
// blk_cols > 0: gtable is block-major, [Ds / blk_cols][V][blk_cols] (one contiguous [V, blk_cols] block per owner of an
// embedding-dim shard); blk_cols = 0: plain [V, Ds].
__global__ void embed_bwd_kernel(__nv_bfloat16* __restrict__ gtable, const long long* __restrict__ ids,
                                 const __nv_bfloat16* __restrict__ dy, long long ld_dy, int col_off, int T, int Ds,
                                 int D, float scale, uint32_t thresh, float drop_scale, uint64_t seed, uint64_t offset,
                                 const unsigned long long* __restrict__ step_ptr, int blk_cols, int V) {
  pdl_prologue();
  if (step_ptr) offset += __ldg(step_ptr) * 65536ull;
  const int per_row = Ds / 8;
  const long long total = (long long)T * per_row;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / per_row), c = (int)(i % per_row) * 8;
    float v[8];
    unpack8(*reinterpret_cast<const uint4*>(dy + (size_t)t * ld_dy + col_off + c), v);
    if (thresh) {
      bool kp[8];
      keep8(seed, offset, (uint64_t)t * D + col_off + c, thresh, kp);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = kp[k] ? v[k] * drop_scale : 0.f;
    }
    __nv_bfloat162* g = blk_cols > 0
        ? reinterpret_cast<__nv_bfloat162*>(gtable + ((size_t)(c / blk_cols) * V + (size_t)ids[t]) * blk_cols + (c % blk_cols))
        : reinterpret_cast<__nv_bfloat162*>(gtable + (size_t)ids[t] * Ds + c);
#pragma unroll
    for (int k = 0; k < 4; ++k) atomicAdd(g + k, __floats2bfloat162_rn(v[2 * k] * scale, v[2 * k + 1] * scale));
  }
}

// ------------------------------------------------------------------------------------------------
// Short-sequence attention (S <= 128, head_dim 64) on packed projections, in fp32 throughout.
// qkv: [T, 3*D] with T = S*B tokens (token = s*B + b). The projection comes out of a column-rotated
// linear, so its columns are grouped per shard: shard j holds [q_j | k_j | v_j], each D/nshard wide.
// out: [T, D], column = head*64 + d. One block per (batch, head).
//
// There are few blocks (batch x heads) and little work in each, so a block's latency is the kernel's time.  Products run
// on register tiles (2 x 2 scores, 2 x 4 outputs a thread) fed by 16-byte shared-memory reads, 256 or 512 threads a block;
// rows of 64 floats hold their 16-byte chunks swizzled by row % 8, so that eight rows read side by side touch different
// banks.  One score per thread from rows of 65 floats, 128 threads: 13 x 12 blocks of S = 50 took 32 us forward and
// 97 us backward, now 13 and 27 us.
// ------------------------------------------------------------------------------------------------
constexpr int kHd = 64;
__device__ __forceinline__ int qkv_col(int head, int which, int D, int nshard, int heads) {
  const int hps = heads / nshard;  // heads per shard
  const int j = head / hps, hl = head % hps;
  return j * (3 * (D / nshard)) + which * (D / nshard) + hl * kHd;
}
// 16-byte chunk c (0..15) of row r
__device__ __forceinline__ float4& chunk_at(float* base, int r, int c) {
  return reinterpret_cast<float4*>(base)[r * 16 + (c ^ (r & 7))];
}
__device__ __forceinline__ float dot4(const float4& a, const float4& b, float acc) {
  acc = fmaf(a.x, b.x, acc); acc = fmaf(a.y, b.y, acc); acc = fmaf(a.z, b.z, acc);
  return fmaf(a.w, b.w, acc);
}
__device__ __forceinline__ void axpy4(float s, const float4& v, float4& acc) {
  acc.x = fmaf(s, v.x, acc.x); acc.y = fmaf(s, v.y, acc.y); acc.z = fmaf(s, v.z, acc.z); acc.w = fmaf(s, v.w, acc.w);
}
// The rows of N operands into shared memory, their loads in flight together: in a loop for each operand a short sequence
// waited for memory once per operand (4 x 4 blocks, S = 8: forward 3.4 -> 2.9 us, backward 4.9 -> 4.0).
template <int N>
__device__ __forceinline__ void fill_rows(float* const (&dst)[N], const __nv_bfloat16* const (&src)[N], const long long (&ld)[N],
                                          const int (&col)[N], const float (&scale)[N], int S, int B, int b) {
  for (int i = threadIdx.x; i < S * 8; i += blockDim.x) {
    const int s = i >> 3, c = i & 7;
    uint4 u[N];
#pragma unroll
    for (int k = 0; k < N; ++k)
      u[k] = *reinterpret_cast<const uint4*>(src[k] + (size_t)(s * B + b) * ld[k] + col[k] + c * 8);
#pragma unroll
    for (int k = 0; k < N; ++k) {
      float f[8];
      unpack8(u[k], f);
      chunk_at(dst[k], s, 2 * c) = make_float4(f[0] * scale[k], f[1] * scale[k], f[2] * scale[k], f[3] * scale[k]);
      chunk_at(dst[k], s, 2 * c + 1) = make_float4(f[4] * scale[k], f[5] * scale[k], f[6] * scale[k], f[7] * scale[k]);
    }
  }
}
// out[r, c] = <a_r, b_c> for c <= r (causal) or all c, -inf / 0 elsewhere (`other`), on 2 x 2 tiles
__device__ __forceinline__ void row_dots(float* a, float* b, float* out, int S, int causal, float other) {
  const int nt = (S + 1) >> 1;
  for (int i = threadIdx.x; i < nt * nt; i += blockDim.x) {
    const int r0 = (i / nt) * 2, c0 = (i % nt) * 2;
    const int r1 = min(r0 + 1, S - 1), c1 = min(c0 + 1, S - 1);
    float d00 = 0.f, d01 = 0.f, d10 = 0.f, d11 = 0.f;
    if (!causal || c0 <= r1) {
#pragma unroll 8
      for (int e = 0; e < 16; ++e) {
        const float4 x0 = chunk_at(a, r0, e), x1 = chunk_at(a, r1, e), y0 = chunk_at(b, c0, e), y1 = chunk_at(b, c1, e);
        d00 = dot4(x0, y0, d00); d01 = dot4(x0, y1, d01); d10 = dot4(x1, y0, d10); d11 = dot4(x1, y1, d11);
      }
    }
    const int ld = S + 1;
    out[r0 * ld + c0] = (!causal || c0 <= r0) ? d00 : other;
    if (c0 + 1 < S) out[r0 * ld + c0 + 1] = (!causal || c0 + 1 <= r0) ? d01 : other;
    if (r0 + 1 < S) {
      out[(r0 + 1) * ld + c0] = (!causal || c0 <= r0 + 1) ? d10 : other;
      if (c0 + 1 < S) out[(r0 + 1) * ld + c0 + 1] = (!causal || c0 + 1 <= r0 + 1) ? d11 : other;
    }
  }
}
// acc[u] = sum_c w(r0 + u, c) v_c[4 e .. 4 e + 3] over c in [lo, hi), w(r, c) = p[r * sr + c * sc]
__device__ __forceinline__ void row_sums(const float* p, int sr, int sc, float* v, int r0, int r1, int e, int lo, int hi,
                                         float4 (&acc)[2]) {
  acc[0] = acc[1] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int c = lo; c < hi; ++c) {
    const float4 x = chunk_at(v, c, e);
    axpy4(p[r0 * sr + c * sc], x, acc[0]);
    axpy4(p[r1 * sr + c * sc], x, acc[1]);
  }
}
__device__ __forceinline__ void store4(__nv_bfloat16* dst, const float4& v, float s) {
  *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(v.x * s, v.y * s), pack_bf16(v.z * s, v.w * s));
}

__global__ void __launch_bounds__(512) attn_small_fwd_kernel(const __nv_bfloat16* __restrict__ qkv, __nv_bfloat16* __restrict__ out,
                                      int S, int B, int heads, int nshard, int causal, float sm_scale, uint32_t thresh,
                                      float drop_scale, uint64_t seed, uint64_t offset,
                                      const unsigned long long* __restrict__ step_ptr) {
  pdl_prologue();
  extern __shared__ __align__(16) float smf[];
  if (step_ptr) offset += __ldg(step_ptr) * 65536ull;
  const int D = heads * kHd;
  const int b = blockIdx.x / heads, h = blockIdx.x % heads;
  float* q = smf;                 // [S][64], pre-scaled
  float* k = q + S * kHd;
  float* v = k + S * kHd;
  float* p = v + S * kHd;         // [S][S+1]
  fill_rows<3>({q, k, v}, {qkv, qkv, qkv}, {3 * D, 3 * D, 3 * D},
               {qkv_col(h, 0, D, nshard, heads), qkv_col(h, 1, D, nshard, heads), qkv_col(h, 2, D, nshard, heads)},
               {sm_scale, 1.f, 1.f}, S, B, b);
  __syncthreads();
  row_dots(q, k, p, S, causal, -INFINITY);
  __syncthreads();
  // softmax per row: one warp per row
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int r = warp; r < S; r += nw) {
    float mx = -INFINITY;
    for (int c = lane; c < S; c += 32) mx = fmaxf(mx, p[r * (S + 1) + c]);
    mx = warp_max(mx);
    float se = 0.f;
    for (int c = lane; c < S; c += 32) {
      float e = __expf(p[r * (S + 1) + c] - mx);
      p[r * (S + 1) + c] = e;
      se += e;
    }
    se = warp_sum(se);
    const float inv = 1.f / se;
    for (int c = lane; c < S; c += 32) {
      float pv = p[r * (S + 1) + c] * inv;
      if (thresh) {
        const uint64_t e = ((uint64_t)blockIdx.x * S + r) * S + c;
        pv = dropout_keep(seed, offset, e, thresh) ? pv * drop_scale : 0.f;
      }
      p[r * (S + 1) + c] = pv;
    }
  }
  __syncthreads();
  const int nt = (S + 1) >> 1;
  for (int i = threadIdx.x; i < nt * 16; i += blockDim.x) {
    const int r0 = (i >> 4) * 2, e = i & 15, r1 = min(r0 + 1, S - 1);
    float4 acc[2];
    row_sums(p, S + 1, 1, v, r0, r1, e, 0, causal ? r0 + 1 : S, acc);
    if (causal && r1 > r0) axpy4(p[r1 * (S + 1) + r1], chunk_at(v, r1, e), acc[1]);   // row r0 does not see key r1
    __nv_bfloat16* o = out + h * kHd + 4 * e;
    store4(o + (size_t)(r0 * B + b) * D, acc[0], 1.f);
    if (r0 + 1 < S) store4(o + (size_t)(r1 * B + b) * D, acc[1], 1.f);
  }
}

__global__ void __launch_bounds__(512) attn_small_bwd_kernel(const __nv_bfloat16* __restrict__ qkv,
                                      const __nv_bfloat16* __restrict__ dout, __nv_bfloat16* __restrict__ dqkv, int S, int B,
                                      int heads, int nshard, int causal, float sm_scale, uint32_t thresh, float drop_scale,
                                      uint64_t seed, uint64_t offset, const unsigned long long* __restrict__ step_ptr) {
  pdl_prologue();
  extern __shared__ __align__(16) float smf[];
  if (step_ptr) offset += __ldg(step_ptr) * 65536ull;
  const int D = heads * kHd;
  const int b = blockIdx.x / heads, h = blockIdx.x % heads;
  float* q = smf;                 // [S][64] (pre-scaled)
  float* k = q + S * kHd;
  float* v = k + S * kHd;
  float* go = v + S * kHd;        // dO
  float* p = go + S * kHd;        // [S][S+1] softmax probabilities (no dropout)
  float* ds = p + S * (S + 1);    // [S][S+1] dP then dS
  const int cq = qkv_col(h, 0, D, nshard, heads), ck = qkv_col(h, 1, D, nshard, heads), cv = qkv_col(h, 2, D, nshard, heads);
  fill_rows<4>({q, k, v, go}, {qkv, qkv, qkv, dout}, {3 * D, 3 * D, 3 * D, D}, {cq, ck, cv, h * kHd},
               {sm_scale, 1.f, 1.f, 1.f}, S, B, b);
  __syncthreads();
  row_dots(q, k, p, S, causal, -INFINITY);
  row_dots(go, v, ds, S, causal, 0.f);                // dP of the dropped probabilities
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int r = warp; r < S; r += nw) {
    float mx = -INFINITY;
    for (int c = lane; c < S; c += 32) mx = fmaxf(mx, p[r * (S + 1) + c]);
    mx = warp_max(mx);
    float se = 0.f;
    for (int c = lane; c < S; c += 32) {
      float e = __expf(p[r * (S + 1) + c] - mx);
      p[r * (S + 1) + c] = e;
      se += e;
    }
    se = warp_sum(se);
    const float inv = 1.f / se;
    float dot = 0.f;
    uint32_t keep = 0;                                // bit j: element lane + 32 j survives (S <= 128)
    for (int c = lane, j = 0; c < S; c += 32, ++j) {
      const float pv = p[r * (S + 1) + c] * inv;
      float m = 1.f;
      if (thresh) {
        const uint64_t e = ((uint64_t)blockIdx.x * S + r) * S + c;
        const bool kp = dropout_keep(seed, offset, e, thresh);
        keep |= (kp ? 1u : 0u) << j;
        m = kp ? drop_scale : 0.f;
      }
      const float dpv = ds[r * (S + 1) + c] * m;      // gradient wrt the un-dropped probability
      p[r * (S + 1) + c] = pv;
      ds[r * (S + 1) + c] = dpv;
      dot += dpv * pv;
    }
    dot = warp_sum(dot);
    for (int c = lane, j = 0; c < S; c += 32, ++j) {
      const float pv = p[r * (S + 1) + c];
      const float dsv = pv * (ds[r * (S + 1) + c] - dot);
      // keep the dropped probability in p for dV
      const float m = thresh ? (((keep >> j) & 1u) ? drop_scale : 0.f) : 1.f;
      p[r * (S + 1) + c] = pv * m;
      ds[r * (S + 1) + c] = dsv;
    }
  }
  __syncthreads();
  // dQ = dS K * scale ; dK = dS^T Q(pre-scaled) ; dV = Pd^T dO
  const int nt = (S + 1) >> 1, ld = S + 1;
  for (int i = threadIdx.x; i < 3 * nt * 16; i += blockDim.x) {
    const int which = i / (nt * 16), j = i - which * (nt * 16);
    const int r0 = (j >> 4) * 2, e = j & 15, r1 = min(r0 + 1, S - 1);
    float4 acc[2];
    // entries above the diagonal are 0 with a causal mask: rows see the keys up to r1, keys the rows from r0 on
    if (which == 0) row_sums(ds, ld, 1, k, r0, r1, e, 0, causal ? r1 + 1 : S, acc);
    else if (which == 1) row_sums(ds, 1, ld, q, r0, r1, e, causal ? r0 : 0, S, acc);
    else row_sums(p, 1, ld, go, r0, r1, e, causal ? r0 : 0, S, acc);
    __nv_bfloat16* o = dqkv + (which == 0 ? cq : which == 1 ? ck : cv) + 4 * e;
    const float sc = which == 0 ? sm_scale : 1.f;
    store4(o + (size_t)(r0 * B + b) * (3 * D), acc[0], sc);
    if (r0 + 1 < S) store4(o + (size_t)(r1 * B + b) * (3 * D), acc[1], sc);
  }
}

// ------------------------------------------------------------------------------------------------
// Column sums of a bf16 matrix [M, N] (pitch ld) into fp32 out[N] (must be zeroed by the caller).
// ------------------------------------------------------------------------------------------------
__global__ void colsum_kernel(const __nv_bfloat16* __restrict__ x, long long ld, int M, int N, float* __restrict__ out,
                              int rows_per_block) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 2;
  if (c >= N) return;
  const int r0 = blockIdx.y * rows_per_block;
  const int r1 = min(M, r0 + rows_per_block);
  float a0 = 0.f, a1 = 0.f;
  for (int r = r0; r < r1; ++r) {
    const uint32_t u = *reinterpret_cast<const uint32_t*>(x + (size_t)r * ld + c);
    a0 += bf16_lo(u);
    a1 += bf16_hi(u);
  }
  atomicAdd(out + c, a0);
  atomicAdd(out + c + 1, a1);
}

// Vector variant: a block of 256 threads owns 64 columns (8 column lanes x 16 bytes) and a range of rows (32 row lanes,
// up to 8 loads in flight per thread); the row lanes are combined in shared memory.  The blocks that share a column
// group form a thread-block cluster along y: each leaves its 64 partial sums in its own shared memory, and the first
// block of the cluster adds them up through distributed shared memory and stores the result (no atomics, no zero-fill).
__global__ void __launch_bounds__(256) colsum_vec_kernel(const __nv_bfloat16* __restrict__ x, long long ld, int M, int N,
                                                         float* __restrict__ out, int rows_per_block, int atomic) {
  pdl_prologue();
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ float red[32][65];
  __shared__ float part[64];
  const int cl = threadIdx.x & 7, rl = threadIdx.x >> 3;
  const int c = blockIdx.x * 64 + cl * 8;
  const int r0 = blockIdx.y * rows_per_block;
  const int r1 = min(M, r0 + rows_per_block);
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  if (c < N) {
    int r = r0 + rl;
    for (; r + 7 * 32 < r1; r += 8 * 32) {
      uint4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldcs(reinterpret_cast<const uint4*>(x + (size_t)(r + u * 32) * ld + c));
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        float f[8];
        unpack8(v[u], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += f[i];
      }
    }
    for (; r + 3 * 32 < r1; r += 4 * 32) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldcs(reinterpret_cast<const uint4*>(x + (size_t)(r + u * 32) * ld + c));
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float f[8];
        unpack8(v[u], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += f[i];
      }
    }
    for (; r < r1; r += 32) {
      float f[8];
      unpack8(__ldcs(reinterpret_cast<const uint4*>(x + (size_t)r * ld + c)), f);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += f[i];
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) red[rl][cl * 8 + i] = acc[i];
  __syncthreads();
  if (threadIdx.x < 64) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) t += red[k][threadIdx.x];
    part[threadIdx.x] = t;
  }
  cluster.sync();
  if (cluster.block_rank() == 0 && threadIdx.x < 64) {
    const int col = blockIdx.x * 64 + threadIdx.x;
    float t = 0.f;
    for (unsigned k = 0; k < cluster.num_blocks(); ++k) t += cluster.map_shared_rank(part, k)[threadIdx.x];
    if (col < N) {
      if (atomic) atomicAdd(out + col, t); else out[col] = t;
    }
  }
  cluster.sync();   // no block leaves while its shared memory may still be read
}

// ------------------------------------------------------------------------------------------------
// Multi-tensor Adam / AdamW with optional gradient value clipping.
// ------------------------------------------------------------------------------------------------
constexpr int kAdamGroups = 2;
// One element's update, rounding by rounding, so that every path gives the same bits.
__device__ __forceinline__ void adam_element(float& p, float g, float& m, float& v, float decay, float beta1, float beta2,
                                             float eps, float weight_decay, int adamw, float clip_value, float grad_scale,
                                             float step_size, float inv_sqrt_bc2) {
  g = __fmul_rn(g, grad_scale);
  if (clip_value > 0.f) g = fminf(fmaxf(g, -clip_value), clip_value);
  if (weight_decay != 0.f) {
    if (adamw) p = __fmul_rn(p, 1.f - decay); else g = __fmaf_rn(weight_decay, p, g);
  }
  m = __fmaf_rn(1.f - beta1, g, __fmul_rn(beta1, m));
  v = __fmaf_rn(__fmul_rn(1.f - beta2, g), g, __fmul_rn(beta2, v));
  p = __fsub_rn(p, __fdividef(__fmul_rn(step_size, m), __fmaf_rn(sqrtf(v), inv_sqrt_bc2, eps)));
}
struct AdamRegs {
  float pv[8], gv[8], mv[8], vv[8];
  long long i0;
  int cnt;
  bool vec, svec;
};
// loads of one group of up to 8 elements (issued for both groups of a thread before either is updated)
__device__ __forceinline__ void adam_load(const RtpAdamTensor& t, long long i0, AdamRegs& r) {
  r.i0 = i0;
  r.cnt = i0 < t.n ? (int)min((long long)8, t.n - i0) : 0;
  if (r.cnt == 0) return;
  const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(t.p) + i0;
  const __nv_bfloat16* g = reinterpret_cast<const __nv_bfloat16*>(t.g) + i0;
  r.vec = r.cnt == 8 && ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g)) & 15) == 0;
  if (r.vec) {
    unpack8(__ldcs(reinterpret_cast<const uint4*>(p)), r.pv);
    unpack8(__ldcs(reinterpret_cast<const uint4*>(g)), r.gv);
  } else {
    _Pragma("unroll") for (int i = 0; i < 8; ++i) if (i < r.cnt) { r.pv[i] = __bfloat162float(p[i]); r.gv[i] = __bfloat162float(g[i]); }
  }
  // state_fp32: 0 = both moments bf16, 1 = both fp32, 2 = first moment bf16, second moment fp32
  r.svec = r.cnt == 8 && ((reinterpret_cast<uintptr_t>(t.m) | reinterpret_cast<uintptr_t>(t.v)) & 15) == 0;
  if (t.state_fp32 == 1) {
    const float* m = reinterpret_cast<const float*>(t.m) + i0;
    if (r.svec) {
      const float4 a = __ldcs(reinterpret_cast<const float4*>(m)), b = __ldcs(reinterpret_cast<const float4*>(m) + 1);
      r.mv[0] = a.x; r.mv[1] = a.y; r.mv[2] = a.z; r.mv[3] = a.w; r.mv[4] = b.x; r.mv[5] = b.y; r.mv[6] = b.z; r.mv[7] = b.w;
    } else {
      _Pragma("unroll") for (int i = 0; i < 8; ++i) if (i < r.cnt) r.mv[i] = m[i];
    }
  } else {
    const __nv_bfloat16* m = reinterpret_cast<const __nv_bfloat16*>(t.m) + i0;
    if (r.svec) unpack8(__ldcs(reinterpret_cast<const uint4*>(m)), r.mv);
    else { _Pragma("unroll") for (int i = 0; i < 8; ++i) if (i < r.cnt) r.mv[i] = __bfloat162float(m[i]); }
  }
  if (t.state_fp32 >= 1) {
    const float* v = reinterpret_cast<const float*>(t.v) + i0;
    if (r.svec) {
      const float4 c = __ldcs(reinterpret_cast<const float4*>(v)), d = __ldcs(reinterpret_cast<const float4*>(v) + 1);
      r.vv[0] = c.x; r.vv[1] = c.y; r.vv[2] = c.z; r.vv[3] = c.w; r.vv[4] = d.x; r.vv[5] = d.y; r.vv[6] = d.z; r.vv[7] = d.w;
    } else {
      _Pragma("unroll") for (int i = 0; i < 8; ++i) if (i < r.cnt) r.vv[i] = v[i];
    }
  } else {
    const __nv_bfloat16* v = reinterpret_cast<const __nv_bfloat16*>(t.v) + i0;
    if (r.svec) unpack8(__ldcs(reinterpret_cast<const uint4*>(v)), r.vv);
    else { _Pragma("unroll") for (int i = 0; i < 8; ++i) if (i < r.cnt) r.vv[i] = __bfloat162float(v[i]); }
  }
}
__device__ __forceinline__ void adam_update_store(const RtpAdamTensor& t, AdamRegs& r, float lr, float beta1, float beta2,
                                                  float eps, float weight_decay, int adamw, float clip_value,
                                                  float grad_scale, float step_size, float inv_sqrt_bc2) {
  if (r.cnt == 0) return;
  _Pragma("unroll") for (int i = 0; i < 8; ++i) if (i < r.cnt) {
    adam_element(r.pv[i], r.gv[i], r.mv[i], r.vv[i], lr * t.lr_mult * weight_decay, beta1, beta2, eps, weight_decay, adamw,
                 clip_value, grad_scale, step_size, inv_sqrt_bc2);
  }
  __nv_bfloat16* p = reinterpret_cast<__nv_bfloat16*>(t.p) + r.i0;
  if (r.vec) __stcs(reinterpret_cast<uint4*>(p), pack8(r.pv));
  else { _Pragma("unroll") for (int i = 0; i < 8; ++i) if (i < r.cnt) p[i] = __float2bfloat16(r.pv[i]); }
  if (t.state_fp32 == 1) {
    float* m = reinterpret_cast<float*>(t.m) + r.i0;
    if (r.svec) {
      __stcs(reinterpret_cast<float4*>(m), make_float4(r.mv[0], r.mv[1], r.mv[2], r.mv[3]));
      __stcs(reinterpret_cast<float4*>(m) + 1, make_float4(r.mv[4], r.mv[5], r.mv[6], r.mv[7]));
    } else {
      _Pragma("unroll") for (int i = 0; i < 8; ++i) if (i < r.cnt) m[i] = r.mv[i];
    }
  } else {
    __nv_bfloat16* m = reinterpret_cast<__nv_bfloat16*>(t.m) + r.i0;
    if (r.svec) __stcs(reinterpret_cast<uint4*>(m), pack8(r.mv));
    else { _Pragma("unroll") for (int i = 0; i < 8; ++i) if (i < r.cnt) m[i] = __float2bfloat16(r.mv[i]); }
  }
  if (t.state_fp32 >= 1) {
    float* v = reinterpret_cast<float*>(t.v) + r.i0;
    if (r.svec) {
      __stcs(reinterpret_cast<float4*>(v), make_float4(r.vv[0], r.vv[1], r.vv[2], r.vv[3]));
      __stcs(reinterpret_cast<float4*>(v) + 1, make_float4(r.vv[4], r.vv[5], r.vv[6], r.vv[7]));
    } else {
      _Pragma("unroll") for (int i = 0; i < 8; ++i) if (i < r.cnt) v[i] = r.vv[i];
    }
  } else {
    __nv_bfloat16* v = reinterpret_cast<__nv_bfloat16*>(t.v) + r.i0;
    if (r.svec) __stcs(reinterpret_cast<uint4*>(v), pack8(r.vv));
    else { _Pragma("unroll") for (int i = 0; i < 8; ++i) if (i < r.cnt) v[i] = __float2bfloat16(r.vv[i]); }
  }
}

// The same update on a full chunk with 16-byte aligned buffers, for one moment policy (CODE as in state_fp32).  What
// bounds it is memory (18 bytes per parameter with mixed moments), so every load of a thread has to be in flight before
// the first is used: the groups stay packed as loaded (20 registers a group with mixed moments) and are unpacked two
// elements at a time.  Unpacked on arrival they take 32 registers a group, two groups did not fit beside each other in
// the 64 registers that four blocks per SM leave, and the loads went out one group after the other.  315 M parameters,
// mixed moments: 1200 -> 819 us (4.7 -> 6.9 TB/s); 26 M: 114 -> 75 us.
template <int CODE>
struct AdamVec {
  static constexpr int MW = CODE == 1 ? 2 : 1, VW = CODE >= 1 ? 2 : 1;   // 16-byte words of eight moments
  uint4 p, g, m[MW], v[VW];
};
__device__ __forceinline__ float word_at(const uint4& u, int i) {
  return __uint_as_float(i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w);
}
__device__ __forceinline__ float bf_at(const uint4& u, int i) {
  const uint32_t w = (i >> 1) == 0 ? u.x : (i >> 1) == 1 ? u.y : (i >> 1) == 2 ? u.z : u.w;
  return (i & 1) ? bf16_hi(w) : bf16_lo(w);
}
__device__ __forceinline__ void word_set(uint4& u, int i, uint32_t w) {
  if (i == 0) u.x = w; else if (i == 1) u.y = w; else if (i == 2) u.z = w; else u.w = w;
}
template <int CODE>
__device__ __forceinline__ void adam_chunk(const RtpAdamTensor& t, long long i0, float lr, float beta1, float beta2, float eps,
                                           float weight_decay, int adamw, float clip_value, float grad_scale, float step_size,
                                           float inv_sqrt_bc2) {
  using Vec = AdamVec<CODE>;
  Vec r[kAdamGroups];
#pragma unroll
  for (int u = 0; u < kAdamGroups; ++u) {
    const long long i = i0 + u * 2048;
    r[u].p = __ldcs(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(t.p) + i));
    r[u].g = __ldcs(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(t.g) + i));
#pragma unroll
    for (int w = 0; w < Vec::MW; ++w)
      r[u].m[w] = __ldcs(reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(t.m) + i * 2 * Vec::MW) + w);
#pragma unroll
    for (int w = 0; w < Vec::VW; ++w)
      r[u].v[w] = __ldcs(reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(t.v) + i * 2 * Vec::VW) + w);
  }
#pragma unroll
  for (int u = 0; u < kAdamGroups; ++u) {
    const long long i = i0 + u * 2048;
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      float pv[2], mv[2], vv[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        pv[e] = bf_at(r[u].p, k + e);
        mv[e] = CODE == 1 ? word_at(r[u].m[(k + e) / 4 % Vec::MW], (k + e) & 3) : bf_at(r[u].m[0], k + e);
        vv[e] = CODE >= 1 ? word_at(r[u].v[(k + e) / 4 % Vec::VW], (k + e) & 3) : bf_at(r[u].v[0], k + e);
        adam_element(pv[e], bf_at(r[u].g, k + e), mv[e], vv[e], lr * t.lr_mult * weight_decay, beta1, beta2, eps, weight_decay,
                     adamw, clip_value, grad_scale, step_size, inv_sqrt_bc2);
      }
      word_set(r[u].p, k / 2, pack_bf16(pv[0], pv[1]));
      if (CODE == 1) {
        word_set(r[u].m[k / 4 % Vec::MW], k & 3, __float_as_uint(mv[0]));
        word_set(r[u].m[k / 4 % Vec::MW], (k & 3) + 1, __float_as_uint(mv[1]));
      } else {
        word_set(r[u].m[0], k / 2, pack_bf16(mv[0], mv[1]));
      }
      if (CODE >= 1) {
        word_set(r[u].v[k / 4 % Vec::VW], k & 3, __float_as_uint(vv[0]));
        word_set(r[u].v[k / 4 % Vec::VW], (k & 3) + 1, __float_as_uint(vv[1]));
      } else {
        word_set(r[u].v[0], k / 2, pack_bf16(vv[0], vv[1]));
      }
    }
    __stcs(reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(t.p) + i), r[u].p);
#pragma unroll
    for (int w = 0; w < Vec::MW; ++w)
      __stcs(reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(t.m) + i * 2 * Vec::MW) + w, r[u].m[w]);
#pragma unroll
    for (int w = 0; w < Vec::VW; ++w)
      __stcs(reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(t.v) + i * 2 * Vec::VW) + w, r[u].v[w]);
  }
}

// One block = kAdamGroups x 2048 elements of one tensor; every thread owns one group of 8 elements in each 2048-element
// sub-chunk.  The last chunk of a tensor and unaligned buffers take the element-wise path.
__global__ void __launch_bounds__(256, 4) adam_kernel(const RtpAdamTensor* __restrict__ tensors,
                                                   const int* __restrict__ block_start, int ntensors,
                                                   const long long* __restrict__ step_ptr, float lr, float beta1,
                                                   float beta2, float eps, float weight_decay, int adamw,
                                                   float clip_value, float grad_scale,
                                                   const int* __restrict__ block_tensor) {
  // locate the tensor this block works on: one load from the per-block table when the caller provides it
  int lo = 0, hi = ntensors - 1;
  if (block_tensor) {
    lo = block_tensor[blockIdx.x];
  } else {
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (block_start[mid] <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
  }
  const RtpAdamTensor t = tensors[lo];
  const long long step = *step_ptr;
  const float bc1 = 1.f - powf(beta1, (float)step);
  const float bc2 = 1.f - powf(beta2, (float)step);
  const float step_size = lr * t.lr_mult / bc1;
  const float inv_sqrt_bc2 = rsqrtf(bc2);
  const long long base = (long long)((int)blockIdx.x - block_start[lo]) * (256 * 8 * kAdamGroups);
  const uintptr_t addr = reinterpret_cast<uintptr_t>(t.p) | reinterpret_cast<uintptr_t>(t.g) |
                         reinterpret_cast<uintptr_t>(t.m) | reinterpret_cast<uintptr_t>(t.v);
  if (base + 256 * 8 * kAdamGroups <= t.n && (addr & 15) == 0) {
    const long long i0 = base + threadIdx.x * 8;
#define RTP_ADAM_CHUNK(CODE) adam_chunk<CODE>(t, i0, lr, beta1, beta2, eps, weight_decay, adamw, clip_value, grad_scale, \
                                              step_size, inv_sqrt_bc2)
    if (t.state_fp32 == 2) RTP_ADAM_CHUNK(2); else if (t.state_fp32 == 1) RTP_ADAM_CHUNK(1); else RTP_ADAM_CHUNK(0);
#undef RTP_ADAM_CHUNK
    return;
  }
#pragma unroll 1
  for (int u = 0; u < kAdamGroups; ++u) {
    AdamRegs r;
    adam_load(t, base + u * (256 * 8) + threadIdx.x * 8, r);
    adam_update_store(t, r, lr, beta1, beta2, eps, weight_decay, adamw, clip_value, grad_scale, step_size, inv_sqrt_bc2);
  }
}

// ------------------------------------------------------------------------------------------------
// Causal softmax over rows of a score matrix stack [rows_total, S] (row r belongs to query i = r % S).
// In place: p[i, j] = softmax_j(scale * s[i, j]) for j <= i, 0 for j > i (those entries may hold anything).
// ------------------------------------------------------------------------------------------------
__global__ void causal_softmax_kernel(__nv_bfloat16* __restrict__ s, long long rows, int S, float scale) {
  __shared__ float red[32];
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    __nv_bfloat16* p = s + row * S;
    const int i = (int)(row % S);
    float mx = -INFINITY;
    for (int c = threadIdx.x * 8; c <= i; c += blockDim.x * 8) {
      float v[8];
      unpack8(*reinterpret_cast<const uint4*>(p + c), v);
#pragma unroll
      for (int k = 0; k < 8; ++k) if (c + k <= i) mx = fmaxf(mx, v[k] * scale);
    }
    mx = block_max(mx, red);
    float se = 0.f;
    for (int c = threadIdx.x * 8; c <= i; c += blockDim.x * 8) {
      float v[8];
      unpack8(*reinterpret_cast<const uint4*>(p + c), v);
#pragma unroll
      for (int k = 0; k < 8; ++k) if (c + k <= i) se += __expf(v[k] * scale - mx);
    }
    se = block_sum(se, red);
    const float inv = 1.f / se;
    for (int c = threadIdx.x * 8; c < S; c += blockDim.x * 8) {
      float v[8];
      if (c <= i) unpack8(*reinterpret_cast<const uint4*>(p + c), v);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = (c + k <= i) ? __expf(v[k] * scale - mx) * inv : 0.f;
      *reinterpret_cast<uint4*>(p + c) = pack8(v);
    }
    __syncthreads();
  }
}
// dS = scale * P * (dP - sum_j P dP), written over dP; entries above the diagonal become 0.
__global__ void causal_softmax_bwd_kernel(const __nv_bfloat16* __restrict__ pm, __nv_bfloat16* __restrict__ dp,
                                          long long rows, int S, float scale) {
  __shared__ float red[32];
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const __nv_bfloat16* p = pm + row * S;
    __nv_bfloat16* d = dp + row * S;
    const int i = (int)(row % S);
    float dot = 0.f;
    for (int c = threadIdx.x * 8; c <= i; c += blockDim.x * 8) {
      float a[8], b[8];
      unpack8(*reinterpret_cast<const uint4*>(p + c), a);
      unpack8(*reinterpret_cast<const uint4*>(d + c), b);
#pragma unroll
      for (int k = 0; k < 8; ++k) if (c + k <= i) dot += a[k] * b[k];
    }
    dot = block_sum(dot, red);
    for (int c = threadIdx.x * 8; c < S; c += blockDim.x * 8) {
      float a[8], b[8], o[8];
      if (c <= i) {
        unpack8(*reinterpret_cast<const uint4*>(p + c), a);
        unpack8(*reinterpret_cast<const uint4*>(d + c), b);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = (c + k <= i) ? scale * a[k] * (b[k] - dot) : 0.f;
      *reinterpret_cast<uint4*>(d + c) = pack8(o);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------------------
// Activations (n % 8 == 0).  mode 0: y = gelu(x) (erf form).  mode 1: y = silu(g) * u with g, u the two column halves
// selected by pointers.  Backward kernels recompute from the saved pre-activations.
// ------------------------------------------------------------------------------------------------
// Normal distribution function from the complementary error function's Chebyshev fit of W. H. Press et al., Numerical
// Recipes (erfcc, fractional error below 1.2e-7 everywhere): a reciprocal, an exponential and ten multiply-adds without a
// branch, and no cancellation in the lower tail, where 1 + erff(x) loses its digits.  With erff the kernels were bound by
// instructions, not memory: 67 M elements forward 77 -> 54 us, backward 92 -> 69 us; results that are the exactly rounded
// ones, inputs N(0, 4): forward 98.6 -> 100.0 %, gradient 99.5 -> 100.0 %.
__device__ __forceinline__ float normal_cdf(float x) {
  const float z = fabsf(x) * 0.70710678118654752f;
  const float t = __fdividef(1.f, fmaf(0.5f, z, 1.f));
  float p = 0.17087277f;
  p = fmaf(p, t, -0.82215223f);
  p = fmaf(p, t, 1.48851587f);
  p = fmaf(p, t, -1.13520398f);
  p = fmaf(p, t, 0.27886807f);
  p = fmaf(p, t, -0.18628806f);
  p = fmaf(p, t, 0.09678418f);
  p = fmaf(p, t, 0.37409196f);
  p = fmaf(p, t, 1.00002368f);
  p = fmaf(p, t, -1.26551223f);
  const float tail = 0.5f * t * __expf(fmaf(-z, z, p));
  return x >= 0.f ? 1.f - tail : tail;
}
__device__ __forceinline__ float gelu_f(float x) { return x * normal_cdf(x); }
__device__ __forceinline__ float gelu_grad_f(float x) {
  return normal_cdf(x) + x * 0.3989422804014327f * __expf(-0.5f * x * x);
}
__global__ void gelu_fwd_kernel(const __nv_bfloat16* x, __nv_bfloat16* y, long long n) {
  const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  float v[8];
  unpack8(*reinterpret_cast<const uint4*>(x + i), v);
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = gelu_f(v[k]);
  *reinterpret_cast<uint4*>(y + i) = pack8(v);
}
__global__ void gelu_bwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* dy, __nv_bfloat16* dx, long long n) {
  const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  float v[8], g[8];
  unpack8(*reinterpret_cast<const uint4*>(x + i), v);
  unpack8(*reinterpret_cast<const uint4*>(dy + i), g);
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = g[k] * gelu_grad_f(v[k]);
  *reinterpret_cast<uint4*>(dx + i) = pack8(v);
}
// g, u: [rows, cols] windows with pitch ld (elements); y dense [rows, cols]
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* g, const __nv_bfloat16* u, long long ld, __nv_bfloat16* y,
                                  long long rows, int cols) {
  const long long it = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int per = cols / 8;
  if (it >= rows * per) return;
  const long long r = it / per;
  const int c = (int)(it % per) * 8;
  float a[8], b[8];
  unpack8(*reinterpret_cast<const uint4*>(g + r * ld + c), a);
  unpack8(*reinterpret_cast<const uint4*>(u + r * ld + c), b);
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = a[k] / (1.f + __expf(-a[k])) * b[k];
  *reinterpret_cast<uint4*>(y + r * cols + c) = pack8(a);
}
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* g, const __nv_bfloat16* u, long long ld, const __nv_bfloat16* dy,
                                  __nv_bfloat16* dg, __nv_bfloat16* du, long long ldo, long long rows, int cols) {
  const long long it = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int per = cols / 8;
  if (it >= rows * per) return;
  const long long r = it / per;
  const int c = (int)(it % per) * 8;
  float a[8], b[8], d[8], og[8], ou[8];
  unpack8(*reinterpret_cast<const uint4*>(g + r * ld + c), a);
  unpack8(*reinterpret_cast<const uint4*>(u + r * ld + c), b);
  unpack8(*reinterpret_cast<const uint4*>(dy + r * cols + c), d);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float sg = 1.f / (1.f + __expf(-a[k]));
    const float silu = a[k] * sg;
    ou[k] = d[k] * silu;
    og[k] = d[k] * b[k] * (sg + silu * (1.f - sg));
  }
  *reinterpret_cast<uint4*>(dg + r * ldo + c) = pack8(og);
  *reinterpret_cast<uint4*>(du + r * ldo + c) = pack8(ou);
}

// ------------------------------------------------------------------------------------------------
// MoE token movement by index (top-2): slot[s, k] is the destination row (expert * capacity + position) of choice k
// of token s, or -1.  One warp per (token, choice).  M % 8 == 0.  fill (may be null): for each group of `cap` destination rows
// one more than its last row that a token went to (zeroed by the caller).
// ------------------------------------------------------------------------------------------------
__global__ void moe_scatter_kernel(const __nv_bfloat16* __restrict__ src, const int* __restrict__ slot,
                                   const float* __restrict__ scale, __nv_bfloat16* __restrict__ dst, int S, int M,
                                   int* fill, int cap) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= 2 * S) return;
  const int sl = slot[w];
  if (sl < 0) return;
  if (fill && lane == 0) {
    const int e = sl / cap, n = sl - e * cap + 1;
    if (n > *reinterpret_cast<volatile int*>(fill + e)) atomicMax(fill + e, n);      // few get here: slots rise with the tokens
  }
  const float sc = scale ? scale[w] : 1.f;
  const __nv_bfloat16* a = src + (size_t)(w >> 1) * M;
  __nv_bfloat16* d = dst + (size_t)sl * M;
  for (int c = lane * 8; c < M; c += 256) {
    float v[8];
    unpack8(*reinterpret_cast<const uint4*>(a + c), v);
    if (scale) {
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] *= sc;
    }
    *reinterpret_cast<uint4*>(d + c) = pack8(v);
  }
}
__global__ void moe_gather_kernel(const __nv_bfloat16* __restrict__ src, const int* __restrict__ slot,
                                  const float* __restrict__ scale, __nv_bfloat16* __restrict__ dst, int S, int M) {
  const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (s >= S) return;
  const int s0 = slot[2 * s], s1 = slot[2 * s + 1];
  const float g0 = scale ? scale[2 * s] : 1.f, g1 = scale ? scale[2 * s + 1] : 1.f;
  for (int c = lane * 8; c < M; c += 256) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, v[8];
    if (s0 >= 0) {
      unpack8(*reinterpret_cast<const uint4*>(src + (size_t)s0 * M + c), v);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += g0 * v[k];
    }
    if (s1 >= 0) {
      unpack8(*reinterpret_cast<const uint4*>(src + (size_t)s1 * M + c), v);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += g1 * v[k];
    }
    *reinterpret_cast<uint4*>(dst + (size_t)s * M + c) = pack8(acc);
  }
}
// out[s, k] = <a[s, :], b[slot[s, k], :]>
__global__ void moe_rowdot_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                                  const int* __restrict__ slot, float* __restrict__ out, int S, int M) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= 2 * S) return;
  const int sl = slot[w];
  float acc = 0.f;
  if (sl >= 0) {
    const __nv_bfloat16* x = a + (size_t)(w >> 1) * M;
    const __nv_bfloat16* y = b + (size_t)sl * M;
    for (int c = lane * 8; c < M; c += 256) {
      float u[8], v[8];
      unpack8(*reinterpret_cast<const uint4*>(x + c), u);
      unpack8(*reinterpret_cast<const uint4*>(y + c), v);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc += u[k] * v[k];
    }
  }
  acc = warp_sum(acc);
  if (lane == 0) out[w] = acc;
}

// out = a + b (bf16), n % 8 == 0 handled vectorised, tail scalar
__global__ void add_kernel(const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* out, long long n) {
  const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * 8;
  if (i + 8 <= n) {
    float x[8], y[8];
    unpack8(*reinterpret_cast<const uint4*>(a + i), x);
    unpack8(*reinterpret_cast<const uint4*>(b + i), y);
    for (int k = 0; k < 8; ++k) x[k] += y[k];
    *reinterpret_cast<uint4*>(out + i) = pack8(x);
  } else {
    for (long long k = i; k < n; ++k) out[k] = __float2bfloat16(__bfloat162float(a[k]) + __bfloat162float(b[k]));
  }
}
// fp32 vector -> bf16 (used for LayerNorm parameter gradients accumulated in fp32)
__global__ void cast_f32_bf16_kernel(const float* in, __nv_bfloat16* out, long long n, float scale) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16(in[i] * scale);
}
// sum of fp32 vector * scale (/ *divisor) -> out[0] (single block)
__global__ void sum_kernel(const float* in, float* out, int n, float scale, const float* __restrict__ divisor) {
  pdl_prologue();
  __shared__ float red[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += in[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) out[0] = divisor ? s * scale / *divisor : s * scale;
}

}  // namespace

extern "C" {

const char* rtp_kernels_last_error(void) { return k_err.c_str(); }

int rtp_norm_fwd(const void* x, const void* sub, const void* gamma, const void* beta, void* h_out, void* y,
                 float* mean, float* rstd, int M, int D, float eps, int rms, float drop_p, unsigned long long seed,
                 unsigned long long offset, const unsigned long long* step_ptr, void* stream) {
  if (D % 8 || D > 8192) { k_err = "norm: D must be a multiple of 8 and at most 8192"; return -1; }
  const float ds = drop_p > 0.f ? 1.f / (1.f - drop_p) : 1.f;
#define RTP_NORM_FWD(T, NG, PER_SM)                                                                                   \
  rtp::launch_k(norm_fwd_kernel<T, NG>, dim3(std::min(M, 148 * PER_SM)), dim3(T), 0, (cudaStream_t)stream,            \
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)sub, (const __nv_bfloat16*)gamma, (const __nv_bfloat16*)beta,    \
      (__nv_bfloat16*)h_out, (__nv_bfloat16*)y, mean, rstd, M, D, eps, rms, host_thresh(drop_p), ds, seed, offset,    \
      step_ptr)
  if (D <= 1024) RTP_NORM_FWD(128, 1, 7); else if (D <= 2048) RTP_NORM_FWD(256, 1, 4);
  else if (D <= 4096) RTP_NORM_FWD(256, 2, 2); else if (D <= 6144) RTP_NORM_FWD(256, 3, 2); else RTP_NORM_FWD(256, 4, 2);
#undef RTP_NORM_FWD
  LAUNCH_CHECK("norm_fwd");
  return 0;
}
// Threads a row and rows in flight per group of a backward launch: no more rows than leave every SM a block or two, one where there
// are fewer rows than SMs (64 x 4096 with dropout, two rows 7.5 us, one 6.9).
struct NormBwdShape { int T, R; };
static NormBwdShape norm_bwd_shape(int M, int D) {
  if (D <= 256) return {32, M <= 2368 ? 1 : 4};
  if (D <= 512) return {64, M <= 148 ? 1 : M <= 1184 ? 2 : 4};
  if (D <= 1024) return {128, M <= 148 ? 1 : M <= 592 ? 2 : 4};
  if (D <= 2048) return {256, M <= 1024 || M >= 4096 ? 2 : 4};
  if (D <= 4096) return {256, M <= 148 ? 1 : 2};
  return {256, 1};
}
// Few blocks: every block ends with one vector atomic per 4 columns of dgamma / dbeta.  Up to 1024 wide rows one block per
// SM (256 x 2048 256 blocks 10.3 us, 128 with two rows each 7.4; 1024 x 3072 256 blocks 18.3, 148 14.6), else two.
static int norm_bwd_blocks(int M, int D) {
  const NormBwdShape s = norm_bwd_shape(M, D);
  const int rows = 256 / s.T * s.R;
  return std::min((M + rows - 1) / rows, M <= 1024 && D > 1024 ? 148 : 296);
}
// part_pitch as in norm_bwd_kernel
static int norm_bwd_launch(const void* dy, const void* h, const void* gamma, const float* mean, const float* rstd, void* dx,
                           void* dsub, float* dgamma, float* dbeta, int M, int D, int rms, float drop_p, unsigned long long seed,
                           unsigned long long offset, const void* dres, const unsigned long long* step_ptr, int part_pitch,
                           void* stream) {
  if (D % 8 || D > 8192) { k_err = "norm: D must be a multiple of 8 and at most 8192"; return -1; }
  const float ds = drop_p > 0.f ? 1.f / (1.f - drop_p) : 1.f;
  const int vec_atomics = ((reinterpret_cast<uintptr_t>(dgamma) | reinterpret_cast<uintptr_t>(dbeta)) & 15) == 0;
  const int R = norm_bwd_shape(M, D).R;
#define RTP_NORM_BWD(T, NG, R, AHEAD)                                                                                 \
  rtp::launch_k(norm_bwd_kernel<T, NG, R, AHEAD>, dim3(norm_bwd_blocks(M, D)), dim3(256), 0, (cudaStream_t)stream,     \
      (const __nv_bfloat16*)dy, (const __nv_bfloat16*)h, (const __nv_bfloat16*)gamma, mean, rstd, (__nv_bfloat16*)dx, \
      (__nv_bfloat16*)dsub, dgamma, dbeta, M, D, rms, host_thresh(drop_p), ds, seed, offset,                          \
      (const __nv_bfloat16*)dres, step_ptr, vec_atomics, part_pitch)
  if (D <= 256) { if (R == 1) RTP_NORM_BWD(32, 1, 1, false); else RTP_NORM_BWD(32, 1, 4, false); }
  else if (D <= 512) {
    if (R == 1) RTP_NORM_BWD(64, 1, 1, false); else if (R == 2) RTP_NORM_BWD(64, 1, 2, false);
    else RTP_NORM_BWD(64, 1, 4, false);
  } else if (D <= 1024) {
    if (R == 1) RTP_NORM_BWD(128, 1, 1, false); else if (R == 2) RTP_NORM_BWD(128, 1, 2, false);
    else RTP_NORM_BWD(128, 1, 4, false);
  } else if (D <= 2048) {
    if (M <= 1024) RTP_NORM_BWD(256, 1, 2, false); else if (R == 4) RTP_NORM_BWD(256, 1, 4, false);
    else RTP_NORM_BWD(256, 1, 2, true);
  } else if (D <= 4096) { if (R == 1) RTP_NORM_BWD(256, 2, 1, false); else RTP_NORM_BWD(256, 2, 2, false); }
  else if (D <= 6144) RTP_NORM_BWD(256, 3, 1, false); else RTP_NORM_BWD(256, 4, 1, false);
#undef RTP_NORM_BWD
  LAUNCH_CHECK("norm_bwd");
  return 0;
}
int rtp_norm_bwd(const void* dy, const void* h, const void* gamma, const float* mean, const float* rstd, void* dx,
                 void* dsub, float* dgamma, float* dbeta, int M, int D, int rms, float drop_p,
                 unsigned long long seed, unsigned long long offset, const void* dres,
                 const unsigned long long* step_ptr, void* stream) {
  return norm_bwd_launch(dy, h, gamma, mean, rstd, dx, dsub, dgamma, dbeta, M, D, rms, drop_p, seed, offset, dres, step_ptr, 0,
                         stream);
}
unsigned long long rtp_norm_bwd_scratch(int M, int D, int has_beta) {
  return (unsigned long long)norm_bwd_blocks(M, D) * (has_beta ? 2 : 1) * D * sizeof(float);
}
int rtp_norm_bwd_params(const void* dy, const void* h, const void* gamma, const float* mean, const float* rstd, void* dx,
                        void* dgamma, void* dbeta, float* scratch, int M, int D, int rms, const void* dres, void* stream) {
  if (M <= 0) { k_err = "norm backward: no rows"; return -1; }
  if (reinterpret_cast<uintptr_t>(scratch) & 15) { k_err = "norm backward: scratch must be 16-byte aligned"; return -1; }
  const int pitch = dbeta ? 2 * D : D;
  if (norm_bwd_launch(dy, h, gamma, mean, rstd, dx, nullptr, scratch, dbeta ? scratch + D : nullptr, M, D, rms, 0.f, 0, 0, dres,
                      nullptr, pitch, stream))
    return -1;
  rtp::launch_k(norm_param_grads_kernel, dim3((D + 63) / 64, dbeta ? 2 : 1), dim3(256), 0, (cudaStream_t)stream, (const float*)scratch,
                norm_bwd_blocks(M, D), pitch, D, (__nv_bfloat16*)dgamma, (__nv_bfloat16*)dbeta);
  LAUNCH_CHECK("norm_param_grads");
  return 0;
}
int rtp_cross_entropy_scaled(void* logits, long long ld, const long long* target, float* loss, int M, int V, float grad_scale,
                             const float* scale_ptr, long long ignore_index, int write_grad, void* grad, long long ldg,
                             void* stream) {
  if (V % 8 || ld % 8 || (grad && ldg % 8)) { k_err = "cross_entropy: V and the row pitches must be multiples of 8"; return -1; }
  if (M > 0 && V > 0 && V <= kCeMaxV) {
    __nv_bfloat16* out = (__nv_bfloat16*)(write_grad ? (grad ? grad : logits) : nullptr);
    const long long ldo = grad ? ldg : ld;
#define RTP_CE(KERNEL, T, X)                                                                                         \
  rtp::launch_k(KERNEL<T, X>, dim3(M), dim3(T), 0, (cudaStream_t)stream, (const __nv_bfloat16*)logits, ld, target,   \
                loss, V, grad_scale, scale_ptr, ignore_index, out, ldo)
#define RTP_CE_HELD(T, WORDS) RTP_CE(ce_row_kernel, T, WORDS)
    // Held rows pay where a block has at most eight words a thread to hold, and for the loss alone only where a few rows
    // leave the SMs idle (256 x 24576 4.4 us, read again 5.8; 512 x 24576 7.4 and 7.3; 2048 x 8192 8.1 and 7.9).
    // As many 16-byte words a thread as the row needs, one kernel for each number: words that the row does not have cost
    // registers.  Against numbers rounded up to a few: 8192 x 5120 42.6 -> 36.6 us, 12288 89.8 -> 83.1.
    if (V > 32768) { if (out) RTP_CE(ce_stream_kernel, 512, true); else RTP_CE(ce_stream_kernel, 512, false); }
    else if (!out && V > 16384 && M >= 512) RTP_CE(ce_stream_kernel, 512, false);
    else if (!out && V > 8192 && V <= 16384 && M >= 2048) RTP_CE(ce_stream_kernel, 256, false);
    else switch (V <= 16384 ? (V + 2047) / 2048 : 4 + (V + 4095) / 4096) {
      case 1: RTP_CE_HELD(256, 1); break; case 2: RTP_CE_HELD(256, 2); break; case 3: RTP_CE_HELD(256, 3); break;
      case 4: RTP_CE_HELD(256, 4); break; case 5: RTP_CE_HELD(256, 5); break; case 6: RTP_CE_HELD(256, 6); break;
      case 7: RTP_CE_HELD(256, 7); break; case 8: RTP_CE_HELD(256, 8); break;
      case 9: RTP_CE_HELD(512, 5); break; case 10: RTP_CE_HELD(512, 6); break; case 11: RTP_CE_HELD(512, 7); break;
      default: RTP_CE_HELD(512, 8); break;
    }
#undef RTP_CE_HELD
#undef RTP_CE
    LAUNCH_CHECK("cross_entropy");
    return 0;
  }
  if (scale_ptr) { k_err = "cross_entropy: a device-side scale needs rows of at most 65536 logits"; return -1; }
  // without dependent launch: 512 x 100352 103 us, with it 119 (its blocks wait where others of the same kernel run)
  const int grid = M < 148 * 8 ? M : 148 * 8;
  ce_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)logits, ld, target, loss, M, V, grad_scale, ignore_index,
                                                    write_grad, (__nv_bfloat16*)grad, ldg);
  LAUNCH_CHECK("cross_entropy");
  return 0;
}
int rtp_ce_count(const long long* target, int M, long long ignore_index, float* out2, void* stream) {
  rtp::launch_k(ce_count_kernel, dim3(1), dim3(1024), 0, (cudaStream_t)stream, target, M, ignore_index, out2);
  LAUNCH_CHECK("ce_count");
  return 0;
}
int rtp_scale_unless_one(void* g, const float* scale, long long n, void* stream) {
  if (n % 8 || (reinterpret_cast<uintptr_t>(g) & 15)) { k_err = "scale: n must be a multiple of 8 and the buffer aligned"; return -1; }
  if (n == 0) return 0;
  const long long blocks = (n / 8 + 255) / 256;
  scale_unless_one_kernel<<<(int)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)g, scale,
                                                                                                     n / 8);
  LAUNCH_CHECK("scale");
  return 0;
}
int rtp_embed_fwd(const void* table, const long long* ids, const void* pe, long long ld_pe, int tokens_per_pos,
                  void* out, long long ld_out, int col_off, int T, int Ds, int D, float scale, float drop_p,
                  unsigned long long seed, unsigned long long offset, const unsigned long long* step_ptr,
                  void* stream) {
  if (Ds % 8 || col_off % 8 || ld_out % 8) { k_err = "embed: widths must be multiples of 8"; return -1; }
  const long long total = (long long)T * (Ds / 8);
  if (total <= 0) return 0;
  int grid = (int)((total + 255) / 256 > 148 * 16 ? 148 * 16 : (total + 255) / 256);
  const float ds = drop_p > 0.f ? 1.f / (1.f - drop_p) : 1.f;
  rtp::launch_k(embed_fwd_kernel, dim3(grid), dim3(256), 0, (cudaStream_t)stream, (const __nv_bfloat16*)table, ids,
                (const __nv_bfloat16*)pe, ld_pe, tokens_per_pos, (__nv_bfloat16*)out, ld_out, col_off, T, Ds, D, scale,
                host_thresh(drop_p), ds, seed, offset, step_ptr);
  LAUNCH_CHECK("embed_fwd");
  return 0;
}
int rtp_embed_bwd(void* gtable, const long long* ids, const void* dy, long long ld_dy, int col_off, int T, int Ds,
                  int D, float scale, float drop_p, unsigned long long seed, unsigned long long offset,
                  const unsigned long long* step_ptr, void* stream) {
  return rtp_embed_bwd_blocks(gtable, ids, dy, ld_dy, col_off, T, Ds, D, scale, drop_p, seed, offset, step_ptr, 0, 0, stream);
}
int rtp_embed_bwd_blocks(void* gtable, const long long* ids, const void* dy, long long ld_dy, int col_off, int T, int Ds,
                         int D, float scale, float drop_p, unsigned long long seed, unsigned long long offset,
                         const unsigned long long* step_ptr, int blk_cols, int V, void* stream) {
  if (Ds % 8 || col_off % 8 || ld_dy % 8 || blk_cols % 8 || (blk_cols > 0 && Ds % blk_cols)) {
    k_err = "embed: widths must be multiples of 8";
    return -1;
  }
  const long long total = (long long)T * (Ds / 8);
  int grid = (int)((total + 255) / 256);
  if (grid > 148 * 16) grid = 148 * 16;
  const float ds = drop_p > 0.f ? 1.f / (1.f - drop_p) : 1.f;
  rtp::launch_k(embed_bwd_kernel, dim3(grid), dim3(256), 0, (cudaStream_t)stream, (__nv_bfloat16*)gtable, ids,
                (const __nv_bfloat16*)dy, ld_dy, col_off, T, Ds, D, scale, host_thresh(drop_p), ds, seed, offset, step_ptr,
                blk_cols, V);
  LAUNCH_CHECK("embed_bwd");
  return 0;
}
static int g_attn_tc = 1;
void rtp_set_attn_tc(int on) { g_attn_tc = on ? 1 : 0; }
static size_t attn_smem(int S, bool bwd) {
  size_t f = (size_t)(bwd ? 4 : 3) * S * kHd + (size_t)(bwd ? 2 : 1) * S * (S + 1);
  return f * sizeof(float);
}
// A 2 x 2 tile of scores per thread and round, and no more threads than there is work for where blocks queue for an SM:
// 32 x 32 blocks of S = 4, forward / backward with 128 and 256 threads 3.8 / 5.7 and 5.5 / 8.2 us, S = 12 7.0 / 12.4 and
// 8.0 / 13.3; 4 blocks of S = 8 3.3 / 4.9 and 2.9 / 4.0.
static int attn_threads(int S, int blocks) {
  if (S <= 4 || (S <= 12 && blocks > 592)) return 128;
  return S <= 40 ? 256 : 512;
}
int rtp_attn_small_fwd(const void* qkv, void* out, int S, int B, int heads, int nshard, int causal, float sm_scale,
                       float drop_p, unsigned long long seed, unsigned long long offset,
                       const unsigned long long* step_ptr, void* stream) {
  if (g_attn_tc && rtp_attn_tc_supported(S, heads, nshard)) {
    const int rc = rtp_attn_tc_fwd(qkv, out, S, B, heads, nshard, causal, sm_scale, drop_p, seed, offset, step_ptr, stream);
    if (rc) k_err = rtp_attn_tc_last_error();
    return rc;
  }
  if (S > 128 || heads % nshard) { k_err = "attn_small: S must be <= 128 and heads divisible by shards"; return -1; }
  const size_t smem = attn_smem(S, false);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(attn_small_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return kfail("attn fwd attr", e);
  }
  const float ds = drop_p > 0.f ? 1.f / (1.f - drop_p) : 1.f;
  rtp::launch_k(attn_small_fwd_kernel, dim3(B * heads), dim3(attn_threads(S, B * heads)), smem, (cudaStream_t)stream,
      (const __nv_bfloat16*)qkv, (__nv_bfloat16*)out, S, B, heads, nshard, causal, sm_scale, host_thresh(drop_p), ds,
      seed, offset, step_ptr);
  LAUNCH_CHECK("attn_small_fwd");
  return 0;
}
int rtp_attn_small_bwd(const void* qkv, const void* dout, void* dqkv, int S, int B, int heads, int nshard, int causal,
                       float sm_scale, float drop_p, unsigned long long seed, unsigned long long offset,
                       const unsigned long long* step_ptr, void* stream) {
  if (g_attn_tc && rtp_attn_tc_supported(S, heads, nshard)) {
    const int rc = rtp_attn_tc_bwd(qkv, dout, dqkv, S, B, heads, nshard, causal, sm_scale, drop_p, seed, offset, step_ptr,
                                   stream);
    if (rc) k_err = rtp_attn_tc_last_error();
    return rc;
  }
  if (heads % nshard) { k_err = "attn_small: heads must be divisible by shards"; return -1; }
  const size_t smem = attn_smem(S, true);
  if (smem > 227 * 1024) { k_err = "attn_small backward: sequence too long for shared memory (S <= 96)"; return -1; }
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(attn_small_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return kfail("attn bwd attr", e);
  }
  const float ds = drop_p > 0.f ? 1.f / (1.f - drop_p) : 1.f;
  rtp::launch_k(attn_small_bwd_kernel, dim3(B * heads), dim3(attn_threads(S, B * heads)), smem, (cudaStream_t)stream,
      (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dqkv, S, B, heads, nshard, causal,
      sm_scale, host_thresh(drop_p), ds, seed, offset, step_ptr);
  LAUNCH_CHECK("attn_small_bwd");
  return 0;
}
int rtp_colsum(const void* x, long long ld, int M, int N, float* out, void* stream) {
  if (N % 2 || ld % 2) { k_err = "colsum: N and ld must be even"; return -1; }
  if (N % 8 == 0 && ld % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0) {
    // clusters of up to 8 blocks split the rows (at least 128 rows per block); very tall matrices get several
    // clusters per column group, whose sums meet in the zeroed output by atomics
    int cy = 8;
    while (cy > 1 && M < cy * 128) cy >>= 1;
    int groups = 1;
    while (groups < 64 && M / (cy * groups) > 1024) groups <<= 1;
    const int rows = (M + cy * groups - 1) / (cy * groups);
    if (groups > 1) {
      cudaError_t e = cudaMemsetAsync(out, 0, (size_t)N * sizeof(float), (cudaStream_t)stream);
      if (e != cudaSuccess) return kfail("colsum memset", e);
    }
    rtp::launch_kc(colsum_vec_kernel, dim3((N + 63) / 64, cy * groups), dim3(256), 0, (cudaStream_t)stream, dim3(1, cy, 1),
                   (const __nv_bfloat16*)x, ld, M, N, out, rows, groups > 1 ? 1 : 0);
    LAUNCH_CHECK("colsum");
    return 0;
  }
  cudaError_t e = cudaMemsetAsync(out, 0, (size_t)N * sizeof(float), (cudaStream_t)stream);
  if (e != cudaSuccess) return kfail("colsum memset", e);
  const int rows_per_block = 64;
  dim3 grid((N / 2 + 127) / 128, (M + rows_per_block - 1) / rows_per_block);
  colsum_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, ld, M, N, out, rows_per_block);
  LAUNCH_CHECK("colsum");
  return 0;
}
int rtp_adam(const RtpAdamTensor* tensors_dev, const int* block_start_dev, int ntensors, int total_blocks,
             const long long* step_dev, float lr, float beta1, float beta2, float eps, float weight_decay, int adamw,
             float clip_value, float grad_scale, const int* block_tensor_dev, void* stream) {
  if (ntensors <= 0 || total_blocks <= 0) return 0;
  adam_kernel<<<total_blocks, 256, 0, (cudaStream_t)stream>>>(tensors_dev, block_start_dev, ntensors, step_dev, lr,
                                                              beta1, beta2, eps, weight_decay, adamw, clip_value,
                                                              grad_scale, block_tensor_dev);
  LAUNCH_CHECK("adam");
  return 0;
}
int rtp_causal_softmax(void* s, long long rows, int S, float scale, void* stream) {
  if (S % 8) { k_err = "causal_softmax: S must be a multiple of 8"; return -1; }
  const int grid = rows < 148 * 16 ? (int)rows : 148 * 16;
  causal_softmax_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)s, rows, S, scale);
  LAUNCH_CHECK("causal_softmax");
  return 0;
}
int rtp_causal_softmax_bwd(const void* p, void* dp, long long rows, int S, float scale, void* stream) {
  if (S % 8) { k_err = "causal_softmax_bwd: S must be a multiple of 8"; return -1; }
  const int grid = rows < 148 * 16 ? (int)rows : 148 * 16;
  causal_softmax_bwd_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)p, (__nv_bfloat16*)dp, rows, S,
                                                                   scale);
  LAUNCH_CHECK("causal_softmax_bwd");
  return 0;
}
int rtp_gelu_fwd(const void* x, void* y, long long n, void* stream) {
  if (n % 8) { k_err = "gelu: n must be a multiple of 8"; return -1; }
  gelu_fwd_kernel<<<(unsigned)((n / 8 + 255) / 256), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)y, n);
  LAUNCH_CHECK("gelu_fwd");
  return 0;
}
int rtp_gelu_bwd(const void* x, const void* dy, void* dx, long long n, void* stream) {
  if (n % 8) { k_err = "gelu: n must be a multiple of 8"; return -1; }
  gelu_bwd_kernel<<<(unsigned)((n / 8 + 255) / 256), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)dy,
                                                                                 (__nv_bfloat16*)dx, n);
  LAUNCH_CHECK("gelu_bwd");
  return 0;
}
int rtp_swiglu_fwd(const void* g, const void* u, long long ld, void* y, long long rows, int cols, void* stream) {
  if (cols % 8 || ld % 8) { k_err = "swiglu: cols and ld must be multiples of 8"; return -1; }
  const long long items = rows * (cols / 8);
  swiglu_fwd_kernel<<<(unsigned)((items + 255) / 256), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)g, (const __nv_bfloat16*)u, ld,
                                                                                   (__nv_bfloat16*)y, rows, cols);
  LAUNCH_CHECK("swiglu_fwd");
  return 0;
}
int rtp_swiglu_bwd(const void* g, const void* u, long long ld, const void* dy, void* dg, void* du, long long ldo,
                   long long rows, int cols, void* stream) {
  if (cols % 8 || ld % 8 || ldo % 8) { k_err = "swiglu: cols and ld must be multiples of 8"; return -1; }
  const long long items = rows * (cols / 8);
  swiglu_bwd_kernel<<<(unsigned)((items + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)g, (const __nv_bfloat16*)u, ld, (const __nv_bfloat16*)dy, (__nv_bfloat16*)dg, (__nv_bfloat16*)du, ldo, rows,
      cols);
  LAUNCH_CHECK("swiglu_bwd");
  return 0;
}
int rtp_moe_scatter(const void* src, const int* slot, const float* scale, void* dst, int S, int M, long long dst_rows,
                    int* fill, int cap, void* stream) {
  if (M % 8) { k_err = "moe: M must be a multiple of 8"; return -1; }
  if (fill && (cap <= 0 || dst_rows % cap)) { k_err = "moe: rows must be whole capacities"; return -1; }
  cudaError_t e = cudaMemsetAsync(dst, 0, (size_t)dst_rows * M * 2, (cudaStream_t)stream);
  if (e == cudaSuccess && fill) e = cudaMemsetAsync(fill, 0, (size_t)(dst_rows / cap) * sizeof(int), (cudaStream_t)stream);
  if (e != cudaSuccess) return kfail("moe memset", e);
  const long long threads = 2ll * S * 32;
  moe_scatter_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)src, slot, scale, (__nv_bfloat16*)dst, S, M, fill, cap);
  LAUNCH_CHECK("moe_scatter");
  return 0;
}
int rtp_moe_gather(const void* src, const int* slot, const float* scale, void* dst, int S, int M, void* stream) {
  if (M % 8) { k_err = "moe: M must be a multiple of 8"; return -1; }
  const long long threads = (long long)S * 32;
  moe_gather_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)src, slot, scale, (__nv_bfloat16*)dst, S, M);
  LAUNCH_CHECK("moe_gather");
  return 0;
}
int rtp_moe_rowdot(const void* a, const void* b, const int* slot, float* out, int S, int M, void* stream) {
  if (M % 8) { k_err = "moe: M must be a multiple of 8"; return -1; }
  const long long threads = 2ll * S * 32;
  moe_rowdot_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)a, (const __nv_bfloat16*)b, slot, out, S, M);
  LAUNCH_CHECK("moe_rowdot");
  return 0;
}
int rtp_add(const void* a, const void* b, void* out, long long n, void* stream) {
  const long long blocks = (n + 2047) / 2048;
  add_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)a, (const __nv_bfloat16*)b,
                                                                 (__nv_bfloat16*)out, n);
  LAUNCH_CHECK("add");
  return 0;
}
int rtp_cast_f32_bf16(const float* in, void* out, long long n, float scale, void* stream) {
  cast_f32_bf16_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(in, (__nv_bfloat16*)out, n, scale);
  LAUNCH_CHECK("cast");
  return 0;
}
int rtp_sum_f32(const float* in, float* out, int n, float scale, const float* divisor, void* stream) {
  rtp::launch_k(sum_kernel, dim3(1), dim3(1024), 0, (cudaStream_t)stream, in, out, n, scale, divisor);
  LAUNCH_CHECK("sum");
  return 0;
}

}  // extern "C"

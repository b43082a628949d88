// Short-sequence attention (S = 32 or 64, head_dim 64) on tcgen05 tensor cores.
//
// One CTA of 128 threads handles 128 / S (batch, head) pairs at once: their query rows and their key rows are stacked into
// 128-row operands, so that every product is one chain of M = 128 UMMAs.  Thread t owns stacked row t (TMEM lane t) and works on
// the columns of its own head, so the softmax of a row and the dS algebra of the backward pass run entirely in that thread's
// registers, without shuffles.
//
//   forward :  S = Q K^T (all pairs of stacked rows)  ->  P = dropout(softmax(scale * S)) of the own head  ->  O = P V
//   backward:  S, dP = dO V^T  ->  dS  ->  dQ = dS K ;  dK = dS^T Q ;  dV = P_drop^T dO
//
// P and dS are [128 x 128] tiles with zeros between different heads.  Where V (forward) or Q, K or dO (backward) hold a value that
// is not finite, these zeros would make NaN of it in the rows of other heads: such a CTA multiplies one head's rows at a time and
// each head keeps what came of its own.  The look for such values is free, it is taken while the tensor cores make S and dP (at the
// end, from the results, it took 0.5 us of a backward of 8).  Written once, row per thread, the dS tile is read K-major for dQ and
// MN-major (transposed) for dK.  P takes the place of operands that are no longer needed, and the results take the place of S and dP
// in TMEM: 48 / 112 KB and 128 / 256 columns, so that two CTAs and more share an SM (one chain a head, with 64 / 144 KB and 256 /
// 512 columns, had one in backward: 1024 heads of 32 x 64 took two rounds).
// us, that form -> this: 1024 heads of 32 with dropout, forward 10.4 -> 8.1, backward 20.0 -> 10.9; 32 heads of 32 5.8 -> 5.2 and
// 10.9 -> 7.9; 1024 heads of 64 17.8 -> 12.8 and 47.4 -> 25.2.
//
// Operands are fetched with plain 16-byte loads into 128-byte-swizzled tiles (the strided token order s*B + b of the
// packed projection needs no tensor map); "fence.proxy.async" publishes them to the tensor core.
//
// Same data layout and dropout stream as the scalar kernels in kernels.cu (attn_small_*), which remain the path for
// every other sequence length.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "launch.h"

namespace {
using namespace rtp;

constexpr int kHd = 64;
constexpr int kRows = 128;                 // stacked rows per CTA
constexpr int kTile = kRows * 128;         // one [128 x 64] bf16 operand tile, 128-byte rows: 16 KB
constexpr int kSlack = 512;                // for the alignment of the tiles, which shared memory starts with anyhow

__device__ unsigned int g_attn_tc_error;        // set when a bounded wait for the CTA's own UMMAs ran out
__device__ unsigned long long* g_attn_trace;   // tuning aid: timeline of CTA 0 (16 words), null = off
#define ATT_STAMP(i) do { if (g_attn_trace && blockIdx.x == 0 && threadIdx.x == 0) g_attn_trace[i] = globaltimer_ns(); } while (0)

struct Ctl {
  uint64_t bar[2];
  uint32_t tmem_base;
  int valid[4];
  int b[4];
  int h[4];
  int cq[4], ck[4], cv[4];
};

__device__ __forceinline__ int qkv_col(int head, int which, int D, int nshard, int heads) {
  const int hps = heads / nshard;  // heads per shard
  const int j = head / hps, hl = head % hps;
  return j * (3 * (D / nshard)) + which * (D / nshard) + hl * kHd;
}
// byte offset of 16-byte chunk `chunk` of row `row` in a 128-byte-swizzled tile of 128-byte rows
__device__ __forceinline__ uint32_t sw128(int row, int chunk) {
  return (uint32_t)row * 128u + (uint32_t)((chunk ^ (row & 7)) << 4);
}
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (globaltimer_ns() - t0 > 1000000000ull) {
      atomicExch(&g_attn_tc_error, 1u);
      return false;
    }
  }
  return true;
}
// Keep bits of the S_T probabilities that start at element e0 (a multiple of 4): bit c set = kept.
template <int S_T>
__device__ __forceinline__ uint64_t keep_row(uint64_t seed, uint64_t offset, uint64_t e0, uint32_t thresh) {
  uint64_t keep = ~0ull;
  if (!thresh) return keep;
  keep = 0;
#pragma unroll
  for (int c4 = 0; c4 < S_T / 4; ++c4) {
    const uint4 rr = philox4x32(seed, offset, (e0 >> 2) + c4);
    const uint32_t k4 = (rr.x >= thresh ? 1u : 0u) | (rr.y >= thresh ? 2u : 0u) | (rr.z >= thresh ? 4u : 0u) | (rr.w >= thresh ? 8u : 0u);
    keep |= (uint64_t)k4 << (4 * c4);
  }
  return keep;
}
// Row `row` of a [128 x 128] tile of two [128 x 64] sub-tiles: the S_T values of head q at its columns, zeros elsewhere.
template <int S_T>
__device__ __forceinline__ void write_diagonal(uint8_t* tile, int row, int q, const float* v) {
  constexpr int N = S_T / 8;
  uint4 w[N];
#pragma unroll
  for (int k = 0; k < N; ++k)
    w[k] = make_uint4(pack_bf16(v[8 * k], v[8 * k + 1]), pack_bf16(v[8 * k + 2], v[8 * k + 3]), pack_bf16(v[8 * k + 4], v[8 * k + 5]),
                      pack_bf16(v[8 * k + 6], v[8 * k + 7]));
#pragma unroll
  for (int g = 0; g < 16 / N; ++g) {
    const bool own = g == q;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int c = g * N + k;
      *reinterpret_cast<uint4*>(tile + (c >> 3) * kTile + sw128(row, c & 7)) = own ? w[k] : make_uint4(0u, 0u, 0u, 0u);
    }
  }
}

// Stacks rows [q * S_T + s] = token (s, b_q), columns col[q] .. col[q] + 64 of `src` (row pitch ld) into swizzled tiles.
// A thread's eight 16-byte loads per tile are all issued before the first shared-memory store, so that they overlap
// (a store in between would order them: the compiler cannot prove that the tile and the control block do not alias).
struct HeadRef {
  int valid, b, col;
};
template <int S_T>
__device__ __forceinline__ void fetch_stack(uint4 (&v)[8], const __nv_bfloat16* __restrict__ src, long long ld, int B,
                                            const HeadRef (&hr)[kRows / S_T], int tid) {
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int i = it * 128 + tid;
    const int row = i >> 3, c = i & 7;
    const int q = row / S_T, s = row % S_T;
    v[it] = make_uint4(0u, 0u, 0u, 0u);
    if (hr[q].valid) v[it] = __ldg(reinterpret_cast<const uint4*>(src + (size_t)(s * B + hr[q].b) * ld + hr[q].col + c * 8));
  }
}
__device__ __forceinline__ void store_stack(uint8_t* dst, const uint4 (&v)[8], int tid) {
#pragma unroll
  for (int it = 0; it < 8; ++it) {
    const int i = it * 128 + tid;
    *reinterpret_cast<uint4*>(dst + sw128(i >> 3, i & 7)) = v[it];
  }
}

template <int S_T>
__device__ __forceinline__ void setup(Ctl* ctl, int tid, int warp, int B, int heads, int nshard, int n_bh,
                                      uint32_t tmem_cols) {
  constexpr int HPC = kRows / S_T;
  const int D = heads * kHd;
  if (tid < HPC) {
    const int bh = blockIdx.x * HPC + tid;
    const int ok = bh < n_bh;
    const int b = ok ? bh / heads : 0, h = ok ? bh % heads : 0;
    ctl->valid[tid] = ok;
    ctl->b[tid] = b;
    ctl->h[tid] = h;
    ctl->cq[tid] = qkv_col(h, 0, D, nshard, heads);
    ctl->ck[tid] = qkv_col(h, 1, D, nshard, heads);
    ctl->cv[tid] = qkv_col(h, 2, D, nshard, heads);
  }
  if (tid == 0) {
    mbar_init(&ctl->bar[0], 1);
    mbar_init(&ctl->bar[1], 1);
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(&ctl->tmem_base, tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();   // every CTA owns its TMEM columns first (see launch.h)
  pdl_wait();   // set-up touched shared memory and TMEM only; the loads below need the previous kernel's output
}

// Row t of the score matrix out of TMEM, scaled; masked entries become -inf.
template <int S_T>
__device__ __forceinline__ void load_row(uint32_t taddr, float (&x)[S_T]) {
#pragma unroll
  for (int j = 0; j < S_T / 32; ++j) {
    uint32_t r[32];
    tmem_ld_32x32(taddr + j * 32, r);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; ++i) x[j * 32 + i] = __uint_as_float(r[i]);
  }
}

// 1 if one of these bf16 is an infinity or a NaN
__device__ __forceinline__ int not_finite(const uint4 (&v)[8]) {
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    m = __vimax3_u16x2(m, v[i].x & 0x7fff7fffu, v[i].y & 0x7fff7fffu);
    m = __vimax3_u16x2(m, v[i].z & 0x7fff7fffu, v[i].w & 0x7fff7fffu);
  }
  return (m & 0xffffu) >= 0x7f80u || (m >> 16) >= 0x7f80u;
}
// The products of a CTA, each over the 128 stacked rows in slices of 16, or over the rows of head g alone.
template <int S_T, typename... Products>
__device__ __forceinline__ void each_slice(bool all, int g, Products... products) {
  auto chain = [](auto product, int j0, auto n) {
#pragma unroll
    for (int i = 0; i < decltype(n)::value; ++i) product(j0 + i, i > 0);
  };
  if (all) (chain(products, 0, std::integral_constant<int, kRows / 16>{}), ...);
  else (chain(products, g * (S_T / 16), std::integral_constant<int, S_T / 16>{}), ...);
}

template <int S_T>
__global__ void __launch_bounds__(128) attn_tc_fwd_kernel(const __nv_bfloat16* __restrict__ qkv,
                                                          __nv_bfloat16* __restrict__ out, int B, int heads, int nshard,
                                                          int causal, float sm_scale, uint32_t thresh, float drop_scale,
                                                          uint64_t seed, uint64_t offset,
                                                          const unsigned long long* __restrict__ step_ptr, int n_bh) {
  constexpr int HPC = kRows / S_T;
  extern __shared__ __align__(1024) uint8_t smem_tiles[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_tiles) + 1023) & ~uintptr_t(1023));
  if (sm - smem_tiles > kSlack) {
    if (threadIdx.x == 0) atomicExch(&g_attn_tc_error, 1u);
    return;
  }
  uint8_t* sQ = sm;
  uint8_t* sK = sm + kTile;
  uint8_t* sV = sm + 2 * kTile;
  uint8_t* sP = sm;                         // [128 x 128], over Q and K
  Ctl* ctl = reinterpret_cast<Ctl*>(sm + 3 * kTile);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int D = heads * kHd;
  ATT_STAMP(0);
  setup<S_T>(ctl, tid, warp, B, heads, nshard, n_bh, 128);
  ATT_STAMP(1);
  const uint32_t tmem = ctl->tmem_base;
  const int q = tid / S_T, s = tid % S_T;
  uint64_t keep;
  uint4 va[8], vb[8], vc[8];
  {
    HeadRef hq[HPC], hk[HPC], hv[HPC];
#pragma unroll
    for (int qq = 0; qq < HPC; ++qq) {
      hq[qq] = {ctl->valid[qq], ctl->b[qq], ctl->cq[qq]};
      hk[qq] = {ctl->valid[qq], ctl->b[qq], ctl->ck[qq]};
      hv[qq] = {ctl->valid[qq], ctl->b[qq], ctl->cv[qq]};
    }
    fetch_stack<S_T>(va, qkv, 3 * D, B, hq, tid);
    fetch_stack<S_T>(vb, qkv, 3 * D, B, hk, tid);
    fetch_stack<S_T>(vc, qkv, 3 * D, B, hv, tid);
    // the dropout bits are worked out while the loads are in flight
    if (step_ptr) offset += __ldg(step_ptr) * 65536ull;
    keep = keep_row<S_T>(seed, offset, ((uint64_t)(blockIdx.x * HPC + q) * S_T + s) * S_T, thresh);
    store_stack(sQ, va, tid);
    store_stack(sK, vb, tid);
    store_stack(sV, vc, tid);
  }
  fence_proxy_async_smem();
  __syncthreads();
  ATT_STAMP(2);

  if (warp == 0 && elect_one()) {
    const uint32_t idesc = make_idesc_bf16(128, 128, 0, 0);
    const uint32_t aq = smem_u32(sQ), bk = smem_u32(sK);
#pragma unroll
    for (int kk = 0; kk < kHd / 16; ++kk)
      umma_bf16(tmem, make_smem_desc(aq + kk * 32, 16, 1024), make_smem_desc(bk + kk * 32, 16, 1024), idesc, kk > 0 ? 1u : 0u);
    umma_commit(&ctl->bar[0]);
  }
  const int odd = not_finite(vc);
  wait_bar(&ctl->bar[0], 0);
  __syncwarp();
  tc_fence_after();
  ATT_STAMP(3);

  const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
  {
    float x[S_T];
    load_row<S_T>(lane_addr + q * S_T, x);
    float mx = -INFINITY;
#pragma unroll
    for (int c = 0; c < S_T; ++c) {
      x[c] = (causal && c > s) ? -INFINITY : x[c] * sm_scale;
      mx = fmaxf(mx, x[c]);
    }
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < S_T; ++c) {
      x[c] = __expf(x[c] - mx);
      sum += x[c];
    }
    const float inv = 1.f / sum, kept = thresh ? inv * drop_scale : inv;
#pragma unroll
    for (int c = 0; c < S_T; ++c) x[c] *= (keep >> c) & 1ull ? kept : 0.f;
    write_diagonal<S_T>(sP, tid, q, x);
  }
  ATT_STAMP(4);
  fence_proxy_async_smem();
  tc_fence_before();
  const int parts = __syncthreads_or(odd) ? HPC : 1;
  ATT_STAMP(5);

#pragma unroll 1
  for (int g = 0; g < parts; ++g) {
    if (warp == 0 && elect_one()) {
      tc_fence_after();
      const uint32_t idesc = make_idesc_bf16(128, kHd, 0, 1);
      const uint32_t ap = smem_u32(sP), bv = smem_u32(sV);
      auto product = [&](int j, bool add) {        // 16 of the stacked keys
        umma_bf16(tmem, make_smem_desc(ap + (j >> 2) * kTile + (j & 3) * 32, 16, 1024), make_smem_desc(bv + j * 2048, 8192, 1024), idesc,
                  add ? 1u : 0u);
      };
      each_slice<S_T>(parts == 1, g, product);
      umma_commit(&ctl->bar[1]);
    }
    wait_bar(&ctl->bar[1], g & 1);
    __syncwarp();
    tc_fence_after();
    ATT_STAMP(6);
    if (parts == 1 || g == q) {
      // a warp's 32 rows belong to one head and to consecutive positions
      float o[kHd];
      load_row<kHd>(lane_addr, o);
      __nv_bfloat16* dst = out + (size_t)((s - lane) * B + ctl->b[q]) * D + ctl->h[q] * kHd;
      const int rows = ctl->valid[q] ? 32 : 0;
      store_rows32(dst, (long long)B * D, rows, o, lane);
      store_rows32(dst + 32, (long long)B * D, rows, o + 32, lane);
    }
    ATT_STAMP(7);
    tc_fence_before();
    __syncthreads();
  }
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 128);
  }
  ATT_STAMP(8);
}

template <int S_T>
__global__ void __launch_bounds__(128) attn_tc_bwd_kernel(const __nv_bfloat16* __restrict__ qkv,
                                                          const __nv_bfloat16* __restrict__ dout,
                                                          __nv_bfloat16* __restrict__ dqkv, int B, int heads, int nshard,
                                                          int causal, float sm_scale, uint32_t thresh, float drop_scale,
                                                          uint64_t seed, uint64_t offset,
                                                          const unsigned long long* __restrict__ step_ptr, int n_bh) {
  constexpr int HPC = kRows / S_T;
  extern __shared__ __align__(1024) uint8_t smem_tiles[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_tiles) + 1023) & ~uintptr_t(1023));
  if (sm - smem_tiles > kSlack) {
    if (threadIdx.x == 0) atomicExch(&g_attn_tc_error, 1u);
    return;
  }
  uint8_t* sQ = sm;
  uint8_t* sK = sm + kTile;
  uint8_t* sG = sm + 2 * kTile;            // dO
  uint8_t* sV = sm + 3 * kTile;
  uint8_t* sP = sV;                        // dropped probabilities [128 x 128], over V and the tile behind it
  uint8_t* sS = sm + 5 * kTile;            // dS [128 x 128]
  Ctl* ctl = reinterpret_cast<Ctl*>(sm + 7 * kTile);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int D = heads * kHd;
  ATT_STAMP(0);
  setup<S_T>(ctl, tid, warp, B, heads, nshard, n_bh, 256);
  ATT_STAMP(1);
  const uint32_t tmem = ctl->tmem_base;
  const int q = tid / S_T, s = tid % S_T;
  uint64_t keep;
  uint4 va[8], vb[8], vc[8], vd[8];
  {
    HeadRef hq[HPC], hk[HPC], hv[HPC], hg[HPC];
#pragma unroll
    for (int qq = 0; qq < HPC; ++qq) {
      hq[qq] = {ctl->valid[qq], ctl->b[qq], ctl->cq[qq]};
      hk[qq] = {ctl->valid[qq], ctl->b[qq], ctl->ck[qq]};
      hv[qq] = {ctl->valid[qq], ctl->b[qq], ctl->cv[qq]};
      hg[qq] = {ctl->valid[qq], ctl->b[qq], ctl->h[qq] * kHd};   // dO has [T, D] layout: column of head h is h * 64
    }
    fetch_stack<S_T>(va, qkv, 3 * D, B, hq, tid);
    fetch_stack<S_T>(vb, qkv, 3 * D, B, hk, tid);
    fetch_stack<S_T>(vc, dout, D, B, hg, tid);
    fetch_stack<S_T>(vd, qkv, 3 * D, B, hv, tid);
    // the dropout bits are worked out while the loads are in flight
    if (step_ptr) offset += __ldg(step_ptr) * 65536ull;
    keep = keep_row<S_T>(seed, offset, ((uint64_t)(blockIdx.x * HPC + q) * S_T + s) * S_T, thresh);
    store_stack(sQ, va, tid);
    store_stack(sK, vb, tid);
    store_stack(sG, vc, tid);
    store_stack(sV, vd, tid);
  }
  fence_proxy_async_smem();
  __syncthreads();
  ATT_STAMP(2);

  if (warp == 0 && elect_one()) {
    const uint32_t idesc = make_idesc_bf16(128, 128, 0, 0);
    const uint32_t aq = smem_u32(sQ), bk = smem_u32(sK), ag = smem_u32(sG), bv = smem_u32(sV);
#pragma unroll
    for (int kk = 0; kk < kHd / 16; ++kk)
      umma_bf16(tmem, make_smem_desc(aq + kk * 32, 16, 1024), make_smem_desc(bk + kk * 32, 16, 1024), idesc, kk > 0 ? 1u : 0u);
#pragma unroll
    for (int kk = 0; kk < kHd / 16; ++kk)
      umma_bf16(tmem + 128, make_smem_desc(ag + kk * 32, 16, 1024), make_smem_desc(bv + kk * 32, 16, 1024), idesc, kk > 0 ? 1u : 0u);
    umma_commit(&ctl->bar[0]);
  }
  const int odd = not_finite(va) | not_finite(vb) | not_finite(vc);
  wait_bar(&ctl->bar[0], 0);
  __syncwarp();
  tc_fence_after();
  ATT_STAMP(3);

  const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
  {
    float x[S_T], dp[S_T];
    load_row<S_T>(lane_addr + q * S_T, x);
    load_row<S_T>(lane_addr + 128 + q * S_T, dp);
    float mx = -INFINITY;
#pragma unroll
    for (int c = 0; c < S_T; ++c) {
      x[c] = (causal && c > s) ? -INFINITY : x[c] * sm_scale;
      mx = fmaxf(mx, x[c]);
    }
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < S_T; ++c) {
      x[c] = __expf(x[c] - mx);
      sum += x[c];
    }
    const float inv = 1.f / sum;
    // x <- P, dp <- m * dP (gradient wrt the un-dropped probability)
    float dot = 0.f;
#pragma unroll
    for (int c = 0; c < S_T; ++c) {
      x[c] *= inv;
      dp[c] = (keep >> c) & 1ull ? dp[c] * drop_scale : 0.f;
      dot += dp[c] * x[c];
    }
    // dS (into dp) and the dropped probabilities (into x)
#pragma unroll
    for (int c = 0; c < S_T; ++c) {
      dp[c] = x[c] * (dp[c] - dot);
      x[c] = (keep >> c) & 1ull ? x[c] * drop_scale : 0.f;
    }
    write_diagonal<S_T>(sS, tid, q, dp);
    write_diagonal<S_T>(sP, tid, q, x);
  }
  ATT_STAMP(4);
  fence_proxy_async_smem();
  tc_fence_before();
  const int parts = __syncthreads_or(odd) ? HPC : 1;   // S and dP have been read everywhere: the results take their TMEM columns
  ATT_STAMP(5);

#pragma unroll 1
  for (int g = 0; g < parts; ++g) {
    if (warp == 0 && elect_one()) {
      tc_fence_after();
      const uint32_t as = smem_u32(sS), ap = smem_u32(sP), bk = smem_u32(sK), bq = smem_u32(sQ), bg = smem_u32(sG);
      const uint32_t id_q = make_idesc_bf16(128, kHd, 0, 1), id_t = make_idesc_bf16(128, kHd, 1, 1);
      // 16 of the stacked keys (dQ) or queries
      auto dq = [&](int j, bool add) {
        umma_bf16(tmem, make_smem_desc(as + (j >> 2) * kTile + (j & 3) * 32, 16, 1024), make_smem_desc(bk + j * 2048, 8192, 1024), id_q,
                  add ? 1u : 0u);
      };
      auto dk = [&](int j, bool add) {
        umma_bf16(tmem + 64, make_smem_desc(as + j * 2048, kTile, 1024), make_smem_desc(bq + j * 2048, 8192, 1024), id_t, add ? 1u : 0u);
      };
      auto dv = [&](int j, bool add) {
        umma_bf16(tmem + 128, make_smem_desc(ap + j * 2048, kTile, 1024), make_smem_desc(bg + j * 2048, 8192, 1024), id_t, add ? 1u : 0u);
      };
      each_slice<S_T>(parts == 1, g, dq, dk, dv);
      umma_commit(&ctl->bar[1]);
    }
    wait_bar(&ctl->bar[1], g & 1);
    __syncwarp();
    tc_fence_after();
    ATT_STAMP(6);
    if (parts == 1 || g == q) {
      // a warp's 32 rows belong to one head and to consecutive positions
      __nv_bfloat16* rowp = dqkv + (size_t)((s - lane) * B + ctl->b[q]) * (3 * D);
      const long long pitch = 3ll * B * D;
      const int rows = ctl->valid[q] ? 32 : 0;
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const int col = r == 0 ? ctl->cq[q] : r == 1 ? ctl->ck[q] : ctl->cv[q];
        float o[kHd];
        load_row<kHd>(lane_addr + r * kHd, o);
        if (r < 2) {
#pragma unroll
          for (int c = 0; c < kHd; ++c) o[c] *= sm_scale;
        }
        store_rows32(rowp + col, pitch, rows, o, lane);
        store_rows32(rowp + col + 32, pitch, rows, o + 32, lane);
      }
    }
    ATT_STAMP(7);
    tc_fence_before();
    __syncthreads();
  }
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 256);
  }
  ATT_STAMP(8);
}

std::string g_err;
constexpr int kFwdSmem = 3 * kTile + kSlack + 256;
constexpr int kBwdSmem = 7 * kTile + kSlack + 256;
static_assert(2 * (kBwdSmem + 1024) <= 233472, "two CTAs of the backward kernel on an SM");
uint32_t thresh_of(float p) {
  if (p <= 0.f) return 0u;
  double t = (double)p * 4294967296.0;
  if (t > 4294967295.0) t = 4294967295.0;
  return (uint32_t)t;
}
template <auto Kern>
int set_smem(int bytes) {
  cudaError_t e = rtp::ensure_smem<Kern>(bytes);
  if (e != cudaSuccess) {
    g_err = std::string("attn_tc: cudaFuncSetAttribute: ") + cudaGetErrorString(e);
    return -1;
  }
  return 0;
}
}  // namespace

extern "C" {

const char* rtp_attn_tc_last_error(void) { return g_err.c_str(); }

// tuning aid: device buffer of 16 words that receives globaltimer stamps of CTA 0 (null switches it off)
int rtp_attn_tc_set_trace(unsigned long long* device_buffer) {
  return cudaMemcpyToSymbol(g_attn_trace, &device_buffer, sizeof(device_buffer)) == cudaSuccess ? 0 : -1;
}

int rtp_attn_tc_supported(int S, int heads, int nshard) { return (S == 32 || S == 64) && heads % nshard == 0; }

// 1 if a bounded wait inside one of the kernels ran out since the last call (and clears the flag); synchronises.
int rtp_attn_tc_error(void) {
  unsigned int v = 0, z = 0;
  if (cudaMemcpyFromSymbol(&v, g_attn_tc_error, sizeof(v)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_attn_tc_error, &z, sizeof(z));
  return (int)v;
}

int rtp_attn_tc_fwd(const void* qkv, void* out, int S, int B, int heads, int nshard, int causal, float sm_scale,
                    float drop_p, unsigned long long seed, unsigned long long offset,
                    const unsigned long long* step_ptr, void* stream) {
  if (!rtp_attn_tc_supported(S, heads, nshard)) { g_err = "attn_tc: S must be 32 or 64"; return -1; }
  const int n_bh = B * heads;
  const float ds = drop_p > 0.f ? 1.f / (1.f - drop_p) : 1.f;
  const int hpc = 128 / S;
  const int grid = (n_bh + hpc - 1) / hpc;
  if (S == 32) {
    if (set_smem<attn_tc_fwd_kernel<32>>(kFwdSmem)) return -1;
    rtp::launch_k(attn_tc_fwd_kernel<32>, dim3(grid), dim3(128), kFwdSmem, (cudaStream_t)stream,
        (const __nv_bfloat16*)qkv, (__nv_bfloat16*)out, B, heads, nshard, causal, sm_scale, thresh_of(drop_p), ds, seed,
        offset, step_ptr, n_bh);
  } else {
    if (set_smem<attn_tc_fwd_kernel<64>>(kFwdSmem)) return -1;
    rtp::launch_k(attn_tc_fwd_kernel<64>, dim3(grid), dim3(128), kFwdSmem, (cudaStream_t)stream,
        (const __nv_bfloat16*)qkv, (__nv_bfloat16*)out, B, heads, nshard, causal, sm_scale, thresh_of(drop_p), ds, seed,
        offset, step_ptr, n_bh);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { g_err = std::string("attn_tc_fwd: ") + cudaGetErrorString(e); return -1; }
  return 0;
}

int rtp_attn_tc_bwd(const void* qkv, const void* dout, void* dqkv, int S, int B, int heads, int nshard, int causal,
                    float sm_scale, float drop_p, unsigned long long seed, unsigned long long offset,
                    const unsigned long long* step_ptr, void* stream) {
  if (!rtp_attn_tc_supported(S, heads, nshard)) { g_err = "attn_tc: S must be 32 or 64"; return -1; }
  const int n_bh = B * heads;
  const float ds = drop_p > 0.f ? 1.f / (1.f - drop_p) : 1.f;
  const int hpc = 128 / S;
  const int grid = (n_bh + hpc - 1) / hpc;
  if (S == 32) {
    if (set_smem<attn_tc_bwd_kernel<32>>(kBwdSmem)) return -1;
    rtp::launch_k(attn_tc_bwd_kernel<32>, dim3(grid), dim3(128), kBwdSmem, (cudaStream_t)stream,
        (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dqkv, B, heads, nshard, causal, sm_scale,
        thresh_of(drop_p), ds, seed, offset, step_ptr, n_bh);
  } else {
    if (set_smem<attn_tc_bwd_kernel<64>>(kBwdSmem)) return -1;
    rtp::launch_k(attn_tc_bwd_kernel<64>, dim3(grid), dim3(128), kBwdSmem, (cudaStream_t)stream,
        (const __nv_bfloat16*)qkv, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dqkv, B, heads, nshard, causal, sm_scale,
        thresh_of(drop_p), ds, seed, offset, step_ptr, n_bh);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { g_err = std::string("attn_tc_bwd: ") + cudaGetErrorString(e); return -1; }
  return 0;
}

}  // extern "C"

// Flash attention on tcgen05 tensor cores: forward, delta and backward kernels (see flash_attn.h for the interface).
//
// A CTA works on 128-row tiles of one (batch, head) at a time.  Twelve warps:
//   warps 0-7  "row" threads: thread = TMEM lane = row of a tile (forward: all 128 columns of a block; backward: 64).  The online
//              softmax of a row (forward) and the dS algebra (backward) run in registers without shuffles.
//   warp 8     TMA producer: Q / K / V / dO tiles, 128 rows x 64 columns per copy, 128-byte swizzle, local memory only.
//   warp 9     UMMA issuer (one elected thread).
//   warp 10    asks for the next piece of work (one elected thread); warp 11 is there for its registers.
//
// Forward, per block of 128 keys:  S = Q K^T (TMEM)  ->  row threads: scale, masks, running max, P = exp2(S - m) as bf16 back into
// TMEM  ->  O += P V with O resident in TMEM.  O is rescaled in TMEM only when a row's maximum has grown by more than 2^8
// since the last rescale (the sum l carries the same offset, so the final O / l is exact); most blocks skip the rescale.
// Output: O / l and the row's log-sum-exp (log2 units).
//
// Backward recomputes P from Q, K and the saved log-sum-exp; nothing of size S x S touches global memory.  delta = rowsum(dO * O)
// comes from a kernel of its own, dQ of a block of queries and dK / dV of a block of keys are pieces of work of one launch.
//
// What it gives (us, before: one row tile a CTA with two threads a row, P and dS through shared memory, dQ and dK / dV in
// launches of their own; now), forward and backward: 1 x 16 heads of 8192 x 8192 x 128 causal 337 -> 237 and 1 131 -> 795,
// 4 x 16 of 2048 causal 123 -> 91 and 401 -> 280, 8 x 20 of 512 x 2048 x 64 118 -> 88 and 433 -> 244, 4 x 8 of 256 x 256 x 64
// 6.4 -> 6.2 and 20 -> 14, 4 x 8 of 64 x 64 x 64 4.9 -> 4.9 and 10.7 -> 9.4.  Heads of one key block that fill more than half of
// the SMs are a little slower: 8 x 16 of 64 x 64 x 64 5.3 -> 5.6 and 11.8 -> 12.8.  Per 128 x 128 block at head_dim 128 (SM
// clocks): forward 1 700 (tensor work 1 024, exponentials 1 024), dK / dV 3 100 (tensor work 2 048), dQ 2 080 (1 536).  The
// forward is bound by the exponentials and the hand-overs between row threads and issuer, dK / dV by the chain P -> dV -> S of
// the next block (TMEM has no room for a second S).
//
// Each kernel is compiled in variants (no mask, key padding only, additive mask; dropout yes or no; more work than SMs or not; backward:
// one head a CTA):
// the mask and Philox code unrolled over a row's registers is several times larger than the plain softmax and, when merely
// branched over, slowed the row threads down through instruction fetch alone.
// Every mbarrier wait is bounded; on expiry the CTA records a status code, drains its copies and UMMAs, frees its TMEM
// and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <string>
#include <type_traits>

#include "common.cuh"
#include "flash_attn.h"
#include "launch.h"
#include "tmap.h"

namespace {
using namespace rtp;

constexpr int kBlk = 128;              // rows of Q per CTA = keys per block
constexpr int kSub = 16384;            // one [128 x 64] bf16 sub-tile with 128-byte rows
constexpr int kThreads = 384;          // two warpgroups of row threads, one of producer, issuer and two idle warps
// A row thread holds 128 scores: of the 168 registers a thread that 384 threads are launched with, the third warpgroup
// hands most to the other two.
constexpr int kRowRegs = 208, kAuxRegs = 88;
static_assert(2 * kRowRegs + kAuxRegs <= 3 * 168, "more registers than the launch has");
constexpr int kProducerWarp = 8, kMmaWarp = 9, kSchedWarp = 10;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kRescaleGap = 8.f;     // rescale O when a row maximum grew by more than 2^8

struct DRef {                          // device copy of an RtpFlashRef
  void* ptr;
  long long sb, ss;
  int col_base, hpg, gstride, hstride;
};
__device__ __forceinline__ int head_col(const DRef& r, int h) {
  if (h < r.hpg) return r.col_base + h * r.hstride;      // one group of heads: no division
  return r.col_base + (h / r.hpg) * r.gstride + (h % r.hpg) * r.hstride;
}
__device__ __forceinline__ __nv_bfloat16* row_ptr(const DRef& r, int b, int s, int h) {
  return reinterpret_cast<__nv_bfloat16*>(r.ptr) + (long long)b * r.sb + (long long)s * r.ss + head_col(r, h);
}

struct MaskArgs {
  const void* mask; long long mask_ld; int mask_fp32;
  const unsigned char* kpm; long long kpm_ld;
  int causal, Sq, Sk;
  float scale_log2, sm_scale;
  uint32_t thresh; float drop_scale;
  unsigned long long seed, offset;
  const unsigned long long* step_ptr;
};

struct alignas(64) FlashParams {
  CUtensorMap mq, mk, mv, mdo;         // 3-D maps {columns, dim1, dim2}; *_seq1 tells which of dim1 / dim2 is the sequence
  int q_seq1, k_seq1, v_seq1, do_seq1;
  DRef q, k, v, o, dout, dq, dk, dv;
  float* lse;
  float* delta;
  int B, H;
  int group;                           // (batch, head) pairs whose CTAs run side by side (see head_group)
  int split;                           // forward: one row tile a CTA, its key blocks dealt to the two warpgroups
  MaskArgs m;
  unsigned long long* status;
  unsigned long long timeout_ns;
  long long* trace;                    // tuning aid (rtp_flash_debug_set_trace): SM clock stamps of CTA 0, else null
};

struct Ctl {
  uint64_t bar[28];
  uint4 next;                          // the scheduler's answer: the work that follows (see schedule)
  uint32_t tmem_base;
  uint32_t abort_flag;
};

__device__ __forceinline__ void tmem_ld32f(uint32_t taddr, float* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
        "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]),
        "=f"(r[16]), "=f"(r[17]), "=f"(r[18]), "=f"(r[19]), "=f"(r[20]), "=f"(r[21]), "=f"(r[22]), "=f"(r[23]),
        "=f"(r[24]), "=f"(r[25]), "=f"(r[26]), "=f"(r[27]), "=f"(r[28]), "=f"(r[29]), "=f"(r[30]), "=f"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32f(uint32_t taddr, const float* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]),
        "f"(r[8]), "f"(r[9]), "f"(r[10]), "f"(r[11]), "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15]),
        "f"(r[16]), "f"(r[17]), "f"(r[18]), "f"(r[19]), "f"(r[20]), "f"(r[21]), "f"(r[22]), "f"(r[23]),
        "f"(r[24]), "f"(r[25]), "f"(r[26]), "f"(r[27]), "f"(r[28]), "f"(r[29]), "f"(r[30]), "f"(r[31])
      : "memory");
}

// 16 columns of this thread's lane: 32 bf16 of a TMEM A operand
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// Loads one [128 rows x 64 * SUB columns] tile of a (batch, head) into SUB swizzled sub-tiles.
template <int SUB>
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, int seq1, int col, int b, int s0,
                                          uint32_t bar) {
  const unsigned long long m = reinterpret_cast<unsigned long long>(map);
#pragma unroll
  for (int u = 0; u < SUB; ++u) {
    if (seq1) tma_load_3d_s(dst + u * kSub, m, col + u * 64, s0, b, bar);
    else tma_load_3d_s(dst + u * kSub, m, col + u * 64, b, s0, bar);
  }
}

// x[i] = log2-domain score of (row, col0 + i): scale, additive mask, key padding, causal and sequence bounds.
// Masked entries become -inf.  `plain` = nothing but the scale applies to this block.  MSK: 0 no masks, 1 key padding only,
// 2 an additive mask (with or without key padding); `dead`: bit i set = key col0 + i is padding (dead_keys).
template <int NC, int MSK>
__device__ __forceinline__ void score_chunk(float* x, int row, int col0, uint32_t dead, const MaskArgs& m, bool plain) {
  static_assert(NC == 32, "one word of bits");
#pragma unroll
  for (int i = 0; i < NC; ++i) x[i] *= m.scale_log2;
  if (plain) return;
  if constexpr (MSK == 2) {
  if (row < m.Sq) {
    if (m.mask_fp32) {
      const float* mp = reinterpret_cast<const float*>(m.mask) + (long long)row * m.mask_ld + col0;
      if (col0 + NC <= m.Sk && (reinterpret_cast<uintptr_t>(mp) & 15) == 0) {
#pragma unroll
        for (int q = 0; q < NC / 4; ++q) {
          const float4 v = __ldg(reinterpret_cast<const float4*>(mp) + q);
          x[4 * q] += v.x * kLog2e; x[4 * q + 1] += v.y * kLog2e; x[4 * q + 2] += v.z * kLog2e; x[4 * q + 3] += v.w * kLog2e;
        }
      } else {
#pragma unroll
        for (int i = 0; i < NC; ++i) if (col0 + i < m.Sk) x[i] += __ldg(mp + i) * kLog2e;
      }
    } else {
      const __nv_bfloat16* mp = reinterpret_cast<const __nv_bfloat16*>(m.mask) + (long long)row * m.mask_ld + col0;
      if (col0 + NC <= m.Sk && (reinterpret_cast<uintptr_t>(mp) & 15) == 0) {
#pragma unroll
        for (int q = 0; q < NC / 8; ++q) {
          const uint4 v = __ldg(reinterpret_cast<const uint4*>(mp) + q);
          x[8 * q] += bf16_lo(v.x) * kLog2e; x[8 * q + 1] += bf16_hi(v.x) * kLog2e;
          x[8 * q + 2] += bf16_lo(v.y) * kLog2e; x[8 * q + 3] += bf16_hi(v.y) * kLog2e;
          x[8 * q + 4] += bf16_lo(v.z) * kLog2e; x[8 * q + 5] += bf16_hi(v.z) * kLog2e;
          x[8 * q + 6] += bf16_lo(v.w) * kLog2e; x[8 * q + 7] += bf16_hi(v.w) * kLog2e;
        }
      } else {
#pragma unroll
        for (int i = 0; i < NC; ++i) if (col0 + i < m.Sk) x[i] += __bfloat162float(__ldg(mp + i)) * kLog2e;
      }
    }
  }
  }
  // bit i: key col0 + i has no weight
  uint32_t off = MSK ? dead : 0u;
  if (m.causal && col0 + NC - 1 > row) off |= row < col0 ? 0xffffffffu : 0xffffffffu << (row + 1 - col0);
  if (col0 + NC > m.Sk) off |= col0 >= m.Sk ? 0xffffffffu : 0xffffffffu << (m.Sk - col0);
  if (off) {
#pragma unroll
    for (int i = 0; i < NC; ++i) if ((off >> i) & 1u) x[i] = -INFINITY;
  }
}
// Padding bits of keys col0 .. col0 + 31, one byte per lane and a ballot (the warp works on one batch entry and one range
// of keys).  Every row thread used to load all of its block's bytes, beside the additive mask's code: 6 x 12 heads of
// 700 x 700, head_dim 64, padded: forward 84 -> 46 us, dQ 64 -> 53, dK / dV 124 -> 61 (unmasked 37, 45, 61).
template <int MSK>
__device__ __forceinline__ uint32_t dead_keys(const MaskArgs& m, int b, int col0, int lane) {
  if constexpr (MSK == 0) return 0u;
  if (!m.kpm) return 0u;
  const int col = col0 + lane;
  return __ballot_sync(0xffffffffu, col < m.Sk && __ldg(m.kpm + (long long)b * m.kpm_ld + col) != 0);
}
// keep bits of the NC probabilities (row, col0 ..) of head-batch bh: bit i set = kept.  Needs Sk % 4 == 0.
template <int NC>
__device__ __forceinline__ uint32_t keep_bits(const MaskArgs& m, unsigned long long offset, long long bh, int row, int col0) {
  static_assert(NC <= 32, "keep mask is one word");
  const unsigned long long e4 = (((unsigned long long)bh * m.Sq + row) * (unsigned long long)m.Sk + col0) >> 2;
  uint32_t bits = 0;
#pragma unroll
  for (int g = 0; g < NC / 4; ++g) {
    const uint4 r = philox4x32(m.seed, offset, e4 + g);
    bits |= ((r.x >= m.thresh ? 1u : 0u) | (r.y >= m.thresh ? 2u : 0u) | (r.z >= m.thresh ? 4u : 0u) |
             (r.w >= m.thresh ? 8u : 0u)) << (4 * g);
  }
  return bits;
}

// Common set-up: barriers, TMEM, abort flag.  Returns the TMEM base.
__device__ __forceinline__ uint32_t setup_cta(Ctl* ctl, const int* counts, int nbar, int warp, int lane) {
  if (warp == kProducerWarp) {
    if (lane < nbar) mbar_init(&ctl->bar[lane], counts[lane]);
    if (lane == 31) ctl->abort_flag = 0;
    mbar_fence_init();
    __syncwarp();
    tmem_alloc(&ctl->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();      // every CTA owns its TMEM columns first (see launch.h)
  pdl_wait();
  return ctl->tmem_base;
}
__device__ __forceinline__ void teardown_cta(uint32_t tmem, int warp) {
  tc_fence_before();
  __syncthreads();
  if (warp == kProducerWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Two fp32 operations in one instruction (each rounded as the single one is).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.ftz.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.ftz.f32x2 x, x, y;\n\t"
      "mov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.ftz.f32x2 x, x, y;\n\t"
      "mov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
// 2^x of two numbers that are not NaN on the multiply-add pipes, x >= -126 or taken as that: 2^round(x) rides in as an exponent, the
// rest is a polynomial of degree 6 in [-1/2, 1/2] (least maximum relative error, by Remez exchange).  Relative error up to 1.1e-7
// in fp32, not above ex2.approx; twice its instructions, but the special-function unit has only four lanes an SM quarter.
__device__ __forceinline__ float2 ex2_poly2(float2 t) {
  const float2 magic = make_float2(12582912.f, 12582912.f);       // 1.5 * 2^23: rounds to integers, which stay in the low bits
  t.x = fmaxf(t.x, -126.f);
  t.y = fmaxf(t.y, -126.f);
  const float2 r = add2(t, magic);
  const float2 n = add2(r, make_float2(-12582912.f, -12582912.f));
  const float2 f = fma2(n, make_float2(-1.f, -1.f), t);
  float2 p = make_float2(1.3652998313773423e-4f, 1.3652998313773423e-4f);
  p = fma2(p, f, make_float2(1.3320884900167584e-3f, 1.3320884900167584e-3f));
  p = fma2(p, f, make_float2(9.6239959821105e-3f, 9.6239959821105e-3f));
  p = fma2(p, f, make_float2(5.550621822476387e-2f, 5.550621822476387e-2f));
  p = fma2(p, f, make_float2(0.24022623896598816f, 0.24022623896598816f));
  p = fma2(p, f, make_float2(0.6931469440460205f, 0.6931469440460205f));
  p = fma2(p, f, make_float2(1.f, 1.f));
  return make_float2(__int_as_float(__float_as_int(p.x) + (__float_as_int(r.x) << 23)),
                     __int_as_float(__float_as_int(p.y) + (__float_as_int(r.y) << 23)));
}
__device__ __forceinline__ float max64(const float* s) {
  float m0 = s[0], m1 = s[1], m2 = s[2], m3 = s[3];
#pragma unroll
  for (int i = 4; i < 60; i += 8) {
    m0 = max3(m0, s[i], s[i + 1]); m1 = max3(m1, s[i + 2], s[i + 3]);
    m2 = max3(m2, s[i + 4], s[i + 5]); m3 = max3(m3, s[i + 6], s[i + 7]);
  }
  return max3(max3(max3(m0, m1, m2), m3, s[60]), s[61], max3(s[61], s[62], s[63]));
}
// The CTAs are persistent: when a role is done with one piece of work it goes on with the next, so that copies and products of
// the next run under the end of the last, and TMEM and barriers are set up once.  A CTA's first work is its own blockIdx.x; from
// then on one thread asks for a CTA that has not started yet (the longest are numbered first).  It asks when every role has begun
// the current piece and the producer has copied all of it, no earlier: asked for at the beginning of the piece before, work was
// tied to CTAs that were not the first to be free (16 heads of 8192 x 8192, head_dim 128, causal: forward 292 us, 249 without
// persistence).  A launch that fits the SMs at once has nothing to ask for (MORE = false)
// and is better off without the instruction: with it in the kernel, dependent launch around it no longer overlaps (32 heads of
// 256 x 256, head_dim 64: backward 10.3 -> 13.5 us).
__device__ __forceinline__ void schedule(Ctl* ctl, uint64_t* full, uint64_t* taken, volatile uint32_t* abort_flag,
                                         unsigned long long* status, unsigned long long tmo) {
  for (uint32_t n = 0;; ++n) {
    if (!mbar_wait(taken, n & 1u, abort_flag, status, tmo)) return;
    fence_proxy_async_smem();          // all roles have read the last answer: the next may be written over it
    mbar_arrive_expect_tx(full, 16);
    clc_try_cancel(&ctl->next, full);
    if (!mbar_wait(full, n & 1u, abort_flag, status, tmo)) {
      const unsigned long long t0 = globaltimer_ns();            // the answer lands (bounded) before the CTA may exit
      while (!mbar_try_wait(full, n & 1u))
        if (globaltimer_ns() - t0 > 2000000ull) break;
      return;
    }
    if (clc_answer(&ctl->next) < 0) return;
  }
}
// For every role, by all lanes of a warp or by one thread: the n-th next piece of work, -1: none, or a wait ran out.  The role
// arrives on `taken` once for each piece, the first included.
__device__ __forceinline__ int next_work(Ctl* ctl, uint64_t* full, uint32_t n, bool whole_warp, volatile uint32_t* abort_flag,
                                         unsigned long long* status, unsigned long long tmo) {
  uint32_t good = mbar_wait(full, n & 1u, abort_flag, status, tmo) ? 1u : 0u;
  if (whole_warp) good = __all_sync(0xffffffffu, good);
  if (!good) return -1;
  const int w = clc_answer(&ctl->next);
  if (whole_warp) __syncwarp();
  return w;
}
// After an abort: wait (bounded) for the copies this thread has issued, so that none lands in a dead CTA.
__device__ __forceinline__ void drain_loads(uint64_t* bars, uint32_t used, uint32_t parity) {
  for (int i = 0; i < 32; ++i) {
    if (!((used >> i) & 1u)) continue;
    const unsigned long long t0 = globaltimer_ns();
    while (!mbar_try_wait(&bars[i], (parity >> i) & 1u)) {
      if (globaltimer_ns() - t0 > 2000000ull) break;
    }
  }
}
__device__ __forceinline__ void drain_mma(uint64_t* bar) {
  umma_commit(bar);
  const unsigned long long t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, 0)) {
    if (globaltimer_ns() - t0 > 2000000ull) break;
  }
}

// bf16 of 32 values into 16 columns of this thread's lane
__device__ __forceinline__ void store_bf16x32(uint32_t taddr, const float* v) {
  uint32_t pk[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) pk[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
  tmem_st16(taddr, pk);
}
// A warp's part of P or dS is in TMEM: one arrival for it.
__device__ __forceinline__ void publish_rows(uint64_t* bar, int lane) {
  tmem_st_wait();
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}
// Waits of all lanes of a warp; false for all if one ran out.  Not polled as the issuer's are: forward and backward of 16 heads of
// 8192 x 8192 x 128 took 1 036 us polled, 1 028 suspended, shorter ones the same either way.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag, unsigned long long* status,
                                          unsigned long long tmo) {
  const uint32_t good = mbar_wait(bar, parity, abort_flag, status, tmo) ? 1u : 0u;
  return __all_sync(0xffffffffu, good);
}
// D[128 x 128] = A B^T of two [128 x HD] K-major tiles
template <int HD>
__device__ __forceinline__ void umma_tiles(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc) {
#pragma unroll
  for (int u = 0; u < HD / 64; ++u)
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      umma_bf16(d, make_smem_desc(a + u * kSub + kk * 32, 16, 1024), make_smem_desc(b + u * kSub + kk * 32, 16, 1024), idesc,
                (u | kk) ? 1u : 0u);
}
// D[128 x HD] += A B: A the two halves of a [128 x 128] bf16 operand in TMEM, 64 columns apart, B a [128 x HD] tile read MN-major
__device__ __forceinline__ void umma_rows(uint32_t d, uint32_t a_tmem, uint32_t b, uint32_t idesc, bool add) {
#pragma unroll
  for (int kk = 0; kk < 8; ++kk)
    umma_bf16_ts(d, a_tmem + (kk >> 2) * 64 + (kk & 3) * 8, make_smem_desc(b + kk * 2048, kSub, 1024), idesc,
                 (add || kk > 0) ? 1u : 0u);
}

// =====================================================================================================  forward
// Two row tiles a CTA, one warpgroup each (thread = row), so that the softmax of one tile runs under the products of the
// other: per 128 x 128 block the tensor cores need 1 024 clocks at head_dim 128 and the exponentials 1 024 (16 a clock),
// and with both tiles in flight neither waits for the other's chain S -> softmax -> P V.  P goes back into the tile's own S
// columns as bf16 and is the TMEM operand of P V: through shared memory (a 32 KB tile written, then read at the rate of the
// UMMA itself) and with one tile a CTA the block took 2 750 clocks, now 1 700.  One exponential in four goes through the
// multiply-add pipes (ex2_poly2): 266 -> 246 us at 16 heads of 8192 x 8192 x 128.  The UMMAs of a CTA run in the order of their issue, so
// S(i + 1) of a tile may follow P V(i) into the same columns, and S(i + 1) complete means O is complete up to i.
// `split`: both tiles are the SAME 128 queries and take turns at the key blocks (tile t: blocks t, t + 2, ..); the two partial
// results are merged at the end.  Taken where the launch has too few row tiles to fill the SMs twice (see rtp_flash_fwd).
// barriers
enum { F_QFULL = 0 /* 2 tiles */, F_QEMPTY = 2 /* 2 */, F_KFULL = 4 /* 2 stages */, F_KEMPTY = 6, F_VFULL = 8, F_VEMPTY = 10,
       F_SFULL = 12 /* 2 tiles */, F_PFULL = 14 /* 2 */, F_PTAIL = 16 /* 2 */, F_OFULL = 18 /* 2 */, F_WFULL = 20, F_TAKEN = 21,
       F_DRAIN = 22 };

// What blockIdx.x stands for: row tiles g0 (and g0 + 1) of head h of batch entry b, with n0 and n1 steps; nload key blocks in all.
struct FwdWork {
  int g0, bh, b, h, n0, n1, nload;
};
__device__ __forceinline__ FwdWork fwd_work(const FlashParams& p, int blk) {
  const int nqb = (p.m.Sq + kBlk - 1) / kBlk, nkb = (p.m.Sk + kBlk - 1) / kBlk, BH = p.B * p.H;
  // row tiles of a piece of work: one or two; heaviest (last) query blocks of a group of heads first
  const int nt = p.split ? nqb : (nqb + 1) >> 1, span = p.group * nt;
  int grp = 0;
  if (blk >= span) {
    const int g = blk / span;
    grp = g * p.group;
    blk -= g * span;
  }
  const int heads = min(p.group, BH - grp), level = blk / heads;
  FwdWork w;
  w.g0 = (nt - 1 - level) * (p.split ? 1 : 2);
  w.bh = grp + blk - level * heads;
  w.b = w.bh / p.H;
  w.h = w.bh - w.b * p.H;
  const int nb0 = p.m.causal ? min(nkb, w.g0 + 1) : nkb;            // key blocks of the first tile, of the second
  const int nb1 = w.g0 + 1 >= nqb ? 0 : p.m.causal ? min(nkb, w.g0 + 2) : nkb;
  w.n0 = p.split ? (nb0 + 1) >> 1 : nb0;
  w.n1 = p.split ? nb0 >> 1 : nb1;
  w.nload = p.split ? nb0 : max(nb0, nb1);
  return w;
}

template <int HD, int MSK, bool DRP, bool MORE>
__global__ void __launch_bounds__(kThreads, 1) flash_fwd_kernel(const __grid_constant__ FlashParams p) {
  constexpr int SUB = HD / 64;
  constexpr int TILE = SUB * kSub;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = sm;                   // 2 tiles (split: the first serves both)
  uint8_t* sK = sQ + 2 * TILE;        // 2 stages
  uint8_t* sV = sK + 2 * TILE;        // 2 stages
  Ctl* ctl = reinterpret_cast<Ctl*>(sV + 2 * TILE);
  float* sX = reinterpret_cast<float*>(sV + 2 * TILE + 256);        // split: {maximum, sum} of each row and tile
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const MaskArgs& M = p.m;
  const bool split = p.split;                                       // one wave: no CTA has a second piece of work

  // counts by barrier index: copies and commits 1 each, P (its first three quarters, its last) 4: one per row warp of the tile,
  // next work 1 and 10 (producer, issuer, eight row warps)
  const int counts[23] = {1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 4, 4, 4, 4, 1, 1, 1, 10, 1};
  // The first work is looked up before the wait for the previous kernel: its divisions took 1 000 clocks between set-up and the first
  // copy, of the 12 000 of a launch of one key block (4 x 8 heads of 64 x 64).
  const FwdWork first = fwd_work(p, (int)blockIdx.x);
  asm volatile("" ::"r"(first.b), "r"(first.h), "r"(first.g0), "r"(first.nload));
  const uint32_t tmem = setup_cta(ctl, counts, 23, warp, lane);
  volatile uint32_t* abort_flag = &ctl->abort_flag;
  unsigned long long* status = p.status;
  const unsigned long long tmo = p.timeout_ns;
  uint64_t* bar = ctl->bar;
  auto following = [&](uint32_t n, bool whole_warp) {
    return MORE ? next_work(ctl, &bar[F_WFULL], n, whole_warp, abort_flag, status, tmo) : -1;
  };

  if (warp >= kProducerWarp) {
  reg_dealloc<kAuxRegs>();
  if (warp == kProducerWarp) {
    // ---------------------------------------------------------------------------------- TMA producer
    if (elect_one()) {
      bool ok = true;
      uint32_t used = 0, par = 0, nkv = 0, nq[2] = {0, 0};          // barriers with copies, parity of their last
      auto load = [&](int full, uint32_t ph, uint8_t* dst, const CUtensorMap* map, int seq1, int col, int b, int s0) {
        mbar_arrive_expect_tx(&bar[full], TILE);
        load_tile<SUB>(smem_u32(dst), map, seq1, col, b, s0, smem_u32(&bar[full]));
        used |= 1u << full;
        par = (par & ~(1u << full)) | (ph << full);
      };
      auto wait = [&](int i, uint32_t ph) { return mbar_wait(&bar[i], ph, abort_flag, status, tmo); };
      uint32_t n = 0;
      for (int blk = (int)blockIdx.x; blk >= 0 && ok; blk = following(n++, false)) {
        const FwdWork w = n == 0 ? first : fwd_work(p, blk);
        const int b = w.b, h = w.h;
        const int cq = head_col(p.q, h), ck = head_col(p.k, h), cv = head_col(p.v, h);
        auto load_q = [&](int t) {
          const uint32_t ph = nq[t]++ & 1u;
          if (!wait(F_QEMPTY + t, ph ^ 1u)) return false;
          load(F_QFULL + t, ph, sQ + t * TILE, &p.mq, p.q_seq1, cq, b, (w.g0 + t) * kBlk);
          return true;
        };
        ok = load_q(0);
        for (int j = 0; j < w.nload && ok; ++j, ++nkv) {
          const int st = nkv & 1;
          const uint32_t ph = (nkv >> 1) & 1u;
          if (!wait(F_KEMPTY + st, ph ^ 1u)) { ok = false; break; }
          load(F_KFULL + st, ph, sK + st * TILE, &p.mk, p.k_seq1, ck, b, j * kBlk);
          if (j == 0 && !split && w.n1 > 0 && !load_q(1)) { ok = false; break; }
          if (!wait(F_VEMPTY + st, ph ^ 1u)) { ok = false; break; }
          load(F_VFULL + st, ph, sV + st * TILE, &p.mv, p.v_seq1, cv, b, j * kBlk);
        }
        if (!ok) break;
        mbar_arrive(&bar[F_TAKEN]);
      }
      if (!ok || *abort_flag) drain_loads(bar, used, par);
    }
  } else if (warp == kMmaWarp) {
    // ---------------------------------------------------------------------------------- UMMA issuer
    if (elect_one()) {
      const uint32_t id_s = make_idesc_bf16(128, 128, 0, 0), id_o = make_idesc_bf16(128, HD, 0, 1);
      const uint32_t aQ = smem_u32(sQ), aK = smem_u32(sK), aV = smem_u32(sV);
      bool ok = true, issued = false;
      auto wait = [&](int i, uint32_t ph) { return mbar_spin(&bar[i], ph, abort_flag, status, tmo); };
      // S of tile t against the c-th block since the start, once that is there; `last`: no other tile needs the block
      auto issue_s = [&](int t, uint32_t c, bool last, bool q_done) {
        if (!wait(F_KFULL + (c & 1), (c >> 1) & 1u)) return false;
        tc_fence_after();
        umma_tiles<HD>(tmem + (uint32_t)(t * 128), aQ + (split ? 0 : t * TILE), aK + (c & 1) * TILE, id_s);
        if (last) umma_commit(&bar[F_KEMPTY + (c & 1)]);
        if (q_done) umma_commit(&bar[F_QEMPTY + t]);
        umma_commit(&bar[F_SFULL + t]);
        issued = true;
        return true;
      };
      uint32_t n = 0, kv0 = 0, np[2] = {0, 0}, nq[2] = {0, 0};      // blocks before this work, P tiles and Q tiles so far
      for (int blk = (int)blockIdx.x; blk >= 0 && ok; blk = following(n++, false)) {
        const FwdWork w = n == 0 ? first : fwd_work(p, blk);
        const int n0 = w.n0, n1 = w.n1;
        mbar_arrive(&bar[F_TAKEN]);
        ok = wait(F_QFULL, nq[0]++ & 1u) && issue_s(0, kv0, split || n1 == 0, !split && n0 == 1);
        if (ok && n1 > 0) {
          if (!split) ok = wait(F_QFULL + 1, nq[1]++ & 1u);
          ok = ok && issue_s(1, kv0 + (split ? 1 : 0), true, !split && n1 == 1);
        }
        const int nmax = max(n0, n1);
        for (int i = 0; i < nmax && ok; ++i) {
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int nt = t ? n1 : n0;
            if (!ok || i >= nt) continue;
            const uint32_t c = kv0 + (split ? 2 * i + t : i);
            const int st = c & 1;
            // the block's second tile releases it; a tile that is done no longer counts
            const bool last = split || t == 1 || i >= n1;
            const uint32_t pp = np[t]++ & 1u;
            if (!wait(F_VFULL + st, (c >> 1) & 1u) || !wait(F_PFULL + t, pp)) { ok = false; break; }
            tc_fence_after();
            const uint32_t vb = aV + st * TILE, pt = tmem + (uint32_t)(t * 128), d = tmem + (uint32_t)(256 + t * HD);
#pragma unroll
            for (int kk = 0; kk < 6; ++kk)
              umma_bf16_ts(d, pt + kk * 8, make_smem_desc(vb + kk * 2048, kSub, 1024), id_o, (i > 0 || kk > 0) ? 1u : 0u);
            if (!wait(F_PTAIL + t, pp)) { ok = false; break; }
            tc_fence_after();
#pragma unroll
            for (int kk = 6; kk < 8; ++kk)
              umma_bf16_ts(d, pt + kk * 8, make_smem_desc(vb + kk * 2048, kSub, 1024), id_o, 1u);
            if (last) umma_commit(&bar[F_VEMPTY + st]);
            if (i + 1 < nt) ok = issue_s(t, split ? c + 2 : c + 1, split || t == 1 || i + 1 >= n1, !split && i + 2 == nt);
            else umma_commit(&bar[F_OFULL + t]);
          }
        }
        kv0 += w.nload;
        if (!ok) break;
      }
      if ((!ok || *abort_flag) && issued) drain_mma(&bar[F_DRAIN]);
    }
  } else if (warp == kSchedWarp) {
    if (MORE && elect_one()) schedule(ctl, &bar[F_WFULL], &bar[F_TAKEN], abort_flag, status, tmo);
  }
  } else {
    reg_alloc<kRowRegs>();
    // ---------------------------------------------------------------------------------- row threads
    const int t = warp >> 2, rt = tid & 127;           // tile and row of this thread
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t aS = lane_addr + (uint32_t)(t * 128), aO = lane_addr + (uint32_t)(256 + t * HD);
    const unsigned long long offset = M.offset + (M.step_ptr ? __ldg(M.step_ptr) * 65536ull : 0ull);
    bool ok = true;
    uint32_t ns = 0, no = 0, n = 0;                    // S tiles, O tiles, pieces of work so far
    // stamps of the two tiles' first warps of CTA 0: [warp 0 | warp 4][step < 16][event < 8]
    long long* tr = (p.trace && blockIdx.x == 0 && lane == 0 && (warp & 3) == 0) ? p.trace + (warp >> 2) * 128 : nullptr;
    for (int blk = (int)blockIdx.x; blk >= 0; blk = following(n++, true)) {
    const FwdWork w = n == 0 ? first : fwd_work(p, blk);
    if (lane == 0) mbar_arrive(&bar[F_TAKEN]);
    const int bh = w.bh, b = w.b, h = w.h, n1 = w.n1;
    const int nt = t ? n1 : w.n0, gt = w.g0 + (split ? 0 : t);
    const int row = gt * kBlk + rt;
    float m_used = -INFINITY, l = 0.f;
    for (int i = 0; i < nt; ++i, ++ns) {
      const int c = split ? 2 * i + t : i, col0 = c * kBlk;
      if (tr && ns < 16) tr[ns * 8 + 0] = clock64();
      uint32_t dead[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) dead[q] = dead_keys<MSK>(M, b, col0 + 32 * q, lane);
      const uint32_t good = mbar_wait(&bar[F_SFULL + t], ns & 1u, abort_flag, status, tmo) ? 1u : 0u;
      if (!__all_sync(0xffffffffu, good)) { ok = false; break; }
      tc_fence_after();
      if (tr && ns < 16) tr[ns * 8 + 1] = clock64();
      // A block that needs more than the scale is put right in TMEM first, 32 or 64 columns at a time, so that the loop below is one
      // for all blocks; one that only needs the scale keeps the raw scores: the scale rides in the exponent's multiply-add.
      const bool plain = MSK != 2 && !(dead[0] | dead[1] | dead[2] | dead[3]) && !(M.causal && c == gt) && (col0 + kBlk <= M.Sk) &&
                         M.scale_log2 >= 0.f;          // the maximum commutes with a positive scale only
      if (!plain) {
        constexpr int NQ = MSK == 2 ? 1 : 2;           // chunks at a time: the additive mask's code is long
#pragma unroll 1
        for (int q = 0; q < 4; q += NQ) {
          float x[32 * NQ];
#pragma unroll
          for (int u = 0; u < NQ; ++u) tmem_ld32f(aS + (uint32_t)((q + u) * 32), x + 32 * u);
          tmem_ld_wait();
#pragma unroll
          for (int u = 0; u < NQ; ++u) {
            const uint32_t dd = q + u == 0 ? dead[0] : q + u == 1 ? dead[1] : q + u == 2 ? dead[2] : dead[3];
            score_chunk<32, MSK>(x + 32 * u, row, col0 + 32 * (q + u), dd, M, false);
            tmem_st32f(aS + (uint32_t)((q + u) * 32), x + 32 * u);
          }
        }
        tmem_st_wait();
      }
      float s[128];
      tmem_ld32f(aS, s);
      tmem_ld32f(aS + 32, s + 32);
      tmem_ld_wait();
      tmem_ld32f(aS + 64, s + 64);
      tmem_ld32f(aS + 96, s + 96);
      float mx = max64(s);
      tmem_ld_wait();
      mx = max3(mx, mx, max64(s + 64));
      if (plain) mx *= M.scale_log2;
      const float cand = fmaxf(m_used, mx);
      const bool need = cand > m_used + kRescaleGap;
      const float m_new = need ? cand : m_used;
      const float mref = (m_new == -INFINITY) ? 0.f : m_new;
      const float mul = plain ? M.scale_log2 : 1.f;
      // some: one exponential in four by polynomial.  That is for blocks without masked scores, which have to become 0, whose rows
      // all have a finite maximum: a NaN or an infinite score has to reach the output, and a row of -inf alone has no weights;
      // a -inf below a finite maximum gets 2^-126 beside 2^-8 or more.
      const bool fin = fabsf(mx) < INFINITY;
      bool some = !DRP && plain;
      if (__any_sync(0xffffffffu, (i > 0 && need) || !fin)) {
        if (i > 0 && __any_sync(0xffffffffu, need)) {
          // the S that was waited for came after the P V of the tile's previous step: O is complete up to there
          const float alpha = need ? ex2_approx(m_used - cand) : 1.f;
#pragma unroll
          for (int q = 0; q < HD / 32; ++q) {
            float o[32];
            tmem_ld32f(aO + (uint32_t)(q * 32), o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] *= alpha;
            tmem_st32f(aO + (uint32_t)(q * 32), o);
          }
          l *= alpha;
        }
        some = some && __all_sync(0xffffffffu, fin);
      }
      float2 ra = make_float2(0.f, 0.f), rb = ra;
      const float2 mul2 = make_float2(mul, mul), ref2 = make_float2(-mref, -mref);
      auto exponentials = [&](auto poly) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float* e = s + 32 * q;
        uint32_t pk[16];
        [[maybe_unused]] uint32_t keep = 0xffffffffu;
        if constexpr (DRP) keep = keep_bits<32>(M, offset, bh, min(row, M.Sq - 1), col0 + 32 * q);
#pragma unroll
        for (int k = 0; k < 32; k += 4) {
          float2 x = fma2(make_float2(e[k], e[k + 1]), mul2, ref2), y = fma2(make_float2(e[k + 2], e[k + 3]), mul2, ref2);
          x = make_float2(ex2_approx(x.x), ex2_approx(x.y));
          if (decltype(poly)::value && (k & 4)) y = ex2_poly2(y);
          else y = make_float2(ex2_approx(y.x), ex2_approx(y.y));
          ra = add2(ra, x);
          rb = add2(rb, y);
          if constexpr (DRP) {
            x.x = ((keep >> k) & 1u) ? x.x * M.drop_scale : 0.f;
            x.y = ((keep >> (k + 1)) & 1u) ? x.y * M.drop_scale : 0.f;
            y.x = ((keep >> (k + 2)) & 1u) ? y.x * M.drop_scale : 0.f;
            y.y = ((keep >> (k + 3)) & 1u) ? y.y * M.drop_scale : 0.f;
          }
          pk[k / 2] = pack_bf16(x.x, x.y);
          pk[k / 2 + 1] = pack_bf16(y.x, y.y);
        }
        tmem_st16(aS + (uint32_t)(q * 16), pk);
        if (q >= 2) {          // three quarters of P: their products run under the exponentials of the last
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar[(q == 2 ? F_PFULL : F_PTAIL) + t]);
        }
      }
      };
      if (some) exponentials(std::true_type{}); else exponentials(std::false_type{});
      m_used = m_new;
      l += (ra.x + ra.y) + (rb.x + rb.y);
      if (tr && ns < 16) tr[ns * 8 + 2] = clock64();
    }
    const int r0 = gt * kBlk + (warp & 3) * 32;        // the warp's first row
    __nv_bfloat16* const dst = row_ptr(p.o, b, r0, h);
    const bool lone = split && n1 == 0;                // one key block: the tile's second warpgroup takes half of the columns
    if (lone) {
      if (t == 0) {
        sX[rt] = m_used;
        sX[128 + rt] = l;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");   // under the product P V
      m_used = sX[rt];
      l = sX[128 + rt];
    }
    const bool stores = nt > 0 || lone;
    if (ok && stores) {
      const uint32_t good = mbar_wait(&bar[F_OFULL + (lone ? 0 : t)], no++ & 1u, abort_flag, status, tmo) ? 1u : 0u;
      if (!__all_sync(0xffffffffu, good)) ok = false;
    }
    tc_fence_after();
    const bool merge = split && n1 > 0;
    constexpr int OC = HD / 64;                        // 32-column chunks of half a row
    float a_own = 1.f, a_other = 0.f;
    if (merge) {
      // Each thread of a row finishes half of its columns: it hands the other half, its maximum and its sum to the other
      // tile's thread.  The products have read K (every S was issued before the last P V), so its stages hold the floats.
      float* xo = reinterpret_cast<float*>(sK) + t * (HD / 2) * 128;
      if (ok) {
#pragma unroll
        for (int q = 0; q < OC; ++q) {
          float o[32];
          tmem_ld32f(aO + (uint32_t)((t ^ 1) * (HD / 2) + q * 32), o);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) xo[(q * 32 + e) * 128 + rt] = o[e];
        }
        sX[t * 256 + rt] = m_used;
        sX[t * 256 + 128 + rt] = l;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");   // all row threads come here, whether their waits ran out or not
      const float m_o = sX[(t ^ 1) * 256 + rt], l_o = sX[(t ^ 1) * 256 + 128 + rt];
      const float m_all = fmaxf(m_used, m_o);
      a_own = m_used == -INFINITY ? 0.f : ex2_approx(m_used - m_all);
      a_other = m_o == -INFINITY ? 0.f : ex2_approx(m_o - m_all);
      l = l * a_own + l_o * a_other;
      m_used = m_all;
    }
    if (ok && stores) {
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const float* xi = reinterpret_cast<const float*>(sK) + (t ^ 1) * (HD / 2) * 128;
      const int c0 = split ? t * OC : 0, c1 = split ? c0 + OC : 2 * OC;
      const uint32_t aR = lone ? lane_addr + 256u : aO;
      for (int q = c0; q < c1; ++q) {
        float o[32];
        tmem_ld32f(aR + (uint32_t)(q * 32), o);
        tmem_ld_wait();
        if (merge) {
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = o[e] * a_own + xi[((q - c0) * 32 + e) * 128 + rt] * a_other;
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] *= inv;
        store_rows32(dst + q * 32, p.o.ss, M.Sq - r0, o, lane);
      }
      if (row < M.Sq && p.lse && !(split && t)) {
        const float mref = (m_used == -INFINITY) ? 0.f : m_used;
        p.lse[(long long)bh * M.Sq + row] = l > 0.f ? mref + log2f(l) : INFINITY;
      }
      tc_fence_before();               // O has been read before the next P is announced
    }
    if (!ok) break;
    }
  }
  teardown_cta(tmem, warp);
}

// =====================================================================================================  backward
// delta[b, h, q] = rowsum(dO * O), HD / 8 lanes a row.  Reads both once (8192 tokens x 16 heads of 128: 67 MB), apart from the
// launch below so that its two kinds of CTAs need nothing of each other.
template <int HD>
__global__ void __launch_bounds__(256) flash_delta_kernel(DRef o, DRef g, float* __restrict__ delta, int Sq, int H, long long rows) {
  pdl_prologue();
  constexpr int LPR = HD / 8;
  const long long r = (blockIdx.x * 256ll + threadIdx.x) / LPR;
  const int c = threadIdx.x % LPR;
  float s = 0.f;
  const long long bs = r / H;                                // rows in memory order: (batch, position, head)
  const int h = (int)(r % H), b = (int)(bs / Sq), q = (int)(bs % Sq);
  if (r < rows) {
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(row_ptr(o, b, q, h)) + c);
    const uint4 y = __ldg(reinterpret_cast<const uint4*>(row_ptr(g, b, q, h)) + c);
    s = bf16_lo(x.x) * bf16_lo(y.x) + bf16_hi(x.x) * bf16_hi(y.x) + bf16_lo(x.y) * bf16_lo(y.y) + bf16_hi(x.y) * bf16_hi(y.y) +
        bf16_lo(x.z) * bf16_lo(y.z) + bf16_hi(x.z) * bf16_hi(y.z) + bf16_lo(x.w) * bf16_lo(y.w) + bf16_hi(x.w) * bf16_hi(y.w);
  }
#pragma unroll
  for (int d = LPR / 2; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  if (r < rows && c == 0) delta[((long long)b * H + h) * Sq + q] = s;
}

// Two kinds of work share one launch, the heaviest of each kind first: together they fill the SMs where either alone would
// leave some idle, and neither has a tail of its own.  The row threads (two a row, 64 of the 128 columns each) make P and then
// dS of a block; the products of one run under the other: while the rows work on dS(i) the tensor cores do dV(i) and S(i + 1),
// while they work on P(i + 1) dK(i) and dP(i + 1).  P and dS go back into the TMEM columns of S and dP as bf16 A operands: in
// shared memory, 64 columns a step, a block took 4 800 clocks in each of the two kernels there were, now 2 080 (dQ) and 3 100.
//
// dK / dV of 128 keys (rows of every product are KEYS), queries walked in blocks of 128, two stages of Q and dO:
//   S^T = K Q^T, dP^T = V dO^T  ->  P^T, dS^T  ->  dV += P^T dO, dK += dS^T Q
// dQ of 128 queries, keys walked in blocks of 128, three stages of K (dQ(i) still reads one while S(i + 2) needs another) and two of
// V, S double-buffered:
//   S = Q K^T, dP = dO V^T  ->  dS = P (dP - delta)  ->  dQ += dS K
//
// ONE: heads of one key block and one query block, a CTA a head: dS^T goes to shared memory too, where dQ reads it transposed.
//
// Shared memory is seven tiles, each with a "full" and an "empty" barrier of its own, whatever it holds: what follows is copied
// into a tile as soon as its last product is done, also across pieces of work.
//   dK / dV:  0 K   1 V   2, 3 Q   4, 5 dO            dQ:  0 Q   1 dO   2, 3, 4 K   5, 6 V
// TMEM: S 0, dP 128; dK / dV: dV 256, dK 256 + HD; dQ: dQ 256, second S 384.
// Barriers: tile t full t, empty 7 + t; the statistics of a block of queries (-log-sum-exp, -delta: the producer warp) beside
// its Q tile; accumulators complete, and read out.
enum { B_FULL = 0, B_EMPTY = 7, B_STAT = 14 /* 2 */, B_SFULL = 16 /* 2 */, B_PFULL = 18, B_DPFULL = 19, B_DSFULL = 20, B_ACC = 21,
       B_ACCREAD = 22, B_WFULL = 23, B_TAKEN = 24, B_DRAIN = 25 };

// What blockIdx.x stands for: the key block kb, or (kb < 0) the query block qb, of head h of batch entry b.
struct BwdWork {
  int kb, qb, bh, b, h;
};
__device__ __forceinline__ BwdWork bwd_work(const FlashParams& p, int blk) {
  const int nq = (p.m.Sq + kBlk - 1) / kBlk, nk = (p.m.Sk + kBlk - 1) / kBlk, BH = p.B * p.H, both = min(nq, nk), span = p.group * (nq + nk);
  // a group of heads: a key block of each, a query block of each and so on, the longest first (causal: first keys, last queries), then
  // what one kind has more
  int grp = 0;
  if (blk >= span) {
    const int g = blk / span;
    grp = g * p.group;
    blk -= g * span;
  }
  const int heads = min(p.group, BH - grp), row = blk / heads;
  BwdWork w = {-1, -1, grp + blk - row * heads, 0, 0};
  if (row < 2 * both) { if (row & 1) w.qb = nq - 1 - (row >> 1); else w.kb = row >> 1; }
  else if (nk > nq) w.kb = row - both;
  else w.qb = nq - 1 + both - row;
  w.b = w.bh / p.H;
  w.h = w.bh - w.b * p.H;
  return w;
}

constexpr int kBwdSlack = 768;          // all that a CTA's shared memory leaves for the alignment of the tiles (its base has it)

template <int HD, int MSK, bool DRP, bool MORE, bool ONE = false>
__global__ void __launch_bounds__(kThreads, 1) flash_bwd_kernel(const __grid_constant__ FlashParams p) {
  constexpr int TILE = (HD / 64) * kSub;
  extern __shared__ __align__(1024) uint8_t smem_tiles[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_tiles) + 1023) & ~uintptr_t(1023));
  if (sm - smem_tiles > kBwdSlack) {
    if (threadIdx.x == 0) atomicCAS(p.status, (unsigned long long)ST_OK, (unsigned long long)ST_BAD_ARGUMENT);
    return;
  }
  Ctl* ctl = reinterpret_cast<Ctl*>(sm + 7 * TILE);
  float* sStat = reinterpret_cast<float*>(sm + 7 * TILE + 256);     // two stages of 128 x -log-sum-exp, 128 x -delta
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const MaskArgs& M = p.m;
  const int nqb = (M.Sq + kBlk - 1) / kBlk, nkb = (M.Sk + kBlk - 1) / kBlk;
  // counts by barrier index: copies and commits 1; statistics 32 (lanes); P and dS, accumulators read 8 (one per row warp); next work
  // 1 and 10 (producer, issuer, eight row warps)
  const int counts[26] = {1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 32, 32, 1, 1, 8, 1, 8, 1, 8, 1, 10, 1};
  const BwdWork first = bwd_work(p, (int)blockIdx.x);       // before the wait for the previous kernel, as in forward
  asm volatile("" ::"r"(first.b), "r"(first.h), "r"(first.kb), "r"(first.qb));
  const uint32_t tmem = setup_cta(ctl, counts, 26, warp, lane);
  volatile uint32_t* abort_flag = &ctl->abort_flag;
  unsigned long long* status = p.status;
  const unsigned long long tmo = p.timeout_ns;
  uint64_t* bar = ctl->bar;
  const uint32_t tS = tmem, tP = tmem + 128, tAcc = tmem + 256;
  auto following = [&](uint32_t n, bool whole_warp) {
    return MORE ? next_work(ctl, &bar[B_WFULL], n, whole_warp, abort_flag, status, tmo) : -1;
  };

  if (warp >= kProducerWarp) {
  reg_dealloc<kAuxRegs>();
  if (warp == kProducerWarp) {
    // ---------------------------------------------------------------------------------- TMA producer
    // the whole warp goes through the work: lane 0 issues the copies, every lane fetches the statistics of four queries
    bool ok = true;
    uint32_t uses = 0, copied = 0, n = 0;               // per tile: parity of its next use; copies issued
    auto load = [&](int t, const CUtensorMap* map, int seq1, int col, int b, int s0) {
      const uint32_t ph = (uses >> t) & 1u;
      if (!warp_wait(&bar[B_EMPTY + t], ph ^ 1u, abort_flag, status, tmo)) return false;
      if (lane == 0) {
        mbar_arrive_expect_tx(&bar[B_FULL + t], TILE);
        load_tile<HD / 64>(smem_u32(sm + t * TILE), map, seq1, col, b, s0, smem_u32(&bar[B_FULL + t]));
      }
      uses ^= 1u << t;
      copied |= 1u << t;
      return true;
    };
    for (int blk = (int)blockIdx.x; blk >= 0 && ok; blk = following(n++, true)) {
      const BwdWork w = n == 0 ? first : bwd_work(p, blk);
      const int b = w.b, h = w.h;
      const int cq = head_col(p.q, h), ck = head_col(p.k, h), cv = head_col(p.v, h), cg = head_col(p.dout, h);
      if (w.kb >= 0) {
        const long long base = (long long)w.bh * M.Sq;
        const int i0 = M.causal ? w.kb : 0;
        ok = load(0, &p.mk, p.k_seq1, ck, b, w.kb * kBlk);
        for (int i = i0; i < nqb && ok; ++i) {
          const int st = (i - i0) & 1, q0 = i * kBlk;
          ok = load(2 + st, &p.mq, p.q_seq1, cq, b, q0);
          if (!ok) break;
          if (i == i0) ok = load(1, &p.mv, p.v_seq1, cv, b, w.kb * kBlk);
          ok = ok && load(4 + st, &p.mdo, p.do_seq1, cg, b, q0);
          float* stat = sStat + st * 2 * kBlk;          // free with its Q tile: dK read that after the rows had read these
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int q = q0 + e * 32 + lane;
            stat[e * 32 + lane] = q < M.Sq ? -__ldg(p.lse + base + q) : -INFINITY;
            stat[kBlk + e * 32 + lane] = q < M.Sq ? -__ldg(p.delta + base + q) : 0.f;
          }
          mbar_arrive(&bar[B_STAT + st]);
        }
      } else {
        const int nb = M.causal ? min(nkb, w.qb + 1) : nkb;
        ok = load(0, &p.mq, p.q_seq1, cq, b, w.qb * kBlk);
        for (int j = 0; j < nb && ok; ++j) {
          ok = load(2 + j % 3, &p.mk, p.k_seq1, ck, b, j * kBlk);
          if (ok && j == 0) ok = load(1, &p.mdo, p.do_seq1, cg, b, w.qb * kBlk);
          ok = ok && load(5 + (j & 1), &p.mv, p.v_seq1, cv, b, j * kBlk);
        }
      }
      if (!ok) break;
      if (lane == 0) mbar_arrive(&bar[B_TAKEN]);
    }
    if (lane == 0 && (!ok || *abort_flag)) drain_loads(bar + B_FULL, copied, ~uses);
  } else if (warp == kMmaWarp) {
    // ---------------------------------------------------------------------------------- UMMA issuer
    if (elect_one()) {
      const uint32_t id_s = make_idesc_bf16(128, 128, 0, 0), id_t = make_idesc_bf16(128, HD, 0, 1);
      [[maybe_unused]] const uint32_t id_q = make_idesc_bf16(128, HD, 1, 1);
      const uint32_t a0 = smem_u32(sm);
      bool ok = true, issued = false;
      uint32_t uses = 0, np = 0, nds = 0, n = 0;        // per tile: parity of its next use; P, dS and pieces of work so far
      auto wait = [&](int i, uint32_t ph) { return mbar_spin(&bar[i], ph, abort_flag, status, tmo); };
      auto tile = [&](int t) {
        const bool got = wait(B_FULL + t, (uses >> t) & 1u);
        uses ^= 1u << t;
        return got;
      };
      auto at = [&](int t) { return a0 + (uint32_t)(t * TILE); };
      auto done_with = [&](int t) { umma_commit(&bar[B_EMPTY + t]); };
      // S or dP = tile a x tile b, the second of which has to be waited for; tiles that are read for the last time are released
      auto product = [&](uint32_t d, int a, int bt, int sig, bool last_a, bool last_b) {
        if (!tile(bt)) return false;
        tc_fence_after();
        umma_tiles<HD>(d, at(a), at(bt), id_s);
        if (last_a) done_with(a);
        if (last_b) done_with(bt);
        umma_commit(&bar[sig]);
        issued = true;
        return true;
      };
      for (int blk = (int)blockIdx.x; blk >= 0 && ok; blk = following(n++, false)) {
        const BwdWork w = n == 0 ? first : bwd_work(p, blk);
        mbar_arrive(&bar[B_TAKEN]);
        const uint32_t read = (n & 1u) ^ 1u;            // the accumulators of the work before have been read out
        if (w.kb >= 0) {
          const int nit = nqb - (M.causal ? w.kb : 0);
          ok = tile(0) && product(tS, 0, 2, B_SFULL, nit == 1, false) && tile(1) && product(tP, 1, 4, B_DPFULL, nit == 1, false) &&
               wait(B_ACCREAD, read);
          for (int it = 0; it < nit && ok; ++it) {
            const int st = it & 1, ot = st ^ 1;
            const bool more = it + 1 < nit, end = it + 2 == nit;
            if (!wait(B_PFULL, np++ & 1u)) { ok = false; break; }
            tc_fence_after();
            umma_rows(tAcc, tS, at(4 + st), id_t, it > 0);
            done_with(4 + st);
            if (more && !product(tS, 0, 2 + ot, B_SFULL, end, false)) { ok = false; break; }
            if (!wait(B_DSFULL, nds++ & 1u)) { ok = false; break; }
            tc_fence_after();
            umma_rows(tAcc + HD, tP, at(2 + st), id_t, it > 0);
            if constexpr (ONE) {                         // dQ from dS^T in shared memory, into the columns of S
#pragma unroll
              for (int kk = 0; kk < 8; ++kk)
                umma_bf16(tS, make_smem_desc(at(5) + kk * 2048, kSub, 1024), make_smem_desc(at(0) + kk * 2048, kSub, 1024), id_q,
                          kk > 0 ? 1u : 0u);
            }
            done_with(2 + st);
            if (more) ok = product(tP, 1, 4 + ot, B_DPFULL, end, false);
            else umma_commit(&bar[B_ACC]);
          }
        } else {
          const int nb = M.causal ? min(nkb, w.qb + 1) : nkb;
          auto issue_s = [&](int j) {
            return product(j & 1 ? tmem + 384 : tS, 0, 2 + j % 3, B_SFULL + (j & 1), j + 1 == nb, false);
          };
          auto issue_dp = [&](int j) { return product(tP, 1, 5 + (j & 1), B_DPFULL, j + 1 == nb, true); };
          ok = tile(0) && issue_s(0) && tile(1) && issue_dp(0) && wait(B_ACCREAD, read) && (nb < 2 || issue_s(1));
          for (int j = 0; j < nb && ok; ++j) {
            if (!wait(B_DSFULL, nds++ & 1u)) { ok = false; break; }
            tc_fence_after();
            umma_rows(tAcc, tP, at(2 + j % 3), id_t, j > 0);
            done_with(2 + j % 3);
            if (j + 1 == nb) umma_commit(&bar[B_ACC]);
            else ok = issue_dp(j + 1) && (j + 2 >= nb || issue_s(j + 2));
          }
        }
        if (!ok) break;
      }
      if ((!ok || *abort_flag) && issued) drain_mma(&bar[B_DRAIN]);
    }
  } else if (warp == kSchedWarp) {
    if (MORE && elect_one()) schedule(ctl, &bar[B_WFULL], &bar[B_TAKEN], abort_flag, status, tmo);
  }
  } else {
    reg_alloc<kRowRegs>();
    // ---------------------------------------------------------------------------------- row threads
    const int wg = warp >> 2, rt = (warp & 3) * 32 + lane;       // column half and row of this thread
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t aP = tP + lane_off + (uint32_t)(wg * 64);
    const unsigned long long offset = M.offset + (M.step_ptr ? __ldg(M.step_ptr) * 65536ull : 0ull);
    const float2 sc = make_float2(M.scale_log2, M.scale_log2);
    bool ok = true;
    uint32_t n = 0, ns = 0, ndp = 0, nst = 0;                    // pieces of work, S per buffer (bits), dP, statistics per stage (bits)
    auto wait = [&](int i, uint32_t ph) { return warp_wait(&bar[i], ph, abort_flag, status, tmo); };
    long long* tr = (p.trace && blockIdx.x == 0 && lane == 0 && (warp & 3) == 0) ? p.trace + (warp >> 2) * 128 : nullptr;
    for (int blk = (int)blockIdx.x; blk >= 0 && ok; blk = following(n++, true)) {
      const BwdWork w = n == 0 ? first : bwd_work(p, blk);
      if (lane == 0) mbar_arrive(&bar[B_TAKEN]);
      const int bh = w.bh, b = w.b, h = w.h;
      if (w.kb >= 0) {
        const int k0 = w.kb * kBlk, i0 = M.causal ? w.kb : 0, nit = nqb - i0;
        const uint32_t aS = tS + lane_off + (uint32_t)(wg * 64);
        const int key = k0 + rt;
        bool key_dead = key >= M.Sk;
        if constexpr (MSK != 0) key_dead = key_dead || (M.kpm && __ldg(M.kpm + (long long)b * M.kpm_ld + key));
        const bool keys_plain = MSK != 2 && !__any_sync(0xffffffffu, key_dead);
        for (int it = 0; it < nit; ++it) {
          const int st = it & 1;
          const int qbase = (i0 + it) * kBlk + wg * 64;          // first query of this thread
          const float* nlse = sStat + st * 2 * kBlk + wg * 64;
          const float* ndel = nlse + kBlk;
          // Dropout bits.  One generator call covers four neighbouring keys, which sit in four neighbouring lanes: each lane
          // calls it for every fourth query and the four exchange their nibbles.
          uint32_t kw[2][4] = {};                                // kw[c][e]: nibble g = keys of the quad, query 32 c + 4 g + e
          if constexpr (DRP) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              uint32_t mine = 0;
#pragma unroll
              for (int g = 0; g < 8; ++g) {
                const int q = min(qbase + 32 * c + 4 * g + (lane & 3), M.Sq - 1);
                const unsigned long long idx = ((unsigned long long)bh * M.Sq + q) * (unsigned long long)M.Sk + (key & ~3);
                const uint4 r = philox4x32(M.seed, offset, idx >> 2);
                mine |= ((r.x >= M.thresh ? 1u : 0u) | (r.y >= M.thresh ? 2u : 0u) | (r.z >= M.thresh ? 4u : 0u) |
                         (r.w >= M.thresh ? 8u : 0u)) << (4 * g);
              }
#pragma unroll
              for (int e = 0; e < 4; ++e) kw[c][e] = __shfl_sync(0xffffffffu, mine, (lane & ~3) + e) >> (lane & 3);
            }
          }
          if (tr && it < 16) tr[it * 8] = clock64();
          if (!wait(B_STAT + st, (nst >> st) & 1u)) { ok = false; break; }
          nst ^= 1u << st;
          float nl[64];                                          // read before S is there: the tensor cores keep shared memory busy
#pragma unroll
          for (int i = 0; i < 64; i += 4) *reinterpret_cast<float4*>(nl + i) = *reinterpret_cast<const float4*>(nlse + i);
          if (!wait(B_SFULL, ns & 1u)) { ok = false; break; }
          ns ^= 1u;
          tc_fence_after();
          if (tr && it < 16) tr[it * 8 + 1] = clock64();
          float x[64];
          tmem_ld32f(aS, x);
          tmem_ld32f(aS + 32, x + 32);
          tmem_ld_wait();
          if (keys_plain && !(M.causal && it == 0)) {            // the diagonal crosses a causal key block's first query block
#pragma unroll
            for (int i = 0; i < 64; i += 2) {
              const float2 u = fma2(make_float2(x[i], x[i + 1]), sc, make_float2(nl[i], nl[i + 1]));
              x[i] = u.x; x[i + 1] = u.y;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 64; ++i) {
              const int q = qbase + i;
              float xs = x[i] * M.scale_log2;
              if constexpr (MSK == 2) {
                if (q < M.Sq && key < M.Sk) {
                  const long long mi = (long long)q * M.mask_ld + key;
                  xs += (M.mask_fp32 ? __ldg(reinterpret_cast<const float*>(M.mask) + mi)
                                     : __bfloat162float(__ldg(reinterpret_cast<const __nv_bfloat16*>(M.mask) + mi))) * kLog2e;
                }
              }
              x[i] = key_dead || (M.causal && key > q) ? -INFINITY : xs + nl[i];
            }
          }
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            float* e = x + 32 * c;
#pragma unroll
            for (int i = 0; i < 32; ++i) e[i] = ex2_approx(e[i]);
            if constexpr (DRP) {
              float d[32];
#pragma unroll
              for (int i = 0; i < 32; ++i) d[i] = (kw[c][i & 3] >> (i & ~3)) & 1u ? e[i] * M.drop_scale : 0.f;
              store_bf16x32(aS + (uint32_t)(c * 16), d);
            } else {
              store_bf16x32(aS + (uint32_t)(c * 16), e);
            }
          }
          publish_rows(&bar[B_PFULL], lane);
          if (tr && it < 16) tr[it * 8 + 2] = clock64();
          if (!wait(B_DPFULL, ndp++ & 1u)) { ok = false; break; }
          tc_fence_after();
          if (tr && it < 16) tr[it * 8 + 3] = clock64();
          float dp[64];
          tmem_ld32f(aP, dp);
          tmem_ld32f(aP + 32, dp + 32);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int i = 32 * c; i < 32 * c + 32; i += 4) {
              const float4 D = *reinterpret_cast<const float4*>(ndel + i);
              if constexpr (DRP) {
#pragma unroll
                for (int e = 0; e < 4; ++e) dp[i + e] = (kw[c][e] >> (i - 32 * c)) & 1u ? dp[i + e] * M.drop_scale : 0.f;
              }
              const float2 u = mul2(make_float2(x[i], x[i + 1]), add2(make_float2(dp[i], dp[i + 1]), make_float2(D.x, D.y)));
              const float2 v = mul2(make_float2(x[i + 2], x[i + 3]), add2(make_float2(dp[i + 2], dp[i + 3]), make_float2(D.z, D.w)));
              x[i] = u.x; x[i + 1] = u.y; x[i + 2] = v.x; x[i + 3] = v.y;
            }
            store_bf16x32(aP + (uint32_t)(c * 16), x + 32 * c);
            if constexpr (ONE) {                         // the same row in shared memory: A of dQ, read MN-major
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float* e = x + 32 * c + 8 * k;
                *reinterpret_cast<uint4*>(sm + 5 * TILE + wg * kSub + rt * 128 + (((4 * c + k) ^ (rt & 7)) << 4)) =
                    make_uint4(pack_bf16(e[0], e[1]), pack_bf16(e[2], e[3]), pack_bf16(e[4], e[5]), pack_bf16(e[6], e[7]));
              }
            }
          }
          if constexpr (ONE) fence_proxy_async_smem();
          publish_rows(&bar[B_DSFULL], lane);
          if (tr && it < 16) tr[it * 8 + 4] = clock64();
        }
      } else {
        const int q0 = w.qb * kBlk, nb = M.causal ? min(nkb, w.qb + 1) : nkb;
        const int row = q0 + rt;
        const bool live = row < M.Sq;
        const float nlse = live ? -__ldg(p.lse + (long long)bh * M.Sq + row) : -INFINITY;
        const float ndel = live ? -__ldg(p.delta + (long long)bh * M.Sq + row) : 0.f;
        const float2 nl = make_float2(nlse, nlse), nd = make_float2(ndel, ndel);
        for (int j = 0; j < nb; ++j) {
          const int col0 = j * kBlk + wg * 64;
          const uint32_t dead[2] = {dead_keys<MSK>(M, b, col0, lane), dead_keys<MSK>(M, b, col0 + 32, lane)};
          uint32_t keep[2] = {0xffffffffu, 0xffffffffu};
          if constexpr (DRP) {
            keep[0] = keep_bits<32>(M, offset, bh, min(row, M.Sq - 1), col0);
            keep[1] = keep_bits<32>(M, offset, bh, min(row, M.Sq - 1), col0 + 32);
          }
          if (!wait(B_SFULL + (j & 1), (ns >> (j & 1)) & 1u)) { ok = false; break; }
          ns ^= 1u << (j & 1);
          tc_fence_after();
          const uint32_t aS = (j & 1 ? tmem + 384 : tS) + lane_off + (uint32_t)(wg * 64);
          float x[64];
          tmem_ld32f(aS, x);
          tmem_ld32f(aS + 32, x + 32);
          tmem_ld_wait();
          const bool plain = MSK != 2 && !(dead[0] | dead[1]) && !(M.causal && j == w.qb) && (j * kBlk + kBlk <= M.Sk);
          if (plain) {
#pragma unroll
            for (int i = 0; i < 64; i += 2) {
              const float2 u = fma2(make_float2(x[i], x[i + 1]), sc, nl);
              x[i] = u.x; x[i + 1] = u.y;
            }
          } else {
            score_chunk<32, MSK>(x, row, col0, dead[0], M, false);
            score_chunk<32, MSK>(x + 32, row, col0 + 32, dead[1], M, false);
#pragma unroll
            for (int i = 0; i < 64; ++i) x[i] += nlse;
          }
#pragma unroll
          for (int i = 0; i < 64; ++i) x[i] = ex2_approx(x[i]);
          if (!wait(B_DPFULL, ndp++ & 1u)) { ok = false; break; }
          tc_fence_after();
          float dp[64];
          tmem_ld32f(aP, dp);
          tmem_ld32f(aP + 32, dp + 32);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int i = 32 * c; i < 32 * c + 32; i += 2) {
              if constexpr (DRP) {
                dp[i] = (keep[c] >> (i & 31)) & 1u ? dp[i] * M.drop_scale : 0.f;
                dp[i + 1] = (keep[c] >> ((i + 1) & 31)) & 1u ? dp[i + 1] * M.drop_scale : 0.f;
              }
              const float2 u = mul2(make_float2(x[i], x[i + 1]), add2(make_float2(dp[i], dp[i + 1]), nd));
              x[i] = u.x; x[i + 1] = u.y;
            }
            store_bf16x32(aP + (uint32_t)(c * 16), x + 32 * c);
          }
          publish_rows(&bar[B_DSFULL], lane);
        }
      }
      if (ok) ok = wait(B_ACC, n & 1u);
      if (!ok) break;
      tc_fence_after();
      const int r0 = (w.kb >= 0 ? w.kb : w.qb) * kBlk + (warp & 3) * 32;      // the warp's first row
      const int nacc = ONE ? 3 : w.kb >= 0 ? 2 : 1;
      for (int a = 0; a < nacc; ++a) {
        const bool is_q = w.kb < 0 || (ONE && a == 2);
        const DRef& out = is_q ? p.dq : a ? p.dk : p.dv;
        const int left = (is_q ? M.Sq : M.Sk) - r0;
        __nv_bfloat16* dst = row_ptr(out, b, r0, h) + wg * (HD / 2);
        const float mul = !is_q && a == 0 ? 1.f : M.sm_scale;
        const uint32_t acc = ONE && a == 2 ? tS : tAcc + (uint32_t)(a * HD);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) {
          float o[32];
          tmem_ld32f(acc + lane_off + (uint32_t)(wg * (HD / 2) + c * 32), o);
          tmem_ld_wait();
          if (a + 1 == nacc && c + 1 == HD / 64) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar[B_ACCREAD]);
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] *= mul;
          store_rows32(dst + c * 32, out.ss, left, o, lane);
        }
      }
    }
  }
  teardown_cta(tmem, warp);
}

// =====================================================================================================  parts
// Twelve variants for each direction and head_dim take 17 s of compilation; the build makes an object of each of the four side by side
// (RTP_FLASH_PART 0 to 3; undefined: all in one).  Part 0 has the entry points.
#ifdef RTP_FLASH_PART
#define RTP_FLASH_HAS(k) (RTP_FLASH_PART == k)
#else
#define RTP_FLASH_HAS(k) 1
#endif

constexpr int smem_fwd(int hd) { return 1024 + (hd / 64) * kSub * 6 + 256 + 2 * 256 * 4; }
// backward: seven tiles, control block, statistics of two blocks of queries
constexpr int smem_bwd(int hd) { return kBwdSlack + (hd / 64) * kSub * 7 + 256 + 2 * 2 * kBlk * 4; }
static_assert(sizeof(Ctl) <= 256, "control block");
static_assert(smem_fwd(128) <= 232448 && smem_bwd(128) <= 232448, "shared memory budget");

template <auto Kern>
cudaError_t launch_flash(const FlashParams& P, int grid, int smem, cudaStream_t stream) {
  const cudaError_t e = ensure_smem<Kern>(smem);
  return e != cudaSuccess ? e : launch_k(Kern, dim3(grid), dim3(kThreads), smem, stream, P);
}
// kind: 0 one piece of work a CTA, 1 persistent, 2 (backward) one head a CTA; mask: none, key padding, additive
#define RTP_FLASH_FWD(HD, MSK, DRP)                                                                                     \
  (kind == 1 ? launch_flash<flash_fwd_kernel<HD, MSK, DRP, true>>(P, grid, smem_fwd(HD), (cudaStream_t)stream)          \
             : launch_flash<flash_fwd_kernel<HD, MSK, DRP, false>>(P, grid, smem_fwd(HD), (cudaStream_t)stream))
#define RTP_FLASH_BWD(HD, MSK, DRP)                                                                                     \
  (kind == 2   ? launch_flash<flash_bwd_kernel<HD, MSK, DRP, false, true>>(P, grid, smem_bwd(HD), (cudaStream_t)stream) \
   : kind == 1 ? launch_flash<flash_bwd_kernel<HD, MSK, DRP, true>>(P, grid, smem_bwd(HD), (cudaStream_t)stream)        \
               : launch_flash<flash_bwd_kernel<HD, MSK, DRP, false>>(P, grid, smem_bwd(HD), (cudaStream_t)stream))
#define RTP_FLASH_PART_FN(NAME, LAUNCH, HD)                                                              \
  extern "C" int NAME(const void* params, int mask, int drp, int kind, int grid, void* stream) {         \
    const FlashParams& P = *reinterpret_cast<const FlashParams*>(params);                                \
    return (int)(mask == 2   ? (drp ? LAUNCH(HD, 2, true) : LAUNCH(HD, 2, false))                        \
                 : mask == 1 ? (drp ? LAUNCH(HD, 1, true) : LAUNCH(HD, 1, false))                        \
                             : (drp ? LAUNCH(HD, 0, true) : LAUNCH(HD, 0, false)));                      \
  }

}  // namespace

// Launches a variant with the FlashParams at `params`; returns a cudaError_t.
typedef int FlashPart(const void* params, int mask, int drp, int kind, int grid, void* stream);
extern "C" {
FlashPart rtp_flash_part_fwd64;
FlashPart rtp_flash_part_fwd128;
FlashPart rtp_flash_part_bwd64;
FlashPart rtp_flash_part_bwd128;
}
#if RTP_FLASH_HAS(0)
RTP_FLASH_PART_FN(rtp_flash_part_fwd64, RTP_FLASH_FWD, 64)
#endif
#if RTP_FLASH_HAS(1)
RTP_FLASH_PART_FN(rtp_flash_part_fwd128, RTP_FLASH_FWD, 128)
#endif
#if RTP_FLASH_HAS(2)
RTP_FLASH_PART_FN(rtp_flash_part_bwd64, RTP_FLASH_BWD, 64)
#endif
#if RTP_FLASH_HAS(3)
RTP_FLASH_PART_FN(rtp_flash_part_bwd128, RTP_FLASH_BWD, 128)
#endif

#if RTP_FLASH_HAS(0)
namespace {
// =====================================================================================================  host
thread_local std::string g_ferr;
long long* g_flash_trace = nullptr;
int ffail(const std::string& s) { g_ferr = s; return -1; }

int device_sms() {
  static int n[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!n[dev]) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
  return n[dev];
}

// How many heads run side by side: as many as leave what their CTAs read again and again well inside L2.  Over all heads at once,
// longest blocks first, long sequences came from HBM each time (16 heads of 8192 x 128: backward 870 us, 790 in groups of 4).
int head_group(long long bytes_per_head, int BH) {
  const long long g = (32ll << 20) / std::max(bytes_per_head, 1ll);
  return (int)std::min<long long>(std::max(g, 1ll), BH);
}

uint32_t thresh_of(float pdrop) {
  if (pdrop <= 0.f) return 0u;
  double t = (double)pdrop * 4294967296.0;
  if (t > 4294967295.0) t = 4294967295.0;
  return (uint32_t)t;
}

// 3-D map {width columns, dim1, dim2} over a [batch, seq, width] view; the dimension with the smaller stride comes first.
int make_map3(CUtensorMap* m, int* seq1, const RtpFlashRef& r, int B, int S, const char* what) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return ffail("cuTensorMapEncodeTiled entry point not found");
  if ((reinterpret_cast<uintptr_t>(r.ptr) & 15) != 0) return ffail(std::string(what) + ": base is not 16-byte aligned");
  if ((r.sb * 2) % 16 || (r.ss * 2) % 16) return ffail(std::string(what) + ": strides must be multiples of 16 bytes");
  if (r.width <= 0) return ffail(std::string(what) + ": width missing");
  const bool s_first = r.ss <= r.sb || B == 1;
  *seq1 = s_first ? 1 : 0;
  cuuint64_t dims[3] = {(cuuint64_t)r.width, (cuuint64_t)(s_first ? S : B), (cuuint64_t)(s_first ? B : S)};
  cuuint64_t strides[2] = {(cuuint64_t)(s_first ? r.ss : r.sb) * 2, (cuuint64_t)(s_first ? r.sb : r.ss) * 2};
  if (B == 1) strides[1] = strides[0] * (cuuint64_t)S;   // a single batch: any legal pitch
  cuuint32_t box[3] = {64u, s_first ? (cuuint32_t)kBlk : 1u, s_first ? 1u : (cuuint32_t)kBlk};
  cuuint32_t estr[3] = {1u, 1u, 1u};
  CUresult rc = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, r.ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) return ffail(std::string(what) + ": cuTensorMapEncodeTiled failed with code " + std::to_string((int)rc));
  return 0;
}
DRef dref(const RtpFlashRef& r) {
  DRef d;
  d.ptr = r.ptr; d.sb = r.sb; d.ss = r.ss;
  d.col_base = r.col_base; d.hpg = r.hpg > 0 ? r.hpg : 1; d.gstride = r.gstride; d.hstride = r.hstride;
  return d;
}
int check_ref(const RtpFlashRef& r, const char* what, int hd) {
  if (!r.ptr) return ffail(std::string(what) + ": null pointer");
  if ((reinterpret_cast<uintptr_t>(r.ptr) & 15) || (r.sb % 8) || (r.ss % 8) || (r.col_base % 8) || (r.gstride % 8) ||
      (r.hstride % 8))
    return ffail(std::string(what) + ": rows of a head must be 16-byte aligned");
  (void)hd;
  return 0;
}
int fill_common(const RtpFlashArgs* a, FlashParams& P) {
  if (a->head_dim != 64 && a->head_dim != 128) return ffail("flash attention: head_dim must be 64 or 128");
  if (a->B <= 0 || a->H <= 0 || a->Sq <= 0 || a->Sk <= 0) return ffail("flash attention: empty problem");
  if (a->causal && a->Sq != a->Sk) return ffail("flash attention: a causal mask needs Sq == Sk");
  if (a->drop_p > 0.f && a->Sk % 4) return ffail("flash attention: dropout needs Sk to be a multiple of 4");
  if (!a->status) return ffail("flash attention: status word required");
  P.B = a->B; P.H = a->H;
  P.m.mask = a->mask; P.m.mask_ld = a->mask_ld; P.m.mask_fp32 = a->mask_fp32;
  P.m.kpm = a->kpm; P.m.kpm_ld = a->kpm_ld;
  P.m.causal = a->causal; P.m.Sq = a->Sq; P.m.Sk = a->Sk;
  P.m.sm_scale = a->sm_scale; P.m.scale_log2 = a->sm_scale * kLog2e;
  P.m.thresh = thresh_of(a->drop_p);
  P.m.drop_scale = a->drop_p > 0.f ? 1.f / (1.f - a->drop_p) : 1.f;
  P.m.seed = a->seed; P.m.offset = a->offset; P.m.step_ptr = a->step_ptr;
  P.status = a->status;
  P.timeout_ns = 2000000000ull;
  P.trace = g_flash_trace;
  P.lse = a->lse;
  P.delta = a->delta;
  if (check_ref(a->q, "q", a->head_dim) || check_ref(a->k, "k", a->head_dim) || check_ref(a->v, "v", a->head_dim) ||
      check_ref(a->o, "o", a->head_dim))
    return -1;
  if (make_map3(&P.mq, &P.q_seq1, a->q, a->B, a->Sq, "q")) return -1;
  if (make_map3(&P.mk, &P.k_seq1, a->k, a->B, a->Sk, "k")) return -1;
  if (make_map3(&P.mv, &P.v_seq1, a->v, a->B, a->Sk, "v")) return -1;
  P.q = dref(a->q); P.k = dref(a->k); P.v = dref(a->v); P.o = dref(a->o);
  return 0;
}
int mask_kind(const RtpFlashArgs* a) { return a->mask ? 2 : a->kpm ? 1 : 0; }
int launched(int e, const char* what) { return e == (int)cudaSuccess ? 0 : ffail(std::string(what) + ": " + cudaGetErrorString((cudaError_t)e)); }

}  // namespace

extern "C" {

const char* rtp_flash_last_error(void) { return g_ferr.c_str(); }
void rtp_flash_debug_set_trace(long long* device_buffer_512_words) { g_flash_trace = device_buffer_512_words; }

int rtp_flash_fwd(const RtpFlashArgs* a, void* stream) {
  static thread_local FlashParams P;
  if (fill_common(a, P)) return -1;
  if (!a->lse) return ffail("flash attention: lse buffer required");
  // One row tile a CTA, its keys shared out, as long as that is one wave; two row tiles a CTA beyond it, where they share the copies
  // of K and V.  Two tiles -> shared out, us: 2 heads of 4096 x 4096 x 128 49 -> 37, 32 of 1024 keys x 128 17.7 -> 13.9, 32 of
  // 256 x 256 x 64 9.2 -> 7.2, 4 of 384 x 384 x 64 9.5 -> 7.6; one key block the same either way.
  const int tiles = (a->Sq + kBlk - 1) / kBlk, BH = a->B * a->H;
  P.split = (long long)tiles * BH <= device_sms();
  P.group = head_group(4ll * a->Sk * a->head_dim, BH);
  const int grid = (P.split ? tiles : (tiles + 1) / 2) * BH;
  const bool more = grid > device_sms();         // 48 heads of 999 x 128: 31 -> 28 us
  return launched((a->head_dim == 64 ? rtp_flash_part_fwd64 : rtp_flash_part_fwd128)(&P, mask_kind(a), P.m.thresh != 0, more, grid, stream),
                  "flash_fwd");
}

int rtp_flash_bwd(const RtpFlashArgs* a, void* stream) {
  static thread_local FlashParams P;
  if (fill_common(a, P)) return -1;
  if (!a->lse || !a->delta) return ffail("flash attention backward: lse and delta buffers required");
  if (check_ref(a->dout, "dout", a->head_dim) || check_ref(a->dq, "dq", a->head_dim) || check_ref(a->dk, "dk", a->head_dim) ||
      check_ref(a->dv, "dv", a->head_dim))
    return -1;
  if (make_map3(&P.mdo, &P.do_seq1, a->dout, a->B, a->Sq, "dout")) return -1;
  P.dout = dref(a->dout); P.dq = dref(a->dq); P.dk = dref(a->dk); P.dv = dref(a->dv);
  const int BH = a->B * a->H;
  // Heads of one block of keys and of queries are a CTA each where two would be two rounds.  us, two -> one: 128 heads of 64 x 64 x 64
  // 16.2 -> 12.8, of 128 x 128 x 128 20.8 -> 15.8; 64 heads, one round either way, 11.2 -> 11.5 and (64 x 64 x 128) 13.7 -> 16.2.
  const bool one = a->Sq <= kBlk && a->Sk <= kBlk && BH <= device_sms() && 2 * BH > device_sms();
  const int grid = one ? BH : ((a->Sq + kBlk - 1) / kBlk + (a->Sk + kBlk - 1) / kBlk) * BH;
  const int kind = one ? 2 : grid > 2 * device_sms();   // one or two rounds are over sooner without (16 heads of 1024 x 1024: 55 us, 60)
  cudaStream_t s = (cudaStream_t)stream;
  P.group = one ? BH : head_group(4ll * (a->Sq + a->Sk) * a->head_dim, BH);
  const long long rows = (long long)a->B * a->Sq * a->H, per = 256 / (a->head_dim / 8);
  const cudaError_t e = launch_k(a->head_dim == 64 ? flash_delta_kernel<64> : flash_delta_kernel<128>,
                                 dim3((unsigned)((rows + per - 1) / per)), dim3(256), 0, s, P.o, P.dout, P.delta, a->Sq, a->H, rows);
  if (e != cudaSuccess) return ffail(std::string("flash_delta: ") + cudaGetErrorString(e));
  return launched((a->head_dim == 64 ? rtp_flash_part_bwd64 : rtp_flash_part_bwd128)(&P, mask_kind(a), P.m.thresh != 0, kind, grid, stream),
                  "flash_bwd");
}

}  // extern "C"
#endif  // part 0

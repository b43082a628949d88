// Warp-specialised tcgen05 GEMM for a ring of one rank.
//
// The rotation kernel (gemm_kernel.cuh) carries a 17 KB program as its launch parameter, polls counters, pushes shards
// and signals peers; on one rank none of that is needed, and for the short GEMMs of a training step the fixed cost was
// most of the time (256 x 1024 x 256: 17 us in a graph, of which the tensor work is 1 us).  This kernel takes up to 16
// plain jobs in a few hundred bytes each:
//
//   warp 0       TMA producer          warps 2-9    epilogue: two warps per TMEM lane quadrant, 64 columns at a time
//   warp 1       UMMA issuer
//
// The column sums of A (the bias gradient of a weight-gradient job) are a job of their own, A times a 16-wide tile of
// ones that stays in shared memory: it loads A alone and adds about 2 % of tensor work.  Tried and dropped: warps that
// add up the staged A tiles of the first tile column (unpack + FADD 450 ns per k-block, mma.sync 650 ns, against 350 ns
// of the tile itself; weight gradient 8192 x 2048 -> 2048 went from 49 to 90 us), and a [1, M] x [M, out] product (a
// 256-row tile per 256 outputs, 12 % of the weight gradient).
//
// Tiles are 256 x {256, 128} on CTA pairs (cta_group::2) or 128 x {128, 64} on single CTAs.  A k-block of a pair tile
// moves 32 or 24 KB into each SM; a single 128 x 128 tile moves 32 KB for half (a quarter) of the work and is bound by
// what an SM takes in (120 GB/s measured, 64 bytes per clock).  Pairs win wherever their tiles fill the grid, single
// CTAs where a launch has few tiles; run() below chooses per launch by a cost model.
#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstring>
#include <string>
#include "common.cuh"
#include "gemm_local.h"
#include "launch.h"
#include "tmap.h"

namespace rtp {
namespace {

constexpr int kTM = 128;                         // rows of a tile that one CTA stages and drains
constexpr int kKB = 64;                          // contraction elements per stage
constexpr int kStages = 8;
constexpr int kABytesL = kTM * kKB * 2;
constexpr int kArea = 196608;                    // stage ring: 6 x 32 KB, 8 x 24 KB
constexpr int kPitch = 128;                      // staged row: 64 bf16, 16-byte chunks swizzled by row % 8
constexpr int kEpiWarps = 8;
constexpr int kStageOut = kEpiWarps * 32 * kPitch;
constexpr int kThreads = 32 * (2 + kEpiWarps);
constexpr int kOnes = 1024;                      // eight 128-byte rows of ones: a CTA's share of a pair's 16-wide tile
constexpr int kSmem = 1024 + kArea + kStageOut + kOnes + 256;
static_assert(kSmem <= 232448, "over the shared memory of a CTA");

struct alignas(64) Job {
  CUtensorMap ma, mb;
  int M, N, bn, kblocks;
  int tile0, tiles_m, tiles_n;                   // first tile of the job in the launch's tile order
  int group;                                     // tile rows of a group (see tile_pos)
  unsigned char a_mn, b_mn, a3, b3;              // a3 / b3: the MN-major map is 3-D {64 mn, k, mn / 64}
  void* d; long long ldd;
  const void* c; long long ldc;
  const void* bias;
  const void* mask; long long ldmask;
  float mask_scale, drop_scale;
  uint32_t drop_thresh;
  int act;
  int kper, slice_tiles;                         // > 0: k-blocks and tiles of a slice (fp32 results, bare sums)
  long long part_stride;                         // between the results of two slices
  int sum;                                       // 1: d[m] = sum_k A[m, k] (+ c[m]); B is the tile of ones, bn = 16
  unsigned long long seed, offset;
  const unsigned long long* step_ptr;
  const int *m_fill, *k_fill;                    // see LocalGemm
};

template <int MAXJ>
struct alignas(64) Params {
  int njobs, total, units, stages, stage_bytes;
  int ones_off;                                  // where the tile of ones starts behind the stage ring; 0: no sums
  unsigned long long* status;
  unsigned long long timeout_ns;
  Job job[MAXJ];
};

struct Ctrl {
  uint64_t full[kStages], empty[kStages], peer_full[kStages];
  uint64_t tmem_full[2], tmem_empty[2], drain;
  uint32_t tmem_base, abort_flag;
};
static_assert(sizeof(Ctrl) <= 256, "control block");

// The t-th tile of a unit.  Tiles are ordered by falling cost and dealt out to and fro (0..U-1, U-1..0, ...), so that a
// unit with an expensive tile in one round gets a cheap one in the next.
__device__ __forceinline__ int unit_tile(int round, int unit, int units) {
  return round * units + ((round & 1) ? units - 1 - unit : unit);
}
// Tile position inside a job: groups of tile rows, column by column, so that the tiles in flight share operands.
__device__ __forceinline__ void tile_pos(const Job& j, int lt, int& tm, int& tn) {
  const int per = j.group * j.tiles_n;
  const int g = lt / per, r = lt - g * per;
  const int rows = min(j.group, j.tiles_m - g * j.group);
  tn = r / rows;
  tm = g * j.group + (r - tn * rows);
}
template <int MAXJ>
__device__ __forceinline__ int find_job(const Params<MAXJ>& P, int t) {
  int j = 0;
  while (j + 1 < P.njobs && t >= P.job[j + 1].tile0) ++j;
  return j;
}

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<unsigned long long>(m)) : "memory");
}
__device__ __forceinline__ void add8(float* v, const uint4& u) {
  v[0] += bf16_lo(u.x); v[1] += bf16_hi(u.x); v[2] += bf16_lo(u.y); v[3] += bf16_hi(u.y);
  v[4] += bf16_lo(u.z); v[5] += bf16_hi(u.z); v[6] += bf16_lo(u.w); v[7] += bf16_hi(u.w);
}

// The slice that the lt-th tile of a job belongs to (0: the contraction is whole); lt becomes its number in the slice.
__device__ __forceinline__ int tile_slice(const Job& j, int& lt) {
  if (!j.kper) return 0;
  const int s = lt / j.slice_tiles;
  lt -= s * j.slice_tiles;
  return s;
}
// k-blocks of a tile of slice s whose first row is row0; 0: nothing to do but to write zeros
template <bool FILL>
__device__ __forceinline__ int tile_kblocks(const Job& J, int s, int row0) {
  int n = J.kper ? min(J.kper, J.kblocks - s * J.kper) : J.kblocks;
  if constexpr (FILL) {
    if (J.m_fill && row0 >= __ldg(J.m_fill)) n = 0;
    if (J.k_fill) n = min(n, (__ldg(J.k_fill) + 63) >> 6);
  }
  return n;
}

// FILL: a job has rows that are not in use (the padded capacity of experts: 8 experts of 2560 rows of which 2048 are filled,
// 2048 <-> 8192, whole layer forward and backward 3919 -> 3628 us).
// SRC: a job adds to its output or masks it; FUN: a job has an activation or dropout.  Merely branched over, that code cost every
// launch: twice the spills, and a fifth of the epilogue's time went into instruction fetch.  With it compiled out and both
// halves of a row's 64 columns fetched at once (us, before -> now): 256 x 64 -> 256 4.5 -> 3.4, 1024 x 512 -> 512 6.6 -> 5.5,
// 1024 x 2048 -> 2048 13.4 -> 12.4, 8192 x 8 -> 8192 73 -> 45, 36864 x 64 -> 288 20 -> 13.6; added to its output 25 -> 21.
template <bool PAIR, int MAXJ, bool SRC, bool FUN, bool FILL>
__global__ void __launch_bounds__(kThreads, 1) local_gemm_kernel(const __grid_constant__ Params<MAXJ> P) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = tiles + kArea;
  Ctrl* ctl = reinterpret_cast<Ctrl*>(staging + kStageOut + kOnes);
  volatile uint32_t* abort_flag = &ctl->abort_flag;
  const uint32_t crank = PAIR ? cluster_ctarank() : 0u;
  constexpr int TM = PAIR ? 256 : 128;
  const int unit = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_stages = P.stages, stage_bytes = P.stage_bytes, units = P.units, total = P.total;
  unsigned long long* status = P.status;
  const unsigned long long tmo = P.timeout_ns;

  if (warp == 2) {
    for (int j = lane; j < 2 * P.njobs; j += 32)
      if (!(j & 1) || !P.job[j >> 1].sum) prefetch_tmap(j & 1 ? &P.job[j >> 1].mb : &P.job[j >> 1].ma);
  }
  if (warp == 0) {
    if (lane < kStages) {
      mbar_init(&ctl->full[lane], 1);
      mbar_init(&ctl->empty[lane], 1);
      mbar_init(&ctl->peer_full[lane], 1);
    } else if (lane < kStages + 2) {
      mbar_init(&ctl->tmem_full[lane - kStages], 1);
      mbar_init(&ctl->tmem_empty[lane - kStages], PAIR ? 2 * kEpiWarps : kEpiWarps);
    } else if (lane == kStages + 2) {
      mbar_init(&ctl->drain, 1);
      ctl->abort_flag = 0;
    }
    mbar_fence_init();
  }
  if (P.ones_off) {
    // 16 rows on a single CTA, 8 on each CTA of a pair (all elements are equal: the swizzle does not matter)
    uint4* ones = reinterpret_cast<uint4*>(tiles + P.ones_off);
    const int n = (PAIR ? 8 : 16) * 128 / 16;
    if (threadIdx.x < n) ones[threadIdx.x] = make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    if (PAIR) { tmem_alloc_pair(&ctl->tmem_base, 512); tmem_relinquish_pair(); }
    else { tmem_alloc(&ctl->tmem_base, 512); tmem_relinquish(); }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  pdl_launch_dependents();           // every CTA owns its TMEM columns first (see launch.h)
  pdl_wait();

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0, issued = 0, parity = 0;
      bool ok = true;
      const uint32_t tiles_s = smem_u32(tiles), full_s = smem_u32(&ctl->full[0]), empty_s = smem_u32(&ctl->empty[0]);
      for (int r = 0; ok; ++r) {
        const int t = unit_tile(r, unit, units);
        if (r * units >= total) break;
        if (t >= total) continue;
        const Job& J = P.job[find_job(P, t)];
        int tm, tn, lt = t - J.tile0;
        const int slice = tile_slice(J, lt), kb0 = slice * J.kper;
        tile_pos(J, lt, tm, tn);
        const int bn_cta = PAIR ? J.bn >> 1 : J.bn;
        const int m0 = tm * TM + (int)crank * kTM, n0 = tn * J.bn + (int)crank * bn_cta;
        const unsigned long long ma = reinterpret_cast<unsigned long long>(&J.ma);
        const unsigned long long mb = reinterpret_cast<unsigned long long>(&J.mb);
        const bool a_mn = J.a_mn, b_mn = J.b_mn, a3 = J.a3, b3 = J.b3;
        const int nb = b_mn ? bn_cta >> 6 : 1;
        const bool sum = J.sum;                     // B is already in shared memory
        const uint32_t tx = sum ? kABytesL : kABytesL + bn_cta * kKB * 2;
        const int kblocks = tile_kblocks<FILL>(J, slice, tm * TM);
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait_s(empty_s + stage * 8, phase ^ 1, abort_flag, status, tmo)) { ok = false; break; }
          const uint32_t sa = tiles_s + stage * stage_bytes, sb = sa + kABytesL, bar = full_s + stage * 8;
          issued |= 1u << stage;
          parity = (parity & ~(1u << stage)) | (phase << stage);
          const int k0 = (kb0 + kb) * kKB;
          mbar_arrive_expect_tx_s(bar, tx);
          if (a3) tma_load_3d_s(sa, ma, 0, k0, m0 >> 6, bar);
          else if (a_mn) {
            tma_load_2d_s(sa, ma, m0, k0, bar);
            tma_load_2d_s(sa + 8192, ma, m0 + 64, k0, bar);
          } else tma_load_2d_s(sa, ma, k0, m0, bar);
          if (sum) {
          } else if (b3) tma_load_3d_s(sb, mb, 0, k0, n0 >> 6, bar);
          else if (b_mn) {
            for (int i = 0; i < nb; ++i) tma_load_2d_s(sb + i * 8192, mb, n0 + i * 64, k0, bar);
          } else tma_load_2d_s(sb, mb, k0, n0, bar);
          if (++stage == n_stages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        for (int s = 0; s < n_stages; ++s) {     // copies in flight land (bounded) before the CTA may exit
          if (!((issued >> s) & 1u)) continue;
          const unsigned long long t0 = globaltimer_ns();
          while (!mbar_try_wait(&ctl->full[s], (parity >> s) & 1u))
            if (globaltimer_ns() - t0 > 2000000ull) break;
        }
      }
    }
  } else if (warp == 1) {
    if (crank == 0 && elect_one()) {
      // -------------------------------------------------------------- UMMA issuer (the leader of a pair drives both SMs)
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true, any = false;
      const uint32_t tiles_s = smem_u32(tiles), full_s = smem_u32(&ctl->full[0]), peer_s = smem_u32(&ctl->peer_full[0]);
      for (int r = 0; ok; ++r) {
        const int t = unit_tile(r, unit, units);
        if (r * units >= total) break;
        if (t >= total) continue;
        const Job& J = P.job[find_job(P, t)];
        int row0 = 0, lt = t - J.tile0;
        const int slice = tile_slice(J, lt);
        if constexpr (FILL) {
          int tm, tn;
          tile_pos(J, lt, tm, tn);
          row0 = tm * TM;
        }
        const int kblocks = tile_kblocks<FILL>(J, slice, row0);
        if (FILL && !kblocks) continue;
        const uint32_t idesc = make_idesc_bf16(TM, J.bn, J.a_mn, J.b_mn);
        const uint32_t a_step = J.a_mn ? 128u : 2u, b_step = J.b_mn ? 128u : 2u;    // 16 elements of k, in 16-byte units
        const uint64_t da0 = make_smem_desc(0, J.a_mn ? 8192u : 16u, 1024), db0 = make_smem_desc(0, J.b_mn ? 8192u : 16u, 1024);
        const uint32_t ones = J.sum ? (tiles_s + P.ones_off) >> 4 : 0u;
        if (!mbar_wait(&ctl->tmem_empty[acc], acc_phase ^ 1, abort_flag, status, tmo)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * 256);
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait_s(full_s + stage * 8, phase, abort_flag, status, tmo)) { ok = false; break; }
          if (PAIR && !mbar_try_wait_cluster_s(peer_s + stage * 8, phase)) {
            if (!mbar_wait_slow_s(peer_s + stage * 8, phase, abort_flag, status, tmo)) { ok = false; break; }
            mbar_try_wait_cluster_s(peer_s + stage * 8, phase);
          }
          tc_fence_after();
          const uint32_t sa = (tiles_s + stage * stage_bytes) >> 4, sb = ones ? ones : sa + (kABytesL >> 4);
#pragma unroll
          for (int kk = 0; kk < kKB / 16; ++kk) {
            const uint64_t da = da0 + (uint64_t)(sa + kk * a_step), db = db0 + (uint64_t)(sb + kk * b_step);
            if (PAIR) umma_bf16_pair(d_tmem, da, db, idesc, (kb | kk) ? 1u : 0u);
            else umma_bf16(d_tmem, da, db, idesc, (kb | kk) ? 1u : 0u);
          }
          any = true;
          if (PAIR) umma_commit_pair(&ctl->empty[stage]); else umma_commit(&ctl->empty[stage]);
          if (++stage == n_stages) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (PAIR) umma_commit_pair(&ctl->tmem_full[acc]); else umma_commit(&ctl->tmem_full[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      if (!ok && any) {
        if (PAIR) umma_commit_pair(&ctl->drain); else umma_commit(&ctl->drain);
        const unsigned long long t0 = globaltimer_ns();
        while (!mbar_try_wait(&ctl->drain, 0))
          if (globaltimer_ns() - t0 > 2000000ull) break;
      }
    } else if (PAIR && crank != 0 && elect_one()) {
      // -------------------------------------------------------------- second CTA: "my half of this stage has landed"
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      const uint32_t full_s = smem_u32(&ctl->full[0]), lead = mapa_u32(smem_u32(&ctl->peer_full[0]), 0);
      for (int r = 0; ok; ++r) {
        const int t = unit_tile(r, unit, units);
        if (r * units >= total) break;
        if (t >= total) continue;
        const Job& J = P.job[find_job(P, t)];
        int row0 = 0, lt = t - J.tile0;
        const int slice = tile_slice(J, lt);
        if constexpr (FILL) {
          int tm, tn;
          tile_pos(J, lt, tm, tn);
          row0 = tm * TM;
        }
        const int kblocks = tile_kblocks<FILL>(J, slice, row0);
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait_s(full_s + stage * 8, phase, abort_flag, status, tmo)) { ok = false; break; }
          mbar_arrive_cluster(lead + stage * 8);
          if (++stage == n_stages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp < 2 + kEpiWarps) {
    // ---------------------------------------------------------------- epilogue
    const int quad = warp & 3, half = (warp - 2) >> 2;
    uint8_t* stg = staging + (warp - 2) * (32 * kPitch);
    uint8_t* own = stg + lane * kPitch;                              // this thread's row; chunk q sits at q ^ (lane % 8)
    const int osw = lane & 7;
    // coalesced view: rows 4 k + lane / 8, chunk lane % 8 (rows of even and odd k differ by 4 in row % 8)
    uint8_t* coal0 = stg + (lane >> 3) * kPitch + (((lane & 7) ^ (lane >> 3)) << 4);
    uint8_t* coal1 = stg + (lane >> 3) * kPitch + (((lane & 7) ^ (lane >> 3) ^ 4) << 4);
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int r = 0; ok; ++r) {
      const int t = unit_tile(r, unit, units);
      if (r * units >= total) break;
      if (t >= total) continue;
      const Job& J = P.job[find_job(P, t)];
      int tm, tn, lt = t - J.tile0;
      const int slice = tile_slice(J, lt);
      tile_pos(J, lt, tm, tn);
      const int M = J.M, N = J.N, bn = J.bn, part = J.kper;
      float* const fd = reinterpret_cast<float*>(J.d) + slice * J.part_stride;      // slices: fp32 results
      [[maybe_unused]] const int act = J.act;
      const int row0 = tm * TM + (int)crank * kTM + quad * 32, n0 = tn * bn;
      const __nv_bfloat16* c = reinterpret_cast<const __nv_bfloat16*>(J.c);
      const __nv_bfloat16* mask = reinterpret_cast<const __nv_bfloat16*>(J.mask);
      const __nv_bfloat16* bias = reinterpret_cast<const __nv_bfloat16*>(J.bias);
      __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(J.d);
      const long long ldd = J.ldd;
      [[maybe_unused]] const long long ldc = J.ldc, ldmask = J.ldmask;
      [[maybe_unused]] const uint32_t thresh = J.drop_thresh;
      [[maybe_unused]] unsigned long long drop_off = 0;
      if constexpr (FUN) drop_off = J.offset + (J.step_ptr ? __ldg(J.step_ptr) * 65536ull : 0ull);
      if constexpr (FILL) {
        if (!tile_kblocks<FILL>(J, slice, tm * TM)) {               // no accumulator: zeros
          if (J.sum) {
            if (half == 0 && row0 + lane < M) d[row0 + lane] = __float2bfloat16(0.f);
          } else {
            for (int ch = half; ch * 64 < bn; ch += 2)
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                const int row = row0 + 4 * k + (lane >> 3), col = n0 + ch * 64 + (lane & 7) * 8;
                if (row < M && col < N) *reinterpret_cast<uint4*>(d + (long long)row * ldd + col) = make_uint4(0u, 0u, 0u, 0u);
              }
          }
          continue;
        }
      }
      bool waited = false;
      if (J.sum && half == 0) {
        uint32_t good = 1;
        if (lane == 0) good = mbar_wait(&ctl->tmem_full[acc], acc_phase, abort_flag, status, tmo) ? 1u : 0u;
        good = __shfl_sync(0xffffffffu, good, 0);
        if (!good) { ok = false; break; }
        tc_fence_after();
        waited = true;
        uint32_t ra[32];
        tmem_ld_32x32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * 256), ra);    // column 0 of 16 equal ones
        tmem_ld_wait();
        const int m = row0 + lane;
        if (m < M) {
          if (part) fd[m] = __uint_as_float(ra[0]);
          else d[m] = __float2bfloat16(__uint_as_float(ra[0]) + (c ? __bfloat162float(c[m]) : 0.f));
        }
      }
      for (int ch = half; !J.sum && ch * 64 < bn; ch += 2) {
        const int col0 = n0 + ch * 64;
        const int ccol = col0 + (lane & 7) * 8;                      // column of this lane in the coalesced view
        // the accumulate source is fetched while the accumulator is still being made
        [[maybe_unused]] uint4 cv[8];
        [[maybe_unused]] const __nv_bfloat16* pre = c ? c : mask;
        if constexpr (SRC) {
          const long long ldpre = c ? ldc : ldmask;
          if (pre) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const int row = row0 + 4 * k + (lane >> 3);
              cv[k] = make_uint4(0u, 0u, 0u, 0u);
              if (row < M && ccol < N) cv[k] = __ldcg(reinterpret_cast<const uint4*>(pre + (long long)row * ldpre + ccol));
            }
          }
        }
        // so is the bias, where no other source takes the registers (a job with both is rare)
        [[maybe_unused]] uint4 bv[8];
        auto bias8 = [&](int q) {
          return bias && col0 + q * 8 < N ? __ldg(reinterpret_cast<const uint4*>(bias + col0 + q * 8)) : make_uint4(0u, 0u, 0u, 0u);
        };
        if constexpr (!SRC) {
#pragma unroll
          for (int q = 0; q < 8; ++q) bv[q] = bias8(q);
        }
        if (!waited) {
          uint32_t good = 1;
          if (lane == 0) good = mbar_wait(&ctl->tmem_full[acc], acc_phase, abort_flag, status, tmo) ? 1u : 0u;
          good = __shfl_sync(0xffffffffu, good, 0);
          if (!good) { ok = false; break; }
          tc_fence_after();
          waited = true;
        }
        uint32_t ra[2][32];                      // 64 columns of this thread's row
        const uint32_t acc_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * 256 + ch * 64);
        if constexpr (SRC) {
          if (pre) {
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 8; ++k) *reinterpret_cast<uint4*>((k & 1 ? coal1 : coal0) + 4 * k * kPitch) = cv[k];
            __syncwarp();
          }
        }
        if (!SRC || part) {
          tmem_ld_32x32(acc_addr, ra[0]);
          tmem_ld_32x32(acc_addr + 32, ra[1]);
          tmem_ld_wait();
        }
        if (part) {          // a slice of a contraction: rows of 256 bytes per thread, a few tiles in all
          if (row0 + lane < M) {
            float* dp = fd + (long long)(row0 + lane) * ldd + col0;
#pragma unroll
            for (int q = 0; q < 16; ++q)
              if (col0 + 4 * q < N)
                reinterpret_cast<uint4*>(dp)[q] = make_uint4(ra[q >> 3][4 * (q & 7)], ra[q >> 3][4 * (q & 7) + 1],
                                                             ra[q >> 3][4 * (q & 7) + 2], ra[q >> 3][4 * (q & 7) + 3]);
          }
          continue;
        }
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int colh = col0 + hh * 32;
          if constexpr (SRC) {
            tmem_ld_32x32(acc_addr + hh * 32, ra[hh]);
            tmem_ld_wait();
          }
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(ra[hh][i]);
          if constexpr (SRC) {
            if (c) {
#pragma unroll
              for (int q = 0; q < 4; ++q) add8(v + 8 * q, *reinterpret_cast<const uint4*>(own + (((4 * hh + q) ^ osw) << 4)));
            }
          }
          if constexpr (SRC) {
            if (bias) {
#pragma unroll
              for (int q = 0; q < 4; ++q) add8(v + 8 * q, bias8(4 * hh + q));
            }
          } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) add8(v + 8 * q, bv[4 * hh + q]);
          }
          if constexpr (FUN) {
            if (act == 1) {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i], 0.f);
            } else if (act == 2) {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = 0.5f * v[i] * (1.f + erff(v[i] * 0.70710678118654752f));
            }
          }
          if constexpr (SRC) {
            if (mask) {
              const float ms = J.mask_scale;
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                uint4 u = make_uint4(0u, 0u, 0u, 0u);
                if (!c) u = *reinterpret_cast<const uint4*>(own + (((4 * hh + q) ^ osw) << 4));
                else if (row0 + lane < M && colh + q * 8 < N)     // both at once is rare: not fetched ahead
                  u = __ldcg(reinterpret_cast<const uint4*>(mask + (long long)(row0 + lane) * ldmask + colh + q * 8));
                const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  v[8 * q + 2 * i] = bf16_lo(w[i]) > 0.f ? v[8 * q + 2 * i] * ms : 0.f;
                  v[8 * q + 2 * i + 1] = bf16_hi(w[i]) > 0.f ? v[8 * q + 2 * i + 1] * ms : 0.f;
                }
              }
            }
          }
          if constexpr (FUN) {
            if (thresh) {
              // element index = position in the logical [M, N] output (N and the column are multiples of 4)
              const unsigned long long e4 = ((unsigned long long)(row0 + lane) * (unsigned long long)N + (unsigned long long)colh) >> 2;
              const float dsc = J.drop_scale;
              const unsigned long long sd = J.seed;
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                const uint4 rr = philox4x32(sd, drop_off, e4 + q);
                v[4 * q] = rr.x >= thresh ? v[4 * q] * dsc : 0.f;
                v[4 * q + 1] = rr.y >= thresh ? v[4 * q + 1] * dsc : 0.f;
                v[4 * q + 2] = rr.z >= thresh ? v[4 * q + 2] * dsc : 0.f;
                v[4 * q + 3] = rr.w >= thresh ? v[4 * q + 3] * dsc : 0.f;
              }
            }
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
            *reinterpret_cast<uint4*>(own + (((4 * hh + q) ^ osw) << 4)) =
                make_uint4(pack_bf16(v[8 * q], v[8 * q + 1]), pack_bf16(v[8 * q + 2], v[8 * q + 3]),
                           pack_bf16(v[8 * q + 4], v[8 * q + 5]), pack_bf16(v[8 * q + 6], v[8 * q + 7]));
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int row = row0 + 4 * k + (lane >> 3);
          if (row < M && ccol < N)
            *reinterpret_cast<uint4*>(d + (long long)row * ldd + ccol) = *reinterpret_cast<const uint4*>((k & 1 ? coal1 : coal0) + 4 * k * kPitch);
        }
        __syncwarp();
      }
      if (!ok) break;
      // a warp without a column chunk (64-wide tiles) follows the accumulators all the same
      if (!waited) {
        uint32_t good = 1;
        if (lane == 0) good = mbar_wait(&ctl->tmem_full[acc], acc_phase, abort_flag, status, tmo) ? 1u : 0u;
        good = __shfl_sync(0xffffffffu, good, 0);
        if (!good) { ok = false; break; }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR && crank != 0) mbar_arrive_cluster(mapa_u32(smem_u32(&ctl->tmem_empty[acc]), 0));
        else mbar_arrive(&ctl->tmem_empty[acc]);
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();      // the other CTA may still signal this one's barriers or read its shared memory
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, 512); else tmem_dealloc(tmem_base, 512);
  }
}

// Adds up the slices of a split contraction, four elements a thread, always in the same order: two ranges of them (a weight
// gradient and its bias gradient).  A few MB that are still in L2: bound by its launch and by the latency of its loads.
__global__ void __launch_bounds__(256) local_reduce_kernel(const float* __restrict__ part, int n, long long stride,
                                                           __nv_bfloat16* __restrict__ out, long long len, long long off2,
                                                           __nv_bfloat16* __restrict__ out2, long long len2) {
  pdl_prologue();
  long long i = (blockIdx.x * 256ll + threadIdx.x) * 4;
  const long long first = (len + 3) / 4 * 4;
  if (i >= first) {
    i -= first;
    part += off2; out = out2; len = len2;
  }
  if (i >= len) return;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int k = 0; k < n; ++k) {
    const float4 v = __ldcs(reinterpret_cast<const float4*>(part + k * stride + i));
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  const float r[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (i + k < len) out[i + k] = __float2bfloat16(r[k]);
}

// ------------------------------------------------------------------------------------------------------------- host
thread_local std::string l_err;
int lfail(const std::string& s) { l_err = s; return -1; }

int encode(CUtensorMap* m, const void* ptr, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return lfail("cuTensorMapEncodeTiled entry point not found");
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(ptr), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : lfail("cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
}
// `mn` rows staged per CTA: one box (K-major), one 3-D box, or 64-wide 2-D boxes where mn is not a multiple of 64
int operand_map(CUtensorMap* m, unsigned char* is3d, const void* ptr, long long mn, long long k, long long ld, int stored_mn,
                int rows) {
  *is3d = 0;
  if (!stored_mn) {
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)mn}, st[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {64u, (cuuint32_t)rows};
    return encode(m, ptr, 2, dims, st, box);
  }
  if (mn % 64 == 0) {
    const cuuint64_t dims[3] = {64u, (cuuint64_t)k, (cuuint64_t)(mn / 64)}, st[2] = {(cuuint64_t)ld * 2, 128u};
    const cuuint32_t box[3] = {64u, 64u, (cuuint32_t)(rows / 64)};
    *is3d = 1;
    return encode(m, ptr, 3, dims, st, box);
  }
  const cuuint64_t dims[2] = {(cuuint64_t)mn, (cuuint64_t)k}, st[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {64u, 64u};
  return encode(m, ptr, 2, dims, st, box);
}
bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int sms() {
  static int n[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!n[dev]) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
  return n[dev];
}

// Tile shapes and what they cost in SM clocks, fitted to measured launches (1024 x 2048 -> 2048, K from 256 to 2048, all
// operands in L2): `clk` per k-block of 64, `epi` for the epilogue of a unit's last tile, which nothing hides.  A pair's
// k-block does four times (256 x 256) or twice (256 x 128) the work of a 128 x 128 tile's; its tensor work alone is 512
// and 256 clocks.  Examples, us with {256 x 256, 256 x 128, 128 x 128, 128 x 64}: forward 1024 x 2048 -> 2048
// {17.3, 14.5, 13.9, 21.1}, its backward {19.1, 23.3, 27.0, 37.8}, forward 1024 x 512 -> 512 {10.0, 8.2, 7.6, 7.2},
// 8192 x 2048 -> 8192 {185, 252, 257, 454}.
// A column-sum tile loads 16 KB per k-block and CTA.
// `drain` is what bounds a tile of few k-blocks: the epilogue's warps empty one accumulator at a time, and two fifths of the
// k-loop's clocks come on top (8192 x 8192 with K = 8 / 512, us: {45, 59, 58, 90} / {62, 79, 80, 139}); three fifths
// of `epi` are left to add for the last one.  Without it the weight gradient of a few tokens fell into 64-wide tiles, each
// as long as a 128-wide one: backward of 8 x 2048 -> 8192 70 to 82 us, now 47 (65 before there was a choice).
constexpr int kSumClk = 330;
struct TileShape { bool pair; int bn, clk, epi, drain; };
constexpr TileShape kShapes[4] = {{true, 256, 650, 4600, 5600}, {true, 128, 545, 1700, 3700},
                                  {false, 128, 530, 700, 3600}, {false, 64, 480, 0, 3000}};
constexpr int kTileFixed = 300;       // hand-over between two tiles of a unit

// a GEMM, or the column sums of its A
struct Item { const LocalGemm* g; bool sum; };
constexpr int kMaxItems = kLocalMaxJobs + kLocalMaxJobs / 2;

// clocks of one tile of an item, how many there are, and what the last one's epilogue adds
struct Tiles { long long cost, count, epi; };
Tiles tiles_of(const Item& x, const TileShape& s) {
  const int tm = s.pair ? 256 : 128;
  const long long kb = (x.g->K + 63) / 64, slices = std::max(x.g->part, 1), k = (kb + slices - 1) / slices;
  const long long rows = (x.g->M + tm - 1) / tm * slices;
  if (x.sum) return Tiles{k * kSumClk + kTileFixed, rows, 0};
  const long long loop = k * s.clk + kTileFixed, drain = s.drain + loop * 2 / 5;
  return Tiles{std::max(loop, drain), rows * ((x.g->N + s.bn - 1) / s.bn), loop >= drain ? s.epi : s.epi * 3 / 5};
}
// Clocks of the longest unit of a launch in which job i uses tile shape sh[i]; `ord` sorts the jobs by falling tile cost.
// A unit's load only changes where some job's first or last partial round ends, so one unit of each stretch between those
// places is looked at, not every tile of every unit: a choice for a backward of 16 tiles or of 1 000 takes 1 us or less on
// the host, where dealing out the tiles one by one took up to 12 us of an eager call (eager backward of 16384 x 256 -> 256
// 31 us, 17 before there was a choice).
long long makespan(const Item* it, int n, const TileShape* const* sh, int units, int* ord) {
  long long cost[kMaxItems], count[kMaxItems], epi = 0;
  for (int i = 0; i < n; ++i) {
    const Tiles t = tiles_of(it[i], *sh[i]);
    cost[i] = t.cost; count[i] = t.count;
    epi = std::max(epi, t.epi);
    ord[i] = i;
  }
  std::sort(ord, ord + n, [&](int a, int b) { return cost[a] != cost[b] ? cost[a] > cost[b] : a < b; });
  long long first[kMaxItems + 1] = {0};          // of the jobs in order, and the end of the last
  long long sum = 0;
  for (int q = 0; q < n; ++q) {
    const int i = ord[q];
    first[q + 1] = first[q] + count[i];
    sum += count[i] * cost[i];
  }
  if (first[n] > 8ll * units) return sum / units + cost[ord[0]] / 2 + epi;     // many rounds: the average is close enough
  // Of the first x tiles a unit takes one of every full round, and one of the last, partial round if the dealing has come
  // to it (see unit_tile): the units below `turn` where that round runs upwards, those from it on where it runs back.
  int rounds[kMaxItems + 1], turn[kMaxItems + 1];
  for (int e = 0; e <= n; ++e) {
    rounds[e] = (int)first[e] / units;
    const int rem = (int)first[e] - rounds[e] * units;
    turn[e] = rounds[e] & 1 ? units - rem : rem;
  }
  long long best = 0;
  for (int e = 0; e <= n; ++e) {
    const int u = turn[e];                       // where a stretch of equal units begins
    if (u == units) continue;
    long long load = 0;
    int before = 0;
    for (int q = 0; q < n; ++q) {
      const int upto = rounds[q + 1] + (rounds[q + 1] & 1 ? u >= turn[q + 1] : u < turn[q + 1]);
      load += (upto - before) * cost[ord[q]];
      before = upto;
    }
    best = std::max(best, load);
  }
  return best + epi;
}

template <bool PAIR, int MAXJ, bool SRC, bool FUN, bool FILL = false>
int launch_local(const Params<MAXJ>& P, cudaStream_t stream) {
  if (ensure_smem<local_gemm_kernel<PAIR, MAXJ, SRC, FUN, FILL>>(kSmem) != cudaSuccess) return lfail("cudaFuncSetAttribute failed");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(PAIR ? 2 * P.units : P.units);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  int nat = 0;
  if (pdl_local()) {
    at[nat].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[nat].val.programmaticStreamSerializationAllowed = 1;
    ++nat;
  }
  if (PAIR) {
    at[nat].id = cudaLaunchAttributeClusterDimension;
    at[nat].val.clusterDim.x = 2; at[nat].val.clusterDim.y = 1; at[nat].val.clusterDim.z = 1;
    ++nat;
  }
  cfg.attrs = at;
  cfg.numAttrs = nat;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, local_gemm_kernel<PAIR, MAXJ, SRC, FUN, FILL>, P);
  return e == cudaSuccess ? 0 : lfail(std::string("launch local_gemm_kernel: ") + cudaGetErrorString(e));
}

// Tile shapes (pairs or single CTAs for the launch, then the wide or the narrow tile for each job) and the order of the
// jobs.  Returns the clocks of the longest unit, -1: no shape for this device.
long long choose(const Item* it, int n, int pair_policy, int n_sm, const TileShape** best_sh, int* best_ord) {
  const TileShape* sh[kMaxItems];
  int ord[kMaxItems];
  long long best = -1;
  for (int s = 0; s < 4; s += 2) {
    const TileShape *wide = &kShapes[s], *narrow = &kShapes[s + 1];
    const int units = wide->pair ? n_sm / 2 : n_sm;
    if (!units || pair_policy == (wide->pair ? 0 : 1)) continue;
    auto consider = [&] {
      const long long v = makespan(it, n, sh, units, ord);
      if (best < 0 || v < best) {
        best = v;
        std::copy(sh, sh + n, best_sh);
        std::copy(ord, ord + n, best_ord);
      }
      return v;
    };
    std::fill(sh, sh + n, wide);
    long long cur = consider();
    for (int i = 0; i < n && n <= 4; ++i) {
      if (it[i].sum) continue;                   // one job at a time: the narrow tile stays where it shortens the launch
      sh[i] = narrow;
      const long long v = consider();
      if (v < cur) cur = v; else sh[i] = wide;
    }
    std::fill(sh, sh + n, narrow);
    consider();
  }
  return best;
}

template <int MAXJ>
int run(const Item* it, int n, int pair_policy, unsigned long long* status, unsigned long long timeout_ns, cudaStream_t stream) {
  const int n_sm = sms();
  const TileShape* best_sh[kMaxItems];
  int best_ord[kMaxItems];
  if (choose(it, n, pair_policy, n_sm, best_sh, best_ord) < 0) return lfail("no tile shape for this device");
  const bool pair = best_sh[0]->pair;

  static thread_local Params<MAXJ> P;
  memset(static_cast<void*>(&P), 0, sizeof(P));
  const int tm = pair ? 256 : 128;
  int widest = 0, total = 0;
  bool sums = false, src = false, fun = false, fill = false;
  for (int q = 0; q < n; ++q) {
    const LocalGemm& x = *it[best_ord[q]].g;
    src = src || x.c || x.mask;
    fun = fun || x.act || x.drop_p > 0.f;
    fill = fill || x.m_fill || x.k_fill;
    Job& J = P.job[q];
    J.sum = it[best_ord[q]].sum ? 1 : 0;
    J.M = x.M; J.kblocks = (x.K + 63) / 64;
    const int slices = std::max(x.part, 1);
    if (x.part) { J.kper = (J.kblocks + slices - 1) / slices; J.part_stride = x.part_stride; }
    J.tile0 = total;
    J.tiles_m = (x.M + tm - 1) / tm;
    J.group = 8;
    J.a_mn = (unsigned char)x.a_mn;
    J.m_fill = J.sum ? nullptr : x.m_fill;
    J.k_fill = x.k_fill;
    if (operand_map(&J.ma, &J.a3, x.a, x.M, x.K, x.lda, x.a_mn, 128)) return -1;
    if (J.sum) {
      sums = true;
      J.bn = J.N = 16; J.tiles_n = 1;
      J.d = x.bsum;
      if (x.bsum_add) J.c = x.bsum;
      J.slice_tiles = J.tiles_m;
      total += J.tiles_m * slices;
      continue;
    }
    J.bn = best_sh[best_ord[q]]->bn;
    const int rows_b = pair ? J.bn / 2 : J.bn;
    widest = std::max(widest, rows_b);
    if (operand_map(&J.mb, &J.b3, x.b, x.N, x.K, x.ldb, x.b_mn, rows_b)) return -1;
    J.b_mn = (unsigned char)x.b_mn;
    J.N = x.N; J.tiles_n = (x.N + J.bn - 1) / J.bn;
    // Every group reads all of B again, so a wide output takes 16 rows a group while their part of A still stays in L2 beside
    // it: forward 4096 x 2048 -> 50304 563 -> 546 us, 8192 rows 1147 -> 1103.  Not for a tall one (weight gradient of 50304 x
    // 2048 over 4096 1238 -> 1298 us) nor a long contraction (8192^3 724 -> 740).
    if (J.tiles_n >= J.tiles_m && 16ll * tm * x.K * 2 <= (32ll << 20)) J.group = 16;
    J.slice_tiles = J.tiles_m * J.tiles_n;
    total += J.slice_tiles * slices;
    J.d = x.d; J.ldd = x.ldd; J.c = x.c; J.ldc = x.ldc; J.bias = x.bias; J.act = x.act;
    J.mask = x.mask; J.ldmask = x.ldmask; J.mask_scale = x.mask_scale;
    if (x.drop_p > 0.f) {
      const double th = (double)x.drop_p * 4294967296.0;
      J.drop_thresh = th > 4294967295.0 ? 4294967295u : (uint32_t)th;
      J.drop_scale = 1.f / (1.f - x.drop_p);
      J.seed = x.seed; J.offset = x.offset; J.step_ptr = x.step_ptr;
    }
  }
  P.njobs = n; P.total = total;
  P.units = std::min(total, pair ? n_sm / 2 : n_sm);
  P.stage_bytes = kABytesL + widest * kKB * 2;
  P.stages = std::min(kStages, kArea / P.stage_bytes);
  if (sums) {
    // pairs: behind the staging rows; single CTAs, whose 16 rows need 2 KB: in place of the last stage (four already
    // keep a single CTA's k-loop at its full rate)
    if (!pair) --P.stages;
    P.ones_off = pair ? kArea + kStageOut : P.stages * P.stage_bytes;
  }
  P.status = status; P.timeout_ns = 2 * timeout_ns;
  if (fill) {
    if (src || fun) return lfail("local_gemm: rows in use go with plain jobs only");
    return pair ? launch_local<true, MAXJ, false, false, true>(P, stream) : launch_local<false, MAXJ, false, false, true>(P, stream);
  }
#define RTP_LOCAL(SRC, FUN) (pair ? launch_local<true, MAXJ, SRC, FUN>(P, stream) : launch_local<false, MAXJ, SRC, FUN>(P, stream))
  return src ? (fun ? RTP_LOCAL(true, true) : RTP_LOCAL(true, false)) : (fun ? RTP_LOCAL(false, true) : RTP_LOCAL(false, false));
#undef RTP_LOCAL
}

int items_of(const LocalGemm* jobs, int n, Item* it) {
  int m = 0;
  for (int i = 0; i < n; ++i) it[m++] = Item{&jobs[i], false};
  for (int i = 0; i < n; ++i)
    if (jobs[i].bsum) {
      if (m == kMaxItems) return -1;
      it[m++] = Item{&jobs[i], true};
    }
  return m;
}

}  // namespace

int local_reduce(const float* part, int n, long long stride, void* out, long long len, long long off2, void* out2, long long len2,
                 cudaStream_t stream) {
  const long long items = (len + 3) / 4 + (len2 + 3) / 4;
  if (items <= 0) return 0;
  const cudaError_t e = launch_k(local_reduce_kernel, dim3((unsigned)((items + 255) / 256)), dim3(256), 0, stream, part, n, stride,
                                 reinterpret_cast<__nv_bfloat16*>(out), len, off2, reinterpret_cast<__nv_bfloat16*>(out2), len2);
  return e == cudaSuccess ? 0 : lfail(std::string("launch local_reduce_kernel: ") + cudaGetErrorString(e));
}

const char* local_gemm_error() { return l_err.c_str(); }

bool local_gemm_ok(const LocalGemm& g) {
  // TMA: 16-byte aligned bases and pitches; epilogue: 16-byte vectors of eight columns
  if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.N % 8) return false;
  if (!al16(g.a) || !al16(g.b) || g.lda % 8 || g.ldb % 8) return false;
  if (!al16(g.d) || g.ldd % 8 || !al16(g.c) || !al16(g.mask) || !al16(g.bias)) return false;
  if ((g.c && g.ldc % 8) || (g.mask && g.ldmask % 8)) return false;
  // every slice has a k-block of its own
  if (g.part < 0 || (g.part && ((g.K + 63) / 64 + g.part - 1) / g.part * (g.part - 1) >= (g.K + 63) / 64)) return false;
  if (g.part && (g.c || g.bias || g.act || g.mask || g.drop_p > 0.f || g.bsum_add)) return false;
  if ((g.m_fill || g.k_fill) && (g.c || g.act || g.mask || g.drop_p > 0.f || g.bsum_add || g.part)) return false;
  return !g.bsum || g.a_mn;
}

int local_gemm(const LocalGemm* jobs, int n, int pair_policy, unsigned long long* status, unsigned long long timeout_ns,
               cudaStream_t stream) {
  if (n < 1 || n > kLocalMaxJobs) return lfail("local_gemm: number of jobs out of range");
  for (int i = 0; i < n; ++i)
    if (!local_gemm_ok(jobs[i])) return lfail("local_gemm: operand not aligned to 16 bytes, or N not a multiple of 8");
  Item it[kMaxItems];
  const int m = items_of(jobs, n, it);
  if (m < 0) return lfail("local_gemm: too many column sums");
  return m <= 3 ? run<3>(it, m, pair_policy, status, timeout_ns, stream)
                : run<kMaxItems>(it, m, pair_policy, status, timeout_ns, stream);
}

}  // namespace rtp

// The choice that a launch of these jobs (4 numbers each: M, N, K, 1 = with the column sums of A) makes on a device of n_sm
// SMs; host only.  out: clocks of the longest unit, units, the epilogue share of those clocks, then cost and number of the
// tiles of each job and sum in the order in which they are dealt out.  Returns the number of those, -1: no such launch.
extern "C" int rtp_lint_local_plan(int n_sm, int pair_policy, int n, const int* mnks, long long* out) {
  using namespace rtp;
  if (n < 1 || n > kLocalMaxJobs) return -1;
  LocalGemm jobs[kLocalMaxJobs] = {};
  for (int i = 0; i < n; ++i) {
    jobs[i].M = mnks[4 * i]; jobs[i].N = mnks[4 * i + 1]; jobs[i].K = mnks[4 * i + 2];
    jobs[i].bsum = mnks[4 * i + 3] ? &jobs[i] : nullptr;
  }
  Item it[kMaxItems];
  const TileShape* sh[kMaxItems];
  int ord[kMaxItems];
  const int m = items_of(jobs, n, it);
  if (m < 0 || (out[0] = choose(it, m, pair_policy, n_sm, sh, ord)) < 0) return -1;
  const bool pair = sh[0]->pair;
  out[1] = pair ? n_sm / 2 : n_sm;
  out[2] = 0;
  for (int q = 0; q < m; ++q) {
    const int i = ord[q];
    const Tiles t = tiles_of(it[i], *sh[i]);
    out[2] = std::max(out[2], t.epi);
    out[3 + 2 * q] = t.cost; out[4 + 2 * q] = t.count;
  }
  return m;
}

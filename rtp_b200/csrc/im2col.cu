// Patch matrices for convolution as GEMM: a rotated Conv2d (output channels sharded, reference rtp/module/conv.py:103-114)
// runs on the rotation GEMM kernels as a column-parallel linear over the unfolded input.
//   im2col : x [B, C, H, W] bf16  ->  cols [B*OH*OW, Kp] bf16, column (c, kh, kw) = c*KH*KW + kh*KW + kw, zero padded to Kp
//   col2im : dcols [B*OH*OW, Kp]  ->  dx [B, C, H, W]  (gather form: every input element sums the patch entries that
//            read it, so there are no atomics and the result does not depend on scheduling)
//   rows   : dy [B, C, P] bf16  ->  [B*P, C]: the output gradient as the GEMM reads it
// Patches overlap, so im2col reads its input from shared memory and col2im keeps the patches of a few output rows there: each
// reads global memory once (or a little more) in whole lines and is bound by the patch matrix.  One thread per patch of a
// channel, every element from global memory, is what is left for inputs whose rows do not fit.  us, that form -> this
// (64 x 32 x 26 x 26, 3 x 3; 64 x 1 x 28 x 28, 3 x 3; 32 x 64 x 32 x 32, 5 x 5, padding 1): im2col 36, 6.2, 314 -> 14.5, 2.6, 57,
// col2im 49, 6.2, 181 -> 23, 3.1, 120.  The patches of one row of 26 positions and 8 channels do not fit from 7 x 7 on: col2im of
// 64 x 32 x 26 x 26, 7 x 7 stays at 195.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <string>

#include "common.cuh"
#include "kernels.h"
#include "launch.h"

namespace {
using namespace rtp;

std::string g_err;

struct ConvGeom {
  int B, C, H, W, KH, KW, OH, OW, sh, sw, ph, pw, dh, dw, Kp;
};

// One thread per (output position m, input channel c): the position is decoded once and the thread writes the channel's
// KH*KW consecutive patch entries (adjacent threads write adjacent channels, so a warp's stores are contiguous).
// Threads with c == C fill the zero padding of the row up to Kp.
__global__ void im2col_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ cols, ConvGeom g) {
  const int KK = g.KH * g.KW;
  const int K = g.C * KK;
  const int cpr = g.C + (g.Kp > K ? 1 : 0);          // work items per output row
  const long long total = (long long)g.B * g.OH * g.OW * cpr;
  const __nv_bfloat16 zero = __float2bfloat16(0.f);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % cpr);
    const long long m = i / cpr;
    __nv_bfloat16* dst = cols + m * g.Kp;
    if (c == g.C) {
      for (int k = K; k < g.Kp; ++k) dst[k] = zero;
      continue;
    }
    const int ow = (int)(m % g.OW), oh = (int)((m / g.OW) % g.OH), b = (int)(m / ((long long)g.OW * g.OH));
    const __nv_bfloat16* src = x + ((long long)b * g.C + c) * g.H * g.W;
    dst += c * KK;
    const int h0 = oh * g.sh - g.ph, w0 = ow * g.sw - g.pw;
    for (int kh = 0; kh < g.KH; ++kh) {
      const int h = h0 + kh * g.dh;
      const bool hok = h >= 0 && h < g.H;
      for (int kw = 0; kw < g.KW; ++kw) {
        const int w = w0 + kw * g.dw;
        dst[kh * g.KW + kw] = (hok && w >= 0 && w < g.W) ? src[(long long)h * g.W + w] : zero;
      }
    }
  }
}

__global__ void col2im_kernel(const __nv_bfloat16* __restrict__ dcols, __nv_bfloat16* __restrict__ dx, ConvGeom g) {
  const long long total = (long long)g.B * g.C * g.H * g.W;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int w = (int)(i % g.W), h = (int)((i / g.W) % g.H), c = (int)((i / ((long long)g.W * g.H)) % g.C);
    const int b = (int)(i / ((long long)g.W * g.H * g.C));
    float acc = 0.f;
    for (int kh = 0; kh < g.KH; ++kh) {
      const int hn = h + g.ph - kh * g.dh;
      if (hn < 0 || hn % g.sh) continue;
      const int oh = hn / g.sh;
      if (oh >= g.OH) continue;
      for (int kw = 0; kw < g.KW; ++kw) {
        const int wn = w + g.pw - kw * g.dw;
        if (wn < 0 || wn % g.sw) continue;
        const int ow = wn / g.sw;
        if (ow >= g.OW) continue;
        const long long m = ((long long)b * g.OH + oh) * g.OW + ow;
        acc += __bfloat162float(dcols[m * g.Kp + (c * g.KH + kh) * g.KW + kw]);
      }
    }
    dx[i] = __float2bfloat16(acc);
  }
}

// im2col through shared memory.  Block: R output rows of one image.  The input rows that they read, halo included, lie in shared
// memory as [C][rows][Wp]; a table holds the place of each patch entry k relative to the patch's origin (entries beyond the
// patch read a zero).  A thread makes 16 bytes of a patch, neighbouring threads neighbouring ones.
constexpr int kSmemConv = 96 * 1024;        // two blocks an SM
struct RowTile {
  int R, rows, Wp;                          // output rows of a block, input rows that they read, row pitch
};
// U loads of a thread in flight.
template <int U>
__global__ void __launch_bounds__(256) im2col_rows_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ cols,
                                                          ConvGeom g, RowTile t) {
  extern __shared__ __align__(16) uint8_t smem[];
  int* place = reinterpret_cast<int*>(smem);                        // Kp entries (a multiple of 8)
  __nv_bfloat16* tile = reinterpret_cast<__nv_bfloat16*>(smem + (size_t)g.Kp * 4);
  const int KK = g.KH * g.KW, K = g.C * KK, plane = t.rows * t.Wp, zero_at = g.C * plane;
  const int per = (g.OH + t.R - 1) / t.R, b = blockIdx.x / per, oh0 = (blockIdx.x % per) * t.R;
  const int nrow = min(t.R, g.OH - oh0), h0 = oh0 * g.sh - g.ph;
  for (int k = threadIdx.x; k < g.Kp; k += 256) {
    const int c = k / KK, r = k - c * KK, kh = r / g.KW, kw = r - kh * g.KW;
    place[k] = k < K ? c * plane + kh * g.dh * t.Wp + kw * g.dw : -1;
  }
  // an element of the tile every 256: (c, r, w) is carried along instead of being divided out each time
  const int dw = 256 % t.Wp, dr = 256 / t.Wp % t.rows, dc = 256 / t.Wp / t.rows;
  int w = threadIdx.x % t.Wp, r = threadIdx.x / t.Wp % t.rows, c = threadIdx.x / t.Wp / t.rows;
  pdl_prologue();
  const __nv_bfloat16* src = x + (size_t)b * g.C * g.H * g.W;
  const unsigned short* src16 = reinterpret_cast<const unsigned short*>(src);
  unsigned short* tile16 = reinterpret_cast<unsigned short*>(tile);
  for (int i = threadIdx.x; i < zero_at; i += U * 256) {
    uint32_t e[U];
    bool in[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int h = h0 + r, v = w - g.pw;
      in[u] = i + u * 256 < zero_at && h >= 0 && h < g.H && v >= 0 && v < g.W;
      e[u] = __ldg(src16 + (in[u] ? (c * g.H + h) * g.W + v : 0));      // an image has fewer than 2^31 elements
      w += dw; r += dr; c += dc;
      if (w >= t.Wp) { w -= t.Wp; ++r; }
      if (r >= t.rows) { r -= t.rows; ++c; }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i + u * 256 < zero_at) tile16[i + u * 256] = in[u] ? (unsigned short)e[u] : (unsigned short)0;
  }
  __syncthreads();
  const int chunks = g.Kp / 8, total = nrow * g.OW * chunks;
  uint4* dst = reinterpret_cast<uint4*>(cols + ((size_t)b * g.OH + oh0) * g.OW * g.Kp);
  const unsigned short* t16 = reinterpret_cast<const unsigned short*>(tile);
  const int dk = 256 % chunks, dm = 256 / chunks;
  int k8 = threadIdx.x % chunks, m = threadIdx.x / chunks;
  for (int i = threadIdx.x; i < total; i += 256) {
    const int o = m / g.OW, at = o * g.sh * t.Wp + (m - o * g.OW) * g.sw;
    const int4 p0 = *reinterpret_cast<const int4*>(place + k8 * 8), p1 = *reinterpret_cast<const int4*>(place + k8 * 8 + 4);
    auto get = [&](int p) { return p >= 0 ? (uint32_t)t16[at + p] : 0u; };
    dst[i] = make_uint4(get(p0.x) | get(p0.y) << 16, get(p0.z) | get(p0.w) << 16, get(p1.x) | get(p1.y) << 16,
                        get(p1.z) | get(p1.w) << 16);
    k8 += dk; m += dm;
    if (k8 >= chunks) { k8 -= chunks; ++m; }
  }
}

// col2im through shared memory.  Block: R input rows and CG channels of one image.  The patches of the output rows that touch them
// lie in shared memory, the CG channels of a position side by side, positions an odd number of words apart: neighbouring threads
// sum neighbouring input columns, which read neighbouring positions (stride 1) without bank conflicts.
// ST > 0: stride known and dilation 1, no divisions; KT > 0: kernel known too, and the loops over a patch are unrolled.
struct FoldTile {
  int R, CG, nout, pitch;                   // input rows and channels of a block, output rows held at most, elements per position
};
template <int KT, int ST>
__global__ void __launch_bounds__(256) col2im_rows_kernel(const __nv_bfloat16* __restrict__ dcols, __nv_bfloat16* __restrict__ dx,
                                                          ConvGeom g, FoldTile t) {
  extern __shared__ __align__(16) uint8_t smem[];
  __nv_bfloat16* tile = reinterpret_cast<__nv_bfloat16*>(smem);
  const int KH = KT ? KT : g.KH, KW = KT ? KT : g.KW, sh = ST ? ST : g.sh, sw = ST ? ST : g.sw, dh = ST ? 1 : g.dh, dw = ST ? 1 : g.dw;
  const int KK = KH * KW, per = (g.H + t.R - 1) / t.R, groups = (g.C + t.CG - 1) / t.CG;
  const int cg = blockIdx.x % groups, hb = blockIdx.x / groups % per, b = blockIdx.x / groups / per;
  const int c0 = cg * t.CG, nc = min(t.CG, g.C - c0), h0 = hb * t.R, nh = min(t.R, g.H - h0);
  // output rows that read input rows h0 .. h0 + nh - 1
  const int lo = h0 + g.ph - (KH - 1) * dh, hi = h0 + nh - 1 + g.ph;
  const int o0 = lo <= 0 ? 0 : (lo + sh - 1) / sh, o1 = min(g.OH - 1, hi / sh), no = max(0, o1 - o0 + 1);
  // a group's columns start at a multiple of 8 (CG is one, or there is a single group) and are read to the next one
  const int chunks = (nc * KK + 7) / 8, total = no * g.OW * chunks;
  const uint4* src = reinterpret_cast<const uint4*>(dcols + (((size_t)b * g.OH + o0) * g.OW) * g.Kp + (size_t)c0 * KK);
  const int dk = 256 % chunks, dm = 256 / chunks;
  int k8 = threadIdx.x % chunks, m = threadIdx.x / chunks;
  pdl_prologue();
  for (int i = threadIdx.x; i < total; i += 4 * 256) {          // four loads in flight
    uint4 v[4];
    int at[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      at[u] = i + u * 256 < total ? m * t.pitch + k8 * 8 : -1;
      if (at[u] >= 0) v[u] = __ldg(src + (size_t)m * (g.Kp / 8) + k8);
      k8 += dk; m += dm;
      if (k8 >= chunks) { k8 -= chunks; ++m; }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (at[u] >= 0) {
        uint32_t* d = reinterpret_cast<uint32_t*>(tile + at[u]);
        d[0] = v[u].x; d[1] = v[u].y; d[2] = v[u].z; d[3] = v[u].w;
      }
  }
  const int outs = nc * nh * g.W;
  const int jw = 256 % g.W, jr = 256 / g.W % nh, jc = 256 / g.W / nh;
  int w = threadIdx.x % g.W, r = threadIdx.x / g.W % nh, c = threadIdx.x / g.W / nh;
  __syncthreads();
  for (int i = threadIdx.x; i < outs; i += 256) {
    const int h = h0 + r, hp = h + g.ph, wp = w + g.pw;
    float acc = 0.f;
#pragma unroll
    for (int kh = 0; kh < KH; ++kh) {
      const int hn = hp - kh * dh, oh = hn / sh;
      if (hn < 0 || oh * sh != hn || oh >= g.OH) continue;
      const __nv_bfloat16* row = tile + ((oh - o0) * g.OW) * t.pitch + (c * KH + kh) * KW;
#pragma unroll
      for (int kw = 0; kw < KW; ++kw) {
        const int wn = wp - kw * dw, ow = wn / sw;
        if (wn >= 0 && ow * sw == wn && ow < g.OW) acc += __bfloat162float(row[ow * t.pitch + kw]);
      }
    }
    dx[(((size_t)b * g.C + c0 + c) * g.H + h) * g.W + w] = __float2bfloat16(acc);
    w += jw; r += jr; c += jc;
    if (w >= g.W) { w -= g.W; ++r; }
    if (r >= nh) { r -= nh; ++c; }
  }
}

// [B, C, P] -> [B * P, C], 64 channels x 64 positions a block.
__global__ void __launch_bounds__(256) rows_kernel(const __nv_bfloat16* __restrict__ src, __nv_bfloat16* __restrict__ dst, int C, int P,
                                                   int bp, int bc) {
  __shared__ __nv_bfloat16 t[64][66];
  const int c0 = (blockIdx.x % bc) * 64, p0 = (blockIdx.x / bc % bp) * 64, b = blockIdx.x / bc / bp;
  pdl_prologue();
  const int a = threadIdx.x & 63;
#pragma unroll 4
  for (int k = threadIdx.x >> 6; k < 64; k += 4)
    if (c0 + k < C && p0 + a < P) t[k][a] = src[((size_t)b * C + c0 + k) * P + p0 + a];
  __syncthreads();
#pragma unroll 4
  for (int k = threadIdx.x >> 6; k < 64; k += 4)
    if (p0 + k < P && c0 + a < C) dst[((size_t)b * P + p0 + k) * C + c0 + a] = t[a][k];
}

int launch_geom(ConvGeom& g, int B, int C, int H, int W, int KH, int KW, int sh, int sw, int ph, int pw, int dh, int dw,
                int Kp) {
  g.B = B; g.C = C; g.H = H; g.W = W; g.KH = KH; g.KW = KW; g.sh = sh; g.sw = sw; g.ph = ph; g.pw = pw; g.dh = dh; g.dw = dw;
  g.OH = (H + 2 * ph - dh * (KH - 1) - 1) / sh + 1;
  g.OW = (W + 2 * pw - dw * (KW - 1) - 1) / sw + 1;
  g.Kp = Kp;
  if (g.OH <= 0 || g.OW <= 0 || Kp < C * KH * KW) { g_err = "im2col: bad geometry"; return -1; }
  return 0;
}

int device_sms() {
  static int n[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!n[dev]) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
  return n[dev];
}

template <int KT, int ST>
cudaError_t launch_fold(const ConvGeom& g, const FoldTile& t, unsigned blocks, size_t bytes, const void* dcols, void* dx, cudaStream_t stream) {
  const cudaError_t e = ensure_smem<col2im_rows_kernel<KT, ST>>(kSmemConv);
  if (e != cudaSuccess) return e;
  return launch_k(col2im_rows_kernel<KT, ST>, dim3(blocks), dim3(256), bytes, stream, (const __nv_bfloat16*)dcols, (__nv_bfloat16*)dx, g, t);
}

}  // namespace

extern "C" {

const char* rtp_im2col_last_error(void) { return g_err.c_str(); }

int rtp_im2col(const void* x, void* cols, int B, int C, int H, int W, int KH, int KW, int sh, int sw, int ph, int pw,
               int dh, int dw, int Kp, void* stream) {
  ConvGeom g;
  if (launch_geom(g, B, C, H, W, KH, KW, sh, sw, ph, pw, dh, dw, Kp)) return -1;
  // as many output rows a block as leave two blocks an SM their shared memory and the launch a few blocks an SM
  RowTile t;
  t.Wp = std::max((g.OW - 1) * sw + (KW - 1) * dw + 1, 1);
  auto bytes = [&](int R) { return (long long)Kp * 4 + (long long)C * ((R - 1) * sh + (KH - 1) * dh + 1) * t.Wp * 2; };
  if (Kp % 8 == 0 && (reinterpret_cast<uintptr_t>(cols) & 15) == 0 && bytes(1) <= kSmemConv && (long long)C * H * W <= 0x7fffffff) {
    t.R = 1;
    while (t.R < 8 && t.R < g.OH && bytes(2 * t.R) <= kSmemConv && (long long)B * ((g.OH + 2 * t.R - 1) / (2 * t.R)) >= 2 * device_sms())
      t.R *= 2;
    t.rows = (t.R - 1) * sh + (KH - 1) * dh + 1;
    const long long blocks = (long long)B * ((g.OH + t.R - 1) / t.R);
    if (blocks <= 0x7fffffff) {
      // Loads in flight pay for tiles of 16 loads a thread and more at stride 1.  us, one in flight and four: 64 x 32 x 26 x 26, 3 x 3 16.1
      // and 14.5, 8 x 512 x 14 x 14, 3 x 3 31.8 and 31.0; 64 x 32 x 26 x 26, 2 x 2 by 2 6.0 and 7.4, 32 x 64 x 32 x 32, 3 x 3 by 2 9.5
      // and 12.4, 64 x 1 x 28 x 28, 3 x 3 2.6 and 2.9.
      const bool four = sh == 1 && (long long)C * t.rows * t.Wp >= 16 * 256;
      cudaError_t e = four ? rtp::ensure_smem<im2col_rows_kernel<4>>(kSmemConv) : rtp::ensure_smem<im2col_rows_kernel<1>>(kSmemConv);
      if (e == cudaSuccess)
        e = rtp::launch_k(four ? im2col_rows_kernel<4> : im2col_rows_kernel<1>, dim3((unsigned)blocks), dim3(256), (size_t)bytes(t.R),
                          (cudaStream_t)stream, (const __nv_bfloat16*)x, (__nv_bfloat16*)cols, g, t);
      if (e != cudaSuccess) { g_err = std::string("im2col: ") + cudaGetErrorString(e); return -1; }
      return 0;
    }
  }
  const long long total = (long long)g.B * g.OH * g.OW * (g.C + 1);
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 32) blocks = 148 * 32;
  im2col_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)cols, g);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { g_err = std::string("im2col: ") + cudaGetErrorString(e); return -1; }
  return 0;
}

int rtp_col2im(const void* dcols, void* dx, int B, int C, int H, int W, int KH, int KW, int sh, int sw, int ph, int pw,
               int dh, int dw, int Kp, void* stream) {
  ConvGeom g;
  if (launch_geom(g, B, C, H, W, KH, KW, sh, sw, ph, pw, dh, dw, Kp)) return -1;
  FoldTile t;
  auto held = [&](int R, int CG) {              // bytes of the patches that a block holds
    t.R = R; t.CG = CG;
    t.nout = std::min(g.OH, (R - 1 + (KH - 1) * dh) / sh + 1);
    t.pitch = (std::min(CG, C) * KH * KW + 7) / 8 * 8 + 2;              // an odd number of words
    return (long long)t.nout * g.OW * t.pitch * 2;
  };
  if (Kp % 8 == 0 && (reinterpret_cast<uintptr_t>(dcols) & 15) == 0) {
    // Small blocks, many to an SM: all channels if a row of them takes 48 KB at most and the rows are blocks enough for two an SM, else
    // groups of a multiple of 8; more rows as long as they fit 32 KB and every SM has two blocks (64 x 32 x 26 x 26: up to 96 KB a
    // block 30 us, 48 KB 23, this 20; 8 x 256 x 14 x 14, 1 x 1, all channels 8.1 us, groups 4.6).
    int CG = C;
    while (CG > 8 && (held(1, CG) > 48 * 1024 || (long long)B * H * ((C + CG - 1) / CG) < 2 * device_sms())) CG = (CG / 2 + 7) / 8 * 8;
    if (held(1, CG) <= kSmemConv) {
      const long long groups = (C + CG - 1) / CG;
      int R = 1;
      while (R < 16 && R < H && held(2 * R, CG) <= 32 * 1024 && B * groups * ((H + 2 * R - 1) / (2 * R)) >= 2 * device_sms()) R *= 2;
      const size_t bytes = (size_t)held(R, CG);
      const long long blocks = B * groups * ((H + R - 1) / R);
      if (blocks <= 0x7fffffff) {
        // A stride that is not known costs two divisions for each entry of a patch.  us, neither known, stride, both: 64 x 32 x 26 x 26,
        // 3 x 3 44, 28, 23; 32 x 64 x 32 x 32, 5 x 5 153, 157, 120, by 2 73, 46, 45; 64 x 32 x 26 x 26, 2 x 2 by 2 33, 18, 1 x 1 17, 11.
        const int st = sh == sw && dh == 1 && dw == 1 && sh <= 2 ? sh : 0, kt = st && KH == KW && (KH == 3 || KH == 5) ? KH : 0;
        const auto launch = kt == 3 ? (st == 1 ? launch_fold<3, 1> : launch_fold<3, 2>)
                            : kt == 5 ? (st == 1 ? launch_fold<5, 1> : launch_fold<5, 2>)
                            : st == 1 ? launch_fold<0, 1> : st == 2 ? launch_fold<0, 2> : launch_fold<0, 0>;
        const cudaError_t e = launch(g, t, (unsigned)blocks, bytes, dcols, dx, (cudaStream_t)stream);
        if (e != cudaSuccess) { g_err = std::string("col2im: ") + cudaGetErrorString(e); return -1; }
        return 0;
      }
    }
  }
  const long long total = (long long)g.B * g.C * g.H * g.W;
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  col2im_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)dcols, (__nv_bfloat16*)dx, g);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { g_err = std::string("col2im: ") + cudaGetErrorString(e); return -1; }
  return 0;
}

// [B, C, P] -> [B * P, C], contiguous bf16
int rtp_nchw_rows(const void* src, void* dst, int B, int C, int P, void* stream) {
  const long long bp = (P + 63) / 64, bc = (C + 63) / 64;
  if (B <= 0 || C <= 0 || P <= 0) return 0;
  if (B * bp * bc > 0x7fffffff) { g_err = "rows: too large"; return -1; }
  const cudaError_t e = rtp::launch_k(rows_kernel, dim3((unsigned)(B * bp * bc)), dim3(256), 0, (cudaStream_t)stream,
                                      (const __nv_bfloat16*)src, (__nv_bfloat16*)dst, C, P, (int)bp, (int)bc);
  if (e != cudaSuccess) { g_err = std::string("rows: ") + cudaGetErrorString(e); return -1; }
  return 0;
}

}  // extern "C"

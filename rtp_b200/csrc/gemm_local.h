// GEMMs of a ring of one rank: nothing is pushed, nothing is waited for, so a launch needs only a few jobs
// D = epilogue(A * B^T (+ C)) that share one grid (see gemm_local.cu).  Host interface, used by gemm.cu.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace rtp {

struct LocalGemm {
  // operands (bf16), rows [M, K] or, with *_mn, stored [K, M]; likewise B with N
  const void* a; long long lda; int a_mn;
  const void* b; long long ldb; int b_mn;
  int M, N, K;
  // epilogue: (+ c) -> (+ bias) -> activation -> mask -> dropout, bf16 result
  void* d; long long ldd;
  const void* c; long long ldc;
  const void* bias;
  int act;
  const void* mask; long long ldmask; float mask_scale;
  float drop_p;
  unsigned long long seed, offset;
  const unsigned long long* step_ptr;
  // column sums of A (a_mn = 1 only): bsum[m] (+)= sum_k A[m, k], in bf16
  void* bsum; int bsum_add;
  // > 0: the contraction falls into this many slices (a multiple of 64 elements each, the last one may be shorter), and d and bsum
  // are fp32 and receive the bare sums of slice s (no c, bias, activation, mask or dropout) at d + s * part_stride and bsum +
  // s * part_stride, for local_reduce to add up; d has a pitch of N
  int part;
  long long part_stride;
  // Rows that are in use, known on the device only (expert capacities); a hint.  m_fill: output rows from there on may be anything:
  // a tile of rows behind it gets zeros, the rest of the tile that it lies in what the product and the bias make of A.  k_fill: elements
  // of the contraction, of which those from there on contribute nothing (A or B is zero there, A if there is a bsum) and up to the next
  // multiple of 64 are finite.  A launch with one of them has no c, mask, activation or dropout.
  const int* m_fill;
  const int* k_fill;
};

// Whether the local kernels take this job (16-byte aligned rows, N a multiple of 8).
bool local_gemm_ok(const LocalGemm& g);
// One launch for all jobs (1 .. kLocalMaxJobs), whose outputs are disjoint and whose inputs are no job's output.
// `pair_policy`: 0 never on CTA pairs, 1 always, -1 by the cost model.
constexpr int kLocalMaxJobs = 16;
int local_gemm(const LocalGemm* jobs, int n, int pair_policy, unsigned long long* status, unsigned long long timeout_ns,
               cudaStream_t stream);
// out[i] = bf16(sum over n parts of part[k * stride + i]), i < len, and out2[i] the same of part[k * stride + off2 + i], i < len2
// (parts 16-byte aligned, stride and off2 multiples of 4)
int local_reduce(const float* part, int n, long long stride, void* out, long long len, long long off2, void* out2, long long len2,
                 cudaStream_t stream);
const char* local_gemm_error();

}  // namespace rtp

// Kernel launch with the programmatic-dependent-launch attribute (see pdl_prologue in common.cuh).
#pragma once
#include <cuda_runtime.h>
#include <stdlib.h>

namespace rtp {

// Programmatic dependent launch: a kernel may start, set itself up and wait (griddepcontrol.wait) while its predecessor in
// the stream drains, which takes 0.5 to 1 us off a launch in a CUDA graph: step of the small LM 225 -> 210 us, of the small
// GPT 995 -> 966, of the README LM 3 657 -> 3 637; steps of many milliseconds stay as they are.  Who is launched with it:
// everything but the streaming kernels (Adam, activations, casts), whose blocks fill the SMs and then only wait: with Adam
// in it the README step took 0.2 ms longer.  Cross-entropy and attention have as many blocks and lose nothing by it (loss and
// gradient of 8192 x 50304 462 us both ways, of 1024 x 8192 13.7 -> 12.5; short launches gain).
// RTP_PDL unset: the kernels that work on this GPU alone.  RTP_PDL=1: the rotation kernels too (on the training step of a
// ring they fill the SMs' registers and shared memory, so a successor rarely finds room before its predecessor has left).
// RTP_PDL=0: none.
// A kernel that uses TMEM gives its dependents leave to start (pdl_launch_dependents) only after its CTA has allocated its
// columns.  A dependent's CTA on the same SM may hold columns while it waits for this kernel to complete; were a CTA of this
// kernel still to allocate, both would wait for good.  So whoever waits for columns waits for kernels that all have theirs.
inline int pdl_env() {
  static int v = -2;
  if (v == -2) {
    const char* e = getenv("RTP_PDL");
    v = !e || !e[0] ? -1 : e[0] == '1' ? 1 : 0;
  }
  return v;
}
inline bool pdl_enabled() { return pdl_env() == 1; }      // rotation kernels
inline bool pdl_local() { return pdl_env() != 0; }        // kernels that only touch this GPU

// Raises the dynamic shared-memory limit of kernel `Kern` on the current device, once per (kernel, device): the
// attribute belongs to the kernel on one device, so a process that drives several GPUs sets it on each.
template <auto Kern>
cudaError_t ensure_smem(int bytes) {
  constexpr int kMaxDev = 64;
  static bool done[kMaxDev] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= kMaxDev) dev = 0;
  if (done[dev]) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done[dev] = true;
  return e;
}

template <typename... KArgs, typename... Args>
cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl_local() ? 1 : 0;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Same, with thread-block clusters of `cluster` CTAs.
template <typename... KArgs, typename... Args>
cudaError_t launch_kc(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, dim3 cluster,
                      Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl_local() ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster.x;
  at[1].val.clusterDim.y = cluster.y;
  at[1].val.clusterDim.z = cluster.z;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace rtp

// Host-side launch helpers.
#pragma once

#include <atomic>
#include <cuda_runtime.h>

namespace fmla {

// Raises the dynamic shared memory limit of kernel `Kern` to `bytes`, once per device: the attribute call costs about a
// microsecond, a fifth of the host time of a launch.
template <auto Kern>
cudaError_t allow_smem(int bytes) {
  static std::atomic<unsigned long long> done{0};      // one bit per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

// Launches `Kern` as a programmatic dependent of the kernel in front of it in the stream: it may become resident while that
// kernel drains and has to call pdl_wait() before it touches anything that kernel reads or writes.
template <class... Params, class... Args>
cudaError_t launch_dependent(void (*kern)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace fmla

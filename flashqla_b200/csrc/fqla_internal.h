// Host-side helpers shared by the translation units of libfqla_sm100.so.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <utility>

#include "../../include/fqla.h"

namespace fqla {

// Opt a kernel in to `bytes` of dynamic shared memory on the current device.  The attribute is per
// device and stays; `done` (one per kernel, static at the call site) remembers the devices it was
// set on.
inline int configure_smem(const void* func, int bytes, std::atomic<unsigned long long>& done) {
  if (bytes <= 48 * 1024) return 0;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (dev < 64 && (done.load(std::memory_order_relaxed) & bit)) return 0;
  e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
  return (int)e;
}

// SMs of the current device (which may differ from call to call)
inline int sm_count() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 148;
}

// Launch with programmatic stream serialisation: the kernel's blocks may start while the kernel
// before it in the stream drains, and its set-up (barriers, tensor memory, descriptor prefetch)
// overlaps that tail and the launch latency.  Every such kernel executes pdl_wait() in every
// block before it touches global memory written (or still read) by earlier work of the stream.
template <typename... KArgs, typename... Args>
inline int launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                      Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace fqla

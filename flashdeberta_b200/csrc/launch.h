// Host helpers around kernel launches.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

namespace fdb {

// Lets `kernel` take `bytes` of dynamic shared memory on the current device: asked for once per device (`done` is the
// kernel's own static, one bit per device).
inline cudaError_t allow_smem(std::atomic<uint64_t>& done, const void* kernel, int bytes) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && ((done.load(std::memory_order_relaxed) >> dev) & 1u)) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && dev < 64) done.fetch_or(uint64_t(1) << dev, std::memory_order_relaxed);
  return e;
}

// Multiprocessors of the current device (0: no device).
inline int sm_count() {
  static std::atomic<int> known[64];
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (dev < 64 && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (dev < 64) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

// Kernel launch with programmatic stream serialisation when `chained` (the kernel before may still be running when this one
// starts its prologue: see grid_wait in sm100_ptx.cuh) and clusters of `cluster` CTAs.
template <typename Args>
inline cudaError_t launch_kernel(void (*kernel)(Args), const Args& args, dim3 grid, int threads, size_t smem, bool chained,
                                 cudaStream_t stream, int cluster = 1) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  unsigned n = 0;
  if (cluster > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = (unsigned)cluster;
    at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
    ++n;
  }
  if (chained) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  void* ptr = const_cast<Args*>(&args);
  return cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(kernel), &ptr);
}

}  // namespace fdb

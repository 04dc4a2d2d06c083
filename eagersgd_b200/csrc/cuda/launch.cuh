// Launches that may begin before the kernel ahead of them in the stream has ended.
//
// Programmatic dependent launch hides the launch latency and the tail of the previous kernel (about a microsecond per
// boundary; a CIFAR step is 200 of them, one image through ResNet-50 sixty): the grid becomes resident as the previous one
// drains and waits inside, in pdl_enter(), until that one has completed and its memory is visible.  EVERY kernel launched
// this way calls pdl_enter() before it touches memory, so completion stays transitive along the stream.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include "launch_count.cuh"

namespace esgd {

__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// SMs of the device; a B200's where there is none (the launchers' host arithmetic is tested without one).
inline int sm_count() {
  static const int count = [] {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 0;
    return n > 0 ? n : 148;
  }();
  return count;
}

// More than 48 KB of dynamic shared memory have to be asked for, once for each kernel and device of the process.
using SmemAllowed = std::atomic<uint64_t>;      // one for each kernel; bit d: asked for on device d
template <class K>
inline int allow_smem(K kernel, int bytes, SmemAllowed& devices) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  const uint64_t bit = dev < 64 ? (uint64_t)1 << dev : 0;
  if (devices.load(std::memory_order_relaxed) & bit) return 0;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) devices.fetch_or(bit, std::memory_order_relaxed);
  return (int)e;
}

// kCluster: CTAs of a cluster (along x).
template <int kCluster = 1, class... K, class... A>
inline int launch(void (*kernel)(K...), dim3 grid, int threads, size_t smem, void* stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (kCluster > 1) {
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = kCluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  count_launch();
  return (int)cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
}

}  // namespace esgd

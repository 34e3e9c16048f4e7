// Programmatic dependent launch for the chain of small kernels of a decode step.  A kernel launched through
// launch_dependent() may be made resident while its predecessor in the stream still runs, once every CTA of the
// predecessor has executed dependents_may_start() (or exited); it must call wait_for_predecessor() before it reads
// anything the predecessor wrote or writes anything the predecessor may still read, and it must not read such data
// through `const __restrict__` pointers or __ldg: loads the compiler may treat as invariant can be moved above the
// wait (seen: a stale position, one chunk early, exactly at chunk boundaries).  Both calls do nothing in a kernel
// that was launched the ordinary way.  MOBA_NO_PDL=1 in the environment makes every launch ordinary (for
// comparison); MOBA_PDL_MASK=<bits> keeps the dependent form only for the kinds whose bit is set (1 projections,
// 2 a step's first launch, 4 routing, 8 attention and a small batch's whole step, 16 arg-max, 32 merge), which is how the rule above was found.
#pragma once
#include <cuda_runtime.h>
#include <stdlib.h>

#include <atomic>

namespace moba {

__device__ __forceinline__ void dependents_may_start() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

inline unsigned dependent_launch_mask() {
  static const unsigned mask = [] {
    const char* e = getenv("MOBA_NO_PDL");
    if (e && e[0] == '1') return 0u;
    const char* m = getenv("MOBA_PDL_MASK");
    return m ? (unsigned)strtoul(m, nullptr, 0) : ~0u;
  }();
  return mask;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(unsigned kind, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (dependent_launch_mask() & kind) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

// SMs of the current device; a full B200's where none answers (sizes asked for without a GPU).
inline int device_sms() {
  static std::atomic<int> cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) return 148;
    cached[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

// The limit of a kernel's dynamic shared memory, which belongs to the function: one value per kernel, set once per device (a call
// of the runtime costs a small prefill as much as a tenth of a launch, and it has four such kernels).
template <auto KERNEL>
inline cudaError_t shared_memory_limit(int bytes) {
  static std::atomic<bool> done[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && done[dev].load(std::memory_order_relaxed)) return cudaSuccess;
  e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && dev < 64) done[dev].store(true, std::memory_order_relaxed);
  return e;
}

// The same for a grid of clusters of `cluster` CTAs along x.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent_cluster(unsigned kind, void (*kernel)(KArgs...), dim3 grid, dim3 block, unsigned cluster, size_t smem,
                                            cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (dependent_launch_mask() & kind) ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

}  // namespace moba

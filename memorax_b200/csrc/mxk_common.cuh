// Shared host/device helpers for the mxk kernels (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "mxk.h"

namespace mxk {

constexpr int kNumSMs = 148;  // B200: 2 dies x 74 SMs; grids are sized against this

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Of the launches since the last call (cudaGetLastError forgets what it reports): once, behind the last launch.
inline int launch_status() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MXK_OK : static_cast<int>(e);
}

// Raises a kernel's dynamic shared memory limit, once per kernel and device (the call costs as much as a launch) -- hence to
// a constant: the most that any launch of the kernel asks for.
constexpr int kMaxSmem = 227 * 1024;
template <auto kKernel, int kBytes>
inline int allow_smem() {
  static_assert(kBytes <= kMaxSmem, "shared memory of an SM");
  static std::atomic<uint64_t> done{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (done.load(std::memory_order_acquire) & bit) return MXK_OK;
  e = cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
  if (e != cudaSuccess) return static_cast<int>(e);
  done.fetch_or(bit, std::memory_order_release);
  return MXK_OK;
}

// Kernel launch that may be set up while the kernel in front of it still runs (programmatic dependent launch: 0.7-1 us
// less between two small kernels).  Every kernel of this library begins with enter_kernel(), which waits for the kernels in
// front before anything is read or written, so the order of effects on a stream is the usual one.  What became of a launch
// is launch_status()'s to say.
template <typename... P, typename... A>
inline void launch_kernel_clusters(void (*kernel)(P...), unsigned cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                  A&&... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
inline void launch_kernel(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  launch_kernel_clusters(kernel, 1, grid, block, smem, stream, static_cast<A&&>(args)...);
}

// First statement of every kernel, executed by all threads.  A grid of at most two blocks per SM lets its successor's
// blocks take their places at once (`brief`: a persistent kernel says whether its blocks have one piece of work only); a
// larger or longer one would have them wait, or pile up on the SMs that empty first (3 % of the 1024 x 1024 LRU layer).
__device__ __forceinline__ void enter_kernel(bool brief = true) {
  if (brief && gridDim.x * gridDim.y * gridDim.z <= 2u * kNumSMs) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// 16-byte streaming accesses: data that is touched once should not displace
// reusable lines (the carried state, chunk tiles) from L1/L2.
__device__ __forceinline__ float4 ld_stream(const float4* p) { return __ldcs(p); }
__device__ __forceinline__ float2 ld_stream(const float2* p) { return __ldcs(p); }
__device__ __forceinline__ float ld_stream(const float* p) { return __ldcs(p); }
__device__ __forceinline__ uint4 ld_stream(const uint4* p) { return __ldcs(p); }
__device__ __forceinline__ void st_stream(float4* p, float4 v) { __stcs(p, v); }
__device__ __forceinline__ void st_stream(float2* p, float2 v) { __stcs(p, v); }
__device__ __forceinline__ void st_stream(float* p, float v) { __stcs(p, v); }

}  // namespace mxk

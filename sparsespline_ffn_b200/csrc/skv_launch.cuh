// Host-side launch helpers of the tensor-core kernels.
#pragma once

#include <atomic>
#include <utility>

#include <cuda_runtime.h>

namespace skv {

// Programmatic dependent launch: a kernel of a call's chain may be scheduled while its predecessor still
// runs (its CTAs have all started); pdl_wait() returns once the predecessor is complete and its
// writes are visible.  Every kernel launched through launch_chained() calls it in every thread that touches what earlier
// kernels wrote, at its end at the latest, so that whoever waits for it has waited for all in front of it.
//
// The first kernel of a call waits in every thread before anything else and only then lets its successor start: from there on the
// call's inputs may be read without a wait.  In a CUDA-core call it is chained to whatever was on the stream (a plain launch
// leaves 1.5 us between two calls); in a tensor-core call, where it is the scan, it is launched plainly (launch_prep says why).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// (What an earlier kernel may have written, of the chain or of the call in front of it, is read through plain pointers or ld16, never
// through const __restrict__ pointers, __ldg or ld.global.nc: those are for memory that nothing writes while the kernel is resident, a
// chained kernel is resident before its wait returns, and the compiler may move such loads above the wait.)
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// 16, 8 and 4 bytes, not moved across pdl_wait().
__device__ __forceinline__ uint4 ld16(const void* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ uint2 ld8(const void* p) {
  uint2 v;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ld4(const void* p) {
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// Raises the kernel's dynamic shared-memory limit to all the device has, once per kernel and device.
template <auto Kernel>
cudaError_t allow_all_smem() {
  static std::atomic<uint64_t> done{0};
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev)) return e;
  const uint64_t bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
  return e;
}

template <auto Kernel, typename... Args>
cudaError_t launch_chained(dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, const Args&... args) {
  if (smem > 48 * 1024)
    if (cudaError_t e = allow_all_smem<Kernel>()) return e;
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
  return cudaLaunchKernelEx(&cfg, Kernel, args...);
}

}  // namespace skv

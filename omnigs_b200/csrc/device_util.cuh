// Small device helpers: relaxed GPU-scope loads/stores for look-back words, bounded spin limits.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <utility>

namespace omnigs {

constexpr unsigned kFullMask = 0xffffffffu;
// Every spin-wait on another block's flag gives up after this many polls (with a short sleep
// between polls), records a status bit and lets the kernel finish.
constexpr int kMaxSpins = 1 << 20;

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Copies to shared memory that hold no register meanwhile.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Waits for all groups but the newest.
__device__ __forceinline__ void cp_async_wait_previous() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Programmatic dependent launch (launch_chained): a kernel of a chain first lets the next one's blocks be
// scheduled as its own finish starting, then waits until everything before it has completed and its
// writes are visible.  A kernel that is launched so calls this before it touches memory; launched
// otherwise it changes nothing.
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31; }

// Launches a kernel that begins with chain_begin(), with `chained` so that its launch overlaps the kernel
// before it on the stream (also inside a captured graph).  Where kernels are a few microseconds long that is
// much of their time (64.5 -> 57.2 us for the forward of 10,000 Gaussians at 512x256); where they are longer it
// costs more than it gains (kChainRecords).
template <class... Params, class... Args>
inline void launch_chained(bool chained, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = chained ? 1 : 0;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace omnigs

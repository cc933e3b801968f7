// How the kernels are launched: programmatic dependent launch, clusters, and the shared-memory attribute set once.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <mutex>

namespace snntc {

// A step of a small network is a chain of kernels of a few microseconds, and between two of them the GPU drains, flushes and
// launches: about 1.5 us each. Every kernel launched by launch_chained begins with chain_wait(), in front of its first access
// to global memory, and then chain_next(): a SMALL next kernel of the stream may be put on the SMs as soon as all CTAs of this
// one have started, does its own launch work meanwhile, and waits in its chain_wait() until this one has finished and its
// writes are visible. A kernel that waits has in turn waited for its own predecessor, so stream order holds throughout.
// Measured: the MLP on one sample 64 -> 54 us. Small means up to four warps per SM: a larger grid that is placed while the
// kernel in front still holds some of the SMs crowds onto the others (the walk of 25 088 -> 1024 at 64 samples behind a sort on
// 64 SMs: the whole layer 1119 -> 1278 us), and has nothing to gain from 1.5 us.
constexpr long kChainThreads = 148L * 128;
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// What a chained kernel reads, the kernel in front of it may still be writing while this one is already on the SMs. Loads through
// the read-only path (__ldg, or any load through a const __restrict__ kernel parameter, which the compiler turns into one) are
// defined for memory that nobody writes during the WHOLE life of a kernel: the compiler may move them in front of chain_wait(),
// and the path need not see the other kernel's stores. So a chained kernel takes none of them: its read pointers carry no
// __restrict__ (the pointers it writes through do, which is all that overlapping the loads needs), and it reads with
//   ld_plain    an ordinary load, ordered behind chain_wait() by its memory clobber
//   ld_l2       past L1: data that is read once and should leave L1 to the weights
//   ld_stream   evict first: data that nobody reads again
//   ld_readonly the read-only path after all, in kernels that are never launched as dependents but in plain stream order. Used
//               where the compiler's freedom to move such loads was measured to pay.
template <typename T>
__device__ __forceinline__ T ld_plain(const T* p) { return *p; }
template <typename T>
__device__ __forceinline__ T ld_readonly(const T* p) { return __ldg(p); }
__device__ __forceinline__ uint2 ld_l2(const uint2* p) {
  uint2 v;
  asm volatile("ld.global.cg.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ uint4 ld_l2(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ float ld_stream(const float* p) {
  float v;
  asm volatile("ld.global.cs.f32 %0, [%1];" : "=f"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}

// A grid, and whether it may be launched as a dependent (the kernel is written for it either way).
struct ChainGrid {
  dim3 grid;
  bool chain = true;
  ChainGrid(dim3 d) : grid(d) {}
  ChainGrid(unsigned x, bool may_chain = true) : grid(x), chain(may_chain) {}
};

template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kernel)(Params...), ChainGrid where, dim3 block, size_t smem, cudaStream_t s, unsigned cluster,
                           Args... args) {
  const dim3 grid = where.grid;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (where.chain && (long)grid.x * grid.y * grid.z * (long)(block.x * block.y * block.z) <= kChainThreads) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 0) {   // 0: none, or the kernel's own __cluster_dims__
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = cluster;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// Raises the kernel's limit of dynamic shared memory on the current device to at least `bytes`; a call into the runtime only
// when it grows. What every kernel may have anyway (48 KB less its static arrays, which are below 16 KB everywhere) is not looked up.
template <auto Kernel>
cudaError_t allow_smem(size_t bytes) {
  if (bytes <= 32 * 1024) return cudaSuccess;
  constexpr int kDevices = 64;
  static std::atomic<int> have[kDevices];
  static std::mutex mutex;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool known = dev >= 0 && dev < kDevices;
  if (known && have[dev].load(std::memory_order_acquire) >= (int)bytes) return cudaSuccess;
  const std::lock_guard<std::mutex> lock(mutex);
  if (known && have[dev].load(std::memory_order_relaxed) >= (int)bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess && known) have[dev].store((int)bytes, std::memory_order_release);
  return e;
}

}  // namespace snntc

// What the walk kernels share: the reference's fire comparisons, the causal-set size, two-lane FP32 arithmetic.
#pragma once
#include "snntc_common.cuh"

namespace snntc {

// "ysum/wsum > c" without a division, as the reference evaluates it after consuming input c
// (snntc/snnfc_kernels.cu.cc:53-55)
__device__ __forceinline__ bool ratio_gt(float ysum, float wsum, float c) {
  const float wa = fabsf(wsum);
  const float ya = wsum < 0.f ? -ysum : ysum;
  return ya > c * wa;
}
// "ysum/wsum <= c" (snntc/snnfc_kernels.cu.cc:46-48)
__device__ __forceinline__ bool ratio_le(float ysum, float wsum, float c) {
  const float wa = fabsf(wsum);
  const float ya = wsum < 0.f ? -ysum : ysum;
  return ya <= c * wa;
}

// Number of list entries whose input value lies strictly below y: the causal-set size of an output that fired
// at y (every consumed input is below the spike value, every other one is not). Binary search, one thread.
__device__ __forceinline__ int entries_below(const WalkEntry* ents, int n, float y) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__uint_as_float(ld_l2(ents + mid).x) < y) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// sm_100 has two-lane FP32 add / sub / fma on 64-bit register pairs: one issue slot, two results, each rounded exactly
// like the scalar instruction. Low word = first lane.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void unpack2i(uint64_t v, int& lo, int& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}


}  // namespace snntc

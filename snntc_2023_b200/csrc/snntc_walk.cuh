// What the walk kernels share: the reference's fire comparisons, the causal-set size, the integer minimum of a step's sign test.
#pragma once
#include "snntc_common.cuh"
#include "snntc_ptx.cuh"

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

// Smallest of three float bit patterns compared as signed integers. For the sign test of the walks that is all that is needed:
// the result is <= 0 exactly when one of the floats is negative, -0 or +0 (negative floats are negative integers, +0 is 0,
// positive floats and NaN patterns with a clear sign bit are positive integers).
__device__ __forceinline__ int imin3(int a, int b, int c) { return min(min(a, b), c); }

}  // namespace snntc

// The walks' bound on the weight sums, formed by the first CTAs of the kernel that builds the lists.
#pragma once
#include "snntc_common.cuh"

namespace snntc {

// bound[cta] = sum over the weight rows of this CTA's warps of max_j |w_ij|: summed over the CTAs an upper bound on every column's sum
// of magnitudes. `padded` (may be null) receives the weights with rows of Jp >= J floats, zeros behind column J.
// A launch of its own in front of the lists, 4 to 5 us, was 4 % of a small layer (784 -> 400 trained at 256 samples 106 us); beside
// the lists it costs nothing that can be measured while a CTA has no more than 32 rows or 8192 weights (401 rows of 10 weights by one CTA
// of four warps, a row after the other: 40 us).
__device__ __forceinline__ void weight_bound(const WeightBound& b, int cta) {
  __shared__ float part[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const bool v4 = b.padded == nullptr && (b.J & 3) == 0 && (reinterpret_cast<uintptr_t>(b.w) & 15) == 0;
  float acc = 0.f;                                     // sum of the row maxima of this warp's rows
  for (int r = cta * warps + warp; r < b.rows; r += b.ctas * warps) {
    const float* wr = b.w + (size_t)r * b.J;
    float m = 0.f;
    if (v4) {
#pragma unroll 4
      for (int j = 4 * lane; j < b.J; j += 128) {
        const float4 v = ld_plain(reinterpret_cast<const float4*>(wr + j));
        m = fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
      }
    } else {
#pragma unroll 4
      for (int j = lane; j < b.Jp; j += 32) {
        const float v = j < b.J ? ld_plain(wr + j) : 0.f;
        m = fmaxf(m, fabsf(v));
        if (b.padded != nullptr) b.padded[(size_t)r * b.Jp + j] = v;
      }
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
    acc += m;
  }
  if (lane == 0) part[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int k = 0; k < warps; ++k) t += part[k];
    b.bound[cta] = t;
  }
}

}  // namespace snntc

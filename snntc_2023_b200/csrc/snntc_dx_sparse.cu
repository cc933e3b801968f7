// Input gradient of SnnCvGrad (snntc/snncvgrad_kernels.cu.cc:15-84) over the outputs that carry a gradient only.
//
//   dX[p,c] = sum over taps t, outputs j of  [x_pc <= y_oj] u_oj W[(t,c),j],   o = the receptive field that sees
//             input pixel p through tap t,  u_oj = grad_oj / (sum w - theta), 0 wherever (o,j) did not fire.
//
// In a network u is sparse twice over: 50-65 % of the outputs of a layer do not fire, and a pooling layer behind
// the convolution sends the gradient to one input of each window only. On the layers in front of a 2x2 pooling
// nine of ten u are exactly zero. The dense register-tile kernel (snn_dx_wide_kernel) multiplies through all of
// them. Here
//   1. snn_act_lists_kernel compacts, per receptive field, the outputs with u != 0 into a list (y, u, j), j ascending;
//   2. snn_weight_transpose_kernel lays the weights out as Wt[tap][j][c], so that the C weights one list entry needs
//      for one tap are contiguous;
//   3. snn_dx_sparse_kernel keeps an input pixel's channels in registers (CPL per lane, C / CPL lanes per pixel),
//      gathers the lists of the receptive fields that cover the pixel, tap by tap, into shared memory and walks them:
//      per entry one broadcast shared-memory read, 16-byte weight reads and a compare + predicated FMA per channel.
//      Pixel-stationary as the dense kernel: no atomics (the reference scatters with atomicAdd,
//      snncvgrad_kernels.cu.cc:83).
// The terms of a sum are added in the same order as in the dense kernel (tap-major, j ascending; the skipped ones
// are +-0), so the two kernels give the same bits.
#include "snntc_common.cuh"
#include "snntc_ptx.cuh"

#include <math_constants.h>

namespace snntc {

namespace {

constexpr int kThreads = 256;

// One warp per receptive field r: list[r*J ..] receives (y bits, u bits, j, 0) for every output with u != 0, in
// ascending j; count[r] their number.
__global__ void __launch_bounds__(kThreads)
snn_act_lists_kernel(const float* out, const float* uv, int R, int J,
                     uint4* __restrict__ list, int* __restrict__ count, const DxGate gate) {
  chain_wait();
  chain_next();
  if (gate.nz != nullptr && ld_plain(gate.nz) > gate.threshold) return;   // the dense kernel takes this call
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < R; r += warps) {
    const float* yr = out + (size_t)r * J;
    const float* ur = uv + (size_t)r * J;
    uint4* dst = list + (size_t)r * J;
    int n = 0;
    float y_next = 0.f, u_next = 0.f;     // read in front of the stores of the outputs before: no load waits behind a store
    if (lane < J) { y_next = ld_plain(yr + lane); u_next = ld_plain(ur + lane); }
    for (int j0 = 0; j0 < J; j0 += 32) {
      const int j = j0 + lane;
      const float y = y_next, u = j < J ? u_next : 0.f;
      if (j + 32 < J) { y_next = ld_plain(yr + j + 32); u_next = ld_plain(ur + j + 32); }
      const bool keep = u != 0.f;
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) dst[n + __popc(m & ((1u << lane) - 1u))] = make_uint4(__float_as_uint(y), __float_as_uint(u), (unsigned)j, 0u);
      n += __popc(m);
    }
    if (lane == 0) count[r] = n;
  }
}

// Wt[(tap*J + j)*C + c] = W[(tap*C + c)*J + j]  (the bias row is not part of dX)
__global__ void snn_weight_transpose_kernel(const float* w, float* __restrict__ wt, int taps, int C, int J,
                                            const DxGate gate) {
  chain_wait();
  chain_next();
  if (gate.nz != nullptr && ld_plain(gate.nz) > gate.threshold) return;
  const size_t n = (size_t)taps * C * J;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    const int c = (int)(e % C);
    const size_t tj = e / C;
    const int j = (int)(tj % J);
    const int tap = (int)(tj / J);
    wt[e] = ld_plain(w + ((size_t)tap * C + c) * J + j);
  }
}

// CPL channels per lane (4, 8 or 16), LPP lanes per pixel (a power of two, LPP * CPL >= C): a warp holds
// PPW = 32 / LPP input pixels at a time.
//
// The lists a pixel needs (one per tap that an output reads it through) are first copied into shared memory by
// the pixel's own lanes, back to back and with the tap folded into the entry (its third word becomes the element
// offset of weight row (tap, j) in Wt), kStage / PPW entries per pixel and round. A lane looks up one tap, a scan over the lanes
// gives where each tap's entries lie in the sequence, and every lane finds the taps of its entries by bisection: two round
// trips to the L2 per round instead of two per tap. The arithmetic then runs over that flat sequence, whose last group is filled
// up with entries that add nothing: one broadcast shared-memory read per entry, UN weight rows in flight.
// What bounds it: the L1 cache, which hands every weight to a single FMA, and instruction issue (a compare at half rate and a
// predicated FMA per channel are 8 of 13 instructions per entry at CPL = 4).
// Measured (B200, the whole dX, with a lookup per tap, entries masked one by one and 64-bit weight pointers -> now): 256 images of
// 32x32, 64 -> 64 channels, 13 % of the outputs with a gradient 543 -> 449 us; 16x16, 64 -> 128, 36 %: 493 -> 467; 37 of 45x39, 20 ->
// 52, 5x5 stride 2: 115 -> 73; 16 of 8x8, 256 -> 256: 83 -> 70. Eight entries in flight at CPL = 4: the last but one 76, a small layer of
// 128 -> 256 72 instead of 77.
constexpr int kStage = 256;   // staged list entries per warp and round

// ONE: a 1x1 window, where there is nothing to look up between the taps (201 images of 23x33, 256 -> 16: 219 us without, 176 so).
template <int CPL, int LPP, bool ONE>
__global__ void __launch_bounds__(kThreads)
snn_dx_sparse_kernel(const Geometry g, const float* x, const float* wt,
                     const uint4* list, const int* count, float* __restrict__ dx,
                     const DxGate gate) {
  chain_wait();
  chain_next();
  if (gate.nz != nullptr && ld_plain(gate.nz) > gate.threshold) return;
  constexpr int PPW = 32 / LPP;                       // pixels per warp
  constexpr int SB = kStage / PPW;                    // staged entries per pixel and round
  constexpr int UN = CPL <= 8 && !(ONE && CPL == 8) ? 4 : 2;   // entries whose weight reads are in flight together
  static_assert(SB % (4 * LPP) == 0 && LPP % UN == 0, "groups of entries are staged whole");
  __shared__ uint4 stage_all[(kThreads / 32) * kStage];
  const int lane = threadIdx.x & 31;
  const int sub = lane / LPP;                         // which of the warp's pixels
  const int gl = lane % LPP;                          // lane within the pixel's group
  const int c0 = gl * CPL;                            // first channel of this lane
  uint4* stage = stage_all + (threadIdx.x >> 5) * kStage + sub * SB;
  const int C = g.C, J = g.J;
  const int P = g.B * g.H * g.W;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const int taps = ONE ? 1 : g.Kh * g.Kw;
  // C % 4 == 0 and CPL % 4 == 0: a lane's float4s are all in or all out; one that is out reads the row's first channels, for inputs of
  // +inf that no output reaches
  unsigned coff[CPL / 4];
#pragma unroll
  for (int k = 0; k < CPL / 4; ++k) coff[k] = c0 + 4 * k < C ? (unsigned)(c0 + 4 * k) : 0u;
  const char* wbytes = reinterpret_cast<const char*>(wt);
  for (int pw = __shfl_sync(0xffffffffu, (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), 0); pw * PPW < P; pw += warps) {
    const int p = pw * PPW + sub;
    const bool pix_ok = p < P;
    float xr[CPL], acc[CPL];
#pragma unroll
    for (int k = 0; k < CPL; ++k) { xr[k] = CUDART_INF_F; acc[k] = 0.f; }
    if (pix_ok) {
#pragma unroll
      for (int k4 = 0; k4 < CPL; k4 += 4) {
        if (c0 + k4 < C) {
          const float4 v = ld_plain(reinterpret_cast<const float4*>(x + (size_t)p * C + c0 + k4));
          xr[k4] = v.x; xr[k4 + 1] = v.y; xr[k4 + 2] = v.z; xr[k4 + 3] = v.w;
        }
      }
    }
    int ph = 0, pwid = 0, pb = 0;
    if (pix_ok) {
      pwid = p % g.W;
      const int t = p / g.W;
      ph = t % g.H;
      pb = t / g.H;
    }
    for (int tap0 = 0; tap0 < taps; tap0 += LPP) {    // (the terms keep their order: tap-major, j ascending)
      // ---- this lane's tap: the receptive field that reads the pixel through (kh, kw), if there is one
      int n = 0, r = 0;
      const int tap = ONE ? 0 : tap0 + gl;
      {
        const int kh = tap / g.Kw, kw = tap - kh * g.Kw;
        const int hh = ph + g.pad_top - kh, ww = pwid + g.pad_left - kw;
        int nh = hh, nw = ww;
        bool ok = pix_ok && tap < taps && hh >= 0 && ww >= 0;
        if (g.Sh != 1 || g.Sw != 1) {
          nh = hh / g.Sh; nw = ww / g.Sw;
          ok = ok && nh * g.Sh == hh && nw * g.Sw == ww;
        }
        if (ok && nh < g.Nh && nw < g.Nw) {
          r = (pb * g.Nh + nh) * g.Nw + nw;
          n = ld_plain(count + r);
        }
      }
      int end = n;                                    // entries up to and with this lane's tap
      if constexpr (!ONE) {
#pragma unroll
        for (int d = 1; d < LPP; d <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, end, d, LPP);
          if (gl >= d) end += v;
        }
      }
      const int total = ONE ? n : __shfl_sync(0xffffffffu, end, LPP - 1, LPP);
      const int most = __reduce_max_sync(0xffffffffu, total);
      for (int first = 0; first < most; first += SB) {
        const int nmax = min(most - first, SB);
        // ---- stage entries first .. first + nmax - 1 of this pixel
        if constexpr (ONE) {
          constexpr int Q = LPP >= 16 ? 1 : 4;
#pragma unroll 1
          for (int i = 0; i < nmax; i += Q * LPP) {
            uint4 en[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
              const int e = first + i + q * LPP + gl;
              en[q] = make_uint4(0xff800000u, 0u, 0u, 0u);
              if (e < total) en[q] = ld_plain(list + (size_t)r * J + e);
            }
#pragma unroll
            for (int q = 0; q < Q; ++q) {
              en[q].z *= (unsigned)C;
              stage[i + q * LPP + gl] = en[q];
            }
          }
        } else {
#pragma unroll 1
          for (int i = 0; i < nmax; i += 4 * LPP) {
            uint4 en[4];
            unsigned at[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int e = first + i + q * LPP + gl;
              int t = 0;                                // taps whose entries all lie in front of e
#pragma unroll
              for (int d = LPP / 2; d >= 1; d >>= 1)
                if (__shfl_sync(0xffffffffu, end, t + d - 1, LPP) <= e) t += d;
              const int start = __shfl_sync(0xffffffffu, end - n, t, LPP), row = __shfl_sync(0xffffffffu, r, t, LPP);
              at[q] = (unsigned)(tap0 + t) * (unsigned)J;
              en[q] = make_uint4(0xff800000u, 0u, 0u, 0u);   // behind the end: y = -inf, u = 0
              if (e < total) en[q] = ld_plain(list + (size_t)row * J + (e - start));
              else at[q] = 0u;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int e = i + q * LPP + gl;
              en[q].z = (at[q] + en[q].z) * (unsigned)C;
              stage[e] = en[q];
            }
          }
        }
        __syncwarp();
        // ---- the arithmetic over the staged entries
#pragma unroll 1
        for (int e = 0; e < nmax; e += UN) {
          uint4 en[UN];
          float4 w4[UN][CPL / 4];
#pragma unroll
          for (int q = 0; q < UN; ++q) en[q] = stage[e + q];
#pragma unroll
          for (int q = 0; q < UN; ++q) {
#pragma unroll
            for (int k = 0; k < CPL / 4; ++k)
              w4[q][k] = ld_readonly(reinterpret_cast<const float4*>(wbytes + (size_t)(en[q].z + coff[k]) * 4u));
          }
#pragma unroll
          for (int q = 0; q < UN; ++q) {
            const float y = __uint_as_float(en[q].x), u = __uint_as_float(en[q].y);
#pragma unroll
            for (int k4 = 0; k4 < CPL; k4 += 4) {
              masked_fma(acc[k4], xr[k4], y, u, w4[q][k4 / 4].x);
              masked_fma(acc[k4 + 1], xr[k4 + 1], y, u, w4[q][k4 / 4].y);
              masked_fma(acc[k4 + 2], xr[k4 + 2], y, u, w4[q][k4 / 4].z);
              masked_fma(acc[k4 + 3], xr[k4 + 3], y, u, w4[q][k4 / 4].w);
            }
          }
        }
        __syncwarp();   // the buffer is rewritten by the next round
      }
    }
    if (pix_ok) {
#pragma unroll
      for (int k4 = 0; k4 < CPL; k4 += 4)
        if (c0 + k4 < C)
          *reinterpret_cast<float4*>(dx + (size_t)p * C + c0 + k4) = make_float4(acc[k4], acc[k4 + 1], acc[k4 + 2], acc[k4 + 3]);
    }
  }
}

size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }

template <int CPL, int LPP>
int launch_one(const Geometry& g, const float* x, const float* wt, const uint4* list, const int* count, float* dx,
               DxGate gate, const LaunchInfo& li, cudaStream_t s) {
  const long P = (long)g.B * g.H * g.W;
  const long warps = (P + (32 / LPP) - 1) / (32 / LPP);
  long grid = (warps + (kThreads / 32) - 1) / (kThreads / 32);
  const long cap = (long)li.num_sms * 16;
  if (grid > cap) grid = cap;
  // (in plain order: the transposed weights are read through the read-only path -- 256 channels: 64 us so, 90 with ordinary loads;
  // 512: 246 and 268)
  if (g.Kh * g.Kw == 1) snn_dx_sparse_kernel<CPL, LPP, true><<<(int)grid, kThreads, 0, s>>>(g, x, wt, list, count, dx, gate);
  else snn_dx_sparse_kernel<CPL, LPP, false><<<(int)grid, kThreads, 0, s>>>(g, x, wt, list, count, dx, gate);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? OK : E_CUDA;
}

}  // namespace

bool dx_sparse_shape_ok(const Geometry& g) {
  return g.is_conv && (g.C & 3) == 0 && g.C >= 16 && g.C <= 512;
}

bool dx_sparse_supported(const Geometry& g, const float* x, const float* dx) {
  if (!dx_sparse_shape_ok(g)) return false;
  return (((uintptr_t)x | (uintptr_t)dx) & 15) == 0;
}

// scratch: the lists (R*J entries of 16 bytes), their lengths, the transposed weights (fan-in x J; a workspace
// query knows the fan-in only as the number of weight rows, bias row included, which is an upper bound)
size_t dx_sparse_bytes(const Geometry& g) {
  return align256((size_t)g.R * g.J * sizeof(uint4)) + align256((size_t)g.R * sizeof(int)) +
         align256((size_t)g.I * g.J * sizeof(float));
}

int launch_dx_sparse(const Geometry& g, const float* uv, const float* x, const float* w, const float* out, float* dx,
                     void* scratch, DxGate gate, const LaunchInfo& li, cudaStream_t s) {
  unsigned char* base = static_cast<unsigned char*>(scratch);
  uint4* list = reinterpret_cast<uint4*>(base);
  int* count = reinterpret_cast<int*>(base + align256((size_t)g.R * g.J * sizeof(uint4)));
  float* wt = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(count) + align256((size_t)g.R * sizeof(int)));

  long grid = ((long)g.R + (kThreads / 32) - 1) / (kThreads / 32);
  if (grid > (long)li.num_sms * 16) grid = (long)li.num_sms * 16;
  (void)launch_chained(snn_act_lists_kernel, (int)grid, kThreads, 0, s, 0, out, uv, g.R, g.J, list, count, gate);
  count_launch();
  if (cudaGetLastError() != cudaSuccess) return E_CUDA;
  const size_t nw = (size_t)g.Kh * g.Kw * g.C * g.J;
  long tg = (long)((nw + 255) / 256);
  if (tg > (long)li.num_sms * 8) tg = (long)li.num_sms * 8;
  (void)launch_chained(snn_weight_transpose_kernel, (int)tg, 256, 0, s, 0, w, wt, g.Kh * g.Kw, g.C, g.J, gate);
  count_launch();
  if (cudaGetLastError() != cudaSuccess) return E_CUDA;

  const int C = g.C;
  if (C <= 16) return launch_one<4, 4>(g, x, wt, list, count, dx, gate, li, s);
  if (C <= 32) return launch_one<4, 8>(g, x, wt, list, count, dx, gate, li, s);
  if (C <= 64) return launch_one<4, 16>(g, x, wt, list, count, dx, gate, li, s);
  if (C <= 128) return launch_one<4, 32>(g, x, wt, list, count, dx, gate, li, s);
  if (C <= 256) return launch_one<8, 32>(g, x, wt, list, count, dx, gate, li, s);
  return launch_one<16, 32>(g, x, wt, list, count, dx, gate, li, s);
}

}  // namespace snntc

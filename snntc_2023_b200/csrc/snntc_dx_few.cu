// Input gradient of a convolution on few channels (SnnCvGrad, snntc/snncvgrad_kernels.cu.cc:15-84), up to 15 of them.
//
//   dX[p,c] = sum over receptive fields o that contain pixel p, outputs j of  [x_pc <= y_oj] u_oj W[(tap,c),j]
//
// The register-tile kernel (snn_dx_wide_kernel) works on 64 channels at a time and on every tap whatever the stride: with 3
// channels and a 7x7 window at stride 2 that is 85 products formed for each one wanted, and a small image leaves most of the GPU
// idle besides. Here a warp takes one pixel, its lanes the outputs j (coalesced reads of y, u and of the weight rows), and the
// channels' sums sit in registers: per receptive field and 32 outputs two loads, then a load, a compare and a predicated FMA
// per channel. Only the fields that really contain the pixel are visited. The lanes' sums are added by shuffles at the end, in a
// fixed order: the same bits every run.
// Where the fan-out is a multiple of four a lane takes four outputs at a time, 16 bytes to a load, and narrow fan-outs leave room
// for several fields at once: a quarter of the load instructions, which bound the version with one output per lane and load.
// What bounds it: instruction issue and the L1 reads of the weights; 30 184 pixels x 3 channels, 7x7 stride 2, 128 outputs: 1517 us
// by the register tiles, 89 with one output per load, 62 with four; 200 704 pixels, 64 outputs: 3914, 439, 234; 65 536 x 8
// channels, 3x3, 64 outputs: 291, 187, 140.
#include "snntc_common.cuh"
#include "snntc_ptx.cuh"

namespace snntc {

namespace {

constexpr int kThreads = 256;

// CT: channels held per lane. V4: a lane takes four outputs at a time by 16-byte loads (J a multiple of 4, y, u and w aligned);
// `lanes` = 4, 8, 16 or 32 of them take a field, 32 / lanes fields at once.
template <int CT, bool V4>
__global__ void __launch_bounds__(kThreads)
snn_dx_few_kernel(const Geometry g, const float* uv, const float* x, const float* w,
                  const float* y, float* __restrict__ dx, int lanes) {
  chain_wait();
  chain_next();
  const int lane = threadIdx.x & 31;
  const int C = g.C, J = g.J;
  const int c0 = blockIdx.y * CT;                // this block's channels c0 .. c0 + CT - 1
  const int P = g.B * g.H * g.W;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < P; p += warps) {
    const int pw = p % g.W, t = p / g.W;
    const int ph = t % g.H + g.pad_top, b = t / g.H, pl = pw + g.pad_left;
    float xr[CT], acc[CT];
#pragma unroll
    for (int c = 0; c < CT; ++c) {
      xr[c] = c0 + c < C ? ld_plain(x + (size_t)p * C + c0 + c) : 0.f;
      acc[c] = 0.f;
    }
    // fields nh with nh*Sh <= ph <= nh*Sh + Kh - 1
    const int nh1 = min(ph / g.Sh, g.Nh - 1), nw1 = min(pl / g.Sw, g.Nw - 1);
    const int nh0 = ph < g.Kh ? 0 : (ph - g.Kh) / g.Sh + 1, nw0 = pl < g.Kw ? 0 : (pl - g.Kw) / g.Sw + 1;
    if constexpr (V4) {
      const int cols = nw1 - nw0 + 1, fields = max(0, nh1 - nh0 + 1) * max(0, cols);
      const int step = 32 / lanes;
      int nh = nh0, nw = nw0 + lane / lanes;
      for (int f = lane / lanes; f < fields; f += step, nw += step) {
        while (nw > nw1) { nw -= cols; ++nh; }
        const int kh = ph - nh * g.Sh, kw = pl - nw * g.Sw;
        const size_t o = ((size_t)(b * g.Nh + nh) * g.Nw + nw) * J;
        const float* wt = w + ((size_t)(kh * g.Kw + kw) * C + c0) * J;
#pragma unroll 2
        for (int j = 4 * (lane & (lanes - 1)); j < J; j += 4 * lanes) {
          const float4 yy = ld_plain(reinterpret_cast<const float4*>(y + o + j));
          const float4 u = ld_plain(reinterpret_cast<const float4*>(uv + o + j));
#pragma unroll
          for (int c = 0; c < CT; ++c) {
            if (c0 + c >= C) break;
            const float4 wv = ld_plain(reinterpret_cast<const float4*>(wt + (size_t)c * J + j));
            masked_fma(acc[c], xr[c], yy.x, u.x, wv.x);
            masked_fma(acc[c], xr[c], yy.y, u.y, wv.y);
            masked_fma(acc[c], xr[c], yy.z, u.z, wv.z);
            masked_fma(acc[c], xr[c], yy.w, u.w, wv.w);
          }
        }
      }
      __syncwarp();
    } else {
      for (int nh = nh0; nh <= nh1; ++nh) {
        for (int nw = nw0; nw <= nw1; ++nw) {
          const int kh = ph - nh * g.Sh, kw = pl - nw * g.Sw;
          const size_t o = ((size_t)(b * g.Nh + nh) * g.Nw + nw) * J;
          const float* wt = w + ((size_t)(kh * g.Kw + kw) * C + c0) * J;
#pragma unroll 2
          for (int j = lane; j < J; j += 32) {
            const float yy = ld_plain(y + o + j), u = ld_plain(uv + o + j);
#pragma unroll
            for (int c = 0; c < CT; ++c)
              if (c0 + c < C) masked_fma(acc[c], xr[c], yy, u, ld_plain(wt + (size_t)c * J + j));
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < CT; ++c) {
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], d);
      if (c0 + c < C && lane == c) dx[(size_t)p * C + c0 + c] = acc[c];
    }
  }
}

template <int CT>
int launch(const Geometry& g, const float* uv, const float* x, const float* w, const float* y, float* dx, const LaunchInfo& li,
           cudaStream_t s) {
  const long P = (long)g.B * g.H * g.W;
  long grid = (P + kThreads / 32 - 1) / (kThreads / 32);
  if (grid > 16L * li.num_sms) grid = 16L * li.num_sms;
  const bool v4 = (g.J & 3) == 0 && (((uintptr_t)uv | (uintptr_t)w | (uintptr_t)y) & 15) == 0;
  const int lanes = g.J > 64 ? 32 : (g.J > 32 ? 16 : (g.J > 16 ? 8 : 4));
  const dim3 grid2((unsigned)grid, (g.C + CT - 1) / CT);
  const cudaError_t e = v4 ? launch_chained(snn_dx_few_kernel<CT, true>, grid2, kThreads, 0, s, 0, g, uv, x, w, y, dx, lanes)
                           : launch_chained(snn_dx_few_kernel<CT, false>, grid2, kThreads, 0, s, 0, g, uv, x, w, y, dx, lanes);
  count_launch();
  return e == cudaSuccess ? OK : E_CUDA;
}

}  // namespace

int launch_dx_few(const Geometry& g, const float* uv, const float* x, const float* w, const float* y, float* dx,
                  const LaunchInfo& li, cudaStream_t s) {
  if (g.C == 1) return launch<1>(g, uv, x, w, y, dx, li, s);
  if (g.C == 3) return launch<3>(g, uv, x, w, y, dx, li, s);
  if (g.C <= 4) return launch<4>(g, uv, x, w, y, dx, li, s);
  return launch<8>(g, uv, x, w, y, dx, li, s);          // (more than eight channels: blocks of eight)
}

}  // namespace snntc

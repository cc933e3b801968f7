// Weight gradient of SnnCvGrad (snntc/snncvgrad_kernels.cu.cc:87-161) that skips the outputs that did not fire.
//
//   dW[i,j] = sum_r [x_ri <= y_rj] (x_ri - y_rj) u_rj,   u_rj = 0 wherever output (r,j) did not fire.
//
// In the networks this library is built for, 50-65 % of the outputs of a layer do not fire, and an output
// channel that rarely fires does so for almost every receptive field. The dense register-tile kernel
// (snn_dw_kernel) multiplies through all of them. Here a warp owns FOUR output channels and every lane 4*QL
// fan-in rows, so "did (r,j) fire" is the same question for all 32 lanes: a warp-uniform branch skips the
// whole row of the tile for that channel, and the inputs of row r are not even read from shared memory when
// none of the warp's four channels fired. What is left costs what the dense kernel costs per element: one
// saturating FMA (the clamp [x<=y](y-x) as the saturation of (y-x)*s, s a power of two, see snn_dw_kernel)
// and half a two-lane FMA.
//
// CTA: 16 warps = 64 output channels (or 8 = 32); 128*QL fan-in rows; blockIdx.z takes a slice of the rows r.
// The x tile (16 rows of r at a time, four or two stages in flight) is gathered straight from the NHWC image with 16-byte
// asynchronous copies (four channels of one tap are contiguous), never passing through registers; taps outside
// the image, rows past the slice and the bias row are plain 16-byte stores of constants (NOT copies from a
// constant in global memory: every CTA fetching the same 16 bytes makes one L2 line the bottleneck of the kernel).
//
// Channel counts or fan-outs that are no multiple of four (VEC = false: the first layer of an image network, mostly) have no
// aligned groups of four to copy: there every thread owns single columns of the x tile, copied 4 bytes at a time, y and u likewise,
// and a lane holds pairs of fan-in rows instead of quadruples, so that the tile comes in steps of 64 and a narrow window does not
// pay for 128.
//
// What bounds it: the copies and the shared memory reads of x where few outputs carry a gradient, then issue. 64 outputs per CTA
// (each input copied once for twice the outputs), stages queued three ahead, one barrier a stage and one wave of CTAs against 32
// outputs, two stages, two barriers and eight waves, dW of 131 072 rows of 829 x 128: all outputs that fired 1445 -> 1213 us, 12 %
// of them 731 -> 506; 65 536 of 325 x 64 at stride 2: 201 -> 146, 135 -> 82. Without VEC, 131 072 of 820 x 128 against the dense
// tile: 2012 -> 1469, 1998 -> 734. Channels dealt out to the warps by their activity instead of four neighbours, the sums out through
// shared memory (whole dW): 200 704 of 148 x 64 284 -> 266, 3136 of 4609 x 512 354 -> 330, 1600 of 3201 x 64, 5x5 stride 2 48 -> 39.
#include "snntc_common.cuh"
#include "snntc_ptx.cuh"

#include <math_constants.h>
#include <algorithm>
#include <type_traits>

namespace snntc {

namespace {

constexpr int kRS = 16;          // rows r per stage

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gmem_src) : "memory");
}

// VEC: C and J multiples of four, 16-byte aligned tensors; a lane holds QL quadruples of fan-in rows, else QL pairs
template <int QL, bool VEC, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW)
snn_dw_skip_kernel(const Geometry g, const float* uv, const float* x,
                   const float* out, float* __restrict__ partial, int rows_per_split,
                   float scale, const int* exact_flag) {
  chain_wait();
  chain_next();
  constexpr int kThreads = 32 * NW, kJT = 4 * NW;   // output channels per CTA, 4 per warp
  constexpr int kDepth = NW == 16 ? 4 : 2;          // stages in shared memory
  constexpr int CW = VEC ? 4 : 2;      // neighbouring fan-in rows of a lane
  constexpr int kTI = 32 * CW * QL;    // fan-in rows per CTA
  constexpr int kCh = 32 * QL;         // chunks of CW per row of the x tile
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* Xs = reinterpret_cast<float*>(smem_raw);                 // [kDepth][kRS][kTI]
  float* Ys = Xs + kDepth * kRS * kTI;                            // [kDepth][kRS][kJT]
  float* Us = Ys + kDepth * kRS * kJT;                            // [kDepth][kRS][kJT]
  __shared__ __align__(16) int order[kJT];          // output channels (of this CTA) by warp, four each
  __shared__ int active[kJT];
  __shared__ float4 own_all[NW][2][kRS];            // a stage's u and y of each warp's four channels
  // float of row rl and channel c in a y or u buffer: the 16-byte chunks are swizzled by the row, so that a channel's 16 rows are read
  // two at a time instead of one after the other
  auto at_field = [](int rl, int c) { return rl * kJT + (((c >> 2) ^ (rl & 7)) << 2 | (c & 3)); };
  int4* rowinfo = reinterpret_cast<int4*>(Us + kDepth * kRS * kJT);    // [2][kRS]: .x element offset of the top-left pixel, .y its h, .z its w, .w row valid

  const int J = g.J, I = g.I, R = g.R;
  const int Itot = I + g.has_bias;
  const bool fast = scale != 1.0f && ld_plain(exact_flag) == 0;
  const float sc = fast ? scale : 1.0f;                 // s
  const float nsc = -sc;
  const float nusc = fast ? -1.0f / scale : -1.0f;      // -1/s, exact: s is a power of two

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i0 = blockIdx.y * kTI, j0 = blockIdx.x * kJT;
  const int r_begin = blockIdx.z * rows_per_split;
  const int r_end = min(R, r_begin + rows_per_split);
  // what stands in for inputs that are not there: an input that never spikes; the bias input and the padding beside it
  const float4 v_never = make_float4(g.maxv, g.maxv, g.maxv, g.maxv);
  const float4 v_bias = make_float4(g.biasvolt, g.maxv, g.maxv, g.maxv);

  // this thread's column chunk of the x tile (threads below kCh): .x element offset of its tap from a row's top-left
  // pixel, .y kh, .z kw, .w 1 = image tap, 2 = bias chunk, 0 = padding behind the last weight row
  int4 tapinfo_reg = make_int4(0, 0, 0, 0);
  // (with more threads, kXG of them own a chunk, each every kXG-th row)
  constexpr int kXG = !VEC || kCh * 2 + 64 > kThreads ? 1 : (kCh * 4 + 64 > kThreads ? 2 : 4);
  const int chunk = tid % kCh, xgroup = tid / kCh;
  if (VEC && tid < kCh * kXG) {
    const int i = i0 + 4 * chunk;
    if (i < I) {
      const int tap = i / g.C, c = i - tap * g.C;
      const int kh = tap / g.Kw, kw = tap - kh * g.Kw;
      tapinfo_reg = make_int4((kh * g.W + kw) * g.C + c, kh, kw, 1);
    } else if (i == I && g.has_bias) {
      tapinfo_reg.w = 2;
    }
  }
  auto fill_rowinfo = [&](int slot, int rb) {
    if (tid < kRS) {
      const int r = rb + tid;
      int4 ri = make_int4(0, 0, 0, 0);
      if (r < r_end) {
        const int nw = r % g.Nw;
        const int t = r / g.Nw;
        const int nh = t % g.Nh;
        const int b = t / g.Nh;
        ri.y = nh * g.Sh - g.pad_top;
        ri.z = nw * g.Sw - g.pad_left;
        ri.x = ((b * g.H + ri.y) * g.W + ri.z) * g.C;
        ri.w = 1;
      }
      rowinfo[slot * kRS + tid] = ri;
    }
  };
  // Queues the asynchronous copies of the 16 rows starting at rb into buffer `buf` (rowinfo[slot] describes them). A thread
  // t < kCh * kXG owns a column chunk of the x tile -- its tap is the same for every row and stays in registers -- and walks the
  // rows; the other threads fetch the y and u tiles (16 rows x kJT / 4 chunks each).
  static_assert(!VEC || kCh * kXG < kThreads, "some threads must be left for the y and u tiles");
  const int4 my_tap = tapinfo_reg;
  // Without VEC: this thread's columns col + kThreads*k (narrow tiles: one column, every kGroups-th row), their offsets
  // and taps; tap -1: the bias row, -2: padding
  constexpr int kCols = (kTI + kThreads - 1) / kThreads;
  constexpr int kGroups = kTI <= kThreads / 2 ? kThreads / kTI : 1;
  const int col = kGroups > 1 ? tid % kTI : tid, group = kGroups > 1 ? tid / kTI : 0;
  int col_off[kCols], col_tap[kCols];
  if constexpr (!VEC) {
#pragma unroll
    for (int k = 0; k < kCols; ++k) {
      const int i = i0 + col + k * kThreads;
      col_off[k] = 0;
      col_tap[k] = i == I && g.has_bias ? -1 : -2;
      if (i < I) {
        const int tap = i / g.C, c = i - tap * g.C;
        const int kh = tap / g.Kw, kw = tap - kh * g.Kw;
        col_off[k] = (kh * g.W + kw) * g.C + c;
        col_tap[k] = kh << 16 | kw;
      }
    }
  }
  auto issue = [&](int buf, int slot, int rb) {
    if constexpr (!VEC) {
#pragma unroll 4
      for (int rl = group < kGroups ? group : kRS; rl < kRS; rl += kGroups) {
        const int4 ri = rowinfo[slot * kRS + rl];
#pragma unroll
        for (int k = 0; k < kCols; ++k) {
          if (col + k * kThreads >= kTI) break;
          float* dst = Xs + (buf * kRS + rl) * kTI + col + k * kThreads;
          const bool in_image = ri.w != 0 && col_tap[k] >= 0 && (unsigned)(ri.y + (col_tap[k] >> 16)) < (unsigned)g.H &&
                                (unsigned)(ri.z + (col_tap[k] & 0xffff)) < (unsigned)g.W;
          if (in_image) cp_async4(dst, x + ((ptrdiff_t)ri.x + col_off[k]));
          else *dst = ri.w != 0 && col_tap[k] == -1 ? g.biasvolt : g.maxv;
        }
      }
#pragma unroll
      for (int e = tid; e < 2 * kRS * kJT; e += kThreads) {
        const int which = e / (kRS * kJT), rl = e / kJT % kRS, jl = e % kJT;
        float* dst = (which == 0 ? Ys : Us) + buf * kRS * kJT + at_field(rl, jl);
        if (rb + rl < r_end && j0 + jl < J) cp_async4(dst, (which == 0 ? out : uv) + (size_t)(rb + rl) * J + j0 + jl);
        else *dst = 0.f;
      }
    } else if (tid < kCh * kXG) {
      float* dst = Xs + buf * kRS * kTI + 4 * chunk;
#pragma unroll
      for (int rk = 0; rk < kRS / kXG; ++rk) {
        const int rl = rk * kXG + xgroup;
        const int4 ri = rowinfo[slot * kRS + rl];   // the same word for the whole warp: a broadcast
        const bool in_image = ri.w != 0 && my_tap.w == 1 && (unsigned)(ri.y + my_tap.y) < (unsigned)g.H &&
                              (unsigned)(ri.z + my_tap.z) < (unsigned)g.W;
        if (in_image) cp_async16(dst + rl * kTI, x + ((ptrdiff_t)ri.x + my_tap.x));
        else *reinterpret_cast<float4*>(dst + rl * kTI) = (ri.w != 0 && my_tap.w == 2) ? v_bias : v_never;
      }
    } else {
      for (int e = tid - kCh * kXG; e < 2 * kRS * (kJT / 4); e += kThreads - kCh * kXG) {
        const int which = e / (kRS * (kJT / 4));            // 0: y, 1: u
        const int h = e - which * (kRS * (kJT / 4));
        const int rl = h / (kJT / 4), cq = h - rl * (kJT / 4);
        const int r = rb + rl, j = j0 + 4 * cq;
        const float* base = which == 0 ? out : uv;
        float* dst = (which == 0 ? Ys : Us) + buf * kRS * kJT + at_field(rl, 4 * cq);
        if (r < r_end && j < J) cp_async16(dst, base + (size_t)r * J + j);
        else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);   // no spike value, no gradient
      }
    }
    copies_commit();
  };

  // acc[c][jj][h]: fan-in rows i0 + CW*(lane + 32c) + 2h, +1 (one 64-bit pair), the warp's channel jj
  uint64_t acc[QL][4][CW / 2];
#pragma unroll
  for (int c = 0; c < QL; ++c)
#pragma unroll
    for (int jj = 0; jj < 4; ++jj)
#pragma unroll
      for (int h = 0; h < CW / 2; ++h) acc[c][jj][h] = pack2(0.f, 0.f);

  unsigned at01 = 0u, at23 = 0u;                  // where this lane's row of the warp's four channels lies in a buffer
  const float* const own_from = lane < kRS ? Us : Ys;
  auto reduce_stage = [&](int buf, auto fast_c) {
    constexpr bool FAST = decltype(fast_c)::value;
    const float* xs = Xs + buf * kRS * kTI;
    // The warp's four channels of the stage, a row per lane (lanes from 16 on: y), put side by side for the loop below. Which of the 16
    // rows carry a gradient for one of the four: one vote.
    float4* own = &own_all[warp][0][0];
    unsigned todo;
    {
      const float* from = own_from + buf * kRS * kJT;
      const float4 v = make_float4(from[at01 & 0xffff], from[at01 >> 16], from[at23 & 0xffff], from[at23 >> 16]);
      todo = __ballot_sync(0xffffffffu, (v.x != 0.f) | (v.y != 0.f) | (v.z != 0.f) | (v.w != 0.f)) & ((1u << kRS) - 1u);
      __syncwarp();                                        // every lane is through with the stage before (a vote orders no memory)
      if (todo != 0u) own[lane] = v;
      __syncwarp();
    }
#pragma unroll 1
    while (todo != 0u) {
      const int rl = __ffs((int)todo) - 1;
      todo &= todo - 1u;
      const float4 u4 = own[rl], y4 = own[kRS + rl];
      float xr[QL][CW];
#pragma unroll
      for (int c = 0; c < QL; ++c) {
        if constexpr (VEC) {
          const float4 v = *reinterpret_cast<const float4*>(xs + rl * kTI + 4 * (lane + 32 * c));
          xr[c][0] = v.x; xr[c][1] = v.y; xr[c][2] = v.z; xr[c][3] = v.w;
        } else {
          const float2 v = *reinterpret_cast<const float2*>(xs + rl * kTI + 2 * (lane + 32 * c));
          xr[c][0] = v.x; xr[c][1] = v.y;
        }
      }
      const float yv[4] = {y4.x, y4.y, y4.z, y4.w};
      const float uu[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        if (uu[jj] == 0.f) continue;              // warp-uniform
        const float ys = yv[jj] * sc;
        const float nu = uu[jj] * nusc;
        const uint64_t nu2 = pack2(nu, nu);
#pragma unroll
        for (int c = 0; c < QL; ++c) {
          float t[CW];
#pragma unroll
          for (int k = 0; k < CW; ++k) t[k] = FAST ? fma_sat(xr[c][k], nsc, ys) : fmaxf(ys - xr[c][k], 0.f);
#pragma unroll
          for (int h = 0; h < CW / 2; ++h) acc[c][jj][h] = fma2(pack2(t[2 * h], t[2 * h + 1]), nu2, acc[c][jj][h]);
        }
      }
    }
  };

  // Stage `it` + kDepth - 1 is queued while stage `it` is worked on; one barrier per stage, behind which that stage's copies are
  // there for everyone and everyone is through with the buffer that is refilled.
  for (int d = 0; d < kDepth - 1; ++d) {
    fill_rowinfo(d & 1, r_begin + d * kRS);
    __syncthreads();
    issue(d, d & 1, r_begin + d * kRS);        // (rows from r_end on: an empty stage)
  }
  fill_rowinfo((kDepth - 1) & 1, r_begin + (kDepth - 1) * kRS);
  // Which four channels a warp takes: dealt out in the order of their activity over the stages that are there first, forth and back
  // (see snn_dw_tma_kernel)
  copies_wait<0>();
  __syncthreads();
  if (tid < kJT) {
    int n = 0;
    for (int d = 0; d < kDepth - 1; ++d)
#pragma unroll
      for (int rl = 0; rl < kRS; ++rl) n += Us[d * kRS * kJT + at_field(rl, tid)] != 0.f;
    active[tid] = n;
  }
  __syncthreads();
  if (tid < kJT) {
    const int n = active[tid];
    int rank = 0;
#pragma unroll 8
    for (int c = 0; c < kJT; ++c) rank += active[c] > n || (active[c] == n && c < tid);
    const int k = rank / NW, w = rank % NW;
    order[4 * (k & 1 ? NW - 1 - w : w) + k] = tid;
  }
  __syncthreads();
  {
    const int4 ch = *reinterpret_cast<const int4*>(order + 4 * warp);
    const int rl = lane & (kRS - 1);
    at01 = (unsigned)at_field(rl, ch.x) | (unsigned)at_field(rl, ch.y) << 16;
    at23 = (unsigned)at_field(rl, ch.z) | (unsigned)at_field(rl, ch.w) << 16;
  }
  int it = 0;
  for (int rb = r_begin; rb < r_end; rb += kRS, ++it) {
    copies_wait<kDepth - 2>();
    __syncthreads();
    issue((it + kDepth - 1) % kDepth, (it + kDepth - 1) & 1, rb + (kDepth - 1) * kRS);
    fill_rowinfo((it + kDepth) & 1, rb + kDepth * kRS);
    if (fast) reduce_stage(it % kDepth, std::true_type{});
    else reduce_stage(it % kDepth, std::false_type{});
  }
  copies_wait<0>();

  // The sums go out through shared memory, where they are turned so that a row's channels lie together: row (f % CW, f / CW) for fan-in
  // row f of the tile, lanes on neighbouring rows.
  __syncthreads();
  constexpr int kPitch = kJT + 1;
  static_assert((size_t)kTI * kPitch <= (size_t)kDepth * kRS * (kTI + 2 * kJT), "the tile of sums fits the stages");
  float* turn = Xs;
  {
    const int4 ch = *reinterpret_cast<const int4*>(order + 4 * warp);
    const int chs[4] = {ch.x, ch.y, ch.z, ch.w};
#pragma unroll
    for (int c = 0; c < QL; ++c)
#pragma unroll
      for (int h = 0; h < CW / 2; ++h)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          float a, b;
          unpack2(acc[c][jj][h], a, b);
          turn[((2 * h) * 32 * QL + 32 * c + lane) * kPitch + chs[jj]] = a;
          turn[((2 * h + 1) * 32 * QL + 32 * c + lane) * kPitch + chs[jj]] = b;
        }
  }
  __syncthreads();
  float* __restrict__ dst = partial + (size_t)blockIdx.z * Itot * J;
  const int j = j0 + 4 * (tid % NW);
  if (j < J) {
    for (int f = tid / NW; f < kTI && i0 + f < Itot; f += 32) {
      const float* from = turn + ((f % CW) * 32 * QL + f / CW) * kPitch + 4 * (tid % NW);
      float* to = dst + (size_t)(i0 + f) * J + j;
      if (VEC || (J & 3) == 0) {
        *reinterpret_cast<float4*>(to) = make_float4(from[0], from[1], from[2], from[3]);
      } else {
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
          if (j + jj < J) to[jj] = from[jj];
      }
    }
  }
}

// Fan-in rows of a tile come in units of 128 (VEC) or 64.
int tile_unit(bool vec) { return vec ? 128 : 64; }
bool vec_shape(const Geometry& g) { return (g.C & 3) == 0 && (g.J & 3) == 0; }

// fan-in tiles: as few as possible with at most 640 rows each, then the narrowest tile that covers the share
void plan_tiles(int Itot, bool vec, int* ntiles, int* ql) {
  const int unit = tile_unit(vec);
  const int n = (Itot + 639) / 640;
  const int per = (Itot + n - 1) / n;
  int q = (per + unit - 1) / unit;
  if (!vec && q > 4) q = (q + 1) & ~1;   // widths that are compiled: 1 to 4, 6, 8 and 10 units of 64
  *ql = q;
  *ntiles = (Itot + unit * q - 1) / (unit * q);
}

// 64 outputs per CTA halve the copies (which bound the kernel where few outputs carry a gradient) and leave room for four
// stages; where that would leave half of a last CTA without outputs, 32 and two CTAs per SM.
int plan_warps(const Geometry& g) { return (g.J & 63) == 0 || (g.J & 63) > 32 ? 16 : 8; }

template <int QL, bool VEC, int NW>
int launch_ql(const Geometry& g, const float* uv, const float* x, const float* out, float* partial, dim3 grid,
              int rows_per_split, float scale, const int* exact_flag, cudaStream_t s) {
  const size_t tile = (size_t)tile_unit(VEC) * QL;
  const size_t smem = (NW == 16 ? 4 : 2) * kRS * (tile + 8 * NW) * sizeof(float) + 2 * kRS * sizeof(int4);
  if (allow_smem<snn_dw_skip_kernel<QL, VEC, NW>>(smem) != cudaSuccess)
    return E_CUDA;
  (void)launch_chained(snn_dw_skip_kernel<QL, VEC, NW>, grid, 32 * NW, smem, s, 0, g, uv, x, out, partial, rows_per_split, scale, exact_flag);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? OK : E_CUDA;
}

}  // namespace

bool dw_skip_supported(const Geometry& g, const float* x, const float* uv, const float* out) {
  if (!g.is_conv) return false;
  if (vec_shape(g) && (((uintptr_t)x | (uintptr_t)uv | (uintptr_t)out) & 15)) return false;
  if ((long long)g.B * g.H * g.W * g.C > 0x7fffffffLL) return false;   // element offsets are 32-bit
  return g.Kh < 32768 && g.Kw < 65536;
}

int dw_skip_splits(const Geometry& g, const LaunchInfo& li, int* rows_per_split) {
  int ntiles = 1, ql = 1;
  plan_tiles(g.I + g.has_bias, vec_shape(g), &ntiles, &ql);
  const int nw = plan_warps(g);
  const long tiles = (long)ntiles * ((g.J + 4 * nw - 1) / (4 * nw));
  long want = std::max(1L, 16L / nw * li.num_sms / tiles);   // one wave of CTAs, 512 threads per SM
  const long max_splits = ((long)g.R + kRS - 1) / kRS;
  if (want > max_splits) want = max_splits;
  if (want > 1024) want = 1024;
  if (want < 1) want = 1;
  long rps = ((long)g.R + want - 1) / want;
  rps = (rps + kRS - 1) / kRS * kRS;
  *rows_per_split = (int)rps;
  return (int)(((long)g.R + rps - 1) / rps);
}

int launch_dw_skip(const Geometry& g, const float* uv, const float* x, const float* out, float* partial,
                   int splits, int rows_per_split, float scale, const int* exact_flag,
                   cudaStream_t s) {
  int ntiles = 1, ql = 1;
  plan_tiles(g.I + g.has_bias, vec_shape(g), &ntiles, &ql);
  const int nw = plan_warps(g), jt = 4 * nw;
  dim3 grid((g.J + jt - 1) / jt, ntiles, splits);
  auto run = [&](auto launch) { return launch(g, uv, x, out, partial, grid, rows_per_split, scale, exact_flag, s); };
  auto pick = [&](auto nw_c) {
    constexpr int NW = decltype(nw_c)::value;
    if (!vec_shape(g)) {
      switch (ql) {
        case 1: return run(launch_ql<1, false, NW>);
        case 2: return run(launch_ql<2, false, NW>);
        case 3: return run(launch_ql<3, false, NW>);
        case 4: return run(launch_ql<4, false, NW>);
        case 6: return run(launch_ql<6, false, NW>);
        case 8: return run(launch_ql<8, false, NW>);
        default: return run(launch_ql<10, false, NW>);
      }
    }
    switch (ql) {
      case 1: return run(launch_ql<1, true, NW>);
      case 2: return run(launch_ql<2, true, NW>);
      case 3: return run(launch_ql<3, true, NW>);
      case 4: return run(launch_ql<4, true, NW>);
      default: return run(launch_ql<5, true, NW>);
    }
  };
  return nw == 16 ? pick(std::integral_constant<int, 16>{}) : pick(std::integral_constant<int, 8>{});
}

}  // namespace snntc

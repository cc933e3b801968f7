// Both gradients of a dense layer (SnnFcGrad, snntc/snnfcgrad_kernels.cu.cc:15-225) in one launch behind the u kernel, for
// up to a few thousand samples.
//
//   dX[r,i] = sum_j [x_ri <= y_rj] u_rj W[i,j]        dW[i,j] = sum_r [x_ri <= y_rj] (x_ri - y_rj) u_rj
//   u[r,j]  = y[r,j] fired ? grad[r,j] * inv[r,j] : 0
//
// What bounds a dense layer at these sizes is not arithmetic but how little of the GPU a call reaches: 256 samples of a
// 784 -> 400 layer are 52 tiles of 64 x 64 for dX, each reducing 400 outputs one after the other. Here
//   - the unit of work is a 32 x 32 tile of dX or dW per WARP, 32 sums per lane, and the warps of a cluster of up to eight
//     CTAs (four warps each) share out tiles AND the reduction: `split` warps take a part each of one tile's reduction
//     and are added in a fixed order through distributed shared memory, so that a layer with few tiles still gives every
//     SM work (32 samples of that layer are 25 tiles: with all of a tile's warps in one CTA, 25 SMs worked for 12 us);
//   - every warp brings its own chunks of 16 reduction steps in with 16-byte asynchronous copies, two buffers deep, as they
//     lie in memory, with no CTA barrier in the loop. dX reads four steps of a row at once (16 bytes), so nothing has to be
//     transposed; rows of 20 floats and a lane's rows 8 apart keep these reads free of bank conflicts. (4-byte copies that
//     transpose on the way took half of the kernel's instructions, register staging was bound by L1 line lookups.)
//   - dX and dW tiles are blocks of one grid: they run side by side without an auxiliary stream.
// Per element dX is a compare and a predicated FMA (bound by the half-rate compare pipe), dW a saturating FMA and half a
// two-lane FMA (the scaled form of relu(y - x), snntc_backward.cu).
// Measured (B200, batch 256, 784 -> 400, every output with a gradient): dX 67 us, dW 22 us and 9 us around them before,
// DENSE_BOTH_US us now.
#include "snntc_common.cuh"

#include <cooperative_groups.h>
#include <math_constants.h>

namespace snntc {

namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxCluster = 8;
constexpr int kT = 32;            // edge of a warp's tile
constexpr int kStep = 16;         // reduction steps per staged chunk
constexpr int kRow = kStep + 4;   // row stride of dX's staged arrays ([32 rows or inputs][16 steps])
constexpr int kTile = kT * kRow;  // floats of one staged array (dW: [16 steps][32], 512 of them)
constexpr int kPad = kT + 4;      // row stride of the tiles that are added over the split
constexpr int kWarpFloats = 2 * 3 * kTile;                              // two buffers of three arrays
constexpr size_t kSmemBytes = (size_t)kWarps * kWarpFloats * sizeof(float);
static_assert(kT * kPad <= kWarpFloats, "the reduction tile lies over the warp's own staging buffers");

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float fma_sat(float a, float b, float c) {
  float r;
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// acc += [x <= y] * u * w as one compare and one predicated FMA
__device__ __forceinline__ void masked_fma(float& acc, float x, float y, float u, float w) {
  asm("{\n\t.reg .pred p;\n\tsetp.le.f32 p, %1, %2;\n\t@p fma.rn.f32 %0, %3, %4, %0;\n\t}"
      : "+f"(acc) : "f"(x), "f"(y), "f"(u), "f"(w));
}
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// 4- and 16-byte asynchronous copies; `ok` false writes zeros and reads nothing
__device__ __forceinline__ void copy4(unsigned dst, const float* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copy16(unsigned dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct DensePlan {
  int cluster;                             // CTAs per cluster; a cluster's warps take (its warps / split) neighbouring tiles
  int dx_clusters, dx_split, dx_tiles_n;   // dX: tiles of [rows][inputs], neighbours along the inputs
  int dw_clusters, dw_split, dw_tiles_m;   // dW: tiles of [weight rows][outputs], neighbours along the weight rows
};

struct DenseArgs {
  const float* u;       // [R,J]
  const float* x;
  const float* w;
  const float* y;       // [R,J]
  float* dx;
  float* dw;
  const int* flags;     // range flags of the u kernel's blocks
  int nflags;
  int R, I, J, has_bias;
  float biasvolt, scale;   // scale: the power of two of the scaled dW loop, 1 = not usable
};

// The sums of a warp's tile (lane -> rows m + MS*k, k < ML, columns n + NS*b, b < NL) are added over the `split` warps of the
// tile in warp order, and the tile goes out in whole rows of 32 columns.
template <int ML, int NL, int MS, int NS>
__device__ __forceinline__ void write_tile(const float (&acc)[ML][NL], float* smem, int gw, int lane, int m, int n, int split,
                                           float* __restrict__ dst, int m0, int M, int n0, int N) {
  cg::cluster_group cl = cg::this_cluster();
  float* mine = smem + (gw % kWarps) * kWarpFloats;    // (this warp's own staging buffers: every copy into them has been waited for)
  __syncwarp();
#pragma unroll
  for (int k = 0; k < ML; ++k)
#pragma unroll
    for (int b = 0; b < NL; ++b) mine[(m + MS * k) * kPad + n + NS * b] = acc[k][b];
  const int part = gw % split, first = gw - part;      // the tile's warps in the cluster: first .. first + split - 1
  if (split == 1) {
    __syncwarp();
    if (n0 + lane < N)
      for (int row = 0; row < kT && m0 + row < M; ++row) dst[(size_t)(m0 + row) * N + n0 + lane] = mine[row * kPad + lane];
    return;
  }
  cl.sync();
  if (n0 + lane < N) {
    for (int row = part; row < kT && m0 + row < M; row += split) {
      float s = 0.f;
      for (int k = 0; k < split; ++k) {
        const float* tile = cl.map_shared_rank(smem, (first + k) / kWarps) + ((first + k) % kWarps) * kWarpFloats;
        s += tile[row * kPad + lane];
      }
      dst[(size_t)(m0 + row) * N + n0 + lane] = s;
    }
  }
  cl.sync();                                           // no CTA leaves while its tiles may still be read
}

// VX: I is a multiple of 4 and x 16-byte aligned; VJ: J is a multiple of 4 and u, y and w 16-byte aligned. Then every copy
// moves 16 bytes, else 4.
template <bool VX, bool VJ>
__global__ void __launch_bounds__(kThreads, 3)
snn_dense_bwd_kernel(const DenseArgs a, const DensePlan p) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  float* mine = smem + warp * kWarpFloats;
  const unsigned mine_at = smem_u32(mine);
  const int R = a.R, I = a.I, J = a.J;
  const int cluster = blockIdx.x / p.cluster;
  const int gw = (blockIdx.x - cluster * p.cluster) * kWarps + warp;    // this warp within its cluster
  const int cluster_warps = p.cluster * kWarps;

  if (cluster < p.dx_clusters) {
    // ---------------------------------------------------------------- dX tile: rows r, columns i, reduced over j
    const int tile = cluster * (cluster_warps / p.dx_split) + gw / p.dx_split;     // (a tile behind the last one has r0 >= R)
    const int r0 = tile / p.dx_tiles_n * kT, i0 = tile % p.dx_tiles_n * kT;
    const int part = gw % p.dx_split;
    const int chunks = (J + kStep - 1) / kStep;
    const int c0 = chunks * part / p.dx_split, c1 = r0 < R ? chunks * (part + 1) / p.dx_split : c0;
    auto issue = [&](int c, int buf) {
      const unsigned at = mine_at + 4u * (unsigned)(buf * 3 * kTile);
      if constexpr (VJ) {
        // lane -> steps 4*(lane & 3) .. +3 of tile rows (lane >> 2) + 8q. What does not exist copies zeros: u = 0, w = 0
        const int j = c * kStep + 4 * (lane & 3), row = lane >> 2;
        const bool jok = j < J;
        const float* gy = a.y + (size_t)(r0 + row) * J + j;
        const float* gu = a.u + (size_t)(r0 + row) * J + j;
        const float* gw = a.w + (size_t)(i0 + row) * J + j;
        const unsigned to = at + 4u * (unsigned)(row * kRow + 4 * (lane & 3));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const bool rok = jok && r0 + row + 8 * q < R, iok = jok && i0 + row + 8 * q < I;
          copy16(to + 4u * (8 * q * kRow), rok ? gy + (size_t)(8 * q) * J : a.y, rok);
          copy16(to + 4u * (8 * q * kRow + kTile), rok ? gu + (size_t)(8 * q) * J : a.u, rok);
          copy16(to + 4u * (8 * q * kRow + 2 * kTile), iok ? gw + (size_t)(8 * q) * J : a.w, iok);
        }
      } else {
        const int j = c * kStep + (lane & 15), row = lane >> 4;
        const bool jok = j < J;
#pragma unroll 4
        for (int q = 0; q < 16; ++q) {
          const int k = row + 2 * q;
          const unsigned to = at + 4u * (unsigned)(k * kRow + (lane & 15));
          const bool rok = jok && r0 + k < R, iok = jok && i0 + k < I;
          copy4(to, rok ? a.y + (size_t)(r0 + k) * J + j : a.y, rok);
          copy4(to + 4u * kTile, rok ? a.u + (size_t)(r0 + k) * J + j : a.u, rok);
          copy4(to + 8u * kTile, iok ? a.w + (size_t)(i0 + k) * J + j : a.w, iok);
        }
      }
      copies_commit();
    };
    if (c0 < c1) issue(c0, 0);
    if (c0 + 1 < c1) issue(c0 + 1, 1);
    const int m = lane >> 2, n = lane & 3;      // this lane's rows m + 8k and inputs n + 4b
    float xr[4][8], acc[4][8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float* gx = a.x + (size_t)(r0 + m + 8 * k) * I + i0 + n;
      const bool rok = r0 + m + 8 * k < R;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        xr[k][b] = (rok && i0 + n + 4 * b < I) ? __ldg(gx + 4 * b) : CUDART_INF_F;
        acc[k][b] = 0.f;
      }
    }
    for (int c = c0; c < c1; ++c) {
      const int buf = (c - c0) & 1;
      if (c + 1 < c1) copies_wait<1>(); else copies_wait<0>();
      __syncwarp();
      const float* Y = mine + buf * 3 * kTile + m * kRow;
      const float* W = mine + buf * 3 * kTile + 2 * kTile + n * kRow;
#pragma unroll
      for (int s = 0; s < kStep; s += 4) {
        float w[8][4];
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const float4 w4 = *reinterpret_cast<const float4*>(W + 4 * b * kRow + s);
          w[b][0] = w4.x; w[b][1] = w4.y; w[b][2] = w4.z; w[b][3] = w4.w;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float4 y4 = *reinterpret_cast<const float4*>(Y + 8 * k * kRow + s);
          const float4 u4 = *reinterpret_cast<const float4*>(Y + kTile + 8 * k * kRow + s);
          const float y[4] = {y4.x, y4.y, y4.z, y4.w}, u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
          for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int b = 0; b < 8; ++b) masked_fma(acc[k][b], xr[k][b], y[t], u[t], w[b][t]);
        }
      }
      __syncwarp();
      if (c + 2 < c1) issue(c + 2, buf);
    }
    write_tile<4, 8, 8, 4>(acc, smem, gw, lane, m, n, p.dx_split, a.dx, r0, R, i0, I);
    return;
  }

  // ------------------------------------------------------------------ dW tile: rows i (bias row last), columns j, reduced over r
  const int Itot = I + a.has_bias;
  const int tile = (cluster - p.dx_clusters) * (cluster_warps / p.dw_split) + gw / p.dw_split;
  const int i0 = tile % p.dw_tiles_m * kT, j0 = tile / p.dw_tiles_m * kT;          // (a tile behind the last one has j0 >= J)
  const int part = gw % p.dw_split;
  const int chunks = (R + kStep - 1) / kStep;
  const int c0 = chunks * part / p.dw_split, c1 = j0 < J ? chunks * (part + 1) / p.dw_split : c0;
  const int ls = lane >> 3, lc = 4 * (lane & 7);    // 16-byte copies: row ls + 4q of the chunk, columns lc .. lc+3
  auto issue = [&](int c, int buf) {
    const unsigned at = mine_at + 4u * (unsigned)(buf * 3 * kTile);
    if constexpr (VX) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int s = ls + 4 * q, r = c * kStep + s;
        const bool ok = r < R && i0 + lc < I;
        copy16(at + 4u * (s * kT + lc), ok ? a.x + (size_t)r * I + i0 + lc : a.x, ok);
      }
    } else {
#pragma unroll
      for (int s = 0; s < kStep; ++s) {
        const int r = c * kStep + s;
        const bool ok = r < R && i0 + lane < I;
        copy4(at + 4u * (s * kT + lane), ok ? a.x + (size_t)r * I + i0 + lane : a.x, ok);
      }
    }
    if constexpr (VJ) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int s = ls + 4 * q, r = c * kStep + s;
        const bool ok = r < R && j0 + lc < J;
        const size_t o = ok ? (size_t)r * J + j0 + lc : 0;
        copy16(at + 4u * (kTile + s * kT + lc), a.y + o, ok);
        copy16(at + 4u * (2 * kTile + s * kT + lc), a.u + o, ok);
      }
    } else {
#pragma unroll
      for (int s = 0; s < kStep; ++s) {
        const int r = c * kStep + s;
        const bool ok = r < R && j0 + lane < J;
        const size_t o = ok ? (size_t)r * J + j0 + lane : 0;
        copy4(at + 4u * (kTile + s * kT + lane), a.y + o, ok);
        copy4(at + 4u * (2 * kTile + s * kT + lane), a.u + o, ok);
      }
    }
    copies_commit();
  };
  if (c0 < c1) issue(c0, 0);
  if (c0 + 1 < c1) issue(c0 + 1, 1);
  int raised = 0;
  for (int k = threadIdx.x; k < a.nflags; k += kThreads) raised |= __ldg(a.flags + k);
  const bool fast = !__syncthreads_or(raised) && a.scale != 1.0f;
  const float sc = fast ? a.scale : 1.0f, nsc = -sc, nusc = fast ? -1.0f / a.scale : -1.0f;   // exact: powers of two
  const int m = 8 * (lane >> 3), n = 4 * (lane & 7);
  const bool bias_tile = a.has_bias && I >= i0 && I < i0 + kT;    // the bias row (x = biasvolt for every r) is one of the tile's
  uint64_t acc2[8][2];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc2[k][0] = acc2[k][1] = pack2(0.f, 0.f);
  for (int c = c0; c < c1; ++c) {
    const int buf = (c - c0) & 1;
    if (c + 1 < c1) copies_wait<1>(); else copies_wait<0>();
    __syncwarp();
    float* X = mine + buf * 3 * kTile;
    if (bias_tile && lane < kStep) X[lane * kT + I - i0] = a.biasvolt;
    // y and u of the chunk scaled in place, once instead of once per lane that reads them
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float4* y = reinterpret_cast<float4*>(X + kTile) + q * 32 + lane;
      float4* u = reinterpret_cast<float4*>(X + 2 * kTile) + q * 32 + lane;
      const float4 yq = *y, uq = *u;
      *y = make_float4(yq.x * sc, yq.y * sc, yq.z * sc, yq.w * sc);
      *u = make_float4(uq.x * nusc, uq.y * nusc, uq.z * nusc, uq.w * nusc);
    }
    __syncwarp();
    auto steps = [&](auto clamp) {
#pragma unroll 8
      for (int s = 0; s < kStep; ++s) {
        const float4 xa = *reinterpret_cast<const float4*>(X + s * kT + m);
        const float4 xb = *reinterpret_cast<const float4*>(X + s * kT + m + 4);
        const float4 y4 = *reinterpret_cast<const float4*>(X + kTile + s * kT + n);
        const ulonglong2 nu2 = *reinterpret_cast<const ulonglong2*>(X + 2 * kTile + s * kT + n);
        const float x[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
        const float y[4] = {y4.x, y4.y, y4.z, y4.w};
        const uint64_t nu[2] = {nu2.x, nu2.y};
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
          for (int b = 0; b < 2; ++b)
            acc2[k][b] = fma2(pack2(clamp(x[k], y[2 * b]), clamp(x[k], y[2 * b + 1])), nu[b], acc2[k][b]);
      }
    };
    if (fast) steps([nsc](float x, float ys) { return fma_sat(x, nsc, ys); });
    else steps([](float x, float y) { return fmaxf(y - x, 0.f); });
    __syncwarp();
    if (c + 2 < c1) issue(c + 2, buf);
  }
  float acc[8][4];
#pragma unroll
  for (int k = 0; k < 8; ++k)
#pragma unroll
    for (int b = 0; b < 2; ++b) unpack2(acc2[k][b], acc[k][2 * b], acc[k][2 * b + 1]);
  write_tile<8, 4, 1, 1>(acc, smem, gw, lane, m, n, p.dw_split, a.dw, i0, Itot, j0, J);
}

// How many warps share one tile's reduction of length L: a power of two up to the 32 warps of the largest cluster that
// minimises (waves of 12 warps per SM) x (steps of a warp + about 20 steps' worth of prologue, pipeline fill and adding up),
// with at least one chunk of 16 steps per warp.
int pick_split(long tiles, int L, const LaunchInfo& li) {
  const long wave = 12L * li.num_sms;
  int best = 1;
  long best_cost = 0;
  for (int s = 1; s <= kMaxCluster * kWarps && (s == 1 || L >= kStep * s); s *= 2) {
    const long waves = (tiles * s + wave - 1) / wave;
    const long cost = waves * ((L + s - 1) / s + 20);
    if (s == 1 || cost < best_cost) { best = s; best_cost = cost; }
  }
  return best;
}

template <bool VX, bool VJ>
int launch(const DenseArgs& a, const DensePlan& p, cudaStream_t s) {
  if (cudaFuncSetAttribute(snn_dense_bwd_kernel<VX, VJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes) != cudaSuccess)
    return E_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((p.dx_clusters + p.dw_clusters) * p.cluster));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, snn_dense_bwd_kernel<VX, VJ>, a, p);
  count_launch();
  return e == cudaSuccess ? OK : E_CUDA;
}

}  // namespace

// Up to 4096 samples: beyond, the row loop of a dW tile is long enough that the row-split register tiles of
// snntc_backward.cu keep the GPU as busy.
bool dense_bwd_supported(const Geometry& g) { return !g.is_conv && g.R <= 4096; }

int launch_dense_bwd(const Geometry& g, const float* uv, const float* x, const float* w, const float* out, float* dx,
                     float* dw, float scale, const int* flags, int nflags, const LaunchInfo& li, cudaStream_t s) {
  DenseArgs a = {uv, x, w, out, dx, dw, flags, nflags, g.R, g.I, g.J, g.has_bias, g.biasvolt, scale};
  DensePlan p = {};
  const long rt = (g.R + kT - 1) / kT, it = (g.I + kT - 1) / kT;                                // dX tiles
  const long wt = (g.I + g.has_bias + kT - 1) / kT, jt = (g.J + kT - 1) / kT;                   // dW tiles
  p.dx_split = dx ? pick_split(rt * it, g.J, li) : 1;
  p.dw_split = dw ? pick_split(wt * jt, g.R, li) : 1;
  const int most = p.dx_split > p.dw_split ? p.dx_split : p.dw_split;
  p.cluster = most <= kWarps ? 1 : most / kWarps;
  const long warps = (long)p.cluster * kWarps;
  p.dx_tiles_n = (int)it;
  p.dw_tiles_m = (int)wt;
  if (dx) p.dx_clusters = (int)((rt * it + warps / p.dx_split - 1) / (warps / p.dx_split));
  if (dw) p.dw_clusters = (int)((jt * wt + warps / p.dw_split - 1) / (warps / p.dw_split));
  if (p.dx_clusters + p.dw_clusters == 0) return OK;
  const bool vx = (g.I & 3) == 0 && ((uintptr_t)x & 15) == 0;
  const bool vj = (g.J & 3) == 0 && (((uintptr_t)uv | (uintptr_t)out | (uintptr_t)w) & 15) == 0;
  if (vx) return vj ? launch<true, true>(a, p, s) : launch<true, false>(a, p, s);
  return vj ? launch<false, true>(a, p, s) : launch<false, false>(a, p, s);
}

}  // namespace snntc

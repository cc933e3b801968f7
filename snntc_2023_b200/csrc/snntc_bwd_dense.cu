// Both gradients of a dense layer (SnnFcGrad, snntc/snnfcgrad_kernels.cu.cc:15-225) in one launch behind the u kernel, for
// up to 2048 samples.
//
//   dX[r,i] = sum_j [x_ri <= y_rj] u_rj W[i,j]        dW[i,j] = sum_r [x_ri <= y_rj] (x_ri - y_rj) u_rj
//   u[r,j]  = y[r,j] fired ? grad[r,j] * inv[r,j] : 0
//
// What bounds a dense layer at these sizes is not arithmetic but how little of the GPU a call reaches: 256 samples of a
// 784 -> 400 layer are 52 tiles of 64 x 64 for dX, each reducing 400 outputs one after the other. Here
//   - the unit of work is a small tile per WARP. dX: 32 x 32 down to 8 x 8 (rows x inputs), the largest that still gives every
//     SM four warps; the reduction over the outputs is one running sum per element, ascending, as in the other dX kernels.
//     dW: 32 x 32, its rows cut into the slices that plan_dw (snntc_backward.cu) gives the register-tile kernel, a warp per
//     slice, and the slices added through the distributed shared memory of a cluster in the order snn_dw_reduce_kernel adds
//     planes. So the sums are the register-tile kernels' bit for bit;
//   - every warp brings its own chunks of 16 reduction steps in with 16-byte asynchronous copies, two buffers deep, as they
//     lie in memory, with no CTA barrier in the loop. dX reads four steps of a row at once (16 bytes), so nothing has to be
//     transposed; rows of 20 floats and a lane's rows 8 apart keep these reads free of bank conflicts. (4-byte copies that
//     transpose on the way took half of the kernel's instructions, register staging was bound by L1 line lookups.)
//   - dX and dW tiles are blocks of one grid: they run side by side without an auxiliary stream.
// Per element dX is a compare and a predicated FMA (bound by the half-rate compare pipe), dW a saturating FMA and half a
// two-lane FMA (the scaled form of relu(y - x), snntc_backward.cu).
// Measured (B200, dX + dW with the u kernel, before -> now): 784 -> 400 at 32 samples 85 -> 16 us, at 256: 98 -> 35, at 1024: 142 -> 99;
// 4096 -> 512 at 256: 166 -> 126; 25 088 -> 1024 at 64: 501 -> 332.
#include "snntc_common.cuh"
#include "snntc_ptx.cuh"

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

// 4- and 16-byte asynchronous copies; `ok` false writes zeros and reads nothing
__device__ __forceinline__ void copy4(unsigned dst, const float* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copy16(unsigned dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

struct DensePlan {
  int cluster;                             // CTAs per cluster
  int dx_clusters, dx_tiles_n;             // dX: tiles of [rows][inputs], a warp each, neighbours along the inputs
  int dw_clusters, dw_tiles_m;             // dW: tiles of [weight rows][outputs], neighbours along the weight rows
  int dw_splits, dw_rows;                  // slices of the rows (at most 32, a warp each) and rows per slice (a multiple of 16)
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

// A warp's tile of MR x NC sums in shared memory goes out in whole rows.
template <int MR, int NC>
__device__ __forceinline__ void store_tile(const float* tile, int lane, float* __restrict__ dst, int m0, int M, int n0, int N) {
#pragma unroll 4
  for (int e = lane; e < MR * NC; e += 32) {
    const int row = e / NC, col = e % NC;
    if (m0 + row < M && n0 + col < N) dst[(size_t)(m0 + row) * N + n0 + col] = tile[row * kPad + col];
  }
}

// VX: I is a multiple of 4 and x 16-byte aligned; VJ: J is a multiple of 4 and u, y and w 16-byte aligned. Then every copy
// moves 16 bytes, else 4.
// ML, NL: rows and inputs of a dX tile per lane (the tile is 8*ML x 4*NL).
template <bool VX, bool VJ, int ML, int NL>
__global__ void __launch_bounds__(kThreads, 3)
snn_dense_bwd_kernel(const DenseArgs a, const DensePlan p) {
  chain_wait();
  chain_next();
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
    constexpr int MR = 8 * ML, NC = 4 * NL;
    const int tile = cluster * cluster_warps + gw;
    const int r0 = tile / p.dx_tiles_n * MR, i0 = tile % p.dx_tiles_n * NC;
    if (r0 >= R) return;                        // (no barrier of the CTA or cluster in this branch)
    const int chunks = (J + kStep - 1) / kStep;
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
        for (int q = 0; q < ML; ++q) {
          const bool rok = jok && r0 + row + 8 * q < R;
          copy16(to + 4u * (8 * q * kRow), rok ? gy + (size_t)(8 * q) * J : a.y, rok);
          copy16(to + 4u * (8 * q * kRow + kTile), rok ? gu + (size_t)(8 * q) * J : a.u, rok);
        }
#pragma unroll
        for (int q = 0; q < (NL + 1) / 2; ++q) {
          const bool iok = jok && i0 + row + 8 * q < I && row + 8 * q < NC;
          copy16(to + 4u * (8 * q * kRow + 2 * kTile), iok ? gw + (size_t)(8 * q) * J : a.w, iok);
        }
      } else {
        const int j = c * kStep + (lane & 15), row = lane >> 4;
        const bool jok = j < J;
        const unsigned to = at + 4u * (unsigned)(row * kRow + (lane & 15));
#pragma unroll 4
        for (int k = 0; k < MR; k += 2) {
          const bool rok = jok && r0 + row + k < R;
          const size_t o = rok ? (size_t)(r0 + row + k) * J + j : 0;
          copy4(to + 4u * (k * kRow), a.y + o, rok);
          copy4(to + 4u * (k * kRow + kTile), a.u + o, rok);
        }
#pragma unroll 4
        for (int k = 0; k < NC; k += 2) {
          const bool iok = jok && i0 + row + k < I;
          copy4(to + 4u * (k * kRow + 2 * kTile), iok ? a.w + (size_t)(i0 + row + k) * J + j : a.w, iok);
        }
      }
      copies_commit();
    };
    issue(0, 0);
    if (chunks > 1) issue(1, 1);
    const int m = lane >> 2, n = lane & 3;      // this lane's rows m + 8k and inputs n + 4b
    float xr[ML][NL], acc[ML][NL];
#pragma unroll
    for (int k = 0; k < ML; ++k) {
      const float* gx = a.x + (size_t)(r0 + m + 8 * k) * I + i0 + n;
      const bool rok = r0 + m + 8 * k < R;
#pragma unroll
      for (int b = 0; b < NL; ++b) {
        xr[k][b] = (rok && i0 + n + 4 * b < I) ? ld_plain(gx + 4 * b) : CUDART_INF_F;
        acc[k][b] = 0.f;
      }
    }
    for (int c = 0; c < chunks; ++c) {
      const int buf = c & 1;
      if (c + 1 < chunks) copies_wait<1>(); else copies_wait<0>();
      __syncwarp();
      const float* Y = mine + buf * 3 * kTile + m * kRow;
      const float* W = mine + buf * 3 * kTile + 2 * kTile + n * kRow;
#pragma unroll
      for (int s = 0; s < kStep; s += 4) {
        float w[NL][4];
#pragma unroll
        for (int b = 0; b < NL; ++b) {
          const float4 w4 = *reinterpret_cast<const float4*>(W + 4 * b * kRow + s);
          w[b][0] = w4.x; w[b][1] = w4.y; w[b][2] = w4.z; w[b][3] = w4.w;
        }
#pragma unroll
        for (int k = 0; k < ML; ++k) {
          const float4 y4 = *reinterpret_cast<const float4*>(Y + 8 * k * kRow + s);
          const float4 u4 = *reinterpret_cast<const float4*>(Y + kTile + 8 * k * kRow + s);
          const float y[4] = {y4.x, y4.y, y4.z, y4.w}, u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
          for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int b = 0; b < NL; ++b) masked_fma(acc[k][b], xr[k][b], y[t], u[t], w[b][t]);
        }
      }
      __syncwarp();
      if (c + 2 < chunks) issue(c + 2, buf);
    }
#pragma unroll
    for (int k = 0; k < ML; ++k)
#pragma unroll
      for (int b = 0; b < NL; ++b) mine[(m + 8 * k) * kPad + n + 4 * b] = acc[k][b];
    __syncwarp();
    store_tile<MR, NC>(mine, lane, a.dx, r0, R, i0, I);
    return;
  }

  // ------------------------------------------------------------------ dW tile: rows i (bias row last), columns j, reduced over r
  const int Itot = I + a.has_bias;
  const int per = cluster_warps / p.dw_splits;                                      // tiles per cluster
  const int mine_tile = gw / p.dw_splits, part = gw % p.dw_splits;
  const int tile = (cluster - p.dx_clusters) * per + mine_tile;
  const int i0 = tile % p.dw_tiles_m * kT, j0 = tile / p.dw_tiles_m * kT;           // (a tile behind the last one has j0 >= J)
  const int r_begin = part * p.dw_rows, r_end = min(R, r_begin + p.dw_rows);
  const int c0 = r_begin / kStep, c1 = mine_tile < per && j0 < J ? (r_end + kStep - 1) / kStep : c0;
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
  for (int k = threadIdx.x; k < a.nflags; k += kThreads) raised |= ld_plain(a.flags + k);
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
  copies_wait<0>();
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    float lo[2], hi[2];
    unpack2(acc2[k][0], lo[0], hi[0]);
    unpack2(acc2[k][1], lo[1], hi[1]);
    *reinterpret_cast<float4*>(mine + (m + k) * kPad + n) = make_float4(lo[0], hi[0], lo[1], hi[1]);
  }
  if (p.dw_splits == 1) {
    __syncwarp();
    if (c0 < c1) store_tile<kT, kT>(mine, lane, a.dw, i0, Itot, j0, J);
    return;
  }
  // the slices of a tile, added as snn_dw_reduce_kernel adds planes: four interleaved sums, then their sum
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  if (mine_tile < per && j0 + lane < J) {
    const int first = gw - part;
    auto slice = [&](int k, int row) {
      const int wk = first + k;
      return cl.map_shared_rank(smem, wk / kWarps)[(wk % kWarps) * kWarpFloats + row * kPad + lane];
    };
    for (int row = part; row < kT && i0 + row < Itot; row += p.dw_splits) {
      float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
      int k = 0;
      for (; k + 8 <= p.dw_splits; k += 8) {
        float v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = slice(k + q, row);
        s0 += v[0]; s1 += v[1]; s2 += v[2]; s3 += v[3];
        s0 += v[4]; s1 += v[5]; s2 += v[6]; s3 += v[7];
      }
      for (; k < p.dw_splits; ++k) s0 += slice(k, row);
      a.dw[(size_t)(i0 + row) * J + j0 + lane] = (s0 + s1) + (s2 + s3);
    }
  }
  cl.sync();                                           // no CTA leaves while its tiles may still be read
}

template <bool VX, bool VJ, int ML, int NL>
int launch(const DenseArgs& a, const DensePlan& p, cudaStream_t s) {
  if (allow_smem<snn_dense_bwd_kernel<VX, VJ, ML, NL>>(kSmemBytes) != cudaSuccess) return E_CUDA;
  const cudaError_t e = launch_chained(snn_dense_bwd_kernel<VX, VJ, ML, NL>, dim3((unsigned)((p.dx_clusters + p.dw_clusters) * p.cluster)),
                                       dim3(kThreads), kSmemBytes, s, (unsigned)p.cluster, a, p);
  count_launch();
  return e == cudaSuccess ? OK : E_CUDA;
}

template <int ML, int NL>
int launch_tile(DenseArgs a, DensePlan p, bool vx, bool vj, cudaStream_t s) {
  if (a.dx) {
    const long m = (a.R + 8 * ML - 1) / (8 * ML), n = (a.I + 4 * NL - 1) / (4 * NL);
    p.dx_tiles_n = (int)n;
    p.dx_clusters = (int)((m * n + p.cluster * kWarps - 1) / (p.cluster * kWarps));
  }
  if (p.dx_clusters + p.dw_clusters == 0) return OK;
  if (vx) return vj ? launch<true, true, ML, NL>(a, p, s) : launch<true, false, ML, NL>(a, p, s);
  return vj ? launch<false, true, ML, NL>(a, p, s) : launch<false, false, ML, NL>(a, p, s);
}

}  // namespace

// Up to 2048 samples, which plan_dw cuts into at most 32 slices: one per warp of the largest cluster. Beyond, the row loop of a
// dW tile is long enough that the register-tile kernels keep the GPU as busy.
bool dense_bwd_supported(const Geometry& g) { return !g.is_conv && g.R <= 2048; }

int launch_dense_bwd(const Geometry& g, const float* uv, const float* x, const float* w, const float* out, float* dx,
                     float* dw, int dw_splits, int dw_rows, float scale, const int* flags, int nflags, const LaunchInfo& li,
                     cudaStream_t s) {
  const DenseArgs a = {uv, x, w, out, dx, dw, flags, nflags, g.R, g.I, g.J, g.has_bias, g.biasvolt, scale};
  DensePlan p = {};
  p.dw_splits = dw ? dw_splits : 1;
  p.dw_rows = dw_rows;
  p.cluster = (p.dw_splits + kWarps - 1) / kWarps;
  if (p.cluster > kMaxCluster) return E_UNSUPPORTED;
  if (dw) {
    // of the cluster sizes the one that takes the fewest CTAs: the warps of a cluster that its tiles leave over have nothing to do
    // (ten slices, 325 tiles: 975 CTAs with one tile to three of them, 815 with two to five, which is two waves instead of three; dW of
    // 785 x 400 with the u kernel at 1024 samples 62 -> 57 us, at 2048 99 -> 90)
    const long m = (g.I + g.has_bias + kT - 1) / kT, n = (g.J + kT - 1) / kT;
    auto clusters = [&](int c) { const long per = c * kWarps / p.dw_splits; return (m * n + per - 1) / per; };
    for (int c = p.cluster + 1; c <= kMaxCluster; ++c)
      if (clusters(c) * c < clusters(p.cluster) * p.cluster) p.cluster = c;
    p.dw_tiles_m = (int)m;
    p.dw_clusters = (int)clusters(p.cluster);
  }
  const bool vx = (g.I & 3) == 0 && ((uintptr_t)x & 15) == 0;
  const bool vj = (g.J & 3) == 0 && (((uintptr_t)uv | (uintptr_t)out | (uintptr_t)w) & 15) == 0;
  // the largest dX tile that leaves every SM four warps (beside those of dW): a large one reads less per product, with few warps latency
  // counts (both gradients, six warps and four, us: 400 x 400 at 1024 samples 62, 58, 784 x 400 at 512 55, 53)
  auto tiles = [&](int m, int n) { return (long)((g.R + m - 1) / m) * ((g.I + n - 1) / n); };
  const long enough = 4L * li.num_sms;
  // (32 rows only where they are not padding: 35 samples of 9893 -> 940 are 289 us with them, 281 with 16)
  const bool rows32 = (g.R + 31) / 32 * 32 * 8 <= (g.R + 15) / 16 * 16 * 9;
  if (!dx || (tiles(32, 32) >= enough && rows32)) return launch_tile<4, 8>(a, p, vx, vj, s);
  if (tiles(16, 32) >= enough) return launch_tile<2, 8>(a, p, vx, vj, s);
  if (tiles(16, 16) >= enough) return launch_tile<2, 4>(a, p, vx, vj, s);
  return launch_tile<1, 4>(a, p, vx, vj, s);
}

}  // namespace snntc

// The sorted walk for a moderate number of (row, 32 outputs) items: a warp walks one, one output per lane, and copies the weight rows its list
// names into shared memory ahead of itself.
//
// Between the walk with a copying warp (snntc_walk_ring.cu), which with a second warp per item is two waves here, and the pairs walk, which
// at fan-outs up to 32 leaves half of its lanes idle and beyond has too few warps to hide its latencies. Weight rows arrive by asynchronous
// copies, kBlock entries to a block, two blocks ahead of the one that is consumed; the sums and sign tests of kBlock / 2 steps are
// formed before one vote, from operands that were read a group ahead. Blocks of 32 entries halve the votes, and take twice the shared
// memory: 16 warps to an SM instead of 32.
// The steps are those of the walk with a copying warp (LaneWalk in snntc_walk.cuh): the same bits. Bound by the latency of the chain of sums
// up to about ten items per SM and by issue beyond. Measured (B200, walk alone; copying warp, this, pairs walk): 2304 -> 32 at 2600 rows
// 77, 65, 83 us, 5400 -> 32 161, 139, 180, 576 -> 32 28, 24, 25; further figures where the choice is made (snntc_forward.cu).
#include "snntc_common.cuh"
#include "snntc_walk.cuh"

#include <limits.h>
#include <math_constants.h>

namespace snntc {

namespace {

constexpr int kWarps = 2;                          // per CTA, each on a row of its own
constexpr int kRing = 3;                           // weight blocks per warp: one consumed, two on their way
constexpr int kListRing = 4;                       // list blocks per warp

template <int kBlock>                              // list entries
struct RingWarp {
  float w[kRing][kBlock][32];
  float x[kListRing][kBlock];
  unsigned off[kListRing][kBlock];                 // element offset of the weight row
};

// (through L1: weights of 17 to 31 columns share lines, 576 -> 20 at 3500 rows 26 us, 32 past it; 32 columns 27 and 26)
__device__ __forceinline__ void copy_async(unsigned dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

template <int kBlock>
__global__ void __launch_bounds__(32 * kWarps)
snn_walk_alone_kernel(const Geometry g, const WalkEntry* lists, const int* nvalid, int istride, const float* w,
                      float* __restrict__ out, int slices) {
  chain_wait();
  chain_next();
  constexpr int kGroup = kBlock / 2;               // steps per vote
  __shared__ __align__(16) RingWarp<kBlock> ring[kWarps];
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  RingWarp<kBlock>& sm = ring[warp];
  const int J = g.J;
  // neighbouring items are rows of the same output slice: the slice's weights stay in L2 while they run
  const long item = (long)blockIdx.x * kWarps + warp;
  if (item >= (long)g.R * slices) return;
  const int r = (int)(item % g.R), j0 = (int)(item / g.R) * 32;
  const WalkEntry* ents = lists + (size_t)r * istride;
  const int n = __shfl_sync(0xffffffffu, ld_plain(nvalid + r), 0);
  const int blocks = (n + kBlock - 1) / kBlock;

  // list block b: read a block ahead into a register, then put into shared memory. Behind the end of the list: offset 0 (a
  // row is copied that nothing consumes)
  WalkEntry pre = make_uint2(0u, 0u);
  auto read_list = [&](int b) {
    pre = make_uint2(0u, 0u);
    if ((kBlock == 32 || lane < kBlock) && b * kBlock + lane < n) pre = ld_l2(ents + b * kBlock + lane);
  };
  auto put_list = [&](int b) {
    if (kBlock == 32 || lane < kBlock) {
      sm.x[b % kListRing][lane] = __uint_as_float(pre.x);
      sm.off[b % kListRing][lane] = pre.y;
    }
  };
  // weight block b: a copy brings four rows, 16 bytes per lane (lanes behind the row copy nothing)
  const int sub = lane >> 3, col = 4 * (lane & 7);
  const bool mine = j0 + col < J;
  const float* wj = w + j0 + col;
  auto copy_weights = [&](int b) {
    const unsigned* off = sm.off[b % kListRing];
    const unsigned to = smem_u32(&sm.w[b % kRing][0][0]);
#pragma unroll
    for (int q = 0; q < kBlock / 4; ++q)
      if (mine) copy_async(to + 512u * q + 16u * lane, wj + off[4 * q + sub]);
  };

  const int j = j0 + lane;
  const bool ok = j < g.jout;
#pragma unroll
  for (int b = 0; b < kRing - 1; ++b) {
    read_list(b);
    put_list(b);
    __syncwarp();
    if (b < blocks) copy_weights(b);
    copies_commit();
  }
  read_list(kRing - 1);
  LaneWalk wk;
  wk.start(g, ok, g.has_bias && ok ? ld_plain(w + (size_t)g.I * J + j) : 0.f);
  bool turned = false;
  for (int b = 0; b < blocks; ++b) {
    put_list(b + kRing - 1);
    __syncwarp();                                  // (and every lane is through with block b - 1, whose buffer is refilled)
    read_list(b + kRing);
    if (b + kRing - 1 < blocks) copy_weights(b + kRing - 1);
    copies_commit();
    copies_wait<kRing - 1>();                      // weight block b
    __syncwarp();
    const float* xb = sm.x[b % kListRing];
    const float* wb = &sm.w[b % kRing][0][lane];
    const int nb = min(kBlock, n - b * kBlock);
    int k = 0;
    // the next group's operands are read while this one's vote is on its way
    float x[2][kGroup], wv[2][kGroup];
    auto read = [&](int at, float (&xs)[kGroup], float (&ws)[kGroup]) {
#pragma unroll
      for (int u = 0; u < kGroup; u += 4) {
        const float4 v = *reinterpret_cast<const float4*>(xb + at + u);
        xs[u] = v.x; xs[u + 1] = v.y; xs[u + 2] = v.z; xs[u + 3] = v.w;
      }
#pragma unroll
      for (int u = 0; u < kGroup; ++u) ws[u] = wb[(at + u) * 32];
    };
    auto group = [&](const auto& xs, auto& ws) {
      int lim = 0;
      if (__builtin_expect(turned, 0)) lim = wk.guard(xs, ws);
      wk.steps(xs, ws, lim);
    };
    read(0, x[0], wv[0]);
    if (nb == kBlock) {
      read(kGroup, x[1], wv[1]);
      group(x[0], wv[0]);
      group(x[1], wv[1]);
      k = kBlock;
    } else if (kGroup <= nb) {
      group(x[0], wv[0]);
      k = kGroup;
    }
    if (kGroup > 8 && k + 8 <= nb) {
      float x8[8], w8[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) { x8[u] = xb[k + u]; w8[u] = wb[(k + u) * 32]; }
      group(x8, w8);
      k += 8;
    }
#pragma unroll 1
    for (; k < nb; ++k) {
      const float x1[1] = {xb[k]};
      float w1[1] = {wb[k * 32]};
      group(x1, w1);
    }
    turned = wk.turn(turned);
    if (!__any_sync(0xffffffffu, wk.live)) break;  // every output has fired
  }
  copies_wait<0>();

  float yv, iv;
  wk.finish(g, yv, iv);
  if (ok) {
    out[(size_t)r * g.jout + j] = yv;
    if (!g.infer) out[(size_t)(g.R + r) * g.jout + j] = iv;
    if (g.khist != nullptr) atomicAdd(g.khist + (yv < g.maxv ? entries_below(ents, n, yv) : g.I + 1), 1);
  }
}

template <int kBlock>
int launch(const Geometry& g, const WalkEntry* lists, const int* nvalid, int istride, const float* w, float* out, int list_ctas,
           const LaunchInfo& li, cudaStream_t s) {
  const int slices = (g.J + 31) / 32;
  const long grid = ((long)g.R * slices + kWarps - 1) / kWarps;
  if (grid > 0x7fffffffL) return E_UNSUPPORTED;
  const cudaError_t e = launch_chained(snn_walk_alone_kernel<kBlock>, {(unsigned)grid, walk_chains(grid, list_ctas, false, li)}, 32 * kWarps, 0, s, 0, g,
                                       lists, nvalid, istride, w, out, slices);
  count_launch();
  return e == cudaSuccess ? OK : E_CUDA;
}

}  // namespace

int launch_walk_alone(const Geometry& g, const WalkEntry* lists, const int* nvalid, int istride, const float* w, float* out,
                      bool large, int list_ctas, const LaunchInfo& li, cudaStream_t s) {
  return large ? launch<32>(g, lists, nvalid, istride, w, out, list_ctas, li, s)
               : launch<16>(g, lists, nvalid, istride, w, out, list_ctas, li, s);
}

}  // namespace snntc

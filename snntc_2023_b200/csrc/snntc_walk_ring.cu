// The sorted walk for layers with few (row, output) pairs: a warp walks one row for 32 outputs, one per lane, and copies the
// weight rows its list names into shared memory ahead of itself.
//
// With few warps on an SM a walk is bound by latency: the walk from global memory (snntc_forward.cu) waits an L2 round trip for
// every four to eight weight rows and a vote with its branch at every step, 75 to 130 cycles a step. Here
//   - weight rows arrive by asynchronous copies, 32 (or 16) entries to a block, two blocks ahead of the one that is consumed;
//   - the sums and sign tests of 16 (or 8) steps are formed before one vote, from operands that were read a group ahead. The
//     sums in front of every step of the group stay in registers, so where the vote finds an output at or near zero, only the
//     steps concerned are taken through the reference's own comparisons (snntc/snnfc_kernels.cu.cc:46-55) and nothing is
//     replayed (groups of four without the read ahead: 30 % slower at one row of 25 088 inputs);
//   - one output per lane: with a warp per scheduler every instruction of the dependent chain costs its latency, so the fewest
//     instructions per step win (two outputs per lane, as pairs in 64-bit registers, took 82 cycles a step).
// Arithmetic, order and decisions are those of walk_row: the same bits. The margin of a sign test is 2^-22 |x * sum w|, formed
// from the output's own sum -- four times the rounding error of the reference's product x * sum w, so every step that
// rounding could decide goes to the reference's comparisons, and no bound over the weight matrix has to be computed first.
// Measured (B200, walk alone, before -> now): 784 -> 400 at 32 samples 58 -> 22 us; 4096 -> 512 at 32: 150 -> 47 us; 25 088 ->
// 1024 at 64: 1918 -> 771 us; 3x3 convolution 256 -> 256 on 64 fields 85 -> 35 us. From about 24 items (row, 32 outputs) per
// SM on the walk from global memory is the faster one: it spends fewer instructions per output.
#include "snntc_common.cuh"
#include "snntc_walk.cuh"

#include <limits.h>
#include <math_constants.h>

namespace snntc {

namespace {

constexpr int kWarps = 2;                          // per CTA, each on an item of its own
constexpr int kRing = 3;                           // weight blocks per warp: one consumed, two on their way
constexpr int kListRing = 4;                       // list blocks per warp

template <int kBlock>
struct RingWarp {
  float w[kRing][kBlock][32];
  float x[kListRing][kBlock];
  unsigned off[kListRing][kBlock];                 // element offset of the weight row
};

template <int BYTES>
__device__ __forceinline__ void copy_async(unsigned dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}

// One output of one lane. wsum = sum w - theta and ysum = sum w*x run on; an output that has fired keeps its sums in fin and
// its running weight sum at -inf, where q stays +inf.
struct Walk {
  float wsum, ysum;
  float2 fin;
  bool live;
  int sticky;             // INT_MIN: the output was at or near zero at the last entry without firing, else INT_MAX
  float xprev;

  template <bool FIRST, int G>
  __device__ __forceinline__ void steps(const float (&x)[G], const float (&w)[G]) {
    float sw[G], sy[G];
    int p[G];
    const float z = -2.384185791015625e-7f * fmaxf(fabsf(x[0]), fabsf(x[G - 1]));   // inputs ascend: |x| peaks at an end
    int m = sticky;
#pragma unroll
    for (int u = 0; u < G; ++u) {
      sw[u] = wsum; sy[u] = ysum;
      p[u] = __float_as_int(fmaf(z, fabsf(wsum), fmaf(-x[u], wsum, ysum)));   // (an output set aside: NaN, a positive integer)
      m = min(m, p[u]);
      wsum += w[u];
      ysum = fmaf(x[u], w[u], ysum);
    }
    if (__builtin_expect(__any_sync(0xffffffffu, m <= 0), 0)) {
      // FIRST: every lane takes its own first step at or near zero through the comparisons, all lanes at once. Nearly always
      // that step fires; where one does not, or was waited for from the group before, the steps are gone through one by one.
      // (784 -> 400 at 32 samples with its sort 19.9 -> 17.3 us; where bandwidth counts the one by one code is the better one:
      // 25 088 -> 1024 at 64 samples 819 us, 882 with FIRST)
      if constexpr (FIRST) {
        float tw = 0.f, ty = 0.f, tx = 0.f, txp = 0.f;
        bool at = false;
#pragma unroll
        for (int u = G - 1; u >= 0; --u) {
          if (p[u] <= 0) { tw = sw[u]; ty = sy[u]; tx = x[u]; txp = u == 0 ? xprev : x[u > 0 ? u - 1 : 0]; at = true; }
        }
        at &= live;
        const bool hit = at & ratio_gt(ty, tw, txp) & ratio_le(ty, tw, tx);
        if (!__any_sync(0xffffffffu, (at & !hit) | (sticky < 0))) {
          if (hit) {
            fin = make_float2(tw, ty);
            wsum = -CUDART_INF_F;
            live = false;
          }
          xprev = x[G - 1];
          return;
        }
      }
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const bool near = live & (p[u] <= 0);
        if (!__any_sync(0xffffffffu, near | (sticky < 0))) continue;
        const float xp = u == 0 ? xprev : x[u > 0 ? u - 1 : 0];
        const bool fire = live & ratio_gt(sy[u], sw[u], xp) & ratio_le(sy[u], sw[u], x[u]);
        if (fire) fin = make_float2(sw[u], sy[u]);
        live = live & !fire;
        sticky = (near & !fire) ? INT_MIN : INT_MAX;
      }
      if (!live) wsum = -CUDART_INF_F;
    }
    xprev = x[G - 1];
  }
};

// VEC: J is a multiple of 4 and w 16-byte aligned: 16-byte weight copies, else 4-byte ones. kBlock: list entries per block, 32,
// or 16 where there are warps to fill the SMs (half the shared memory per warp: 58 against 68 us for 784 -> 400 at 256 samples).
template <bool VEC, int kBlock>
__global__ void __launch_bounds__(32 * kWarps)
snn_walk_ring_kernel(const Geometry g, const WalkEntry* lists, const int* nvalid, int istride,
                     const float* w, float* __restrict__ out, int slices) {
  chain_wait();
  chain_next();
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
  // weight block b. VEC: a copy brings four rows of 32 outputs, 16 bytes per lane (columns outside the row: column 0 again)
  // Else 4 bytes per lane, 32 / columns rows at a time.
  const int cols = J - j0 < 32 ? J - j0 : 32;
  const int per = VEC ? 4 : 32 / cols, sub = VEC ? lane >> 3 : min(lane / cols, per - 1);
  const int col = VEC ? (4 * (lane & 7) < cols ? 4 * (lane & 7) : 0) : lane % cols;
  const float* wj = w + j0 + col;
  auto copy_weights = [&](int b) {
    const unsigned* off = sm.off[b % kListRing];
    const unsigned to = smem_u32(&sm.w[b % kRing][0][0]);
    if constexpr (VEC) {
#pragma unroll
      for (int q = 0; q < kBlock / 4; ++q) copy_async<16>(to + 512u * q + 16u * lane, wj + off[4 * q + sub]);
    } else {
#pragma unroll 4
      for (int e = sub; e < kBlock; e += per) copy_async<4>(to + 128u * e + 4u * col, wj + off[e]);
    }
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
  Walk wk;
  wk.wsum = -g.theta;
  wk.ysum = 0.f;
  if (g.has_bias) {   // the bias input (value biasvolt, weight row I) is always consumed first
    const float wb = ok ? ld_plain(w + (size_t)g.I * J + j) : 0.f;
    wk.wsum += wb;
    wk.ysum = g.biasvolt * wb;
  }
  if (!ok) wk.wsum = -CUDART_INF_F;
  wk.live = ok;
  wk.fin = make_float2(0.f, 0.f);
  wk.sticky = INT_MAX;
  wk.xprev = g.has_bias ? g.biasvolt : 0.f;
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
    constexpr int kGroup = kBlock / 2;             // steps per vote
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
    read(0, x[0], wv[0]);
#pragma unroll 1
    for (; k + 2 * kGroup <= nb; k += 2 * kGroup) {
      read(k + kGroup, x[1], wv[1]);
      wk.steps<kBlock == 32, kGroup>(x[0], wv[0]);
      read(k + 2 * kGroup < kBlock ? k + 2 * kGroup : 0, x[0], wv[0]);
      wk.steps<kBlock == 32, kGroup>(x[1], wv[1]);
    }
    if (k + kGroup <= nb) {
      wk.steps<kBlock == 32, kGroup>(x[0], wv[0]);
      k += kGroup;
    }
    if (kGroup > 8 && k + 8 <= nb) {
      float x8[8], w8[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) { x8[u] = xb[k + u]; w8[u] = wb[(k + u) * 32]; }
      wk.steps<kBlock == 32, 8>(x8, w8);
      k += 8;
    }
#pragma unroll 1
    for (; k < nb; ++k) {
      const float x1[1] = {xb[k]}, w1[1] = {wb[k * 32]};
      wk.steps<false, 1>(x1, w1);
    }
    if (!__any_sync(0xffffffffu, wk.live)) break;  // every output has fired
  }
  copies_wait<0>();

  // an output that stopped has fired; one that consumed every input fires iff it is armed
  float ws = wk.fin.x, ys = wk.fin.y;
  bool fired = true;
  if (wk.live) {
    ws = wk.wsum; ys = wk.ysum;
    fired = ratio_gt(ys, ws, wk.xprev);
  }
  float yv = g.maxv, iv = 0.f;
  if (fired) {
    iv = __fdividef(1.0f, ws);
    yv = ys * iv;
    if (yv >= g.maxv) { yv = g.maxv; iv = 0.f; }
  }
  if (ok) {
    out[(size_t)r * g.jout + j] = yv;
    if (!g.infer) out[(size_t)(g.R + r) * g.jout + j] = iv;
    if (g.khist != nullptr) atomicAdd(g.khist + (yv < g.maxv ? entries_below(ents, n, yv) : g.I + 1), 1);
  }
}

}  // namespace

int launch_walk_ring(const Geometry& g, const WalkEntry* lists, const int* nvalid, int istride, const float* w, float* out,
                     const LaunchInfo& li, cudaStream_t s) {
  const int slices = (g.J + 31) / 32;
  const long grid = ((long)g.R * slices + kWarps - 1) / kWarps;
  if (grid > 0x7fffffffL) return E_UNSUPPORTED;
  const bool vec = (g.J & 3) == 0 && ((uintptr_t)w & 15) == 0;
  const bool small = grid * kWarps > 8L * li.num_sms;
  auto go = [&](auto kernel) { (void)launch_chained(kernel, (unsigned)grid, 32 * kWarps, 0, s, 0, g, lists, nvalid, istride, w, out, slices); };
  if (vec) small ? go(snn_walk_ring_kernel<true, 16>) : go(snn_walk_ring_kernel<true, 32>);
  else small ? go(snn_walk_ring_kernel<false, 16>) : go(snn_walk_ring_kernel<false, 32>);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? OK : E_CUDA;
}

}  // namespace snntc

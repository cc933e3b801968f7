// The sorted walk for layers with few (row, output) pairs: a warp walks one row for 32 outputs, one per lane, and a warp beside it
// copies the weight rows that the list names into shared memory ahead of it.
//
// With few warps on an SM a walk is bound by latency: the walk from global memory (snntc_forward.cu) waits an L2 round trip for
// every four to eight weight rows and a vote with its branch per step or two, 75 to 130 cycles a step. Here
//   - a warp of its own copies the list and, from it, the weight rows, 32 entries to a block, two blocks ahead of the one that is
//     walked; one barrier per block. A warp that does both spends 38 cycles an entry (one row of 4096 -> 512, 51 us), one that only
//     walks 25 (36 us). Two warps that walk the same row share the copies: 25 088 -> 1024 at 64 samples 804 us with each copying for
//     itself, 463 so (copies past L1: 531 through it);
//   - the sums and sign tests of 16 steps are formed before one vote. The sums in front of every step of the group stay in registers,
//     so where the vote finds an output at or near zero, only the steps concerned are taken through the reference's own
//     comparisons (snntc/snnfc_kernels.cu.cc:46-55) and nothing is replayed;
//   - one output per lane: with a warp per scheduler every instruction of the dependent chain costs its latency, so the fewest
//     instructions per step win (two outputs per lane, as pairs in 64-bit registers, took 82 cycles a step).
// Arithmetic, order and decisions (LaneWalk in snntc_walk.cuh) are those of walk_row: the same bits.
// Measured (B200, walk alone, each warp copying for itself -> now): one row of 784 -> 400 18.6 -> 14.3 us, 64 of 2304 -> 256 30 -> 25,
// 128 of 2000 -> 512 76 -> 43, 100 of 6000 -> 1000 219 -> 164, 64 of 25 088 -> 1024 802 -> 424 (of which the outputs that rounding
// keeps from firing, turn() below, 150).
#include "snntc_common.cuh"
#include "snntc_walk.cuh"

#include <limits.h>
#include <math_constants.h>

namespace snntc {

namespace {

constexpr int kBlock = 32;                         // list entries
constexpr int kGroup = 16;                         // steps per vote
constexpr int kRing = 3;                           // blocks of weights: one consumed, two on their way
constexpr int kListAhead = 2;                      // blocks that the list is copied ahead of the weights it names

template <int BYTES>
__device__ __forceinline__ void copy_async(unsigned dst, const void* src, bool valid) {   // not valid: zeros
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? BYTES : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(valid ? BYTES : 0) : "memory");
}

// A CTA takes a row and 32 * C outputs: C warps walk 32 outputs each, one more warp copies for them. VEC: J is a multiple of 4 and w
// 16-byte aligned: 16-byte weight copies, else 4-byte ones (C = 1).
template <int C>
struct RingShared {
  float w[kRing][kBlock][32 * C];
  float x[kRing][kBlock];
  WalkEntry list[2 * kListAhead][kBlock];
};

template <bool VEC, int C>
__global__ void __launch_bounds__(32 * (C + 1))
snn_walk_ring_kernel(const Geometry g, const WalkEntry* lists, const int* nvalid, int istride, const float* w,
                     float* __restrict__ out) {
  chain_wait();
  chain_next();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RingShared<C>& sm = *reinterpret_cast<RingShared<C>*>(smem_raw);
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int J = g.J;
  // neighbouring CTAs are rows of the same output slice: the slice's weights stay in L2 while they run
  const int r = (int)(blockIdx.x % (unsigned)g.R), j0 = (int)(blockIdx.x / (unsigned)g.R) * 32 * C;
  const WalkEntry* ents = lists + (size_t)r * istride;
  const int n = __shfl_sync(0xffffffffu, ld_plain(nvalid + r), 0);
  const int blocks = (n + kBlock - 1) / kBlock;

  if (warp == C) {
    // list block b: a lane per entry. Behind the end of the list: the last input again with weights of zero, which change no sum and
    // can fire nothing
    auto copy_list = [&](int b) {
      if (b < blocks)
        copy_async<8>(smem_u32(&sm.list[b % (2 * kListAhead)][lane]), ents + min(b * kBlock + lane, n - 1), true);
    };
    // VEC: a copy instruction brings 4 / C rows of 32 * C outputs, 16 bytes per lane. Else 4 bytes per lane, 32 / columns rows at a time.
    // (Lanes behind the row copy nothing: with the row's first column once more 1024 rows of 400 -> 10 took 47 us, 15 so.)
    const int cols = J - j0 < 32 * C ? J - j0 : 32 * C;
    const int per = VEC ? 4 / C : 32 / cols, sub = VEC ? lane / (8 * C) : min(lane / cols, per - 1);
    const int at = VEC ? 4 * (lane % (8 * C)) : lane % cols;
    const float* wj = w + j0 + at;
    const bool mine = !VEC || at < cols;
    int s = 0;                                     // buffer of the block that is filled next
    auto fill = [&](int b) {
      if (b >= blocks) return;
      const WalkEntry e = sm.list[b % (2 * kListAhead)][lane];
      sm.x[s][lane] = __uint_as_float(e.x);
      const unsigned to = smem_u32(&sm.w[s][0][at]);
      // (the offsets of eight copies are shuffled together: one by one each waits for its own, 28 cycles a copy)
#pragma unroll 1
      for (int q = 0; q < kBlock; q += 8 * per) {
        unsigned off[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) off[i] = __shfl_sync(0xffffffffu, e.y, (q + i * per + sub) & 31);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int k = q + i * per + sub;
          if (VEC ? mine : k < kBlock) copy_async<VEC ? 16 : 4>(to + 128u * C * k, wj + off[i], b * kBlock + k < n);
        }
      }
      s = s + 1 == kRing ? 0 : s + 1;
    };
#pragma unroll
    for (int b = 0; b < kRing - 1 + kListAhead; ++b) copy_list(b);
    copies_commit();
    copies_wait<0>();
    __syncwarp();
#pragma unroll 1
    for (int b = 0; b < kRing - 1; ++b) {
      fill(b);
      copies_commit();
    }
    for (int b = 0; b < blocks; ++b) {
      copies_wait<kRing - 2>();                    // block b, and the list of block b + kListAhead
      if (!__syncthreads_or(0)) break;             // (and every warp has read block b - 1, whose buffer is refilled)
      fill(b + kRing - 1);
      copy_list(b + kRing - 1 + kListAhead);
      copies_commit();
    }
    copies_wait<0>();
    return;
  }

  const int j = j0 + 32 * warp + lane;
  const bool ok = j < g.jout;
  LaneWalk wk;
  wk.start(g, ok, g.has_bias && ok ? ld_plain(w + (size_t)g.I * J + j) : 0.f);
  if (blocks > 0 && __syncthreads_or(wk.live)) {
    bool more = true, turned = false;
    // (one copy of the steps: reading the next group ahead of a vote takes two, and costs more in instructions that have to be
    // fetched than it hides)
    int half = 0;                                  // of the 2 * kRing halves of the buffers
#pragma unroll 1
    for (int h = 0; more; ++h) {
      float x[kGroup], wv[kGroup];
      const float* xb = &sm.x[0][0] + half * kGroup;
      const float* wb = &sm.w[0][0][32 * warp + lane] + half * (kGroup * 32 * C);
      half = half + 1 == 2 * kRing ? 0 : half + 1;
#pragma unroll
      for (int u = 0; u < kGroup; u += 4) {
        const float4 v = *reinterpret_cast<const float4*>(xb + u);
        x[u] = v.x; x[u + 1] = v.y; x[u + 2] = v.z; x[u + 3] = v.w;
      }
#pragma unroll
      for (int u = 0; u < kGroup; ++u) wv[u] = wb[u * 32 * C];
      // a block's barrier lies behind the reads of the block in front of it, not behind its steps
      if (h & 1) more = (h >> 1) + 1 < blocks && __syncthreads_or(wk.live);
      int lim = 0;
      if (__builtin_expect(turned, 0)) lim = wk.guard(x, wv);
      wk.steps(x, wv, lim);
      turned = wk.turn(turned);
    }
  }

  float yv, iv;
  wk.finish(g, yv, iv);
  if (ok) {
    out[(size_t)r * g.jout + j] = yv;
    if (!g.infer) out[(size_t)(g.R + r) * g.jout + j] = iv;
    if (g.khist != nullptr) atomicAdd(g.khist + (yv < g.maxv ? entries_below(ents, n, yv) : g.I + 1), 1);
  }
}

template <bool VEC, int C>
int launch(const Geometry& g, const WalkEntry* lists, const int* nvalid, int istride, const float* w, float* out, int list_ctas,
           const LaunchInfo& li, cudaStream_t s) {
  const long grid = (long)g.R * ((g.J + 32 * C - 1) / (32 * C));
  if (grid > 0x7fffffffL) return E_UNSUPPORTED;
  constexpr size_t smem = sizeof(RingShared<C>);
  if (allow_smem<snn_walk_ring_kernel<VEC, C>>(smem) != cudaSuccess) return E_CUDA;
  const cudaError_t e = launch_chained(snn_walk_ring_kernel<VEC, C>, {(unsigned)grid, walk_chains(grid, list_ctas, C == 1, li)}, 32 * (C + 1), smem, s, 0, g,
                                       lists, nvalid, istride, w, out);
  count_launch();
  return e == cudaSuccess ? OK : E_CUDA;
}

}  // namespace

// How many warps of 32 outputs share a list and a copying warp: one for fan-outs up to 32 (with a second, idle one 64 us instead of 48
// for 1430 rows of 2304 -> 32) and while every CTA has an SM to itself (one row of 4096 -> 512 36 us,
// 38 with two), two up to six CTAs per SM, which is what the registers hold. Beyond, four where that makes it one wave again (25 088 ->
// 1024 at 64 samples 424 us, 515 with two; 2000 -> 512 at 128 43, 53): the copying warp, 28 cycles an entry, holds four back (9000 ->
// 700 at 30 samples 115 us, 89 with two).
int launch_walk_ring(const Geometry& g, const WalkEntry* lists, const int* nvalid, int istride, const float* w, float* out,
                     int list_ctas, const LaunchInfo& li, cudaStream_t s) {
  const bool vec = (g.J & 3) == 0 && ((uintptr_t)w & 15) == 0;
  if (!vec) return launch<false, 1>(g, lists, nvalid, istride, w, out, list_ctas, li, s);
  auto ctas = [&](int c) { return (long)g.R * ((g.J + 32 * c - 1) / (32 * c)); };
  if (g.J <= 32 || ctas(1) <= li.num_sms) return launch<true, 1>(g, lists, nvalid, istride, w, out, list_ctas, li, s);
  if (ctas(2) > 6L * li.num_sms && ctas(4) <= 4L * li.num_sms) return launch<true, 4>(g, lists, nvalid, istride, w, out, list_ctas, li, s);
  return launch<true, 2>(g, lists, nvalid, istride, w, out, list_ctas, li, s);
}

}  // namespace snntc

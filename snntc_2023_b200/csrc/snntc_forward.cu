// SNN-TC forward (SnnFc / SnnCv) for sm_100a: sorted lists of the inputs that can spike -> sorted walk.
//
// Rows are dense samples or conv receptive fields (gathered straight from the NHWC image with MAX
// outside it). A scratch buffer of sorted lists in global memory -- per row the inputs at or below MAX-0.1 as
// (value, element offset of the weight row), ascending -- joins two stages:
//   1. the lists. Stride-1 convolutions up to 3x3 on 16 to 512 channels: per-pixel sort and two levels of
//      merging (snntc_lists.cu). Rows of at most 64 inputs: a sorting network in registers, one warp per row
//      (snntc_lists.cu). Everything else: a bucket sort per row (snntc_sort.cu);
//   2. the walk (walk kernels): every warp takes (row, block of outputs) items and walks the row's list, which it
//      stages through shared memory 32 entries at a time. The running sum(w)-theta and sum(w*x) stay in
//      registers, in sorted order, bias first, with the arithmetic of the reference kernel
//      (snntc/snnfc_kernels.cu.cc:33-69); the causality test is the sign of q = ysum - x*wsum per step -- one FMA
//      per output, the lane's smallest q as an integer, one warp vote -- backed by the reference's exact
//      division-free comparisons wherever the sign is not certain (PairWalk in snntc_walk.cuh, walk_row). Three layouts of
//      a lane's outputs: one pair or two pairs of neighbours in 64-bit registers (walk_pairs), or outputs lane + 32*m
//      (odd fan-out, unaligned weights).
#include "snntc_common.cuh"
#include "snntc_walk.cuh"

#include <limits.h>
#include <math.h>
#include <algorithm>
#include <math_constants.h>
#include <type_traits>

namespace snntc {

namespace {

// A CTA of the walks from global memory is two warps with one item each: the rows differ in length and in when their outputs have
// fired, and small CTAs leave it to the hardware to give a free place the next item (eight warps that took every grid-th
// item, 8 CTAs per SM: 2570 us for 131 072 rows of 576 x 128, 2370 so; 4096 of 1152 x 128: 135, 120; one item per warp but eight
// warps: 2387, 135).
constexpr int kFwdThreads = 64;
constexpr int kFwdWarps = kFwdThreads / 32;

typedef unsigned long long u64;

// Index of this warp in its CTA, broadcast from lane 0: the value is the same for all 32 lanes anyway, but only
// a shuffle from a fixed lane lets the compiler treat everything derived from it (row numbers, list lengths,
// loop bounds) as warp-uniform, and with that it drops the divergence check in front of every warp vote.
__device__ __forceinline__ int uniform_warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// ------------------------------------------------------------------------------------------- walk

// How close to zero q = ysum - x*wsum may be before the sign of q stops deciding. The reference compares
// ysum against the ROUNDED product x*wsum (ratio_gt / ratio_le below), so it can see "ysum <= x*wsum" while the
// exact difference is still positive by up to half an ulp of the product, and the other way round for the test
// against the previous input. The walk therefore hands a step over to the reference's comparisons whenever
// q <= tol, tol = 2^-21 * |x| * (|theta| + B), B = sum of g.wbound[] >= sum_i |w_ij| for every output j: |wsum| never
// exceeds |theta| + B, so tol is at least eight times the largest rounding error of the product, and small enough
// to be met by chance about once in 10^5 output steps. Compared as integers: tol >= +0, negative q are negative.
__device__ __forceinline__ float walk_tolerance_base(const Geometry& g) {
  const int lane = threadIdx.x & 31;
  float b = lane < g.wbound_n ? ld_plain(g.wbound + lane) : 0.f;
  if (lane + 32 < g.wbound_n) b += ld_plain(g.wbound + lane + 32);
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) b += __shfl_xor_sync(0xffffffffu, b, d);
  return 4.76837158203125e-7f * (fabsf(g.theta) + b) * 1.0001f;   // (a little slack for the rounding of the sums)
}

// One warp walks one row for 32*JPT outputs. Let q_k = ysum - x_k*wsum be taken just before input k is
// consumed. The reference fires at step k when "ysum/wsum > previous input" and "ysum/wsum <= x_k", i.e.
// sign(wsum)*q_{k-1} > 0 >= sign(wsum)*q_k (q_{k-1} re-evaluated with the sums of step k, which leaves its
// value unchanged). With a positive denominator -- the only case in which an output of sorted inputs at or
// above the bias input can fire -- that is the first k with q_k <= 0. The loop therefore computes one extra FMA
// per output and step (q, with its exact sign), takes the smallest q of the lane and one warp vote; only when
// some lane sees q <= 0 does the warp evaluate the reference's own rounded, division-free tests
// (snntc/snnfc_kernels.cu.cc:46-55) for its live outputs, so the decision is the reference's, an exact tie
// (q == 0) included. An output whose q is not positive but which the reference test did not fire -- q within an
// ulp of zero, or a NEGATIVE denominator, which inputs below the bias input can produce and for which the
// reference fires on the way back up through zero -- makes the lane "sticky": the exact tests run again at
// the next step whatever q is, until no live output of the lane is in that state any more.
template <int JPT, int CH, bool FULL>
__device__ __forceinline__ void walk_row(const Geometry& g, const WalkEntry* ents, int nvalid,
                                         const float* w, int jbase, int lane,
                                         float* __restrict__ y_row, float* __restrict__ inv_row,
                                         WalkEntry* __restrict__ sbuf) {
  const int J = g.J;
  int jl[JPT];
  bool jok[JPT];
  float wsum[JPT], ysum[JPT], wfin[JPT], yfin[JPT];
  int livemask[JPT];
#pragma unroll
  for (int m = 0; m < JPT; ++m) {
    const int j = jbase + lane + 32 * m;
    jok[m] = FULL || j < g.jout;
    jl[m] = jok[m] ? j : J - 1;   // (padding behind jout: weights of zero, never stored)
    wsum[m] = -g.theta;
    ysum[m] = 0.f;
    if (g.has_bias) {  // the bias input (value biasvolt, weight row I) is always consumed first
      const float wb = ld_plain(w + (size_t)g.I * J + jl[m]);
      wsum[m] += wb;
      ysum[m] = g.biasvolt * wb;
    }
    wfin[m] = wsum[m];
    yfin[m] = ysum[m];
    livemask[m] = -1;
    if (!jok[m]) {   // no output: parked from the start like one that has fired, or the walk would wait for it
      livemask[m] = 0;
      wsum[m] = -CUDART_INF_F;
    }
  }
  // Without bias the sums start at (-theta, 0), for which "ysum/wsum > c" is false for every c >= 0, so the
  // first step needs no special case; with bias the previous input is the bias input itself.
  float xprev = g.has_bias ? g.biasvolt : 0.f;
  int sticky = INT_MAX;   // INT_MIN while some live output of this lane must be tested exactly at the next step
  const float tolbase = walk_tolerance_base(g);
  int qlim = 0;           // bits of the largest q that still goes to the exact tests (see walk_tolerance_base)

  const float* wl = w + (FULL ? jbase + lane : 0);
  auto load_weights = [&](unsigned eoff, float (&wv)[JPT]) {
    const float* wrow = wl + eoff;
#pragma unroll
    for (int m = 0; m < JPT; ++m) wv[m] = FULL ? ld_plain(wrow + 32 * m) : ld_plain(wrow + jl[m]);
  };

  // one step for all JPT outputs of this lane: sign test, (rarely) exact test, then consume
  auto step = [&](const float x, const float xprev, const float (&wv)[JPT]) {
    int q[JPT];
#pragma unroll
    for (int m = 0; m < JPT; ++m) q[m] = __float_as_int(fmaf(-x, wsum[m], ysum[m]));
    int qmin;
    if constexpr (JPT == 1) qmin = min(q[0], sticky);
    else if constexpr (JPT == 2) qmin = imin3(q[0], q[1], sticky);
    else qmin = imin3(imin3(q[0], q[1], q[2]), q[3], sticky);
    if (__builtin_expect(__any_sync(0xffffffffu, qmin <= qlim), 0)) {
      // rare path: the reference's own rounded comparisons for the live outputs concerned (usually one of the
      // lane's outputs in one lane: skip the others with a warp-uniform test each)
      bool again = false;
#pragma unroll
      for (int m = 0; m < JPT; ++m) {
        if (JPT > 1 && !__any_sync(0xffffffffu, (q[m] <= qlim) | (sticky < 0))) continue;
        const bool live = livemask[m] != 0;
        const bool fire = live & ratio_gt(ysum[m], wsum[m], xprev) & ratio_le(ysum[m], wsum[m], x);
        if (fire) {
          livemask[m] = 0;  // spike lies in (previous input, x]: keep the sums aside ...
          wfin[m] = wsum[m];
          yfin[m] = ysum[m];
          // ... and park the running ones where q can never be non-positive again: with wsum = -inf,
          // q = ysum + x*inf = +inf at every later step
          wsum[m] = -CUDART_INF_F;
        }
        again |= live & !fire & (q[m] <= qlim);
      }
      sticky = again ? INT_MIN : INT_MAX;
    }
#pragma unroll
    for (int m = 0; m < JPT; ++m) {
      wsum[m] += wv[m];
      ysum[m] = fmaf(x, wv[m], ysum[m]);
    }
  };

  bool all_done = false;
  auto check_done = [&]() {
    int any_live = 0;
#pragma unroll
    for (int m = 0; m < JPT; ++m) any_live |= livemask[m];
    all_done = !__any_sync(0xffffffffu, any_live != 0);
  };
  // One chunk of CH steps: entries, two by one 16-byte read, then their weight rows, then the arithmetic.
  static_assert(CH % 2 == 0, "entries are fetched two at a time");
  auto chunk = [&](const WalkEntry* cur) {
    float xs[CH];
    float wv[CH][JPT];
#pragma unroll
    for (int u = 0; u < CH; u += 2) {
      const uint4 e2 = *reinterpret_cast<const uint4*>(cur + u);
      xs[u] = __uint_as_float(e2.x);
      load_weights(e2.y, wv[u]);
      xs[u + 1] = __uint_as_float(e2.z);
      load_weights(e2.w, wv[u + 1]);
    }
    qlim = __float_as_int(tolbase * fmaxf(fabsf(xs[0]), fabsf(xs[CH - 1])));   // inputs ascend: |x| peaks at an end
#pragma unroll
    for (int u = 0; u < CH; ++u) step(xs[u], u == 0 ? xprev : xs[u > 0 ? u - 1 : 0], wv[u]);
    xprev = xs[CH - 1];   // the previous input is only read when an output is about to fire: no copy per step
  };
  auto single = [&](const WalkEntry e) {
    float wv[JPT];
    load_weights(e.y, wv);
    qlim = __float_as_int(tolbase * fabsf(__uint_as_float(e.x)));
    step(__uint_as_float(e.x), xprev, wv);
    xprev = __uint_as_float(e.x);
  };
  // The list goes through shared memory 32 entries at a time: one coalesced read per lane and block, issued a
  // whole block ahead, instead of one L2 round trip in front of every chunk; a step then reads its entry with
  // one broadcast shared-memory load. Two buffers of 32 entries per warp.
  WalkEntry pre = make_uint2(0u, 0u);
  if (lane < nvalid) pre = ld_l2(ents + lane);
  int b = 0;
  for (int base = 0; base < nvalid && !all_done; base += 32, b ^= 32) {
    sbuf[b + lane] = pre;
    __syncwarp();
    if (base + 32 + lane < nvalid) pre = ld_l2(ents + base + 32 + lane);
    const int nb = min(32, nvalid - base);
    const WalkEntry* cur = sbuf + b;
    int kk = 0;
#pragma unroll 1
    for (; kk + CH <= nb; kk += CH) chunk(cur + kk);
    for (; kk < nb; ++kk) single(cur[kk]);
    check_done();   // one "has every output fired" vote per block
  }

#pragma unroll
  for (int m = 0; m < JPT; ++m) {
    // an output that stopped has fired; one that consumed every input fires iff it is armed
    bool fired = true;
    float ws = wfin[m], ys = yfin[m];
    if (livemask[m]) {
      ws = wsum[m]; ys = ysum[m];
      fired = ratio_gt(ys, ws, xprev);
    }
    float yv = g.maxv, iv = 0.f;
    if (fired) {
      iv = __fdividef(1.0f, ws);
      yv = ys * iv;
      if (yv >= g.maxv) { yv = g.maxv; iv = 0.f; }
    }
    if (jok[m]) {
      const int j = jbase + lane + 32 * m;
      y_row[j] = yv;
      if (inv_row != nullptr) inv_row[j] = iv;
      if (g.khist != nullptr) atomicAdd(g.khist + (yv < g.maxv ? entries_below(ents, nvalid, yv) : g.I + 1), 1);
    }
  }
}

// ---- outputs in pairs, two to a 64-bit register (PairWalk in snntc_walk.cuh): one pair of neighbouring outputs per lane (P = 1, 64 per
// warp) or two (P = 2, 128 per warp). Requires J a multiple of 2 * P and the weights aligned to 8 * P bytes.
// WS: the weights of this warp's 64 outputs sit in shared memory as [fan-in row][64] (see snn_walk2_smemw_kernel);
// `ws_lane` is the shared-memory byte address of this lane's pair in row 0 and `wmul` = 256 / J (J = 64, 128 or 256): a
// list entry's element offset (source index * J) times wmul is the row's byte offset in the slice -- one integer
// multiply-add on the FMA pipe per weight read.
// The list goes through shared memory 32 entries at a time (sbuf: a block and the entry in front of it), one coalesced read per lane
// issued a block ahead instead of an L2 round trip per step. CH entries and their weight rows are read together.
constexpr int kPairsStage = 34;                   // entries staged per warp: 33, and to a multiple of 16 bytes

template <int P, int CH, bool WS = false, bool FULL = WS>
__device__ __forceinline__ void walk_pairs(const Geometry& g, const WalkEntry* ents, int nvalid, const float* w, int jbase, int lane,
                                           float* __restrict__ y_row, float* __restrict__ inv_row, WalkEntry* __restrict__ sbuf,
                                           float* __restrict__ fin, unsigned ws_lane = 0u, unsigned wmul = 0u) {
  const int j0 = jbase + 2 * P * lane;                    // this lane's outputs: 2 * P from j0 on
  const unsigned lane_off = (unsigned)(jbase + 2 * P * (FULL ? lane : min(lane, (g.J - jbase) / (2 * P) - 1)));   // (behind the row: its last)
  const char* wbase = reinterpret_cast<const char*>(w);
  // a 32-bit element offset from the (uniform) weight base, widened before the scaling to bytes: a 64-bit pointer per lane plus the
  // entry's offset takes two instructions more per step
  auto load_row = [&](unsigned eoff, uint64_t (&wv)[P]) {
    if constexpr (WS) {
      static_assert(P == 1, "slices of 64 outputs");
      asm("ld.shared.b64 %0, [%1];" : "=l"(wv[0]) : "r"(eoff * wmul + ws_lane));
    } else if constexpr (P == 1) {
      wv[0] = ld_plain(reinterpret_cast<const unsigned long long*>(wbase + (size_t)(eoff + lane_off) * 4u));
    } else {
      const ulonglong2 v = ld_plain(reinterpret_cast<const ulonglong2*>(wbase + (size_t)(eoff + lane_off) * 4u));
      wv[0] = v.x; wv[1] = v.y;
    }
  };
  PairWalk<P> pw;
  pw.fin = fin + lane;
  {
    float wb[2 * P];
    bool ok[2 * P];
#pragma unroll
    for (int m = 0; m < 2 * P; ++m) {   // the bias input (value biasvolt, weight row I) is always consumed first
      wb[m] = g.has_bias ? ld_plain(w + (size_t)g.I * g.J + lane_off + m) : 0.f;
      ok[m] = FULL || j0 + m < g.jout;
    }
    // (the smallest input is read by all lanes from one address: taken out of lane 0's entry below it cost a divergence check in
    // front of every vote)
    pw.start(g, walk_tolerance_base(g), nvalid > 0 ? __uint_as_float(ld_l2(ents).x) : 0.f, wb, ok);
  }
  WalkEntry pre = make_uint2(0u, 0u);
  if (lane < nvalid) pre = ld_l2(ents + lane);
  // entry k of the list is staged at k % 32, the one in front of the block at 32
  if (lane == 0) sbuf[32] = make_uint2(__float_as_uint(g.has_bias ? g.biasvolt : 0.f), 0u);
  __syncwarp();                                           // (a row without spiking inputs goes straight on to reading it)
  auto inputs = [&](int at) { return make_float2(__uint_as_float(sbuf[at].x), __uint_as_float(sbuf[at > 0 ? at - 1 : 32].x)); };
  bool flipped = false;
  auto block = [&](int base, auto flip_c) {
    constexpr bool FLIP = decltype(flip_c)::value;
    constexpr int N = FLIP ? 2 : CH;                      // (FLIP with four: the walk spills more, 4 % slower)
    const int nb = min(32, nvalid - base);
    pw.margin(__uint_as_float(sbuf[0].x), __uint_as_float(sbuf[nb - 1].x));   // inputs ascend: |x| peaks at an end
    int kk = 0;
#pragma unroll 1
    for (; kk + N <= nb; kk += N) {
      uint64_t x2[N], wv[N][P];
#pragma unroll
      for (int u = 0; u < N; u += 2) {
        const uint4 e2 = *reinterpret_cast<const uint4*>(sbuf + kk + u);
        x2[u] = pack2(__uint_as_float(e2.x), __uint_as_float(e2.x));
        load_row(e2.y, wv[u]);
        x2[u + 1] = pack2(__uint_as_float(e2.z), __uint_as_float(e2.z));
        load_row(e2.w, wv[u + 1]);
      }
      if constexpr (FLIP) {
#pragma unroll
        for (int u = 0; u < N; ++u) pw.template step<true>(x2[u], wv[u], [&] { return inputs(kk + u); });
      } else {
#pragma unroll
        for (int u = 0; u < N; u += 2)
          pw.step2(x2[u], wv[u], x2[u + 1], wv[u + 1], [&] { return inputs(kk + u); }, [&] { return inputs(kk + u + 1); });
      }
    }
#pragma unroll 1
    for (; kk < nb; ++kk) {
      const WalkEntry e = sbuf[kk];
      uint64_t wv[P];
      load_row(e.y, wv);
      pw.template step<FLIP>(pack2(__uint_as_float(e.x), __uint_as_float(e.x)), wv, [&] { return inputs(kk); });
    }
    flipped = pw.template flip<FLIP>(__uint_as_float(sbuf[nb - 1].x));
  };
  for (int base = 0; base < nvalid; base += 32) {
    __syncwarp();                                         // (every lane is through with the block that goes)
    if (lane == 31 && base > 0) sbuf[32] = sbuf[31];      // (that lane's own store)
    sbuf[lane] = pre;
    __syncwarp();
    if (base + 32 + lane < nvalid) pre = ld_l2(ents + base + 32 + lane);
    if (__builtin_expect(flipped, 0)) block(base, std::true_type{});
    else block(base, std::false_type{});
    if (pw.done()) break;   // every output has fired
  }
  const float xprev = __uint_as_float(sbuf[nvalid > 0 ? (nvalid - 1) & 31 : 32].x);
#pragma unroll
  for (int m = 0; m < 2 * P; ++m) {
    const int j = j0 + m;
    if (!FULL && j >= g.jout) continue;
    float y, inv;
    pw.finish(g, m, xprev, y, inv);
    y_row[j] = y;
    if (inv_row != nullptr) inv_row[j] = inv;
    if (g.khist != nullptr) atomicAdd(g.khist + (y < g.maxv ? entries_below(ents, nvalid, y) : g.I + 1), 1);
  }
}

// ------------------------------------------------------------------------------------------- kernels
// Walk kernel: every warp takes (row, block of 32*JPT outputs) items, adjacent warps share a row.
template <int JPT>
__global__ void __launch_bounds__(kFwdThreads, 1024 / kFwdThreads)   // 64 registers, 32 warps per SM
snn_walk_kernel(const Geometry g, const WalkEntry* keys_g, const int* nvalid_g, int istride,
                const float* w, float* __restrict__ out) {
  chain_wait();
  chain_next();
  __shared__ __align__(16) WalkEntry stage[kFwdWarps * 64];   // two blocks of 32 list entries per warp
  WalkEntry* sbuf = stage + (threadIdx.x >> 5) * 64;
  const int R = g.R;
  const int lane = threadIdx.x & 31;
  const int jchunks = (g.jout + 32 * JPT - 1) / (32 * JPT);
  const bool full_j = (g.jout % (32 * JPT)) == 0;
  float* __restrict__ y_out = out;
  float* __restrict__ inv_out = g.infer ? nullptr : out + (size_t)R * g.jout;
  const long items = (long)R * jchunks;
  const long wstride = (long)gridDim.x * kFwdWarps;
  constexpr int CH = JPT == 4 ? 4 : 8;
  for (long item = (long)blockIdx.x * kFwdWarps + uniform_warp_index(); item < items; item += wstride) {
    const int r = (int)(item / jchunks), jc = (int)(item - (long)r * jchunks);
    const WalkEntry* krow = keys_g + (size_t)r * istride;
    const int n = __shfl_sync(0xffffffffu, ld_plain(nvalid_g + r), 0);
    if (full_j)
      walk_row<JPT, CH, true>(g, krow, n, w, jc * 32 * JPT, lane, y_out + (size_t)r * g.jout, (inv_out ? inv_out + (size_t)r * g.jout : nullptr), sbuf);
    else
      walk_row<JPT, CH, false>(g, krow, n, w, jc * 32 * JPT, lane, y_out + (size_t)r * g.jout, (inv_out ? inv_out + (size_t)r * g.jout : nullptr), sbuf);
    __syncwarp();   // the next row's first block goes into the buffer this row may have read last
  }
}

// The same items with the outputs of a lane held in pairs (walk_pairs): a warp covers 64 * P outputs.
template <int P, bool FULL>
__global__ void __launch_bounds__(kFwdThreads, 1024 / kFwdThreads)
snn_walk_pairs_kernel(const Geometry g, const WalkEntry* keys_g, const int* nvalid_g, int istride, const float* w,
                      float* __restrict__ out) {
  chain_wait();
  chain_next();
  __shared__ __align__(16) WalkEntry stage[kFwdWarps * kPairsStage];
  __shared__ float fins[kFwdWarps * PairWalk<P>::kFloats];
  constexpr int CH = P == 2 ? 4 : 8;
  WalkEntry* sbuf = stage + (threadIdx.x >> 5) * kPairsStage;
  float* fin = fins + (threadIdx.x >> 5) * PairWalk<P>::kFloats;
  const int J = g.jout, R = g.R;
  const int lane = threadIdx.x & 31;
  const int jchunks = (J + 64 * P - 1) / (64 * P);
  float* __restrict__ y_out = out;
  float* __restrict__ inv_out = g.infer ? nullptr : out + (size_t)R * J;
  const long items = (long)R * jchunks;
  const long wstride = (long)gridDim.x * kFwdWarps;
  for (long item = (long)blockIdx.x * kFwdWarps + uniform_warp_index(); item < items; item += wstride) {
    const int r = (int)(item / jchunks), jc = (int)(item - (long)r * jchunks);
    const WalkEntry* krow = keys_g + (size_t)r * istride;
    const int n = __shfl_sync(0xffffffffu, ld_plain(nvalid_g + r), 0);
    float* yr = y_out + (size_t)r * J;
    float* ir = inv_out ? inv_out + (size_t)r * J : nullptr;
    walk_pairs<P, CH, false, FULL>(g, krow, n, w, jc * 64 * P, lane, yr, ir, sbuf, fin);
    __syncwarp();   // the next row's first block goes into the buffer this row may have read last
  }
}

// ---- the pairs walk with its weights staged in shared memory ---------------------------------------------
// Where all fan-in rows of 64 outputs fit into one CTA's shared memory ((I + bias) * 256 bytes beside 784 for each warp's list and the sums
// of its spikes), a persistent CTA of 32 warps copies that slice of the weight matrix in once -- one asynchronous bulk copy
// (cp.async.bulk) per weight row, all completing on one mbarrier -- and every step of every walk then reads its
// weight pair with one shared-memory load instead of a global load through L1. CTA c takes output slice
// c % (J/64) and every (gridDim.x / (J/64))-th row of that slice.
// Where that leaves less room than 32 warps need (from 803 rows on), the CTA has fewer, down to 21 at 835 rows: 65 536 rows of 821 -> 64, 26
// warps, 880 us, of 831 -> 64, 22 warps, 928 (walk from global memory 1020, 1031; 32 768 rows of 831, half of the inputs spiking, 285, 287).
constexpr int kSmemwThreads = 1024;
constexpr size_t kSmemwFewest = 20;                    // warps
constexpr size_t kSmemwWarpBytes = kPairsStage * sizeof(WalkEntry) + PairWalk<1>::kFloats * sizeof(float);
constexpr long long kSmemwWaitClocks = 2000000000LL;   // SM clocks a CTA waits for its weight copies (about a second)
__device__ unsigned g_walk_copy_timeouts = 0u;          // CTAs that gave up waiting since the library was loaded

__global__ void __launch_bounds__(kSmemwThreads, 1)
snn_walk2_smemw_kernel(const Geometry g, const WalkEntry* keys_g, const int* nvalid_g,
                       int istride, const float* w, float* __restrict__ out, unsigned wmul) {
  chain_wait();
  chain_next();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long copy_done;
  const int J = g.J, R = g.R;
  const int rows_w = g.I + g.has_bias;
  float* ws = reinterpret_cast<float*>(smem_raw);                                        // [rows_w][64]
  const int warps = blockDim.x >> 5;
  WalkEntry* stage = reinterpret_cast<WalkEntry*>(smem_raw + (size_t)rows_w * 256);      // [warps][kPairsStage]
  float* fins = reinterpret_cast<float*>(stage + warps * kPairsStage);                   // [warps][PairWalk<1>::kFloats]
  const int lane = threadIdx.x & 31;
  const int warp = uniform_warp_index();
  const int slices = J >> 6;
  const int slice = blockIdx.x % slices;
  const int j0 = slice << 6;
  const unsigned bar = smem_u32(&copy_done);

  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (warp == 0) {
    if (lane == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((unsigned)rows_w * 256u) : "memory");
    __syncwarp();
    for (int row = lane; row < rows_w; row += 32)
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 256, [%2];"
                   ::"r"(smem_u32(ws + row * 64)), "l"(__cvta_generic_to_global(w + (size_t)row * J + j0)), "r"(bar) : "memory");
  }
  // Every thread waits for the copies itself (phase 0 of the barrier), for at most about a second of SM clocks. If
  // they have not arrived by then the CTA counts a timeout and walks with the weights read from global memory, like
  // snn_walk_pairs_kernel; before it leaves it gives the copies the same time once more, so that none is in flight into
  // shared memory that the next CTA on this SM owns.
  auto copies_arrived = [&]() {
    const long long t0 = clock64();
    bool arrived = false;
    while (!arrived && clock64() - t0 < kSmemwWaitClocks) {
      unsigned ok;
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                   : "=r"(ok) : "r"(bar) : "memory");
      arrived = ok != 0u;
    }
    return arrived;
  };
  const bool staged = !__syncthreads_or(!copies_arrived());
  if (!staged && threadIdx.x == 0) atomicAdd(&g_walk_copy_timeouts, 1u);

  WalkEntry* sbuf = stage + warp * kPairsStage;
  float* fin = fins + warp * PairWalk<1>::kFloats;
  float* __restrict__ y_out = out;
  float* __restrict__ inv_out = g.infer ? nullptr : out + (size_t)R * J;
  const unsigned ws_lane = smem_u32(ws) + 8u * (unsigned)lane;
  const int ctas = gridDim.x / slices;                 // CTAs that share this slice (the host makes gridDim.x a multiple)
  const int cta = blockIdx.x / slices;
  for (int r = cta * warps + warp; r < R; r += ctas * warps) {
    const WalkEntry* krow = keys_g + (size_t)r * istride;
    const int n = __shfl_sync(0xffffffffu, ld_plain(nvalid_g + r), 0);
    float* yr = y_out + (size_t)r * J;
    float* ir = inv_out ? inv_out + (size_t)r * J : nullptr;
    if (staged) walk_pairs<1, 8, true>(g, krow, n, w, j0, lane, yr, ir, sbuf, fin, ws_lane, wmul);
    else walk_pairs<1, 8>(g, krow, n, w, j0, lane, yr, ir, sbuf, fin);
    __syncwarp();
  }
  if (!staged) {
    __syncthreads();
    (void)copies_arrived();
  }
}

int key_stride(const Geometry& g) { return (g.I + 3) & ~3; }  // a multiple of four entries: rows of keys start 32-byte aligned

size_t keys_bytes(const Geometry& g) { return (size_t)g.R * key_stride(g) * sizeof(u64); }
// list lengths, then 256 bytes that hold the weight bound of the walk (up to 64 partial sums)
size_t nvalid_only_bytes(const Geometry& g) { return ((size_t)g.R * sizeof(int) + 255) & ~(size_t)255; }
size_t nvalid_bytes(const Geometry& g) { return nvalid_only_bytes(g) + 256; }

template <int JPT>
int launch_walk(const Geometry& g, const WalkEntry* keys_g, const int* nvalid_g, const float* w, float* out,
                cudaStream_t s) {
  const int jchunks = (g.jout + 32 * JPT - 1) / (32 * JPT);
  const long items = (long)g.R * jchunks;
  long grid = (items + kFwdWarps - 1) / kFwdWarps;
  if (grid > 0x7fffffffL) grid = 0x7fffffffL;      // (a warp goes on to item + warps of the grid)
  (void)launch_chained(snn_walk_kernel<JPT>, (int)grid, kFwdThreads, 0, s, 0, g, keys_g, nvalid_g, key_stride(g), w, out);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? OK : E_CUDA;
}

template <int P>
int launch_walk_pairs(const Geometry& g, const WalkEntry* keys_g, const int* nvalid_g, const float* w, float* out, cudaStream_t s) {
  const long items = (long)g.R * ((g.jout + 64 * P - 1) / (64 * P));
  long grid = (items + kFwdWarps - 1) / kFwdWarps;
  if (grid > 0x7fffffffL) grid = 0x7fffffffL;      // (a warp goes on to item + warps of the grid)
  // FULL (no lane behind the row) for lists of at most 64 entries, where a row costs more to begin and to end than to walk: 94 248 rows of
  // 9 -> 128 with their lists 120 -> 112 us, 31 958 of 27 -> 256 97.7 -> 92.0. Long lists run slower in it (65 536 of 576 -> 128 628 -> 632).
  if (g.I <= 64 && g.jout % (64 * P) == 0)
    (void)launch_chained(snn_walk_pairs_kernel<P, true>, (int)grid, kFwdThreads, 0, s, 0, g, keys_g, nvalid_g, key_stride(g), w, out);
  else
    (void)launch_chained(snn_walk_pairs_kernel<P, false>, (int)grid, kFwdThreads, 0, s, 0, g, keys_g, nvalid_g, key_stride(g), w, out);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? OK : E_CUDA;
}

// The pairs walk with the weights staged in shared memory: fan-out a power-of-two multiple of 64, weights 16-byte
// aligned, all (I + bias) rows of a 64-output slice plus the list staging buffers within one CTA's shared memory.
bool walk_smemw_ok(const Geometry& g, const float* w, const LaunchInfo& li, int* warps, int* wmul) {
  if ((g.J != 64 && g.J != 128 && g.J != 256) || (reinterpret_cast<uintptr_t>(w) & 15) != 0) return false;
  if (g.jout != g.J) return false;      // J is the kernel's output stride too
  const size_t rows_w = (size_t)g.I + g.has_bias;
  const size_t room = (size_t)li.max_smem_optin - 2048;
  if (rows_w * 256 + kSmemwFewest * kSmemwWarpBytes > room) return false;
  if ((g.J >> 6) > li.num_sms) return false;
  *warps = (int)std::min<size_t>(kSmemwThreads / 32, (room - rows_w * 256) / kSmemwWarpBytes);
  *wmul = 256 / g.J;
  return true;
}

int launch_walk2_smemw(const Geometry& g, const WalkEntry* keys_g, const int* nvalid_g, const float* w, float* out,
                       const LaunchInfo& li, cudaStream_t s, int warps, int wmul) {
  const int slices = g.J >> 6;
  long per_slice = li.num_sms / slices;                       // persistent: one CTA per SM
  const long need = ((long)g.R + warps - 1) / warps;
  if (per_slice > need) per_slice = need;
  if (per_slice < 1) per_slice = 1;
  const int grid = (int)(per_slice * slices);
  const size_t smem = ((size_t)g.I + g.has_bias) * 256 + warps * kSmemwWarpBytes;
  if (allow_smem<snn_walk2_smemw_kernel>(smem) != cudaSuccess) return E_CUDA;
  (void)launch_chained(snn_walk2_smemw_kernel, grid, 32 * warps, smem, s, 0, g, keys_g, nvalid_g, key_stride(g), w, out, (unsigned)wmul);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? OK : E_CUDA;
}

// What a walk from global memory takes with n warps to an SM, in microseconds for rows of 500 inputs of which half spike: 32 warps
// run at once, each full wave of them takes `wave`, the last one first + n * warp. Fitted on the scalar steps, which one, two and four outputs
// lane + 32 m still take; with the packed ones pairs and quads became faster alike, and the choice between them was measured again: at 300 to 2304 inputs, half or all of them
// spiking, 400 to 20 000 rows and fan-outs 70 to 512, 89 sizes, the one it takes is never more than 4 % behind the other. They cross at about
// 32 warps of 64 outputs per SM (500 rows of 2304 -> 256: 89 us with pairs, 112 with quads, 1200 rows 166, 130).
struct WalkCost { double wave, first, warp; };
constexpr WalkCost kCostPairs = {27, 20, 0.6};                                        // 64 outputs per warp
constexpr WalkCost kCostQuads = {43, 29, 0.8};                                        // 128
constexpr WalkCost kCostLanes[3] = {{25, 20, 0.37}, {36, 21.5, 0.67}, {69, 30, 1.3}};    // 32, 64, 128 by 4-byte loads
double walk_cost(double n, const WalkCost& c) {
  const double waves = n > 32 ? ceil(n / 32) - 1 : 0;
  return waves * c.wave + c.first + (n - 32 * waves) * c.warp;
}

// Lists of a conv layer are built by per-pixel sorting and merging when the geometry allows it and there is enough to do:
// the bucket sort sorts every input pixel of a 3x3 stride-1 convolution nine times over, but spreads a small layer over the
// GPU, where the merges are three launches of long serial threads (64 fields of 2304 inputs: 46 against 7 us). The two cross at
// 4.7 M inputs over all fields for up to 128 channels, at 7 M for 256 and 13 M for 512.
bool use_merge_lists(const Geometry& g, const Options& opt, const LaunchInfo& li) {
  const int want = opt.list_builder & 3;
  if (want == 1 || want == 3 || !merge_lists_supported(g)) return false;
  if (want == 2) return true;
  const double line = 30000.0 * li.num_sms * (g.C > 170 ? g.C / 170.0 : 1.0);
  return (double)g.R * g.I > line;
}

// Short rows (a first layer on a few image channels) are sorted by a network in registers.
bool use_small_rows(const Geometry& g, const Options& opt) {
  const int want = opt.list_builder & 3;
  if (want == 1 || want == 2 || !small_rows_supported(g)) return false;
  return true;
}

}  // namespace

unsigned long long walk_copy_timeouts() {
  unsigned n = 0;
  if (cudaMemcpyFromSymbol(&n, g_walk_copy_timeouts, sizeof(n)) != cudaSuccess) note_cuda_error(cudaGetLastError());
  return n;
}

// Where the padded copy of the weights lies in the workspace (fan-out no multiple of four), behind the sorted lists, their
// lengths and (conv layers that qualify) the scratch of the merging list builder.
static size_t padded_weights_at(const Geometry& g) {
  return (keys_bytes(g) + nvalid_bytes(g) + (merge_lists_shape_ok(g) ? merge_lists_bytes(g) : 0) + 255) & ~(size_t)255;
}
static size_t padded_weights_bytes(const Geometry& g) {
  return (g.J & 3) == 0 ? 0 : (size_t)(g.I + 1) * ((g.J + 3) & ~3) * sizeof(float);
}

size_t forward_workspace_bytes(const Geometry& g) {
  return padded_weights_at(g) + padded_weights_bytes(g);
}

int launch_forward(const Geometry& g_in, const float* x, const float* w, float* out, void* ws, size_t ws_bytes,
                   const LaunchInfo& li, const Options& opt, cudaStream_t s) {
  if (!ws || ws_bytes < forward_workspace_bytes(g_in)) return E_WORKSPACE;
  WalkEntry* keys_g = static_cast<WalkEntry*>(ws);
  int* nvalid_g = reinterpret_cast<int*>(static_cast<unsigned char*>(ws) + keys_bytes(g_in));
  float* wbound = reinterpret_cast<float*>(static_cast<unsigned char*>(ws) + keys_bytes(g_in) + nvalid_only_bytes(g_in));
  void* merge_scratch = static_cast<unsigned char*>(ws) + keys_bytes(g_in) + nvalid_bytes(g_in);
  Geometry g = g_in;
  g.wbound = wbound;
  const int istride = key_stride(g);

  const int fparts = opt.forward_parts;
  g.jout = g.J;
  const bool own = opt.walk_layout == 0 && opt.walk_outputs == 0;    // the library's own choice
  const long ring_items = (long)g.R * ((g.J + 31) / 32);
  // A fan-out that is no multiple of four: with more than a few items, or more inputs than the 4-byte copies of the walk below
  // take as long over as one more launch (2 rows of 6852 -> 135: 176 -> 82 us with the sort, 30 of 991 -> 126: 36 -> 22, 20 of
  // 200 -> 501: 14 -> 12), the weights are copied with padded rows (by the kernel that reads them for the bound), so that every
  // walk reads them 16 bytes at a time. Up to 16 outputs a 4-byte copy brings two rows or more, which keeps up with the walk.
  const int jp = (g.J + 3) & ~3;
  // (from six items per SM on, four at up to 64 inputs: 800 to 1184 rows of 40 -> 10 6.2 to 6.3 us so, 6.5 to 7.1 by 4-byte copies, of
  // 400 -> 10 14.7 to 15.7, 14.2 to 16.6)
  const long pad_line = (g.J > 32 ? 8 : (g.I <= 64 ? 4 : 6)) * (long)li.num_sms;
  const bool pad = own && jp != g.J && (ring_items > pad_line || (g.I >= 200 && g.J > 16)) && (long long)(g.I + 1) * jp <= INT_MAX;
  const float* const w_in = w;
  float* const w_padded = reinterpret_cast<float*>(static_cast<unsigned char*>(ws) + padded_weights_at(g_in));
  if (pad) {
    w = w_padded;
    g.J = jp;
  }
  const bool copies16 = (g.J & 3) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
  // With few warps on an SM latency is what counts, with many the instructions per output. In turn:
  //   - the walk with a copying warp while its CTAs are one wave: six to an SM with two walking warps, four with four (784 -> 128, 592 rows
  //     27.6 us, each warp copying for itself 29.8, pairs walk 39; 740 rows, beyond, 35.3, 33.6, 41), for long lists two waves (4096 -> 256, 370
  //     rows 117, 123, 130; 2000 -> 256, 333 rows 64, 65, 70). For fan-outs up to 32, where a CTA is one walking warp and the copying one, up
  //     to six items (rows) per SM (784 -> 32, 888 rows 20.9, 24.4 and in blocks of 32 entries 22.0; 1184 rows 24.8, 25.6, 23.8), fewer where
  //     lists are short, for it takes longer to begin, and where rows are no whole sectors, since it copies past L1 (200 -> 24, 888 rows 12.2,
  //     12.2, 11.4; 40 -> 12, 592 rows 6.8, 5.8, 5.5; 40 -> 128, 592 rows 7.8, 6.7). Eight items where rows have to be copied 4 bytes at a time.
  //   - the walk whose warps copy for themselves, up to 24 items of 32 outputs per SM (21 at 300 to 1200 inputs; 784 -> 400 input spikes, 250
  //     rows, 22 items, 65, pairs walk 51; 100 -> 400, 273 rows, 24 items, 12.4, 14.0, 319 rows 14.0, 14.3), in blocks of 32 entries up to one wave of
  //     those (16 items) where lists are not short or the fan-out is not above 32 (2000 -> 64, 1036 rows 60, in blocks of 16 64; 400 -> 16, 1480 rows
  //     19.5, 20.5, pairs walk 51, 2960 rows (20 items) 30.1, 25.8, 37; 40 -> 256, 296 rows 8.0, 6.7).
  const long sms = li.num_sms;
  long line = 6;                                       // rows per SM of the walk with a copying warp at fan-outs up to 32
  if (g.I <= 64) line = (g.J & 7) ? 1 : 4;
  else if (g.I <= 256) line = (g.J & 7) ? 3 : 5;
  bool few = ring_items <= (copies16 ? line : 8) * sms;
  if (copies16 && g.J > 32) {
    const long pairs_of_warps = (long)g.R * ((g.J + 63) / 64);
    few = pairs_of_warps <= 6 * sms || (long)g.R * ((g.J + 127) / 128) <= 4 * sms;
    if (g.I <= 64) few = few && ring_items <= 10 * sms;
    if (g.I > 1200) few = few || (ring_items > 16 * sms && pairs_of_warps <= 12 * sms);
  }
  const bool ring = (opt.walk_layout & 16) != 0 || (own && few);
  const long most = (g.J > 32 && g.I > 300 && g.I <= 1200 ? 21 : 24) * sms;
  const bool alone = copies16 && ((opt.walk_layout & 384) != 0 || (own && !ring && ring_items <= most));
  const bool large = own ? ring_items <= 16 * sms && (g.J <= 32 || g.I > 400) : (opt.walk_layout & 256) != 0;
  // Several rows per warp for fan-out up to 64, where that leaves enough warps: 5 per SM at eight rows to a warp (fan-out 16;
  // 10 where the weights miss the L1 cache), 11 at four (32), 40 at two (64). With fewer the pairs walk, a warp per row, hides
  // its latencies better. Pairs against rows, us: 576 -> 16 4000 rows 35, 39, 7000 rows 53, 39; 576 -> 32 35, 37 and 54, 43; 147 -> 64 8000
  // rows 25, 27, 14 000 37, 35; 500 -> 64 8000 54, 61, 14 000 85, 85, -> 36 80, 76.
  bool rows = !ring && !alone && walk_rows_ok(g, w) && (own || (opt.walk_layout & 96) != 0);
  if (rows && own) {
    const int lanes = g.J > 32 ? 16 : (g.J > 16 ? 8 : 4);
    const long warps_per_sm = (long)g.R * lanes / 32 / li.num_sms;
    const bool in_l1 = (size_t)(g.I + 1) * g.J * sizeof(float) <= (size_t)128 << 10;
    rows = warps_per_sm >= (lanes == 16 ? 40 : (lanes == 8 ? 11 : (in_l1 ? 5 : 10)));
    // (65 536 rows of 576 x 64: 364 us with the pairs walk and its weights in shared memory, 380 so, but 16 384 rows 130 and 113;
    // 262 144 of 27 x 64: 222, 208, but 59 400 of 64 x 64 75, 83; where the weights do not fit shared memory the pairs walk from
    // global memory is ahead too: 65 536 of 900 x 64 649, 672)
    if (g.jout == 64 && g.I >= 64 && g.R >= 32768) rows = false;
  }
  // the walk's bound on the weight sums (see walk_tolerance_base), by up to 64 CTAs of 8192 weights and more beside the lists. (Lists
  // without a walk: whatever walk the next call names may need it.)
  WeightBound wb = {w_in, g.I + g.has_bias, g.jout, g.J, wbound, pad ? w_padded : nullptr, 0};
  if (!(ring || alone) || pad || !(fparts & 2)) {
    const long long n = (long long)wb.rows * g.J;
    // With few rows to sort the bound may take longer than they do: no more than 32 weight rows to a CTA then (a few weights each are
    // as long as 8192 weights; 401 x 10 by one CTA 40 us beside a sort of 5), and padded rows, which are copied by 4 bytes, count twice
    // (800 x 302 at 317 rows 45.0 us with the walk, 42 so). In front of many rows the CTAs only take their places (13 986 rows of 501 -> 52,
    // trained, 220 us with 4 CTAs, 222 with 16, 227 with 32).
    const bool hurry = g.R <= 4096;
    const long long ctas = std::max((n + 8191) / 8192 * (pad && hurry ? 2 : 1), wb.rows / (hurry ? 32LL : 128LL) + 1);
    wb.ctas = (int)std::min(ctas, 64LL);
    g.wbound_n = wb.ctas;
  }
  // Variants of the walk from global memory: 1 = output pairs in 64-bit registers, 64 outputs per warp; 3 = four consecutive outputs
  // per lane, 128 per warp; 2 = outputs lane + 32*m (odd fan-out, weights that are not even 8-byte aligned). More outputs per warp
  // share a step's list entry, address and vote, fewer make more warps: priced by walk_cost.
  const bool al8 = (g.J % 2 == 0) && (reinterpret_cast<uintptr_t>(w) % 8 == 0);
  const bool al16 = (g.J % 4 == 0) && (reinterpret_cast<uintptr_t>(w) % 16 == 0);
  auto cost = [&](int outputs, const WalkCost& c) {
    return walk_cost((double)g.R * ((g.J + outputs - 1) / outputs) / li.num_sms, c);
  };
  int variant = 2, lanes = 0;                          // lanes: variant 2 with 1, 2 or 4 outputs per lane
  for (int c = 1; c < 3; ++c)
    if (cost(32 << c, kCostLanes[c]) < cost(32 << lanes, kCostLanes[lanes])) lanes = c;
  if (al8) variant = al16 && g.J > 64 && cost(128, kCostQuads) < cost(64, kCostPairs) ? 3 : 1;
  // a layout that the call names, where the weights allow it
  const int named = opt.walk_layout & 3;
  if (named == 2 || (named == 1 && al8) || (named == 3 && al16)) variant = named;
  if (opt.walk_outputs >= 1 && opt.walk_outputs <= 3) lanes = opt.walk_outputs - 1;
  int smemw_warps = 0, smemw_mul = 0;
  // weights staged in shared memory: where they fit, for fan-out 64 with enough rows to keep one CTA of 32 warps per SM busy (walk alone,
  // 262 144 rows of 576 -> 64 1210 us, from global memory 1535). At fan-out 128 and 256 two and four staged slices are level with four
  // outputs per lane from global memory: 65 536 of 576 -> 128 630, 629, 131 072 with every input spiking 2222, 2197, 16 384 of 576 -> 256 325,
  // 320, of 768 -> 256 739, 738. walk_layout 8 asks for it wherever it fits, a named layout switches it off
  const bool smemw = walk_smemw_ok(g, w, li, &smemw_warps, &smemw_mul) &&
                     ((opt.walk_layout & 8) != 0 || ((opt.walk_layout & 3) == 0 && g.J == 64 && g.R >= 32768));
  // CTAs of the last kernel that builds the lists: eight rows each (sorting network), one row each (bucket sort of few rows), many
  const int list_ctas = use_merge_lists(g, opt, li) ? li.num_sms : (use_small_rows(g, opt) ? (g.R + 7) / 8 : g.R) + wb.ctas;
  auto walk = [&]() -> int {
    if (!(fparts & 2)) return OK;
    if (alone) return launch_walk_alone(g, keys_g, nvalid_g, key_stride(g), w, out, large, list_ctas, li, s);
    if (ring) return launch_walk_ring(g, keys_g, nvalid_g, key_stride(g), w, out, list_ctas, li, s);
    if (rows) return launch_walk_rows(g, keys_g, nvalid_g, key_stride(g), w, out, own ? g.J > 32 && g.R >= 32768 : (opt.walk_layout & 64) != 0, li, s);
    if (smemw) return launch_walk2_smemw(g, keys_g, nvalid_g, w, out, li, s, smemw_warps, smemw_mul);
    if (variant == 1) return launch_walk_pairs<1>(g, keys_g, nvalid_g, w, out, s);
    if (variant == 3) return launch_walk_pairs<2>(g, keys_g, nvalid_g, w, out, s);
    if (lanes == 0) return launch_walk<1>(g, keys_g, nvalid_g, w, out, s);
    if (lanes == 1) return launch_walk<2>(g, keys_g, nvalid_g, w, out, s);
    return launch_walk<4>(g, keys_g, nvalid_g, w, out, s);
  };

  if (use_merge_lists(g, opt, li)) {
    if (fparts & 1) {
      const int rc = launch_merge_lists(g, x, keys_g, nvalid_g, istride, merge_scratch, (opt.list_builder >> 2) - 1, wb, li, s);
      if (rc != OK) return rc;
    }
    return walk();
  }
  if (use_small_rows(g, opt)) {
    if (fparts & 1) {
      const int rc = launch_small_rows(g, x, keys_g, nvalid_g, istride, wb, li, s);
      if (rc != OK) return rc;
    }
    return walk();
  }

  if (fparts & 1) {
    const int rc = launch_row_sort(g, x, keys_g, nvalid_g, istride, wb, li, s);
    if (rc != OK) return rc;
  }
  return walk();
}

}  // namespace snntc

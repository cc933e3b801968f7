// The sorted walk for fan-out up to 64: several rows per warp, four consecutive outputs per lane.
//
// A walk that gives a warp to each (row, 64 outputs) leaves three quarters of it idle at fan-out 16 and pays a step's list entry,
// vote and branch for 64 outputs at best. Here 16, 8 or 4 lanes (for fan-out up to 64, 32, 16) take a row with its own list, so a
// warp's step advances 128 outputs whatever the fan-out. The steps are those of PairWalk (snntc_walk.cuh) with two pairs per lane:
// the same bits as every other walk. Rows of one warp are neighbours (receptive
// fields next to each other), so their lists are about equally long; behind the end of its list a row repeats its last input
// with weight zero, which changes no sum and can fire nothing.
// WS: all weights fit one CTA's shared memory beside lists and sums (177 KB, 708 rows of 64; 161 KB, 2 576 of 16): a persistent CTA of
// 32 warps per SM holds them, since rows of 64 to 256 bytes picked at random miss the L1 cache beside everything else that goes
// through it.
// What bounds it: instruction issue and the latency of a step's chain.
// Measured (B200, walk alone): against the pairs walk 65 536 rows of 144 -> 16 inputs 123 -> 51 us, of 288 -> 32: 223 -> 131; 61 440
// of 576 -> 48: 401 -> 346; 18 000 of 3136 -> 32: 1219 -> 743, all with scalar steps; with PairWalk 262 144 of 27 -> 64 265 -> 235 and
// 16 384 of 576 -> 64 109 -> 101. The weights in shared memory pay from fan-out 33 and 32 768 rows on.
#include "snntc_common.cuh"
#include "snntc_walk.cuh"

#include <limits.h>
#include <math_constants.h>
#include <type_traits>

namespace snntc {

namespace {

constexpr int kChunk = 4;                        // steps whose entries and weights are read together

template <int LPR>
struct Shape {
  static constexpr int rows = 32 / LPR;          // per warp
  static constexpr int block = LPR >= 16 ? 32 : 16;   // list entries staged per row
};


template <int LPR, bool WS>
__global__ void __launch_bounds__(WS ? 1024 : 256, WS ? 1 : 4)
snn_walk_rows_kernel(const Geometry g, const WalkEntry* lists, const int* nvalid, int istride,
                     const float* w, float* __restrict__ out) {
  chain_wait();
  chain_next();
  constexpr int RPW = Shape<LPR>::rows, BLK = Shape<LPR>::block, PER = BLK / LPR;
  constexpr int WARPS = (WS ? 1024 : 256) / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WalkEntry* stage_all = reinterpret_cast<WalkEntry*>(smem_raw);              // [warps][rows][BLK]
  float* fins = reinterpret_cast<float*>(smem_raw + (size_t)WARPS * RPW * BLK * sizeof(WalkEntry));       // [warps][kFloats]
  float* ws_smem = fins + WARPS * PairWalk<2>::kFloats;                                                    // [I + bias][J]
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int sub = lane / LPR, gl = lane % LPR;
  const int J = g.J, jout = g.jout;
  if constexpr (WS) {
    const size_t n16 = (size_t)(g.I + g.has_bias) * J / 4;
    for (size_t e = threadIdx.x; e < n16; e += 1024)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(ws_smem + 4 * e)), "l"(w + 4 * e) : "memory");
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  }
  WalkEntry* stage = stage_all + (size_t)(warp * RPW + sub) * BLK;
  float tolbase;                                  // see walk_tolerance_base in snntc_forward.cu
  {
    float b = lane < g.wbound_n ? ld_plain(g.wbound + lane) : 0.f;
    if (lane + 32 < g.wbound_n) b += ld_plain(g.wbound + lane + 32);
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) b += __shfl_xor_sync(0xffffffffu, b, d);
    tolbase = 4.76837158203125e-7f * (fabsf(g.theta) + b) * 1.0001f;
  }
  const int j = 4 * gl;
  const bool in_row = j < J;                      // J % 4 == 0
  const unsigned lane_off = in_row ? (unsigned)j : 0u;
  const char* wbytes = reinterpret_cast<const char*>(w);
  const unsigned ws_lane = smem_u32(ws_smem) + 4u * lane_off;
  auto load_weights = [&](unsigned eoff, uint64_t (&wv)[2]) {
    if constexpr (WS) {
      asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(wv[0]), "=l"(wv[1]) : "r"(4u * eoff + ws_lane));
    } else {
      const ulonglong2 v = ld_plain(reinterpret_cast<const ulonglong2*>(wbytes + (size_t)(eoff + lane_off) * 4u));
      wv[0] = v.x; wv[1] = v.y;
    }
  };
  PairWalk<2> pw;
  pw.fin = fins + warp * PairWalk<2>::kFloats + lane;

  const int groups = (g.R + RPW - 1) / RPW;
  for (int grp = blockIdx.x * WARPS + warp; grp < groups; grp += gridDim.x * WARPS) {
    const int r = grp * RPW + sub;
    const bool row_ok = r < g.R;
    const int n = row_ok ? ld_plain(nvalid + r) : 0;
    const int nmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
    const int nmin = (int)__reduce_min_sync(0xffffffffu, (unsigned)n);
    const WalkEntry* ents = lists + (size_t)(row_ok ? r : 0) * istride;
    // the bias input (value biasvolt, weight row I) is always consumed first
    {
      uint64_t b2[2] = {0, 0};
      if (g.has_bias) load_weights((unsigned)g.I * (unsigned)J, b2);
      float wb[4];
      unpack2(b2[0], wb[0], wb[1]);
      unpack2(b2[1], wb[2], wb[3]);
      bool ok[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) ok[m] = row_ok & (j + m < jout);   // (padding behind jout never fires: the walk would wait for it)
      const WalkEntry head = ld_l2(ents);
      pw.start(g, tolbase, n > 0 ? __uint_as_float(head.x) : 0.f, wb, ok);
    }
    float xprev = g.has_bias ? g.biasvolt : 0.f;

    // entries c .. c + 3 of the staged block; LAST: some row's list ends among them (`left` entries of this row are valid): behind its
    // end a row repeats its last input with weight zero
    auto chunk = [&](int c, int left, auto last_c, auto flip_c) {
      constexpr bool LAST = decltype(last_c)::value, FLIP = decltype(flip_c)::value;
      float xs[kChunk];
      uint64_t wv[kChunk][2];
#pragma unroll
      for (int u = 0; u < kChunk; u += 2) {
        const uint4 e2 = *reinterpret_cast<const uint4*>(stage + c + u);
        xs[u] = __uint_as_float(e2.x);
        xs[u + 1] = __uint_as_float(e2.z);
        unsigned o0 = e2.y, o1 = e2.w;
        if (LAST) {
          if (u >= left) { xs[u] = u > 0 ? xs[u > 0 ? u - 1 : 0] : xprev; o0 = 0u; }
          if (u + 1 >= left) { xs[u + 1] = xs[u]; o1 = 0u; }
        }
        load_weights(o0, wv[u]);
        load_weights(o1, wv[u + 1]);
        if (LAST) {
          if (u >= left) wv[u][0] = wv[u][1] = 0;
          if (u + 1 >= left) wv[u + 1][0] = wv[u + 1][1] = 0;
        }
      }
      auto inputs = [&](int u) { return make_float2(xs[u], u == 0 ? xprev : xs[u > 0 ? u - 1 : 0]); };
      pw.margin(xs[0], xs[kChunk - 1]);           // inputs ascend: |x| peaks at an end
#pragma unroll
      for (int u = 0; u < kChunk; u += 2) {
        const uint64_t xa = pack2(xs[u], xs[u]), xb = pack2(xs[u + 1], xs[u + 1]);
        if constexpr (FLIP) {
          pw.step<true>(xa, wv[u], [&] { return inputs(u); });
          pw.step<true>(xb, wv[u + 1], [&] { return inputs(u + 1); });
        } else {
          pw.step2(xa, wv[u], xb, wv[u + 1], [&] { return inputs(u); }, [&] { return inputs(u + 1); });
        }
      }
      xprev = xs[kChunk - 1];
    };

    WalkEntry pre[PER];
    auto read_block = [&](int base) {
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const int k = base + gl + q * LPR;
        pre[q] = make_uint2(0u, 0u);
        if (k < n) pre[q] = ld_l2(ents + k);
      }
    };
    read_block(0);
    bool flipped = false;
    for (int base = 0; base < nmax; base += BLK) {
      __syncwarp();
#pragma unroll
      for (int q = 0; q < PER; ++q) stage[gl + q * LPR] = pre[q];
      __syncwarp();
      if (base + BLK < nmax) read_block(base + BLK);
      if (__builtin_expect(flipped, 0)) {
#pragma unroll 1
        for (int c = 0; c < BLK && base + c < nmax; c += kChunk) chunk(c, n - base - c, std::true_type{}, std::true_type{});
        pw.flip<true>(xprev);
      } else {
#pragma unroll 1
        for (int c = 0; c < BLK && base + c < nmax; c += kChunk) {
          if (base + c + kChunk <= nmin) chunk(c, kChunk, std::false_type{}, std::false_type{});
          else chunk(c, n - base - c, std::true_type{}, std::false_type{});
        }
        flipped = pw.flip<false>(xprev);
      }
      if (pw.done()) break;   // every output has fired
    }

    float yo[4], io[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) pw.finish(g, m, xprev, yo[m], io[m]);
    if (row_ok && in_row) {
      float* yr = out + (size_t)r * jout + j;
      float* ir = yr + (size_t)g.R * jout;
      if ((jout & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && ((size_t)g.R * jout & 3) == 0) {
        *reinterpret_cast<float4*>(yr) = make_float4(yo[0], yo[1], yo[2], yo[3]);
        if (!g.infer) *reinterpret_cast<float4*>(ir) = make_float4(io[0], io[1], io[2], io[3]);
      } else {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          if (j + m < jout) {
            yr[m] = yo[m];
            if (!g.infer) ir[m] = io[m];
          }
        }
      }
      if (g.khist != nullptr) {
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (j + m < jout) atomicAdd(g.khist + (yo[m] < g.maxv ? entries_below(ents, n, yo[m]) : g.I + 1), 1);
      }
    }
  }
}

template <int LPR, bool WS>
int launch(const Geometry& g, const WalkEntry* lists, const int* nvalid, int istride, const float* w, float* out,
           const LaunchInfo& li, cudaStream_t s) {
  constexpr int threads = WS ? 1024 : 256, warps = threads / 32;
  const size_t smem = (size_t)warps * (Shape<LPR>::rows * Shape<LPR>::block * sizeof(WalkEntry) + PairWalk<2>::kFloats * sizeof(float)) +
                      (WS ? (size_t)(g.I + g.has_bias) * g.J * sizeof(float) : 0);
  if (allow_smem<snn_walk_rows_kernel<LPR, WS>>(smem) != cudaSuccess) return E_CUDA;
  const long groups = ((long)g.R + Shape<LPR>::rows - 1) / Shape<LPR>::rows;
  long grid = (groups + warps - 1) / warps;
  const long most = WS ? li.num_sms : 8L * li.num_sms;
  if (grid > most) grid = most;
  const cudaError_t e = launch_chained(snn_walk_rows_kernel<LPR, WS>, (unsigned)grid, threads, smem, s, 0, g, lists, nvalid, istride, w, out);
  count_launch();
  return e == cudaSuccess ? OK : E_CUDA;
}

template <int LPR>
int launch_lanes(const Geometry& g, const WalkEntry* lists, const int* nvalid, int istride, const float* w, float* out,
                 bool resident, const LaunchInfo& li, cudaStream_t s) {
  const size_t need = (size_t)32 * (Shape<LPR>::rows * Shape<LPR>::block * sizeof(WalkEntry) + PairWalk<2>::kFloats * sizeof(float)) +
                      (size_t)(g.I + g.has_bias) * g.J * sizeof(float);
  if (resident && need + 2048 <= (size_t)li.max_smem_optin) return launch<LPR, true>(g, lists, nvalid, istride, w, out, li, s);
  return launch<LPR, false>(g, lists, nvalid, istride, w, out, li, s);
}

}  // namespace

bool walk_rows_ok(const Geometry& g, const float* w) {
  return g.J <= 64 && (g.J & 3) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
}

int launch_walk_rows(const Geometry& g, const WalkEntry* lists, const int* nvalid, int istride, const float* w, float* out,
                     bool resident, const LaunchInfo& li, cudaStream_t s) {
  if (g.J > 32) return launch_lanes<16>(g, lists, nvalid, istride, w, out, resident, li, s);
  if (g.J > 16) return launch_lanes<8>(g, lists, nvalid, istride, w, out, resident, li, s);
  return launch_lanes<4>(g, lists, nvalid, istride, w, out, resident, li, s);
}

}  // namespace snntc

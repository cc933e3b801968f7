// The sorted walk for fan-out up to 64: several rows per warp, four consecutive outputs per lane.
//
// A walk that gives a warp to each (row, 64 outputs) leaves three quarters of it idle at fan-out 16 and pays a step's list entry,
// vote and branch for 64 outputs at best. Here 16, 8 or 4 lanes (for fan-out up to 64, 32, 16) take a row with its own list, so a
// warp's step advances 128 outputs whatever the fan-out. Per step and lane: q of four outputs, their smallest as an integer,
// one vote, and the reference's own comparisons (snntc/snnfc_kernels.cu.cc:46-55) where some q is at or near zero -- the
// arithmetic, order and decisions of walk_row in snntc_forward.cu: the same bits. Rows of one warp are neighbours (receptive
// fields next to each other), so their lists are about equally long; behind the end of its list a row repeats its last input
// with weight zero, which changes no sum and can fire nothing.
// WS: all weights fit one CTA's shared memory (up to 200 KB: 780 rows of 64, 3 100 of 16): a persistent CTA of 32 warps per SM
// holds them, since rows of 64 to 256 bytes picked at random miss the L1 cache beside everything else that goes through it.
// What bounds it: instruction issue, about 26 instructions per step of 128 outputs.
// Measured (B200, walk alone, before -> now): 65 536 rows of 144 -> 16 inputs 123 -> 51 us, of 288 -> 32: 223 -> 131; 61 440 of 576 ->
// 48: 401 -> 346; 18 000 of 3136 -> 32: 1219 -> 743. The weights in shared memory pay from fan-out 33 and 32 768 rows on.
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
  float* ws_smem = reinterpret_cast<float*>(smem_raw + (size_t)WARPS * RPW * BLK * sizeof(WalkEntry));   // [I + bias][J]
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
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) b += __shfl_xor_sync(0xffffffffu, b, d);
    tolbase = 4.76837158203125e-7f * (fabsf(g.theta) + b) * 1.0001f;
  }
  const int j = 4 * gl;
  const bool in_row = j < J;                      // J % 4 == 0
  const unsigned lane_off = in_row ? (unsigned)j : 0u;
  const char* wbytes = reinterpret_cast<const char*>(w);
  const unsigned ws_lane = smem_u32(ws_smem) + 4u * lane_off;
  auto load_weights = [&](unsigned eoff) -> float4 {
    if constexpr (WS) {
      float4 v;
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(4u * eoff + ws_lane));
      return v;
    } else {
      return ld_plain(reinterpret_cast<const float4*>(wbytes + (size_t)(eoff + lane_off) * 4u));
    }
  };

  const int groups = (g.R + RPW - 1) / RPW;
  for (int grp = blockIdx.x * WARPS + warp; grp < groups; grp += gridDim.x * WARPS) {
    const int r = grp * RPW + sub;
    const bool row_ok = r < g.R;
    const int n = row_ok ? ld_plain(nvalid + r) : 0;
    const int nmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
    const int nmin = (int)__reduce_min_sync(0xffffffffu, (unsigned)n);
    const WalkEntry* ents = lists + (size_t)(row_ok ? r : 0) * istride;
    // the bias input (value biasvolt, weight row I) is always consumed first
    float wsum[4] = {-g.theta, -g.theta, -g.theta, -g.theta}, ysum[4] = {0.f, 0.f, 0.f, 0.f};
    if (g.has_bias) {
      const float4 wb = load_weights((unsigned)g.I * (unsigned)J);
      wsum[0] += wb.x; wsum[1] += wb.y; wsum[2] += wb.z; wsum[3] += wb.w;
      ysum[0] = g.biasvolt * wb.x; ysum[1] = g.biasvolt * wb.y; ysum[2] = g.biasvolt * wb.z; ysum[3] = g.biasvolt * wb.w;
    }
    float wfin[4], yfin[4];
    int live[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      wfin[m] = 0.f; yfin[m] = 0.f;
      live[m] = row_ok && j + m < jout ? -1 : 0;   // (padding behind jout never fires: the walk would wait for it)
      if (live[m] == 0) wsum[m] = -CUDART_INF_F;
    }
    float xprev = g.has_bias ? g.biasvolt : 0.f;
    int sticky = INT_MAX, qlim = 0;

    auto step = [&](const float x, const float xp, const float4& w4) {
      const float wv[4] = {w4.x, w4.y, w4.z, w4.w};
      int q[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) q[m] = __float_as_int(fmaf(-x, wsum[m], ysum[m]));
      const int qmin = imin3(imin3(q[0], q[1], q[2]), q[3], sticky);
      if (__builtin_expect(__any_sync(0xffffffffu, qmin <= qlim), 0)) {
        bool again = false;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          if (!__any_sync(0xffffffffu, (q[m] <= qlim) | (sticky < 0))) continue;
          const bool lv = live[m] != 0;
          const bool fire = lv & ratio_gt(ysum[m], wsum[m], xp) & ratio_le(ysum[m], wsum[m], x);
          if (fire) {
            live[m] = 0;                          // spike lies in (previous input, x]: keep the sums aside and park the running ones
            wfin[m] = wsum[m];
            yfin[m] = ysum[m];
            wsum[m] = -CUDART_INF_F;
          }
          again |= lv & !fire & (q[m] <= qlim);
        }
        sticky = again ? INT_MIN : INT_MAX;
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        wsum[m] += wv[m];
        ysum[m] = fmaf(x, wv[m], ysum[m]);
      }
    };
    // entries c .. c + 3 of the staged block; LAST: some row's list ends among them (`left` entries of this row are valid)
    auto chunk = [&](int c, int left, auto last_c) {
      constexpr bool LAST = decltype(last_c)::value;
      float xs[kChunk];
      float4 wv[kChunk];
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
        wv[u] = load_weights(o0);
        wv[u + 1] = load_weights(o1);
        if (LAST) {
          if (u >= left) wv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (u + 1 >= left) wv[u + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      qlim = __float_as_int(tolbase * fmaxf(fabsf(xs[0]), fabsf(xs[kChunk - 1])));   // inputs ascend: |x| peaks at an end
#pragma unroll
      for (int u = 0; u < kChunk; ++u) step(xs[u], u == 0 ? xprev : xs[u > 0 ? u - 1 : 0], wv[u]);
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
    for (int base = 0; base < nmax; base += BLK) {
      __syncwarp();
#pragma unroll
      for (int q = 0; q < PER; ++q) stage[gl + q * LPR] = pre[q];
      __syncwarp();
      if (base + BLK < nmax) read_block(base + BLK);
#pragma unroll 1
      for (int c = 0; c < BLK && base + c < nmax; c += kChunk) {
        if (base + c + kChunk <= nmin) chunk(c, kChunk, std::false_type{});
        else chunk(c, n - base - c, std::true_type{});
      }
      if (!__any_sync(0xffffffffu, (live[0] | live[1] | live[2] | live[3]) != 0)) break;   // every output has fired
    }

    float yo[4], io[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      // an output that stopped has fired; one that consumed every input fires iff it is armed
      bool fired = true;
      float ws = wfin[m], yy = yfin[m];
      if (live[m]) {
        ws = wsum[m]; yy = ysum[m];
        fired = ratio_gt(yy, ws, xprev);
      }
      yo[m] = g.maxv; io[m] = 0.f;
      if (fired) {
        io[m] = __fdividef(1.0f, ws);
        yo[m] = yy * io[m];
        if (yo[m] >= g.maxv) { yo[m] = g.maxv; io[m] = 0.f; }
      }
    }
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
  const size_t smem = (size_t)warps * Shape<LPR>::rows * Shape<LPR>::block * sizeof(WalkEntry) +
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
  const size_t need = (size_t)32 * Shape<LPR>::rows * Shape<LPR>::block * sizeof(WalkEntry) + (size_t)(g.I + g.has_bias) * g.J * sizeof(float);
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

// Weight gradient of SnnCvGrad (snntc/snncvgrad_kernels.cu.cc:87-161) for stride-1 convolutions on a power-of-two
// number of channels: the row-skipping kernel of snntc_dw_skip.cu with its tiles brought in by the tensor memory
// accelerator instead of per-thread copies.
//
//   dW[i,j] = sum_r [x_ri <= y_rj] (x_ri - y_rj) u_rj,   u_rj = 0 wherever output (r,j) carries no gradient.
//
// As there, a warp owns FOUR output channels and every lane 4*QL fan-in rows, a CTA 64 (or 32) channels, a slice of the
// rows r (blockIdx.z) and a tile of the fan-in (blockIdx.y), and the rows of a stage of 16 whose four channels
// carry no gradient are skipped by a warp-uniform branch. What differs is how a stage gets into shared memory. In
// snn_dw_skip_kernel 160 threads issue sixteen 16-byte copies each per stage, with the tap arithmetic and the
// image-border tests in front of every copy -- a third of the instructions of the warps that also do the
// arithmetic. Here one tiled bulk copy per tap of the kernel window, a lane each, does it. A stage is a block of
// hseg x wseg = 16 receptive fields of one image (16 columns of one row of the output map, or 8 columns of two rows,
// ... where the map is narrower than 16): through tap (kh, kw) they read a box of [rows][columns][channels] of the
// NHWC image, which is exactly what a 4-D tensor map describes. Coordinates outside the image are legal for a load
// and read as the fill value -- NaN here, which behaves like an input that never spikes: the saturating FMA of the
// inner loop flushes a NaN to +0 (PTX .sat), and fmaxf(NaN, 0) of the unscaled loop is 0. The y and u tiles are two
// more boxes, of the outputs seen as [image][row][column][channel]; where the map's width or height is no multiple
// of the block, the fields past its edge read as u = 0 (zero fill) and are skipped like any field without a
// gradient. Every copy completes on the `full` mbarrier of its buffer; a warp waits for that (with a time limit),
// does its arithmetic and arrives on the buffer's `empty` barrier, which whoever refills the buffer waits for. Nothing
// holds the warps together stage by stage: how much a warp has to do depends on how many of its four channels carry
// gradients, and with a barrier per stage every warp took the time of the busiest (the largest stall of the kernel).
//
// What bounds it: the latency of a row's chain (read, test, FMAs) at four warps per scheduler, and the warp with the most to do. Which
// channels a warp owns is therefore dealt out by their activity (see `order`). With dW of 262 144 rows of 577 x 64, 12 % of the
// outputs carrying a gradient, 353 -> 256 us against two stages, a CTA barrier per stage, 32 outputs per CTA and eight waves of CTAs; 200 704
// x 1153 x 128 790 -> 658 us. Channels by activity instead of four neighbours (the whole dW, its u kernel and reduction with it): 262 144 x
// 577 x 64, 13 % active, 438 -> 378 us; 65 536 x 577 x 128, 36 % 410 -> 341; 16 384 x 1153 x 256, 36 % 461 -> 338; 65 536 x 1153 x 128, 13 %
// 360 -> 359 (the neighbours there are nearly even); 131 072 x 576 x 128, 79 % 1032 -> 1014.
//
// The x tile of a stage is laid out [tap][row][channel] (one box after the other), so a fan-in tile is made of
// whole taps, taps_per_tile = 640 / C of them; the bias row (x = biasvolt for every r) is a sum per output channel
// that the CTAs of the last fan-in tile keep beside their tile.
#include "snntc_common.cuh"
#include "snntc_ptx.cuh"

#include <cuda.h>
#include <math_constants.h>
#include <algorithm>
#include <mutex>
#include <type_traits>

namespace snntc {

namespace {

constexpr int kRS = 16;          // rows r per stage
constexpr int kMaxTileFloats = 640;
constexpr int kMaxDepth = 8;     // stages in flight at most
constexpr long long kWaitClocks = 2000000000LL;   // SM clocks a thread waits for a stage's copies (about a second)
__device__ unsigned g_dw_copy_timeouts = 0u;        // CTAs that gave up waiting since the library was loaded

// x box: coordinates (channel, column, row, image); the channel coordinate is always 0 (16-byte aligned)
__device__ __forceinline__ void tma_load_4d(unsigned dst, const CUtensorMap* map, unsigned bar, int c, int w, int h, int b) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c), "r"(w), "r"(h), "r"(b) : "memory");
}
// (the y / u boxes use the same instruction: coordinates (output channel, column, row, image), the channel
// coordinate a multiple of 32)

// C256: 256 channels (a chunk column is half a tap), else a power of two up to 128; NW warps
template <int QL, bool C256, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW)
snn_dw_tma_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_y,
                  const __grid_constant__ CUtensorMap map_u, const Geometry g, float* __restrict__ partial,
                  int stages_per_split, float scale, const int* exact_flag, int taps_per_tile,
                  int wseg_log2, int depth) {
  constexpr int kJT = 4 * NW;                                      // output channels per CTA, 4 per warp
  chain_wait();
  chain_next();
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long full[kMaxDepth], empty[kMaxDepth];
  __shared__ int gave_up;
  __shared__ __align__(16) int order[kJT];                         // output channels (of this CTA) by warp, four each
  __shared__ int active[kJT];
  __shared__ float4 own_all[NW][2][kRS];                           // a stage's u and y of each warp's four channels
  unsigned char* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // swizzled boxes: 1024-byte boundaries
  const int C = g.C, J = g.J, I = g.I;
  const int Itot = I + g.has_bias;
  const int taps = g.Kh * g.Kw;
  const int tap0 = blockIdx.y * taps_per_tile;
  const int ntap = max(0, min(taps_per_tile, taps - tap0));
  const bool bias_here = g.has_bias && blockIdx.y == gridDim.y - 1;
  const int xfloats = taps_per_tile * kRS * C;                     // floats of one x buffer
  float* Xs = reinterpret_cast<float*>(base);                      // [depth][taps_per_tile][kRS][C]
  float* Ys = Xs + ((depth * xfloats + 255) & ~255);               // [depth][kJT / 32][kRS][32], chunks swizzled (see at_field)
  float* Us = Ys + depth * kRS * kJT;                              // the same

  const bool fast = scale != 1.0f && ld_plain(exact_flag) == 0;
  const float sc = fast ? scale : 1.0f;                 // s
  const float nsc = -sc;
  const float nusc = fast ? -1.0f / scale : -1.0f;      // -1/s, exact: s is a power of two

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int j0 = blockIdx.x * kJT;
  // stages: blocks of hseg x wseg fields, column blocks fastest, then row blocks, then images
  const int wseg = 1 << wseg_log2, hseg = kRS >> wseg_log2;
  const int WB = (g.Nw + wseg - 1) >> wseg_log2, HB = (g.Nh + hseg - 1) / hseg;
  const int total_stages = g.B * HB * WB;
  const int s_begin = blockIdx.z * stages_per_split;
  const int nstages = max(0, min(total_stages, s_begin + stages_per_split) - s_begin);

  if (tid == 0) {
    for (int d = 0; d < depth; ++d) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[d])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&empty[d])), "r"(NW) : "memory");
    }
    gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();

  // The calling warp queues the copies of stage `st` into buffer `buf`, a box per lane: the taps, then the y box and the u box.
  auto issue = [&](int st, int buf) {
    const int sg = s_begin + st;
    const int nw0 = (sg % WB) << wseg_log2;
    const int t = sg / WB;
    const int nh0 = (t % HB) * hseg;
    const int b = t / HB;
    const unsigned bar = smem_u32(&full[buf]);
    if (lane == 0) {
      const unsigned bytes = (unsigned)(ntap * kRS * C + 2 * kRS * kJT) * 4u;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    }
    __syncwarp();
    for (int tl = lane; tl < ntap + 2 * (kJT / 32); tl += 32) {
      if (tl < ntap) {
        const int tap = tap0 + tl;
        const int kh = tap / g.Kw, kw = tap - kh * g.Kw;
        tma_load_4d(smem_u32(Xs + buf * xfloats + tl * kRS * C), &map_x, bar, 0, nw0 - g.pad_left + kw,
                    nh0 - g.pad_top + kh, b);
      } else {
        const int part = (tl - ntap) >> 1;          // 32 output channels
        float* to = ((tl - ntap) & 1 ? Us : Ys) + buf * kRS * kJT + part * kRS * 32;
        tma_load_4d(smem_u32(to), (tl - ntap) & 1 ? &map_u : &map_y, bar, j0 + 32 * part, nw0, nh0, b);
      }
    }
    __syncwarp();
  };
  // try_wait suspends the thread until the phase completes or a hardware time limit passes, so a waiting warp does
  // not take issue slots from the SM's other CTA; the clock bounds the number of attempts
  auto passed = [&](const unsigned long long* barrier, unsigned parity) {
    const unsigned bar = smem_u32(barrier);
    auto attempt = [&]() {
      unsigned ok;
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                   : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
      return ok != 0u;
    };
    bool arrived = attempt();
    if (!arrived) {
      const long long t0 = clock64();
      do arrived = attempt(); while (!arrived && clock64() - t0 < kWaitClocks);
    }
    return __all_sync(0xffffffffu, arrived) != 0;
  };

  // This lane's 16-byte chunks of the fan-in tile: chunk q = lane + 32c holds fan-in floats f = 4*lane + 128c of the
  // tile, i.e. channel f % C of tap f / C, at float (f / C)*16*C + f % C of row 0 of an x buffer. C is a power of two:
  // for C <= 128 a step of c is 128 / C whole taps (2048 floats), for C = 256 it is half a tap, so the offset is a
  // part that depends on the lane plus a compile-time constant per c. A chunk behind the tile's taps is read all
  // the same (what it reads lies inside the CTA's shared memory: the other x buffer or the y/u tiles) and its sums
  // are dropped at the end.
  const int lane_part = C256 ? 4 * lane : ((4 * lane) / C) * kRS * C + (4 * lane) % C;
  // the bias row: x = biasvolt for every r, one sum per output channel, kept by every lane alike (it takes two
  // instructions per row and channel beside the thirty of a fan-in chunk)
  float accb[4] = {0.f, 0.f, 0.f, 0.f};

  // acc[c][jj][h]: fan-in floats 4*lane + 128*c + 2h, +1 of the tile (one 64-bit pair), the warp's channel jj
  uint64_t acc[QL][4][2];
#pragma unroll
  for (int c = 0; c < QL; ++c)
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) acc[c][jj][0] = acc[c][jj][1] = pack2(0.f, 0.f);

  // float of field `row` and channel c in a y or u buffer: rows of 32 channels, whose 16-byte chunks the copy swizzles by the row, so
  // that a channel's 16 fields are read two at a time instead of one after the other
  auto at_field = [](int row, int c) { return (c >> 5) * (kRS * 32) + row * 32 + ((((c >> 2) ^ row) & 7) << 2) + (c & 3); };

  unsigned at01 = 0u, at23 = 0u;                  // where this lane's field of the warp's four channels lies in a buffer
  const float* const own_from = lane < kRS ? Us : Ys;

  auto reduce_stage = [&](int buf, auto fast_c) {
    constexpr bool FAST = decltype(fast_c)::value;
    const float* xb = Xs + buf * xfloats + lane_part;
    // The warp's four channels of the stage, a field per lane (lanes from 16 on: y), put side by side for the loop below. Which of the
    // 16 rows carry a gradient for one of the four: one vote.
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
      const float uu[4] = {u4.x, u4.y, u4.z, u4.w}, yv[4] = {y4.x, y4.y, y4.z, y4.w};
      float xr[QL][4];
      const float* xrow = xb + rl * C;
#pragma unroll
      for (int c = 0; c < QL; ++c) {
        const float4 v = *reinterpret_cast<const float4*>(xrow + (C256 ? (c >> 1) * kRS * 256 + (c & 1) * 128 : 2048 * c));
        xr[c][0] = v.x; xr[c][1] = v.y; xr[c][2] = v.z; xr[c][3] = v.w;
      }
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        if (uu[jj] == 0.f) continue;              // warp-uniform
        const float ys = yv[jj] * sc;
        const float nu = uu[jj] * nusc;
        const uint64_t nu2 = pack2(nu, nu);
        if (bias_here) accb[jj] = fmaf(FAST ? fma_sat(g.biasvolt, nsc, ys) : fmaxf(ys - g.biasvolt, 0.f), nu, accb[jj]);
#pragma unroll
        for (int c = 0; c < QL; ++c) {
          float t[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) t[k] = FAST ? fma_sat(xr[c][k], nsc, ys) : fmaxf(ys - xr[c][k], 0.f);
          acc[c][jj][0] = fma2(pack2(t[0], t[1]), nu2, acc[c][jj][0]);
          acc[c][jj][1] = fma2(pack2(t[2], t[3]), nu2, acc[c][jj][1]);
        }
      }
    }
  };

  // The warps are not held together by a barrier per stage: a warp that is through with a stage says so on the buffer's `empty`
  // barrier and goes on, ahead of the slowest by what is in flight. In turn, warp k mod NW when it comes to stage k, they wait
  // until everyone is through with stage k - lag and queue stage k - lag + depth in its place.
  const int first_stages = min(depth, nstages);
  for (int st = warp; st < first_stages; st += NW) issue(st, st);
  const int lag = min(2, depth - 1);
  bool failed = false;

  // Which four channels a warp takes. Channels differ in how often they carry a gradient (one in four never, one in four nearly
  // always), and a stage lasts as long as the warp with the most to do: of four neighbouring channels 1.7 to 2.2 times the mean, with
  // the channels dealt out in the order of their activity, forth and back, 1.05 to 1.2 times. The activity is counted over the first
  // stages, by every CTA for itself: which warp adds up a channel changes no sum.
  for (int d = 0; d < first_stages && !failed; ++d) failed = !passed(&full[d], 0u);
  if (tid < kJT) {
    int n = 0;
    if (!failed)
      for (int d = 0; d < first_stages; ++d)
#pragma unroll
        for (int row = 0; row < kRS; ++row) n += Us[d * kRS * kJT + at_field(row, tid)] != 0.f;
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
  failed = __syncthreads_or(failed) != 0;
  {
    const int4 ch = *reinterpret_cast<const int4*>(order + 4 * warp);
    const int row = lane & (kRS - 1);
    at01 = (unsigned)at_field(row, ch.x) | (unsigned)at_field(row, ch.y) << 16;
    at23 = (unsigned)at_field(row, ch.z) | (unsigned)at_field(row, ch.w) << 16;
  }

  int buf = 0, rbuf = depth - lag;        // buffers of stages it and it - lag
  unsigned phase = 0u, rphase = 1u;       // and the parities of their phases
  for (int it = 0; it < nstages && !failed; ++it) {
    if (it >= lag && it % NW == warp && it - lag + depth < nstages) {
      failed = !passed(&empty[rbuf], rphase);
      if (failed) break;
      issue(it - lag + depth, rbuf);
    }
    failed = !passed(&full[buf], phase);
    if (failed) break;
    if (fast) reduce_stage(buf, std::true_type{});
    else reduce_stage(buf, std::false_type{});
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty[buf])) : "memory");
    if (++buf == depth) { buf = 0; phase ^= 1u; }
    if (++rbuf == depth) { rbuf = 0; rphase ^= 1u; }
  }
  if (failed) gave_up = 1;
  __syncthreads();
  if (gave_up != 0) {
    // give the copies that may still be in flight the same time once more before the shared memory is handed on
    if (tid == 0) atomicAdd(&g_dw_copy_timeouts, 1u);
    const long long t0 = clock64();
    while (clock64() - t0 < kWaitClocks) {}
    __syncthreads();
  }

  // The sums go out through shared memory (no copy is in flight any more), where they are turned so that a row's channels lie
  // together: row (f % 4, f / 4) for fan-in float f of the tile, lanes on neighbouring rows.
  constexpr int kPitch = kJT + 1;
  float* turn = reinterpret_cast<float*>(base);
  {
    const int4 ch = *reinterpret_cast<const int4*>(order + 4 * warp);
    const int chs[4] = {ch.x, ch.y, ch.z, ch.w};
#pragma unroll
    for (int c = 0; c < QL; ++c) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          float a, b;
          unpack2(acc[c][jj][h], a, b);
          turn[((2 * h) * 32 * QL + 32 * c + lane) * kPitch + chs[jj]] = a;
          turn[((2 * h + 1) * 32 * QL + 32 * c + lane) * kPitch + chs[jj]] = b;
        }
      }
    }
    if (bias_here && lane == 0) {
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) turn[128 * QL * kPitch + chs[jj]] = accb[jj];
    }
  }
  __syncthreads();
  float* __restrict__ dst = partial + (size_t)blockIdx.z * Itot * J;
  const int j = j0 + 4 * (tid % NW);
  if (j < J) {
    for (int f = tid / NW; f <= ntap * C; f += 32) {
      const bool bias_row = f == ntap * C;
      if (bias_row && !bias_here) break;
      const float* from = turn + (bias_row ? 128 * QL : (f & 3) * 32 * QL + (f >> 2)) * kPitch + 4 * (tid % NW);
      const int i = bias_row ? I : tap0 * C + f;
      *reinterpret_cast<float4*>(dst + (size_t)i * J + j) = make_float4(from[0], from[1], from[2], from[3]);
    }
  }
}

struct TmaPlan { int taps_per_tile, ntiles, ql, nw, depth; size_t smem; };

TmaPlan plan(const Geometry& g) {
  TmaPlan p;
  const int taps = g.I / g.C > 0 ? g.I / g.C : 1;      // (a workspace query knows the fan-in, not the kernel window)
  int tpt = kMaxTileFloats / g.C;
  if (tpt < 1) tpt = 1;
  if (tpt > taps) tpt = taps;
  p.taps_per_tile = tpt;
  p.ntiles = (taps + tpt - 1) / tpt;                   // the bias row rides in the last tile
  p.ql = (tpt * g.C + 127) / 128;
  // 64 outputs per CTA read every input once for twice the outputs and leave room for four stages in flight; where that would
  // leave half of a last CTA without outputs, 32 and two CTAs per SM (96 outputs: 54 against 58 us)
  p.nw = (g.J & 63) == 0 || (g.J & 63) > 32 ? 16 : 8;
  const size_t stage = (size_t)kRS * (tpt * g.C + 8 * p.nw) * sizeof(float);
  const size_t room = (p.nw == 16 ? 216 : 106) * 1024;
  p.depth = (int)std::min<size_t>(kMaxDepth, room / stage);
  // (the tile of sums that goes out through the same memory: 640 fan-in rows and the bias row of 65 or 33 floats at most)
  p.smem = std::max(p.depth * stage, (size_t)(128 * p.ql + 1) * (4 * p.nw + 1) * sizeof(float)) + 2048;
  return p;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// the driver's cuTensorMapEncodeTiled, looked up once through the runtime (the library does not link libcuda)
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
    else
      (void)cudaGetLastError();
  });
  return fn;
}

// how the 16 fields of a stage are laid over the output map: wseg columns (a power of two, at most 16) x 16/wseg rows
int stage_wseg_log2(const Geometry& g) {
  int lg = 0;
  while ((1 << lg) < kRS && (1 << lg) < g.Nw) ++lg;
  return lg;
}
long stage_count(const Geometry& g) {
  const int lg = stage_wseg_log2(g);
  const int wseg = 1 << lg, hseg = kRS >> lg;
  return (long)g.B * ((g.Nh + hseg - 1) / hseg) * ((g.Nw + wseg - 1) / wseg);
}

template <int QL, bool C256, int NW>
int launch_ql(const CUtensorMap& mx, const CUtensorMap& my, const CUtensorMap& mu, const Geometry& g, float* partial,
              dim3 grid, int stages_per_split, float scale, const int* exact_flag, const TmaPlan& p, cudaStream_t s) {
  if (allow_smem<snn_dw_tma_kernel<QL, C256, NW>>(p.smem) != cudaSuccess)
    return E_CUDA;
  (void)launch_chained(snn_dw_tma_kernel<QL, C256, NW>, grid, 32 * NW, p.smem, s, 0, mx, my, mu, g, partial, stages_per_split, scale, exact_flag,
                       p.taps_per_tile, stage_wseg_log2(g), p.depth);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? OK : E_CUDA;
}

}  // namespace

bool dw_tma_shape_ok(const Geometry& g) {
  if (!g.is_conv || g.Sh != 1 || g.Sw != 1) return false;
  if (g.C < 4 || g.C > 256 || (g.C & (g.C - 1)) != 0 || (g.J & 3) != 0) return false;   // channels: a power of two
  if (g.Nh < 1 || g.Nw < 1 || g.B < 1) return false;
  if ((long long)g.B * g.H * g.W * g.C > 0x7fffffffLL) return false;
  if (stage_count(g) > 0x7fffffffL) return false;
  return true;
}

bool dw_tma_supported(const Geometry& g, const float* x, const float* uv, const float* out) {
  if (!dw_tma_shape_ok(g)) return false;
  if (((uintptr_t)x | (uintptr_t)uv | (uintptr_t)out) & 15) return false;
  return encode_tiled() != nullptr;
}

// The stages are cut into `return value` slices of *stages_per_split stages each (blockIdx.z).
int dw_tma_splits(const Geometry& g, const LaunchInfo& li, int* stages_per_split) {
  const TmaPlan p = plan(g);
  const long tiles = (long)p.ntiles * ((g.J + 4 * p.nw - 1) / (4 * p.nw));
  const long stages = stage_count(g);
  // one wave of CTAs (512 threads per SM): what a second one evens out is less than what its start and its planes cost (15 layers,
  // sum of the times with 1, 2, 4 and 8 waves: 4829, 4968, 5107, 5511 us)
  long want = std::max(1L, 16L / p.nw * li.num_sms / tiles);
  if (want > stages) want = stages;
  if (want > 1024) want = 1024;
  if (want < 1) want = 1;
  const long sps = (stages + want - 1) / want;
  *stages_per_split = (int)sps;
  return (int)((stages + sps - 1) / sps);
}

int launch_dw_tma(const Geometry& g, const float* uv, const float* x, const float* out, float* partial, int splits,
                  int stages_per_split, float scale, const int* exact_flag, cudaStream_t s) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return E_UNSUPPORTED;
  const TmaPlan p = plan(g);
  const int lg = stage_wseg_log2(g);
  const cuuint32_t wseg = 1u << lg, hseg = (cuuint32_t)kRS >> lg;
  const cuuint32_t jt = 4u * p.nw;   // output channels per CTA, copied 32 at a time (128 bytes: a swizzle's width)
  const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
  CUtensorMap mx, my, mu;
  {
    const cuuint64_t dims[4] = {(cuuint64_t)g.C, (cuuint64_t)g.W, (cuuint64_t)g.H, (cuuint64_t)g.B};
    const cuuint64_t strides[3] = {(cuuint64_t)g.C * 4, (cuuint64_t)g.W * g.C * 4, (cuuint64_t)g.H * g.W * g.C * 4};
    const cuuint32_t box[4] = {(cuuint32_t)g.C, wseg, hseg, 1u};
    if (enc(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(x), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NAN_REQUEST_ZERO_FMA) != CUDA_SUCCESS)
      return E_UNSUPPORTED;
  }
  {
    // the outputs as [image][row][column][channel]: fields past the edge of the map read as zero
    const cuuint64_t dims[4] = {(cuuint64_t)g.J, (cuuint64_t)g.Nw, (cuuint64_t)g.Nh, (cuuint64_t)g.B};
    const cuuint64_t strides[3] = {(cuuint64_t)g.J * 4, (cuuint64_t)g.Nw * g.J * 4, (cuuint64_t)g.Nh * g.Nw * g.J * 4};
    const cuuint32_t box[4] = {32u, wseg, hseg, 1u};
    if (enc(&my, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(out), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return E_UNSUPPORTED;
    if (enc(&mu, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(uv), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return E_UNSUPPORTED;
  }
  dim3 grid((g.J + jt - 1) / jt, p.ntiles, splits);
  auto run = [&](auto launch) { return launch(mx, my, mu, g, partial, grid, stages_per_split, scale, exact_flag, p, s); };
  auto pick = [&](auto nw) {
    constexpr int NW = decltype(nw)::value;
    if (g.C == 256)   // tiles of one or two taps: 2 or 4 chunk columns
      return p.ql <= 2 ? run(launch_ql<2, true, NW>) : run(launch_ql<4, true, NW>);
    switch (p.ql) {
      case 1: return run(launch_ql<1, false, NW>);
      case 2: return run(launch_ql<2, false, NW>);
      case 3: return run(launch_ql<3, false, NW>);
      case 4: return run(launch_ql<4, false, NW>);
      default: return run(launch_ql<5, false, NW>);
    }
  };
  return p.nw == 16 ? pick(std::integral_constant<int, 16>{}) : pick(std::integral_constant<int, 8>{});
}

unsigned long long dw_copy_timeouts() {
  unsigned n = 0;
  if (cudaMemcpyFromSymbol(&n, g_dw_copy_timeouts, sizeof(n)) != cudaSuccess) note_cuda_error(cudaGetLastError());
  return n;
}

}  // namespace snntc

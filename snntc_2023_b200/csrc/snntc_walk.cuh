// What the walk kernels share: the reference's fire comparisons, the causal-set size, the integer minimum of a step's sign test, and the
// steps of a walk with a lane's outputs in pairs (PairWalk) and with one output per lane (LaneWalk).
#pragma once
#include "snntc_common.cuh"
#include "snntc_ptx.cuh"

#include <limits.h>
#include <math_constants.h>

namespace snntc {

// "ysum/wsum > c" without a division, as the reference evaluates it after consuming input c
// (snntc/snnfc_kernels.cu.cc:53-55)
__device__ __forceinline__ bool ratio_gt(float ysum, float wsum, float c) {
  const float wa = fabsf(wsum);
  const float ya = wsum < 0.f ? -ysum : ysum;
  return ya > c * wa;
}
// "ysum/wsum <= c" (snntc/snnfc_kernels.cu.cc:46-48)
__device__ __forceinline__ bool ratio_le(float ysum, float wsum, float c) {
  const float wa = fabsf(wsum);
  const float ya = wsum < 0.f ? -ysum : ysum;
  return ya <= c * wa;
}

// Number of list entries whose input value lies strictly below y: the causal-set size of an output that fired
// at y (every consumed input is below the spike value, every other one is not). Binary search, one thread.
__device__ __forceinline__ int entries_below(const WalkEntry* ents, int n, float y) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__uint_as_float(ld_l2(ents + mid).x) < y) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Smallest of three float bit patterns compared as signed integers. For the sign test of the walks that is all that is needed:
// the result is <= 0 exactly when one of the floats is negative, -0 or +0 (negative floats are negative integers, +0 is 0,
// positive floats and NaN patterns with a clear sign bit are positive integers).
__device__ __forceinline__ int imin3(int a, int b, int c) { return min(min(a, b), c); }

// The outputs of one lane as P pairs in 64-bit registers, walked with the two-lane FP32 instructions: q, the weight sum and the
// weighted sum of two outputs are one instruction each. The weight sum is carried NEGATED (n = theta - sum w), so that
// q = fma(x, n, ysum) needs no negated copy of x; negation is exact, so every value is bit for bit the scalar walk's -- except the
// sign of an exactly cancelled sum, which is why it is read back as 0 - n: 1/(+0) = +inf clamps to "no spike", 1/(-0) would not.
//
// Two steps share a vote. Where it finds some q at or below the margin tol, nearly always an output has q < -tol, and that output
// has fired, without the reference's comparisons: let X bound the inputs consumed so far (0 <= inputs, ascending; |biasvolt|),
// tol = 8 * 2^-24 * X * (|theta| + B) with |sum w - theta| <= |theta| + B and |ysum| <= X * B.
//   - the step before left q > tol (an output that did not is `again`, below), i.e. ysum' - x' wsum' > tol. Consuming x' rounds
//     ysum and wsum once each and the reference rounds x' * wsum: together at most 3 * 2^-24 * X * (|theta| + B), so the
//     reference sees ysum > x' * wsum;
//   - q < -tol leaves ysum <= x * wsum whatever way that product is rounded;
//   - q fell from above tol to below -tol with x' <= x: wsum > 0.
// So "armed" and "fire" both hold. An output within tol of zero, of either sign, is taken through the reference's rounded
// comparisons (exact()); if it does not fire there, so is every output of the lane at the next step (`again`), and so is the first
// step of a row. Rows for which X is no bound (an input below zero, a NaN, or sums that may overflow: `careful`) take the
// comparisons whenever q <= tol. An output that has fired is parked at n = +inf: q = +inf (x > 0) or a positive NaN (x = 0) from
// then on, or a NaN behind a weight that is infinite or NaN, where nothing fires again either. So n tells who need not be waited for,
// and whether there is a spike to write is read beside its sums, in shared memory (as registers they took the walk beyond its 64).
//
// An output may also cross zero without firing (the two rounded comparisons of the reference can both miss it, about once in 10^5
// spikes) and then stays below, taking its row through the comparisons at every step: twice the time of its neighbours, and where
// the rows are one wave, of the whole launch. So between two blocks such an output changes the sign of its sums (flip()). Its q is
// positive again, and below -tol it fires again: q rose through zero, the denominator is NEGATIVE, and the proof above holds with
// both signs turned. From then on the row is walked by the FLIP steps, which give the weights each output's sign.
// Measured (B200, walk alone, scalar steps with a vote each -> now), four outputs per lane from global memory: 1024 rows of 784 -> 400 130 -> 109
// us, 65 536 of 576 -> 128 687 -> 629, 16 384 of 2304 -> 256 1243 -> 1107; instructions per step of 128 outputs 24.5 -> 17.4 where nothing
// fires. One pair per lane: 262 144 of 576 -> 64 1632 -> 1535, 250 of 4096 -> 512 158 -> 127, with the weights in shared memory 262 144 of
// 576 -> 64 1384 -> 1210. Rows with an input below zero, where every spike is compared: 16 384 of 576 -> 128 186 -> 220 (scalar 206).
// Asking shared memory after every block which outputs have fired took 0.5 to 3 % more; a second copy of the walk in the kernel, for warps
// without lanes behind the row, up to 20 % (784 -> 400 at 256 rows by pairs 62 us, 51 with one copy).
// What bounds it: the chain q - minimum - vote - branch at 32 warps per SM (issue slots 64 % busy) and the FMA pipe that takes the packed
// instructions.
template <int P>
struct PairWalk {
  static constexpr int kFloats = 128 * P;   // of shared memory per warp
  uint64_t n[P], ys[P];
  float* fin;       // this lane's column of [2 * P][2][32] floats: an output's sums once it has fired; until then the sign that its
                    // running sums carry, and a NaN (the sums of a spike are numbers: both ways to it have compared them)
  float tolbase, xmag;
  int qlim;         // bits of tol, or INT_MAX: every output of this lane goes to the comparisons at the next step
  int qtol;         // bits of tol
  bool careful;     // q < -tol is no proof in this row

  // sums with the bias input consumed (value biasvolt, weight wb), which is always the first; first: the row's smallest input
  __device__ __forceinline__ void start(const Geometry& g, float tolerance_base, float first, const float (&wb)[2 * P],
                                        const bool (&ok)[2 * P]) {
    tolbase = tolerance_base;
    xmag = g.has_bias ? fabsf(g.biasvolt) : 0.f;
    careful = !(first >= 0.f) | !(tolbase * 4194304.f * fmaxf(xmag, fabsf(g.maxv)) < CUDART_INF_F);   // 2^22 tolbase = 2 (|theta| + B)
    qlim = INT_MAX;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      float nn[2], yy[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = 2 * p + h;
        nn[h] = ok[m] ? g.theta - wb[m] : CUDART_INF_F;   // (no output: parked, or the walk would wait for it)
        yy[h] = g.has_bias ? g.biasvolt * wb[m] : 0.f;
        fin[64 * m] = 1.f; fin[64 * m + 32] = CUDART_NAN_F;
      }
      n[p] = pack2(nn[0], nn[1]);
      ys[p] = pack2(yy[0], yy[1]);
    }
  }
  // the margin of steps whose inputs lie in [x0, x1]
  __device__ __forceinline__ void margin(float x0, float x1) {
    const float a = fmaxf(xmag, fabsf(x0)), b = fabsf(x1);
    qtol = __float_as_int(tolbase * (b <= a ? a : b));     // (a NaN for a NaN at the end of the list)
    if (qlim != INT_MAX) qlim = qtol;
  }
  // no output of the warp may fire any more (one whose weight sum has overflowed to -inf cannot)
  __device__ __forceinline__ bool done() const {
    bool live = false;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      float a, b;
      unpack2(n[p], a, b);
      live |= (a != CUDART_INF_F) | (b != CUDART_INF_F);
    }
    return !__any_sync(0xffffffffu, live);
  }

  // ---- one or two steps. x2: the input twice; inputs() gives the input and the one in front of it, for the comparisons
  template <bool FLIP, typename Inputs>
  __device__ __forceinline__ void step(uint64_t x2, const uint64_t (&w)[P], Inputs&& inputs) {
    int q[2 * P];
    form_q(x2, n, ys, q);
    if (__builtin_expect(__any_sync(0xffffffffu, smallest(q) <= qlim), 0)) {
      uint64_t n0[P];
#pragma unroll
      for (int p = 0; p < P; ++p) n0[p] = n[p];
      hit<FLIP>(q, n0, ys, n, inputs);
    }
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const uint64_t ws = FLIP ? mul2(w[p], signs(p)) : w[p];
      n[p] = sub2(n[p], ws);
      ys[p] = fma2(x2, ws, ys[p]);
    }
  }
  template <typename InputsA, typename InputsB>
  __device__ __forceinline__ void step2(uint64_t xa, const uint64_t (&wa)[P], uint64_t xb, const uint64_t (&wb)[P], InputsA&& ia,
                                        InputsB&& ib) {
    int qa[2 * P], qb[2 * P];
    uint64_t n1[P], ys1[P];
    form_q(xa, n, ys, qa);
#pragma unroll
    for (int p = 0; p < P; ++p) {
      n1[p] = sub2(n[p], wa[p]);
      ys1[p] = fma2(xa, wa[p], ys[p]);
    }
    form_q(xb, n1, ys1, qb);
    int m;
    if constexpr (P == 1) m = min(imin3(qa[0], qa[1], qb[0]), qb[1]);
    else m = min(imin3(qa[0], qa[1], qa[2]), imin3(imin3(qa[3], qb[0], qb[1]), qb[2], qb[3]));
    if (__builtin_expect(__any_sync(0xffffffffu, m <= qlim), 0)) {
      if (__any_sync(0xffffffffu, smallest(qa) <= qlim)) {
        hit<false>(qa, n, ys, n1, ia);
        form_q(xb, n1, ys1, qb);
      }
      if (__any_sync(0xffffffffu, smallest(qb) <= qlim)) {
        uint64_t n0[P];
#pragma unroll
        for (int p = 0; p < P; ++p) n0[p] = n1[p];
        hit<false>(qb, n0, ys1, n1, ib);
      }
    }
#pragma unroll
    for (int p = 0; p < P; ++p) {
      n[p] = sub2(n1[p], wb[p]);
      ys[p] = fma2(xb, wb[p], ys1[p]);
    }
  }

  // Between two blocks: outputs below zero that have not fired change their sign. xprev: the last input consumed. FLIP: the warp
  // has such outputs already. Returns whether it has any.
  template <bool FLIP>
  __device__ __forceinline__ bool flip(float xprev) {
    const bool look = (qlim == INT_MAX) & !careful;
    if (__builtin_expect(!__any_sync(0xffffffffu, look), 1)) return FLIP;
    const float tol = __int_as_float(qtol);
    bool any = false, sure = look;                        // sure: no live output of this lane is within the margin any more (a NaN never fires)
    int q[2 * P];
    form_q(pack2(xprev, xprev), n, ys, q);
#pragma unroll
    for (int p = 0; p < P; ++p) {
      float nn[2], s[2];
      unpack2(n[p], nn[0], nn[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float qm = __int_as_float(q[2 * p + h]);
        const bool live = nn[h] != CUDART_INF_F, below = look & live & (qm < -tol);
        s[h] = below ? -1.f : 1.f;
        if (below) fin[64 * (2 * p + h)] *= -1.f;
        any |= below;
        sure &= !live | !(fabsf(qm) <= tol);
      }
      n[p] = mul2(n[p], pack2(s[0], s[1]));
      ys[p] = mul2(ys[p], pack2(s[0], s[1]));
    }
    __syncwarp();
    if (sure) qlim = qtol;
    return FLIP | (bool)__any_sync(0xffffffffu, any);
  }

  // spike value and 1/(sum w - theta) of output m once the list is consumed: an output that stopped has fired; one that consumed
  // every input fires iff it is armed
  __device__ __forceinline__ void finish(const Geometry& g, int m, float xprev, float& y, float& inv) const {
    float nn[2], yy[2];
    unpack2(n[m / 2], nn[0], nn[1]);
    unpack2(ys[m / 2], yy[0], yy[1]);
    float a = fin[64 * m], ws = 0.f - a, yv = fin[64 * m + 32];
    bool fired = true;
    if (yv != yv) {
      ws = 0.f - a * nn[m & 1]; yv = a * yy[m & 1];
      fired = (nn[m & 1] != CUDART_INF_F) & ratio_gt(yv, ws, xprev);
    }
    y = g.maxv; inv = 0.f;
    if (fired) {
      inv = __fdividef(1.0f, ws);
      y = yv * inv;
      if (y >= g.maxv) { y = g.maxv; inv = 0.f; }
    }
  }

 private:
  static __device__ __forceinline__ void form_q(uint64_t x2, const uint64_t (&n)[P], const uint64_t (&ys)[P], int (&q)[2 * P]) {
#pragma unroll
    for (int p = 0; p < P; ++p) unpack2i(fma2(x2, n[p], ys[p]), q[2 * p], q[2 * p + 1]);
  }
  static __device__ __forceinline__ int smallest(const int (&q)[2 * P]) {
    return P == 1 ? min(q[0], q[1]) : min(imin3(q[0], q[1], q[2 * P - 2]), q[2 * P - 1]);
  }
  // signs of a pair (of an output that has fired: the sign of a sum, which its parked n does not feel)
  __device__ __forceinline__ uint64_t signs(int p) const { return pack2(copysignf(1.f, fin[128 * p]), copysignf(1.f, fin[128 * p + 64])); }
  // true sums of a pair
  template <bool FLIP>
  __device__ __forceinline__ void sums(const uint64_t (&n)[P], const uint64_t (&ys)[P], int p, float (&nn)[2], float (&yy)[2]) const {
    unpack2(FLIP ? mul2(n[p], signs(p)) : n[p], nn[0], nn[1]);
    unpack2(FLIP ? mul2(ys[p], signs(p)) : ys[p], yy[0], yy[1]);
  }
  // both sums of an output that fires. Predicated, and with the park added to n instead of put in its place: a branch here, or halves
  // of n that are written alone, cost a divergence check per vote and copies of all sums per step
  static __device__ __forceinline__ void store_if(bool fire, float* to, float a, float b) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.f32 [%1], %2;\n\t@p st.shared.f32 [%1 + 128], %3;\n\t}"
                 ::"r"((unsigned)fire), "r"(smem_u32(to)), "f"(a), "f"(b) : "memory");
  }
  // a step whose vote has passed. n0, ys0: the sums in front of it; what fires is parked in n1
  template <bool FLIP, typename Inputs>
  __device__ __forceinline__ void hit(const int (&q)[2 * P], const uint64_t (&n0)[P], const uint64_t (&ys0)[P], uint64_t (&n1)[P],
                                      Inputs&& inputs) {
    const float tol = careful ? CUDART_NAN_F : __int_as_float(qlim);   // (INT_MAX is a NaN, too: nothing below fires)
    float near = CUDART_INF_F;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      float nn[2], yy[2], park[2];
      sums<FLIP>(n0, ys0, p, nn, yy);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = 2 * p + h;
        const float qm = __int_as_float(q[m]);
        park[h] = qm < -tol ? CUDART_INF_F : 0.f;
        store_if(qm < -tol, fin + 64 * m, nn[h], yy[h]);
        near = fminf(near, fabsf(qm));
      }
      n1[p] = add2(n1[p], pack2(park[0], park[1]));
    }
    if (__any_sync(0xffffffffu, !(near > tol))) {
      const float2 xx = inputs();
      exact<FLIP>(q, tol, n0, ys0, n1, xx.x, xx.y);
    }
  }
  // the reference's own comparisons, for all outputs of the lanes concerned that have not fired
  template <bool FLIP>
  __device__ __forceinline__ void exact(const int (&q)[2 * P], float tol, const uint64_t (&n0)[P], const uint64_t (&ys0)[P], uint64_t (&n1)[P],
                                        float x, float xp) {
    bool again = false;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      float nn[2], yy[2], before[2], park[2] = {0.f, 0.f};
      sums<FLIP>(n0, ys0, p, nn, yy);
      unpack2(n0[p], before[0], before[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m = 2 * p + h;
        if (!__any_sync(0xffffffffu, q[m] <= qlim)) continue;
        const bool live = (before[h] != CUDART_INF_F) & !(__int_as_float(q[m]) < -tol);   // (below: parked by hit())
        const float wsum = 0.f - nn[h];
        const bool fire = live & ratio_gt(yy[h], wsum, xp) & ratio_le(yy[h], wsum, x);
        park[h] = fire ? CUDART_INF_F : 0.f;
        store_if(fire, fin + 64 * m, nn[h], yy[h]);
        again |= live & !fire & (q[m] <= qtol);
      }
      n1[p] = add2(n1[p], pack2(park[0], park[1]));
    }
    qlim = again ? INT_MAX : qtol;
  }
};

// One output of one lane, for walks that are bound by the latency of the chain of sums: the sums and sign tests of G steps are formed
// before one vote. wsum = sum w - theta and ysum = sum w*x run on; an output that has fired keeps its sums in fin and its running
// weight sum at -inf, where q stays +inf. The margin of a sign test is 2^-22 |x * sum w|, formed from the output's own sum -- four
// times the rounding error of the reference's product x * sum w, so every step that rounding could decide goes to the
// reference's comparisons, and no bound over the weight matrix is needed.
struct LaneWalk {
  float wsum, ysum;       // times sign
  float2 fin;
  bool live;
  int sticky;             // INT_MIN: the output was at or near zero at the last entry without firing, else INT_MAX
  float xprev;
  float sign;             // -1: the output has crossed zero without firing (turn)

  // sums with the bias input consumed (value biasvolt, weight wb), which is always the first; not ok: no output, nothing waits for it
  __device__ __forceinline__ void start(const Geometry& g, bool ok, float wb) {
    wsum = -g.theta;
    ysum = 0.f;
    if (g.has_bias) {
      wsum += wb;
      ysum = g.biasvolt * wb;
    }
    if (!ok) wsum = -CUDART_INF_F;
    live = ok;
    fin = make_float2(0.f, 0.f);
    sticky = INT_MAX;
    xprev = g.has_bias ? g.biasvolt : 0.f;
    sign = 1.f;
  }
  // spike value and 1/(sum w - theta) once the list is consumed: an output that stopped has fired; one that consumed every input fires
  // iff it is armed
  __device__ __forceinline__ void finish(const Geometry& g, float& y, float& inv) const {
    float ws = fin.x, ys = fin.y;
    bool spike = true;
    if (live) {
      ws = plain(wsum); ys = plain(ysum);
      spike = ratio_gt(ys, ws, xprev);
    }
    y = g.maxv; inv = 0.f;
    if (spike) {
      inv = __fdividef(1.0f, ws);
      y = ys * inv;
      if (y >= g.maxv) { y = g.maxv; inv = 0.f; }
    }
  }

  __device__ __forceinline__ float plain(float v) const { return sign < 0.f ? 0.f - v : v; }   // (an exactly cancelled sum stays +0)

  // lim: bits of the q beyond the margin that still goes to the comparisons, 0 unless the output has been turned
  template <int G>
  __device__ __forceinline__ void steps(const float (&x)[G], const float (&w)[G], const int lim) {
    float sw[G], sy[G];
    int p[G];
    const float z = -2.384185791015625e-7f * fmaxf(fabsf(x[0]), fabsf(x[G - 1]));   // inputs ascend: |x| peaks at an end
    int m = sticky;
#pragma unroll
    for (int u = 0; u < G; ++u) {
      sw[u] = wsum; sy[u] = ysum;
      p[u] = __float_as_int(fmaf(z, fabsf(wsum), fmaf(-x[u], wsum, ysum)));   // (an output set aside: NaN, a positive integer)
      if (u & 1) m = imin3(m, p[u - (u > 0)], p[u]);
      else if (u == G - 1) m = min(m, p[u]);
      wsum += w[u];
      ysum = fmaf(x[u], w[u], ysum);
    }
    if (__builtin_expect(__any_sync(0xffffffffu, m <= lim), 0)) {
      // Every lane takes its own first step at or near zero through the comparisons, all lanes at once. Nearly always that step
      // fires; where one does not, or was waited for from the group before, the steps are gone through one by one.
      {
        float tw = 0.f, ty = 0.f, tx = 0.f, txp = 0.f;
        bool at = false;
#pragma unroll
        for (int u = G - 1; u >= 0; --u) {
          if (p[u] <= lim) { tw = sw[u]; ty = sy[u]; tx = x[u]; txp = u == 0 ? xprev : x[u > 0 ? u - 1 : 0]; at = true; }
        }
        at &= live;
        tw = plain(tw); ty = plain(ty);
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
        const bool near = live & (p[u] <= lim);
        if (!__any_sync(0xffffffffu, near | (sticky < 0))) continue;
        const float xp = u == 0 ? xprev : x[u > 0 ? u - 1 : 0], tw = plain(sw[u]), ty = plain(sy[u]);
        const bool fire = live & ratio_gt(ty, tw, xp) & ratio_le(ty, tw, x[u]);
        if (fire) fin = make_float2(tw, ty);
        live = live & !fire;
        sticky = (near & !fire) ? INT_MIN : INT_MAX;
      }
      if (!live) wsum = -CUDART_INF_F;
    }
    xprev = x[G - 1];
  }

  // Between two groups. An output may cross zero without firing (both rounded comparisons of the reference can miss it: about once
  // in 10^5 spikes at some hundred inputs, once in some hundred at 25 000) and would take its warp through the steps one by one to the
  // end of the list. Beyond the margin its sums change their sign, and with them its q: it cannot fire before q comes back to zero.
  // (A positive sum: not armed, if the present sums, too, see the last input beyond zero -- guard() widens the margin by what the
  // step between may have added. A negative sum: not yet back.) Returns whether the warp has any such output.
  __device__ __forceinline__ bool turn(bool turned) {
    if (__builtin_expect(__any_sync(0xffffffffu, sticky < 0), 0)) {
      const float q = fmaf(-xprev, wsum, ysum);
      if (sticky < 0 && live && fabsf(q) > 2.384185791015625e-7f * fabsf(xprev * wsum)) {
        sticky = INT_MAX;
        if (q < 0.f) { sign = -sign; wsum = 0.f - wsum; ysum = 0.f - ysum; }
      }
      turned |= (bool)__any_sync(0xffffffffu, sign < 0.f);
    }
    return turned;
  }
  // weights of a group in a warp with turned outputs: their sign, and the limit for steps()
  template <int G>
  __device__ __forceinline__ int guard(const float (&x)[G], float (&w)[G]) const {
    float most = 0.f;
#pragma unroll
    for (int u = 0; u < G; ++u) {
      most = fmaxf(most, fabsf(w[u]));
      w[u] *= sign;
    }
    return sign < 0.f ? __float_as_int(2.384185791015625e-7f * most * fmaxf(fabsf(x[0]), fabsf(x[G - 1]))) : 0;
  }
};

}  // namespace snntc

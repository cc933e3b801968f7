// Sorted lists of rows that neither the merging builder nor the register network (snntc_lists.cu) covers: rows of more than 64
// inputs, dense or receptive fields of strided, larger or small convolutions. One bucket pass, then every bucket ranked in place.
//
// A list holds the row's inputs at or below MAX - 0.1, ascending in (value, source index). Per row:
//   1. the keys (values as sortable 32-bit integers) of the inputs that can spike, their smallest and largest;
//   2. the key range is cut into NB buckets of equal width in key bits (spike times fill a few binades evenly); a histogram by
//      shared-memory atomics, its prefix sum, and a scatter into bucket order;
//   3. every key's rank inside its bucket -- one or two keys on average -- by counting the smaller (key, index) pairs, and the
//      entry goes straight to its place in the list. A bucket of more than 128 keys (many equal inputs, as the background of
//      an image gives) is first sorted in place by a bitonic network.
// Against the stable radix sort this replaces (three to four passes over the row, ranking by warp-wide digit matches) a key
// costs about a third of the instructions, and a row is shared by up to 1024 threads where there are few of them.
// Measured (B200, half of the inputs spiking, before -> now): 784 inputs at 32 samples 19 -> 6 us, at 1024: 24 -> 7; 4096 at 32:
// 65 -> 8; 25 088 at 64: 376 -> 31; 17 020 fields of 5x5x20 inputs 106 -> 58; 3136 fields of 3x3x128, stride 2: 60 -> 36.
#include "snntc_bound.cuh"
#include "snntc_common.cuh"

namespace snntc {

namespace {

constexpr int kBigBucket = 128;

// Where element i of a conv row sits relative to the row's top-left input pixel, built once per CTA: off[i] in elements,
// khw[i] = kh << 8 | kw (Kh, Kw <= 255).
__host__ __device__ __forceinline__ size_t tap_table_bytes(const Geometry& g) {
  return g.is_conv ? ((((size_t)g.I * 6) + 15) & ~(size_t)15) : 0;
}

// The threads that share a row: a warp, or the CTA.
template <int TPR>
__device__ __forceinline__ void row_sync() {
  if constexpr (TPR == 32) __syncwarp(); else __syncthreads();
}

// Sum over the row's threads of everything in front of this thread (exclusive), and the total. `tmp`: 33 words.
template <int TPR>
__device__ __forceinline__ unsigned exclusive_sum(unsigned v, unsigned* tmp, unsigned& total) {
  const int lane = threadIdx.x & 31;
  unsigned incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  if constexpr (TPR == 32) {
    total = __shfl_sync(0xffffffffu, incl, 31);
    return incl - v;
  } else {
    const int warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 31) tmp[warp] = incl;
    __syncthreads();
    unsigned before = 0, all = 0;
#pragma unroll
    for (int k = 0; k < TPR / 32; ++k) {
      const unsigned t = tmp[k];
      before += k < warp ? t : 0u;
      all += t;
    }
    total = all;
    return before + incl - v;
  }
}

// Bitonic network over the (key, index) pairs [0, n) of one bucket, in place. Every compare-exchange moves the smaller pair to
// the lower index, so the virtual infinite elements behind n never move and need no storage.
template <int TPR>
__device__ __forceinline__ void sort_bucket(uint32_t* key, unsigned short* idx, int n, int t) {
  auto exchange = [&](int i, int p) {
    if (p < n) {
      const uint32_t a = key[i], b = key[p];
      const unsigned short ia = idx[i], ib = idx[p];
      if (a > b || (a == b && ia > ib)) { key[i] = b; key[p] = a; idx[i] = ib; idx[p] = ia; }
    }
  };
  int npad = 2;
  while (npad < n) npad <<= 1;
  const int half = npad >> 1;
  for (int k = 2; k <= npad; k <<= 1) {
    const int hk = k >> 1;
    for (int q = t; q < half; q += TPR) {
      const int o = q & (hk - 1), base = (q - o) << 1;
      exchange(base + o, base + k - 1 - o);
    }
    row_sync<TPR>();
    for (int j = hk >> 1; j >= 1; j >>= 1) {
      for (int q = t; q < half; q += TPR) {
        const int o = q & (j - 1), i = ((q - o) << 1) + o;
        exchange(i, i + j);
      }
      row_sync<TPR>();
    }
  }
}

// Shared memory of one row: keys and indices in bucket order, the buckets, (warp per row) the keys in index order.
template <int TPR>
__host__ __device__ __forceinline__ size_t row_bytes(int I, int nb_log2) {
  const size_t padded = ((size_t)I + 7) & ~(size_t)7;
  return padded * 4 + padded * 2 + ((size_t)4 << nb_log2) + (TPR == 32 ? padded * 4 : 0);
}

// TPR threads per row (32: several rows per CTA, else one), EPT keys per thread in registers (0: in shared memory).
template <int TPR, int EPT>
__global__ void __launch_bounds__(TPR == 32 ? 256 : TPR)
snn_bucket_sort_kernel(const Geometry g, const float* x, WalkEntry* __restrict__ lists, int* __restrict__ nvalid,
                       int istride, int nb_log2, int table, const WeightBound wb) {
  chain_wait();
  chain_next();
  if ((int)blockIdx.x < wb.ctas) return weight_bound(wb, blockIdx.x);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned tmp[33], tmp_max[TPR > 32 ? TPR / 32 : 1];
  constexpr int kMostBig = TPR == 32 ? 8 : 256;      // at most I / 129 buckets hold more than 128 keys
  __shared__ int big_count[TPR == 32 ? 8 : 1], big_list[TPR == 32 ? 8 : 1][kMostBig];
  const int I = g.I;
  const int t = TPR == 32 ? (threadIdx.x & 31) : threadIdx.x;
  const int group = TPR == 32 ? (threadIdx.x >> 5) : 0, groups = TPR == 32 ? (blockDim.x >> 5) : 1;
  int* tap_off = reinterpret_cast<int*>(smem_raw);
  unsigned short* tap_khw = reinterpret_cast<unsigned short*>(tap_off + I);
  const int padded = (I + 7) & ~7;
  unsigned char* mine = smem_raw + (table ? tap_table_bytes(g) : 0) + (size_t)group * row_bytes<TPR>(I, nb_log2);
  uint32_t* key = reinterpret_cast<uint32_t*>(mine);                       // bucket order
  unsigned* bin = reinterpret_cast<unsigned*>(key + padded);
  unsigned short* idx = reinterpret_cast<unsigned short*>(bin + (1 << nb_log2));
  uint32_t* in_order = reinterpret_cast<uint32_t*>(idx + padded);          // TPR == 32 only
  const int nb = 1 << nb_log2;
  if (table) {
    for (int i = threadIdx.x; i < I; i += blockDim.x) {
      const int tap = i / g.C, c = i - tap * g.C;
      const int kh = tap / g.Kw, kw = tap - kh * g.Kw;
      tap_off[i] = (kh * g.W + kw) * g.C + c;
      tap_khw[i] = (unsigned short)(kh << 8 | kw);
    }
    __syncthreads();
  }
  const float maxcomp = g.maxv - 0.1f;

  for (int r = (blockIdx.x - wb.ctas) * groups + group; r < g.R; r += (gridDim.x - wb.ctas) * groups) {
    const float* xr = x + (size_t)r * I;
    int h0 = 0, w0 = 0;
    if (g.is_conv) {
      const int nw = r % g.Nw, q = r / g.Nw;
      const int nh = q % g.Nh, b = q / g.Nh;
      h0 = nh * g.Sh - g.pad_top;
      w0 = nw * g.Sw - g.pad_left;
      // the row's top-left input pixel; may lie outside the image, in which case it is never dereferenced
      xr = x + ((ptrdiff_t)b * g.H * g.W + (ptrdiff_t)h0 * g.W + w0) * g.C;
    }
    auto load = [&](int i) {        // MAX where there is nothing
      float v = g.maxv;
      if (i < I) {
        if (table) {
          const unsigned khw = tap_khw[i];
          if ((unsigned)(h0 + (int)(khw >> 8)) < (unsigned)g.H && (unsigned)(w0 + (int)(khw & 255u)) < (unsigned)g.W) v = ld_plain(xr + tap_off[i]);
        } else if (g.is_conv) {     // a window too large for the table
          const int tap = i / g.C, c = i - tap * g.C;
          const int kh = tap / g.Kw, kw = tap - kh * g.Kw;
          if ((unsigned)(h0 + kh) < (unsigned)g.H && (unsigned)(w0 + kw) < (unsigned)g.W) v = ld_plain(xr + (ptrdiff_t)(kh * g.W + kw) * g.C + c);
        } else {
          v = ld_plain(xr + i);
        }
      }
      return v;
    };
    // ---- keys; an input that never spikes has the key 0xFFFFFFFF, which no kept input has (it would be a NaN with all
    // bits set: such an input takes the next smaller key)
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    auto to_key = [&](float v) {
      const uint32_t k = float_to_sortable(v);
      return v > maxcomp ? kNone : (k == kNone ? kNone - 1u : k);
    };
    uint32_t kmin = kNone, kmax = 0u;
    uint32_t mykey[EPT > 0 ? EPT : 1];
    if constexpr (EPT > 0) {
#pragma unroll
      for (int e = 0; e < EPT; ++e) mykey[e] = to_key(load(e * TPR + t));
#pragma unroll
      for (int e = 0; e < EPT; ++e)
        if (mykey[e] != kNone) { kmin = min(kmin, mykey[e]); kmax = max(kmax, mykey[e]); }
    } else {
      for (int i0 = 0; i0 < I; i0 += 4 * TPR) {      // four loads in flight per lane
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = load(i0 + q * TPR + t);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t k = to_key(v[q]);
          if (i0 + q * TPR + t < I) in_order[i0 + q * TPR + t] = k;
          if (k != kNone) { kmin = min(kmin, k); kmax = max(kmax, k); }
        }
      }
    }
    kmin = __reduce_min_sync(0xffffffffu, kmin);
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    if constexpr (TPR > 32) {
      __syncthreads();
      if ((t & 31) == 0) { tmp[t >> 5] = kmin; tmp_max[t >> 5] = kmax; }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < TPR / 32; ++k) { kmin = min(kmin, tmp[k]); kmax = max(kmax, tmp_max[k]); }
    }
    // bucket of a key: (key - kmin) >> shift < nb
    const int bits = kmax > kmin ? 32 - __clz(kmax - kmin) : 0;
    const int shift = bits > nb_log2 ? bits - nb_log2 : 0;
    auto each = [&](auto f) {       // every kept key of this thread
      if constexpr (EPT > 0) {
#pragma unroll
        for (int e = 0; e < EPT; ++e)
          if (mykey[e] != kNone) f(mykey[e], e * TPR + t);
      } else {
        for (int i = t; i < I; i += TPR) {
          const uint32_t k = in_order[i];
          if (k != kNone) f(k, i);
        }
      }
    };
    for (int b = t; b < nb; b += TPR) bin[b] = 0u;
    if (t == 0) big_count[group] = 0;
    row_sync<TPR>();
    each([&](uint32_t k, int) { atomicAdd(&bin[(k - kmin) >> shift], 1u); });
    row_sync<TPR>();
    // ---- starts of the buckets: a thread owns nb / TPR neighbouring ones
    const int per = nb / TPR;
    unsigned s = 0, total;
    auto start_of = [&](unsigned c, int b, unsigned& at) {
      if (c > kBigBucket) big_list[group][atomicAdd(&big_count[group], 1)] = b;
      const unsigned first = at;
      at += c;
      return first;
    };
    if (per % 4 == 0) {
      uint4* mine4 = reinterpret_cast<uint4*>(bin + t * per);
      for (int q = 0; q < per / 4; ++q) { const uint4 c = mine4[q]; s += c.x + c.y + c.z + c.w; }
      unsigned at = exclusive_sum<TPR>(s, tmp, total);
      for (int q = 0; q < per / 4; ++q) {
        uint4 c = mine4[q];
        const int b = t * per + 4 * q;
        c.x = start_of(c.x, b, at); c.y = start_of(c.y, b + 1, at); c.z = start_of(c.z, b + 2, at); c.w = start_of(c.w, b + 3, at);
        mine4[q] = c;
      }
    } else {
      for (int q = 0; q < per; ++q) s += bin[t * per + q];
      unsigned at = exclusive_sum<TPR>(s, tmp, total);
      for (int q = 0; q < per; ++q) bin[t * per + q] = start_of(bin[t * per + q], t * per + q, at);
    }
    const int n = (int)total;
    row_sync<TPR>();
    each([&](uint32_t k, int i) {
      const unsigned p = atomicAdd(&bin[(k - kmin) >> shift], 1u);   // afterwards bin[b] is the end of bucket b
      key[p] = k;
      idx[p] = (unsigned short)i;
    });
    row_sync<TPR>();
    for (int q = 0; q < big_count[group]; ++q) {
      const int b = big_list[group][q];
      const int first = b > 0 ? (int)bin[b - 1] : 0;
      sort_bucket<TPR>(key + first, idx + first, (int)bin[b] - first, t);
    }
    // ---- ranks inside the buckets
    WalkEntry* dst = lists + (size_t)r * istride;
    for (int p = t; p < n; p += TPR) {
      const uint32_t k = key[p];
      const unsigned i = idx[p];
      const unsigned b = (k - kmin) >> shift;
      const int first = b > 0 ? (int)bin[b - 1] : 0, last = (int)bin[b];
      int rank = p;
      if (last - first <= kBigBucket) {
        rank = first;
        for (int q = first; q < last; ++q) {
          const uint32_t o = key[q];
          rank += (o < k) | ((o == k) & (idx[q] < i));
        }
      }
      dst[rank] = make_uint2(__float_as_uint(sortable_to_float(k)), i * (unsigned)g.J);
    }
    if (t == 0) nvalid[r] = n;
    row_sync<TPR>();                // the next row's keys go into the same memory
  }
}

template <int TPR, int EPT>
int launch(const Geometry& g, const float* x, WalkEntry* lists, int* nvalid, int istride, int nb_log2, const WeightBound& wb,
           const LaunchInfo& li, cudaStream_t s) {
  const size_t row = row_bytes<TPR>(g.I, nb_log2);
  size_t table = g.is_conv && g.Kh <= 255 && g.Kw <= 255 ? tap_table_bytes(g) : 0;
  const size_t budget = (size_t)li.max_smem_optin - 12 * 1024;              // (static arrays, the per-CTA reserve)
  if (table + row > budget) table = 0;
  int rows_per_cta = 1;
  if (TPR == 32) {
    rows_per_cta = 8;
    while (rows_per_cta > 1 && table + rows_per_cta * row > budget / 4) rows_per_cta >>= 1;
  }
  const size_t smem = table + rows_per_cta * row;
  if (smem > budget) return E_UNSUPPORTED;
  if (allow_smem<snn_bucket_sort_kernel<TPR, EPT>>(smem) != cudaSuccess) return E_CUDA;
  const int threads = TPR == 32 ? 32 * rows_per_cta : TPR;
  long resident = (long)(budget / (smem + 10 * 1024));
  if (resident > 2048 / threads) resident = 2048 / threads;
  if (resident < 1) resident = 1;
  long grid = ((long)g.R + rows_per_cta - 1) / rows_per_cta;
  if (grid > resident * li.num_sms) grid = resident * li.num_sms;
  (void)launch_chained(snn_bucket_sort_kernel<TPR, EPT>, (int)grid + wb.ctas, threads, smem, s, 0, g, x, lists, nvalid, istride, nb_log2, table > 0, wb);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? OK : E_CUDA;
}

}  // namespace

// Rows of up to 31 000 inputs. Enough rows to fill the GPU's warps (16 per SM): a warp per row for up to 512 inputs, for
// receptive fields up to 1024 (the tap arithmetic then hides what a warp loses on longer rows: 784 inputs at 10 000 rows are
// 63 us by warps and 57 by CTAs when dense, 80 against 88 as fields). Else a CTA per row of as many threads as leave a
// thread eight keys (32 in the longest rows). Buckets: about one per two inputs, at least one per thread.
int launch_row_sort(const Geometry& g, const float* x, WalkEntry* lists, int* nvalid, int istride, const WeightBound& wb,
                    const LaunchInfo& li, cudaStream_t s) {
  if (g.I > 32768) return E_UNSUPPORTED;
  int lg = 5;
  while ((1 << lg) * 2 < g.I && lg < 13) ++lg;
  if (g.R <= li.num_sms && g.I <= 4096) {          // a CTA per SM at most: the fewest keys one after the other
    if (g.I <= 512) return launch<128, 4>(g, x, lists, nvalid, istride, lg < 7 ? 7 : lg, wb, li, s);
    if (g.I <= 1024) return launch<256, 4>(g, x, lists, nvalid, istride, lg < 8 ? 8 : lg, wb, li, s);
    if (g.I <= 2048) return launch<512, 4>(g, x, lists, nvalid, istride, lg < 9 ? 9 : lg, wb, li, s);
    return launch<1024, 4>(g, x, lists, nvalid, istride, lg < 10 ? 10 : lg, wb, li, s);
  }
  if (g.I <= 1024) {
    if (g.R >= 16 * li.num_sms && (g.is_conv || g.I <= 512)) return launch<32, 0>(g, x, lists, nvalid, istride, lg, wb, li, s);
    return launch<128, 8>(g, x, lists, nvalid, istride, lg < 7 ? 7 : lg, wb, li, s);
  }
  if (g.I <= 2048) return launch<256, 8>(g, x, lists, nvalid, istride, lg < 8 ? 8 : lg, wb, li, s);
  if (g.I <= 4096) return launch<512, 8>(g, x, lists, nvalid, istride, lg < 9 ? 9 : lg, wb, li, s);
  if (g.I <= 8192) return launch<1024, 8>(g, x, lists, nvalid, istride, lg < 10 ? 10 : lg, wb, li, s);
  return launch<1024, 32>(g, x, lists, nvalid, istride, lg, wb, li, s);
}

}  // namespace snntc

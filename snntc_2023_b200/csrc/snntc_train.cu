// The pieces of a training step that sit around the four SNN-TC operators in the reference's example
// trainers, as single kernels over flat fp32 buffers:
//   - input encoding      x = exp(scale * (1 - p))  or  exp(scale * p)            (snntc-mnist.py:75, snntc-cifar10.py)
//   - loss                mean softmax cross-entropy on the NEGATED spike times, its gradient and the
//                         arg-min accuracy count                                    (SNN_TC_Modules.py:286-288, snntc-mnist.py:82)
//   - weight cost         K * mean_j max(0, 1 - sum_i w_ij) + K2 * mean(w^2) and its gradient   (snntc-mnist.py:55-59)
//   - optimiser           Adam and SGD with momentum in the Keras formulation, reading the (all-reduced)
//                         gradient bucket in place                                  (snntc-mnist.py:70, snntc-imagenet.py:238)
// The reference runs these as TensorFlow graph ops; nothing here has native code in the reference.
#include "../../include/snntc_b200.h"
#include "snntc_launch.cuh"

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

namespace snntc { void count_launch(int n = 1); }

namespace {

using snntc::chain_next;
using snntc::chain_wait;
using snntc::ld_plain;
using snntc::launch_chained;

int grid_for(size_t n, int per_block = 256) {
  size_t b = (n + per_block - 1) / per_block;
  if (b > 148 * 16) b = 148 * 16;
  if (b < 1) b = 1;
  return (int)b;
}

__global__ void encode_kernel(const float* p, float* __restrict__ x, size_t n, float scale, int one_minus) {
  chain_wait();
  chain_next();
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    const float v = ld_plain(p + e);
    x[e] = expf(scale * (one_minus ? 1.0f - v : v));
  }
}

// One warp per sample: logits z = -y. loss_b = logsumexp(z) - z[label]; grad_y = -(softmax(z) - onehot) * gscale.
// sums[0] += loss_b * lscale, sums[1] += (argmin_j y == label). Ties in the arg-min go to the lowest index,
// as tf.argmin does.
__global__ void loss_ce_kernel(const float* __restrict__ y, const long long* __restrict__ labels, float* __restrict__ grad,
                               float* __restrict__ sums, int B, int J, float lscale, float gscale) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  float loss_acc = 0.f, hit_acc = 0.f;
  for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < B; b += warps) {
    const float* row = y + (size_t)b * J;
    float zmax = -CUDART_INF_F;
    int amin = 0x7fffffff;
    float ymin = CUDART_INF_F;
    for (int j = lane; j < J; j += 32) {
      const float v = __ldg(row + j);
      zmax = fmaxf(zmax, -v);
      if (v < ymin) { ymin = v; amin = j; }
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
      zmax = fmaxf(zmax, __shfl_xor_sync(0xffffffffu, zmax, d));
      const float oy = __shfl_xor_sync(0xffffffffu, ymin, d);
      const int oa = __shfl_xor_sync(0xffffffffu, amin, d);
      if (oy < ymin || (oy == ymin && oa < amin)) { ymin = oy; amin = oa; }
    }
    float se = 0.f;
    for (int j = lane; j < J; j += 32) se += expf(-__ldg(row + j) - zmax);
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) se += __shfl_xor_sync(0xffffffffu, se, d);
    const float lse_rel = logf(se);   // logsumexp(z) - zmax: the loss is lse_rel + (zmax - z[label]), never lse itself,
                                      // which would lose the small term beside a large |zmax| (all outputs at MAX)
    const int lab = (int)labels[b];
    const float inv = 1.0f / se;
    if (grad != nullptr) {
      for (int j = lane; j < J; j += 32) {
        const float sm = expf(-__ldg(row + j) - zmax) * inv;
        grad[(size_t)b * J + j] = -(sm - (j == lab ? 1.0f : 0.0f)) * gscale;
      }
    }
    if (lane == 0) {
      const float zl = (lab >= 0 && lab < J) ? -__ldg(row + lab) : zmax;
      loss_acc += (lse_rel + (zmax - zl)) * lscale;
      hit_acc += (amin == lab) ? 1.0f : 0.0f;
    }
  }
  if (lane == 0) {
    if (loss_acc != 0.f) atomicAdd(sums, loss_acc);
    if (hit_acc != 0.f) atomicAdd(sums + 1, hit_acc);
  }
}

// column sums of w[rows, J] into colsum[J] (zeroed by the caller) and sum of squares into sq[0]
__global__ void wcost_sums_kernel(const float* __restrict__ w, float* __restrict__ colsum, float* __restrict__ sq,
                                  int rows, int J, int rows_per_block) {
  const int r0 = blockIdx.y * rows_per_block;
  const int r1 = min(rows, r0 + rows_per_block);
  float s2 = 0.f;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < J; j += gridDim.x * blockDim.x) {
    float s = 0.f;
    for (int r = r0; r < r1; ++r) {
      const float v = __ldg(w + (size_t)r * J + j);
      s += v;
      s2 = fmaf(v, v, s2);
    }
    atomicAdd(colsum + j, s);
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, d);
  if ((threadIdx.x & 31) == 0 && s2 != 0.f) atomicAdd(sq, s2);
}

// cost[0] += K * mean_j max(0, 1 - colsum_j) + K2 * sq / (rows*J)   (block 0, thread-serial over a small J is
// avoided: every block adds its share), gw[i,j] += -K/J * [1 - colsum_j > 0] + 2*K2/(rows*J) * w[i,j]
__global__ void wcost_apply_kernel(const float* __restrict__ w, const float* __restrict__ colsum,
                                   const float* __restrict__ sq, float* __restrict__ gw, float* __restrict__ cost,
                                   int rows, int J, float K, float K2) {
  const size_t n = (size_t)rows * J;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const float a = -K / (float)J, b2 = 2.0f * K2 / (float)n;
  if (gw != nullptr) {
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
      const int j = (int)(e % J);
      const float hinge = (1.0f - __ldg(colsum + j)) > 0.f ? a : 0.f;
      gw[e] += hinge + b2 * __ldg(w + e);
    }
  }
  if (cost != nullptr) {
    float c = 0.f;
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < (size_t)J; j += stride)
      c += fmaxf(0.f, 1.0f - __ldg(colsum + j));
    c *= K / (float)J;
    if (blockIdx.x == 0 && threadIdx.x == 0) c += K2 * __ldg(sq) / (float)n;
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) c += __shfl_xor_sync(0xffffffffu, c, d);
    if ((threadIdx.x & 31) == 0 && c != 0.f) atomicAdd(cost, c);
  }
}

// Keras Adam: lr_t = lr * sqrt(1 - b2^t) / (1 - b1^t); m += (g - m)(1 - b1); v += (g^2 - v)(1 - b2);
// w -= lr_t * m / (sqrt(v) + eps). The step count t lives on the device (step[0] = steps taken so far), so that
// a captured CUDA graph replays with the count advancing; a one-thread kernel increments it after the update.
__global__ void adam_kernel(float* __restrict__ w, const float* g, float* __restrict__ m, float* __restrict__ v,
                            size_t n, float lr, float b1, float b2, float eps, float gscale,
                            const int* step) {
  chain_wait();
  chain_next();
  const int t = ld_plain(step) + 1;
  const float c1 = 1.0f - powf(b1, (float)t), c2 = 1.0f - powf(b2, (float)t);
  const float lrt = lr * sqrtf(c2) / c1;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    const float ge = ld_plain(g + e) * gscale;
    const float me = m[e] + (ge - m[e]) * (1.0f - b1);
    const float ve = v[e] + (ge * ge - v[e]) * (1.0f - b2);
    m[e] = me;
    v[e] = ve;
    w[e] -= lrt * me / (sqrtf(ve) + eps);
  }
}
__global__ void step_inc_kernel(int* step) { chain_wait(); chain_next(); *step += 1; }

// Keras SGD with momentum: vel = momentum * vel - lr * g; w += vel
__global__ void sgdm_kernel(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ vel, size_t n,
                            float lr, float momentum, float gscale) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += stride) {
    const float ve = momentum * vel[e] - lr * (__ldg(g + e) * gscale);
    vel[e] = ve;
    w[e] += ve;
  }
}

// ---- loss of a whole batch, no zeroed accumulators, in a fixed order of summation: the same bits every run. G lanes per sample
// (16 for up to 16 classes, else 32).
// Small batches: one launch of one cluster of eight CTAs, whose partial sums are added over distributed shared memory in rank
// order. Bound by latency (a few rounds of loads and shuffles per group): against the pair of a zero fill and an atomic
// accumulation it takes a launch off a step.
// Large ones (loss_in_one_cluster): CTAs over the whole GPU, each leaves its sum in a workspace, and a second launch adds them.
constexpr int kLossThreads = 512;
constexpr int kLossCluster = 8;

struct RowStats { float zmax, lse; int amin; };   // max of z = -y, sum exp(z - zmax), arg-min of y (lowest index on ties)

template <int G>
__device__ __forceinline__ RowStats row_stats(const float* row, int J, int gl) {
  RowStats s;
  s.zmax = -CUDART_INF_F;
  s.amin = 0x7fffffff;
  float ymin = CUDART_INF_F;
  for (int j = gl; j < J; j += G) {
    const float v = ld_plain(row + j);
    s.zmax = fmaxf(s.zmax, -v);
    if (v < ymin) { ymin = v; s.amin = j; }
  }
#pragma unroll
  for (int d = G / 2; d >= 1; d >>= 1) {
    s.zmax = fmaxf(s.zmax, __shfl_xor_sync(0xffffffffu, s.zmax, d));
    const float oy = __shfl_xor_sync(0xffffffffu, ymin, d);
    const int oa = __shfl_xor_sync(0xffffffffu, s.amin, d);
    if (oy < ymin || (oy == ymin && oa < s.amin)) { ymin = oy; s.amin = oa; }
  }
  float se = 0.f;
  for (int j = gl; j < J; j += G) se += expf(-ld_plain(row + j) - s.zmax);
#pragma unroll
  for (int d = G / 2; d >= 1; d >>= 1) se += __shfl_xor_sync(0xffffffffu, se, d);
  s.lse = se;
  return s;
}

// Sum of (a, b) over the cluster, valid in thread 0 of CTA 0: lanes, warps and CTAs in a fixed order.
__device__ __forceinline__ float2 cluster_sum(float a, float b) {
  namespace cg = cooperative_groups;
  __shared__ float2 part[33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, d);
    b += __shfl_xor_sync(0xffffffffu, b, d);
  }
  if (lane == 0) part[warp] = make_float2(a, b);
  __syncthreads();
  cg::cluster_group cl = cg::this_cluster();
  if (threadIdx.x == 0) {
    float2 t = part[0];
    for (int k = 1; k < warps; ++k) { t.x += part[k].x; t.y += part[k].y; }
    part[32] = t;
  }
  cl.sync();
  float2 sum = make_float2(0.f, 0.f);
  if (threadIdx.x == 0 && cl.block_rank() == 0)
    for (unsigned k = 0; k < cl.num_blocks(); ++k) {
      const float2 o = *cl.map_shared_rank(&part[32], k);
      sum.x += o.x;
      sum.y += o.y;
    }
  cl.sync();   // no CTA leaves while its shared memory may still be read
  return sum;
}

// (loss, hits) of the samples that this thread's group of G lanes takes, `groups` in step: in lane 0 of the group
template <int G>
__device__ __forceinline__ float2 loss_of_samples(const float* y, const long long* labels, int B, int J, float lscale, int groups) {
  const int gl = threadIdx.x % G;
  float loss_acc = 0.f, hit_acc = 0.f;
  for (int b0 = 0; b0 < B; b0 += groups) {
    const int b = b0 + (blockIdx.x * blockDim.x + threadIdx.x) / G;
    const bool ok = b < B;                       // (shuffles run with all lanes: a group without a sample repeats the last)
    const float* row = y + (size_t)(ok ? b : B - 1) * J;
    const RowStats s = row_stats<G>(row, J, gl);
    if (ok && gl == 0) {
      const int lab = (int)labels[b];
      // the loss is log(se) + (zmax - z[label]), never logsumexp itself, which would lose the small term beside a large
      // |zmax| (all outputs at MAX)
      const float zl = (lab >= 0 && lab < J) ? -ld_plain(row + lab) : s.zmax;
      loss_acc += (logf(s.lse) + (s.zmax - zl)) * lscale;
      hit_acc += (s.amin == lab) ? 1.0f : 0.0f;
    }
  }
  return make_float2(loss_acc, hit_acc);
}

template <int G>
__global__ void __cluster_dims__(kLossCluster, 1, 1) __launch_bounds__(kLossThreads)
loss_fwd_kernel(const float* y, const long long* labels, float* __restrict__ loss, float* __restrict__ hits, int B, int J,
                float lscale) {
  chain_wait();
  chain_next();
  const float2 mine = loss_of_samples<G>(y, labels, B, J, lscale, kLossCluster * kLossThreads / G);
  const float2 sum = cluster_sum(mine.x, mine.y);
  if (blockIdx.x == 0 && threadIdx.x == 0) { *loss = sum.x; *hits = sum.y; }
}

constexpr int kLossWideThreads = 256;
constexpr int kLossWideCtas = 592;      // four per SM of a B200 at most; fixed, so that the order of summation is

template <int G>
__global__ void __launch_bounds__(kLossWideThreads)
loss_partial_kernel(const float* y, const long long* labels, float2* __restrict__ partial, int B, int J, float lscale) {
  chain_wait();
  chain_next();
  const float2 mine = loss_of_samples<G>(y, labels, B, J, lscale, (int)gridDim.x * (kLossWideThreads / G));
  const float2 sum = cluster_sum(mine.x, mine.y);     // (every CTA is a cluster of its own)
  if (threadIdx.x == 0) partial[blockIdx.x] = sum;
}

__global__ void __launch_bounds__(kLossWideThreads)
loss_total_kernel(const float2* partial, int n, float* __restrict__ loss, float* __restrict__ hits) {
  chain_wait();
  chain_next();
  float2 mine = make_float2(0.f, 0.f);
  for (int k = threadIdx.x; k < n; k += kLossWideThreads) {
    const float2 p = ld_plain(partial + k);
    mine.x += p.x;
    mine.y += p.y;
  }
  const float2 sum = cluster_sum(mine.x, mine.y);
  if (threadIdx.x == 0) { *loss = sum.x; *hits = sum.y; }
}

// grad_y = -(softmax(-y) - onehot) * gscale * (*gloss): the softmax again from y instead of a gradient kept by the forward
template <int G>
__global__ void __launch_bounds__(256)
loss_bwd_kernel(const float* y, const long long* labels, const float* gloss,
                float* __restrict__ grad, int B, int J, float gscale) {
  chain_wait();
  chain_next();
  const int gl = threadIdx.x % G;
  const int b = (blockIdx.x * 256 + threadIdx.x) / G;
  const bool ok = b < B;
  const float* row = y + (size_t)(ok ? b : B - 1) * J;
  const RowStats s = row_stats<G>(row, J, gl);
  if (!ok) return;
  const int lab = (int)labels[b];
  const float inv = 1.0f / s.lse, up = ld_plain(gloss);
  for (int j = gl; j < J; j += G) {
    const float sm = expf(-ld_plain(row + j) - s.zmax) * inv;
    grad[(size_t)b * J + j] = -(sm - (j == lab ? 1.0f : 0.0f)) * gscale * up;
  }
}

// ---- the weight cost of several tensors at once. A network has one small tensor per layer, and cost and gradient of
// each used to be two memsets, two kernels and three framework operations; here all tensors share three launches.
// Column sums go through partial sums of row slices that are added in a fixed order: no atomics, same bits every run.
constexpr int kCostMax = 16;          // tensors per launch
constexpr int kCostThreads = 256;
constexpr int kCostChunk = 4096;      // elements per CTA of the gradient kernel

struct CostTensors {
  int count;
  const float* w[kCostMax];
  float* gw[kCostMax];
  int rows[kCostMax], cols[kCostMax];
  int slices[kCostMax];               // row slices of the column-sum pass
  int first_cta[kCostMax + 1];        // of the column-sum pass: slices * blocks of kCostThreads columns
  int first_col[kCostMax + 1];        // offset of the tensor's columns in colsum
  int first_chunk[kCostMax + 1];      // of the gradient pass
  long long partial[kCostMax];        // offset of the tensor's [slices][cols] partial column sums
};

__device__ __forceinline__ int tensor_of(const int* first, int count, int at) {
  int t = 0;
  while (t + 1 < count && at >= first[t + 1]) ++t;
  return t;
}

// CTA = (tensor, block of up to 256 columns, slice of the rows): a thread owns one column and every (256 / columns)-th
// row of the slice, eight loads in flight; the threads of a column are added through shared memory.
__global__ void __launch_bounds__(kCostThreads)
cost_sums_kernel(const __grid_constant__ CostTensors c, float* __restrict__ partial, float* __restrict__ sq) {
  chain_wait();
  chain_next();
  __shared__ float part[kCostThreads];
  const int t = tensor_of(c.first_cta, c.count, blockIdx.x);
  const int local = blockIdx.x - c.first_cta[t];
  const int rows = c.rows[t], J = c.cols[t], slices = c.slices[t];
  const int slice = local % slices, j0 = (local / slices) * kCostThreads;
  const int width = min(kCostThreads, J - j0);
  const int lines = kCostThreads / width;            // rows in step
  const int line = threadIdx.x / width, col = threadIdx.x % width;
  const int per = (rows + slices - 1) / slices;
  const int r0 = slice * per, r1 = min(rows, r0 + per);
  const float* w = c.w[t] + j0 + col;
  float s = 0.f, s2 = 0.f;
  if (line < lines) {
    int r = r0 + line;
    for (; r + 7 * lines < r1; r += 8 * lines) {
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = ld_plain(w + (size_t)(r + q * lines) * J);
#pragma unroll
      for (int q = 0; q < 8; ++q) { s += v[q]; s2 = fmaf(v[q], v[q], s2); }
    }
    for (; r < r1; r += lines) {
      const float v = ld_plain(w + (size_t)r * J);
      s += v;
      s2 = fmaf(v, v, s2);
    }
  }
  part[threadIdx.x] = s;
  __syncthreads();
  if (line == 0) {
    for (int k = 1; k < lines; ++k) s += part[k * width + col];
    partial[c.partial[t] + (long long)slice * J + j0 + col] = s;
  }
  __syncthreads();
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, d);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s2;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < kCostThreads / 32; ++k) s2 += part[k];
    sq[blockIdx.x] = s2;
  }
}

// One cluster: column sums out of the partial ones, and the cost of all tensors (added to *cost when `add` is set).
__global__ void __cluster_dims__(kLossCluster, 1, 1) __launch_bounds__(kLossThreads)
cost_total_kernel(const __grid_constant__ CostTensors c, const float* partial, const float* sq,
                  float* __restrict__ colsum, float* __restrict__ cost, float K, float K2, int add) {
  chain_wait();
  chain_next();
  const int me = blockIdx.x * kLossThreads + threadIdx.x;
  constexpr int kAll = kLossCluster * kLossThreads;
  float total = 0.f;
  for (int col = me; col < c.first_col[c.count]; col += kAll) {
    const int t = tensor_of(c.first_col, c.count, col);
    const int J = c.cols[t];
    const float* p = partial + c.partial[t] + (col - c.first_col[t]);
    float s = 0.f;
#pragma unroll 8
    for (int k = 0; k < c.slices[t]; ++k) s += ld_plain(p + (long long)k * J);
    colsum[col] = s;
    total += fmaxf(0.f, 1.0f - s) * (K / (float)J);
  }
  for (int k = me; k < c.first_cta[c.count]; k += kAll) {
    const int t = tensor_of(c.first_cta, c.count, k);
    total += ld_plain(sq + k) * (K2 / ((float)c.rows[t] * (float)c.cols[t]));
  }
  const float2 sum = cluster_sum(total, 0.f);
  if (blockIdx.x == 0 && threadIdx.x == 0) *cost = add ? *cost + sum.x : sum.x;
}

// gw = gcost * (-K/J [colsum < 1] + 2 K2 / n * w), or gw += it, a CTA per 4096 elements of one tensor
template <bool ADD>
__global__ void __launch_bounds__(kCostThreads)
cost_grad_kernel(const __grid_constant__ CostTensors c, const float* colsum, const float* gcost,
                 float K, float K2) {
  chain_wait();
  chain_next();
  const int t = tensor_of(c.first_chunk, c.count, blockIdx.x);
  const int J = c.cols[t];
  const unsigned n = (unsigned)c.rows[t] * (unsigned)J;
  const unsigned e0 = (unsigned)(blockIdx.x - c.first_chunk[t]) * kCostChunk;
  const unsigned e1 = min(n, e0 + kCostChunk);
  const float up = ld_plain(gcost);
  const float a = -K / (float)J, b2 = 2.0f * K2 / (float)n;
  const float* cs = colsum + c.first_col[t];
  const float* w = c.w[t];
  float* gw = c.gw[t];
  if ((J & 3) == 0 && (((uintptr_t)w | (uintptr_t)gw) & 15) == 0) {
    for (unsigned e = e0 + 4 * threadIdx.x; e < e1; e += 4 * kCostThreads) {
      const unsigned j = e % (unsigned)J;
      const float4 v = ld_plain(reinterpret_cast<const float4*>(w + e));
      float4 r;
      r.x = ((1.0f - ld_plain(cs + j)) > 0.f ? a : 0.f) + b2 * v.x;
      r.y = ((1.0f - ld_plain(cs + j + 1)) > 0.f ? a : 0.f) + b2 * v.y;
      r.z = ((1.0f - ld_plain(cs + j + 2)) > 0.f ? a : 0.f) + b2 * v.z;
      r.w = ((1.0f - ld_plain(cs + j + 3)) > 0.f ? a : 0.f) + b2 * v.w;
      // (the product is rounded before it is added, as when a gradient tensor of its own is added to the bucket)
      float4 o = make_float4(__fmul_rn(up, r.x), __fmul_rn(up, r.y), __fmul_rn(up, r.z), __fmul_rn(up, r.w));
      if (ADD) {
        const float4 have = *reinterpret_cast<const float4*>(gw + e);
        o = make_float4(have.x + o.x, have.y + o.y, have.z + o.z, have.w + o.w);
      }
      *reinterpret_cast<float4*>(gw + e) = o;
    }
  } else {
    for (unsigned e = e0 + threadIdx.x; e < e1; e += kCostThreads) {
      const float r = __fmul_rn(up, ((1.0f - ld_plain(cs + e % (unsigned)J)) > 0.f ? a : 0.f) + b2 * ld_plain(w + e));
      gw[e] = ADD ? gw[e] + r : r;
    }
  }
}

// Tensors [at, at + 16) of a list; the column sums of the earlier ones take the first `cols_before` floats of colsum.
// Row slices: about 64 rows each, at most 128, so that a large tensor spreads over the GPU.
CostTensors cost_tensors(int count, const float* const* w, float* const* gw, const int* rows, const int* cols, int at) {
  CostTensors c;
  c.count = count - at < kCostMax ? count - at : kCostMax;
  int cta = 0, col = 0, chunk = 0;
  long long partial = 0;
  for (int k = 0; k < c.count; ++k) {
    const int r = rows[at + k], J = cols[at + k];
    c.w[k] = w ? w[at + k] : nullptr;
    c.gw[k] = gw ? gw[at + k] : nullptr;
    c.rows[k] = r;
    c.cols[k] = J;
    int slices = (r + 63) / 64;
    if (slices > 128) slices = 128;
    c.slices[k] = slices;
    c.first_cta[k] = cta;
    c.first_col[k] = col;
    c.first_chunk[k] = chunk;
    c.partial[k] = partial;
    cta += slices * ((J + kCostThreads - 1) / kCostThreads);
    col += J;
    chunk += (int)(((long long)r * J + kCostChunk - 1) / kCostChunk);
    partial += (long long)slices * J;
  }
  c.first_cta[c.count] = cta;
  c.first_col[c.count] = col;
  c.first_chunk[c.count] = chunk;
  return c;
}
size_t cost_partial_floats(const CostTensors& c) {
  size_t n = 0;
  for (int k = 0; k < c.count; ++k) n += (size_t)c.slices[k] * c.cols[k];
  return n;
}

int loss_lanes(int J) { return J <= 16 ? 16 : 32; }
int loss_wide_ctas(int B, int J) {
  const long long ctas = ((long long)B * loss_lanes(J) + kLossWideThreads - 1) / kLossWideThreads;
  return ctas < kLossWideCtas ? (int)ctas : kLossWideCtas;
}
// One cluster takes about 0.9 us for a round of its 4096 lanes and 0.1 us for each load of a lane in it, two launches over the whole
// GPU 6.5 us and up: they cross at 1024 samples of 10 classes (6.2 us in one cluster, 6.5 in two launches; 4096: 17.5 and 7.0), 256 of
// 300 (6.2, 6.5) and 128 of 1000 (6.6, 7.2; 256: 10.2, 7.6; 1024: 32 and 8.6; 65 536: 2850 and 95).
bool loss_in_one_cluster(int B, int J) {
  const int G = loss_lanes(J);
  constexpr int lanes = kLossCluster * kLossThreads;
  const long long rounds = ((long long)B * G + lanes - 1) / lanes;
  return rounds * (9 + (J + G - 1) / G) <= 42;
}

int done() {
  snntc::count_launch();
  return cudaGetLastError() == cudaSuccess ? SNNTC_OK : SNNTC_E_CUDA;
}

}  // namespace

extern "C" {

int snntc_encode(const float* p, float* x, size_t n, float scale, int one_minus, void* stream) {
  if (!p || !x) return SNNTC_E_NULL;
  if (n == 0) return SNNTC_OK;
  (void)launch_chained(encode_kernel, grid_for(n), 256, 0, (cudaStream_t)stream, 0, p, x, n, scale, one_minus);
  return done();
}

int snntc_loss_ce(const float* y, const long long* labels, float* grad, float* sums2, int B, int J,
                  float loss_scale, float grad_scale, void* stream) {
  if (!y || !labels || !sums2) return SNNTC_E_NULL;
  if (B <= 0 || J <= 0) return SNNTC_E_SHAPE;
  loss_ce_kernel<<<grid_for((size_t)B * 32), 256, 0, (cudaStream_t)stream>>>(y, labels, grad, sums2, B, J, loss_scale,
                                                                            grad_scale);
  return done();
}

int snntc_loss_forward(const float* y, const long long* labels, float* loss, float* hits, int B, int J, float loss_scale,
                       void* stream) {
  if (!y || !labels || !loss || !hits) return SNNTC_E_NULL;
  if (B <= 0 || J <= 0) return SNNTC_E_SHAPE;
  if (J <= 16) (void)launch_chained(loss_fwd_kernel<16>, kLossCluster, kLossThreads, 0, (cudaStream_t)stream, 0, y, labels, loss, hits, B, J, loss_scale);
  else (void)launch_chained(loss_fwd_kernel<32>, kLossCluster, kLossThreads, 0, (cudaStream_t)stream, 0, y, labels, loss, hits, B, J, loss_scale);
  return done();
}

size_t snntc_loss_forward_workspace_bytes(int B, int J) {
  if (B <= 0 || J <= 0 || loss_in_one_cluster(B, J)) return 0;
  return (size_t)loss_wide_ctas(B, J) * sizeof(float2);
}

int snntc_loss_forward_ws(const float* y, const long long* labels, float* loss, float* hits, int B, int J, float loss_scale,
                          void* workspace, size_t workspace_bytes, void* stream) {
  const size_t need = snntc_loss_forward_workspace_bytes(B, J);
  if (need == 0) return snntc_loss_forward(y, labels, loss, hits, B, J, loss_scale, stream);
  if (!y || !labels || !loss || !hits || !workspace) return SNNTC_E_NULL;
  if (workspace_bytes < need) return SNNTC_E_WORKSPACE;
  const int ctas = loss_wide_ctas(B, J);
  float2* partial = static_cast<float2*>(workspace);
  if (J <= 16) (void)launch_chained(loss_partial_kernel<16>, ctas, kLossWideThreads, 0, (cudaStream_t)stream, 0, y, labels, partial, B, J, loss_scale);
  else (void)launch_chained(loss_partial_kernel<32>, ctas, kLossWideThreads, 0, (cudaStream_t)stream, 0, y, labels, partial, B, J, loss_scale);
  if (done() != SNNTC_OK) return SNNTC_E_CUDA;
  (void)launch_chained(loss_total_kernel, 1, kLossWideThreads, 0, (cudaStream_t)stream, 0, partial, ctas, loss, hits);
  return done();
}

int snntc_loss_backward(const float* y, const long long* labels, const float* gloss, float* grad, int B, int J,
                        float grad_scale, void* stream) {
  if (!y || !labels || !gloss || !grad) return SNNTC_E_NULL;
  if (B <= 0 || J <= 0) return SNNTC_E_SHAPE;
  const int G = J <= 16 ? 16 : 32;
  const int grid = (int)(((long long)B * G + 255) / 256);
  if (G == 16) (void)launch_chained(loss_bwd_kernel<16>, grid, 256, 0, (cudaStream_t)stream, 0, y, labels, gloss, grad, B, J, grad_scale);
  else (void)launch_chained(loss_bwd_kernel<32>, grid, 256, 0, (cudaStream_t)stream, 0, y, labels, gloss, grad, B, J, grad_scale);
  return done();
}

size_t snntc_weight_costs_workspace_bytes(int count, const int* rows, const int* cols) {
  if (count <= 0 || !rows || !cols) return 0;
  size_t most = 0;
  for (int at = 0; at < count; at += kCostMax) {
    const CostTensors c = cost_tensors(count, nullptr, nullptr, rows, cols, at);
    const size_t n = cost_partial_floats(c) + (size_t)c.first_cta[c.count];
    if (n > most) most = n;
  }
  return most * sizeof(float);
}

int snntc_weight_costs(int count, const float* const* w, const int* rows, const int* cols, float K, float K2, float* colsum,
                       float* cost, void* workspace, size_t workspace_bytes, void* stream) {
  if (!w || !rows || !cols || !colsum || !cost || !workspace) return SNNTC_E_NULL;
  if (count <= 0) return SNNTC_E_SHAPE;
  for (int k = 0; k < count; ++k) {
    if (!w[k]) return SNNTC_E_NULL;
    if (rows[k] <= 0 || cols[k] <= 0) return SNNTC_E_SHAPE;
    if ((long long)rows[k] * cols[k] > 0x7fffffffLL) return SNNTC_E_TOO_LARGE;
  }
  if (workspace_bytes < snntc_weight_costs_workspace_bytes(count, rows, cols)) return SNNTC_E_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  for (int at = 0; at < count; at += kCostMax) {
    const CostTensors c = cost_tensors(count, w, nullptr, rows, cols, at);
    float* partial = static_cast<float*>(workspace);
    float* sq = partial + cost_partial_floats(c);
    (void)launch_chained(cost_sums_kernel, c.first_cta[c.count], kCostThreads, 0, s, 0, c, partial, sq);
    if (done() != SNNTC_OK) return SNNTC_E_CUDA;
    (void)launch_chained(cost_total_kernel, kLossCluster, kLossThreads, 0, s, 0, c, partial, sq, colsum, cost, K, K2, at > 0);
    if (done() != SNNTC_OK) return SNNTC_E_CUDA;
    colsum += c.first_col[c.count];
  }
  return SNNTC_OK;
}

int snntc_weight_cost_grads(int count, const float* const* w, float* const* gw, const int* rows, const int* cols, float K,
                            float K2, const float* colsum, const float* gcost, int add, void* stream) {
  if (!w || !gw || !rows || !cols || !colsum || !gcost) return SNNTC_E_NULL;
  if (count <= 0) return SNNTC_E_SHAPE;
  for (int k = 0; k < count; ++k) {
    if (!w[k] || !gw[k]) return SNNTC_E_NULL;
    if (rows[k] <= 0 || cols[k] <= 0) return SNNTC_E_SHAPE;
    if ((long long)rows[k] * cols[k] > 0x7fffffffLL) return SNNTC_E_TOO_LARGE;
  }
  for (int at = 0; at < count; at += kCostMax) {
    const CostTensors c = cost_tensors(count, w, gw, rows, cols, at);
    if (add) (void)launch_chained(cost_grad_kernel<true>, c.first_chunk[c.count], kCostThreads, 0, (cudaStream_t)stream, 0, c, colsum, gcost, K, K2);
    else (void)launch_chained(cost_grad_kernel<false>, c.first_chunk[c.count], kCostThreads, 0, (cudaStream_t)stream, 0, c, colsum, gcost, K, K2);
    if (done() != SNNTC_OK) return SNNTC_E_CUDA;
    colsum += c.first_col[c.count];
  }
  return SNNTC_OK;
}

size_t snntc_weight_cost_workspace_bytes(int J) { return ((size_t)J + 1) * sizeof(float); }

int snntc_weight_cost(const float* w, float* gw, float* cost, int rows, int J, float K, float K2,
                      void* workspace, size_t workspace_bytes, void* stream) {
  if (!w || !workspace) return SNNTC_E_NULL;
  if (rows <= 0 || J <= 0) return SNNTC_E_SHAPE;
  if (workspace_bytes < snntc_weight_cost_workspace_bytes(J)) return SNNTC_E_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  float* colsum = static_cast<float*>(workspace);
  float* sq = colsum + J;
  if (cudaMemsetAsync(workspace, 0, snntc_weight_cost_workspace_bytes(J), s) != cudaSuccess) return SNNTC_E_CUDA;
  const int rpb = 64;
  dim3 grid((J + 255) / 256, (rows + rpb - 1) / rpb);
  wcost_sums_kernel<<<grid, 256, 0, s>>>(w, colsum, sq, rows, J, rpb);
  if (done() != SNNTC_OK) return SNNTC_E_CUDA;
  wcost_apply_kernel<<<grid_for((size_t)rows * J), 256, 0, s>>>(w, colsum, sq, gw, cost, rows, J, K, K2);
  return done();
}

int snntc_adam_step(float* w, const float* g, float* m, float* v, size_t n, float lr, float beta1, float beta2,
                    float eps, float grad_scale, int* step, void* stream) {
  if (!w || !g || !m || !v || !step) return SNNTC_E_NULL;
  if (n == 0) return SNNTC_OK;
  (void)launch_chained(adam_kernel, grid_for(n), 256, 0, (cudaStream_t)stream, 0, w, g, m, v, n, lr, beta1, beta2, eps, grad_scale, step);
  if (done() != SNNTC_OK) return SNNTC_E_CUDA;
  (void)launch_chained(step_inc_kernel, 1, 1, 0, (cudaStream_t)stream, 0, step);
  return done();
}

int snntc_sgdm_step(float* w, const float* g, float* vel, size_t n, float lr, float momentum, float grad_scale,
                    void* stream) {
  if (!w || !g || !vel) return SNNTC_E_NULL;
  if (n == 0) return SNNTC_OK;
  sgdm_kernel<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(w, g, vel, n, lr, momentum, grad_scale);
  return done();
}

}  // extern "C"

// BatchNorm over dim 1 of an NC(HW) tensor with fused residual add and ReLU.
//
// Replaces `torch::batch_norm` (flodl-sys/ops_training.cpp:1025-1046, cuDNN) plus the separate
// add and ReLU nodes of a residual block (ddp-bench/src/models/resnet.rs:209-301):
//     y = relu( (x - mean_c) * rstd_c * gamma_c + beta_c + residual )      (residual, relu optional)
// Training mode: batch statistics, biased variance for normalisation, unbiased for the running
// estimate (momentum update in place), as libtorch does. Eval mode uses the running statistics.
//
// Forward = one partial-statistics pass + one normalise pass; backward = one partial-reduction pass
// (sum dy', sum dy'*xhat with dy' = dy masked by the ReLU) + one pass writing dx and d(residual).
// Per-channel partials go to a scratch buffer of C * kSplits * 2 floats and are folded by every
// block that needs them (kSplits is small), which avoids a third launch and any atomics.
//
// Work split: block (c, s) owns the samples n = s, s + kSplits, ... of channel c. Their HW-element
// rows are walked as ONE flattened index space in 16-byte vectors, so all 256 threads stay busy
// for 8x8 feature maps as well as 32x32 ones (a per-row loop leaves 3/4 of the block idle at HW = 64).
#include "../include/flodl_b200.h"
#include "common.cuh"

namespace fb {

constexpr int kBnSplits = 16;
constexpr int kBnThreads = 256;

// Calls f(offset, count) for this block's elements: `count` consecutive elements (V when the
// vector path applies, else 1) starting at `offset` from the tensor base.
template <int V, typename F>
__device__ __forceinline__ void bn_for_each(int N, int C, int HW, int c, int s, F f) {
  const int rows = (N - s + kBnSplits - 1) / kBnSplits;     // samples owned by this block
  if (rows <= 0) return;
  if (HW % V == 0) {
    const int per_row = HW / V;
    const int total = rows * per_row;
    for (int q = threadIdx.x; q < total; q += kBnThreads) {
      const int r = q / per_row;
      const int i = (q - r * per_row) * V;
      const long long off = (static_cast<long long>(s + r * kBnSplits) * C + c) * HW + i;
      f(off, true);
    }
  } else {
    const long long total = static_cast<long long>(rows) * HW;
    for (long long q = threadIdx.x; q < total; q += kBnThreads) {
      const int r = static_cast<int>(q / HW);
      const int i = static_cast<int>(q - static_cast<long long>(r) * HW);
      const long long off = (static_cast<long long>(s + r * kBnSplits) * C + c) * HW + i;
      f(off, false);
    }
  }
}

template <typename T>
__device__ __forceinline__ bool bn_aligned(const void* p) {
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

// grid (C, kBnSplits)
template <typename T>
__global__ void __launch_bounds__(kBnThreads)
bn_stats_kernel(const T* __restrict__ x, float* __restrict__ partial, int N, int C, int HW) {
  pdl_entry();
  constexpr int V = VecIO<T>::kVec;
  __shared__ float scratch[32];
  const int c = blockIdx.x, s = blockIdx.y;
  float sum = 0.f, sq = 0.f;
  const bool vec_ok = bn_aligned<T>(x);
  if (vec_ok) {
    bn_for_each<V>(N, C, HW, c, s, [&](long long off, bool vec) {
      if (vec) {
        float v[V];
        VecIO<T>::load(x + off, v);
#pragma unroll
        for (int j = 0; j < V; ++j) { sum += v[j]; sq += v[j] * v[j]; }
      } else {
        const float v = VecIO<T>::get(x + off);
        sum += v; sq += v * v;
      }
    });
  } else {
    bn_for_each<1>(N, C, HW, c, s, [&](long long off, bool) {
      const float v = VecIO<T>::get(x + off);
      sum += v; sq += v * v;
    });
  }
  sum = block_sum(sum, scratch);
  sq = block_sum(sq, scratch);
  if (threadIdx.x == 0) {
    partial[(c * kBnSplits + s) * 2] = sum;
    partial[(c * kBnSplits + s) * 2 + 1] = sq;
  }
}

// grid (C, kBnSplits)
template <typename T>
__global__ void __launch_bounds__(kBnThreads)
bn_apply_kernel(const T* __restrict__ x, const T* __restrict__ residual, const float* __restrict__ gamma,
                const float* __restrict__ beta, const float* __restrict__ partial, float* __restrict__ running_mean,
                float* __restrict__ running_var, float* __restrict__ save_mean, float* __restrict__ save_rstd,
                T* __restrict__ y, int N, int C, int HW, float eps, float momentum, int relu, int training) {
  pdl_entry();
  constexpr int V = VecIO<T>::kVec;
  const int c = blockIdx.x, s = blockIdx.y;
  float mean, rstd;
  if (training) {
    float sum = 0.f, sq = 0.f;
#pragma unroll
    for (int i = 0; i < kBnSplits; ++i) {
      sum += partial[(c * kBnSplits + i) * 2];
      sq += partial[(c * kBnSplits + i) * 2 + 1];
    }
    const float cnt = static_cast<float>(N) * HW;
    mean = sum / cnt;
    const float var = fmaxf(sq / cnt - mean * mean, 0.f);
    rstd = rsqrtf(var + eps);
    if (s == 0 && threadIdx.x == 0) {
      save_mean[c] = mean;
      save_rstd[c] = rstd;
      if (running_mean) running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * mean;
      if (running_var) running_var[c] = (1.f - momentum) * running_var[c] + momentum * var * (cnt / fmaxf(cnt - 1.f, 1.f));
    }
  } else {
    mean = running_mean[c];
    rstd = rsqrtf(running_var[c] + eps);
  }
  const float g = gamma ? gamma[c] : 1.f, b = beta ? beta[c] : 0.f;
  const float scale = rstd * g, shift = b - mean * scale;
  const bool vec_ok = bn_aligned<T>(x) && bn_aligned<T>(y) && (!residual || bn_aligned<T>(residual));
  auto one = [&](long long off) {
    float v = VecIO<T>::get(x + off) * scale + shift;
    if (residual) v += VecIO<T>::get(residual + off);
    if (relu) v = fmaxf(v, 0.f);
    VecIO<T>::put(y + off, v);
  };
  if (vec_ok) {
    bn_for_each<V>(N, C, HW, c, s, [&](long long off, bool vec) {
      if (!vec) { one(off); return; }
      float v[V], r[V];
      VecIO<T>::load(x + off, v);
      if (residual) VecIO<T>::load(residual + off, r);
#pragma unroll
      for (int j = 0; j < V; ++j) {
        float o = fmaf(v[j], scale, shift);
        if (residual) o += r[j];
        v[j] = relu ? fmaxf(o, 0.f) : o;
      }
      VecIO<T>::store(y + off, v);
    });
  } else {
    bn_for_each<1>(N, C, HW, c, s, [&](long long off, bool) { one(off); });
  }
}

template <typename T>
__global__ void __launch_bounds__(kBnThreads)
bn_bwd_reduce_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ y,
                     const float* __restrict__ save_mean, const float* __restrict__ save_rstd, float* __restrict__ partial,
                     int N, int C, int HW, int relu) {
  pdl_entry();
  constexpr int V = VecIO<T>::kVec;
  __shared__ float scratch[32];
  const int c = blockIdx.x, s = blockIdx.y;
  const float mean = save_mean[c], rstd = save_rstd[c];
  float s1 = 0.f, s2 = 0.f;
  const bool vec_ok = bn_aligned<T>(dy) && bn_aligned<T>(x) && bn_aligned<T>(y);
  auto one = [&](long long off) {
    float g = VecIO<T>::get(dy + off);
    if (relu && VecIO<T>::get(y + off) <= 0.f) g = 0.f;
    s1 += g;
    s2 += g * (VecIO<T>::get(x + off) - mean) * rstd;
  };
  if (vec_ok) {
    bn_for_each<V>(N, C, HW, c, s, [&](long long off, bool vec) {
      if (!vec) { one(off); return; }
      float g[V], xv[V], yv[V];
      VecIO<T>::load(dy + off, g);
      VecIO<T>::load(x + off, xv);
      if (relu) VecIO<T>::load(y + off, yv);
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const float gj = (relu && yv[j] <= 0.f) ? 0.f : g[j];
        s1 += gj;
        s2 += gj * (xv[j] - mean) * rstd;
      }
    });
  } else {
    bn_for_each<1>(N, C, HW, c, s, [&](long long off, bool) { one(off); });
  }
  s1 = block_sum(s1, scratch);
  s2 = block_sum(s2, scratch);
  if (threadIdx.x == 0) {
    partial[(c * kBnSplits + s) * 2] = s1;
    partial[(c * kBnSplits + s) * 2 + 1] = s2;
  }
}

template <typename T>
__global__ void __launch_bounds__(kBnThreads)
bn_bwd_apply_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ y, const float* __restrict__ gamma,
                    const float* __restrict__ save_mean, const float* __restrict__ save_rstd, const float* __restrict__ partial,
                    T* __restrict__ dx, T* __restrict__ dres, float* __restrict__ dgamma, float* __restrict__ dbeta,
                    int accumulate, int N, int C, int HW, int relu) {
  pdl_entry();
  constexpr int V = VecIO<T>::kVec;
  const int c = blockIdx.x, s = blockIdx.y;
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int i = 0; i < kBnSplits; ++i) {
    s1 += partial[(c * kBnSplits + i) * 2];
    s2 += partial[(c * kBnSplits + i) * 2 + 1];
  }
  if (s == 0 && threadIdx.x == 0) {
    if (dgamma) dgamma[c] = accumulate ? dgamma[c] + s2 : s2;
    if (dbeta) dbeta[c] = accumulate ? dbeta[c] + s1 : s1;
  }
  const float cnt = static_cast<float>(N) * HW;
  const float mean = save_mean[c], rstd = save_rstd[c];
  const float g = gamma ? gamma[c] : 1.f;
  const float m1 = s1 / cnt, m2 = s2 / cnt;
  const float k = g * rstd;
  const bool vec_ok = bn_aligned<T>(dy) && bn_aligned<T>(x) && bn_aligned<T>(y) && bn_aligned<T>(dx) && (!dres || bn_aligned<T>(dres));
  auto one = [&](long long off) {
    float gy = VecIO<T>::get(dy + off);
    if (relu && VecIO<T>::get(y + off) <= 0.f) gy = 0.f;
    const float xh = (VecIO<T>::get(x + off) - mean) * rstd;
    VecIO<T>::put(dx + off, k * (gy - m1 - xh * m2));
    if (dres) VecIO<T>::put(dres + off, gy);
  };
  if (vec_ok) {
    bn_for_each<V>(N, C, HW, c, s, [&](long long off, bool vec) {
      if (!vec) { one(off); return; }
      float gy[V], xv[V], yv[V];
      VecIO<T>::load(dy + off, gy);
      VecIO<T>::load(x + off, xv);
      if (relu) VecIO<T>::load(y + off, yv);
#pragma unroll
      for (int j = 0; j < V; ++j) {
        if (relu && yv[j] <= 0.f) gy[j] = 0.f;
        xv[j] = k * (gy[j] - m1 - (xv[j] - mean) * rstd * m2);
      }
      VecIO<T>::store(dx + off, xv);
      if (dres) VecIO<T>::store(dres + off, gy);
    });
  } else {
    bn_for_each<1>(N, C, HW, c, s, [&](long long off, bool) { one(off); });
  }
}


// =============================================================================== channels-last
// The same four passes for an N-H-W-C tensor, seen as a [P, C] matrix (P = N*H*W pixels, the C
// channels of a pixel contiguous). This is the layout the tensor-core convolutions want, so a
// ResNet that stays channels-last end to end never pays for a layout transpose.
//
// A thread owns one 16-byte vector of channels (a fixed column group) and walks down the pixels;
// per-channel sums are folded across the block in shared memory and written as one partial row per
// block. The last block to finish (device counter) folds the partial rows, so each pass is still
// one launch: statistics pass -> mean / rstd / running stats, backward reduction -> dgamma, dbeta
// and the two means the dx pass needs.
constexpr int kBnMaxBlocks = 592;     // partial rows that the scratch holds; the passes take at most this many blocks

template <typename T>
struct NhwcMap {
  static constexpr int V = VecIO<T>::kVec;
  int cv, lanes;          // vectors per pixel, pixels per block iteration
  __device__ NhwcMap(int C) : cv(C / V), lanes(kBnThreads / (C / V)) {}
  __device__ bool active() const { return static_cast<int>(threadIdx.x) < lanes * cv; }
  __device__ int col() const { return (threadIdx.x % cv) * V; }
  __device__ int lane() const { return threadIdx.x / cv; }
};

// Fold this block's per-thread channel sums (a[V], b[V]) and publish them as partial row
// blockIdx.x; returns true in the block that finished last.
template <typename T>
__device__ __forceinline__ bool nhwc_publish(const NhwcMap<T>& m, int C, const float (&a)[VecIO<T>::kVec], const float (&b)[VecIO<T>::kVec],
                                             float* __restrict__ partial, unsigned int* __restrict__ counter, float* sm) {
  constexpr int V = VecIO<T>::kVec;
  // sm: [2][lanes][C]
  __shared__ bool last;
  if (m.active()) {
#pragma unroll
    for (int j = 0; j < V; j += 4) {
      *reinterpret_cast<float4*>(sm + m.lane() * C + m.col() + j) = make_float4(a[j], a[j + 1], a[j + 2], a[j + 3]);
      *reinterpret_cast<float4*>(sm + (m.lanes + m.lane()) * C + m.col() + j) = make_float4(b[j], b[j + 1], b[j + 2], b[j + 3]);
    }
  }
  __syncthreads();
  // the 2C columns over all threads: `slices` threads share one
  const int slices = kBnThreads / (2 * C);
  float* row = partial + static_cast<long long>(blockIdx.x) * 2 * C;
  if (slices > 1) {
    const int c = threadIdx.x % (2 * C), sl = threadIdx.x / (2 * C), which = c / C, ch = c - which * C;
    float acc = 0.f;
    if (sl < slices)
      for (int l = sl; l < m.lanes; l += slices) acc += sm[(which * m.lanes + l) * C + ch];
    __syncthreads();
    sm[threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.x < 2 * C) {
      acc = 0.f;
      for (int k = 0; k < slices; ++k) acc += sm[k * 2 * C + threadIdx.x];
      row[threadIdx.x] = acc;
    }
  } else {
    for (int c = threadIdx.x; c < 2 * C; c += kBnThreads) {
      const int which = c / C, ch = c - which * C;
      float acc = 0.f;
      for (int l = 0; l < m.lanes; ++l) acc += sm[(which * m.lanes + l) * C + ch];
      row[c] = acc;
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// Sum of partial rows [0, nrows) for every channel, both planes, by the whole block: a thread takes four columns of every
// slices-th row, eight rows in flight (one block reads all rows while the device waits, so what counts is the chain of L2 latencies);
// slices are then folded through shared memory. Results land in sm[0 .. 2C): plane 0 then plane 1.
// The backward's reduction over a ResNet-20 step, us per launch, with one column and four rows in flight against this: batch 1000
// 21.8 -> 17.5, batch 128 9.1 -> 8.0.
__device__ __forceinline__ void nhwc_fold(const float* __restrict__ partial, int nrows, int C, float* sm) {
  constexpr int kRows = 8;
  const int four = C / 2, slices = kBnThreads / four;       // C is a multiple of 4 and at most kBnThreads
  const int c4 = (threadIdx.x % four) * 4, sl = threadIdx.x / four;
  const bool whole = (reinterpret_cast<uintptr_t>(partial) & 15) == 0;
  auto load = [&](int row) {
    const float* p = partial + static_cast<long long>(row) * 2 * C + c4;
    return whole ? __ldcg(reinterpret_cast<const float4*>(p)) : make_float4(__ldcg(p), __ldcg(p + 1), __ldcg(p + 2), __ldcg(p + 3));
  };
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (sl < slices) {
    for (int i = sl; i < nrows; i += kRows * slices) {
      float4 v[kRows];
#pragma unroll
      for (int u = 0; u < kRows; ++u) v[u] = i + u * slices < nrows ? load(i + u * slices) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int u = 0; u < kRows; ++u) { acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w; }
    }
  }
  __syncthreads();
  // sm has room for 4 * kBnThreads floats: 2 * lanes * C of them, lanes * C more than kBnThreads * V less one pixel's
  *reinterpret_cast<float4*>(sm + 4 * threadIdx.x) = acc;
  __syncthreads();
  float t[2] = {0.f, 0.f};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = threadIdx.x + h * kBnThreads;
    if (c < 2 * C)
      for (int k = 0; k < slices; ++k) t[h] += sm[k * 2 * C + c];
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (threadIdx.x + h * kBnThreads < 2 * C) sm[threadIdx.x + h * kBnThreads] = t[h];
  __syncthreads();
}

// The channels-last passes below read up to three tensors and write up to two, once each: HBM (or, at CIFAR batches, L2) bounds them if enough
// loads are in flight. A thread fetches four pixels of every tensor before it works on the first, on as many blocks per SM as the registers of that
// allow, in one wave; the statistics pass, one tensor and two sums, does better with more blocks and a loop that the compiler unrolls.
// us back to back, bf16, [pixels, channels] of 128 x 32 x 32 x 16 / 1000 x 32 x 32 x 64, in brackets all passes with two pixels and three blocks: statistics
// 5.7 / 31 (6.4 / 55), apply 3.2 / 43 (3.4 / 51), with residual 3.5 / 64 (3.8 / 63), backward sums 6.7 / 65 (7.7 / 67), backward apply 3.6 / 79 (5.7 / 97).
constexpr int kBnBatch = 4;
constexpr int kBnStatsPerSm = 4, kBnApplyPerSm = 3, kBnBwdPerSm = 2;

template <typename T>
__global__ void __launch_bounds__(kBnThreads, kBnStatsPerSm)
bn_nhwc_stats_kernel(const T* __restrict__ x, float* __restrict__ partial, unsigned int* __restrict__ counter,
                     float* __restrict__ running_mean, float* __restrict__ running_var, float* __restrict__ save_mean,
                     float* __restrict__ save_rstd, long long P, int C, float eps, float momentum) {
  pdl_entry();
  constexpr int V = VecIO<T>::kVec;
  extern __shared__ __align__(16) float sm[];
  const NhwcMap<T> m(C);
  float a[V], b[V];
#pragma unroll
  for (int j = 0; j < V; ++j) a[j] = b[j] = 0.f;
  if (m.active()) {
    for (long long p = static_cast<long long>(blockIdx.x) * m.lanes + m.lane(); p < P; p += static_cast<long long>(gridDim.x) * m.lanes) {
      float v[V];
      VecIO<T>::load(x + p * C + m.col(), v);
#pragma unroll
      for (int j = 0; j < V; ++j) { a[j] += v[j]; b[j] += v[j] * v[j]; }
    }
  }
  if (!nhwc_publish<T>(m, C, a, b, partial, counter, sm)) return;
  nhwc_fold(partial, static_cast<int>(gridDim.x), C, sm);
  for (int c = threadIdx.x; c < C; c += kBnThreads) {
    const float sum = sm[c], sq = sm[C + c];
    const float cnt = static_cast<float>(P);
    const float mean = sum / cnt;
    const float var = fmaxf(sq / cnt - mean * mean, 0.f);
    save_mean[c] = mean;
    save_rstd[c] = rsqrtf(var + eps);
    if (running_mean) running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * mean;
    if (running_var) running_var[c] = (1.f - momentum) * running_var[c] + momentum * var * (cnt / fmaxf(cnt - 1.f, 1.f));
  }
  if (threadIdx.x == 0) *counter = 0;      // ready for the next launch
}

// kFromSums: the per-channel sum and sum of squares were accumulated by the kernel that produced x (the
// convolution's epilogue); every thread derives mean and 1/std of its own channels from them, block 0
// also records them for the backward pass and updates the running statistics. One launch, no
// statistics pass over x.
template <typename T, bool kFromSums>
__global__ void __launch_bounds__(kBnThreads, kBnApplyPerSm)
bn_nhwc_apply_kernel(const T* __restrict__ x, const T* __restrict__ residual, const float* __restrict__ gamma,
                     const float* __restrict__ beta, const float* __restrict__ mean, const float* __restrict__ rstd,
                     T* __restrict__ y, long long P, int C, int relu, const float* __restrict__ sums, float* __restrict__ save_mean,
                     float* __restrict__ save_rstd, float* __restrict__ running_mean, float* __restrict__ running_var, float eps,
                     float momentum) {
  pdl_entry();
  constexpr int V = VecIO<T>::kVec;
  const NhwcMap<T> m(C);
  if (!m.active()) return;
  float scale[V], shift[V];
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int c = m.col() + j;
    const float g = gamma ? gamma[c] : 1.f, b = beta ? beta[c] : 0.f;
    float mu, rs;
    if (kFromSums) {
      const float cnt = static_cast<float>(P);
      mu = sums[c] / cnt;
      const float var = fmaxf(sums[C + c] / cnt - mu * mu, 0.f);
      rs = rsqrtf(var + eps);
      if (blockIdx.x == 0 && m.lane() == 0) {
        save_mean[c] = mu;
        save_rstd[c] = rs;
        if (running_mean) running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * mu;
        if (running_var) running_var[c] = (1.f - momentum) * running_var[c] + momentum * var * (cnt / fmaxf(cnt - 1.f, 1.f));
      }
    } else {
      mu = mean[c];
      rs = rstd[c];
    }
    scale[j] = rs * g;
    shift[j] = b - mu * scale[j];
  }
  const long long step = static_cast<long long>(gridDim.x) * m.lanes;
  for (long long p0 = static_cast<long long>(blockIdx.x) * m.lanes + m.lane(); p0 < P; p0 += kBnBatch * step) {
    uint4 xr[kBnBatch], rr[kBnBatch];
#pragma unroll
    for (int u = 0; u < kBnBatch; ++u) {
      const long long at = (p0 + u * step) * C + m.col();
      if (p0 + u * step < P) {
        xr[u] = *reinterpret_cast<const uint4*>(x + at);
        if (residual) rr[u] = *reinterpret_cast<const uint4*>(residual + at);
      }
    }
#pragma unroll
    for (int u = 0; u < kBnBatch; ++u) {
      if (p0 + u * step >= P) break;
      float v[V], r[V];
      VecIO<T>::unpack(xr[u], v);
      if (residual) VecIO<T>::unpack(rr[u], r);
#pragma unroll
      for (int j = 0; j < V; ++j) {
        float o = fmaf(v[j], scale[j], shift[j]);
        if (residual) o += r[j];
        v[j] = relu ? fmaxf(o, 0.f) : o;
      }
      VecIO<T>::store(y + (p0 + u * step) * C + m.col(), v);
    }
  }
}

// fold[0..C) = mean of dy', fold[C..2C) = mean of dy' * xhat
template <typename T>
__global__ void __launch_bounds__(kBnThreads, kBnBwdPerSm)
bn_nhwc_bwd_reduce_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ y, const float* __restrict__ mean,
                          const float* __restrict__ rstd, float* __restrict__ partial, unsigned int* __restrict__ counter,
                          float* __restrict__ fold, float* __restrict__ dgamma, float* __restrict__ dbeta, int accumulate,
                          long long P, int C, int relu) {
  pdl_entry();
  constexpr int V = VecIO<T>::kVec;
  extern __shared__ __align__(16) float sm[];
  const NhwcMap<T> m(C);
  float a[V], b[V], mu[V];
#pragma unroll
  for (int j = 0; j < V; ++j) a[j] = b[j] = 0.f;
  if (m.active()) {
#pragma unroll
    for (int j = 0; j < V; ++j) mu[j] = mean[m.col() + j];
    const long long step = static_cast<long long>(gridDim.x) * m.lanes;
    for (long long p0 = static_cast<long long>(blockIdx.x) * m.lanes + m.lane(); p0 < P; p0 += kBnBatch * step) {
      uint4 gr[kBnBatch], xr[kBnBatch], yr[kBnBatch];
#pragma unroll
      for (int u = 0; u < kBnBatch; ++u) {
        const long long at = (p0 + u * step) * C + m.col();
        if (p0 + u * step < P) {
          gr[u] = *reinterpret_cast<const uint4*>(dy + at);
          xr[u] = *reinterpret_cast<const uint4*>(x + at);
          if (relu) yr[u] = *reinterpret_cast<const uint4*>(y + at);
        }
      }
#pragma unroll
      for (int u = 0; u < kBnBatch; ++u) {
        if (p0 + u * step >= P) break;
        float g[V], xv[V], yv[V];
        VecIO<T>::unpack(gr[u], g);
        VecIO<T>::unpack(xr[u], xv);
        if (relu) VecIO<T>::unpack(yr[u], yv);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          const float gj = (relu && yv[j] <= 0.f) ? 0.f : g[j];
          a[j] += gj;
          b[j] += gj * (xv[j] - mu[j]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < V; ++j) b[j] *= rstd[m.col() + j];       // a column's own factor: once, not per pixel
  }
  if (!nhwc_publish<T>(m, C, a, b, partial, counter, sm)) return;
  nhwc_fold(partial, static_cast<int>(gridDim.x), C, sm);
  for (int c = threadIdx.x; c < C; c += kBnThreads) {
    const float s1 = sm[c], s2 = sm[C + c];
    if (dgamma) dgamma[c] = accumulate ? dgamma[c] + s2 : s2;
    if (dbeta) dbeta[c] = accumulate ? dbeta[c] + s1 : s1;
    fold[c] = s1 / static_cast<float>(P);
    fold[C + c] = s2 / static_cast<float>(P);
  }
  if (threadIdx.x == 0) *counter = 0;
}

template <typename T>
__global__ void __launch_bounds__(kBnThreads, kBnBwdPerSm)
bn_nhwc_bwd_apply_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ y, const float* __restrict__ gamma,
                         const float* __restrict__ mean, const float* __restrict__ rstd, const float* __restrict__ fold,
                         T* __restrict__ dx, T* __restrict__ dres, long long P, int C, int relu) {
  pdl_entry();
  constexpr int V = VecIO<T>::kVec;
  const NhwcMap<T> m(C);
  if (!m.active()) return;
  float mu[V], k[V], m1[V], q[V];
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int c = m.col() + j;
    const float rs = rstd[c];
    mu[j] = mean[c];
    k[j] = (gamma ? gamma[c] : 1.f) * rs;
    m1[j] = fold[c];
    q[j] = rs * fold[C + c];
  }
  const long long step = static_cast<long long>(gridDim.x) * m.lanes;
  for (long long p0 = static_cast<long long>(blockIdx.x) * m.lanes + m.lane(); p0 < P; p0 += kBnBatch * step) {
    uint4 gr[kBnBatch], xr[kBnBatch], yr[kBnBatch];
#pragma unroll
    for (int u = 0; u < kBnBatch; ++u) {
      const long long at = (p0 + u * step) * C + m.col();
      if (p0 + u * step < P) {
        gr[u] = *reinterpret_cast<const uint4*>(dy + at);
        xr[u] = *reinterpret_cast<const uint4*>(x + at);
        if (relu) yr[u] = *reinterpret_cast<const uint4*>(y + at);
      }
    }
#pragma unroll
    for (int u = 0; u < kBnBatch; ++u) {
      if (p0 + u * step >= P) break;
      const long long at = (p0 + u * step) * C + m.col();
      float g[V], xv[V], yv[V];
      VecIO<T>::unpack(gr[u], g);
      VecIO<T>::unpack(xr[u], xv);
      if (relu) VecIO<T>::unpack(yr[u], yv);
#pragma unroll
      for (int j = 0; j < V; ++j) {
        if (relu && yv[j] <= 0.f) g[j] = 0.f;
        xv[j] = k[j] * (g[j] - m1[j] - (xv[j] - mu[j]) * q[j]);
      }
      VecIO<T>::store(dx + at, xv);
      if (dres) VecIO<T>::store(dres + at, g);
    }
  }
}

static int nhwc_iters() {
  static int it = 0;
  if (!it) {
    const char* e = getenv("FLODL_B200_BN_ITERS");
    it = e ? atoi(e) : 4;      // pixels per thread; measured on a ResNet-20 step: 8 -> 1.398 ms, 4 -> 1.327, 2 -> 1.341, 1 -> 1.400
    if (it < 1) it = 4;
  }
  return it;
}
static int nhwc_grid(long long P, int C, int V, int per_sm) {
  const int lanes = kBnThreads / (C / V);
  const long long per = static_cast<long long>(lanes) * nhwc_iters();
  long long want = (P + per - 1) / per;
  if (want < 1) want = 1;
  int wave = sm_count() * per_sm;
  if (wave > kBnMaxBlocks) wave = kBnMaxBlocks;
  return static_cast<int>(want < wave ? want : wave);
}

}  // namespace fb

// Channels-last entry points. C must be a multiple of the 16-byte vector (8 bf16 / 4 fp32) and at most
// 256; scratch holds fb_bn_nhwc_scratch_floats(C) floats; `counter` is one zero-initialised word the
// kernels leave at zero.
extern "C" int fb_bn_nhwc_scratch_floats(int C) { return (fb::kBnMaxBlocks * 2 + 2) * C; }

extern "C" int fb_bn_nhwc_fwd(const void* x, const void* residual, const float* gamma, const float* beta, float* running_mean,
                              float* running_var, void* y, float* save_mean, float* save_rstd, float* scratch, unsigned int* counter,
                              long long P, int C, float eps, float momentum, int relu, int training, int is_bf16, void* stream) {
  using namespace fb;
  if (P <= 0 || C <= 0) return 0;
  const int V = is_bf16 ? 8 : 4;
  if (C % V || C > kBnThreads) return -4;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid_stats = nhwc_grid(P, C, V, kBnStatsPerSm), grid = nhwc_grid(P, C, V, kBnApplyPerSm);
  const int lanes = kBnThreads / (C / V);
  const size_t smem = sizeof(float) * 2 * lanes * C;
  const float* mean = training ? save_mean : running_mean;
  if (is_bf16) {
    using T = __nv_bfloat16;
    if (training)
      launch_pdl(bn_nhwc_stats_kernel<T>, dim3(grid_stats), dim3(kBnThreads), smem, st, static_cast<const T*>(x), scratch, counter, running_mean, running_var,
                                                             save_mean, save_rstd, P, C, eps, momentum);
    else return -6;   // evaluation mode goes through the framework's generic path
    launch_pdl(bn_nhwc_apply_kernel<T, false>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(x), static_cast<const T*>(residual), gamma, beta, mean,
                                                               save_rstd, static_cast<T*>(y), P, C, relu, nullptr, nullptr, nullptr, nullptr,
                                                               nullptr, 0.f, 0.f);
  } else {
    using T = float;
    if (training)
      launch_pdl(bn_nhwc_stats_kernel<T>, dim3(grid_stats), dim3(kBnThreads), smem, st, static_cast<const T*>(x), scratch, counter, running_mean, running_var,
                                                             save_mean, save_rstd, P, C, eps, momentum);
    else return -6;
    launch_pdl(bn_nhwc_apply_kernel<T, false>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(x), static_cast<const T*>(residual), gamma, beta, mean,
                                                               save_rstd, static_cast<T*>(y), P, C, relu, nullptr, nullptr, nullptr, nullptr,
                                                               nullptr, 0.f, 0.f);
  }
  return static_cast<int>(cudaGetLastError());
}

// Training-mode forward whose statistics come from `sums` (fp32 [2][C]: per-channel sum and sum of
// squares of x over its P pixels, e.g. from fb_conv_fprop). One launch.
extern "C" int fb_bn_nhwc_fwd_sums(const void* x, const void* residual, const float* gamma, const float* beta, float* running_mean,
                                   float* running_var, void* y, float* save_mean, float* save_rstd, const float* sums, long long P, int C,
                                   float eps, float momentum, int relu, int is_bf16, void* stream) {
  using namespace fb;
  if (P <= 0 || C <= 0) return 0;
  const int V = is_bf16 ? 8 : 4;
  if (C % V || C > kBnThreads || !sums) return -4;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = nhwc_grid(P, C, V, kBnApplyPerSm);
  if (is_bf16) {
    using T = __nv_bfloat16;
    launch_pdl(bn_nhwc_apply_kernel<T, true>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(x), static_cast<const T*>(residual), gamma, beta, nullptr,
                                                              nullptr, static_cast<T*>(y), P, C, relu, sums, save_mean, save_rstd, running_mean,
                                                              running_var, eps, momentum);
  } else {
    using T = float;
    launch_pdl(bn_nhwc_apply_kernel<T, true>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(x), static_cast<const T*>(residual), gamma, beta, nullptr,
                                                              nullptr, static_cast<T*>(y), P, C, relu, sums, save_mean, save_rstd, running_mean,
                                                              running_var, eps, momentum);
  }
  return static_cast<int>(cudaGetLastError());
}

extern "C" int fb_bn_nhwc_bwd(const void* dy, const void* x, const void* y, const float* gamma, const float* save_mean,
                              const float* save_rstd, void* dx, void* dresidual, float* dgamma, float* dbeta, int accumulate,
                              float* scratch, unsigned int* counter, long long P, int C, int relu, int is_bf16, void* stream) {
  using namespace fb;
  if (P <= 0 || C <= 0) return 0;
  const int V = is_bf16 ? 8 : 4;
  if (C % V || C > kBnThreads) return -4;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = nhwc_grid(P, C, V, kBnBwdPerSm);
  const int lanes = kBnThreads / (C / V);
  const size_t smem = sizeof(float) * 2 * lanes * C;
  float* fold = scratch + static_cast<long long>(kBnMaxBlocks) * 2 * C;
  if (is_bf16) {
    using T = __nv_bfloat16;
    launch_pdl(bn_nhwc_bwd_reduce_kernel<T>, dim3(grid), dim3(kBnThreads), smem, st, static_cast<const T*>(dy), static_cast<const T*>(x), static_cast<const T*>(y),
                                                                save_mean, save_rstd, scratch, counter, fold, dgamma, dbeta, accumulate, P, C, relu);
    launch_pdl(bn_nhwc_bwd_apply_kernel<T>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(dy), static_cast<const T*>(x), static_cast<const T*>(y), gamma,
                                                            save_mean, save_rstd, fold, static_cast<T*>(dx), static_cast<T*>(dresidual), P, C, relu);
  } else {
    using T = float;
    launch_pdl(bn_nhwc_bwd_reduce_kernel<T>, dim3(grid), dim3(kBnThreads), smem, st, static_cast<const T*>(dy), static_cast<const T*>(x), static_cast<const T*>(y),
                                                                save_mean, save_rstd, scratch, counter, fold, dgamma, dbeta, accumulate, P, C, relu);
    launch_pdl(bn_nhwc_bwd_apply_kernel<T>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(dy), static_cast<const T*>(x), static_cast<const T*>(y), gamma,
                                                            save_mean, save_rstd, fold, static_cast<T*>(dx), static_cast<T*>(dresidual), P, C, relu);
  }
  return static_cast<int>(cudaGetLastError());
}

extern "C" int fb_bn_scratch_floats(int C) { return C * fb::kBnSplits * 2; }

// scratch: fb_bn_scratch_floats(C) floats.
extern "C" int fb_bn_fwd(const void* x, const void* residual, const float* gamma, const float* beta, float* running_mean,
                         float* running_var, void* y, float* save_mean, float* save_rstd, float* scratch, int N, int C,
                         int HW, float eps, float momentum, int relu, int training, int is_bf16, void* stream) {
  using namespace fb;
  if (N <= 0 || C <= 0 || HW <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  dim3 grid(C, kBnSplits);
  if (is_bf16) {
    using T = __nv_bfloat16;
    if (training) launch_pdl(bn_stats_kernel<T>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(x), scratch, N, C, HW);
    launch_pdl(bn_apply_kernel<T>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(x), static_cast<const T*>(residual), gamma, beta, scratch,
                                                    running_mean, running_var, save_mean, save_rstd, static_cast<T*>(y), N, C, HW,
                                                    eps, momentum, relu, training);
  } else {
    using T = float;
    if (training) launch_pdl(bn_stats_kernel<T>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(x), scratch, N, C, HW);
    launch_pdl(bn_apply_kernel<T>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(x), static_cast<const T*>(residual), gamma, beta, scratch,
                                                    running_mean, running_var, save_mean, save_rstd, static_cast<T*>(y), N, C, HW,
                                                    eps, momentum, relu, training);
  }
  return static_cast<int>(cudaGetLastError());
}

extern "C" int fb_bn_bwd(const void* dy, const void* x, const void* y, const float* gamma, const float* save_mean,
                         const float* save_rstd, void* dx, void* dresidual, float* dgamma, float* dbeta, int accumulate,
                         float* scratch, int N, int C, int HW, int relu, int is_bf16, void* stream) {
  using namespace fb;
  if (N <= 0 || C <= 0 || HW <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  dim3 grid(C, kBnSplits);
  if (is_bf16) {
    using T = __nv_bfloat16;
    launch_pdl(bn_bwd_reduce_kernel<T>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(dy), static_cast<const T*>(x), static_cast<const T*>(y),
                                                         save_mean, save_rstd, scratch, N, C, HW, relu);
    launch_pdl(bn_bwd_apply_kernel<T>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(dy), static_cast<const T*>(x), static_cast<const T*>(y),
                                                        gamma, save_mean, save_rstd, scratch, static_cast<T*>(dx),
                                                        static_cast<T*>(dresidual), dgamma, dbeta, accumulate, N, C, HW, relu);
  } else {
    using T = float;
    launch_pdl(bn_bwd_reduce_kernel<T>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(dy), static_cast<const T*>(x), static_cast<const T*>(y),
                                                         save_mean, save_rstd, scratch, N, C, HW, relu);
    launch_pdl(bn_bwd_apply_kernel<T>, dim3(grid), dim3(kBnThreads), 0, st, static_cast<const T*>(dy), static_cast<const T*>(x), static_cast<const T*>(y),
                                                        gamma, save_mean, save_rstd, scratch, static_cast<T*>(dx),
                                                        static_cast<T*>(dresidual), dgamma, dbeta, accumulate, N, C, HW, relu);
  }
  return static_cast<int>(cudaGetLastError());
}

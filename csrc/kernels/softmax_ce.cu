// Fused softmax cross-entropy: one pass for the row statistics, one pass that writes the gradient.
//
// Replaces `at::cross_entropy_loss` (flodl-sys/ops_training.cpp:926-937; mean reduction,
// ignore_index) and the log_softmax / nll backward kernels libtorch runs for it. Logits may be
// bf16 or fp32; all math is fp32. The gradient (softmax - onehot) / n_valid is produced in the
// forward launch (it may overwrite the logits), so the backward pass is a scalar multiply that the
// consumer GEMMs take as their `alpha`.
#include <type_traits>

#include "../include/flodl_b200.h"
#include "common.cuh"

namespace fb {

__global__ void ce_count_kernel(const long long* __restrict__ targets, int rows, long long ignore_index,
                                float* __restrict__ count_inv /* [0]=count, [1]=1/max(count,1) */) {
  pdl_entry();
  __shared__ float scratch[32];
  float c = 0.f;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) c += (targets[i] != ignore_index) ? 1.f : 0.f;
  c = block_sum(c, scratch);
  if (threadIdx.x == 0) {
    count_inv[0] = c;
    count_inv[1] = 1.f / fmaxf(c, 1.f);
  }
}

// A row of `n` values as 16-byte vectors and the few values before the first and after the last whole one: rows of an odd
// length, one after the other, start at any multiple of the element size. `b` (may be null) is a second row walked in step;
// if the two are aligned differently everything is left to the single values.
template <typename T>
struct RowSplit {
  int head, nvec, tail;       // values [0, head) and [tail, n) one by one, nvec vectors from `head` on
  __device__ RowSplit(const T* a, const T* b, int n) {
    constexpr int V = VecIO<T>::kVec;
    const uintptr_t pa = reinterpret_cast<uintptr_t>(a), pb = b ? reinterpret_cast<uintptr_t>(b) : pa;
    head = (pa ^ pb) & 15 ? n : min(n, static_cast<int>(((16 - (pa & 15)) & 15) / sizeof(T)));
    nvec = (n - head) / V;
    tail = head + nvec * V;
  }
};

// exp(v - base) of two values: the difference first, then the power of two, as for one.
__device__ __forceinline__ F2 f2_exp_from(F2 v, F2 minus_base) {
  float lo, hi;
  f2_get(f2_mul(f2_add(v, minus_base), f2_splat(1.4426950408889634f)), lo, hi);
  return f2_make(ex2_approx(lo), ex2_approx(hi));
}
// Maximum and sum of exponentials relative to it, over a stream of values; -inf values (and rows of nothing else) add nothing.
struct OnlineSum {
  float m = -INFINITY;
  F2 s2 = f2_splat(0.f);
  __device__ __forceinline__ void reach(float vm) {
    if (vm > m) {
      s2 = f2_mul(s2, f2_splat(__expf(m - vm)));
      m = vm;
    }
  }
  template <int N>
  __device__ __forceinline__ void add(const float (&v)[N]) {
    float vm = v[0];
#pragma unroll
    for (int j = 1; j < N; ++j) vm = fmaxf(vm, v[j]);
    reach(vm);
    const F2 minus = f2_splat(m == -INFINITY ? 0.f : -m);
#pragma unroll
    for (int j = 0; j < N; j += 2) s2 = f2_add(s2, f2_exp_from(f2_make(v[j], v[j + 1]), minus));
  }
  __device__ __forceinline__ void add(float v) {
    reach(v);
    s2 = f2_add(s2, f2_make(__expf(v - (m == -INFINITY ? 0.f : m)), 0.f));
  }
  __device__ __forceinline__ float sum() const {
    float lo, hi;
    f2_get(s2, lo, hi);
    return lo + hi;
  }
};
// A sum without a maximum is 0, or NaN if all its values were NaN, and stays what it is.
__device__ __forceinline__ float sum_rebased(float s, float m, float to) { return m == -INFINITY ? s : s * __expf(m - to); }

// One row per block or, for short rows, per warp. The row is read twice, for the statistics and for the gradient, and written once. What bounds it is
// HBM where the second read finds the row in L2, so that a row's threads times the resident blocks' rows decide: few threads to a row keep the
// barrier and the exponentials of one row behind the loads of others, but put more rows in flight; long rows then leave L2 between their reads.
// Exponentials (two a value) and issue slots are not far behind, so the arithmetic goes two values an instruction and the target is looked for once
// per vector. us for a mean loss with its gradient; in brackets one value an instruction, before that a 256-thread block per row:
//   bf16 4000 x 3000 17.5 (20.3, 19.8), 8192 x 8000 64.5 (74.2, 72.7), 4096 x 32000 114 (126), 8192 x 32000 219 (238, 266), 2048 x 50304 88 (103);
//   fp32 8192 x 4000 57.1 (56.6, 64.0), 2094 x 23544 81 (81, 107), 4096 x 30522 181 (187, 396).
// kUnroll vectors in flight per thread, kBlocks blocks of kThreads on an SM.
template <typename T, bool kWarpRow, int kThreads, int kBlocks, int kUnroll>
__global__ void __launch_bounds__(kThreads, kBlocks)
ce_fwd_kernel(const T* __restrict__ logits, long long ld, const long long* __restrict__ targets, int rows,
              int V, long long ignore_index, T* __restrict__ dlogits, long long ldd,
              const float* __restrict__ count_inv, float* __restrict__ row_loss, const int* __restrict__ counts) {
  pdl_entry();
  constexpr int VEC = VecIO<T>::kVec;
  constexpr int kWarps = kThreads / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int me = kWarpRow ? lane : threadIdx.x, row = kWarpRow ? blockIdx.x * kWarps + warp : blockIdx.x;
  constexpr int step = kWarpRow ? 32 : kThreads;
  if (kWarpRow && row >= rows) return;
  if (counts) (void)FB_INDEX_OK(counts[0], static_cast<long long>(rows) + 1, 202);
  if (counts && row >= counts[1]) {      // compacted input: nothing lives past the padded count
    if (row_loss && me == 0) row_loss[row] = 0.f;
    return;
  }
  const long long t = targets[row];
  const T* lr = logits + static_cast<long long>(row) * ld;
  T* dr = dlogits ? dlogits + static_cast<long long>(row) * ldd : nullptr;
  const RowSplit<T> sp(lr, dr, V);
  if (t != ignore_index) (void)FB_INDEX_OK(t, V, 201);        // a label outside the vocabulary is recorded (and treated as ignored)
  if (t == ignore_index || t < 0 || t >= V) {
    if (row_loss && me == 0) row_loss[row] = 0.f;
    if (dr) {
      float z[VEC];
#pragma unroll
      for (int j = 0; j < VEC; ++j) z[j] = 0.f;
      for (int k = me; k < sp.head; k += step) VecIO<T>::put(dr + k, 0.f);
      for (int i = me; i < sp.nvec; i += step) VecIO<T>::store(dr + sp.head + i * VEC, z);
      for (int k = sp.tail + me; k < V; k += step) VecIO<T>::put(dr + k, 0.f);
    }
    return;
  }
  const float x_t = me == 0 && row_loss ? VecIO<T>::get(lr + t) : 0.f;      // before the gradient may overwrite it
  if constexpr (kWarpRow) __syncwarp();

  OnlineSum acc;
  for (int k = me; k < sp.head; k += step) acc.add(VecIO<T>::get(lr + k));
  for (int k = sp.tail + me; k < V; k += step) acc.add(VecIO<T>::get(lr + k));
  const T* body = lr + sp.head;
  int i = me;
  for (; i + (kUnroll - 1) * step < sp.nvec; i += kUnroll * step) {
    float v[kUnroll][VEC];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) VecIO<T>::load(body + static_cast<long long>(i + u * step) * VEC, v[u]);
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) acc.add(v[u]);
  }
  for (; i < sp.nvec; i += step) {
    float v[VEC];
    VecIO<T>::load(body + static_cast<long long>(i) * VEC, v);
    acc.add(v);
  }
  float gmax = warp_max(acc.m);
  float gsum = warp_sum(sum_rebased(acc.sum(), acc.m, gmax));
  if constexpr (!kWarpRow) {
    __shared__ float red_m[kWarps], red_s[kWarps];
    if (lane == 0) { red_m[warp] = gmax; red_s[warp] = gsum; }
    __syncthreads();
    const float wm = lane < kWarps ? red_m[lane] : -INFINITY, ws = lane < kWarps ? red_s[lane] : 0.f;
    gmax = warp_max(wm);
    gsum = warp_sum(sum_rebased(ws, wm, gmax));
  }
  if (row_loss && me == 0) row_loss[row] = __logf(gsum) + gmax - x_t;
  if (!dr) return;

  const float inv_n = count_inv ? count_inv[1] : 1.f, inv_sum = 1.f / gsum;
  T* dbody = dr + sp.head;
  auto grad = [&](float x, int k) { return (__expf(x - gmax) * inv_sum - (k == t ? 1.f : 0.f)) * inv_n; };
  // a vector's: two values an instruction, and the target looked for once per vector
  const F2 minus = f2_splat(-gmax), scale = f2_splat(inv_sum * inv_n);
  const int t_vec = t >= sp.head && t < sp.tail ? static_cast<int>(t - sp.head) / VEC : -1, t_at = static_cast<int>(t - sp.head) % VEC;
  auto grads = [&](float (&v)[VEC], int vec) {
    float x_target = 0.f;
    if (vec == t_vec) {
#pragma unroll
      for (int j = 0; j < VEC; ++j)
        if (j == t_at) x_target = v[j];
    }
#pragma unroll
    for (int j = 0; j < VEC; j += 2) f2_get(f2_mul(f2_exp_from(f2_make(v[j], v[j + 1]), minus), scale), v[j], v[j + 1]);
    if (vec == t_vec) {
#pragma unroll
      for (int j = 0; j < VEC; ++j)
        if (j == t_at) v[j] = (__expf(x_target - gmax) * inv_sum - 1.f) * inv_n;
    }
  };
  for (int k = me; k < sp.head; k += step) VecIO<T>::put(dr + k, grad(VecIO<T>::get(lr + k), k));
  for (int k = sp.tail + me; k < V; k += step) VecIO<T>::put(dr + k, grad(VecIO<T>::get(lr + k), k));
  i = me;
  for (; i + (kUnroll - 1) * step < sp.nvec; i += kUnroll * step) {
    float v[kUnroll][VEC];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) VecIO<T>::load(body + static_cast<long long>(i + u * step) * VEC, v[u]);
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      grads(v[u], i + u * step);
      VecIO<T>::store(dbody + static_cast<long long>(i + u * step) * VEC, v[u]);
    }
  }
  for (; i < sp.nvec; i += step) {
    float v[VEC];
    VecIO<T>::load(body + static_cast<long long>(i) * VEC, v);
    grads(v, i);
    VecIO<T>::store(dbody + static_cast<long long>(i) * VEC, v);
  }
}

// loss = sum(row_loss) / max(count, 1), in a fixed order (deterministic).
__global__ void ce_finalize_kernel(const float* __restrict__ row_loss, int rows, const float* __restrict__ count_inv,
                                   float* __restrict__ loss) {
  pdl_entry();
  __shared__ float scratch[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) s += row_loss[i];
  s = block_sum(s, scratch);
  if (threadIdx.x == 0) loss[0] = s * count_inv[1];
}

// x[r][c] *= *scalar (device scalar); rows of length `cols` with leading dimension `ld`. A factor of one, which is what the
// gradient of a loss that is differentiated itself arrives with, leaves x as it is and costs the launch only.
template <typename T>
__global__ void __launch_bounds__(256) scale_rows_kernel(T* __restrict__ x, long long ld, int rows, int cols, const float* __restrict__ scalar) {
  pdl_entry();
  constexpr int VEC = VecIO<T>::kVec;
  const float a = *scalar;
  if (a == 1.f) return;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    T* xr = x + static_cast<long long>(r) * ld;
    const RowSplit<T> sp(xr, nullptr, cols);
    for (int c = threadIdx.x; c < sp.head; c += blockDim.x) VecIO<T>::put(xr + c, VecIO<T>::get(xr + c) * a);
    for (int c = sp.tail + threadIdx.x; c < cols; c += blockDim.x) VecIO<T>::put(xr + c, VecIO<T>::get(xr + c) * a);
    for (int i = threadIdx.x; i < sp.nvec; i += blockDim.x) {
      float v[VEC];
      VecIO<T>::load(xr + sp.head + i * VEC, v);
#pragma unroll
      for (int j = 0; j < VEC; ++j) v[j] *= a;
      VecIO<T>::store(xr + sp.head + i * VEC, v);
    }
  }
}

}  // namespace fb

// count_inv: 2 floats, row_loss: `rows` floats, loss: 1 float (all device memory, caller-owned).
extern "C" int fb_softmax_ce_dyn(const void* logits, long long ld, const long long* targets, int rows, int V,
                                 long long ignore_index, void* dlogits, long long ldd, float* count_inv,
                                 float* row_loss, float* loss, int is_bf16, const int* counts, void* stream) {
  if (rows <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  fb::launch_pdl(fb::ce_count_kernel, dim3(1), dim3(1024), 0, st, targets, rows, ignore_index, count_inv);
  // By the row's bytes and by how many rows there are to an SM; the lines lie where the measured curves cross. Up to 1 KB, or 2 KB of many rows, a
  // warp. Few rows are a latency: 256 threads each. Otherwise as few threads as fill the loads: 128 up to 32 KB in bf16, 20 KB in fp32; beyond, rows
  // have to find themselves in L2 again, so 256 threads of more values each in bf16, 512 from 96 KB on; in fp32 256 up to 32 KB,
  // 512 up to 96 KB and then 1024.
  const long long bytes = static_cast<long long>(V) * (is_bf16 ? 2 : 4);
  const int per_sm = rows / fb::sm_count();
  auto go = [&](auto kern, int threads, int rows_per_block, auto* x, auto* dx) {
    fb::launch_pdl(kern, dim3((rows + rows_per_block - 1) / rows_per_block), dim3(threads), 0, st, x, ld, targets, rows, V, ignore_index, dx, ldd, count_inv, row_loss, counts);
  };
  auto pick = [&](auto* x, auto* dx) {
    using T = std::remove_pointer_t<decltype(dx)>;
    constexpr int one = sizeof(T) == 2 ? 1 : 2;      // vectors that make eight values
    if (bytes <= 1024 || (bytes <= 2048 && per_sm >= 16)) return go(fb::ce_fwd_kernel<T, true, 128, 16, one>, 128, 4, x, dx);
    if constexpr (sizeof(T) == 2) {
      if (per_sm < 4) go(fb::ce_fwd_kernel<T, false, 256, 4, 2 * one>, 256, 1, x, dx);
      else if (bytes <= 32768) go(fb::ce_fwd_kernel<T, false, 128, 12, 2 * one>, 128, 1, x, dx);
      else if (bytes <= 98304) go(fb::ce_fwd_kernel<T, false, 256, 6, 2 * one>, 256, 1, x, dx);
      else go(fb::ce_fwd_kernel<T, false, 512, 3, 2 * one>, 512, 1, x, dx);
    } else {
      if (bytes <= 20480 && per_sm >= 4) go(fb::ce_fwd_kernel<T, false, 128, 16, one>, 128, 1, x, dx);
      else if (bytes <= 32768) go(fb::ce_fwd_kernel<T, false, 256, 8, one>, 256, 1, x, dx);
      else if (bytes <= 98304) go(fb::ce_fwd_kernel<T, false, 512, 4, one>, 512, 1, x, dx);
      else go(fb::ce_fwd_kernel<T, false, 1024, 2, one>, 1024, 1, x, dx);
    }
  };
  if (is_bf16) pick(static_cast<const __nv_bfloat16*>(logits), static_cast<__nv_bfloat16*>(dlogits));
  else pick(static_cast<const float*>(logits), static_cast<float*>(dlogits));
  if (loss) fb::launch_pdl(fb::ce_finalize_kernel, dim3(1), dim3(1024), 0, st, row_loss, rows, count_inv, loss);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int fb_softmax_ce(const void* logits, long long ld, const long long* targets, int rows, int V,
                             long long ignore_index, void* dlogits, long long ldd, float* count_inv,
                             float* row_loss, float* loss, int is_bf16, void* stream) {
  return fb_softmax_ce_dyn(logits, ld, targets, rows, V, ignore_index, dlogits, ldd, count_inv, row_loss, loss, is_bf16, nullptr, stream);
}

extern "C" int fb_scale_rows(void* x, long long ld, int rows, int cols, const float* scalar, int is_bf16, void* stream) {
  if (rows <= 0 || cols <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = rows < 148 * 8 ? rows : 148 * 8;
  if (is_bf16)
    fb::launch_pdl(fb::scale_rows_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, st, static_cast<__nv_bfloat16*>(x), ld, rows, cols, scalar);
  else
    fb::launch_pdl(fb::scale_rows_kernel<float>, dim3(grid), dim3(256), 0, st, static_cast<float*>(x), ld, rows, cols, scalar);
  return static_cast<int>(cudaGetLastError());
}

FB_BOUNDS_ATTACH(softmax_ce)

// Fused LayerNorm forward / backward, one warp per row, the row held in registers.
//
// Replaces `at::native_layer_norm` (flodl-sys/ops_tensor.cpp:442-460) and, for the encoder
// blocks, the separate dropout + residual add that precede it
// (flodl-hf/src/models/transformer_layer.rs:224-263):
//     pre = residual + dropout(x)        (both optional)
//     y   = (pre - mean) * rstd * gamma + beta
// The dropout mask is a pure function of (seed, element index), so the backward pass
// regenerates it and nothing but `pre`, mean and rstd is saved.
//
// Backward produces d(pre) (which is also the residual-branch gradient), optionally
// d(x) = d(pre) * mask, and dgamma / dbeta.
#include "../include/flodl_b200.h"
#include "common.cuh"

namespace fb {

constexpr int kLnWarps = 4;

// N consecutive fp32 values p[off .. off+N) as 16-byte loads (N is 4 or 8, off a multiple of N, the
// array 16-byte aligned as every parameter slot is); `fill` when p is null.
template <int N>
__device__ __forceinline__ void load_f32_vec(const float* __restrict__ p, int off, float fill, float (&out)[N]) {
  if (!p) {
#pragma unroll
    for (int j = 0; j < N; ++j) out[j] = fill;
    return;
  }
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
#pragma unroll
    for (int j = 0; j < N; j += 4) {
      const float4 q = __ldg(reinterpret_cast<const float4*>(p + off + j));
      out[j] = q.x; out[j + 1] = q.y; out[j + 2] = q.z; out[j + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < N; ++j) out[j] = __ldg(p + off + j);
  }
}

// N consecutive parameters as they are in memory, fp32 or bf16 (a model cast to bf16 for inference): loaded, and converted where they are used, so that
// a warp has all its loads in flight. A parameter off the alignment of a vector is read value by value; a missing one is `fill`.
template <typename P, int N>
struct Param;
template <int N>
struct Param<float, N> {
  float v[N];
  __device__ __forceinline__ void load(const float* __restrict__ p, int off, float fill) { load_f32_vec<N>(p, off, fill, v); }
  __device__ __forceinline__ float get(int j) const { return v[j]; }
};
template <int N>
struct Param<__nv_bfloat16, N> {
  static_assert(N == 4 || N == 8, "");
  uint32_t h[N / 2];
  __device__ __forceinline__ void load(const __nv_bfloat16* __restrict__ p, int off, float fill) {
    if (!p) {
#pragma unroll
      for (int j = 0; j < N / 2; ++j) h[j] = __float_as_uint(fill) >> 16 | (__float_as_uint(fill) & 0xffff0000u);
    } else if ((reinterpret_cast<uintptr_t>(p) & (2 * N - 1)) == 0) {
      if constexpr (N == 8) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(p + off));
        h[0] = q.x; h[1] = q.y; h[2] = q.z; h[3] = q.w;
      } else {
        const uint2 q = __ldg(reinterpret_cast<const uint2*>(p + off));
        h[0] = q.x; h[1] = q.y;
      }
    } else {
      const uint16_t* u = reinterpret_cast<const uint16_t*>(p + off);
#pragma unroll
      for (int j = 0; j < N / 2; ++j) h[j] = static_cast<uint32_t>(__ldg(u + 2 * j)) | static_cast<uint32_t>(__ldg(u + 2 * j + 1)) << 16;
    }
  }
  __device__ __forceinline__ float get(int j) const { return __uint_as_float(j & 1 ? h[j / 2] & 0xffff0000u : h[j / 2] << 16); }
};

// Blocks per SM: of one row of `size`-byte values in the forward pass (one more for fp32 makes a whole wave of 4096 rows: 1024 wide 6.2 us, with six 9.0),
// and in the backward pass what `values` columns per lane and two rows in flight leave registers for.
constexpr int ln_fwd_blocks(int size) { return size == 4 ? 7 : 6; }
constexpr int ln_bwd_blocks(int values) { return values <= 16 ? 4 : values <= 24 ? 3 : 2; }

// A warp per row, all its loads issued before anything is done with them, six or seven blocks on an SM: a row's two warp-wide sums are a serial chain of
// shuffles, which other warps' loads cover. HBM bounds it (65536 x 768 bf16, residual, pre kept: 61 us, 6.5 TB/s), below some 16 MB L2.
// us, plain / with residual, in brackets a load where it is used, and one wave of warps that walk the rows with the next row's loads in flight:
// bf16 65536 x 768 49 / 61 (60 / 81, 50 / 65), 4096 x 768 5.0 / 5.6 (5.6 / 6.0, 6.2 / 6.5), 65536 x 256 20 / 25 (21 / 30, 31 / 36), 4096 x 1024 6.2 / 6.9
// (6.4 / 6.8, 7.8 / 8.4), fp32 4096 x 1024 6.2 / 8.7 (7.3 / 9.3, 10.9 / 11.2), 65536 x 1024 95 / 166 (110 / 165, 119 / 156).
// kFew, for as many rows as two blocks on each SM take: such a launch is one chain of latencies, so that gamma and beta are brought to L2 while the
// previous kernel still runs and loaded along with the row instead of after its sums, in registers that many rows need for more warps. bf16 768 wide,
// residual, pre kept: 77 rows 2.0 us (2.6), 1184 rows 2.6 (3.1), 2368 rows 4.2 against 3.7; an encoder of bf16 parameters, cold: 5.0 -> 3.0 a launch, of
// which half is the parameters' conversion, which had made each of six loads wait for the one before.
template <typename T, int VPL, typename P, bool kFew>
__global__ void __launch_bounds__(kLnWarps * 32, kFew ? 2 : ln_fwd_blocks(sizeof(T)))
ln_fwd_kernel(const T* __restrict__ x, const T* __restrict__ residual, const P* __restrict__ gamma,
              const P* __restrict__ beta, T* __restrict__ y, T* __restrict__ pre_out,
              float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int cols, float eps,
              float p_drop, uint64_t seed_in, const unsigned long long* __restrict__ seed_dev) {
  if constexpr (kFew) {
    const int at = threadIdx.x * (128 / static_cast<int>(sizeof(P)));
    if (at < cols) {
      if (gamma) asm volatile("prefetch.global.L2 [%0];" ::"l"(gamma + at));
      if (beta) asm volatile("prefetch.global.L2 [%0];" ::"l"(beta + at));
    }
  }
  pdl_entry();
  constexpr int V = VecIO<T>::kVec;
  const uint64_t seed = seed_in + (seed_dev ? *seed_dev : 0ull);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = cols / V;
  const float inv_keep = p_drop > 0.f ? 1.f / (1.f - p_drop) : 1.f;

  const int row = blockIdx.x * kLnWarps + warp;
  if (row >= rows) return;
  // all loads of the row before anything is done with them
  uint4 nx[VPL], nr[VPL];
  const uint4* xr = reinterpret_cast<const uint4*>(x + static_cast<long long>(row) * cols);
  const uint4* rr = reinterpret_cast<const uint4*>(residual + static_cast<long long>(row) * cols);
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int vi = lane + i * 32;
    if (vi < nvec) {
      nx[i] = xr[vi];
      if (residual) nr[i] = rr[vi];
    }
  }
  Param<P, V> g[VPL], b[VPL];
  if constexpr (kFew) {
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int vi = lane + i * 32;
      if (vi < nvec) {
        g[i].load(gamma, vi * V, 1.f);
        b[i].load(beta, vi * V, 0.f);
      }
    }
  }
  float v[VPL][V];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int vi = lane + i * 32;
    if (vi < nvec) {
      VecIO<T>::unpack(nx[i], v[i]);
      if (p_drop > 0.f) {
        const uint64_t base = static_cast<uint64_t>(row) * cols + static_cast<uint64_t>(vi) * V;
#pragma unroll
        for (int j = 0; j < V; j += 4) {
          float s[4];
          dropout_scale4(seed, base + j, p_drop, inv_keep, s);
#pragma unroll
          for (int k = 0; k < 4; ++k) v[i][j + k] *= s[k];
        }
      }
      if (residual) {
        float r[V];
        VecIO<T>::unpack(nr[i], r);
#pragma unroll
        for (int j = 0; j < V; ++j) v[i][j] += r[j];
      }
      if (pre_out) {
        // keep what the backward pass will see: the value rounded to the storage type
        VecIO<T>::store(pre_out + static_cast<long long>(row) * cols + vi * V, v[i]);
      }
#pragma unroll
      for (int j = 0; j < V; ++j) sum += v[i][j];
    } else {
#pragma unroll
      for (int j = 0; j < V; ++j) v[i][j] = 0.f;
    }
  }
  const float mean = warp_sum(sum) / cols;
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    if (lane + i * 32 < nvec) {
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const float d = v[i][j] - mean;
        sq += d * d;
      }
    }
  }
  const float rstd = rsqrtf(warp_sum(sq) / cols + eps);
  if (lane == 0) {
    if (mean_out) mean_out[row] = mean;
    if (rstd_out) rstd_out[row] = rstd;
  }
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int vi = lane + i * 32;
    if (vi < nvec) {
      float o[V];
      if constexpr (!kFew) {
        g[i].load(gamma, vi * V, 1.f);
        b[i].load(beta, vi * V, 0.f);
      }
#pragma unroll
      for (int j = 0; j < V; ++j) o[j] = fmaf((v[i][j] - mean) * rstd, g[i].get(j), b[i].get(j));
      VecIO<T>::store(y + static_cast<long long>(row) * cols + vi * V, o);
    }
  }
}

// One resident wave of blocks walks the rows, because each keeps sums for the parameter gradients, and each warp has the next row's 16-byte loads
// in flight while it reduces and writes this one. HBM bounds it. bf16, parameter gradients accumulated, against a block per four rows: 65536 x 768
// 54 us (5.5 TB/s) against 104, 65536 x 1024, where two blocks fit an SM, 133 against 245; fp32 32768 x 768 60 against 97.
template <typename T, int VPL>
__global__ void __launch_bounds__(kLnWarps * 32, ln_bwd_blocks(VPL * VecIO<T>::kVec))
ln_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ pre, const float* __restrict__ mean,
              const float* __restrict__ rstd, const float* __restrict__ gamma, T* __restrict__ dpre,
              T* __restrict__ dx_drop, float* __restrict__ partial, float* __restrict__ dgamma, float* __restrict__ dbeta,
              int rows, int cols, float p_drop, uint64_t seed_in, const unsigned long long* __restrict__ seed_dev) {
  pdl_entry();
  constexpr int V = VecIO<T>::kVec;
  const uint64_t seed = seed_in + (seed_dev ? *seed_dev : 0ull);
  __shared__ __align__(16) float red[kLnWarps][32 * VPL * V + 4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = cols / V;
  const float inv_keep = p_drop > 0.f ? 1.f / (1.f - p_drop) : 1.f;
  float dg[VPL][V], db[VPL][V];
#pragma unroll
  for (int i = 0; i < VPL; ++i)
#pragma unroll
    for (int j = 0; j < V; ++j) dg[i][j] = db[i][j] = 0.f;

  // gamma does not change from row to row: in registers where they allow it
  constexpr bool kKeep = VPL * V <= 24;
  float gm[kKeep ? VPL : 1][V];
  if constexpr (kKeep) {
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (lane + i * 32 < nvec) {
        load_f32_vec<V>(gamma, (lane + i * 32) * V, 1.f, gm[i]);
      } else {
#pragma unroll
        for (int j = 0; j < V; ++j) gm[i][j] = 1.f;
      }
    }
  }
  auto gain = [&](int i, float (&g)[V]) {
    if constexpr (kKeep) {
#pragma unroll
      for (int j = 0; j < V; ++j) g[j] = gm[i][j];
    } else {
      load_f32_vec<V>(gamma, (lane + i * 32) * V, 1.f, g);
    }
  };
  // dy and pre stay packed: xhat is computed twice from them, which costs less than the registers of a second row in fp32
  uint4 na[VPL], nb[VPL];
  float nmu = 0.f, nrs = 0.f;
  auto fetch = [&](int row) {
    const uint4* ar = reinterpret_cast<const uint4*>(dy + static_cast<long long>(row) * cols);
    const uint4* br = reinterpret_cast<const uint4*>(pre + static_cast<long long>(row) * cols);
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int vi = lane + i * 32;
      if (vi < nvec) { na[i] = ar[vi]; nb[i] = br[vi]; }
    }
    nmu = mean[row];
    nrs = rstd[row];
  };
  int row = blockIdx.x * kLnWarps + warp;
  if (row < rows) fetch(row);
  for (; row < rows; row += gridDim.x * kLnWarps) {
    uint4 ca[VPL], cb[VPL];
    const float mu = nmu, rs = nrs;
#pragma unroll
    for (int i = 0; i < VPL; ++i) { ca[i] = na[i]; cb[i] = nb[i]; }
    if (row + gridDim.x * kLnWarps < rows) fetch(row + gridDim.x * kLnWarps);
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (lane + i * 32 < nvec) {
        float a[V], b[V], g[V];
        VecIO<T>::unpack(ca[i], a);
        VecIO<T>::unpack(cb[i], b);
        gain(i, g);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          const float xh = (b[j] - mu) * rs;
          dg[i][j] += a[j] * xh;
          db[i][j] += a[j];
          s1 += a[j] * g[j];
          s2 += a[j] * g[j] * xh;
        }
      }
    }
    s1 = warp_sum(s1) / cols;
    s2 = warp_sum(s2) / cols;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int vi = lane + i * 32;
      if (vi < nvec) {
        float a[V], b[V], g[V], o[V];
        VecIO<T>::unpack(ca[i], a);
        VecIO<T>::unpack(cb[i], b);
        gain(i, g);
#pragma unroll
        for (int j = 0; j < V; ++j) o[j] = rs * (a[j] * g[j] - s1 - (b[j] - mu) * rs * s2);
        VecIO<T>::store(dpre + static_cast<long long>(row) * cols + vi * V, o);
        if (dx_drop) {
          const uint64_t base = static_cast<uint64_t>(row) * cols + static_cast<uint64_t>(vi) * V;
#pragma unroll
          for (int j = 0; j < V; j += 4) {
            float s[4];
            dropout_scale4(seed, base + j, p_drop, inv_keep, s);
#pragma unroll
            for (int k = 0; k < 4; ++k) o[j + k] *= s[k];
          }
          VecIO<T>::store(dx_drop + static_cast<long long>(row) * cols + vi * V, o);
        }
      }
    }
  }
  if (!partial && !dgamma && !dbeta) return;
  // Fold the 4 warps of the block. The sums are added straight into the gradients where those accumulate (a 16-byte reduction
  // per four columns; it saves a launch, a write and a read of the partial rows); otherwise one partial row per block,
  // [dgamma | dbeta], is left to ln_bwd_finalize_kernel.
  for (int pass = 0; pass < 2; ++pass) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < VPL; ++i)
#pragma unroll
      for (int j = 0; j < V; j += 4)
        *reinterpret_cast<float4*>(&red[warp][(lane + i * 32) * V + j]) = pass == 0 ? make_float4(dg[i][j], dg[i][j + 1], dg[i][j + 2], dg[i][j + 3])
                                                                                     : make_float4(db[i][j], db[i][j + 1], db[i][j + 2], db[i][j + 3]);
    __syncthreads();
    float* out = partial ? partial + (static_cast<long long>(blockIdx.x) * 2 + pass) * cols : (pass == 0 ? dgamma : dbeta);
    if (!out) continue;
    const bool whole = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    for (int c = threadIdx.x * 4; c < cols; c += blockDim.x * 4) {       // cols is a multiple of 4
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < kLnWarps; ++w) {
        const float4 q = *reinterpret_cast<const float4*>(&red[w][c]);
        s.x += q.x; s.y += q.y; s.z += q.z; s.w += q.w;
      }
      if (partial) {
        if (whole) *reinterpret_cast<float4*>(out + c) = s;
        else { out[c] = s.x; out[c + 1] = s.y; out[c + 2] = s.z; out[c + 3] = s.w; }
      } else {
        if (whole) red_add_v4(out + c, s.x, s.y, s.z, s.w);
        else { atomicAdd(out + c, s.x); atomicAdd(out + c + 1, s.y); atomicAdd(out + c + 2, s.z); atomicAdd(out + c + 3, s.w); }
      }
    }
  }
}

// dgamma / dbeta = the column sums of the partial rows: 32 columns x 32 row groups per block, four rows in flight per thread.
__global__ void __launch_bounds__(1024)
ln_bwd_finalize_kernel(const float* __restrict__ partial, float* __restrict__ dgamma, float* __restrict__ dbeta, int nblocks, int cols) {
  pdl_entry();
  __shared__ float rg[32][33], rb[32][33];
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float g = 0.f, b = 0.f;
  if (c < cols) {
    int i = grp;
    for (; i + 96 < nblocks; i += 128) {
      float gg[4], bb[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        gg[u] = partial[(static_cast<long long>(i + 32 * u) * 2) * cols + c];
        bb[u] = partial[(static_cast<long long>(i + 32 * u) * 2 + 1) * cols + c];
      }
      g += (gg[0] + gg[1]) + (gg[2] + gg[3]);
      b += (bb[0] + bb[1]) + (bb[2] + bb[3]);
    }
    for (; i < nblocks; i += 32) {
      g += partial[(static_cast<long long>(i) * 2) * cols + c];
      b += partial[(static_cast<long long>(i) * 2 + 1) * cols + c];
    }
  }
  rg[grp][lane] = g;
  rb[grp][lane] = b;
  __syncthreads();
  // warp w folds column w of both arrays (32 warps, 32 columns)
  g = warp_sum(rg[lane][grp]);
  b = warp_sum(rb[lane][grp]);
  const int col = blockIdx.x * 32 + grp;
  if (lane == 0 && col < cols) {
    if (dgamma) dgamma[col] = g;
    if (dbeta) dbeta[col] = b;
  }
}

template <typename T, int VPL, typename P>
static int ln_fwd_launch(const void* x, const void* res, const P* gamma, const P* beta, void* y,
                         void* pre, float* mean, float* rstd, int rows, int cols, float eps, float p,
                         uint64_t seed, const unsigned long long* seed_dev, cudaStream_t st) {
  const int blocks = (rows + kLnWarps - 1) / kLnWarps;
  auto go = [&](auto kern) {
    launch_pdl(kern, dim3(blocks), dim3(kLnWarps * 32), 0, st, static_cast<const T*>(x), static_cast<const T*>(res), gamma, beta, static_cast<T*>(y),
               static_cast<T*>(pre), mean, rstd, rows, cols, eps, p, seed, seed_dev);
  };
  if (blocks <= 2 * sm_count()) go(ln_fwd_kernel<T, VPL, P, true>);
  else go(ln_fwd_kernel<T, VPL, P, false>);
  return static_cast<int>(cudaGetLastError());
}

// `most` is the number of partial rows the caller's buffer holds.
template <typename T, int VPL>
static int ln_bwd_launch(const void* dy, const void* pre, const float* mean, const float* rstd,
                         const float* gamma, void* dpre, void* dxd, float* partial, float* dgamma, float* dbeta, int accumulate, int most,
                         int rows, int cols, float p, uint64_t seed, const unsigned long long* seed_dev, cudaStream_t st) {
  // A block ends with a reduction into, or a partial row for, every parameter: few short rows are given to fewer blocks, up to four to a warp, the more
  // the fewer bytes a row has (and the fewer with dropout, whose random numbers take as long), though to two blocks on each SM.
  // us, gradients accumulated, bf16, against a full wave: 2048 x 256 4.2 (5.8), 4096 x 256 4.9 (7.1), 2048 x 512 4.6 (6.4), 4096 x 768 7.5 (7.8).
  const int sms = sm_count(), wave = sms * ln_bwd_blocks(VPL * VecIO<T>::kVec), need = (rows + kLnWarps - 1) / kLnWarps;
  const int cheap = (p > 0.f ? 48 : 150) / static_cast<int>(VPL * VecIO<T>::kVec * sizeof(T)), each = cheap < 1 ? 1 : cheap > 4 ? 4 : cheap;
  int grid = (need + each - 1) / each;
  if (grid < 2 * sms) grid = 2 * sms;
  if (grid > wave) grid = wave;
  if (grid > most) grid = most;
  const bool fold = partial && !accumulate && (dgamma || dbeta);      // through the partial rows
  const bool add = partial && accumulate;
  launch_pdl(ln_bwd_kernel<T, VPL>, dim3(grid), dim3(kLnWarps * 32), 0, st, static_cast<const T*>(dy), static_cast<const T*>(pre), mean, rstd, gamma, static_cast<T*>(dpre),
      static_cast<T*>(dxd), fold ? partial : nullptr, add ? dgamma : nullptr, add ? dbeta : nullptr, rows, cols, p, seed, seed_dev);
  if (fold) launch_pdl(ln_bwd_finalize_kernel, dim3((cols + 31) / 32), dim3(1024), 0, st, partial, dgamma, dbeta, grid, cols);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace fb

// FN<T, VPL> or FN<T, VPL, P> for the row's type and length; PARAM is FB_LN_PARAM(P) or empty.
#define FB_LN_DISPATCH(FN, PARAM, ...)                                              \
  do {                                                                              \
    const int vec = is_bf16 ? 8 : 4;                                                \
    const int vpl = (cols / vec + 31) / 32;                                         \
    if (is_bf16) {                                                                  \
      switch (vpl) {                                                                \
        case 1: return fb::FN<__nv_bfloat16, 1 PARAM>(__VA_ARGS__);                 \
        case 2: return fb::FN<__nv_bfloat16, 2 PARAM>(__VA_ARGS__);                 \
        case 3: return fb::FN<__nv_bfloat16, 3 PARAM>(__VA_ARGS__);                 \
        case 4: return fb::FN<__nv_bfloat16, 4 PARAM>(__VA_ARGS__);                 \
        default: return -4;                                                         \
      }                                                                             \
    } else {                                                                        \
      switch (vpl) {                                                                \
        case 1: return fb::FN<float, 1 PARAM>(__VA_ARGS__);                         \
        case 2: return fb::FN<float, 2 PARAM>(__VA_ARGS__);                         \
        case 3: return fb::FN<float, 3 PARAM>(__VA_ARGS__);                         \
        case 4: return fb::FN<float, 4 PARAM>(__VA_ARGS__);                         \
        case 5: case 6: return fb::FN<float, 6 PARAM>(__VA_ARGS__);                 \
        case 7: case 8: return fb::FN<float, 8 PARAM>(__VA_ARGS__);                 \
        default: return -4;                                                         \
      }                                                                             \
    }                                                                               \
  } while (0)
#define FB_LN_PARAM(P) , P

extern "C" int fb_layernorm_max_cols(int is_bf16) { return 1024; }

namespace {
template <typename P>
int layernorm_fwd(const void* x, const void* residual, const P* gamma, const P* beta, void* y, void* pre_out, float* mean, float* rstd, int rows, int cols,
                  float eps, float p_drop, unsigned long long seed, const unsigned long long* seed_dev, int is_bf16, void* stream) {
  if (rows <= 0) return 0;
  if (cols % (is_bf16 ? 8 : 4) || cols > 1024) return -4;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  FB_LN_DISPATCH(ln_fwd_launch, FB_LN_PARAM(P), x, residual, gamma, beta, y, pre_out, mean, rstd, rows, cols, eps, p_drop, seed, seed_dev, st);
}
}  // namespace

extern "C" int fb_layernorm_fwd(const void* x, const void* residual, const float* gamma, const float* beta,
                                void* y, void* pre_out, float* mean, float* rstd, int rows, int cols,
                                float eps, float p_drop, unsigned long long seed, const unsigned long long* seed_dev, int is_bf16, void* stream) {
  return layernorm_fwd(x, residual, gamma, beta, y, pre_out, mean, rstd, rows, cols, eps, p_drop, seed, seed_dev, is_bf16, stream);
}

extern "C" int fb_layernorm_fwd_p16(const void* x, const void* residual, const void* gamma, const void* beta,
                                    void* y, void* pre_out, float* mean, float* rstd, int rows, int cols,
                                    float eps, float p_drop, unsigned long long seed, const unsigned long long* seed_dev, int is_bf16, void* stream) {
  return layernorm_fwd(x, residual, static_cast<const __nv_bfloat16*>(gamma), static_cast<const __nv_bfloat16*>(beta), y, pre_out, mean, rstd, rows, cols, eps,
                       p_drop, seed, seed_dev, is_bf16, stream);
}

// The most blocks the backward kernel uses: one resident wave (its dgamma / dbeta sums stay in registers).
extern "C" int fb_layernorm_bwd_grid(int rows) {
  const int cap = 4 * fb::sm_count(), g = (rows + fb::kLnWarps - 1) / fb::kLnWarps;
  return g < cap ? g : cap;
}

// `partial` must hold fb_layernorm_bwd_grid(rows) * 2 * cols floats.
extern "C" int fb_layernorm_bwd(const void* dy, const void* pre, const float* mean, const float* rstd,
                                const float* gamma, void* dpre, void* dx_drop, float* partial, float* dgamma,
                                float* dbeta, int accumulate, int rows, int cols, float p_drop,
                                unsigned long long seed, const unsigned long long* seed_dev, int is_bf16, void* stream) {
  if (rows <= 0) return 0;
  if (cols % (is_bf16 ? 8 : 4) || cols > 1024) return -4;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int most = fb_layernorm_bwd_grid(rows);
  FB_LN_DISPATCH(ln_bwd_launch, , dy, pre, mean, rstd, gamma, dpre, dx_drop, partial, dgamma, dbeta, accumulate, most, rows, cols, p_drop, seed, seed_dev, st);
}

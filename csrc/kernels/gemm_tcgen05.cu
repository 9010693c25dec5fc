// bf16 GEMM on the 5th-generation tensor cores: D[m,n] = sum_k A(m,k) * B(n,k), fp32 accumulate.
//
// Replaces the cuBLAS call behind `torch::linear` that the reference issues for every Linear
// layer (flodl-sys/ops_training.cpp:306-318) and for the dX / dW products libtorch's autograd
// derives from it.
//
// Shape of the kernel
//   * persistent: one CTA (or one CTA pair) per SM walks a list of output tiles;
//   * warp 0 feeds a multi-stage shared-memory ring with TMA (`cp.async.bulk.tensor`, 128-byte
//     swizzle), warp 1 issues `tcgen05.mma` (both run their loops whole, one elected lane issues), warps 2..9
//     drain the accumulator from TMEM with `tcgen05.ld` and run the epilogue;
//   * two accumulator buffers in TMEM, so the epilogue of tile i overlaps the main loop of
//     tile i+1;
//   * `kCG == 2` pairs two CTAs of a cluster on one 256-row tile (`cta_group::2`): each CTA loads
//     its own half of A and B with plain (non-multicast) TMA loads that credit the leader's
//     mbarrier, the leader issues the MMAs, commits are multicast to both CTAs.
//   * operands may be K-major (row = M/N index) or MN-major (row = K index); the second form is
//     what dX = dY * W and dW = dY^T * X need, so no transposes are materialised.
//   * epilogue: optional alpha (device scalar), bias, GELU (erf or tanh; pre-activation saved to
//     `aux`), GELU' (multiply by gelu'(aux)), accumulate into C, split-K added to memory in fp32;
//   * the gradients of a linear layer as one launch: dX's tiles, then dW's reduction cut where the tiles of dX leave time, and
//     two more warps for the bias gradient (`fb_gemm_backward`).
//
// All waits are bounded (see ptx_sm100.cuh); a give-up is reported through `status`.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstring>
#include <type_traits>
#include <mutex>
#include <unordered_map>

#include "../include/flodl_b200.h"
#include "common.cuh"
#include "ptx_sm100.cuh"

// The per-CTA timeline (`ts`) is a tuning aid: it is compiled in only with -DFB_TIMELINE=1
// (FLODL_B200_TIMELINE=1 at build time); a regular build ignores the argument.
#ifndef FB_TIMELINE
#define FB_TIMELINE 0
#endif
#if FB_TIMELINE
#define FB_TIMELINE_ONLY(stmt) stmt
#else
#define FB_TIMELINE_ONLY(stmt)
#endif

namespace fb {

// gemm_small.cu
int gemm_small_split(int M, int N, int K, bool several = false);
bool gemm_small_aligned(int N, const void* C, long long ldc, const void* aux, long long ldaux);
int gemm_small(const void* A, const void* const* B, void* C, int M, int group, int groups, int K, long long lda, long long ldb, long long ldc, int b_mn,
               const void* const* bias, int bias_fp32, int epi, void* aux, long long ldaux, const float* alpha, int split, int* status, cudaStream_t stream);

constexpr int BM = 128;  // rows of the tile held by ONE CTA
constexpr int BK = 64;   // K per stage = one 128-byte swizzle row of bf16
constexpr int kEpiWarps = 8;
constexpr int kGemmThreads = 32 * (2 + kEpiWarps);

struct GemmParams {
  int M, N, K;
  int a_mn, b_mn;
  void* C;
  long long ldc;
  int c_fp32;
  const void* bias;
  int bias_fp32;
  int epi;
  void* aux;
  long long ldaux;
  const float* alpha;
  int accumulate;
  int split_k;
  int c_mode;      // 0 = per-thread global stores, 1 = staged TMA store, 2 = staged TMA reduce-add (fp32)
  int part_groups; // of kernels with kParts: the device cuts K for as many pairs (parts_for); C is [parts][rows of whole tiles][N] fp32, written and not
                   // added to, or with one part [M][N] bf16 through the map `aux`
  int kind;        // EpiKind: what the epilogue does
  int band;        // column tiles per band of the tile order (tile_of)
  int aux_tma;     // 1: the GELU pre-activation goes out through its own staged TMA store; 2: GELU' takes it in through TMA loads
  int* status;
  long long* ts;   // optional per-CTA timeline (8 slots each), for tuning
  // Optional device-side problem sizes (produced by an earlier kernel of the stream): the kernel
  // works on min(M, *m_dyn) rows / min(K, *k_dyn) of the reduction. Buffers and tensor maps keep
  // their full static size, so a captured graph can replay with a different count every step.
  const int* m_dyn;
  const int* k_dyn;
};

template <int kCG, int kBN>
struct GemmCfg {
  static constexpr int BN_CTA = kBN / kCG;
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN_CTA * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (160 * 1024) / STAGE_BYTES;
  // two accumulators side by side; the allocation size must be a power of two
  static constexpr int TMEM_COLS = (2 * kBN <= 32) ? 32 : (2 * kBN <= 64) ? 64 : (2 * kBN <= 128) ? 128 : (2 * kBN <= 256) ? 256 : 512;
  // the 8 epilogue warps are 4 TMEM lane quarters x 2 column ranges; ranges are multiples of 64
  // columns (one staged bf16 store), so a 192-wide tile splits 128 + 64
  static constexpr int EPI_SPLIT = (kBN == 192) ? 128 : kBN / 2;
  // epilogue staging: 4 KB (32 rows x 128 B, swizzled) per epilogue warp for C, the same again for aux
  static constexpr int EPI_BYTES = 2 * kEpiWarps * 4096;
  static constexpr int BAR_BYTES = 512, BIAS_BYTES = 2 * 256 * 4;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_BYTES + BAR_BYTES + BIAS_BYTES;
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
  static_assert((2 * STAGES + 5 + 2 * kEpiWarps) * 8 + 8 <= BAR_BYTES, "barrier block");
  static_assert(TMEM_COLS <= 512, "accumulators do not fit TMEM");
};

// The epilogue runs on 8 warps while the tensor cores work on the next tile, so its budget per
// output element is about a dozen FP32 instructions and one special-function op (for K = 768 the
// main loop of a 128x256 tile is ~3000 cycles). libdevice's erff/tanhf cost 3-4x that, which made
// the GELU epilogue, not the MMA, the critical path. These bf16-output versions use the hardware
// tanh (see common.cuh): erf through a fitted odd polynomial inside tanh, |error| < 6e-5 in GELU.
__device__ __forceinline__ float gelu_erf_f(float x) { return gelu_erf_fast(x); }
__device__ __forceinline__ float dgelu_erf_f(float x) { return dgelu_erf_fast(x); }
__device__ __forceinline__ float gelu_tanh_f(float x) { return gelu_tanh_fast(x); }
__device__ __forceinline__ float dgelu_tanh_f(float x) { return dgelu_tanh_fast(x); }

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void unpack_bf16x2(uint32_t w, float& lo, float& hi) {
  const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
  lo = f.x;
  hi = f.y;
}

// v[0..32) += bias[col0 .. col0+32). Every lane of a warp reads the same addresses (one output row
// per lane, the same 32 columns), so wide loads are broadcasts: 8 (fp32) or 4 (bf16) load
// instructions per 32 columns instead of 32.
__device__ __forceinline__ void add_bias32(const GemmParams& p, int col0, int nvalid, float (&v)[32]) {
  if (p.bias_fp32) {
    const float* b = static_cast<const float*>(p.bias) + col0;
    if (nvalid == 32 && (reinterpret_cast<uintptr_t>(b) & 15) == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(b) + j);
        v[4 * j] += q.x; v[4 * j + 1] += q.y; v[4 * j + 2] += q.z; v[4 * j + 3] += q.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (i < nvalid) v[i] += __ldg(b + i);
    }
  } else {
    const __nv_bfloat16* b = static_cast<const __nv_bfloat16*>(p.bias) + col0;
    if (nvalid == 32 && (reinterpret_cast<uintptr_t>(b) & 15) == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(b) + j);
        float h[8];
        unpack_bf16x2(q.x, h[0], h[1]); unpack_bf16x2(q.y, h[2], h[3]);
        unpack_bf16x2(q.z, h[4], h[5]); unpack_bf16x2(q.w, h[6], h[7]);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[8 * j + i] += h[i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (i < nvalid) v[i] += __bfloat162float(b[i]);
    }
  }
}

// Epilogue for 32 consecutive columns of one output row. Every loop over the 32 values is fully
// unrolled with compile-time indices (tails are handled by predicates), so the values stay in
// registers: a dynamically indexed copy would be demoted to local memory and every access to it
// would become a memory transaction.
// Registers-only part: alpha, bias, activation. `v` receives the output values, `pre` the
// pre-activation (only meaningful for the GELU epilogues). Rows/cols outside the problem yield
// harmless values; the caller's store clips them.
__device__ __forceinline__ void epilogue_compute32(const GemmParams& p, const uint32_t (&acc)[32], int row, int col0,
                                                   bool add_bias, float (&v)[32], float (&pre)[32]) {
  if (p.alpha) {
    const float alpha = __ldg(p.alpha);
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(acc[i]) * alpha;
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(acc[i]);
  }
  const int nvalid = (col0 + 32 <= p.N) ? 32 : (p.N > col0 ? p.N - col0 : 0);
  if (p.bias && add_bias) add_bias32(p, col0, nvalid, v);
  if (p.epi == FB_EPI_GELU_ERF) {
#pragma unroll
    for (int i = 0; i < 32; ++i) { pre[i] = v[i]; v[i] = gelu_erf_f(v[i]); }
  } else if (p.epi == FB_EPI_GELU_TANH) {
#pragma unroll
    for (int i = 0; i < 32; ++i) { pre[i] = v[i]; v[i] = gelu_tanh_f(v[i]); }
  } else if ((p.epi == FB_EPI_DGELU_ERF || p.epi == FB_EPI_DGELU_TANH) && row < p.M) {
    const __nv_bfloat16* a =
        static_cast<const __nv_bfloat16*>(p.aux) + static_cast<long long>(row) * p.ldaux + col0;
    const bool vec = nvalid == 32 && ((reinterpret_cast<uintptr_t>(a) & 15) == 0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float h[8];
      if (vec) {
        const uint4 raw = *reinterpret_cast<const uint4*>(a + j * 8);
        unpack_bf16x2(raw.x, h[0], h[1]);
        unpack_bf16x2(raw.y, h[2], h[3]);
        unpack_bf16x2(raw.z, h[4], h[5]);
        unpack_bf16x2(raw.w, h[6], h[7]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) h[i] = (j * 8 + i < nvalid) ? __bfloat162float(a[j * 8 + i]) : 0.f;
      }
      if (p.epi == FB_EPI_DGELU_ERF) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[j * 8 + i] *= dgelu_erf_f(h[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[j * 8 + i] *= dgelu_tanh_f(h[i]);
      }
    }
  }
}

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// 16-byte piece `piece` (0..7) of row `row` (0..31) in a 32 x 128-byte tile with the 128-byte swizzle.
__device__ __forceinline__ uint32_t stage_addr(uint32_t base, int row, int piece) {
  return base + row * 128 + ((piece ^ (row & 7)) << 4);
}
__device__ __forceinline__ void tma_reduce_add_2d(const void* tmap, const void* smem_src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(tmap),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}

__device__ __forceinline__ uint32_t f2_pack_bf16(F2 a) {
  float lo, hi;
  f2_get(a, lo, hi);
  return pack_bf16x2(lo, hi);
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 q;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w) : "r"(addr) : "memory");
  return q;
}

// What a staged epilogue does. One of these per launch: testing the kernel's parameters for every 64 columns took 350 cycles of them.
enum EpiKind { kEpiDirect, kEpiPlain, kEpiGelu, kEpiGeluAux, kEpiDgelu, kEpiDgeluTanh, kEpiF32 };

// An epilogue warp's 32 rows: the two staging tiles, which take turns, and the stores issued so far.
struct EpiWarp {
  uint8_t* stage[2];
  uint64_t* aux_bar;       // pre-activations landed in stage[0], stage[1]
  uint32_t staged;
  int lane;
};

// This lane's row of a 32 x 64 bf16 staging tile.
__device__ __forceinline__ void stage_row64(uint32_t tile, int lane, const F2 (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
    st_shared_v4(stage_addr(tile, lane, j), f2_pack_bf16(v[4 * j]), f2_pack_bf16(v[4 * j + 1]), f2_pack_bf16(v[4 * j + 2]), f2_pack_bf16(v[4 * j + 3]));
}
// This lane's row of a staging tile that holds pre-activations: each 16-byte piece is replaced by v times the activation's derivative there.
template <bool kTanh>
__device__ __forceinline__ void dgelu_row64(uint32_t tile, int lane, const F2 (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t addr = stage_addr(tile, lane, j);
    const uint4 q = ld_shared_v4(addr);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float lo, hi;
      unpack_bf16x2(w[i], lo, hi);
      const F2 x = f2_make(lo, hi);
      o[i] = f2_pack_bf16(f2_mul(v[4 * j + i], kTanh ? f2_dgelu_tanh(x) : f2_dgelu_erf(x)));
    }
    st_shared_v4(addr, o[0], o[1], o[2], o[3]);
  }
}

// fp32 results: 32 columns (128 bytes of a row) per staged store or reduction.
template <typename HandBack>
__device__ __forceinline__ void epilogue_tile_f32(const GemmParams& p, const CUtensorMap& tmC, EpiWarp& w, uint32_t taddr, int col0, int row0, int cols, uint32_t bias,
                                                  const HandBack& hand_back) {
#pragma unroll 1
  for (int c = 0; c < cols; c += 32) {
    uint32_t acc[32];
    tmem_ld32_sync(taddr + c, acc);
    if (c + 32 >= cols) hand_back();
    if (p.alpha) {
      const float alpha = __ldg(p.alpha);
#pragma unroll
      for (int i = 0; i < 32; ++i) acc[i] = __float_as_uint(__uint_as_float(acc[i]) * alpha);
    }
    if (bias) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint4 q = ld_shared_v4(bias + c * 4 + j * 16);
        acc[4 * j] = __float_as_uint(__uint_as_float(acc[4 * j]) + __uint_as_float(q.x));
        acc[4 * j + 1] = __float_as_uint(__uint_as_float(acc[4 * j + 1]) + __uint_as_float(q.y));
        acc[4 * j + 2] = __float_as_uint(__uint_as_float(acc[4 * j + 2]) + __uint_as_float(q.z));
        acc[4 * j + 3] = __float_as_uint(__uint_as_float(acc[4 * j + 3]) + __uint_as_float(q.w));
      }
    }
    uint8_t* tile = w.stage[w.staged++ & 1];
    if (w.lane == 0) tma_store_wait_read_but_one();
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 8; ++j) st_shared_v4(stage_addr(smem_u32(tile), w.lane, j), acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
    fence_proxy_async_smem();
    __syncwarp();
    if (w.lane == 0) {
      if (p.c_mode == 2) tma_reduce_add_2d(&tmC, tile, col0 + c, row0);
      else tma_store_2d(&tmC, tile, col0 + c, row0);
      tma_store_commit();
    }
  }
}

// `chunks` times 64 columns from `col0` of rows [row0, row0 + 32), out of TMEM columns from `taddr` on. `bias`: shared memory, one fp32 per column
// (0: none). `hand_back` runs when the accumulator has been read, `next_aux` (lane 0) issues the next load of pre-activations. False: a wait gave up.
// Unrolled over 64 columns: rolled over 16 or 32, with the next ones on their way from TMEM, GELU at 4096 x 3072 x 768 took 25.5 us instead of 24.0.
template <int kKind, typename HandBack, typename NextAux>
__device__ __forceinline__ bool epilogue_tile(const GemmParams& p, const CUtensorMap& tmC, const CUtensorMap& tmAux, EpiWarp& w, uint32_t taddr, int col0, int row0,
                                              int chunks, uint32_t bias, volatile int* abort_flag, const HandBack& hand_back, const NextAux& next_aux) {
#pragma unroll 1
  for (int ch = 0; ch < chunks; ++ch) {
    const int col = col0 + ch * 64;
    F2 v[32];
    {
      uint32_t a[32], b[32];
      tmem_ld64_sync(taddr + ch * 64, a, b);
      if (ch == chunks - 1) hand_back();
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        v[i] = f2_make(__uint_as_float(a[2 * i]), __uint_as_float(a[2 * i + 1]));
        v[16 + i] = f2_make(__uint_as_float(b[2 * i]), __uint_as_float(b[2 * i + 1]));
      }
    }
    if (p.alpha) {
      const F2 alpha = f2_splat(__ldg(p.alpha));
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = f2_mul(v[i], alpha);
    }
    if (bias) {          // every lane reads the same 16 bytes: a load serves four columns of 32 rows
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const uint4 q = ld_shared_v4(bias + ch * 256 + j * 16);
        v[2 * j] = f2_add(v[2 * j], f2_make(__uint_as_float(q.x), __uint_as_float(q.y)));
        v[2 * j + 1] = f2_add(v[2 * j + 1], f2_make(__uint_as_float(q.z), __uint_as_float(q.w)));
      }
    }
    if constexpr (kKind == kEpiDgelu || kKind == kEpiDgeluTanh) {
      const uint32_t b = w.staged & 1;
      const bool ok = mbar_wait(&w.aux_bar[b], (w.staged >> 1) & 1, abort_flag, p.status, kStatusWaitFull);
      if (!__all_sync(0xffffffffu, ok)) return false;
      dgelu_row64<kKind == kEpiDgeluTanh>(smem_u32(w.stage[b]), w.lane, v);
      ++w.staged;
      fence_proxy_async_smem();
      __syncwarp();
      if (w.lane == 0) {
        tma_store_2d(&tmC, w.stage[b], col, row0);
        tma_store_commit();
        if (ch == chunks - 1) {         // the next tile's loads, each once its staging tile has been read
          if (chunks == 2) {
            tma_store_wait_read_but_one();
            next_aux();
          }
          tma_store_wait_read();
          next_aux();
        }
      }
    } else {
      const auto take_turn = [&]() -> uint8_t* {      // the staging tile whose store two turns ago has been read
        if (w.lane == 0) tma_store_wait_read_but_one();
        __syncwarp();
        return w.stage[w.staged++ & 1];
      };
      const auto send = [&](const CUtensorMap* map, const uint8_t* tile, int x) {
        fence_proxy_async_smem();
        __syncwarp();
        if (w.lane == 0) {
          tma_store_2d(map, tile, x, row0);
          tma_store_commit();
        }
      };
      if constexpr (kKind == kEpiGeluAux) {
        uint8_t* tile = take_turn();
        stage_row64(smem_u32(tile), w.lane, v);
        send(&tmAux, tile, col);
      }
      if constexpr (kKind == kEpiGelu || kKind == kEpiGeluAux) {
        if (p.epi == FB_EPI_GELU_ERF) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = f2_gelu_erf(v[i]);
        } else if (p.epi == FB_EPI_GELU_TANH) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = f2_gelu_tanh(v[i]);
        }
      }
      uint8_t* tile = take_turn();
      stage_row64(smem_u32(tile), w.lane, v);
      send(&tmC, tile, col);
    }
  }
  return true;
}

__device__ __forceinline__ void epilogue_store32(const GemmParams& p, const uint32_t (&acc)[32],
                                                 int row, int col0, bool add_bias) {
  if (row >= p.M || col0 >= p.N) return;
  float v[32];
  if (p.alpha) {
    const float alpha = __ldg(p.alpha);
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(acc[i]) * alpha;
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(acc[i]);
  }
  const bool full = (col0 + 32 <= p.N);
  const int nvalid = full ? 32 : (p.N - col0);
  if (p.bias && add_bias) add_bias32(p, col0, nvalid, v);
  if (p.epi == FB_EPI_GELU_ERF || p.epi == FB_EPI_GELU_TANH) {
    if (p.aux) {  // save the pre-activation for the backward pass
      __nv_bfloat16* a = static_cast<__nv_bfloat16*>(p.aux) + static_cast<long long>(row) * p.ldaux + col0;
      if (full && ((reinterpret_cast<uintptr_t>(a) & 15) == 0)) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 pk;
          pk.x = pack_bf16x2(v[j * 8 + 0], v[j * 8 + 1]);
          pk.y = pack_bf16x2(v[j * 8 + 2], v[j * 8 + 3]);
          pk.z = pack_bf16x2(v[j * 8 + 4], v[j * 8 + 5]);
          pk.w = pack_bf16x2(v[j * 8 + 6], v[j * 8 + 7]);
          *reinterpret_cast<uint4*>(a + j * 8) = pk;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (i < nvalid) a[i] = __float2bfloat16(v[i]);
      }
    }
    if (p.epi == FB_EPI_GELU_ERF) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = gelu_erf_f(v[i]);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = gelu_tanh_f(v[i]);
    }
  } else if (p.epi == FB_EPI_DGELU_ERF || p.epi == FB_EPI_DGELU_TANH) {
    const __nv_bfloat16* a =
        static_cast<const __nv_bfloat16*>(p.aux) + static_cast<long long>(row) * p.ldaux + col0;
    const bool vec = full && ((reinterpret_cast<uintptr_t>(a) & 15) == 0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float h[8];
      if (vec) {
        const uint4 raw = *reinterpret_cast<const uint4*>(a + j * 8);
        unpack_bf16x2(raw.x, h[0], h[1]);
        unpack_bf16x2(raw.y, h[2], h[3]);
        unpack_bf16x2(raw.z, h[4], h[5]);
        unpack_bf16x2(raw.w, h[6], h[7]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) h[i] = (j * 8 + i < nvalid) ? __bfloat162float(a[j * 8 + i]) : 0.f;
      }
      if (p.epi == FB_EPI_DGELU_ERF) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[j * 8 + i] *= dgelu_erf_f(h[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[j * 8 + i] *= dgelu_tanh_f(h[i]);
      }
    }
  }

  if (p.c_fp32) {
    float* c = static_cast<float*>(p.C) + static_cast<long long>(row) * p.ldc + col0;
    const bool vec = full && ((reinterpret_cast<uintptr_t>(c) & 15) == 0);
    if (p.split_k > 1 || p.accumulate) {       // added without being read
      if (vec) {
#pragma unroll
        for (int j = 0; j < 8; ++j) red_add_v4(c + 4 * j, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (i < nvalid) atomicAdd(c + i, v[i]);
      }
    } else if (vec) {
#pragma unroll
      for (int j = 0; j < 8; ++j) *reinterpret_cast<float4*>(c + 4 * j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (i < nvalid) c[i] = v[i];
    }
  } else {
    __nv_bfloat16* c = static_cast<__nv_bfloat16*>(p.C) + static_cast<long long>(row) * p.ldc + col0;
    if (full && ((reinterpret_cast<uintptr_t>(c) & 15) == 0)) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (p.accumulate) {
          const uint4 raw = *reinterpret_cast<const uint4*>(c + j * 8);
          float o[8];
          unpack_bf16x2(raw.x, o[0], o[1]);
          unpack_bf16x2(raw.y, o[2], o[3]);
          unpack_bf16x2(raw.z, o[4], o[5]);
          unpack_bf16x2(raw.w, o[6], o[7]);
#pragma unroll
          for (int i = 0; i < 8; ++i) v[j * 8 + i] += o[i];
        }
        uint4 pk;
        pk.x = pack_bf16x2(v[j * 8 + 0], v[j * 8 + 1]);
        pk.y = pack_bf16x2(v[j * 8 + 2], v[j * 8 + 3]);
        pk.z = pack_bf16x2(v[j * 8 + 4], v[j * 8 + 5]);
        pk.w = pack_bf16x2(v[j * 8 + 6], v[j * 8 + 7]);
        *reinterpret_cast<uint4*>(c + j * 8) = pk;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (i < nvalid) {
          float o = v[i];
          if (p.accumulate) o += __bfloat162float(c[i]);
          c[i] = __float2bfloat16(o);
        }
      }
    }
  }
}

// Tile t of the list: bands of `band` column tiles, in a band column tiles fastest.
__device__ __forceinline__ void tile_of(int t, int num_m, int num_n, int band, int& tm, int& tn) {
  int first = 0, width = num_n;
  if (band < num_n) {
    const int b = t / (band * num_m);
    first = b * band;
    t -= first * num_m;
    width = min(band, num_n - first);
  }
  tm = t / width;
  tn = first + t - tm * width;
}

// One product, or two in one launch: the data gradient of a linear layer and the weight gradient from the same dY, whose column sums (the bias
// gradient) two more warps of every CTA take on the side.
template <int kProblems>
struct alignas(64) GemmLaunch {
  CUtensorMap a[kProblems], b[kProblems], c[kProblems], aux;      // aux: the first product's
  GemmParams p[kProblems];
  // The second product's K blocks in one line, tile after tile: the pairs that have a tile of the first product more than the others (the first
  // `ahead` of them) take `share_ahead` of these each, the others `share`, in 1/256 of a block.
  int ahead, share_ahead, share;
  const __nv_bfloat16* sum_x;
  float* sum_out;
  int sum_rows, sum_cols;
  long long sum_ld;
};

// A reduction of `blocks` K blocks in at most `parts` equal ones: as many as hold a block. One without would add an accumulator that no product has
// written (17 blocks each for 500 in 31 parts: the last two would start behind the end).
__host__ __device__ constexpr int parts_with_blocks(int blocks, int parts) {
  if (blocks <= 0 || parts <= 1) return 1;
  const int per = (blocks + parts - 1) / parts;
  return (blocks + per - 1) / per;
}

// Parts to cut a reduction into for `groups` pairs that have `tiles` tiles: a part for every pair, none shorter than kPartBlocks, whose addition or
// storing would cost more than it spreads. The kernel that sums the parts asks again, with the same row count from the device.
constexpr int kPartBlocks = 16;
__host__ __device__ constexpr int parts_for(int tiles, int blocks, int groups) {
  if (tiles <= 0) return 1;
  const int spread = groups / tiles, most = blocks / kPartBlocks;
  return parts_with_blocks(blocks, spread < most ? spread : most);
}

// What a pair (or CTA) works on next: K blocks [kb0, kb1) of a tile.
struct Segment {
  int prob, tm, tn, kb0, kb1, ks;
};
template <int kCG, int kBN, int kProblems, bool kParts>
struct Worklist {
  const GemmLaunch<kProblems>& g;
  int step, num_m, num_n, num_kb, split, kb_per, units, u;      // the first product: whole tiles, or their K splits
  int num_m1, num_n1, num_kb1, at, end;                  // the second: a stretch of its K blocks

  __device__ __forceinline__ Worklist(const GemmLaunch<kProblems>& g_, int group, int groups, int m_eff, int k_eff) : g(g_), step(groups), u(group) {
    const GemmParams& p = g.p[0];
    num_m = (m_eff + BM * kCG - 1) / (BM * kCG);
    num_n = (p.N + kBN - 1) / kBN;
    num_kb = (k_eff + BK - 1) / BK;
    if (kParts) split = parts_for(num_m * num_n, num_kb, p.part_groups);
    kb_per = (num_kb + parts() - 1) / parts();
    units = num_kb > 0 ? num_m * num_n * parts() : 0;
    if constexpr (kProblems == 2) {
      const GemmParams& q = g.p[1];
      num_m1 = (q.M + BM * kCG - 1) / (BM * kCG);
      num_n1 = (q.N + kBN - 1) / kBN;
      num_kb1 = (q.K + BK - 1) / BK;
      const int total = num_m1 * num_n1 * num_kb1;
      // stretches begin at every fourth block: a part shorter than that costs more to add to memory than to compute
      const auto start = [&](int pair) {
        const int v = pair < g.ahead ? pair * g.share_ahead : g.ahead * g.share_ahead + (pair - g.ahead) * g.share;
        return min(total, v >> 8 & ~3);
      };
      at = start(group);
      end = group + 1 < groups ? start(group + 1) : total;
    }
  }
  // Each has a block: parts_for says so, or the host, which does not split a length that it does not know.
  __device__ __forceinline__ int parts() const { return kParts ? split : g.p[0].split_k; }
  __device__ __forceinline__ bool next(Segment& s) {
    if (u < units) {
      int t = u;
      s.ks = 0;
      if (kProblems == 1 && parts() > 1) {
        t = u / parts();
        s.ks = u - t * parts();
      }
      tile_of(t, num_m, num_n, g.p[0].band, s.tm, s.tn);
      s.prob = 0;
      s.kb0 = s.ks * kb_per;
      s.kb1 = min(num_kb, s.kb0 + kb_per);
      u += step;
      return true;
    }
    if (kProblems == 2 && at < end) {
      const int t = at / num_kb1;
      s.prob = 1;
      s.ks = 0;
      s.kb0 = at - t * num_kb1;
      s.kb1 = min(num_kb1, s.kb0 + end - at);
      at += s.kb1 - s.kb0;
      tile_of(t, num_m1, num_n1, g.p[1].band, s.tm, s.tn);
      return true;
    }
    return false;
  }
};

// Column sums of sum_x added to sum_out, by two warps of every CTA: 256 columns by a stretch of rows at a time, eight rows in flight.
template <int kProblems>
__device__ __forceinline__ void column_sums(const GemmLaunch<kProblems>& g, int warp, int lane) {
  const int col_groups = (g.sum_cols + 255) / 256, warps = 2 * static_cast<int>(gridDim.x);
  const int parts = max(1, min(warps / col_groups, g.sum_rows / 32)), per = (g.sum_rows + parts - 1) / parts;
  for (int item = 2 * blockIdx.x + warp; item < col_groups * parts; item += warps) {
    const int part = item / col_groups, col = (item - part * col_groups) * 256 + lane * 8;
    const int r0 = part * per, r1 = min(g.sum_rows, r0 + per);
    if (col >= g.sum_cols || r0 >= r1) continue;
    F2 acc[4] = {f2_splat(0.f), f2_splat(0.f), f2_splat(0.f), f2_splat(0.f)};
    const __nv_bfloat16* x = g.sum_x + col;
    for (int r = r0; r < r1; r += 8) {
      uint4 q[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) q[i] = r + i < r1 ? __ldg(reinterpret_cast<const uint4*>(x + static_cast<long long>(r + i) * g.sum_ld)) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t w[4] = {q[i].x, q[i].y, q[i].z, q[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float lo, hi;
          unpack_bf16x2(w[j], lo, hi);
          acc[j] = f2_add(acc[j], f2_make(lo, hi));
        }
      }
    }
    float v[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (g.p[0].alpha) acc[j] = f2_mul(acc[j], f2_splat(__ldg(g.p[0].alpha)));
      f2_get(acc[j], v[2 * j], v[2 * j + 1]);
    }
    red_add_v4(g.sum_out + col, v[0], v[1], v[2], v[3]);
    red_add_v4(g.sum_out + col + 4, v[4], v[5], v[6], v[7]);
  }
}

constexpr int gemm_threads(int problems) { return kGemmThreads + (problems == 2 ? 64 : 0); }

// kParts: a kernel of its own for the reduction in parts; the choices below cost the others' epilogue (8192 x 2048 x 512 with GELU 23.8 -> 24.8 us).
template <int kCG, int kBN, int kProblems, bool kParts>
__global__ void __launch_bounds__(gemm_threads(kProblems), 1)
gemm_bf16_kernel(const __grid_constant__ GemmLaunch<kProblems> g) {
  const GemmParams& p = g.p[0];
  using Cfg = GemmCfg<kCG, kBN>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // 1024-byte alignment: the 128-byte swizzle pattern is a function of address bits [4,10). Dynamic shared memory starts so where a kernel has no
  // other; there is no room to round up.
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023) {
    set_status(p.status, kStatusBadArg);
    return;
  }
  uint8_t* stage_base = smem;
  uint8_t* epi_smem = smem + Cfg::STAGES * Cfg::STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(epi_smem + Cfg::EPI_BYTES);
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* tfull_bar = empty_bar + Cfg::STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint64_t* aux_bar = tempty_bar + 2;          // two per epilogue warp
  uint64_t* peer_bar = aux_bar + 2 * kEpiWarps;      // the pair's other CTA holds its TMEM
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(peer_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* bias_smem = reinterpret_cast<float*>(epi_smem + Cfg::EPI_BYTES + Cfg::BAR_BYTES);

  const int warp = uniform_warp();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = (kCG == 2) ? cluster_ctarank() : 0u;
  const int group = blockIdx.x / kCG;          // CTA (pair) index
  const int num_groups = gridDim.x / kCG;

#if FB_TIMELINE
  if (p.ts && threadIdx.x == 0) {
    unsigned long long g;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(g));
    p.ts[blockIdx.x * 8 + 0] = static_cast<long long>(g);
    p.ts[blockIdx.x * 8 + 1] = clock64();
  }
#endif
  // The loads wait for the barriers alone (of both CTAs), not for the TMEM allocation, which the other warps hear of through barrier 1.
  if (warp == 0) {
    if (lane == 0) {
      for (int s = 0; s < Cfg::STAGES; ++s) {
        mbar_init(&full_bar[s], 1);
        mbar_init(&empty_bar[s], 1);
      }
      for (int a = 0; a < 2; ++a) {
        mbar_init(&tfull_bar[a], 1);
        mbar_init(&tempty_bar[a], kEpiWarps * kCG);
      }
      if (p.aux_tma == 2)
        for (int w = 0; w < 2 * kEpiWarps; ++w) mbar_init(&aux_bar[w], 1);
      if (kCG == 2) mbar_init(peer_bar, 1);
      *abort_flag = 0;
      mbar_fence_init();
    }
    __syncwarp();
  }
  if constexpr (kCG == 2) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  if (warp == 0) {
    asm volatile("bar.arrive 1, %0;" ::"n"(kGemmThreads) : "memory");
    if (lane == 0) {
      for (int i = 0; i < kProblems; ++i) {
        tma_prefetch_desc(&g.a[i]);
        tma_prefetch_desc(&g.b[i]);
      }
    }
    __syncwarp();
  } else if (warp < 2 + kEpiWarps) {
    if (warp == 2 && lane == 0) {
      for (int i = 0; i < kProblems; ++i)
        if (g.p[i].c_mode) tma_prefetch_desc(&g.c[i]);
      if (p.aux_tma) tma_prefetch_desc(&g.aux);
    }
    if (warp == 1) {
      tmem_alloc<kCG>(tmem_slot, Cfg::TMEM_COLS);
      tmem_relinquish<kCG>();
    }
    tc_fence_before_sync();
    asm volatile("bar.sync 1, %0;" ::"n"(kGemmThreads) : "memory");
    tc_fence_after_sync();
  }
  if constexpr (kCG == 2) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if constexpr (kCG == 1) __syncthreads();        // one CTA: nothing to gain by starting its loads earlier
  const uint32_t tmem_base = warp == 0 || warp >= 2 + kEpiWarps ? 0 : *tmem_slot;
  if constexpr (kCG == 2)
    if (warp == 1 && lane == 0 && rank == 1) mbar_arrive_cluster(peer_bar, 0);
  // Programmatic dependent launch: everything above (barriers, descriptor prefetch, TMEM) touched
  // no global data and may run while the previous kernel of the stream drains; from here on this
  // kernel reads what that kernel wrote.
  FB_TIMELINE_ONLY(if (p.ts && threadIdx.x == 0) p.ts[blockIdx.x * 8 + 7] = clock64();)
  pdl_wait();
  pdl_launch_dependents();

  int m_eff = p.M, k_eff = p.K;
  if (kProblems == 1 && p.m_dyn) m_eff = max(0, min(p.M, *p.m_dyn));
  if (kProblems == 1 && p.k_dyn) k_eff = max(0, min(p.K, *p.k_dyn));
  Worklist<kCG, kBN, kProblems, kParts> work(g, group, num_groups, m_eff, k_eff);
  Segment seg;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      while (ok && work.next(seg)) {
        const int prob = kProblems == 1 ? 0 : seg.prob;
        const CUtensorMap *tmA = &g.a[prob], *tmB = &g.b[prob];
        const int a_mn = g.p[prob].a_mn, b_mn = g.p[prob].b_mn;
        const int m0 = seg.tm * BM * kCG + static_cast<int>(rank) * BM;
        const int n0 = seg.tn * kBN + static_cast<int>(rank) * Cfg::BN_CTA;
        for (int kb = seg.kb0; kb < seg.kb1; ++kb) {
          ok = warp_wait(&empty_bar[s], ph ^ 1, abort_flag, p.status, kStatusWaitEmpty);
          if (!ok) break;
          uint8_t* sa = stage_base + s * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + Cfg::A_BYTES;
          if (elect_one()) {
            if (kCG == 1 || rank == 0) mbar_expect_tx(&full_bar[s], Cfg::STAGE_BYTES * kCG);
            const auto load = [&](uint8_t* to, const CUtensorMap* map, int x, int y) {
              if constexpr (kCG == 1) tma_load_2d(to, map, &full_bar[s], x, y);
              else tma_load_2d_pair(to, map, &full_bar[s], x, y);
            };
            if (!a_mn) {
              load(sa, tmA, kb * BK, m0);
            } else {
              load(sa, tmA, m0, kb * BK);
              load(sa + 8192, tmA, m0 + 64, kb * BK);
            }
            if (!b_mn) {
              load(sb, tmB, kb * BK, n0);
            } else {
#pragma unroll
              for (int q = 0; q < Cfg::BN_CTA / 64; ++q) load(sb + q * 8192, tmB, n0 + q * 64, kb * BK);
            }
          }
          __syncwarp();
          if (++s == Cfg::STAGES) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (rank == 0) {
      const uint32_t hi = smem_desc_hi(1024);
      int s = 0;
      uint32_t ph = 0;
      int it = 0;
      bool ok = true;
      if constexpr (kCG == 2) ok = warp_wait(peer_bar, 0, abort_flag, p.status, kStatusWaitEpi);
      for (; ok && work.next(seg); ++it) {
        const int a_mn = g.p[kProblems == 1 ? 0 : seg.prob].a_mn, b_mn = g.p[kProblems == 1 ? 0 : seg.prob].b_mn;
        const uint32_t idesc = make_idesc_bf16(BM * kCG, kBN, a_mn, b_mn);
        const uint32_t a_kstep = (a_mn ? 2048u : 32u) >> 4, b_kstep = (b_mn ? 2048u : 32u) >> 4;
        const uint32_t a_first = smem_desc_lo(smem_u32(stage_base), a_mn ? 8192u : 16u), b_first = smem_desc_lo(smem_u32(stage_base) + Cfg::A_BYTES, b_mn ? 8192u : 16u);
        const int acc = it & 1;
        ok = warp_wait(&tempty_bar[acc], ((it >> 1) & 1) ^ 1, abort_flag, p.status, kStatusWaitEpi);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * kBN;
        for (int kb = seg.kb0; kb < seg.kb1; ++kb) {
          ok = warp_wait(&full_bar[s], ph, abort_flag, p.status, kStatusWaitFull);
          if (!ok) break;
          tc_fence_after_sync();
          FB_TIMELINE_ONLY(if (p.ts && it == 0 && kb == seg.kb0) p.ts[blockIdx.x * 8 + 2] = clock64();)
          const uint32_t a_lo = a_first + s * (Cfg::STAGE_BYTES >> 4), b_lo = b_first + s * (Cfg::STAGE_BYTES >> 4);
          if (elect_one()) {
#pragma unroll
            for (int k4 = 0; k4 < BK / 16; ++k4)
              umma_bf16<kCG>(d_tmem, desc_of(a_lo + k4 * a_kstep, hi), desc_of(b_lo + k4 * b_kstep, hi), idesc, (kb > seg.kb0 || k4 > 0) ? 1u : 0u);
            if constexpr (kCG == 1) umma_commit(&empty_bar[s]);
            else umma_commit_pair(&empty_bar[s], 3);
          }
          __syncwarp();
          if (++s == Cfg::STAGES) { s = 0; ph ^= 1; }
        }
        if (!ok) break;
        if (elect_one()) {
          if constexpr (kCG == 1) umma_commit(&tfull_bar[acc]);
          else umma_commit_pair(&tfull_bar[acc], 3);
        }
        __syncwarp();
        FB_TIMELINE_ONLY(if (p.ts && it == 0) p.ts[blockIdx.x * 8 + 3] = clock64();)
      }
    }
  } else if (kProblems == 2 && warp >= 2 + kEpiWarps) {
    if (g.sum_out) column_sums(g, warp - 2 - kEpiWarps, lane);
  } else {
    // ------------------------------------------------------------------ epilogue warps
    // What bounds a tile of a short reduction (K = 768: 6.1k cycles of products) is this part, so it is kept below that: 64 columns come out
    // of TMEM per wait, two values share an instruction, the accumulator is handed back before the last columns are worked on, the bias waits in
    // shared memory, and GELU' finds the pre-activations in the staging tile, where a TMA load of the previous tile's time has put them, and
    // leaves its result in their place. Cycles per tile of a launch's first tiles, before and now: plain 3.7k and 2.0k, bias 4.7k and 2.6k, GELU
    // with its pre-activation 9.2k and 7.2k, GELU' 21k (its loads of 64 bytes per row were not coalesced) and 9k. At 4096 x 3072 x 768: 21.6 -> 20.0,
    // 29.0 -> 24.3 and 44.8 -> 26.8 us. Sixteen epilogue warps instead of eight shorten a tile further but start 0.3 us later: 20.0 us again.
    const int q = warp & 3;                 // TMEM lane quarter this warp may touch
    const int half = (warp - 2) >> 2;       // which half of the tile's columns
    constexpr int kSplit = Cfg::EPI_SPLIT;
    const int cols = half ? kBN - kSplit : kSplit;
    constexpr bool kStaged = kBN >= 128;    // a warp of a 64-wide tile has less than a staged store's 64 columns
    EpiWarp w;
    w.stage[0] = epi_smem + (warp - 2) * 4096;
    w.stage[1] = epi_smem + (kEpiWarps + warp - 2) * 4096;
    w.aux_bar = aux_bar + 2 * (warp - 2);
    w.staged = 0;
    w.lane = lane;
    int aux_u = group, aux_c = 0;           // where the next load of pre-activations starts (lane 0)
    uint32_t aux_issued = 0;
    const auto load_aux = [&] {             // the next 64 columns of this warp's rows, into the staging tile whose turn it is
      for (; aux_u < work.units; aux_u += num_groups, aux_c = 0) {
        int tm, tn;
        tile_of(aux_u, work.num_m, work.num_n, p.band, tm, tn);
        const int col = tn * kBN + half * kSplit + aux_c;
        if (aux_c >= cols || col >= p.N) continue;
        const uint32_t b = aux_issued++ & 1;
        mbar_expect_tx(&w.aux_bar[b], 4096);
        tma_load_2d(w.stage[b], &g.aux, &w.aux_bar[b], col, tm * BM * kCG + static_cast<int>(rank) * BM + q * 32);
        aux_c += 64;
        return;
      }
    };
    if (kStaged && p.aux_tma == 2 && lane == 0) {
      load_aux();
      load_aux();
    }
    // Thread i of the four warps of a half keeps column i's bias of the tile to come.
    const bool staged_bias = kStaged && kProblems == 1 && p.bias != nullptr && p.kind != kEpiDirect;
    const auto bias_of = [&](int u) -> float {
      if (u >= work.units) return 0.f;
      int tm, tn;
      tile_of(u / work.parts(), work.num_m, work.num_n, p.band, tm, tn);
      const int c = q * 32 + lane, col = tn * kBN + half * kSplit + c;
      if (c >= cols || col >= p.N) return 0.f;
      return p.bias_fp32 ? __ldg(static_cast<const float*>(p.bias) + col) : __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[col]);
    };
    float next_bias = staged_bias ? bias_of(group) : 0.f;
    int it = 0;
    bool ok = true;
    for (; work.next(seg); ++it) {
      const GemmParams& pp = g.p[kProblems == 1 ? 0 : seg.prob];
      const CUtensorMap& tmC = g.c[kProblems == 1 ? 0 : seg.prob];
      const int row0 = (kParts ? seg.tm + seg.ks * work.num_m : seg.tm) * BM * kCG + static_cast<int>(rank) * BM + q * 32;
      const int ncol0 = seg.tn * kBN + half * kSplit;
      const int acc = it & 1;
      uint32_t bias = 0;
      if (staged_bias) {
        // Two slices in turn: this one was last read a tile before the previous barrier. A warp whose wait gave up still comes here for every
        // tile, so the barrier never lacks one.
        float* slice = bias_smem + acc * 256 + half * 128;
        slice[q * 32 + lane] = next_bias;
        if (half) asm volatile("bar.sync 3, 128;" ::: "memory");
        else asm volatile("bar.sync 2, 128;" ::: "memory");
        next_bias = bias_of(work.u);
        if (seg.ks == 0) bias = smem_u32(slice);
      }
      if (ok) ok = warp_wait(&tfull_bar[acc], (it >> 1) & 1, abort_flag, p.status, kStatusWaitAccum);
      if (!ok) continue;
      tc_fence_after_sync();
      FB_TIMELINE_ONLY(if (p.ts && it == 0 && warp == 2 && lane == 0) p.ts[blockIdx.x * 8 + 4] = clock64();)
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * kBN + half * kSplit;
      const auto hand_back = [&] {          // this warp has read all it needs of the accumulator
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          if (kCG == 1 || rank == 0) mbar_arrive(&tempty_bar[acc]);
          else mbar_arrive_cluster_tmem(&tempty_bar[acc], 0);
        }
      };
      if constexpr (kStaged) {
        // (of a part, whose rows reach to the end of its last tile, only those that are read)
        const bool unread = kParts && seg.tm * BM * kCG + static_cast<int>(rank) * BM + q * 32 >= m_eff;
        const int chunks = ncol0 >= pp.N || unread ? 0 : (min(cols, pp.N - ncol0) + 63) / 64;
        const auto run = [&](auto kind) {
          ok = epilogue_tile<decltype(kind)::value>(pp, kParts ? g.aux : tmC, g.aux, w, taddr, ncol0, row0, chunks, bias, abort_flag, hand_back, load_aux);
        };
        if constexpr (kParts) {
          if (chunks == 0) hand_back();
          else if (work.split == 1) run(std::integral_constant<int, kEpiPlain>());
          else epilogue_tile_f32(pp, tmC, w, taddr, ncol0, row0, min(cols, pp.N - ncol0), bias, hand_back);
          continue;
        }
        if (pp.kind != kEpiDirect) {
          if (chunks == 0) hand_back();
          else if (pp.kind == kEpiPlain) run(std::integral_constant<int, kEpiPlain>());
          else if (pp.kind == kEpiF32) epilogue_tile_f32(pp, tmC, w, taddr, ncol0, row0, min(cols, pp.N - ncol0), bias, hand_back);
          else if (pp.kind == kEpiGelu) run(std::integral_constant<int, kEpiGelu>());
          else if (pp.kind == kEpiGeluAux) run(std::integral_constant<int, kEpiGeluAux>());
          else if (pp.kind == kEpiDgelu) run(std::integral_constant<int, kEpiDgelu>());
          else run(std::integral_constant<int, kEpiDgeluTanh>());
          continue;
        }
      }
#pragma unroll 1
      for (int c = 0; c < cols; c += 32) {
        uint32_t v[32];
        tmem_ld32(taddr + c, v);
        tmem_ld_wait();
        epilogue_store32(pp, v, row0 + lane, ncol0 + c, seg.ks == 0);
      }
      hand_back();
      FB_TIMELINE_ONLY(if (p.ts && it == 0 && warp == 2 && lane == 0) p.ts[blockIdx.x * 8 + 5] = clock64();)
    }
    // The staging tiles must have been read, and loads into them must have landed, before the CTA (and its shared memory) goes away; the
    // writes themselves complete with the grid, as every other global store does.
    if (kStaged && p.kind != kEpiDirect && lane == 0) {
      tma_store_wait_read();
      for (uint32_t n = w.staged; n < aux_issued; ++n)      // none, unless a wait gave up
        for (uint32_t polls = 0; polls < (1u << 20) && !mbar_test(&w.aux_bar[n & 1], (n >> 1) & 1); ++polls) __nanosleep(40);
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
#if FB_TIMELINE
  if (p.ts && threadIdx.x == 0) {
    p.ts[blockIdx.x * 8 + 6] = clock64();
    unsigned long long g;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(g));
    p.ts[blockIdx.x * 8 + 7] = static_cast<long long>(g);   // wall-clock end
  }
#endif
  if constexpr (kCG == 2) cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc<kCG>(tmem_base, Cfg::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------
// 256x256 pair tiles with the reduction split over two pairs
// ---------------------------------------------------------------------------------------------
// For a bf16 result of so few 256x256 tiles that half the SMs would idle (4096 x 512, 2048 x 1024), and a reduction long enough to be
// worth halving. What bounds such a product is the rate at which an SM takes operands from L2, and a pair tile takes half of what
// 128x128 tiles on every SM do for the same arithmetic. A cluster of four CTAs works on one tile: CTAs 0, 1 sum the first half of K,
// CTAs 2, 3 the second. Each CTA hands its partner (two ranks on) the 128 columns that the partner finishes, through the partner's
// shared memory, adds what it was handed to its own and runs the epilogue.
// Back to back in one graph, us, against the best of the persistent kernel's tiles: 4096 x 512 x 2048 12.7 (14.4), x 4096 18.6 (24.4);
// 2048 x 768 x 3072 14.8 (19.0); 2048 x 1024 x 4096 17.6 (23.8); 1024 x 768 x 2048 11.3 (13.7).
struct SplitCfg {
  static constexpr int STAGES = 4, STAGE_BYTES = 2 * BM * BK * 2;
  static constexpr int XCHG_BYTES = BM * 128 * 4;       // 16-byte chunk c of row r at (c * 128 + r) * 16: lanes (rows) side by side
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + XCHG_BYTES + 1024 /*align slack*/ + 256 /*barriers*/;
  static_assert(2 * kEpiWarps * 4096 <= STAGES * STAGE_BYTES, "the epilogue stages its stores where the operands were");
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
};
// Below this the hand-over costs more than half the reduction: 4096 x 512, K = 1024 10.2 against 9.8 us, 1280 10.9 both, 1536 11.5 against 12.2.
constexpr int kSplitMinK = 1280;

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ float4 ld_shared_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// grid = (4, row tiles, column tiles), cluster (4, 1, 1)
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
                  const __grid_constant__ CUtensorMap tmAux, const __grid_constant__ GemmParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using Cfg = SplitCfg;
  uint8_t* xchg = smem + Cfg::STAGES * Cfg::STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(xchg + Cfg::XCHG_BYTES);
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* done_bar = empty_bar + Cfg::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank()), side = rank & 1, part = rank >> 1;
  const int m0 = blockIdx.y * 2 * BM + side * BM, n0 = blockIdx.z * 256;
  const int num_kb = (p.K + BK - 1) / BK, kb_half = (num_kb + 1) / 2;      // num_kb >= 2
  const int kb0 = part * kb_half, kb1 = part ? num_kb : kb_half;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmC);
    if (p.aux_tma == 1) tma_prefetch_desc(&tmAux);
  }
  if (warp == 1) {
    tmem_alloc<2>(tmem_slot, 256);
    tmem_relinquish<2>();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();
  pdl_launch_dependents();

  // what this CTA finishes: columns [part * 128, part * 128 + 128) of the tile
  const int q = warp & 3, half = (warp - 2) >> 2, row0 = m0 + q * 32;
  const uint32_t lane_base = tmem + (static_cast<uint32_t>(q * 32) << 16);
  bool ok = true;
  if (warp == 0) {
    int s = 0;
    uint32_t ph = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!warp_wait(&empty_bar[s], ph ^ 1, abort_flag, p.status, kStatusWaitEmpty)) break;
      uint8_t* sa = smem + s * Cfg::STAGE_BYTES;
      uint8_t* sb = sa + BM * BK * 2;
      if (elect_one()) {
        if (side == 0) mbar_expect_tx(&full_bar[s], 2 * Cfg::STAGE_BYTES);
        tma_load_2d_pair(sa, &tmA, &full_bar[s], kb * BK, m0);
        if (!p.b_mn) {
          tma_load_2d_pair(sb, &tmB, &full_bar[s], kb * BK, n0 + side * 128);
        } else {
          tma_load_2d_pair(sb, &tmB, &full_bar[s], n0 + side * 128, kb * BK);
          tma_load_2d_pair(sb + 8192, &tmB, &full_bar[s], n0 + side * 128 + 64, kb * BK);
        }
      }
      __syncwarp();
      if (++s == Cfg::STAGES) { s = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    if (side == 0) {
      const uint32_t idesc = make_idesc_bf16(2 * BM, 256, 0, p.b_mn);
      const uint32_t b_lbo = p.b_mn ? 8192u : 16u, b_kstep = p.b_mn ? 2048u : 32u;
      const uint16_t pair = static_cast<uint16_t>(3 << (rank & 2));
      int s = 0;
      uint32_t ph = 0;
      for (int kb = kb0; kb < kb1 && ok; ++kb) {
        ok = warp_wait(&full_bar[s], ph, abort_flag, p.status, kStatusWaitFull);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t sa = smem_u32(smem + s * Cfg::STAGE_BYTES), sb = sa + BM * BK * 2;
        if (elect_one()) {
#pragma unroll
          for (int k4 = 0; k4 < BK / 16; ++k4)
            umma_bf16<2>(tmem, make_smem_desc(sa + k4 * 32, 16, 1024), make_smem_desc(sb + k4 * b_kstep, b_lbo, 1024), idesc, (kb > kb0 || k4 > 0) ? 1u : 0u);
          umma_commit_pair(&empty_bar[s], pair);
        }
        __syncwarp();
        if (++s == Cfg::STAGES) { s = 0; ph ^= 1; }
      }
      if (ok && elect_one()) umma_commit_pair(done_bar, pair);
      __syncwarp();
    }
  } else {
    ok = warp_wait(done_bar, 0, abort_flag, p.status, kStatusWaitAccum);
    if (ok) {       // the partner's columns into the partner's shared memory
      tc_fence_after_sync();
      uint32_t there;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(smem_u32(xchg)), "r"(rank ^ 2));
#pragma unroll 1
      for (int c = half * 64; c < half * 64 + 64; c += 32) {
        uint32_t v[32];
        tmem_ld32(lane_base + (part ^ 1) * 128 + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          st_cluster_v4(there + ((c / 4 + j) * 128 + q * 32 + lane) * 16, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      }
    }
  }
  __syncwarp();
  cluster_sync_all();      // every thread gets here, also after a wait that gave up
  if (warp >= 2) {
    const int col0 = n0 + part * 128 + half * 64;
    if (ok && !*abort_flag && row0 < p.M && col0 < p.N) {
      uint8_t* stage = smem + (warp - 2) * 4096;           // every product that reads the operands has retired
      uint8_t* stage_x = smem + (kEpiWarps + warp - 2) * 4096;
      const uint32_t sc = smem_u32(stage), sx = smem_u32(stage_x), mine = smem_u32(xchg);
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int c = half * 64 + 32 * hh;
        uint32_t acc[32];
        tmem_ld32(lane_base + part * 128 + c, acc);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 t = ld_shared_f4(mine + ((c / 4 + j) * 128 + q * 32 + lane) * 16);
          acc[4 * j] = __float_as_uint(__uint_as_float(acc[4 * j]) + t.x);
          acc[4 * j + 1] = __float_as_uint(__uint_as_float(acc[4 * j + 1]) + t.y);
          acc[4 * j + 2] = __float_as_uint(__uint_as_float(acc[4 * j + 2]) + t.z);
          acc[4 * j + 3] = __float_as_uint(__uint_as_float(acc[4 * j + 3]) + t.w);
        }
        float v0[32], p0[32];
        epilogue_compute32(p, acc, row0 + lane, col0 + 32 * hh, true, v0, p0);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          st_shared_v4(stage_addr(sc, lane, 4 * hh + j), pack_bf16x2(v0[8 * j], v0[8 * j + 1]), pack_bf16x2(v0[8 * j + 2], v0[8 * j + 3]),
                       pack_bf16x2(v0[8 * j + 4], v0[8 * j + 5]), pack_bf16x2(v0[8 * j + 6], v0[8 * j + 7]));
        if (p.aux_tma == 1) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            st_shared_v4(stage_addr(sx, lane, 4 * hh + j), pack_bf16x2(p0[8 * j], p0[8 * j + 1]), pack_bf16x2(p0[8 * j + 2], p0[8 * j + 3]),
                         pack_bf16x2(p0[8 * j + 4], p0[8 * j + 5]), pack_bf16x2(p0[8 * j + 6], p0[8 * j + 7]));
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tmC, stage, col0, row0);
        if (p.aux_tma == 1) tma_store_2d(&tmAux, stage_x, col0, row0);
        tma_store_commit();
        tma_store_wait_read();       // before the shared memory goes away
      }
      __syncwarp();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();        // the pair frees its TMEM together
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc<2>(tmem, 256);
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

// The tensor-map encoder is a driver-API call and wants a context current on the calling thread;
// autograd's backward threads only have the runtime's lazy binding, so bind once per thread. The call that does it is refused while a stream is
// captured, and a thread's first product may be under capture, so it is made in the relaxed mode.
void ensure_thread_context() {
  static thread_local bool ready = false;
  if (!ready) {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    cudaFree(nullptr);
    cudaThreadExchangeStreamCaptureMode(&mode);
    ready = true;
  }
}

// 2-D bf16 tensor map over a row-major [rows][ld] matrix with a {box_inner, box_outer} box.
int make_tmap_bf16_2d(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld_elems,
                      uint32_t box_inner, uint32_t box_outer) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return -1;
  ensure_thread_context();
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld_elems * 2};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

// Tensor map for a staged epilogue store: 32 rows x 128 bytes per box, 128-byte swizzle.
static int make_tmap_out(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows, uint64_t ld_elems, bool fp32) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return -1;
  ensure_thread_context();
  const uint64_t esz = fp32 ? 4 : 2;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld_elems * esz};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / esz), 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(out, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
                  strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

template <int kCG, int kBN, int kProblems, bool kParts = false>
static int launch_gemm(const GemmLaunch<kProblems>& g, int groups, cudaStream_t stream) {
  using Cfg = GemmCfg<kCG, kBN>;
  auto kern = gemm_bf16_kernel<kCG, kBN, kProblems, kParts>;
  if (const cudaError_t e = allow_smem<gemm_bf16_kernel<kCG, kBN, kProblems, kParts>>(Cfg::SMEM_BYTES)) return static_cast<int>(e);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(groups * kCG, 1, 1);
  cfg.blockDim = dim3(gemm_threads(kProblems), 1, 1);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kCG;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (pdl_enabled()) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, g));
}
template <int kCG, int kBN>
static int launch_one(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tx, const GemmParams& p, cudaStream_t stream) {
  GemmLaunch<1> g;
  std::memset(&g, 0, sizeof(g));
  g.a[0] = ta; g.b[0] = tb; g.c[0] = tc; g.aux = tx; g.p[0] = p;
  const int units = ((p.M + BM * kCG - 1) / (BM * kCG)) * ((p.N + kBN - 1) / kBN) * p.split_k;
  return launch_gemm<kCG, kBN, 1>(g, units < sm_count() / kCG ? units : sm_count() / kCG, stream);
}

// Bands of at most 12 column tiles: the pairs at work at one time then share about as many column as row panels of the operands (row tiles fastest,
// all read one column's), and rows are read from HBM once where they used to be again for every column. 24576 x 768 x 3072 109 -> 95 us, 24576 x 3072 x 768
// with GELU 129 -> 114, 8192 x 2048 x 512 (dX) 18.7 -> 17.7; bands of 8 or 16 are within 1 % of these.
static int band_of(int N, int tile) {
  const int tiles = (N + tile - 1) / tile, bands = (tiles + 11) / 12;
  return (tiles + bands - 1) / bands;
}

// Whether dX and dW of a linear layer go out as one launch (fb_gemm_backward). Us against dX, dW and db on two streams, rows x n x k: 4096 x 768 x 768
// 15.9 (19.5), 4096 x 768 x 3072 with GELU' 39.2 (47.7), 4096 x 3072 x 768 33.3 (39.5), 8192 x 512 x 512 15.6 (20.6), 2048 x 512 x 512 8.5 (11.2), 512 x 128 x 128
// 6.2 (10.2). Not for few rows, whose dX has few tiles and whose dW has little to sum per tile (77 x 768 x 768 12.7 against 10.9), nor for a dX of few
// tiles with a long reduction, which others split over a cluster (1024 x 3072 x 768 19.4 against 17.1, 768 x 3072 x 768 19.2 against 21.7).
// Nor where a tile of dX alone (`chain` K blocks) takes longer than a pair's share of everything (`share`), when that is long: the caller splits its
// reduction (2048 x 32000 x 512 187 against 153, 4096 x 32000 x 512 207 against 255).
static bool backward_in_one(int rows, int n, int tiles0, long long chain, long long share) {
  return rows >= 256 && (n < 2304 || tiles0 > 12) && (n < 6400 || chain * 4 <= share * 5);
}

// Whether they go out in 128 x 64 tiles of one CTA instead of 256 x 256 tiles of a pair. A small layer has less than a tile for each pair, and then the time
// is that of one tile's chain (its loads, its products, its epilogue of 256 columns), of which a 64-wide tile has a third. That holds as long as dX's tiles
// leave SMs to dW; beyond, and where an SM has more than some 50 K blocks to go through, the wide tiles' fewer bytes per product count. Below 65 rows
// there is nothing to sum in dW. Us against pair tiles: 256 x 128 x 128 4.1 (6.2), 512 x 512 x 128 4.7 (7.1), 512 x 128 x 512 with GELU' 5.6 (8.9),
// 512 x 512 x 512 4.7 (7.8), 512 x 768 x 768 6.2 (8.4), 1024 x 2048 x 512 9.8 (14.6), 4096 x 1024 x 256 10.8 (12.9); 1536 x 768 x 768, whose dX has 144 tiles,
// 9.5 (9.2), 512 x 768 x 3072 with GELU', 192 tiles, 16.5 (13.8). Against dX beside dW and db, where pair tiles are not taken: 77 x 768 x 768 5.5 (6.5), 200 x 512 x 512
// 4.6 (6.5), 512 x 3072 x 768 13.8 (18.7), 768 x 3072 x 768 15.7 (22.2); 16 x 768 x 768 8.0 (5.9), 1024 x 3072 x 768, 62 blocks an SM, 19.2 (18.0).
static bool backward_narrow(int rows, int n, int k) {
  const long long tiles0 = static_cast<long long>((rows + BM - 1) / BM) * ((k + 63) / 64), tiles1 = static_cast<long long>((n + BM - 1) / BM) * ((k + 63) / 64);
  const int kb0 = (n + BK - 1) / BK, kb1 = (rows + BK - 1) / BK, sms = sm_count();
  return rows > 64 && tiles0 * 8 <= sms * 7 && kb0 <= 50 && tiles0 * kb0 + tiles1 * kb1 <= 50 * sms;
}

static cudaLaunchConfig_t split_config(int M, int N, cudaLaunchAttribute* attr, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(4, (M + 2 * BM - 1) / (2 * BM), (N + 255) / 256);
  cfg.blockDim = dim3(kGemmThreads, 1, 1);
  cfg.dynamicSmemBytes = SplitCfg::SMEM_BYTES;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 4;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// How many clusters of gemm_split_kernel the device holds at once (0: none, or it cannot be told).
static int split_clusters() {
  static PerDevice held;
  return held.get([] {
    if (allow_smem<gemm_split_kernel>(SplitCfg::SMEM_BYTES) != cudaSuccess) return 0;
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = split_config(2 * BM, 256, attr, nullptr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, gemm_split_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return clusters;
  });
}

// Long reductions (kSplitMinK) with no more tiles than the device holds clusters at once: one more and the last tile would run
// alone, when the persistent kernel does not need the pairs' full number. Mostly padding (less than 0.8 useful) is left to narrower tiles.
// Products of so few tiles of 128 x 64 that gemm_small.cu applies went there before this is asked.
static bool split_applies(int M, int N, int K) {
  const long long tiles = static_cast<long long>((M + 2 * BM - 1) / (2 * BM)) * ((N + 255) / 256);
  return K >= kSplitMinK && tiles <= split_clusters() && static_cast<long long>(M) * N * 10 >= tiles * 256 * 256 * 8;
}

static int launch_split(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tx, const GemmParams& p, cudaStream_t stream) {
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = split_config(p.M, p.N, attr, stream);
  if (pdl_enabled()) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  return static_cast<int>(cudaLaunchKernelEx(&cfg, gemm_split_kernel, ta, tb, tc, tx, p));
}

}  // namespace fb

extern "C" int fb_gemm_bf16_ts(const void*, const void*, void*, int, int, int, long long, long long, long long, int, int, int, const void*, int,
                               int, void*, long long, const float*, int, int, int, int*, long long*, void*);
extern "C" int fb_gemm_bf16_dyn(const void*, const void*, void*, int, int, int, long long, long long, long long, int, int, int, const void*, int,
                                int, void*, long long, const float*, int, int, int, int*, long long*, const int*, const int*, void*);

extern "C" int fb_gemm_pick_config(int M, int N, int K, int split_k) {
  // Score = SM occupancy of the last wave x a per-tile efficiency prior (bigger tiles re-use
  // operands more and are less L2-bound). Configs: 0 = pair 256x256, 1 = 128x256, 2 = 128x128, 3 = 128x64, 4 = 128x192, 5 = pair 256x192.
  const int sms = 148;
  // Single-CTA tiles read A and the whole B tile from shared memory for every MMA and run close to
  // the shared-memory bandwidth limit; the pair configs (each CTA reads half of B) do not, hence
  // their higher prior. (Back to back in isolation the single-CTA 128x192 tile is the fastest shape for N = 768, 9.2 against
  // 9.9 / 10.4 us, but inside a BERT-base step, where these GEMMs share the GPU with the weight-gradient stream, preferring it
  // made the step 1.7 % slower: 6.01 against 5.90 ms in an A/B within one run. The prior stays at 0.80.) The 256x192 pair needs a K-major B (its 96-column half tile is not a whole
  // number of 64-column panels), so fb_gemm_bf16 falls back to 256x256 when B is MN-major.
  static const float prior192 = [] {      // tuning knob: FLODL_B200_GEMM_PRIOR192 overrides the 128x192 tile's prior
    const char* e = std::getenv("FLODL_B200_GEMM_PRIOR192");
    return e ? static_cast<float>(std::atof(e)) : 0.80f;
  }();
  const struct { int cg, bn; float prior; } cand[6] = {{2, 256, 1.00f}, {1, 256, 0.85f}, {1, 128, 0.70f}, {1, 64, 0.50f}, {1, 192, prior192}, {2, 192, 0.98f}};
  int best = 2;
  float best_score = -1.f;
  for (int i = 0; i < 6; ++i) {
    const int num_m = (M + 128 * cand[i].cg - 1) / (128 * cand[i].cg);
    const int num_n = (N + cand[i].bn - 1) / cand[i].bn;
    const long units = 1L * num_m * num_n * split_k;
    const int slots = sms / cand[i].cg;
    const long waves = (units + slots - 1) / slots;
    // useful fraction of the padded tile grid
    const float useful = (1.f * M * N) / (1.f * num_m * 128 * cand[i].cg * num_n * cand[i].bn);
    const float score = cand[i].prior * useful * (1.f * units) / (1.f * waves * slots);
    if (score > best_score) { best_score = score; best = i; }
  }
  (void)K;
  return best;
}

extern "C" int fb_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                            long long ldb, long long ldc, int a_mn, int b_mn, int c_fp32, const void* bias,
                            int bias_fp32, int epi, void* aux, long long ldaux, const float* alpha,
                            int accumulate, int split_k, int config, int* status, void* stream_) {
  return fb_gemm_bf16_ts(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, c_fp32, bias, bias_fp32, epi, aux, ldaux, alpha, accumulate, split_k,
                         config, status, nullptr, stream_);
}

extern "C" int fb_gemm_bf16_ts(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                               long long ldb, long long ldc, int a_mn, int b_mn, int c_fp32, const void* bias,
                               int bias_fp32, int epi, void* aux, long long ldaux, const float* alpha,
                               int accumulate, int split_k, int config, int* status, long long* ts, void* stream_) {
  return fb_gemm_bf16_dyn(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, c_fp32, bias, bias_fp32, epi, aux, ldaux, alpha, accumulate, split_k,
                          config, status, ts, nullptr, nullptr, stream_);
}

extern "C" int fb_gemm_bf16_dyn(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                                long long ldb, long long ldc, int a_mn, int b_mn, int c_fp32, const void* bias,
                                int bias_fp32, int epi, void* aux, long long ldaux, const float* alpha,
                                int accumulate, int split_k, int config, int* status, long long* ts, const int* m_dyn,
                                const int* k_dyn, void* stream_) {
  using namespace fb;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (split_k < 1) split_k = 1;
  if (split_k > 1 && !c_fp32) return -2;
  if (split_k > 1 && !accumulate) accumulate = 1;          // parts are added to what the caller has zeroed, also if only one of them holds a block
  split_k = k_dyn ? 1 : parts_with_blocks((K + BK - 1) / BK, split_k);
  if ((lda % 8) || (ldb % 8) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return -3;
  bool over_pairs = false;       // the reduction split over two pairs of a cluster
  if (config < 0) {
    // few output tiles, plain bf16 result: the cluster split (gemm_small.cu)
    if (!c_fp32 && !a_mn && !accumulate && split_k == 1 && !m_dyn && !k_dyn && !ts && gemm_small_aligned(N, C, ldc, aux, ldaux))
      if (const int split = gemm_small_split(M, N, K))
        return gemm_small(A, &B, C, M, N, 1, K, lda, ldb, ldc, b_mn, &bias, bias_fp32, epi, aux, ldaux, alpha, split, status, stream);
    const bool act = epi == FB_EPI_GELU_ERF || epi == FB_EPI_GELU_TANH;
    if (!c_fp32 && !a_mn && !accumulate && split_k == 1 && !m_dyn && !k_dyn && !ts && ldc % 8 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0 &&
        (!act || !aux || (ldaux % 8 == 0 && (reinterpret_cast<uintptr_t>(aux) & 15) == 0)) && split_applies(M, N, K))
      over_pairs = true;
    config = over_pairs ? 0 : fb_gemm_pick_config(M, N, K, split_k);
    if (config == 5 && b_mn) config = 0;          // 256x192 pair tiles need a K-major B
  }
  if (config == 5 && b_mn) return -5;
  const int cg = (config == 0 || config == 5) ? 2 : 1;
  const int bn = (config == 0 || config == 1) ? 256 : (config == 2 ? 128 : (config == 4 || config == 5 ? 192 : 64));
  const int bn_cta = bn / cg;

  CUtensorMap ta, tb;
  int r;
  if (!a_mn) r = make_tmap_bf16_2d(&ta, A, K, M, lda, BK, BM);
  else       r = make_tmap_bf16_2d(&ta, A, M, K, lda, 64, BK);
  if (r) return r;
  if (!b_mn) r = make_tmap_bf16_2d(&tb, B, K, N, ldb, BK, bn_cta);
  else       r = make_tmap_bf16_2d(&tb, B, N, K, ldb, 64, BK);
  if (r) return r;

  // epilogue path: staged TMA stores need 16-byte aligned rows; bf16 accumulate keeps the direct path
  const size_t c_esz = c_fp32 ? 4 : 2;
  const bool c_aligned = (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (ldc * c_esz) % 16 == 0;
  int c_mode = 0;
  if (c_aligned) {
    if (c_fp32) c_mode = (accumulate || split_k > 1) ? 2 : 1;
    else if (!accumulate) c_mode = 1;
  }
  const bool gelu_fwd = (epi == FB_EPI_GELU_ERF || epi == FB_EPI_GELU_TANH);
  if (c_fp32 && gelu_fwd) c_mode = 0;
  if (bn < 128) c_mode = 0;   // 32 columns per epilogue warp: narrower than one staged bf16 box
  int aux_tma = 0;
  if (gelu_fwd && aux) {
    if (c_mode == 1 && !c_fp32 && (reinterpret_cast<uintptr_t>(aux) & 15) == 0 && (ldaux * 2) % 16 == 0) aux_tma = 1;
    else c_mode = 0;
  }
  if (epi == FB_EPI_DGELU_ERF || epi == FB_EPI_DGELU_TANH) {
    if (over_pairs) {                          // that kernel reads the pre-activations itself, at any alignment, and stores C through its tensor map
    } else if (c_mode == 1 && !c_fp32 && (reinterpret_cast<uintptr_t>(aux) & 15) == 0 && (ldaux * 2) % 16 == 0) aux_tma = 2;
    else c_mode = 0;
  }
  CUtensorMap tc, tx;
  std::memset(&tc, 0, sizeof(tc));
  std::memset(&tx, 0, sizeof(tx));
  if (c_mode && (r = make_tmap_out(&tc, C, N, M, ldc, c_fp32 != 0))) return r;
  if (aux_tma && (r = make_tmap_out(&tx, aux, N, M, ldaux, false))) return r;

  GemmParams p;
  p.c_mode = c_mode; p.aux_tma = aux_tma;
  p.kind = c_mode == 0 ? kEpiDirect : c_fp32 ? kEpiF32 : aux_tma == 2 ? (epi == FB_EPI_DGELU_ERF ? kEpiDgelu : kEpiDgeluTanh) : aux_tma == 1 ? kEpiGeluAux : gelu_fwd ? kEpiGelu : kEpiPlain;
  p.M = M; p.N = N; p.K = K; p.a_mn = a_mn; p.b_mn = b_mn; p.C = C; p.ldc = ldc; p.c_fp32 = c_fp32;
  p.bias = bias; p.bias_fp32 = bias_fp32; p.epi = epi; p.aux = aux; p.ldaux = ldaux; p.alpha = alpha;
  p.accumulate = accumulate; p.split_k = split_k; p.status = status; p.ts = ts;
  p.m_dyn = m_dyn; p.k_dyn = k_dyn; p.part_groups = 0;
  p.band = band_of(N, bn);
  if (over_pairs) return launch_split(ta, tb, tc, tx, p, stream);
  switch (config) {
    case 0: return launch_one<2, 256>(ta, tb, tc, tx, p, stream);
    case 1: return launch_one<1, 256>(ta, tb, tc, tx, p, stream);
    case 2: return launch_one<1, 128>(ta, tb, tc, tx, p, stream);
    case 4: return launch_one<1, 192>(ta, tb, tc, tx, p, stream);
    case 5: return launch_one<2, 192>(ta, tb, tc, tx, p, stream);
    default: return launch_one<1, 64>(ta, tb, tc, tx, p, stream);
  }
}

// C[:, g * N : (g + 1) * N] = A B_g^T + bias_g for `groups` (at most three) K-major B's of one shape and leading dimension: one launch where
// the products are small together, else one after the other. bias: null, or an array with an entry (null or [N]) per product.
extern "C" int fb_gemm_bf16_grouped(const void* A, const void* const* B, void* C, int M, int N, int K, int groups, long long lda, long long ldb, long long ldc,
                                    const void* const* bias, int bias_fp32, int* status, void* stream_) {
  using namespace fb;
  if (M <= 0 || N <= 0 || K <= 0 || groups <= 0) return 0;
  if (groups > 3) return -2;
  const void* none[3] = {nullptr, nullptr, nullptr};
  if (!bias) bias = none;
  bool aligned = lda % 8 == 0 && ldb % 8 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0 && N % 64 == 0 && gemm_small_aligned(N, C, ldc, nullptr, 0);
  for (int g = 0; g < groups; ++g) aligned = aligned && (reinterpret_cast<uintptr_t>(B[g]) & 15) == 0;
  const int split = aligned ? gemm_small_split(M, N * groups, K, groups > 1) : 0;
  if (split)
    return gemm_small(A, B, C, M, N, groups, K, lda, ldb, ldc, 0, bias, bias_fp32, FB_EPI_NONE, nullptr, 0, nullptr, split, status, static_cast<cudaStream_t>(stream_));
  for (int g = 0; g < groups; ++g) {
    const int r = fb_gemm_bf16(A, B[g], static_cast<__nv_bfloat16*>(C) + static_cast<long long>(g) * N, M, N, K, lda, ldb, ldc, 0, 0, 0, bias[g], bias_fp32, FB_EPI_NONE,
                               nullptr, 0, nullptr, 0, 1, -1, status, stream_);
    if (r) return r;
  }
  return 0;
}

// The gradients of y = x W^T + b from dY in one launch: dX = dY W (times the activation's derivative at `aux`, the pre-activation that x came from,
// with `epi`), dW += dY^T x, db += column sums of dY (db may be null). dY [rows, n], W [n, k], x [rows, k] bf16; dX bf16; dW, db fp32.
// Returns -7 where two launches serve better or the layout does not fit: nothing has been launched then.
//
// All three times *alpha (may be null).
//
// dX comes in whole 256 x 256 tiles, one or two to a pair of SMs, which alone leave up to half the pairs idle at the end; dW's reduction can be
// cut anywhere, for its parts are added to memory, so it fills what dX leaves: each pair's share of dW's K blocks makes its total the same. One launch
// also has one start-up and one draining end instead of three of each, and leaves the stream's chain of programmatic launches whole.
extern "C" int fb_gemm_backward(const void* dY, const void* W, const void* X, void* dX, float* dW, float* db, int rows, int n, int k, long long ldy,
                                long long ldw, long long ldx, long long lddx, long long lddw, int epi, const void* aux, long long ldaux,
                                const float* alpha, int* status, void* stream_) {
  using namespace fb;
  const auto aligned = [](const void* q, long long ld, int esz) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0 && (ld * esz) % 16 == 0; };
  if (rows <= 0 || n <= 0 || k <= 0) return -7;
  if (!aligned(dY, ldy, 2) || !aligned(W, ldw, 2) || !aligned(X, ldx, 2) || !aligned(dX, lddx, 2) || !aligned(dW, lddw, 4)) return -7;
  if (db && ((reinterpret_cast<uintptr_t>(db) & 15) || n % 8)) return -7;
  const bool dgelu = epi == FB_EPI_DGELU_ERF || epi == FB_EPI_DGELU_TANH;
  if (dgelu ? !aux || !aligned(aux, ldaux, 2) : epi != FB_EPI_NONE) return -7;
  const int kb0 = (n + BK - 1) / BK, kb1 = (rows + BK - 1) / BK;
  const bool narrow = backward_narrow(rows, n, k);
  const int tm = narrow ? BM : 2 * BM, tn = narrow ? 64 : 256;
  const int tiles0 = ((rows + tm - 1) / tm) * ((k + tn - 1) / tn), tiles1 = ((n + tm - 1) / tm) * ((k + tn - 1) / tn);
  int groups = narrow ? sm_count() : sm_count() / 2;
  // Work is counted in K blocks of 64, which a pair's products take 530 cycles for; a tile of dX costs its epilogue on top, or that alone where it is
  // the longer.
  const int cost = (dgelu && !narrow ? (kb0 > 15 ? kb0 : 15) : kb0) + 3;
  if (!narrow && !backward_in_one(rows, n, tiles0, static_cast<long long>((tiles0 + groups - 1) / groups) * cost,
                                  (static_cast<long long>(tiles0) * cost + static_cast<long long>(tiles1) * kb1) / groups))
    return -7;
  if (tiles1 * static_cast<long long>(kb1) > (1 << 22)) return -7;       // shares are counted in 1/256 of a block
  if (const int most = tiles0 + tiles1 * kb1 / 4; most < groups) groups = most > 0 ? most : 1;

  GemmLaunch<2> g;
  std::memset(&g, 0, sizeof(g));
  int r;
  if ((r = make_tmap_bf16_2d(&g.a[0], dY, n, rows, ldy, BK, BM)) || (r = make_tmap_bf16_2d(&g.b[0], W, k, n, ldw, 64, BK)) ||
      (r = make_tmap_bf16_2d(&g.a[1], dY, n, rows, ldy, 64, BK)) || (r = make_tmap_bf16_2d(&g.b[1], X, k, rows, ldx, 64, BK)) ||
      (r = make_tmap_out(&g.c[0], dX, k, rows, lddx, false)) || (r = make_tmap_out(&g.c[1], dW, k, n, lddw, true)))
    return r;
  if (dgelu && !narrow && (r = make_tmap_out(&g.aux, aux, k, rows, ldaux, false))) return r;
  GemmParams& p = g.p[0];
  p.M = rows; p.N = k; p.K = n; p.a_mn = 0; p.b_mn = 1; p.C = dX; p.ldc = lddx; p.epi = epi; p.aux = const_cast<void*>(aux); p.ldaux = ldaux;
  p.split_k = 1; p.c_mode = narrow ? 0 : 1; p.aux_tma = dgelu && !narrow ? 2 : 0;
  p.kind = narrow ? kEpiDirect : !dgelu ? kEpiPlain : epi == FB_EPI_DGELU_ERF ? kEpiDgelu : kEpiDgeluTanh;
  p.band = band_of(k, tn); p.status = status; p.alpha = alpha;
  GemmParams& q = g.p[1];
  q.alpha = alpha;
  q.M = n; q.N = k; q.K = rows; q.a_mn = 1; q.b_mn = 1; q.C = dW; q.ldc = lddw; q.c_fp32 = 1; q.accumulate = 1; q.split_k = 1; q.c_mode = narrow ? 0 : 2;
  q.kind = narrow ? kEpiDirect : kEpiF32; q.band = band_of(k, tn); q.status = status;
  const long long total = static_cast<long long>(tiles1) * kb1;
  g.ahead = tiles0 % groups;
  const long long rest = groups - g.ahead, level = g.ahead ? cost : 0;
  g.share_ahead = total > rest * level ? static_cast<int>((total - rest * level) * 256 / groups) : 0;
  g.share = static_cast<int>((total * 256 - static_cast<long long>(g.ahead) * g.share_ahead) / rest);
  g.sum_x = static_cast<const __nv_bfloat16*>(dY); g.sum_out = db; g.sum_rows = rows; g.sum_cols = n; g.sum_ld = ldy;
  if (narrow) return launch_gemm<1, 64, 2>(g, groups, static_cast<cudaStream_t>(stream_));
  return launch_gemm<2, 256, 2>(g, groups, static_cast<cudaStream_t>(stream_));
}

// dX = alpha dY W where few rows make few tiles of a long reduction: the parts into which it is cut go to a scratch, in fp32, and are summed from there
// in their order, so that two calls give the same bits (added to one buffer as they came, three parts and more did not).
// With `counts`, only the first counts[0] rows take part, and row i's sum goes to row idx[i] of dX.
namespace fb {
namespace {
constexpr int kPartTile = 256;

__host__ __device__ constexpr int tiles_of(int n) { return (n + kPartTile - 1) / kPartTile; }

// Rows of the scratch for up to M rows: tiles * parts is at most what there are pairs, unless there is one part.
long long part_rows(int M, int N, int K, bool counted, int groups) {
  const int num_m = tiles_of(M), num_n = tiles_of(N), num_kb = (K + BK - 1) / BK;
  if (!counted) return static_cast<long long>(parts_for(num_m * num_n, num_kb, groups)) * num_m * kPartTile;
  const long long spread = groups / num_n, most = static_cast<long long>(num_m) * (num_kb / kPartBlocks);
  const long long parted = spread < most ? spread : most;
  return (parted > num_m ? parted : num_m) * kPartTile;
}

// Four columns a thread, up to eight parts in flight. Where that leaves threads without work, four of them take every fourth part each and meet in
// shared memory, in their order. One part is bf16 already and only goes to its place.
// A chain of latencies: the grid is what two waves hold, so that many rows are walked and few are shared. The whole of fb_gemm_parts, us, a block for every
// 64 quads instead: 2048 x 768 x 8200 26.5 (45.5), 4096 x 768 x 30522 with 614 rows 38.0 (63.3); without the four lanes 64 x 768 x 50257 20.6 (27.8).
constexpr int kSumThreads = 256, kSumLanes = 4, kSumBlocks = 8;
__global__ void __launch_bounds__(kSumThreads, 4) sum_parts_kernel(const float* __restrict__ parts, int rows, int cols, int num_kb, int groups,
                                                                            const int* __restrict__ idx, const int* __restrict__ counts,
                                                                            __nv_bfloat16* __restrict__ dx, long long ld) {
  __shared__ float4 meet[kSumLanes - 1][kSumThreads / kSumLanes];
  pdl_entry();
  if (counts) (void)FB_INDEX_OK(counts[0], static_cast<long long>(rows) + 1, 107);
  const int m = counts ? max(0, min(rows, counts[0])) : rows, quads = cols / 4, num_m = tiles_of(m), n = parts_for(num_m * tiles_of(cols), num_kb, groups);
  const long long stride = static_cast<long long>(num_m) * kPartTile * cols, items = static_cast<long long>(m) * quads;
  const auto put = [&](long long item, uint2 v) {
    const long long row = item / quads, to = idx ? idx[row] : row;
    if (FB_INDEX_OK(to, rows, 108)) *reinterpret_cast<uint2*>(dx + to * ld + (item - row * quads) * 4) = v;
  };
  const auto sum_of = [&](long long item, int first, int step) {
    const float4* p = reinterpret_cast<const float4*>(parts + item * 4);
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = first; i < n; i += 8 * step) {
      float4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (i + j * step < n) v[j] = p[(i + j * step) * (stride / 4)];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (i + j * step < n) { sum.x += v[j].x; sum.y += v[j].y; sum.z += v[j].z; sum.w += v[j].w; }
    }
    return sum;
  };
  const auto pack = [](float4 v) { return make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w)); };
  if (n == 1 || items * kSumLanes > static_cast<long long>(gridDim.x) * kSumThreads) {
    for (long long item = static_cast<long long>(blockIdx.x) * kSumThreads + threadIdx.x; item < items; item += static_cast<long long>(gridDim.x) * kSumThreads)
      put(item, n == 1 ? reinterpret_cast<const uint2*>(parts)[item] : pack(sum_of(item, 0, 1)));
    return;
  }
  const int quad = threadIdx.x % (kSumThreads / kSumLanes), lane = threadIdx.x / (kSumThreads / kSumLanes);
  const long long item = static_cast<long long>(blockIdx.x) * (kSumThreads / kSumLanes) + quad;
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
  if (item < items) sum = sum_of(item, lane, kSumLanes);
  if (lane) meet[lane - 1][quad] = sum;
  __syncthreads();
  if (lane || item >= items) return;
#pragma unroll
  for (int j = 0; j < kSumLanes - 1; ++j) {
    const float4 v = meet[j][quad];
    sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
  }
  put(item, pack(sum));
}
}  // namespace
}  // namespace fb

extern "C" int fb_gemm_part_count(int M, int N, int K, int groups) {
  using namespace fb;
  return parts_for(tiles_of(M) * tiles_of(N), (K + BK - 1) / BK, groups);
}

extern "C" long long fb_gemm_part_rows(int M, int N, int K, int counted, int groups) { return fb::part_rows(M, N, K, counted != 0, groups); }

// Rows of scratch for a reduction in parts, 0 where one product serves better. Parts save K blocks that run one after the other, `chain` in the kernel
// that would take the product otherwise, and cost the scratch and a launch, about the time of 20 blocks; a cluster of two pairs saves as much as two parts.
// us against one product, rows x columns x reduction: 64 x 128 x 18440 11.5 (13.6), 256 x 512 x 32000 16.1 (23.6), 512 x 512 x 32000 23.7 (40.3),
// 1024 x 512 x 32000 34.1 (77.6), 2048 x 512 x 32000 56.7 (93.4), 2048 x 768 x 8200 26.6 (27.0); left: 256 x 512 x 8200 13.3 (12.7), 512 x 512 x 8200 14.1 (14.8),
// 64 x 512 x 2056 12.4 (4.9). Counted rows are taken for a sixth of M here (a masked-LM batch has about that many labels); the device then cuts for what it
// counts, so that a wrong guess costs little. With the zero fill and the scatter, 4096 x 768 x 30522 of which 614 38.0 (147.5), all 158.5 (157.3); 8192 x
// 768 x 30522, 1228 57.8 (154), all 329 (330); 24576 x 512 x 32000, 3686 106.7 (184), all 588 (605); 1024 x 512 x 2056, 153 rows, left, 16.8 (14.4).
extern "C" long long fb_gemm_parts_apply(int M, int N, int K, int counted) {
  using namespace fb;
  if (M <= 0 || N <= 0 || K <= 0 || N % 8) return 0;
  const int groups = sm_count() / 2, num_kb = (K + BK - 1) / BK;
  const int parts = fb_gemm_part_count(counted ? (M + 5) / 6 : M, N, K, groups), small = counted ? 0 : gemm_small_split(M, N, K);
  const int chain = small ? (num_kb + small - 1) / small : !counted && split_applies(M, N, K) ? (num_kb + 1) / 2 : num_kb;
  if (parts < (counted ? 2 : 3) || chain - num_kb / parts < 20) return 0;
  return part_rows(M, N, K, counted != 0, groups);
}

extern "C" int fb_gemm_parts(const void* dY, const void* W, void* dX, float* scratch, int M, int N, int K, long long ldy, long long ldw, long long ldx, const float* alpha,
                             const int* idx, const int* counts, int* status, void* stream_) {
  using namespace fb;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (ldy % 8 || ldw % 8 || N % 8 || ldx % 4 || (reinterpret_cast<uintptr_t>(dY) & 15) || (reinterpret_cast<uintptr_t>(W) & 15) || (reinterpret_cast<uintptr_t>(dX) & 7) ||
      (reinterpret_cast<uintptr_t>(scratch) & 15) || !idx != !counts)
    return -3;
  const int groups = sm_count() / 2, num_kb = (K + BK - 1) / BK;
  const long long quads = (static_cast<long long>(M) * (N / 4) + kSumThreads / kSumLanes - 1) / (kSumThreads / kSumLanes);
  const int blocks = quads < kSumBlocks * sm_count() ? static_cast<int>(quads) : kSumBlocks * sm_count();
  GemmLaunch<1> g;
  std::memset(&g, 0, sizeof(g));
  int r;
  if ((r = make_tmap_bf16_2d(&g.a[0], dY, K, M, ldy, BK, BM)) || (r = make_tmap_bf16_2d(&g.b[0], W, N, K, ldw, 64, BK)) ||
      (r = make_tmap_out(&g.c[0], scratch, N, part_rows(M, N, K, counts != nullptr, groups), N, true)) || (r = make_tmap_out(&g.aux, scratch, N, M, N, false)))
    return r;
  GemmParams& p = g.p[0];
  p.M = M; p.N = N; p.K = K; p.b_mn = 1; p.C = scratch; p.ldc = N; p.c_fp32 = 1; p.alpha = alpha; p.split_k = 1; p.part_groups = groups; p.c_mode = 1; p.kind = kEpiF32;
  p.band = band_of(N, kPartTile); p.status = status; p.m_dyn = counts;
  const long long units = static_cast<long long>(tiles_of(M)) * tiles_of(N) * (counts ? groups : parts_for(tiles_of(M) * tiles_of(N), num_kb, groups));
  if ((r = launch_gemm<2, 256, 1, true>(g, units < groups ? static_cast<int>(units) : groups, stream))) return r;
  launch_pdl(sum_parts_kernel, dim3(blocks), dim3(kSumThreads), 0, stream, scratch, M, N, num_kb, groups, idx, counts,
             static_cast<__nv_bfloat16*>(dX), ldx);
  return static_cast<int>(cudaGetLastError());
}

FB_BOUNDS_ATTACH(gemm)
